// Harness of tests/test_raise_target.py: host raise targets of a pot fraction.
// Reads lines "num den pot cb mrt", prints the target.
#include <cstdio>
#include <cstring>

#include "game.cuh"

int main() {
  int num, den, pot, cb, mrt;
  while (std::scanf("%d %d %d %d %d", &num, &den, &pot, &cb, &mrt) == 5) {
    mccfr::GameParams g;
    std::memset(&g, 0, sizeof(g));
    mccfr::set_pot_fraction(g, 0, num, den);
    std::printf("%d\n", mccfr::raise_target(g, 0, pot, cb, mrt));
  }
}
