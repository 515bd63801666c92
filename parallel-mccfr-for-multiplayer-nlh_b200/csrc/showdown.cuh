// showdown.cuh — showdown-evaluation microbenchmark kernels.
//
// Two forms of the rank-table gathers that training's showdown rests on
// (cfr_gpu.cu:114-150 for the chains, 694-753 for the showdown):
//   * k_deal_eval7: random 7-card hands drawn on the device (counter-based
//     Philox, partial Fisher-Yates over the 52 cards, the deal's multiply-shift)
//     and ranked by 7 dependent gathers each;
//   * k_showdown_masks: the deals of a training update (deal_one's Philox words
//     and Fisher-Yates, so exactly the cards training deals), each seat's 7-card
//     rank with the 5-card board walked once and shared by every seat (5 + 2 per
//     seat gathers: the table's state depends only on the card set), and a mask
//     of the seats holding the best rank (several bits: a split pot).
// Both are gathers from a 130 MB table, whose upper states are hot: the 7-card
// kernel walks its cards in ascending order, so that the states of the first cards
// are those of few low-card sets and hit more often (2^24 hands: 0.315 ms unsorted,
// 0.270 ms sorted; 0.51 ms when the shuffle kept a list of swapped positions).  The
// six-seat kernel sorts its board and each hand (2^22 deals: 0.281 -> 0.257 ms).
#pragma once
#include "game.cuh"
#include "traverse_ref.cuh"

namespace mccfr {

constexpr uint32_t kEval7Stream = 0x300u;  // Philox counter word of the microbenchmark's hands

// The rank-table codes (to_rm) of a partial Fisher-Yates' first 7 cards, without a
// deck: draw k swaps positions k and j = k + (w_k * (52 - k)) >> 32 and yields the
// card now at position k, so a position holds its own card unless an earlier draw
// moved one there, the last such draw counting.
__device__ __forceinline__ void draw7(const uint32_t (&words)[7], int (&rm)[7]) {
  int at[7], moved[7];  // draw i moved card moved[i] to position at[i]
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    const int j = k + (int)__umulhi(words[k], (uint32_t)(52 - k));
    int cj = j, ck = k;
#pragma unroll
    for (int i = 0; i < k; ++i) {
      if (at[i] == j) cj = moved[i];
      if (at[i] == k) ck = moved[i];
    }
    at[k] = j;
    moved[k] = ck;
    rm[k] = to_rm(cj);
  }
}

// Ascending order: a 16-comparator network for seven values.
__device__ __forceinline__ void sort7(int (&v)[7]) {
  const auto cx = [&](int a, int b) {
    const int lo = min(v[a], v[b]);
    v[b] = max(v[a], v[b]);
    v[a] = lo;
  };
  cx(0, 6); cx(2, 3); cx(4, 5);
  cx(0, 2); cx(1, 4); cx(3, 6);
  cx(0, 1); cx(2, 5); cx(3, 4);
  cx(1, 2); cx(4, 6);
  cx(2, 3); cx(4, 5);
  cx(1, 2); cx(3, 4); cx(5, 6);
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_deal_eval7(const int32_t* __restrict__ T, uint32_t seed_lo, uint32_t seed_hi, uint32_t stream,
             unsigned long long n, uint16_t* __restrict__ ranks) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)BLOCK + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * BLOCK) {
    const U4 w0 = philox(U4{(uint32_t)i, stream, kEval7Stream, (uint32_t)(i >> 32)}, seed_lo, seed_hi);
    const U4 w1 = philox(U4{(uint32_t)i, stream, kEval7Stream + 1u, (uint32_t)(i >> 32)}, seed_lo, seed_hi);
    const uint32_t words[7] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z};
    int rm[7];
    draw7(words, rm);
    sort7(rm);
    int32_t p = 53;
#pragma unroll
    for (int k = 0; k < 7; ++k) p = __ldg(T + p + rm[k]);
    ranks[i] = (uint16_t)decode16((uint32_t)p & 0xFFFF);
  }
}

// The 6-seat deal draws 17 cards, too many to keep by draw: its deck lies in shared
// memory (Deck).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_showdown_masks(const GameParams G, const int32_t* __restrict__ T, uint32_t uid, unsigned n,
                 uint8_t* __restrict__ masks) {
  __shared__ uint32_t s_deck[BLOCK * kDeckWords];
  const Deck<BLOCK> deck{s_deck + threadIdx.x};
  const int N = G.N;
  for (unsigned t = blockIdx.x * BLOCK + threadIdx.x; t < n; t += gridDim.x * BLOCK) {
    deck.shuffle(G, t, uid, 2 * N + 5);
    // board first (positions 2N .. 2N+4), shared by every seat
    int rm[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) rm[i] = to_rm(deck.at(2 * N + i));
    const auto cx = [&](int x, int y) {
      const int lo = min(rm[x], rm[y]);
      rm[y] = max(rm[x], rm[y]);
      rm[x] = lo;
    };
    cx(0, 3); cx(1, 4);
    cx(0, 2); cx(1, 3);
    cx(0, 1); cx(2, 4);
    cx(1, 2); cx(3, 4);
    cx(2, 3);
    int32_t b = 53;
#pragma unroll
    for (int i = 0; i < 5; ++i) b = __ldg(T + b + rm[i]);
    uint32_t rk[kMaxPlayers];
#pragma unroll
    for (int q = 0; q < kMaxPlayers; ++q) {
      rk[q] = 0;
      if (q < N) {
        const int c0 = to_rm(deck.at(2 * q)), c1 = to_rm(deck.at(2 * q + 1));
        const int32_t s6 = __ldg(T + b + min(c0, c1));
        rk[q] = decode16((uint32_t)__ldg(T + s6 + max(c0, c1)) & 0xFFFF);
      }
    }
    uint32_t best = 0;
#pragma unroll
    for (int q = 0; q < kMaxPlayers; ++q) best = max(best, rk[q]);
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < kMaxPlayers; ++q)
      if (q < N && rk[q] == best) m |= 1u << q;
    masks[t] = (uint8_t)m;
  }
}

}  // namespace mccfr
