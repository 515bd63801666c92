// traverse_walk.cuh — external-sampling traversal, every warp on its own trees.
//
// The same player-update as k_traverse_es and the level kernels (a traversal's
// tree, cfr_gpu.cu:644-860, cut into *seeds* at the updating player's decision
// nodes: a traversal's root, or a node's state after one of its legal actions),
// in one launch.  A warp takes roots from a counter and keeps everything its
// trees need to itself:
//   * a stack of seeds in shared memory; an idle lane takes the newest one, loads
//     its parent's 128-byte record and walks the opponents' sampled nodes until a
//     terminal or the next updating-player node;
//   * a pool of node records (betting state, row, children's values) in global
//     memory that stays in L1/L2 because the newest records are reused first;
//   * per open node a count of children still out; the lane that delivers the
//     last value lists the node as ready.  32 ready nodes at a time are regret
//     matched, added to their rows and handed to their own parents;
//   * queues of showdowns and of visits off a row's canonical mask, worked off 32 at
//     a time: each takes hundreds of instructions that few lanes of a step need.
// So no lane waits for a level of the whole update, no counter in global memory
// is shared but the roots', and an update is one launch whatever its depth,
// which is what small updates cost in the level form (38 dependent launches).
// Taking the newest seed first bounds the pool: a seed is taken only while the
// pool could still hold one node for every lane that walks and one per remaining
// decision; with no lane walking one seed at a time always fits (depth first).
//
// A step of the warp: fill idle lanes, apply the lanes' pending actions and sort
// out terminals (their lanes are filled again, until enough lanes stand at a
// decision), then the decisions together: legal mask, key, and for opponents the
// row's sector, the draw and the sampled action.  The betting state is packed
// two seats to a word and the seats still to act are a mask searched from the
// seat after the last actor (seats act in cyclic order), so that no per-player
// array is indexed.
//
// Every sum that reaches the table is an integer (fixed point) and every draw is
// keyed by the node's action path, so the rows after an update are those of the
// other forms, bit for bit, whatever the order of the walks.
//
// What bounds it: the dependent issue of a step's code (about 1,450 instructions for
// 23 decisions; 41% of issue slots, no unit above half its rate) and, in tables far
// beyond L2, random 64-byte accesses: 16 G visits/s in a 33 MB table, 10 G in one of
// 17 GB.  6-max 100BB at 2^20 traversals per update takes the level kernels 12.5 ms
// in iteration 6 and 16.4 in the mean of iterations 6-25, this one 5.6 and 7.0; a
// 1,000-traversal heads-up update took them 220 us and takes this one 60 us.  Six blocks of 80 registers per SM:
// five and seven are within 3%, eight spill and are 5% slower.
#pragma once
#include "game.cuh"
#include "table.cuh"
#include "traverse_ref.cuh"
#include "traverse_es.cuh"
#include "traverse_levels.cuh"

namespace mccfr {

constexpr int kWalkBlock = 128;
constexpr int kWalkWarps = kWalkBlock / 32;
constexpr int kWalkNodes = 192;                  // open updating-player nodes of a warp (128: heads-up 15% slower)
constexpr int kWalkSeeds = kSlots * kWalkNodes;  // their children not yet taken
constexpr int kWalkQueue = 64;                   // queue entries: 31 left over + 32 of one step
constexpr int kWalkReady = 24;                   // lanes at a decision that end the filling of a step (28: up to 7% slower, 20: equal)
constexpr uint32_t kWalkRoot = 0xFFFFu;          // parent of a traversal's root

// Counters of one update, zeroed by the deal that precedes the walk.
struct WalkCtl {
  unsigned work;                // traversals handed out
  unsigned pad[31];
  uint32_t nodes[kMaxLevels];   // updating-player nodes reached from each level's seeds
  uint32_t seeds[kMaxLevels];   // their children (seeds of the next level)
};

// Betting state of a lane's walk.
//   seats = folded | all-in << 8 | still to act << 16 | seat to search from << 24
//   prog  = street | dealer << 4 | raises << 8 | depth << 16 | level << 24
struct WalkState {
  uint32_t inv0, inv1, inv2, bet0, bet1, bet2;  // chips in the hand and in this street, two seats per word
  int pot, cb;
  uint64_t path;
  int lfr;
  uint32_t abits;
  uint32_t aux;  // traversal
  uint32_t seats, prog;
};

// An open updating-player node: its state, row, own seed, and children's values.
struct __align__(128) WalkNode {
  Sector a;   // inv0, inv1 | inv2, bet0 | bet1, bet2 | pot, cb
  Sector b;   // path | lfr, abits | aux, seats | prog, row slot
  Sector v;   // children's values, by action
  uint2 own;  // parent record << 3 | action (its own seed), legal mask
};
static_assert(sizeof(WalkNode) == 128, "a node record is one line");

struct WalkShowdown {
  uint32_t ref, aux, inv0, inv1, inv2;  // ref: seed | folded << 16
};

// A warp's own lists.
struct WalkWarp {
  uint16_t seeds[kWalkSeeds];          // record << 3 | action
  uint16_t spare[kWalkNodes];          // free records
  uint16_t ready[kWalkNodes];          // nodes whose children are all in
  uint32_t out[kWalkNodes / 8];        // children still out, 4 bits per record
  WalkShowdown show[kWalkQueue];
  uint2 off[kWalkQueue];               // row slot, legal mask
  unsigned roots, full;                // traversals taken, updating-player nodes that found no row
};

struct WalkBufs {
  WalkNode* nodes;  // [warps][kWalkNodes]
  WalkCtl* ctl;
  int decisions;    // most updating-player decisions on a path
  int grab;         // traversals a warp takes at a time
};

__device__ __forceinline__ int seat16(uint32_t w0, uint32_t w1, uint32_t w2, int p) {
  const uint32_t w = p < 2 ? w0 : (p < 4 ? w1 : w2);
  return (int)((w >> ((p & 1) << 4)) & 0xFFFFu);
}

// Adds x to seat p's half word (sums stay below 2^16).
__device__ __forceinline__ void seat16_add(uint32_t& w0, uint32_t& w1, uint32_t& w2, int p, uint32_t x) {
  const uint32_t d = x << ((p & 1) << 4);
  w0 += p < 2 ? d : 0u;
  w1 += (p >> 1) == 1 ? d : 0u;
  w2 += p >= 4 ? d : 0u;
}

// Root state of traversal t (es_begin).
__device__ __forceinline__ void walk_root(const GameParams& G, const DealRec* D, uint32_t t, WalkState& s) {
  const int N = G.N;
  const int dealer = D->dealer;
  const uint32_t all = (1u << N) - 1;
  s.aux = t;
  s.inv0 = s.inv1 = s.inv2 = s.bet0 = s.bet1 = s.bet2 = 0;
  s.abits = 0;
  s.path = kPathSeed;
  s.lfr = G.bb;
  if (G.sub_street) {
    const uint32_t x = (uint32_t)(G.sub_pot / N), xx = x | (x << 16);
    s.inv0 = xx;
    s.inv1 = N > 3 ? xx : (N > 2 ? x : 0u);
    s.inv2 = N > 5 ? xx : (N > 4 ? x : 0u);
    s.pot = G.sub_pot;
    s.cb = 0;
    s.seats = (all << 16) | ((uint32_t)seat_after(dealer, 1, N) << 24);
    s.prog = (uint32_t)G.sub_street | ((uint32_t)dealer << 4);
  } else {
    const int next = seat_after(dealer, 1, N);
    const int sbp = N == 2 ? dealer : next;
    const int bbp = N == 2 ? next : seat_after(next, 1, N);
    const int sba = min(G.sb, G.stack), bba = min(G.bb, G.stack);
    seat16_add(s.bet0, s.bet1, s.bet2, sbp, (uint32_t)sba);
    seat16_add(s.bet0, s.bet1, s.bet2, bbp, (uint32_t)bba);
    s.inv0 = s.bet0;
    s.inv1 = s.bet1;
    s.inv2 = s.bet2;
    s.pot = sba + bba;
    s.cb = bba;
    uint32_t allin = 0;
    if (G.stack == sba) allin |= 1u << sbp;
    if (G.stack == bba) allin |= 1u << bbp;
    s.seats = (allin << 8) | ((all & ~allin) << 16) | ((uint32_t)seat_after(bbp, 1, N) << 24);
    s.prog = (uint32_t)dealer << 4;
  }
}

// Next seat to act: the first of `mask` at or after `from`, cyclically.
__device__ __forceinline__ int walk_next(uint32_t seats, int N) {
  const uint32_t mask = (seats >> 16) & 0xFFu;
  const int from = (int)(seats >> 24);
  return seat_after(from, __ffs((int)((mask | (mask << N)) >> from)) - 1, N);
}

// Applies action a of `player` (es_apply).  FNV: the game's keys may be FNV slots,
// which hash the last ten actions; the walk of path-hash keys carries no abits.
template <bool FNV>
__device__ __forceinline__ void walk_apply(const GameParams& G, WalkState& s, int player, int a) {
  const int N = G.N;
  const uint32_t bit = 1u << player;
  const int after = seat_after(player, 1, N);
  if (FNV) s.abits = ((s.abits << 3) | (uint32_t)a) & 0x3FFFFFFFu;
  s.path = path_step(s.path, a);
  s.prog += 1u << 16;  // depth
  uint32_t folded = s.seats & 0xFFu, allin = (s.seats >> 8) & 0xFFu, act = ((s.seats >> 16) & 0xFFu) & ~bit;
  const int k = G.kind[a];
  if (k == 0) {
    folded |= bit;
  } else if (k != 1) {
    const int pbet = seat16(s.bet0, s.bet1, s.bet2, player);
    const int pstack = G.stack_base - seat16(s.inv0, s.inv1, s.inv2, player);
    const int chips = chips_for(G, a, s.pot, pstack, s.cb - pbet, s.cb, s.lfr);
    seat16_add(s.bet0, s.bet1, s.bet2, player, (uint32_t)chips);
    seat16_add(s.inv0, s.inv1, s.inv2, player, (uint32_t)chips);
    s.pot += chips;
    if (pstack == chips) allin |= bit;
    const int nbet = pbet + chips;
    if (nbet > s.cb) {
      const int rs = nbet - s.cb;
      if (rs >= s.lfr || s.cb == 0) s.lfr = rs;
      s.cb = nbet;
      s.prog = (s.prog & ~0xFF00u) | ((s.prog + 0x100u) & 0xFF00u);  // raises, modulo 256
      act = ((1u << N) - 1) & ~(folded | allin | bit);
    }
  }
  s.seats = folded | (allin << 8) | (act << 16) | ((uint32_t)after << 24);
}

// Sorts out what follows an applied action: kLvDone with the terminal's value,
// kLvShow for a showdown, kLvGoOn at a decision node (after a street change
// where one is due).
__device__ __forceinline__ int walk_events(const GameParams& G, WalkState& s, int up, float& value) {
  const int N = G.N;
  const uint32_t live = ((1u << N) - 1) & ~s.seats;
  value = 0.0f;
  if ((int)((s.prog >> 16) & 0xFFu) >= G.max_depth) return kLvDone;
  if ((live & (live - 1)) == 0) {
    const int inv_up = seat16(s.inv0, s.inv1, s.inv2, up);
    value = (live >> up) & 1 ? (float)(s.pot - inv_up) : (float)(-inv_up);
    return kLvDone;
  }
  if (s.seats & 0x00FF0000u) return kLvGoOn;
  if ((s.prog & 0xFu) >= 3u) return kLvShow;
  const uint32_t act = live & ~(s.seats >> 8);
  if (!act) return kLvShow;
  s.bet0 = s.bet1 = s.bet2 = 0;
  s.cb = 0;
  s.lfr = G.bb;
  s.prog = (s.prog + 1u + (1u << 16)) & ~0xFF00u;  // street and depth on, no raises
  s.seats = (s.seats & 0xFFFFu) | (act << 16) | ((uint32_t)seat_after((int)((s.prog >> 4) & 0xFu), 1, N) << 24);
  return (int)((s.prog >> 16) & 0xFFu) >= G.max_depth ? kLvDone : kLvGoOn;
}

// Side-pot payoff of the updating player (side_pot_payoff).  A folded player, or
// one beaten by a live seat with at least its chips, loses what it put in; one
// that no live seat ties or beats takes its share of every seat's chips (sums of
// whole chips below 2^24, exact in any order).  Only ties, and wins over some of
// the side pots, need the pots one by one.
__device__ __forceinline__ float walk_showdown(int N, int up, uint32_t folded, uint32_t inv0, uint32_t inv1,
                                               uint32_t inv2, const DealRec* D) {
  const uint2 k01 = __ldg(reinterpret_cast<const uint2*>(D->rank));
  const uint32_t k2 = __ldg(reinterpret_cast<const uint32_t*>(D->rank + 4));
  const int mine = seat16(inv0, inv1, inv2, up), rank = seat16(k01.x, k01.y, k2, up);
  // (no chips in: the pots leave the negative zero that they start from)
  bool beaten = ((folded >> up) & 1) || mine == 0, contested = false;
  int take = 0;
#pragma unroll
  for (int q = 0; q < kMaxPlayers; ++q) {
    if (q >= N) break;
    const int iq = (int)(((q < 2 ? inv0 : q < 4 ? inv1 : inv2) >> (16 * (q & 1))) & 0xFFFFu);
    const int rq = (int)(((q < 2 ? k01.x : q < 4 ? k01.y : k2) >> (16 * (q & 1))) & 0xFFFFu);
    const bool live = q != up && !((folded >> q) & 1);
    take += min(iq, mine);
    contested |= live && rq >= rank;
    beaten |= live && rq > rank && iq >= mine;
  }
  if (beaten) return -(float)mine;
  if (!contested) return (float)(take - mine);
  return lv_showdown(N, up, folded, inv0, inv1, inv2, D);
}

// A warp's lists as walk_update expects and leaves them.
__device__ __forceinline__ void walk_init(WalkWarp& W) {
  const int lane = threadIdx.x & 31;
  for (int i = lane; i < kWalkNodes; i += 32) W.spare[i] = (uint16_t)(kWalkNodes - 1 - i);
  for (int i = lane; i < kWalkNodes / 8; i += 32) W.out[i] = 0;
  if (lane == 0) W.roots = W.full = 0;
  __syncwarp();
}

// The walk of one table's update by one warp, until no traversal is left to take
// and all that it took are done.  `levels` (may be null): the block's level counts.
template <bool DIRECT, bool FNV>
__device__ __forceinline__ void walk_update(const GameParams& G, const TableView& tv, const DealRec* __restrict__ deals,
                                            int up, uint32_t uid, uint32_t epoch, int batch, float rscale, int grab,
                                            int decisions, unsigned* work, Counters* counters, WalkWarp& W,
                                            WalkNode* const pool, uint32_t* s_nodes, uint32_t* s_seeds) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int N = G.N;
  // warp-uniform list lengths and counters
  int n_seeds = 0, n_spare = kWalkNodes, n_ready = 0, n_show = 0, n_off = 0;
  unsigned c_vis = 0, c_nodes = 0, c_kids = 0;
  bool more = true;  // roots may be left
  int stalled = 0;
  // the lane's walk: idle, an action to apply, or standing at a decision
  enum { kIdle = 0, kApply = 1, kDecide = 2 };
  int st = kIdle;
  WalkState s;
  uint32_t ref = kWalkRoot;  // its seed
  int pl = -1, pa = 0;       // pending action (pl < 0: a root, nothing to apply), or the seat to act
  uint32_t cw = 0;           // that seat's cards (DealRec::ctx)

  // Hands lane values to their parents (ref), listing nodes whose last child it was.
  auto deliver = [&](bool on, float v) {
    const bool has = on && ref != kWalkRoot;
    if (has) reinterpret_cast<float*>(&pool[ref >> 3].v)[ref & 7] = v;
    __syncwarp();
    bool last = false;
    if (has) {
      const unsigned sh = 4u * ((ref >> 3) & 7u);
      last = ((atomicSub(&W.out[ref >> 6], 1u << sh) >> sh) & 15u) == 1u;
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, last);
    if (last) W.ready[n_ready + __popc(m & below)] = (uint16_t)(ref >> 3);
    n_ready += __popc(m);
    __syncwarp();
  };

  for (;;) {
    const unsigned idlem = __ballot_sync(0xFFFFFFFFu, st == kIdle);
    const int n_idle = __popc(idlem);
    const bool starved = n_idle == 32 && n_seeds == 0 && !more;
    // seeds the pool has room for: every walking lane may still open one node,
    // and one seed walked depth first opens one per decision
    const int room = n_spare - (32 - n_idle) - decisions;
    const bool low = room < 1;

    if (n_show >= 32 || (n_show && (starved || low))) {
      // showdowns, one per lane
      const int nb = min(32, n_show);
      n_show -= nb;
      const bool on = lane < nb;
      const WalkShowdown r = W.show[n_show + (on ? lane : 0)];
      const uint32_t keep = ref;
      float v = 0.0f;
      if (on) {
        v = walk_showdown(N, up, r.ref >> 16, r.inv0, r.inv1, r.inv2, deals + r.aux);
        ref = r.ref & 0xFFFFu;
      }
      deliver(on, v);
      ref = keep;
      continue;
    }
    if (n_ready >= 32 || (n_ready && (starved || low))) {
      // ready nodes, one per lane: regret matching, row sums, own value
      const int nb = min(32, n_ready);
      n_ready -= nb;
      const bool on = lane < nb;
      const uint32_t keep = ref;
      float vh = 0.0f;
      uint32_t id = 0;
      if (on) {
        id = W.ready[n_ready + lane];
        const WalkNode* nd = pool + id;
        const unsigned long long slot = nd->b.w >> 32;
        const uint2 own = nd->own;
        const uint32_t vm = own.y;
        const unsigned long long k = __ldcg(row_key(tv, slot));
        float reg[kSlots], strat[kSlots], v[kSlots];
        load_regrets(tv, (long long)slot, reg);
        const Sector cv = ld_own_sector(&nd->v);
        v[0] = lo_float(cv.x); v[1] = hi_float(cv.x); v[2] = lo_float(cv.y); v[3] = hi_float(cv.y);
        v[4] = lo_float(cv.z); v[5] = hi_float(cv.z); v[6] = lo_float(cv.w); v[7] = hi_float(cv.w);
        // a direct-mapped row's key was left to this pass
        if (DIRECT && k != slot + 1) __stcg(row_key(tv, slot), slot + 1);
        mark_wide(tv, slot);
        node_strategy(reg, vm, strat);
#pragma unroll
        for (int a = 0; a < kSlots; ++a)
          if ((vm >> a) & 1) vh = __fadd_rn(vh, __fmul_rn(strat[a], v[a]));
        const long long fv = fix_r(vh, rscale);
#pragma unroll
        for (int a = 0; a < kSlots; ++a)
          if ((vm >> a) & 1) atomicAdd(row_da(tv, slot) + a, (unsigned long long)(fix_r(v[a], rscale) - fv));
        atomicAdd(row_cnt(tv, slot), 1ull << 32);
        ref = own.x;
      }
      __syncwarp();
      if (on) W.spare[n_spare + lane] = (uint16_t)id;
      n_spare += nb;
      deliver(on, vh);
      ref = keep;
      continue;
    }
    if (n_off >= 32 || (n_off && starved)) {
      // visits off the canonical mask: every legal slot's strategy weight
      const int nb = min(32, n_off);
      n_off -= nb;
      if (lane < nb) {
        const uint2 e = W.off[n_off + lane];
        float reg[kSlots], strat[kSlots];
        load_regrets(tv, (long long)e.x, reg);
        node_strategy(reg, e.y, strat);
        atomicOr(row_flags(tv, e.x), kFlagDs);
        atomicAdd(row_cnt(tv, e.x), 1ull << 32);
#pragma unroll
        for (int a = 0; a < kSlots; ++a)
          if ((e.y >> a) & 1) {
            const long long d = fix_s(strat[a]);
            if (d) atomicAdd(row_ds(tv, e.x) + a, (unsigned long long)d);
          }
      }
      __syncwarp();
      continue;
    }
    if (starved) break;

    // ---- fill idle lanes: the newest seeds, else new roots
    bool filled = false;
    if (n_idle) {
      const int allowed = n_idle == 32 ? max(room, 1) : room;
      const int rank = __popc(idlem & below);
      const int take = min(min(n_idle, n_seeds), allowed);
      if (take > 0) {
        n_seeds -= take;
        if (st == kIdle && rank < take) {
          ref = W.seeds[n_seeds + take - 1 - rank];
          const WalkNode* nd = pool + (ref >> 3);
          const Sector a = ld_own_sector(&nd->a), b = ld_own_sector(&nd->b);
          s.inv0 = (uint32_t)a.x; s.inv1 = (uint32_t)(a.x >> 32); s.inv2 = (uint32_t)a.y; s.bet0 = (uint32_t)(a.y >> 32);
          s.bet1 = (uint32_t)a.z; s.bet2 = (uint32_t)(a.z >> 32); s.pot = (int)(uint32_t)a.w; s.cb = (int)(a.w >> 32);
          s.path = b.x;
          s.lfr = (int)(uint32_t)b.y;
          if (FNV) s.abits = (uint32_t)(b.y >> 32);
          s.aux = (uint32_t)b.z; s.seats = (uint32_t)(b.z >> 32); s.prog = (uint32_t)b.w;
          s.prog += 1u << 24;  // one level down
          pl = up;
          pa = (int)(ref & 7u);
          st = kApply;
        }
        filled = true;
      } else if (n_seeds == 0 && more && allowed > 0) {
        const int want = min(min(n_idle, allowed), grab);
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(work, (unsigned)want);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        const int got = base < (unsigned)batch ? min(want, (int)((unsigned)batch - base)) : 0;
        if (got < want) more = false;
        if (st == kIdle && rank < got) {
          walk_root(G, deals + base + rank, base + (uint32_t)rank, s);
          ref = kWalkRoot;
          pl = -1;
          st = kApply;
        }
        if (lane == 0) W.roots += got;
        filled = got > 0;
      }
    }

    // ---- pending actions and what follows from them
    if (__any_sync(0xFFFFFFFFu, st == kApply)) {
      stalled = 0;
      int r = -1;
      float v = 0.0f;
      if (st == kApply) {
        if (pl >= 0) walk_apply<FNV>(G, s, pl, pa);
        r = walk_events(G, s, up, v);
        st = kIdle;
        if (r == kLvGoOn) {
          st = kDecide;
          pl = walk_next(s.seats, N);
          cw = __ldg(deals[s.aux].ctx + pl);
        }
      }
      const unsigned showm = __ballot_sync(0xFFFFFFFFu, r == kLvShow);
      const unsigned donem = __ballot_sync(0xFFFFFFFFu, r == kLvDone);
      if (r == kLvShow) {
        WalkShowdown& q = W.show[n_show + __popc(showm & below)];
        q.ref = ref | (s.seats << 16);
        q.aux = s.aux;
        q.inv0 = s.inv0;
        q.inv1 = s.inv1;
        q.inv2 = s.inv2;
      }
      n_show += __popc(showm);
      if (donem) deliver(r == kLvDone, v);
      __syncwarp();
    }
    // lanes freed by terminals are filled again before the decisions run
    const unsigned decm = __ballot_sync(0xFFFFFFFFu, st == kDecide);
    if (filled && __popc(decm) < kWalkReady && (n_seeds > 0 || more)) continue;
    if (!decm) {
      // every round of the loop above takes, fills or finishes something; a round
      // that does not would never end
      if (++stalled > 8) {
        if (lane == 0) atomicOr(tv.err, kErrStackOverflow);
        break;
      }
      continue;
    }

    // ---- decisions
    bool isup = false, off = false;
    uint32_t vm = 0;
    long long slot = -1;
    c_vis += __popc(decm);
    if (st == kDecide) {
      const int player = pl;
      const int street = (int)(s.prog & 0xFu);
      const int to_call = s.cb - seat16(s.bet0, s.bet1, s.bet2, player);
      vm = valid_mask(G, s.pot, G.stack_base - seat16(s.inv0, s.inv1, s.inv2, player), to_call, s.cb, s.lfr,
                      (int)((s.prog >> 8) & 0xFFu));
      uint32_t hb, bkt;
      if (G.sub_street) {  // exact combo; the river card once it is dealt
        hb = cw & 0xFFFF;
        bkt = (street == 3 && G.sub_street == 2) ? (cw >> 16) : 0u;
      } else {
        hb = cw & 0xFF;
        bkt = street ? ((cw >> (8 * street)) & 0xFF) : 0u;
      }
      const unsigned long long key = FNV ? info_key(G, player, hb, bkt, street, s.abits, s.path)
                                         : id64_key(G, player, hb, bkt, street, s.path);
      isup = player == up;
      // in a direct-mapped table the updating player's row is left to the ready pass
      slot = DIRECT ? (long long)(key - 1) : table_insert<1>(tv, key);
      if (!isup) {
        const bool ok = DIRECT || slot >= 0;
        Sector row{0ull, 0ull, 0ull, 0ull};  // key, tag, strategy
        if (ok) row = ld_sector(row_ptr(tv, (unsigned long long)slot));
        const U4 d = philox(U4{s.aux, uid, (uint32_t)s.path, (uint32_t)(s.path >> 32) | 0x80000000u}, G.seed_lo,
                            G.seed_hi);
        if (DIRECT && row.x != key) __stcg(row_key(tv, (unsigned long long)slot), key);
        pa = sample_stored(G, make_uint4((uint32_t)row.z, (uint32_t)(row.z >> 32), (uint32_t)row.w,
                                         (uint32_t)(row.w >> 32)), vm, uniform01(d.x));
        st = kApply;
        if (ok) {
          if (touch_row_from(tv, (unsigned long long)slot, epoch, vm, row.y))
            atomicAdd(row_cnt(tv, (unsigned long long)slot), (1ull << 32) | 1ull);
          else
            off = true;
        }
      }
    }
    const unsigned offm = __ballot_sync(0xFFFFFFFFu, off);
    if (off) W.off[n_off + __popc(offm & below)] = make_uint2((uint32_t)slot, vm);
    n_off += __popc(offm);
    // other lanes read the entries, and the votes on the way there order no memory
    if (offm) __syncwarp();
    // ---- updating-player nodes: a record and one seed per legal action
    if (__any_sync(0xFFFFFFFFu, isup)) {
      const unsigned full = __ballot_sync(0xFFFFFFFFu, isup && slot < 0);  // no row: nothing to update
      bool open = isup && slot >= 0;
      unsigned upm = __ballot_sync(0xFFFFFFFFu, open);
      if (__popc(upm) > n_spare) {  // cannot happen while seeds are taken within `room`
        if (lane == 0) atomicOr(tv.err, kErrStackOverflow);
        open = false;
        upm = 0;
      }
      const int k = open ? __popc(vm) : 0;
      int before = 0, total = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const unsigned kb = __ballot_sync(0xFFFFFFFFu, (k >> b) & 1);
        before += __popc(kb & below) << b;
        total += __popc(kb) << b;
      }
      const int cnt = __popc(upm);
      // the lanes go on with their node's first action while the pool is far from full
      const bool go_on = n_spare - cnt - 32 >= decisions;
      c_nodes += cnt;
      c_kids += total;
      if (go_on) {
        before -= __popc(upm & below);
        total -= cnt;
      }
      if (open) {
        const uint32_t id = W.spare[n_spare - 1 - __popc(upm & below)];
        WalkNode* nd = pool + id;
        st_own_sector(&nd->a, Sector{two_words(s.inv0, s.inv1), two_words(s.inv2, s.bet0), two_words(s.bet1, s.bet2),
                                     two_words((uint32_t)s.pot, (uint32_t)s.cb)});
        st_own_sector(&nd->b, Sector{s.path, two_words((uint32_t)s.lfr, FNV ? s.abits : 0u), two_words(s.aux, s.seats),
                                     two_words(s.prog, (uint32_t)slot)});
        nd->own = make_uint2(ref, vm);
        atomicAdd(&W.out[id >> 3], (unsigned)k << (4u * (id & 7u)));
        int o = n_seeds + before;
        uint32_t left = vm;
        if (go_on) left &= left - 1;
        for (; left; left &= left - 1) W.seeds[o++] = (uint16_t)((id << 3) | (uint32_t)(__ffs(left) - 1));
        if (s_nodes) {
          const int level = (int)(s.prog >> 24);
          atomicAdd(&s_nodes[level], 1u);
          atomicAdd(&s_seeds[level], (unsigned)k);
        }
        if (go_on) {
          pa = __ffs((int)vm) - 1;
          ref = (id << 3) | (uint32_t)pa;
          s.prog += 1u << 24;
        }
      }
      n_spare -= cnt;
      n_seeds += total;
      __syncwarp();
      if (full) {
        deliver(isup && slot < 0, 0.0f);
        if (lane == 0) W.full += __popc(full);
      }
      if (isup) st = open && go_on ? kApply : kIdle;
    }
  }
  if (lane == 0) {
    if (W.roots) {
      atomicAdd(&counters->traversals, (unsigned long long)W.roots);
      atomicAdd(&counters->evals, (unsigned long long)W.roots * (unsigned)N);
      atomicAdd(&counters->visits, (unsigned long long)c_vis);
      // every root and seed ended at a terminal, an updating-player node, or a node
      // that found no row
      atomicAdd(&counters->terminals, (unsigned long long)W.roots + c_kids - c_nodes - W.full);
      if (c_nodes) atomicAdd(&counters->updates, (unsigned long long)c_nodes);
    }
    W.roots = W.full = 0;
  }
  __syncwarp();
  if (stalled > 8) walk_init(W);  // given up with the error flag set: nothing of this table is left in the lists
}

template <bool DIRECT, bool FNV>
__global__ void __launch_bounds__(kWalkBlock, 6)
k_walk(const GameParams G, const TableView tv, const DealRec* __restrict__ deals, const Sched* __restrict__ sched,
       int batch, float rscale, const WalkBufs wb, Counters* __restrict__ counters) {
  __shared__ WalkWarp s_warp[kWalkWarps];
  __shared__ uint32_t s_nodes[kMaxLevels], s_seeds[kMaxLevels];
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x < kMaxLevels) s_nodes[threadIdx.x] = s_seeds[threadIdx.x] = 0;
  walk_init(s_warp[warp]);
  __syncthreads();
  walk_update<DIRECT, FNV>(G, tv, deals, sched->player, update_id(sched, G.N), *table_epoch(tv), batch, rscale, wb.grab,
                      wb.decisions, &wb.ctl->work, counters, s_warp[warp],
                      wb.nodes + (size_t)(blockIdx.x * kWalkWarps + warp) * kWalkNodes, s_nodes, s_seeds);
  __syncthreads();
  if (threadIdx.x < kMaxLevels) {
    if (s_nodes[threadIdx.x]) atomicAdd(&wb.ctl->nodes[threadIdx.x], s_nodes[threadIdx.x]);
    if (s_seeds[threadIdx.x]) atomicAdd(&wb.ctl->seeds[threadIdx.x], s_seeds[threadIdx.x]);
  }
}

}  // namespace mccfr
