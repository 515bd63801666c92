// traverse_path.cuh — traversal kernel of the reference's update rule.
//
// Under the reference's rule every node samples one action, so a traversal is a
// single root-to-terminal path and every node on it returns the terminal payoff u
// (cfr_gpu.cu:809-818).  Persistent lanes walk one path each (the packed state and
// events of traverse_walk.cuh) and take the next traversal when theirs is done, so
// that a warp does not wait for its longest path.  A sampled visit reads the row's
// stored strategy, one 16-byte load in a direct-mapped table; the updating
// player's nodes are recorded in shared memory, and lanes whose u is known wait
// for each other so that a good part of the warp folds its records together (an
// accumulator update is far more code than a step of the walk).
//
// What bounds it: instruction issue (58% of slots) with its lanes at different kinds
// of nodes (14 of 32 active); at small updates the chain of a long path's loads.
// 2^18 traversals of 6-max 100BB take 147 us (one thread per traversal: 400), 65,536
// of the reference's heads-up game 65 us (146).
#pragma once
#include "traverse_walk.cuh"

namespace mccfr {

constexpr int kPathBlock = 128;
// lanes with a known payoff that start a fold, idle lanes that start a refill (12 and
// 6: the reference's defaults 6% slower, its rule on 6-max the same; 20: 2% slower)
constexpr int kPathFold = 16;
constexpr int kPathRefill = 12;
constexpr int kMaxRec = 24;      // updating-player nodes of a path

// Adds lane's recorded nodes with payoff u to their rows.
__device__ __forceinline__ void path_fold(const TableView& tv, uint32_t epoch, float rscale, float u, int nrec,
                                          const uint32_t* slots, const uint16_t* sv, const float* qs) {
  const long long fu = fix_r(u, rscale);
  for (int i = 0; i < nrec; ++i) {
    const uint32_t slot = slots[i * kPathBlock];
    const uint32_t x = sv[i * kPathBlock];
    const int s = (int)(x & 0xFFu);
    const uint32_t vm = x >> 8;
    const long long dsamp = fix_r(__fsub_rn(__fdiv_rn(u, qs[i * kPathBlock]), u), rscale);
    mark_wide(tv, slot);
    if (touch_row(tv, slot, epoch, vm)) {
      atomicAdd(row_cnt(tv, slot), (1ull << 32) | 1ull);
      atomicAdd(row_su(tv, slot), (unsigned long long)fu);
      atomicAdd(row_da(tv, slot) + s, (unsigned long long)(dsamp + fu));
    } else {
      // mask differs from the row's canonical one (a row shared by states with
      // different legal actions): every term directly
      atomicAdd(row_cnt(tv, slot), 1ull << 32);
      float reg[kSlots], strat[kSlots];
      load_regrets(tv, slot, reg);
      node_strategy(reg, vm, strat);
      long long dr[kSlots], dw[kSlots];
#pragma unroll
      for (int a = 0; a < kSlots; ++a) {
        dr[a] = (a == s) ? dsamp : -fu;
        dw[a] = fix_s(strat[a]);
      }
      add_direct(tv, slot, vm, dr, dw);
    }
  }
}

template <bool DIRECT, bool FNV, bool TRACE>
__global__ void __launch_bounds__(kPathBlock, 6)
k_path(const GameParams G, const TableView tv, const DealRec* __restrict__ deals, const Sched* __restrict__ sched,
       int batch, float rscale, Counters* __restrict__ counters, unsigned* __restrict__ work,
       mccfr_trace* __restrict__ trace) {
  // updating-player nodes of each lane's path: slot, sampled | mask << 8, q
  __shared__ uint32_t s_slot[kMaxRec][kPathBlock];
  __shared__ uint16_t s_sv[kMaxRec][kPathBlock];
  __shared__ float s_q[kMaxRec][kPathBlock];
  const int tid = threadIdx.x, lane = tid & 31;
  const unsigned below = (1u << lane) - 1u;
  const int N = G.N;
  const int up = sched->player;
  const uint32_t uid = update_id(sched, N), epoch = *table_epoch(tv);
  unsigned c_trav = 0, c_vis = 0, c_upd = 0;
  bool more = true;
  enum { kIdle = 0, kApply = 1, kDecide = 2, kFold = 3 };
  int st = kIdle;
  WalkState s;
  int pl = -1, pa = 0, nrec = 0, n_act = 0;
  uint32_t cw = 0;
  float u = 0.0f;
  bool show = false;
  for (;;) {
    const unsigned idlem = __ballot_sync(0xFFFFFFFFu, st == kIdle);
    const int n_idle = __popc(idlem);
    bool filled = false;
    if (more && (n_idle >= kPathRefill || n_idle == 32)) {
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(work, (unsigned)n_idle);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      const int got = base < (unsigned)batch ? min(n_idle, (int)((unsigned)batch - base)) : 0;
      if (got < n_idle) more = false;
      const int rank = __popc(idlem & below);
      if (st == kIdle && rank < got) {
        walk_root(G, deals + base + rank, base + (uint32_t)rank, s);
        st = kApply;
        pl = -1;
        nrec = n_act = 0;
      }
      c_trav += got;
      filled = got > 0;
    }
    if (__any_sync(0xFFFFFFFFu, st == kApply)) {
      if (st == kApply) {
        if (pl >= 0) walk_apply<FNV>(G, s, pl, pa);
        const int r = walk_events(G, s, up, u);
        st = kFold;
        show = r == kLvShow;
        if (r == kLvGoOn) {
          st = kDecide;
          pl = walk_next(s.seats, N);
          cw = __ldg(deals[s.aux].ctx + pl);
        }
      }
    }
    const unsigned foldm = __ballot_sync(0xFFFFFFFFu, st == kFold);
    const unsigned decm = __ballot_sync(0xFFFFFFFFu, st == kDecide);
    if (foldm && (__popc(foldm) >= kPathFold || !decm)) {
      if (st == kFold) {
        if (show) u = walk_showdown(N, up, s.seats & 0xFFu, s.inv0, s.inv1, s.inv2, deals + s.aux);
        path_fold(tv, epoch, rscale, u, nrec, &s_slot[0][tid], &s_sv[0][tid], &s_q[0][tid]);
        if (TRACE) {
          mccfr_trace& tr = trace[s.aux];
          const DealRec& D = deals[s.aux];
          for (int i = 0; i < 12; ++i) tr.hole[i] = D.hole[i];
          for (int i = 0; i < 5; ++i) tr.board[i] = D.board[i];
          tr.dealer = D.dealer;
          tr.n_actions = (uint8_t)n_act;
          tr.n_traverser_nodes = (uint8_t)nrec;
          for (int p = 0; p < 6; ++p) {
            const uint32_t c = D.ctx[p];
            tr.hole_bucket[p] = (uint8_t)(c & 0xFF);
            tr.board_bucket[p][0] = 0;
            tr.board_bucket[p][1] = (uint8_t)(c >> 8);
            tr.board_bucket[p][2] = (uint8_t)(c >> 16);
            tr.board_bucket[p][3] = (uint8_t)(c >> 24);
          }
          tr.payoff = u;
          tr.reserved = 0;
        }
        st = kIdle;
      }
      __syncwarp();
      if (more) continue;  // refill before the decisions
    }
    if (!decm) {
      if (n_idle == 32 && !filled && !more) break;
      continue;
    }
    c_vis += __popc(decm);
    const bool isup = st == kDecide && pl == up;
    c_upd += __popc(__ballot_sync(0xFFFFFFFFu, isup));
    if (st == kDecide) {
      const int street = (int)(s.prog & 0xFu);
      const int to_call = s.cb - seat16(s.bet0, s.bet1, s.bet2, pl);
      const uint32_t vm = valid_mask(G, s.pot, G.stack_base - seat16(s.inv0, s.inv1, s.inv2, pl), to_call, s.cb, s.lfr,
                                     (int)((s.prog >> 8) & 0xFFu));
      uint32_t hb, bkt;
      if (G.sub_street) {  // exact combo; the river card once it is dealt
        hb = cw & 0xFFFF;
        bkt = (street == 3 && G.sub_street == 2) ? (cw >> 16) : 0u;
      } else {
        hb = cw & 0xFF;
        bkt = street ? ((cw >> (8 * street)) & 0xFF) : 0u;
      }
      const unsigned long long key = FNV ? info_key(G, pl, hb, bkt, street, s.abits, s.path)
                                         : id64_key(G, pl, hb, bkt, street, s.path);
      // an opponent's missing row reads as no regrets (in a direct map its stored
      // strategy is zero until training writes it); the updating player's is inserted
      const long long slot = DIRECT ? (long long)(key - 1) : isup ? table_insert(tv, key) : table_find(tv, key);
      uint4 sg = make_uint4(0u, 0u, 0u, 0u);
      float reg[kSlots];
      unsigned long long have = key;
      if (slot >= 0) {
        sg = __ldg(row_strat(tv, (unsigned long long)slot));
        if (isup) {
          if (DIRECT) have = __ldcg(row_key(tv, (unsigned long long)slot));
          load_regrets(tv, slot, reg);
        }
      }
      const U4 d = philox(U4{s.aux, uid, (uint32_t)s.path, (uint32_t)(s.path >> 32) | 0x80000000u}, G.seed_lo,
                          G.seed_hi);
      pa = sample_stored(G, sg, vm, uniform01(d.x));
      st = kApply;
      if (isup && slot >= 0) {
        if (DIRECT && have != key) __stcg(row_key(tv, (unsigned long long)slot), key);
        if (nrec < kMaxRec) {
          // the sampled action's regret-matched probability (node_strategy), at least 0.05
          float sum = 0.0f, mine = 0.0f;
#pragma unroll
          for (int a = 0; a < kSlots; ++a)
            if ((vm >> a) & 1) {
              sum = __fadd_rn(sum, fmaxf(0.0f, reg[a]));
              if (a == pa) mine = reg[a];
            }
          float q = 0.0f;
          if (sum > 1e-7f) q = mine > 0.0f ? __fdiv_rn(mine, sum) : 0.0f;
          else if ((vm >> pa) & 1) q = __fdiv_rn(1.0f, (float)__popc(vm));
          s_slot[nrec][tid] = (uint32_t)slot;
          s_sv[nrec][tid] = (uint16_t)((uint32_t)pa | (vm << 8));
          s_q[nrec][tid] = fmaxf(q, 0.05f);
          nrec++;
        } else {
          atomicOr(tv.err, kErrRecordOverflow);
        }
      }
      if (TRACE) {
        if (n_act < 40) trace[s.aux].actions[n_act] = (uint8_t)pa;
      }
      n_act++;
    }
  }
  if (lane == 0 && c_trav) {
    atomicAdd(&counters->traversals, (unsigned long long)c_trav);
    atomicAdd(&counters->visits, (unsigned long long)c_vis);
    atomicAdd(&counters->updates, (unsigned long long)c_upd);
    atomicAdd(&counters->terminals, (unsigned long long)c_trav);
    atomicAdd(&counters->evals, (unsigned long long)c_trav * (unsigned)N);
  }
}

}  // namespace mccfr
