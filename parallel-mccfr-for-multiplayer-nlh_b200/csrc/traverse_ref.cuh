// traverse_ref.cuh — deals, and what every traversal form shares.
//
// The reference runs one recursive traversal per thread, dealing and bucketing
// at its start, with its game state in local memory (cfr_gpu.cu:644-1011).  Here
// k_deal deals every traversal of a player-update (counter-based Philox, the
// reference's partial Fisher-Yates) and computes its buckets and river ranks into a
// 64-byte record, which the traversal kernels read; the rank chains of all players
// share the 3-card board prefix (the table's state depends only on the set of
// cards, which the tests check).
#pragma once
#include "game.cuh"
#include "table.cuh"
#include "../../include/mccfr.h"

namespace mccfr {

struct Sched {
  long long iteration;  // 1-based
  int player;
  int pad;
};

struct HandView {
  const int32_t* hr;      // rank table
  const uint8_t* pre;     // preflop LUT [52*52]
  const uint8_t* cdf;     // rank-CDF LUTs [3][7463], then the states' buckets
};

// Rank-CDF buckets of the rank table's 5- and 6-card states, one byte per state
// (613 KB beside the LUTs): a flop or turn bucket is one gather from a small
// table instead of the state's rank from the 130 MB one and then its LUT.
constexpr int kStateBuckets = 22400;  // offset: 3 * 7463 rounded up
constexpr int kStates = MCCFR_HAND_TABLE_ENTRIES / 53;
constexpr size_t kCdfBytes = kStateBuckets + kStates;

// One traversal's deal.  ctx[p] = hole bucket | flop << 8 | turn << 16 | river << 24.
struct DealRec {
  uint32_t ctx[kMaxPlayers];
  uint16_t rank[kMaxPlayers];
  uint8_t hole[2 * kMaxPlayers];
  uint8_t board[5];
  uint8_t dealer;
  uint8_t pad[10];
};
static_assert(sizeof(DealRec) == 64, "deal record is one 64-byte pair of sectors");

struct Counters {
  unsigned long long traversals, visits, updates, terminals, evals;
};

__device__ __forceinline__ void warp_add_counters(Counters* c, unsigned t, unsigned v, unsigned u,
                                                  unsigned x, unsigned e) {
  const unsigned m = __activemask();
  t = __reduce_add_sync(m, t);
  v = __reduce_add_sync(m, v);
  u = __reduce_add_sync(m, u);
  x = __reduce_add_sync(m, x);
  e = __reduce_add_sync(m, e);
  // only non-zero sums are added: a launch over an empty level adds nothing
  if ((threadIdx.x & 31) == (__ffs(m) - 1)) {
    if (t) atomicAdd(&c->traversals, (unsigned long long)t);
    if (v) atomicAdd(&c->visits, (unsigned long long)v);
    if (u) atomicAdd(&c->updates, (unsigned long long)u);
    if (x) atomicAdd(&c->terminals, (unsigned long long)x);
    if (e) atomicAdd(&c->evals, (unsigned long long)e);
  }
}

__device__ __forceinline__ uint32_t update_id(const Sched* s, int N) {
  return (uint32_t)((s->iteration - 1) * N + s->player);
}

// Subgame deal: every player's hole combo from its range, all combos drawn
// together and redrawn (up to 16 times) until no two share a card; after that,
// player by player, the drawn combo or the next one of positive weight that
// fits.  On the turn the river card is then uniform among the unused cards.
// ctx[p] = combo | (river card + 1) << 16 (the river card enters the river keys).
//
// Eight lanes per traversal (`gl` = lane of the group): they draw eight attempts
// at once and keep the first that fits, then lane p writes player p's fields.  The
// draws are chains of dependent range lookups (11 per combo), and with six players
// three of four attempts collide, so one thread per traversal spent most of a
// small update here (1,024 six-player turn deals: 236 us).
constexpr int kDealGroup = 8;

__device__ __forceinline__ void deal_subgame(const GameParams& G, const int32_t* __restrict__ T, uint32_t t,
                                             uint32_t uid, DealRec* __restrict__ out, int gl, unsigned gmask) {
  const int N = G.N;
  const int nb = G.sub_street == 2 ? 4 : 5;
  uint64_t used_board = 0;
  for (int i = 0; i < nb; ++i) used_board |= 1ull << G.sub_board[i];
  int combo[kMaxPlayers], first[kMaxPlayers];  // this attempt's combos, the first round's
  uint64_t used = used_board;
  int winner = -1;
  for (int round = 0; round < 16 / kDealGroup && winner < 0; ++round) {
    const uint32_t attempt = 0x100u + (uint32_t)(round * kDealGroup + gl);
    const U4 w0 = philox(U4{t, uid, attempt, 0u}, G.seed_lo, G.seed_hi);
    const U4 w1 = philox(U4{t, uid, attempt, 1u}, G.seed_lo, G.seed_hi);
    const uint32_t words[kMaxPlayers] = {w0.x >> 1, w0.y >> 1, w0.z >> 1, w0.w >> 1, w1.x >> 1, w1.y >> 1};
    // each player's first combo whose cumulative weight exceeds its word, by
    // bisection, the players' side by side
    int lo[kMaxPlayers], hi[kMaxPlayers];
#pragma unroll
    for (int p = 0; p < kMaxPlayers; ++p) {
      lo[p] = 0;
      hi[p] = p < N ? 1325 : 0;
    }
    for (int step = 0; step < 11; ++step) {
#pragma unroll
      for (int p = 0; p < kMaxPlayers; ++p)
        if (lo[p] < hi[p]) {
          const int mid = (lo[p] + hi[p]) >> 1;
          if (words[p] < __ldg(G.range_cdf + 1326 * p + mid)) hi[p] = mid;
          else lo[p] = mid + 1;
        }
    }
    used = used_board;
    bool ok = true;
#pragma unroll
    for (int p = 0; p < kMaxPlayers; ++p) {
      combo[p] = lo[p];
      if (round == 0) first[p] = lo[p];
      if (p < N) {
        const uint64_t m = combo_bits(lo[p]);
        ok &= (used & m) == 0;
        used |= m;
      }
    }
    const unsigned fit = __ballot_sync(gmask, ok) & gmask;
    if (fit) winner = __ffs((int)fit) - 1;
  }
  if (winner < 0) {
    // player by player from the first attempt's draws (the group's first lane's),
    // eight combos of the search at a time: neighbours share their higher card, so a
    // search often passes dozens
    winner = __ffs((int)gmask) - 1;
    used = used_board;
#pragma unroll
    for (int p = 0; p < kMaxPlayers; ++p) {
      if (p >= N) break;
      const uint32_t* cdf = G.range_cdf + 1326 * p;
      const int start = __shfl_sync(gmask, first[p], winner);
      int pick = start;  // kept when the range is exhausted by card removal
      for (int k = 0; k < 1326; k += kDealGroup) {
        const int c = start + k + gl < 1326 ? start + k + gl : start + k + gl - 1326;
        bool fits = false;
        if (k + gl < 1326) fits = __ldg(cdf + c) != (c ? __ldg(cdf + c - 1) : 0u) && !(used & combo_bits(c));
        const unsigned fit = __ballot_sync(gmask, fits) & gmask;
        if (fit) {
          pick = __shfl_sync(gmask, c, __ffs((int)fit) - 1);
          break;
        }
      }
      combo[p] = pick;
      used |= combo_bits(pick);
    }
  }
  int mine = 0;
#pragma unroll
  for (int p = 0; p < kMaxPlayers; ++p) {
    const int c = __shfl_sync(gmask, combo[p], winner);
    if (p == gl) mine = c;
  }
  used = (uint64_t)__shfl_sync(gmask, (unsigned)used, winner) |
         (uint64_t)__shfl_sync(gmask, (unsigned)(used >> 32), winner) << 32;
  int river = nb == 4 ? 0 : -1, fifth = G.sub_board[4];
  if (nb == 4) {
    const U4 w = philox(U4{t, uid, 0x200u, 0u}, G.seed_lo, G.seed_hi);
    uint64_t spare = ~used & ((1ull << 52) - 1);
    int k = (int)(((unsigned long long)w.x * (unsigned long long)__popcll(spare)) >> 32);
    for (; k > 0; --k) spare &= spare - 1;
    river = __ffsll((long long)spare) - 1;
    fifth = river;
  }
  uint32_t* const words = reinterpret_cast<uint32_t*>(out);
  if (gl < kMaxPlayers) {
    uint32_t ctx = 0;
    uint16_t rank = 0, hole = 0;
    if (gl < N) {
      int32_t b = __ldg(T + 53 + to_rm(G.sub_board[0]));
      for (int i = 1; i < 4; ++i) b = __ldg(T + b + to_rm(G.sub_board[i]));
      b = __ldg(T + b + to_rm(fifth));
      int lo, hi;
      combo_cards(mine, lo, hi);
      const int32_t s6 = __ldg(T + b + to_rm(lo));
      rank = (uint16_t)decode16((uint32_t)__ldg(T + s6 + to_rm(hi)) & 0xFFFF);
      ctx = (uint32_t)mine | ((uint32_t)(river + 1) << 16);
      hole = (uint16_t)(lo | hi << 8);
    }
    words[gl] = ctx;
    out->rank[gl] = rank;
    reinterpret_cast<uint16_t*>(out->hole)[gl] = hole;
  } else if (gl == kMaxPlayers) {
    words[12] = (uint32_t)G.sub_board[0] | (uint32_t)G.sub_board[1] << 8 | (uint32_t)G.sub_board[2] << 16 |
                (uint32_t)G.sub_board[3] << 24;
    words[13] = (uint32_t)fifth | (uint32_t)(N - 1) << 8;  // river card, dealer
  } else {
    words[14] = words[15] = 0;
  }
}

// One thread's 52-card deck in shared memory, as 13 words of four cards, a block's
// width apart: whatever cards a warp's threads touch, each works in its own bank.
// (As a thread's own array the shuffle's indexing put it in local memory, and as
// rows of 13 words the threads' banks met at random.)
constexpr int kDeckWords = 13;
template <int STRIDE>
struct Deck {
  uint32_t* col;
  __device__ __forceinline__ uint8_t& at(int i) const {
    return reinterpret_cast<uint8_t*>(col + (i >> 2) * STRIDE)[i & 3];
  }
  __device__ __forceinline__ uint32_t word(int w) const { return col[w * STRIDE]; }

  // The first `n_deal` cards of traversal t's shuffle in update `uid`
  // (cfr_gpu.cu:460-470): partial Fisher-Yates by multiply-shift, four draws per
  // Philox block; returns the word after the last draw.
  __device__ __forceinline__ uint32_t shuffle(const GameParams& G, uint32_t t, uint32_t uid, int n_deal) const {
#pragma unroll
    for (int w = 0; w < kDeckWords; ++w) col[w * STRIDE] = 0x03020100u + 0x04040404u * (uint32_t)w;  // cards 4w .. 4w+3
    uint32_t next = 0;
    for (int blk = 0; 4 * blk <= n_deal; ++blk) {
      const U4 o = philox(U4{t, uid, 0u, (uint32_t)blk}, G.seed_lo, G.seed_hi);
      const uint32_t wv[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 4 * blk + e;
        if (i < n_deal) {
          uint8_t& mine = at(i);
          uint8_t& drawn = at(i + (int)__umulhi(wv[e], (uint32_t)(52 - i)));
          const uint8_t tmp = mine;
          mine = drawn;
          drawn = tmp;
        } else if (i == n_deal) {
          next = wv[e];
        }
      }
    }
    return next;
  }
};

// Deal, buckets and river ranks of traversal t of update `uid`
// (cfr_gpu.cu:460-470, 476-489, 942-952, 963).  `pre` is the 52x52 preflop LUT
// (shared or global memory), `cdf` the rank-CDF LUTs.
template <int STRIDE>
__device__ __forceinline__ void deal_one(const GameParams& G, const int32_t* __restrict__ T, const uint8_t* pre,
                                         const uint8_t* __restrict__ cdf, uint32_t t, uint32_t uid,
                                         DealRec* __restrict__ out, const Deck<STRIDE> deck) {
  const int N = G.N;
  const uint32_t dealer = deck.shuffle(G, t, uid, 2 * N + 5) % (uint32_t)N;
  int board[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) board[i] = deck.at(2 * N + i);
  int32_t b = __ldg(T + 53 + to_rm(board[0]));
  b = __ldg(T + b + to_rm(board[1]));
  b = __ldg(T + b + to_rm(board[2]));
  int32_t s5[kMaxPlayers], s6[kMaxPlayers], r7[kMaxPlayers], s4[kMaxPlayers];
#pragma unroll
  for (int p = 0; p < kMaxPlayers; ++p)
    if (p < N) s4[p] = __ldg(T + b + to_rm(deck.at(2 * p)));
#pragma unroll
  for (int p = 0; p < kMaxPlayers; ++p)
    if (p < N) s5[p] = __ldg(T + s4[p] + to_rm(deck.at(2 * p + 1)));
  const int rm3 = to_rm(board[3]), rm4 = to_rm(board[4]);
#pragma unroll
  for (int p = 0; p < kMaxPlayers; ++p)
    if (p < N) s6[p] = __ldg(T + s5[p] + rm3);
#pragma unroll
  for (int p = 0; p < kMaxPlayers; ++p)
    if (p < N) r7[p] = __ldg(T + s6[p] + rm4);
  uint32_t ctx[kMaxPlayers], rank[kMaxPlayers];
#pragma unroll
  for (int p = 0; p < kMaxPlayers; ++p) {
    ctx[p] = 0;
    rank[p] = 0;
    if (p >= N) continue;
    const uint32_t hb = pre[deck.at(2 * p) * 52 + deck.at(2 * p + 1)];
    const uint32_t rr = decode16((uint32_t)r7[p] & 0xFFFF);
    uint32_t b1, b2, b3;
    if (G.postflop_mode == 0) {
      // the reference decodes the 5th/6th chain value (a state) as a rank
      b1 = ref_linear_bucket(decode16((uint32_t)s5[p] & 0xFFFF), G.post_b[0]);
      b2 = ref_linear_bucket(decode16((uint32_t)s6[p] & 0xFFFF), G.post_b[1]);
      b3 = ref_linear_bucket(rr, G.post_b[2]);
    } else {
      b1 = __ldg(cdf + kStateBuckets + (uint32_t)s5[p] / 53u);
      b2 = __ldg(cdf + kStateBuckets + (uint32_t)s6[p] / 53u);
      b3 = __ldg(cdf + 2 * 7463 + rr);
    }
    ctx[p] = hb | (b1 << 8) | (b2 << 16) | (b3 << 24);
    rank[p] = rr;
  }
  // the record, whole: ctx, ranks, hole cards (the deck's first 2N), board, dealer
  uint4* const dst = reinterpret_cast<uint4*>(out);
  dst[0] = make_uint4(ctx[0], ctx[1], ctx[2], ctx[3]);
  dst[1] = make_uint4(ctx[4], ctx[5], rank[0] | rank[1] << 16, rank[2] | rank[3] << 16);
  const uint32_t h1 = N == 2 ? 0u : N == 3 ? deck.word(1) & 0xFFFFu : deck.word(1);
  const uint32_t h2 = N <= 4 ? 0u : N == 5 ? deck.word(2) & 0xFFFFu : deck.word(2);
  dst[2] = make_uint4(rank[4] | rank[5] << 16, deck.word(0), h1, h2);
  dst[3] = make_uint4((uint32_t)board[0] | (uint32_t)board[1] << 8 | (uint32_t)board[2] << 16 |
                          (uint32_t)board[3] << 24, (uint32_t)board[4] | dealer << 8, 0u, 0u);
}

// Deals of `players` successive updates (the schedule's and the following players'),
// `batch` traversals each, update after update.  The deal starts an update: it
// advances the table's epoch and zeroes `ctl`, the counters of the traversal that
// follows (may be null), so that neither needs a launch of its own.  SUB: a subgame
// (eight lanes per traversal).
template <bool SUB>
__global__ void __launch_bounds__(128) k_deal(const GameParams G, const HandView hv, const Sched* __restrict__ sched,
                                              int batch, int players, DealRec* __restrict__ out,
                                              uint32_t* __restrict__ epoch, uint32_t* __restrict__ ctl,
                                              int ctl_words) {
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) *epoch += 1;
    for (int i = threadIdx.x; i < ctl_words; i += blockDim.x) ctl[i] = 0;
  }
  const uint32_t n = (uint32_t)batch * (uint32_t)players;
  const uint32_t uid = update_id(sched, G.N);
  if constexpr (SUB) {
    const uint32_t i = blockIdx.x * (128 / kDealGroup) + threadIdx.x / kDealGroup;
    if (i >= n) return;  // whole groups
    const uint32_t p = players > 1 ? i / (uint32_t)batch : 0u;
    const int gl = (int)threadIdx.x & (kDealGroup - 1);
    deal_subgame(G, hv.hr, i - p * (uint32_t)batch, uid + p, out + i, gl,
                 ((1u << kDealGroup) - 1u) << ((threadIdx.x & 31) & ~(kDealGroup - 1)));
  } else {
    __shared__ uint8_t s_pre[52 * 52];
    __shared__ uint32_t s_deck[128 * kDeckWords];
    for (int i = threadIdx.x; i < 52 * 52 / 4; i += blockDim.x)
      reinterpret_cast<uint32_t*>(s_pre)[i] = __ldg(reinterpret_cast<const uint32_t*>(hv.pre) + i);
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const uint32_t p = players > 1 ? i / (uint32_t)batch : 0u;
      deal_one(G, hv.hr, s_pre, hv.cdf, i - p * (uint32_t)batch, uid + p, out + i,
               Deck<128>{s_deck + threadIdx.x});
    }
  }
}

// Side-pot showdown for player `up` (cfr_gpu.cu:694-753).  The distinct non-zero
// invested amounts are visited in ascending order as "the smallest amount above
// the previous level", which is the reference's sorted level list without an
// array; invested chips and ranks are read through the caller's accessors.
template <class InvF, class RankF>
__device__ __forceinline__ float side_pot_payoff(int N, int up, uint32_t folded, InvF inv, RankF rank) {
  // The players' amounts and ranks are read once into fixed slots, so the
  // loops below index them with constants.
  int iv[kMaxPlayers];
  uint32_t rk[kMaxPlayers];
#pragma unroll
  for (int q = 0; q < kMaxPlayers; ++q) {
    iv[q] = q < N ? inv(q) : 0;
    rk[q] = q < N ? (uint32_t)rank(q) : 0u;
  }
  int inv_up = 0;
  uint32_t rk_up = 0;
#pragma unroll
  for (int q = 0; q < kMaxPlayers; ++q)
    if (q == up) {
      inv_up = iv[q];
      rk_up = rk[q];
    }
  const bool up_live = !((folded >> up) & 1);
  float payoff = -(float)inv_up;
  int prev = 0;
  for (int guard = 0; guard < kMaxPlayers; ++guard) {
    int L = 0x7FFFFFFF;
#pragma unroll
    for (int q = 0; q < kMaxPlayers; ++q)
      if (q < N && iv[q] > prev && iv[q] < L) L = iv[q];
    if (L == 0x7FFFFFFF) break;
    int layer = 0;
    uint32_t best = 0;
#pragma unroll
    for (int q = 0; q < kMaxPlayers; ++q)
      if (q < N) {
        layer += max(0, min(iv[q], L) - prev);
        if (!((folded >> q) & 1) && iv[q] >= L) best = max(best, rk[q]);
      }
    if (best > 0) {
      int nwin = 0;
#pragma unroll
      for (int q = 0; q < kMaxPlayers; ++q)
        if (q < N && !((folded >> q) & 1) && iv[q] >= L && rk[q] == best) nwin++;
      if (up_live && inv_up >= L && rk_up == best) payoff = __fadd_rn(payoff, __fdiv_rn((float)layer, (float)nwin));
    }
    prev = L;
  }
  return payoff;
}

__device__ __forceinline__ void load_regrets(const TableView& tv, long long slot, float* reg) {
  if (slot >= 0) {
    const float4* p = row_reg(tv, (unsigned long long)slot);
    const float4 r0 = __ldg(p), r1 = __ldg(p + 1);
    reg[0] = r0.x; reg[1] = r0.y; reg[2] = r0.z; reg[3] = r0.w;
    reg[4] = r1.x; reg[5] = r1.y; reg[6] = r1.z; reg[7] = r1.w;
  } else {
#pragma unroll
    for (int a = 0; a < kSlots; ++a) reg[a] = 0.0f;
  }
}

}  // namespace mccfr
