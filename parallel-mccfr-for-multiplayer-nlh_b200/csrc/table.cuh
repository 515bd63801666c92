// table.cuh — open-addressed info-set table in HBM.
//
// Replaces the reference's direct-mapped SoA tables [8 x 2^26] (cfr_gpu.cu:
// 1106-1136).  Each row is one 256-byte record (two 128-byte lines); what a
// visit reads comes first, and a row that only opponents visited in an update
// is folded from its first line alone:
//     0  key    u64   0 = empty; linear probing from the key's home slot, or row k-1
//                       for key k when every key fits (direct map)
//     8  tag    u64   (epoch of the last update with sampled visits) << 8 | canonical
//                       action mask: that of the update's first sampled visit
//    16  strat[8] bf16  current strategy max(0, reg) / sum over all slots, rounded to
//                       BF16 as sampling takes it (0 while the sum is at most 1e-7)
//    32  cnt    u64   (all visits << 32) | visits whose mask is the canonical one
//    40  su     i64   sum of fix(u) (reference rule) or fix(v_h) (external sampling)
//    48  visits u64   updates received since creation
//    56  flags  u32   bit 0: ds holds values
//    64  reg[8] f32   regrets (snapshot within an update)
//    96  ssum[8] f32  average-strategy sums
//   128  da[8]  i64   per-action regret deltas, 2^-rb units
//   192  ds[8]  i64   strategy weights of non-canonical visits, 2^-32 units
// cnt/su/da/ds/flags are per-update accumulators, zeroed by the apply kernel.
// strat follows reg: whoever writes regrets stores it (pack_strategy), so a sampled visit reads one 32-byte sector and divides nothing.
//
// Touched rows are marked in two bitmaps, one bit per row: rows with sampled
// visits, and rows whose da was added to ("wide": the updating player's).  A mark
// is a plain OR whose result nobody waits for, the bitmaps fit L2, and the apply
// kernel meets the rows in address order.  Above 2^28 rows the two bitmaps exceed L2
// (128 MB at 2^29) and every update would read them from memory, so there each run of
// 1,024 rows also has a byte that says whether any of its words are to be read.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>

namespace mccfr {

constexpr int kRowBytes = 256;
constexpr int kOffKey = 0, kOffTag = 8, kOffStrat = 16, kOffCnt = 32, kOffSu = 40, kOffVisits = 48, kOffFlags = 56,
              kOffReg = 64, kOffSsum = 96, kOffDa = 128, kOffDs = 192;
constexpr unsigned kFlagDs = 1u;
struct TableView {
  unsigned char* rows;       // [cap][256]
  unsigned int* bits;        // [2][n_words] touched rows: sampled visits, wide
  unsigned char* runs;       // one byte per 32 words: some row of theirs is marked; null: every word is read
  unsigned int n_words;      // words of one bitmap: one bit per row that a key can own
  // counters, kCounterStride words apart, by epoch parity: touched rows (0, 1) and
  // wide ones among them (2, 3) of the update; the epoch (4): updates begun since
  // the table was cleared; blocks of the apply kernel that are done (5)
  unsigned int* counters;
  unsigned long long mask;   // cap - 1
  int log2cap;
  int direct;                // every key is at most cap: key k owns row k-1, no probing
  int* err;
};

enum : int {
  kErrTableFull = 1,
  kErrRecordOverflow = 2,
  kErrStackOverflow = 4,
};

constexpr int kProbeLimit = 1 << 14;
constexpr int kCounterStride = 32;  // counters 128 bytes apart (separate lines)

__device__ __forceinline__ unsigned char* row_ptr(const TableView& tv, unsigned long long s) {
  return tv.rows + (s << 8);
}
__device__ __forceinline__ unsigned long long* row_key(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned long long*>(row_ptr(tv, s) + kOffKey);
}
__device__ __forceinline__ unsigned long long* row_tag(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned long long*>(row_ptr(tv, s) + kOffTag);
}
// Key and tag.
__device__ __forceinline__ ulonglong2* row_head(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<ulonglong2*>(row_ptr(tv, s));
}
__device__ __forceinline__ uint4* row_strat(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<uint4*>(row_ptr(tv, s) + kOffStrat);
}
__device__ __forceinline__ unsigned long long* row_cnt(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned long long*>(row_ptr(tv, s) + kOffCnt);
}
__device__ __forceinline__ unsigned long long* row_su(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned long long*>(row_ptr(tv, s) + kOffSu);
}
__device__ __forceinline__ float4* row_reg(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<float4*>(row_ptr(tv, s) + kOffReg);
}
__device__ __forceinline__ float4* row_ssum(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<float4*>(row_ptr(tv, s) + kOffSsum);
}
__device__ __forceinline__ unsigned long long* row_da(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned long long*>(row_ptr(tv, s) + kOffDa);
}
__device__ __forceinline__ unsigned long long* row_ds(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned long long*>(row_ptr(tv, s) + kOffDs);
}
__device__ __forceinline__ unsigned long long* row_visits(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned long long*>(row_ptr(tv, s) + kOffVisits);
}
__device__ __forceinline__ unsigned int* row_flags(const TableView& tv, unsigned long long s) {
  return reinterpret_cast<unsigned int*>(row_ptr(tv, s) + kOffFlags);
}

__device__ __forceinline__ unsigned long long home_slot(const TableView& tv, unsigned long long key) {
  return (key * 0x9E3779B97F4A7C15ull) >> (64 - tv.log2cap);
}

// Read-only lookup; returns the slot or -1.  W keys are loaded per probe step
// (independent loads issued together); W is an autotuned probe width.  A
// direct-mapped table reads the key's own row only.
template <int W = 1>
__device__ __forceinline__ long long table_find(const TableView& tv, unsigned long long key) {
  if (tv.direct) return __ldcg(row_key(tv, key - 1)) == key ? (long long)(key - 1) : -1ll;
  unsigned long long s = home_slot(tv, key);
  for (int step = 0; step < kProbeLimit; step += W) {
    unsigned long long k[W];
#pragma unroll
    for (int i = 0; i < W; ++i) k[i] = __ldcg(row_key(tv, (s + i) & tv.mask));
#pragma unroll
    for (int i = 0; i < W; ++i) {
      if (k[i] == key) return (long long)((s + i) & tv.mask);
      if (k[i] == 0) return -1;
    }
    s = (s + W) & tv.mask;
  }
  return -1;
}

// Find or insert; returns the slot, or -1 when the probe limit is exceeded.
// In a direct-mapped table row k-1 can hold no key but k, so every writer of
// the key stores the same value and no atomic is needed.
template <int W = 1>
__device__ __forceinline__ long long table_insert(const TableView& tv, unsigned long long key) {
  if (tv.direct) {
    unsigned long long* kp = row_key(tv, key - 1);
    if (__ldcg(kp) != key) __stcg(kp, key);
    return (long long)(key - 1);
  }
  unsigned long long s = home_slot(tv, key);
  for (int step = 0; step < kProbeLimit; step += W) {
    unsigned long long k[W];
#pragma unroll
    for (int i = 0; i < W; ++i) k[i] = __ldcg(row_key(tv, (s + i) & tv.mask));
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const unsigned long long slot = (s + i) & tv.mask;
      if (k[i] == key) return (long long)slot;
      if (k[i] == 0) {
        const unsigned long long prev = atomicCAS(row_key(tv, slot), 0ull, key);
        if (prev == 0 || prev == key) return (long long)slot;
      }
    }
    s = (s + W) & tv.mask;
  }
  atomicOr(tv.err, kErrTableFull);
  return -1;
}

__host__ __device__ __forceinline__ unsigned int* touched_count(const TableView& tv, uint32_t epoch) {
  return tv.counters + (size_t)kCounterStride * (epoch & 1);
}
__host__ __device__ __forceinline__ unsigned int* wide_count(const TableView& tv, uint32_t epoch) {
  return tv.counters + (size_t)kCounterStride * (2 + (epoch & 1));
}
__host__ __device__ __forceinline__ unsigned int* table_epoch(const TableView& tv) {
  return tv.counters + (size_t)kCounterStride * 4;
}
__host__ __device__ __forceinline__ unsigned int* apply_ticket(const TableView& tv) {
  return tv.counters + (size_t)kCounterStride * 5;
}
// Bytes of the counter block (the six above, then the error flag).
constexpr size_t kCounterBytes = (size_t)kCounterStride * 4 * 6 + 128;

// Rows above which runs of rows carry a mark of their own: where the bitmaps exceed
// L2.  Heads-up under the reference's rule, the apply pass of a 256-traversal update
// takes 101 us in a 2^29-row table when it reads both bitmaps whole and 14 us with the
// runs' marks (lists of touched rows took 39), that of 1,000 external-sampling
// traversals 106 and 28 us.  An update that touches most runs pays for them: 65,536
// heads-up traversals in 2^29 rows 39 us of 420, in 2^26 rows 11 us of 293, and 2^20
// traversals of 6-max 0.9%; up to 2^28 rows no update was slower than with lists.
constexpr unsigned long long kRunRows = 1ull << 28;

__device__ __forceinline__ void mark_run(const TableView& tv, unsigned long long slot) {
  if (tv.runs) tv.runs[slot >> 10] = 1;  // plain: every writer stores the same
}
__device__ __forceinline__ void mark_wide(const TableView& tv, unsigned long long slot) {
  mark_run(tv, slot);
  atomicOr(tv.bits + tv.n_words + (unsigned)(slot >> 5), 1u << (slot & 31));
}

// Marks the row as sampled in the update of `epoch` and returns whether `vm` is
// its canonical mask there (the first visitor's).  `tag` is the row's as the
// caller read it; a stale one only makes the compare-and-swap fail, and then the
// row belongs to this update already.
__device__ __forceinline__ bool touch_row_from(const TableView& tv, unsigned long long slot, uint32_t epoch,
                                               uint32_t vm, unsigned long long tag) {
  if ((tag >> 8) != epoch) {
    tag = atomicCAS(row_tag(tv, slot), tag, ((unsigned long long)epoch << 8) | vm);
    if ((tag >> 8) != epoch) {
      mark_run(tv, slot);
      atomicOr(tv.bits + (unsigned)(slot >> 5), 1u << (slot & 31));
      return true;
    }
  }
  return (uint32_t)(tag & 0xFF) == vm;
}
__device__ __forceinline__ bool touch_row(const TableView& tv, unsigned long long slot, uint32_t epoch, uint32_t vm) {
  return touch_row_from(tv, slot, epoch, vm, __ldcg(row_tag(tv, slot)));
}

// One 32-byte sector by one lane (256-bit accesses; L2 only).
struct __align__(32) Sector {
  unsigned long long x, y, z, w;
};
__device__ __forceinline__ Sector ld_sector(const void* p) {
  Sector s;
  asm volatile("ld.global.cg.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(s.x), "=l"(s.y), "=l"(s.z), "=l"(s.w) : "l"(__cvta_generic_to_global(p)) : "memory");
  return s;
}
__device__ __forceinline__ void st_sector(void* p, const Sector& s) {
  asm volatile("st.global.cg.v4.u64 [%0], {%1, %2, %3, %4};"
               :: "l"(__cvta_generic_to_global(p)), "l"(s.x), "l"(s.y), "l"(s.z), "l"(s.w) : "memory");
}
// The same through L1, for data that only this SM's warp reads back.
__device__ __forceinline__ Sector ld_own_sector(const void* p) {
  Sector s;
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(s.x), "=l"(s.y), "=l"(s.z), "=l"(s.w) : "l"(__cvta_generic_to_global(p)) : "memory");
  return s;
}
__device__ __forceinline__ void st_own_sector(void* p, const Sector& s) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};"
               :: "l"(__cvta_generic_to_global(p)), "l"(s.x), "l"(s.y), "l"(s.z), "l"(s.w) : "memory");
}
__device__ __forceinline__ unsigned long long two_words(uint32_t lo, uint32_t hi) {
  return (unsigned long long)lo | (unsigned long long)hi << 32;
}
__device__ __forceinline__ float lo_float(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi_float(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ unsigned long long two_floats(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | (unsigned long long)__float_as_uint(hi) << 32;
}

// A row's BF16 sampling strategy from its regrets: the sums and roundings of
// sampling (cfr_gpu.cu:318-351).
__device__ __forceinline__ uint4 pack_strategy(const float* reg) {
  float sum = 0.0f;
#pragma unroll
  for (int a = 0; a < 8; ++a) sum = __fadd_rn(sum, fmaxf(0.0f, reg[a]));
  uint32_t h[8];
#pragma unroll
  for (int a = 0; a < 8; ++a)
    h[a] = __bfloat16_as_ushort(__float2bfloat16_rn(sum > 1e-7f && reg[a] > 0.0f ? __fdiv_rn(reg[a], sum) : 0.0f));
  return make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
}

// Adds one visit whose legal mask differs from the row's canonical one: every
// legal action's regret term and strategy weight directly.
__device__ __forceinline__ void add_direct(const TableView& tv, unsigned long long slot, uint32_t vm,
                                           const long long* dr, const long long* dsw) {
  if (dsw) atomicOr(row_flags(tv, slot), kFlagDs);
  for (int a = 0; a < 8; ++a) {
    if (!((vm >> a) & 1)) continue;
    if (dr) atomicAdd(row_da(tv, slot) + a, (unsigned long long)dr[a]);
    if (dsw) atomicAdd(row_ds(tv, slot) + a, (unsigned long long)dsw[a]);
  }
}

}  // namespace mccfr
