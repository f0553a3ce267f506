// qeg_agg.cu -- hash GROUP BY on sm_103a: replaces qe::Aggregate
// (ops/aggregate.h:102-144, ops/aggregate.cpp).
//
// Table layout (HBM). One row of 64-bit words per group:
//   single key : [key word][fields...]            + 2 side rows at index cap
//                (key word 0, which doubles as the empty marker) and cap+1
//                (the NULL key group)
//   multi key  : [state][null mask][key words...][fields...]; state 0 = empty,
//                1 = being published, >= 2 = the row's hash tag
//   global     : one row [unused][fields...]
// Fields hold the reference's AggCell state (ops/agg_internal.h:47-51) in a
// form where all-zero bits are the identity of every aggregate, so tables are
// initialised by memset: row count, per-column NULL count (non-null count =
// rows - nulls), integer / F64 sums, and MIN/MAX as order-preserving unsigned
// encodings updated with atomicMax (qeg_device.cuh).
//
// Kernels: for single keys each CTA keeps a private shared-memory table
// (first-come insertion, or preloaded with heavy hitters) that lanes update row
// by row (qeg_privagg.cuh), and falls back to the global table, whose
// key words are claimed with one CAS; inputs whose global table would not stay
// in L2 are partitioned by key hash first. Rows whose key cannot be placed within
// the probe limit are spilled (row index) and re-run after the host grows the
// table (rehash) -- the GPU form of HashTable::grow (ops/hashtable.cpp:75-91).
#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <unordered_map>

#include "qeg_agg.h"
#include "qeg_privagg.cuh"
#include "qeg_warpagg.cuh"

namespace qeg {

namespace {

__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Acquire load: a state word published after the key words (a fence, then
// the atomic exchange of the tag) makes those key words visible to the loads
// that follow it.
__device__ __forceinline__ uint64_t ld_acquire(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Probe length once the global table is nearly full: what is not found by then
// waits for the larger table. 64M rows with a first table of fixed size, at 16
// slots and at 4: 3M uniform groups 14.7 / 13.4 ms, 10M 17.5 / 15.6, Zipf(1.1)
// over 64M keys 8.2 / 7.5.
constexpr int kFullProbe = 4;
// The partitioned strategy is chosen (QEG_AGG_AUTO) for inputs of at least
// kPartMinRows rows whose estimated global table would take kPartMinTableBytes
// or more (half of L2: its random rows would mostly come from DRAM).
constexpr uint64_t kPartMinRows = 1ull << 22;
constexpr uint64_t kPartMinTableBytes = 64ull << 20;
// At most 2^kPartMaxBits partitions (the sizing pass keeps a 32-bit counter
// per partition in shared memory), and QEG_AGG_AUTO partitions only while the
// estimate averages at most kPartMaxFill of a second-pass table per partition.
constexpr int kPartMaxBits = 15;
constexpr double kPartMaxFill = 0.6;
// Share of a second-pass table that the estimate should fill: short searches
// are worth more partitions (and the tables to clear for them). 48M uniform
// rows, whole call, at 0.6 and at 0.15, two bits more: 3M groups 3.55 / 2.96
// ms, 5M 3.96 / 3.49, 10M 5.17 / 4.79, 16M 7.08 / 6.38; 16M rows over 4M groups
// 2.33 / 1.99, over 12M 3.31 / 3.30; one bit more still: 2.98, 3.57, 2.02 ms
// (3M, 5M, 16M rows over 4M groups).
constexpr double kPartFill = 0.15;
// Share of the rows that the heavy hitters must carry for the partitioned
// passes to look every row up among them.
constexpr double kPartMinHotShare = 0.1;

__device__ __forceinline__ uint64_t ld_volatile_shared(const uint64_t* p) {
  return *reinterpret_cast<const volatile uint64_t*>(p);
}

// Loads the values of one row for every referenced value column.
template <int NV>
__device__ __forceinline__ void load_values(const AggK& P, uint64_t p, bool (&vv)[kMaxVals],
                                            uint64_t (&vb)[kMaxVals]) {
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    vv[c] = false;
    vb[c] = 0;
    if (c < P.nvals) {
      const DevCol& col = P.val[c];
      vv[c] = col_valid(col, p);
      if (vv[c]) {
        if (col.type == kF64)
          vb[c] = static_cast<uint64_t>(__ldg(static_cast<const long long*>(col.data) + p));
        else
          vb[c] = static_cast<uint64_t>(int_value(col, p));
      }
    }
  }
}

// Hash of a single-key table's key word: two multiplies (about 7 instructions;
// the two-round splitmix64 of the composite rows takes about 40). A bijection,
// so distinct keys never share a full hash.
__host__ __device__ __forceinline__ uint64_t key_hash1(uint64_t k) {
  uint64_t x = k * 0x9E3779B97F4A7C15ull;
  x ^= x >> 32;
  return x * 0xD1342543DE82EF95ull;
}

// Home slot of hash h in a table of `cap` slots: the hash scaled to the table,
// by its top 32 bits where the table has fewer than 2^31 slots.
__device__ __forceinline__ uint64_t home_slot(uint64_t h, uint64_t cap) {
  if ((cap >> 31) == 0) return ((h >> 32) * cap) >> 32;
  return __umul64hi(h, cap);
}

// Single-key global lookup/insert of up to U keys per lane (k[u], nonzero,
// where want[u]) from their home slots s[u], whose key words were last read as
// cur[u]: the row of each, or nullptr when it could not be placed within the
// probe limit. Linear probing. A key word never changes once set, so a stale
// non-empty value stays correct. Behind the home slot a few slots are loaded
// per step, for all U keys together, and examined in order; only one that
// reads as empty is claimed by a compare-and-swap. (A compare-and-swap per
// probe is one round trip less for an insert, but an atomic for every look at
// a taken slot: 256M Zipf(1.1) rows over 64M keys, 16.6M groups, forced through
// the private tables 33.9 ms, now 19.0; through the global table alone 107,
// now 65.) One key takes four slots per step, two keys two each: four would spill
// registers at 1024 threads (64M uniform rows over 20k groups: 2.31 ms with one
// or two, 2.80 with four).
template <int U>
__device__ __forceinline__ void global_rows1(const AggK& P, bool (&want)[U], const uint64_t (&k)[U], uint64_t (&s)[U],
                                             const uint64_t (&cur)[U], uint64_t* (&r)[U],
                                             unsigned long long& inserted, int limit) {
  constexpr int kLook = U == 1 ? 4 : 2;
  const int W = P.row_words;
  auto claim = [&](uint64_t* at, uint64_t key) -> bool {  // whether the slot is the key's now
    const unsigned long long old =
        atomicCAS(reinterpret_cast<unsigned long long*>(at), 0ull, static_cast<unsigned long long>(key));
    inserted += old == 0;
    return old == 0 || old == key;
  };
  bool any = false;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    r[u] = nullptr;
    if (!want[u]) continue;
    uint64_t* const at = P.table + s[u] * W;
    if (cur[u] == k[u] || (cur[u] == 0 && claim(at, k[u]))) {
      r[u] = at;
      want[u] = false;
    } else {
      if (++s[u] == P.cap) s[u] = 0;
      any = true;
    }
  }
  for (int t = 1; any && t < limit; t += kLook) {
    uint64_t w[U][kLook];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < kLook; ++j) {
        w[u][j] = 0;
        if (want[u]) w[u][j] = ld_relaxed(P.table + (s[u] + j < P.cap ? s[u] + j : s[u] + j - P.cap) * W);
      }
    any = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int j = 0; j < kLook; ++j) {
        if (!want[u]) continue;
        uint64_t* const at = P.table + s[u] * W;
        if (w[u][j] == k[u] || (w[u][j] == 0 && claim(at, k[u]))) {
          r[u] = at;
          want[u] = false;
        } else if (++s[u] == P.cap) {
          s[u] = 0;
        }
      }
      any |= want[u];
    }
  }
}

// The same for any key: the NULL key and key word 0 have rows of their own.
__device__ __forceinline__ uint64_t* global_row1(const AggK& P, bool kv, uint64_t k, uint64_t h,
                                                 unsigned long long& inserted, int limit) {
  if (!kv) return P.table + (P.cap + 1) * P.row_words;
  if (k == 0) return P.table + P.cap * P.row_words;
  bool want[1] = {true};
  const uint64_t key[1] = {k};
  uint64_t s[1] = {home_slot(h, P.cap)};
  const uint64_t cur[1] = {ld_relaxed(P.table + s[0] * P.row_words)};
  uint64_t* r[1];
  global_rows1<1>(P, want, key, s, cur, r, inserted, limit);
  return r[0];
}

// Multi-key global lookup/insert with a publish protocol: claim (0 -> 1), write
// null mask and key words, fence, publish the tag. Readers wait (bounded) on a
// row being published.
__device__ __forceinline__ uint64_t* global_rowN(const AggK& P, const uint64_t* words, uint64_t nullmask,
                                                 uint64_t h, unsigned long long& inserted) {
  const int W = P.row_words;
  const uint64_t tag = (h >> 32) | 2ull;
  uint64_t s = home_slot(h, P.cap);
  for (int t = 0; t < P.probe_limit; ++t) {
    uint64_t* r = P.table + s * W;
    uint64_t st = ld_acquire(r);
    if (st == 0) {
      const unsigned long long old = atomicCAS(reinterpret_cast<unsigned long long*>(r), 0ull, 1ull);
      if (old == 0) {
        r[1] = nullmask;
        for (int j = 0; j < P.nkeys; ++j) r[2 + j] = words[j];
        __threadfence();
        atomicExch(reinterpret_cast<unsigned long long*>(r), static_cast<unsigned long long>(tag));
        ++inserted;
        return r;
      }
      st = old;
    }
    st = wait_published(r, st, kSpinLimit, P.err);
    if (st == kRowClaimed) return nullptr;
    if (st == tag) {
      bool eq = ld_relaxed(r + 1) == nullmask;
      for (int j = 0; eq && j < P.nkeys; ++j) eq = ld_relaxed(r + 2 + j) == words[j];
      if (eq) return r;
    }
    s = (s + 1 == P.cap) ? 0 : s + 1;
  }
  return nullptr;
}

__device__ __forceinline__ void spill_row(const AggK& P, uint64_t p) {
  const unsigned long long i = atomicAdd(P.counters + 0, 1ull);
  if (i < P.spill_cap)
    P.spill_rows[i] = static_cast<uint32_t>(p);
  else
    atomicOr(P.err, kDevSpillOverflow);
}

// Row of key word k (nonzero) in a finished single-key table, or nullptr.
__device__ __forceinline__ uint64_t* find_row1(uint64_t* table, uint64_t cap, int W, uint64_t k) {
  uint64_t s = home_slot(key_hash1(k), cap);
  for (uint64_t t = 0; t < cap; ++t) {
    uint64_t* r = table + s * W;
    const uint64_t cur = r[0];
    if (cur == k) return r;
    if (cur == 0) return nullptr;
    if (++s == cap) s = 0;
  }
  return nullptr;
}

// Merges one field block `src` (a partial aggregate) into `dst`.
__device__ __forceinline__ void merge_fields(uint64_t* dst, const uint64_t* src, const AggK& P) {
  for (int f = 0; f < P.nfields; ++f) {
    const uint64_t v = src[f];
    if (v == 0) continue;  // zero is the identity of every field
    unsigned long long* d = reinterpret_cast<unsigned long long*>(dst + f);
    switch (P.fkind[f]) {
      case F_ROWS:
      case F_NULLS:
      case F_SUMI: atomicAdd(d, static_cast<unsigned long long>(v)); break;
      case F_SUMF: atomicAdd(reinterpret_cast<double*>(d), __longlong_as_double(static_cast<long long>(v))); break;
      default: atomicMax(d, static_cast<unsigned long long>(v)); break;
    }
  }
}

// Combines the rows of every peer group and lets each group's leader apply the
// result to `f` (its field block; ignored on other lanes). `space` says where
// `f` lives (RowSpace): a warp-private row is updated without atomics (one
// leader per group and one group per row within a warp), shared and global
// rows with reductions of their state space. One loop over the fields keeps
// the code small.
template <int NV>
__device__ __forceinline__ void warp_apply(uint64_t* f, bool leader, int space, unsigned peers, const PeerPlan& pp,
                                           const AggK& P, const bool (&vv)[kMaxVals],
                                           const uint64_t (&vb)[kMaxVals]) {
  if (leader) field_red_at(space, f, F_ROWS, static_cast<uint64_t>(__popc(peers)));
#pragma unroll 1
  for (int fi = 1; fi < P.nfields; ++fi) {
    const uint8_t kind = P.fkind[fi];
    const int c = P.fcol[fi];
    bool v = false;
    uint64_t b = 0;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      if (j == c) {
        v = vv[j];
        b = vb[j];
      }
    }
    const uint64_t x = peer_reduce(field_contrib(kind, v, b), kind, pp);
    if (leader) field_red_at(space, f + fi, kind, x);
  }
}

// ---------------------------------------------------------------------------
// The aggregation kernel. MODE 0: global (no key), 1: single key, 2: multi key.
// Warps walk the rows 32 at a time (blockDim.x is a multiple of 32), so every
// lane reaches the warp-wide intrinsics.
// ---------------------------------------------------------------------------
// Table-full signal (all lanes of the warp call it): inserts are counted per
// warp and published every 64; once the count passes P.full_at, lookups of new
// keys give up after a short probe and spill instead of walking probe_limit
// slots of a full table.
__device__ __forceinline__ void track_full(const AggK& P, unsigned lane, uint32_t iter, unsigned inserted_now,
                                           unsigned& pending, bool& full) {
  pending += __reduce_add_sync(0xffffffffu, inserted_now);
  if (pending >= 64 || (iter & 15) == 15) {
    if (lane == 0) {
      if (pending) {
        const unsigned long long before = atomicAdd(P.counters + 3, static_cast<unsigned long long>(pending));
        if (before + pending >= P.full_at) atomicExch(P.full_flag, 1u);
      }
      full = full || ld_relaxed_u32(P.full_flag) != 0;
    }
    pending = 0;
    full = __shfl_sync(0xffffffffu, full, 0);
  }
}

// Field sets with kernels of their own (qeg_warpagg.cuh): COUNT/SUM/MIN/MAX
// over an integer column plus SUM over an F64 column, and COUNT/SUM/AVG/MIN/
// MAX over one F64 column, each without and with NULL counts, and COUNT(*).
constexpr uint32_t kSpecIntF64 = 6u | spec_field(1, 0, 0) | spec_field(2, F_SUMI, 0) | spec_field(3, F_MINI, 0) |
                                 spec_field(4, F_MAXI, 0) | spec_field(5, 0, 1) | spec_field(6, F_SUMF, 1);
constexpr uint32_t kSpecIntF64Nulls = 6u | spec_field(1, F_NULLS, 0) | spec_field(2, F_SUMI, 0) |
                                      spec_field(3, F_MINI, 0) | spec_field(4, F_MAXI, 0) |
                                      spec_field(5, F_NULLS, 1) | spec_field(6, F_SUMF, 1);
constexpr uint32_t kSpecF64 = 4u | spec_field(1, 0, 0) | spec_field(2, F_SUMF, 0) | spec_field(3, F_MINF, 0) |
                              spec_field(4, F_MAXF, 0);
constexpr uint32_t kSpecF64Nulls = 4u | spec_field(1, F_NULLS, 0) | spec_field(2, F_SUMF, 0) |
                                   spec_field(3, F_MINF, 0) | spec_field(4, F_MAXF, 0);
constexpr uint32_t kSpecCount = 0u;
// SUM over an integer column plus SUM/MIN/MAX over an F64 column (bar-style
// aggregates: volume, then mean/low/high price) likewise.
constexpr uint32_t kSpecIntSumF64Stats = 6u | spec_field(1, 0, 0) | spec_field(2, F_SUMI, 0) | spec_field(3, 0, 1) |
                                         spec_field(4, F_SUMF, 1) | spec_field(5, F_MINF, 1) |
                                         spec_field(6, F_MAXF, 1);
constexpr uint32_t kSpecIntSumF64StatsNulls = kSpecIntSumF64Stats | spec_field(1, F_NULLS, 0) | spec_field(3, F_NULLS, 1);

// MODE 0 (no key) keeps one row per warp; MODE 1 (single key, QEG_AGG_GLOBAL)
// and MODE 2 (composite key) update the global table alone. The rows of a warp
// that share a group are combined before they are applied (warp peer
// aggregation), so a heavy hitter costs one global reduction per warp and
// field instead of one per row.
template <int MODE, int NV, uint32_t SPEC>
__global__ void __launch_bounds__(1024) agg_kernel(const AggK P) {
  extern __shared__ uint64_t sm[];
  // MODE 0: one row per warp, then the CTA's row. An odd stride in 8-byte
  // words, so the same field of different rows falls in different banks.
  const int SW = P.row_words | 1;
  const int fo = (MODE == 2) ? 2 + P.nkeys : 1;  // field offset within a global row
  const unsigned lane = threadIdx.x & 31u;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  uint64_t* wrows = sm + SW;
  if (MODE == 0) {
    for (int i = threadIdx.x; i < (1 + nwarps) * SW; i += blockDim.x) sm[i] = 0;
    __syncthreads();
  }

  unsigned long long inserted = 0;
  unsigned pending = 0;  // table-full signal state (track_full)
  bool full = MODE == 1 && P.full_flag && ld_relaxed_u32(P.full_flag) != 0;
  uint32_t iter = 0;
  const uint64_t step = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t base = static_cast<uint64_t>(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u); base < P.nrows;
       base += step, ++iter) {
    const uint64_t i = base + lane;
    bool live = i < P.nrows;
    uint64_t p = i;
    if (live && P.sel) {
      p = P.sel[i];
      if (p >= P.len) {
        atomicOr(P.err, kDevBadInput);
        live = false;
      }
    }
    bool vv[kMaxVals];
    uint64_t vb[kMaxVals];
#pragma unroll
    for (int c = 0; c < kMaxVals; ++c) {
      vv[c] = false;
      vb[c] = 0;
    }
    if (live) load_values<NV>(P, p, vv, vb);
    const unsigned livemask = __ballot_sync(0xffffffffu, live);

    if (MODE == 0) {
      const unsigned peers = live ? livemask : (1u << lane);
      const PeerPlan pp = plan_peers(peers, lane);
      if constexpr (SPEC != kGenericSpec)
        spec_apply<SPEC, NV>(&wrows[warp * SW + 1], live && __ffs(peers) - 1 == static_cast<int>(lane), kRowPrivate,
                             peers, pp, vv, vb);
      else
        warp_apply<NV>(&wrows[warp * SW + 1], live && __ffs(peers) - 1 == static_cast<int>(lane), kRowPrivate, peers,
                       pp, P, vv, vb);
      continue;
    }
    if (MODE == 1) {
      const DevCol& kc = P.key[0];
      const bool kv = live && col_valid(kc, p);
      const uint64_t k = kv ? key_word(kc, p) : 0;
      const bool key32 = kc.type == kI32 || kc.type == kSTR || kc.type == kBOOL;  // key words fit 32 bits
      // Peers: live lanes with the same key word and the same validity.
      const unsigned same = match_word64(k, lane, key32);
      const unsigned vmask = __ballot_sync(0xffffffffu, kv);
      unsigned peers = live ? (same & livemask & (kv ? vmask : ~vmask)) : (1u << lane);
      const bool leader = live && __ffs(peers) - 1 == static_cast<int>(lane);
      // The leader finds (or places) the group's row.
      uint64_t* f = nullptr;
      const unsigned long long ins0 = inserted;
      if (leader) {
        uint64_t* r = global_row1(P, kv, k, key_hash1(k), inserted, full ? kFullProbe : P.probe_limit);
        if (r) f = r + 1;
      }
      // A group whose row could not be placed spills each of its rows.
      const unsigned placed = __ballot_sync(0xffffffffu, f != nullptr);
      const bool ok = live && ((placed >> (__ffs(peers) - 1)) & 1u);
      if (live && !ok) {
        spill_row(P, p);
        peers = 1u << lane;
      }
      const PeerPlan pp = plan_peers(ok ? peers : (1u << lane), lane);
      if constexpr (SPEC != kGenericSpec) spec_apply<SPEC, NV>(f, leader && ok, kRowGlobal, peers, pp, vv, vb);
      else warp_apply<NV>(f, leader && ok, kRowGlobal, peers, pp, P, vv, vb);
      if (P.full_flag) track_full(P, lane, iter, inserted != ins0, pending, full);
      continue;
    }
    // MODE 2: composite key, global table only. Lanes with the same key tuple
    // combine like MODE 1: they match on the tuple hash, then every lane
    // checks its words against the match group's first lane (a lane that
    // differs -- a hash collision inside the warp -- goes alone), and the
    // group's leader finds the row and applies the combined fields.
    uint64_t words[kMaxKeys];
    uint64_t nullmask = live ? 0 : ~0ull, h = kHashSeed;
#pragma unroll
    for (int j = 0; j < kMaxKeys; ++j) {
      words[j] = 0;
      if (live && j < P.nkeys) {
        const bool kv = col_valid(P.key[j], p);
        words[j] = kv ? key_word(P.key[j], p) : 0;
        if (!kv) nullmask |= 1ull << j;
        h = hash_fold(h, kv ? words[j] : 0x9E3779B97F4A7C15ull);
      }
    }
    // (Matched on a 32-bit fold of the tuple hash; the word check below
    // drops any lane that collides.)
    const uint64_t hm = live ? h : ~static_cast<uint64_t>(lane);
    const unsigned same = __match_any_sync(0xffffffffu, static_cast<uint32_t>(hm ^ (hm >> 32)));
    const int ref = __ffs(same) - 1;
    const uint64_t ref_h = __shfl_sync(0xffffffffu, hm, ref);
    const uint64_t ref_nm = __shfl_sync(0xffffffffu, nullmask, ref);
    bool eq = ref_h == hm && ref_nm == nullmask;
#pragma unroll
    for (int j = 0; j < kMaxKeys; ++j)
      if (j < P.nkeys) eq &= __shfl_sync(0xffffffffu, words[j], ref) == words[j];
    const unsigned eqmask = __ballot_sync(0xffffffffu, eq);
    unsigned peers = (live && eq) ? (same & eqmask & livemask) : (1u << lane);
    const bool leader = live && __ffs(peers) - 1 == static_cast<int>(lane);
    uint64_t* f = nullptr;
    if (leader) {
      uint64_t* r = global_rowN(P, words, nullmask, h, inserted);
      if (r) f = r + fo;
    }
    const unsigned placed = __ballot_sync(0xffffffffu, f != nullptr);
    const bool ok = live && ((placed >> (__ffs(peers) - 1)) & 1u);
    if (live && !ok) {
      spill_row(P, p);
      peers = 1u << lane;
    }
    const PeerPlan pp = plan_peers(ok ? peers : (1u << lane), lane);
    if constexpr (SPEC != kGenericSpec) spec_apply<SPEC, NV>(f, leader && ok, kRowGlobal, peers, pp, vv, vb);
    else warp_apply<NV>(f, leader && ok, kRowGlobal, peers, pp, P, vv, vb);
  }

  if (MODE == 0) {  // the warps' rows into the CTA's, that into the table's
    __syncthreads();
    for (int i = threadIdx.x; i < nwarps; i += blockDim.x)
      if (wrows[i * SW + 1]) merge_fields(&sm[1], &wrows[i * SW + 1], P);
    __syncthreads();
    if (threadIdx.x == 0 && sm[1]) merge_fields(P.table + 1, &sm[1], P);
  }
  // Occupancy accounting: one atomic per warp.
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if ((threadIdx.x & 31) == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}

// Fills a private table's key words with the heavy hitters' table (hot_table:
// S key words, then the slots of the kPrivReps most frequent ones, which also
// get replica rows). A barrier must follow.
__device__ __forceinline__ void priv_preload(uint64_t* keys, int S, const uint64_t* hot, uint8_t* rep, uint16_t* rslot) {
  for (int i = threadIdx.x; i < S; i += blockDim.x) keys[i] = __ldg(hot + i);
  if (rep && threadIdx.x < kPrivReps) {
    const uint64_t s = __ldg(hot + S + threadIdx.x);
    rslot[threadIdx.x] = static_cast<uint16_t>(s);
    if (s < static_cast<uint64_t>(S)) rep[s] = static_cast<uint8_t>(threadIdx.x + 1);
  }
}

// ---------------------------------------------------------------------------
// Single key with a CTA-private table (QEG_AGG_SMEM). Each CTA walks one
// contiguous range of rows. A row whose key has a place in the private table
// (first come, four-slot buckets) is added there by its own lane with
// shared-memory reductions; any other row goes to the global table by its own
// lane with fire-and-forget reductions, its home slot's load issued before
// the shared-memory work. Lanes on one private word would serialise, so slots
// that a warp hits three times at once get a row per lane (priv_promote);
// that replaces combining the lanes' rows first (a match, a shuffle plan and a
// tree per field), which cost 917 warp instructions per 32 rows. Every
// kPrivWindow steps the CTA looks at the share of rows that missed: when it
// passes a quarter the table is flushed and refilled (keys clustered in time:
// the resident ones go stale), less and less often while that does not help.
// ---------------------------------------------------------------------------
constexpr int kPrivWindow = 8;
template <int NV>
constexpr int priv_rows() {  // rows per thread in flight (registers)
  return NV <= 2 ? 2 : 1;
}

// Merges the private table into the global table and clears it (every thread
// of the CTA calls it). A row that finds no place there stays for the next
// flush, or goes to the partial-row list at the final one. CTAs start at
// different slots, so they do not merge the same group at the same time.
template <bool SSUM = false>
__device__ __forceinline__ void priv_flush1(uint64_t* keys, const PrivT& T, const PrivK& A, const AggK& P, uint8_t* rep,
                                            uint16_t* rslot, unsigned* nrep, bool final,
                                            unsigned long long& inserted) {
  priv_fence();
  priv_fold<SSUM>(T, A, rslot, *nrep, P.fkind, P.nfields);
  priv_fence();
  const int S = A.slots, W = P.row_words;
  const int rot = static_cast<int>((blockIdx.x * 97u) % static_cast<unsigned>(S + 2));
  const int limit = P.full_flag && ld_relaxed_u32(P.full_flag) != 0 ? kFullProbe : P.probe_limit;
  for (int i = threadIdx.x; i < S + 2; i += blockDim.x) {
    int sr = i + rot;
    if (sr >= S + 2) sr -= S + 2;
    rep[sr] = 0;
    if (priv_load<SSUM>(T, A, 0, F_ROWS, sr) == 0) continue;
    const uint64_t k = sr < S ? keys[sr] : 0;
    uint64_t* dst = global_row1(P, sr != S + 1, k, key_hash1(k), inserted, limit);
    if (dst) {
#pragma unroll 1
      for (int f = 0; f < P.nfields; ++f) {
        if ((A.skip >> f) & 1u) continue;
        const uint8_t kind = P.fkind[f];
        field_red<kRowGlobal>(dst + 1 + f, kind, priv_load<SSUM>(T, A, f, kind, sr));
      }
    } else if (final) {
      const unsigned long long j = atomicAdd(P.counters + 1, 1ull);
      if (j < P.part_cap) {
        P.spill_parts[j * W] = k;
        for (int f = 0; f < P.nfields; ++f)
          P.spill_parts[j * W + 1 + f] = ((A.skip >> f) & 1u) ? 0 : priv_load<SSUM>(T, A, f, P.fkind[f], sr);
      } else {
        atomicOr(P.err, kDevSpillOverflow);
      }
    } else {
      continue;
    }
    if (final) continue;
    for (int f = 0; f < P.nfields; ++f)
      if (!((A.skip >> f) & 1u)) priv_clear<SSUM>(T, A, f, P.fkind[f], sr);
    if (sr < S) keys[sr] = 0;
  }
  if (threadIdx.x == 0) *nrep = 0;
  __syncthreads();
}

template <int NV, uint32_t SPEC, bool SSUM = false>
__global__ void __launch_bounds__(1024) agg_private_kernel(const __grid_constant__ AggK P,
                                                           const __grid_constant__ PrivK A) {
  constexpr int kPrivU = priv_rows<NV>();
  extern __shared__ __align__(16) uint64_t sm[];
  __shared__ unsigned s_nrep, s_miss[3];
  __shared__ uint16_t s_rslot[kPrivReps];
  uint64_t* keys = sm;
  const PrivT T = priv_init(sm, A);
  uint8_t* rep = reinterpret_cast<uint8_t*>(sm) + A.rep_off;
  const int S = A.slots, W = P.row_words;
  const unsigned lane = threadIdx.x & 31u;
  if (threadIdx.x == 0) {
    s_nrep = 0;
    s_miss[0] = s_miss[1] = s_miss[2] = 0;
  }
  __syncthreads();
  const int insert = P.smem_insert;
  if (P.nhot > 0) {  // preloaded heavy hitters, the first ones with replicas
    priv_preload(keys, S, P.hot, rep, s_rslot);
    if (threadIdx.x == 0) s_nrep = kPrivReps;
    __syncthreads();
  }

  unsigned long long inserted = 0, tracked = 0;
  unsigned pending = 0;  // table-full signal state (track_full)
  bool full = P.full_flag && ld_relaxed_u32(P.full_flag) != 0;
  unsigned missed = 0;             // this warp's rows of the window that missed the private table
  unsigned before = 0;             // the CTA's misses in the window before the last flush
  int wait = 0, backoff = 0;       // windows until the next flush may happen
  int judge = 0;                   // windows until the last flush is judged
  unsigned decision = 0;           // windows whose misses were summed
  const DevCol& kc = P.key[0];
  const uint64_t per = ((P.nrows + gridDim.x - 1) / gridDim.x + 31) & ~31ull;
  const uint64_t lo = min(per * blockIdx.x, P.nrows), hi = min(lo + per, P.nrows);
  const uint64_t span = static_cast<uint64_t>(blockDim.x) * kPrivU;
  uint32_t step = 0;
  for (uint64_t b0 = lo; b0 < hi; b0 += span, ++step) {
    bool live[kPrivU], kv[kPrivU], vv[kPrivU][kMaxVals];
    uint64_t p[kPrivU], k[kPrivU], vb[kPrivU][kMaxVals];
#pragma unroll
    for (int u = 0; u < kPrivU; ++u) {
      const uint64_t i = b0 + static_cast<uint64_t>(u) * blockDim.x + threadIdx.x;
      live[u] = i < hi;
      p[u] = i;
      if (live[u] && P.sel) {
        p[u] = P.sel[i];
        if (p[u] >= P.len) {
          atomicOr(P.err, kDevBadInput);
          live[u] = false;
        }
      }
#pragma unroll
      for (int c = 0; c < kMaxVals; ++c) {
        vv[u][c] = false;
        vb[u][c] = 0;
      }
      kv[u] = false;
      k[u] = 0;
      if (live[u]) {
        kv[u] = col_valid(kc, p[u]);
        if (kv[u]) k[u] = key_word(kc, p[u]);
        load_values<NV>(P, p[u], vv[u], vb[u]);
      }
    }
    // Private slots, and the home slots of the rows that have none.
    int slot[kPrivU];
    uint64_t home[kPrivU], cur[kPrivU];
#pragma unroll
    for (int u = 0; u < kPrivU; ++u) {
      slot[u] = -1;
      home[u] = cur[u] = 0;
      if (live[u]) {
        const uint64_t h = key_hash1(k[u]);
        slot[u] = !kv[u] ? S + 1 : (k[u] == 0 ? S : (insert ? priv_slot(keys, S, k[u], h) : hot_slot(keys, S, k[u], h)));
        if (slot[u] < 0) {
          home[u] = home_slot(h, P.cap);
          cur[u] = ld_relaxed(P.table + home[u] * W);
        }
      }
      missed += __popc(__ballot_sync(0xffffffffu, live[u] && slot[u] < 0));
    }
    if (insert && (step < 4 || (step & 7) == 0)) priv_promote(slot[0], rep, s_rslot, &s_nrep, lane);
#pragma unroll
    for (int u = 0; u < kPrivU; ++u) {
      if (slot[u] >= 0) {
        const int id = rep[slot[u]];
        priv_apply<SPEC, NV, SSUM>(T, A, id ? S + 2 + (id - 1) * 32 + static_cast<int>(lane) : slot[u], P.fkind, P.fcol,
                             P.nfields, vv[u], vb[u]);
      }
    }
    bool cold[kPrivU];
    uint64_t* r[kPrivU];
#pragma unroll
    for (int u = 0; u < kPrivU; ++u) cold[u] = live[u] && slot[u] < 0;
    global_rows1<kPrivU>(P, cold, k, home, cur, r, inserted, full ? kFullProbe : P.probe_limit);
#pragma unroll
    for (int u = 0; u < kPrivU; ++u) {
      if (live[u] && slot[u] < 0) {
        if (r[u]) global_apply<SPEC, NV>(r[u] + 1, P.fkind, P.fcol, P.nfields, vv[u], vb[u]);
        else spill_row(P, p[u]);
      }
    }
    if (P.full_flag) {
      // (With the rows that a flush inserted: without them a table that is
      // too small was never found full, and every row searched it to the
      // probe limit.)
      track_full(P, lane, step, static_cast<unsigned>(inserted - tracked), pending, full);
      tracked = inserted;
    }
    if (insert && (step & (kPrivWindow - 1)) == kPrivWindow - 1) {
      if (judge > 1 || (judge == 0 && wait > 0)) {
        // Nothing to decide: no barrier.
        if (judge > 1) --judge;
        else --wait;
        missed = 0;
        continue;
      }
      // The window's misses, summed over the CTA (three sums in turn: the one
      // cleared here is next used after another barrier).
      unsigned* sum = &s_miss[decision % 3];
      // Not once the global table is full: a flush would search it in vain for
      // most groups, and its refill would spill.
      if (lane == 0 && missed && !full) atomicAdd(sum, missed);
      missed = 0;
      __syncthreads();
      const unsigned m = *sum;
      if (threadIdx.x == 0) s_miss[(decision + 2) % 3] = 0;
      ++decision;
      // A flush is judged by the second window after it: in the first the
      // refill alone keeps the misses low.
      if (judge > 0) {
        judge = 0;
        backoff = m < before - before / 5 ? 0 : min(2 * backoff + 1, 63);
        wait = backoff;
      }
      if (wait > 0) {
        --wait;
      } else if (m > span * kPrivWindow / 4) {
        priv_flush1<SSUM>(keys, T, A, P, rep, s_rslot, &s_nrep, false, inserted);
        before = m;
        judge = 2;
      }
    }
  }
  priv_flush1<SSUM>(keys, T, A, P, rep, s_rslot, &s_nrep, true, inserted);
  // Occupancy accounting: one atomic per warp.
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if (lane == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}

// ---------------------------------------------------------------------------
// Composite keys with a CTA-private table (QEG_AGG_SMEM in mode 2, opt-in).
// Each CTA walks one contiguous range of rows and keeps the groups it meets
// in a shared-memory table of composite rows ([state][null mask][key
// words][fields], the global row format), which it flushes into the global
// table whenever half of it is in use, and at the end. It pays off when the
// groups live at one time in a CTA's range fit its table (input with
// locality); most rows then cost shared-memory reductions, and the global
// table sees one merge per (CTA, group, flush) instead of one per row. Groups
// that miss the private table (probe limit, or no free slot while the global
// table is full) take the global path and spill as usual; partial rows that
// cannot be merged at the final flush go to the partial-row list, merged
// after the host grows the table.
// ---------------------------------------------------------------------------
constexpr int kPrivProbe = 16;

// Composite-row hash of a row's key words and NULL mask (the kernels' rule).
__device__ __forceinline__ uint64_t row_hashN(const AggK& P, const uint64_t* words, uint64_t nullmask) {
  uint64_t h = kHashSeed;
  for (int j = 0; j < P.nkeys; ++j) h = hash_fold(h, ((nullmask >> j) & 1ull) ? 0x9E3779B97F4A7C15ull : words[j]);
  return h;
}

// The private-table slot of a key tuple (found, or claimed when `may_insert`),
// or -1. A claim publishes the key words before the row's tag (fence within
// the CTA); a lookup that sees a claim in progress waits for it, bounded.
__device__ __forceinline__ int priv_row(uint64_t* sm, int S, int SW, const AggK& P, const uint64_t* words,
                                        uint64_t nullmask, uint64_t h, unsigned* used, bool may_insert) {
  const uint64_t tag = (h >> 32) | 2ull;
  int s = static_cast<int>(h & static_cast<uint64_t>(S - 1));
  for (int t = 0; t < kPrivProbe; ++t) {
    uint64_t* r = &sm[s * SW];
    uint64_t st = ld_volatile_shared(r);
    if (st == 0) {
      if (!may_insert) return -1;
      const unsigned long long old = atomicCAS(reinterpret_cast<unsigned long long*>(r), 0ull, 1ull);
      if (old == 0) {
        r[1] = nullmask;
        for (int j = 0; j < P.nkeys; ++j) r[2 + j] = words[j];
        __threadfence_block();
        atomicExch(reinterpret_cast<unsigned long long*>(r), static_cast<unsigned long long>(tag));
        atomicAdd(used, 1u);
        return s;
      }
      st = old;
    }
    int spins = 0;
    while (st == 1) {
      if (++spins > kSpinLimit) {
        atomicOr(P.err, kDevSpinTimeout);
        return -1;
      }
      st = ld_volatile_shared(r);
    }
    if (st == tag) {
      __threadfence_block();
      bool eq = ld_volatile_shared(r + 1) == nullmask;
      for (int j = 0; eq && j < P.nkeys; ++j) eq = ld_volatile_shared(r + 2 + j) == words[j];
      if (eq) return s;
    }
    s = (s + 1) & (S - 1);
  }
  return -1;
}

// Merges the private table into the global table (every thread of the CTA
// calls it). Rows that merge are cleared; the rest stay (global table full)
// or, at the final flush, go to the partial-row list.
__device__ __forceinline__ void priv_flush(uint64_t* sm, int S, int SW, const AggK& P, unsigned* used,
                                           unsigned* left, int* gfull, bool final, unsigned long long& inserted) {
  const int W = P.row_words;
  const int fo = 2 + P.nkeys;
  if (threadIdx.x == 0) *left = 0;
  __syncthreads();
  for (int slot = threadIdx.x; slot < S; slot += blockDim.x) {
    uint64_t* src = &sm[slot * SW];
    if (src[0] < 2) continue;
    uint64_t words[kMaxKeys];
    for (int j = 0; j < P.nkeys; ++j) words[j] = src[2 + j];
    uint64_t* dst = global_rowN(P, words, src[1], row_hashN(P, words, src[1]), inserted);
    if (dst) {
      merge_fields(dst + fo, src + fo, P);
    } else if (final) {
      const unsigned long long i = atomicAdd(P.counters + 1, 1ull);
      if (i < P.part_cap) {
        for (int w = 0; w < W; ++w) P.spill_parts[i * W + w] = src[w];
      } else {
        atomicOr(P.err, kDevSpillOverflow);
      }
    } else {
      atomicAdd(left, 1u);
      continue;
    }
    for (int w = 0; w < W; ++w) src[w] = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *used = *left;
    if (*left >= static_cast<unsigned>(S / 2)) *gfull = 1;
  }
  __syncthreads();
}

template <int NV, uint32_t SPEC>
__global__ void __launch_bounds__(512, 2) agg2_private_kernel(const AggK P) {
  extern __shared__ uint64_t sm[];
  const int W = P.row_words;
  const int SW = W | 1;
  const int S = P.smem_slots;
  const int fo = 2 + P.nkeys;
  const unsigned lane = threadIdx.x & 31u;
  __shared__ unsigned s_used, s_left;
  __shared__ int s_gfull;
  for (int i = threadIdx.x; i < S * SW; i += blockDim.x) sm[i] = 0;
  if (threadIdx.x == 0) {
    s_used = 0;
    s_gfull = 0;
  }
  __syncthreads();
  unsigned long long inserted = 0;
  const uint64_t per = (P.nrows + gridDim.x - 1) / gridDim.x;
  const uint64_t chunk = (per + blockDim.x - 1) / blockDim.x * blockDim.x;
  const uint64_t r0 = static_cast<uint64_t>(blockIdx.x) * chunk;
  const uint64_t r1 = r0 + chunk < P.nrows ? r0 + chunk : P.nrows;
  // Block-uniform loop: every thread makes the same passes (the flush check
  // synchronises the CTA after each one).
  for (uint64_t base = r0; base < r1; base += blockDim.x) {
    const uint64_t i = base + threadIdx.x;
    bool live = i < r1;
    uint64_t p = i;
    if (live && P.sel) {
      p = P.sel[i];
      if (p >= P.len) {
        atomicOr(P.err, kDevBadInput);
        live = false;
      }
    }
    bool vv[kMaxVals];
    uint64_t vb[kMaxVals];
#pragma unroll
    for (int c = 0; c < kMaxVals; ++c) {
      vv[c] = false;
      vb[c] = 0;
    }
    if (live) load_values<NV>(P, p, vv, vb);
    const unsigned livemask = __ballot_sync(0xffffffffu, live);
    uint64_t words[kMaxKeys];
    uint64_t nullmask = live ? 0 : ~0ull, h = kHashSeed;
#pragma unroll
    for (int j = 0; j < kMaxKeys; ++j) {
      words[j] = 0;
      if (live && j < P.nkeys) {
        const bool kv = col_valid(P.key[j], p);
        words[j] = kv ? key_word(P.key[j], p) : 0;
        if (!kv) nullmask |= 1ull << j;
        h = hash_fold(h, kv ? words[j] : 0x9E3779B97F4A7C15ull);
      }
    }
    // Peers: lanes with the same key tuple (hash match, then an exact check
    // against the match group's first lane), as in agg_kernel's mode 2.
    // (Matched on a 32-bit fold of the tuple hash; the word check below
    // drops any lane that collides.)
    const uint64_t hm = live ? h : ~static_cast<uint64_t>(lane);
    const unsigned same = __match_any_sync(0xffffffffu, static_cast<uint32_t>(hm ^ (hm >> 32)));
    const int ref = __ffs(same) - 1;
    const uint64_t ref_h = __shfl_sync(0xffffffffu, hm, ref);
    const uint64_t ref_nm = __shfl_sync(0xffffffffu, nullmask, ref);
    bool eq = ref_h == hm && ref_nm == nullmask;
#pragma unroll
    for (int j = 0; j < kMaxKeys; ++j)
      if (j < P.nkeys) eq &= __shfl_sync(0xffffffffu, words[j], ref) == words[j];
    const unsigned eqmask = __ballot_sync(0xffffffffu, eq);
    unsigned peers = (live && eq) ? (same & eqmask & livemask) : (1u << lane);
    const bool leader = live && __ffs(peers) - 1 == static_cast<int>(lane);
    uint64_t* f = nullptr;
    int space = kRowGlobal;
    if (leader) {
      const int slot = priv_row(sm, S, SW, P, words, nullmask, h, &s_used, s_gfull == 0);
      if (slot >= 0) {
        f = &sm[slot * SW + fo];
        space = kRowShared;
      } else {
        uint64_t* r = global_rowN(P, words, nullmask, h, inserted);
        if (r) f = r + fo;
      }
    }
    const unsigned placed = __ballot_sync(0xffffffffu, f != nullptr);
    const bool ok = live && ((placed >> (__ffs(peers) - 1)) & 1u);
    if (live && !ok) {
      spill_row(P, p);
      peers = 1u << lane;
    }
    const PeerPlan pp = plan_peers(ok ? peers : (1u << lane), lane);
    if constexpr (SPEC != kGenericSpec) spec_apply<SPEC, NV>(f, leader && ok, space, peers, pp, vv, vb);
    else warp_apply<NV>(f, leader && ok, space, peers, pp, P, vv, vb);
    // One CTA-wide decision (a barrier that also ORs the predicate), so every
    // thread enters the flush, or none does.
    if (__syncthreads_or(threadIdx.x == 0 && s_used >= static_cast<unsigned>(S / 2) && s_gfull == 0))
      priv_flush(sm, S, SW, P, &s_used, &s_left, &s_gfull, false, inserted);
  }
  __syncthreads();
  priv_flush(sm, S, SW, P, &s_used, &s_left, &s_gfull, true, inserted);
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if ((threadIdx.x & 31) == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}

// Re-inserts every occupied row of `old` into the (zeroed) table of P.
template <int MODE>
__global__ void rehash_kernel(const AggK P, const uint64_t* __restrict__ old, uint64_t old_cap) {
  const int W = P.row_words;
  unsigned long long inserted = 0;
  const uint64_t total = (MODE == 1) ? old_cap + 2 : old_cap;
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < total;
       s += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t* src = old + s * W;
    uint64_t* dst = nullptr;
    if (MODE == 1) {
      if (s == old_cap) {
        dst = P.table + P.cap * W;
      } else if (s == old_cap + 1) {
        dst = P.table + (P.cap + 1) * W;
      } else {
        const uint64_t k = src[0];
        if (k == 0) continue;
        // The new table has room for every row: probe as far as it takes.
        dst = global_row1(P, true, k, key_hash1(k), inserted, static_cast<int>(P.cap < (1ull << 30) ? P.cap : (1ull << 30)));
      }
      if (!dst) {
        atomicOr(P.err, kDevSpillOverflow);
        continue;
      }
      for (int f = 1; f < W; ++f) dst[f] = src[f];
    } else {
      const uint64_t st = src[0];
      if (st < 2) continue;
      uint64_t words[kMaxKeys];
      for (int j = 0; j < P.nkeys; ++j) words[j] = src[2 + j];
      uint64_t h = kHashSeed;
      for (int j = 0; j < P.nkeys; ++j) h = hash_fold(h, ((src[1] >> j) & 1) ? 0x9E3779B97F4A7C15ull : words[j]);
      dst = global_rowN(P, words, src[1], h, inserted);
      if (!dst) {
        atomicOr(P.err, kDevSpillOverflow);
        continue;
      }
      for (int f = 2 + P.nkeys; f < W; ++f) dst[f] = src[f];
    }
  }
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if ((threadIdx.x & 31) == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}

// ---------------------------------------------------------------------------
// Partitioned strategy (QEG_AGG_PARTITIONED, single key), for tables far
// beyond what L2 holds. Three passes over the batch: a sizing pass counts, per
// key-hash partition, the rows that are not heavy hitters; the first pass
// aggregates the heavy hitters (the sketch's most frequent keys) in read-only
// CTA-private tables and appends every other row to its partition's region of
// the pool; the second pass aggregates one partition per CTA in a private
// table and appends the groups to the tail rows. A pool row is the key word,
// one word per value column and, where a value may be NULL, a word of validity
// bits, padded so that one 16- or 32-byte store (or a few) writes it. The
// partition is the top bits of the key hash, a second-pass slot the bits below.
// ---------------------------------------------------------------------------
// Words of a pool row; MASK: with validity bits (where padding leaves room
// for them they are always there).
template <int NV, bool MASK>
constexpr int pool_words() {
  const int w = 1 + NV + ((MASK || NV >= 2) ? 1 : 0);
  return w <= 2 ? 2 : (w + 3) / 4 * 4;
}

template <int PW>
__device__ __forceinline__ void pool_store(uint64_t* p, const uint64_t (&w)[PW]) {
  if constexpr (PW == 2) {
    asm volatile("st.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(w[0]), "l"(w[1]) : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < PW; i += 4)
      asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p + i), "l"(w[i]), "l"(w[i + 1]), "l"(w[i + 2]),
                   "l"(w[i + 3])
                   : "memory");
  }
}

template <int PW>
__device__ __forceinline__ void pool_load(const uint64_t* p, uint64_t (&w)[PW]) {
  if constexpr (PW == 2) {
    asm volatile("ld.global.L1::no_allocate.v2.b64 {%0, %1}, [%2];" : "=l"(w[0]), "=l"(w[1]) : "l"(p));
  } else {
#pragma unroll
    for (int i = 0; i < PW; i += 4)
      asm volatile("ld.global.L1::no_allocate.v4.b64 {%0, %1, %2, %3}, [%4];"
                   : "=l"(w[i]), "=l"(w[i + 1]), "=l"(w[i + 2]), "=l"(w[i + 3])
                   : "l"(p + i));
  }
}

// Cursors lie in sectors of their own: packed, those of a thousand partitions
// would share a few L2 slices that every row's atomic goes to.
constexpr int kCursorWords = 8;

// The pool and its partitions (np = 2^(64 - shift) of them).
struct PoolK {
  uint64_t* rows;
  uint32_t* cursor;  // next pool row of each partition, kCursorWords apart
  uint32_t* hist;    // sizing pass: rows per partition
  uint32_t* off;     // [np + 1] first pool row of each partition
  uint64_t total;    // pool rows
  int shift;         // partition of a key = key_hash1(key) >> shift
};

// Sizing pass: rows per partition of every row that will reach the pool (a
// non-NULL key other than key word 0 and not a heavy hitter). 32-bit counters
// per CTA in shared memory, added to Q.hist at the end. Each thread has R
// rows in flight per iteration, their key loads issued before any is used.
template <int R>
__global__ void __launch_bounds__(1024) part_hist_kernel(const __grid_constant__ AggK P, const PoolK Q, int S) {
  extern __shared__ uint64_t hsm[];
  uint32_t* cnt = reinterpret_cast<uint32_t*>(hsm + S);
  const uint32_t np = 1u << (64 - Q.shift);
  for (uint32_t i = threadIdx.x; i < np; i += blockDim.x) cnt[i] = 0;
  for (int i = threadIdx.x; i < S; i += blockDim.x) hsm[i] = 0;
  __syncthreads();
  if (P.nhot > 0) priv_preload(hsm, S, P.hot, nullptr, nullptr);
  __syncthreads();
  const DevCol& kc = P.key[0];
  const uint64_t tile = static_cast<uint64_t>(blockDim.x) * R;
  for (uint64_t base = blockIdx.x * tile; base < P.nrows; base += static_cast<uint64_t>(gridDim.x) * tile) {
    uint64_t kw[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const uint64_t i = base + static_cast<uint64_t>(j) * blockDim.x + threadIdx.x;
      bool ok = i < P.nrows;
      uint64_t p = i;
      if (ok && P.sel) {
        p = P.sel[i];
        ok = p < P.len;  // (the first pass reports it)
      }
      ok = ok && col_valid(kc, p);
      kw[j] = ok ? key_word(kc, p) : 0;
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const uint64_t k = kw[j], h = key_hash1(k);
      if (k != 0 && (P.nhot == 0 || hot_slot(hsm, S, k, h) < 0)) atomicAdd(&cnt[h >> Q.shift], 1u);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < np; i += blockDim.x)
    if (cnt[i]) atomicAdd(Q.hist + i, cnt[i]);
}

// Region starts: one CTA scans the (at most 2^15) counts into Q.off and the
// append cursors, and leaves the total in *total. Thread t of the CTA holds
// counts t, t + 1024, ...: every load is coalesced and in flight at once.
__global__ void __launch_bounds__(1024) part_scan_kernel(const PoolK Q, unsigned long long* total) {
  constexpr int kPer = 1 << (kPartMaxBits - 10);
  __shared__ uint32_t s_sum[kPer * 32], s_warp[32];
  const uint32_t np = 1u << (64 - Q.shift);
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  auto warp_scan = [&](uint32_t v) {  // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= static_cast<unsigned>(o)) v += t;
    }
    return v;
  };
  uint32_t cnt[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t i = j * 1024 + threadIdx.x;
    cnt[j] = i < np ? Q.hist[i] : 0;
  }
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t v = warp_scan(cnt[j]);
    if (lane == 31) s_sum[j * 32 + warp] = v;
  }
  __syncthreads();
  // The kPer * 32 warp sums, scanned by the CTA (kPer = 32: one per thread).
  static_assert(kPer == 32, "one warp sum per thread");
  const uint32_t own = s_sum[threadIdx.x], incl = warp_scan(own);
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = s_warp[lane];
    s_warp[lane] = warp_scan(w) - w;
  }
  __syncthreads();
  s_sum[threadIdx.x] = s_warp[warp] + incl - own;
  if (threadIdx.x == 1023) {
    Q.off[np] = s_warp[warp] + incl;
    *total = s_warp[warp] + incl;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t i = j * 1024 + threadIdx.x;
    const uint32_t at = s_sum[j * 32 + warp] + warp_scan(cnt[j]) - cnt[j];
    if (i < np) Q.off[i] = Q.cursor[i * kCursorWords] = at;
  }
}

// First pass. Heavy hitters (and the NULL key and key word 0, which always
// have rows) are added to the CTA's private table, lane by lane; every other
// row is appended to its partition's region: one atomic reserves its place,
// issued before the shared-memory work of the heavy hitters, and one or two
// wide stores write it (the open ends of all regions stay in L2, which merges
// them into whole lines). At the end each CTA merges its table into the
// global one.
template <int NV, uint32_t SPEC, bool MASK>
__global__ void __launch_bounds__(1024) part_pass1_kernel(const __grid_constant__ AggK P,
                                                          const __grid_constant__ PrivK A, const PoolK Q) {
  constexpr int U = priv_rows<NV>();
  constexpr int PW = pool_words<NV, MASK>();
  extern __shared__ __align__(16) uint64_t sm[];
  __shared__ unsigned s_nrep;
  __shared__ uint16_t s_rslot[kPrivReps];
  uint64_t* keys = sm;
  const PrivT T = priv_init(sm, A);
  uint8_t* rep = reinterpret_cast<uint8_t*>(sm) + A.rep_off;
  const int S = A.slots;
  const unsigned lane = threadIdx.x & 31u;
  __syncthreads();
  if (P.nhot > 0) priv_preload(keys, S, P.hot, rep, s_rslot);
  if (threadIdx.x == 0) s_nrep = P.nhot > 0 ? kPrivReps : 0;
  __syncthreads();
  const DevCol& kc = P.key[0];
  const uint64_t span = static_cast<uint64_t>(blockDim.x) * U;
  for (uint64_t b0 = blockIdx.x * span; b0 < P.nrows; b0 += gridDim.x * span) {
    bool live[U], vv[U][kMaxVals];
    uint64_t p[U], k[U], vb[U][kMaxVals];
    int slot[U];
    uint32_t at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t i = b0 + static_cast<uint64_t>(u) * blockDim.x + threadIdx.x;
      live[u] = i < P.nrows;
      p[u] = i;
      if (live[u] && P.sel) {
        p[u] = P.sel[i];
        if (p[u] >= P.len) {
          atomicOr(P.err, kDevBadInput);
          live[u] = false;
        }
      }
#pragma unroll
      for (int c = 0; c < kMaxVals; ++c) {
        vv[u][c] = false;
        vb[u][c] = 0;
      }
      k[u] = 0;
      slot[u] = -1;
      if (live[u]) {
        slot[u] = col_valid(kc, p[u]) ? -1 : S + 1;
        if (slot[u] < 0) k[u] = key_word(kc, p[u]);
        load_values<NV>(P, p[u], vv[u], vb[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      at[u] = 0;
      if (live[u] && slot[u] < 0) {
        const uint64_t h = key_hash1(k[u]);
        if (k[u] == 0) slot[u] = S;
        else if (P.nhot > 0) slot[u] = hot_slot(keys, S, k[u], h);
        if (slot[u] < 0) at[u] = atomicAdd(Q.cursor + (h >> Q.shift) * kCursorWords, 1u);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (slot[u] >= 0) {
        const int id = rep[slot[u]];
        priv_apply<SPEC, NV>(T, A, id ? S + 2 + (id - 1) * 32 + static_cast<int>(lane) : slot[u], P.fkind, P.fcol,
                             P.nfields, vv[u], vb[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (live[u] && slot[u] < 0) {
        if (at[u] < Q.total) {
          uint64_t w[PW], mask = 0;
          w[0] = k[u];
#pragma unroll
          for (int c = 0; c < NV; ++c) {
            w[1 + c] = vb[u][c];
            mask |= vv[u][c] ? 1ull << c : 0;
          }
          if constexpr (PW > 1 + NV) {
            w[1 + NV] = mask;
#pragma unroll
            for (int i = 2 + NV; i < PW; ++i) w[i] = 0;
          }
          pool_store<PW>(Q.rows + static_cast<uint64_t>(at[u]) * PW, w);
        } else {
          spill_row(P, p[u]);  // (the sizing pass counted every such row: not reached)
        }
      }
    }
  }
  unsigned long long inserted = 0;
  priv_flush1(keys, T, A, P, rep, s_rslot, &s_nrep, true, inserted);
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if (lane == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}

// Reads one pool row into a key word and values.
template <int NV, bool MASK>
__device__ __forceinline__ void pool_row(const uint64_t (&w)[pool_words<NV, MASK>()], int nvals, uint64_t& k,
                                         bool (&vv)[kMaxVals], uint64_t (&vb)[kMaxVals]) {
  constexpr int PW = pool_words<NV, MASK>();
  k = w[0];
#pragma unroll
  for (int c = 0; c < kMaxVals; ++c) {
    vv[c] = false;
    vb[c] = 0;
    if (c < NV) {
      vb[c] = w[1 + c];
      if constexpr (PW > 1 + NV) vv[c] = (w[1 + NV] >> c) & 1u;
      else vv[c] = c < nvals;
    }
  }
}

// Second pass: each CTA takes partitions in turn and aggregates the
// partition's pool rows (every key nonzero and non-NULL) in a private table,
// lane by lane, R rows per thread loaded before any is applied; then it
// appends the table's groups to the tail rows with one reservation per CTA and
// clears the rows it used. Two CTAs per SM: one's loads and group output
// overlap the other's table work. A partition with more groups than the table
// holds is listed as failed and appends nothing (its rows go to the global
// table instead), so the pass can be re-run with a larger tail buffer.
template <int NV, uint32_t SPEC, bool MASK>
__global__ void __launch_bounds__(512, 2) part_agg_kernel(const __grid_constant__ AggK P,
                                                          const __grid_constant__ PrivK A, const PoolK Q,
                                                          const PartB B) {
  constexpr int PW = pool_words<NV, MASK>();
  constexpr int R = PW == 2 ? 4 : (PW == 4 ? 2 : 1);
  extern __shared__ __align__(16) uint64_t sm[];
  __shared__ int s_fail;
  __shared__ unsigned s_groups;
  __shared__ unsigned long long s_base;
  uint64_t* keys = sm;
  const PrivT T = priv_init(sm, A);
  // The slots in use, in the order they were claimed (after the table).
  uint16_t* used = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(sm) + A.bytes);
  const int W = P.row_words, S = A.slots;
  const int bits = 64 - Q.shift;
  const uint32_t np = 1u << bits;
  for (uint32_t part = blockIdx.x; part < np; part += gridDim.x) {
    if (threadIdx.x == 0) s_fail = 0, s_groups = 0;
    __syncthreads();
    const uint32_t begin = Q.off[part], n = Q.off[part + 1] - begin;
    for (uint32_t b0 = 0; b0 < n; b0 += blockDim.x * R) {
      uint64_t w[R][PW];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const uint32_t at = b0 + j * blockDim.x + threadIdx.x;
#pragma unroll
        for (int i = 0; i < PW; ++i) w[j][i] = 0;
        if (at < n) pool_load<PW>(Q.rows + static_cast<uint64_t>(begin + at) * PW, w[j]);
      }
      int slot[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const uint64_t k = w[j][0];  // (pool keys are nonzero: zero marks a row past the partition's end)
        const uint64_t h = key_hash1(k);
        uint32_t s = static_cast<uint32_t>((((h << bits) >> 32) * static_cast<uint32_t>(S)) >> 32);
        slot[j] = -1;
        bool look = k != 0;
        for (int t = 0; look && t <= S / 2; ++t) {
          unsigned long long cur = *reinterpret_cast<const volatile unsigned long long*>(keys + s);
          if (cur == 0) {
            cur = atomicCAS(reinterpret_cast<unsigned long long*>(keys + s), 0ull, static_cast<unsigned long long>(k));
            if (cur == 0) {
              used[atomicAdd(&s_groups, 1u)] = static_cast<uint16_t>(s);
              cur = k;
            }
          }
          if (cur == k) {
            slot[j] = static_cast<int>(s);
            look = false;
          } else if (++s == static_cast<uint32_t>(S)) {
            s = 0;
          }
        }
        if (look) s_fail = 1;
      }
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (slot[j] < 0) continue;
        uint64_t k;
        bool vv[kMaxVals];
        uint64_t vb[kMaxVals];
        pool_row<NV, MASK>(w[j], P.nvals, k, vv, vb);
        priv_apply<SPEC, NV>(T, A, slot[j], P.fkind, P.fcol, P.nfields, vv, vb);
      }
    }
    priv_fence();
    const bool failed = s_fail != 0;
    // Groups out, one reservation per CTA.
    const unsigned ng = s_groups;
    if (threadIdx.x == 0) {
      if (failed) {
        const unsigned long long fi = atomicAdd(B.counters + 1, 1ull);
        if (fi < np) B.failed[fi] = part;
      } else if (ng) {
        s_base = atomicAdd(B.counters + 0, static_cast<unsigned long long>(ng));
      }
    }
    __syncthreads();
    for (unsigned g = threadIdx.x; g < ng; g += blockDim.x) {
      const int s = used[g];
      const unsigned long long o = s_base + g;
      uint64_t* dst = !failed && o < B.tails_cap ? B.tails + o * W : nullptr;
      if (dst) dst[0] = keys[s];
      keys[s] = 0;
#pragma unroll 1
      for (int f = 0; f < P.nfields; ++f) {
        const bool none = (A.skip >> f) & 1u;
        if (dst) dst[1 + f] = none ? 0 : priv_load(T, A, f, P.fkind[f], s);
        if (!none) priv_clear(T, A, f, P.fkind[f], s);
      }
    }
    __syncthreads();
  }
}

// Adds pool rows to the global table: the rows of the failed partitions, or
// the listed pool rows (`list`, `nlist`). A row that finds no place is listed
// in P.spill_rows by its pool position.
template <int NV, uint32_t SPEC, bool MASK>
__global__ void __launch_bounds__(512) pool_insert_kernel(const __grid_constant__ AggK P, const PoolK Q,
                                                          const uint32_t* failed, uint32_t nfailed,
                                                          const uint32_t* list, uint64_t nlist) {
  constexpr int PW = pool_words<NV, MASK>();
  unsigned long long inserted = 0;
  auto add = [&](uint32_t at) {
    uint64_t w[PW], k, vb[kMaxVals];
    bool vv[kMaxVals];
    pool_load<PW>(Q.rows + static_cast<uint64_t>(at) * PW, w);
    pool_row<NV, MASK>(w, P.nvals, k, vv, vb);
    uint64_t* r = global_row1(P, true, k, key_hash1(k), inserted, P.probe_limit);
    if (r) global_apply<SPEC, NV>(r + 1, P.fkind, P.fcol, P.nfields, vv, vb);
    else spill_row(P, at);
  };
  if (list) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < nlist;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
      add(list[i]);
  } else {
    for (uint32_t i = blockIdx.x; i < nfailed; i += gridDim.x)
      for (uint32_t at = Q.off[failed[i]] + threadIdx.x; at < Q.off[failed[i] + 1]; at += blockDim.x) add(at);
  }
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if ((threadIdx.x & 31) == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}

// Merges spilled partial rows (single-key rows, or composite rows of the
// composite private tables) into the table.
template <int MODE>
__global__ void merge_parts_kernel(const AggK P, const uint64_t* __restrict__ parts, uint64_t n) {
  const int W = P.row_words;
  unsigned long long inserted = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t* src = parts + i * W;
    uint64_t* dst;
    int fo;
    if (MODE == 2) {
      uint64_t words[kMaxKeys];
      for (int j = 0; j < P.nkeys; ++j) words[j] = src[2 + j];
      dst = global_rowN(P, words, src[1], row_hashN(P, words, src[1]), inserted);
      fo = 2 + P.nkeys;
    } else {
      const uint64_t k = src[0];
      // The caller sized the table for these rows: probe as far as it takes.
      dst = global_row1(P, true, k, key_hash1(k), inserted, static_cast<int>(P.cap < (1ull << 30) ? P.cap : (1ull << 30)));
      fo = 1;
    }
    if (!dst) {
      atomicOr(P.err, kDevSpillOverflow);
      continue;
    }
    merge_fields(dst + fo, src + fo, P);
  }
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if ((threadIdx.x & 31) == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}

// Writes one output value of result type `t` from a 64-bit word.
__device__ __forceinline__ void store_typed(void* base, uint64_t i, int32_t t, uint64_t w) {
  switch (t) {
    case kI32:
    case kSTR: static_cast<int32_t*>(base)[i] = static_cast<int32_t>(static_cast<uint32_t>(w)); break;
    case kBOOL: static_cast<uint8_t*>(base)[i] = static_cast<uint8_t>(w & 1ull); break;
    default: static_cast<uint64_t*>(base)[i] = w; break;
  }
}

// Compacts occupied rows into dense output columns (keys, then aggregates),
// applying the reference's finalisation (ops/agg_internal.h:169-229).
template <int MODE>
__global__ void __launch_bounds__(1024) finalize_kernel(const AggK P, const FinK F) {
  const int W = P.row_words;
  const int fo = (MODE == 2) ? 2 + P.nkeys : 1;
  const uint64_t total = (MODE == 0) ? 1 : (MODE == 1 ? P.cap + 2 : P.cap);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // Output positions: one atomic per CTA and pass (the warps' counts are
  // prefixed in shared memory), not one per warp -- a sparse table of tens of
  // millions of slots would otherwise serialise on the counter.
  __shared__ unsigned int wpos[32];
  __shared__ unsigned int s_rows;
  __shared__ unsigned long long s_first;
  // kFinPer slots per thread and pass: fewer passes, so fewer barriers.
  constexpr int kFinPer = 4;
  // The occupied slots of a pass, side by side, so that the rows are finalised
  // by full warps: slot by slot, the half-empty warps of a half-full table took
  // twice the instructions, FP64 divisions above all (minute bars of 50M
  // trades, 3.9M groups: 3.20 ms the call, 3.11 now).
  __shared__ uint16_t list[1024 * kFinPer];
  const uint64_t span = static_cast<uint64_t>(blockDim.x) * kFinPer;
  for (uint64_t base = blockIdx.x * span; base < total; base += gridDim.x * span) {
    bool occk[kFinPer];
    unsigned mk[kFinPer];
    unsigned cnt = 0;
#pragma unroll
    for (int k = 0; k < kFinPer; ++k) {
      const uint64_t sk = base + static_cast<uint64_t>(k) * blockDim.x + threadIdx.x;
      bool o = false;
      if (sk < total) {
        const uint64_t* rk = P.table + sk * W;
        if (MODE == 0) o = true;
        else if (MODE == 1) o = (sk < P.cap) ? (rk[0] != 0) : (rk[1] != 0);
        else o = rk[0] >= 2;
        if (MODE == 1 && o && F.merge_table && sk < P.cap) {
          // The key also has a row in the second table: merge into it there.
          uint64_t* m = find_row1(F.merge_table, F.merge_cap, W, rk[0]);
          if (m) {
            merge_fields(m + 1, rk + 1, P);
            o = false;
          }
        }
      }
      occk[k] = o;
      mk[k] = __ballot_sync(0xffffffffu, o);
      cnt += __popc(mk[k]);
    }
    if (lane == 0) wpos[warp] = cnt;
    __syncthreads();
    if (warp == 0) {
      const unsigned c = lane < nwarps ? wpos[lane] : 0;
      unsigned incl = c;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      wpos[lane] = incl - c;
      if (lane == 31) {
        s_rows = incl;
        s_first = incl ? atomicAdd(F.out_count, static_cast<unsigned long long>(incl)) : 0;
      }
    }
    __syncthreads();
    unsigned at = wpos[warp];
#pragma unroll
    for (int k = 0; k < kFinPer; ++k) {
      if (occk[k])
        list[at + __popc(mk[k] & ((1u << lane) - 1u))] = static_cast<uint16_t>(k * blockDim.x + threadIdx.x);
      at += __popc(mk[k]);
    }
    const unsigned nrows = s_rows;
    const unsigned long long first = s_first;
    __syncthreads();  // (wpos, s_rows and s_first are rewritten after the next pass's first barrier)
    for (unsigned i = threadIdx.x; i < nrows; i += blockDim.x) {
      const uint64_t s = base + list[i];
      const uint64_t* r = P.table + s * W;
      const uint64_t o = first + i;
      if (o >= F.out_cap) {
        atomicOr(P.err, kDevSpillOverflow);
        continue;
      }
      // keys
      for (int j = 0; j < P.nkeys; ++j) {
        bool isnull;
        uint64_t w;
        if (MODE == 1) {
          isnull = (s == P.cap + 1);
          w = (s == P.cap) ? 0 : r[0];
          if (F.packed_pair) {  // two 4-byte keys packed in one word
            isnull = false;
            w = j == 0 ? w >> 32 : w & 0xffffffffull;
          } else if (F.packed_width > 0) {  // (partition key, bucket index) packed in one word
            isnull = false;
            w = j == 0 ? static_cast<uint64_t>(static_cast<int64_t>(static_cast<int32_t>(static_cast<uint32_t>(w >> 32))))
                       : static_cast<uint64_t>(static_cast<int64_t>(static_cast<int32_t>(static_cast<uint32_t>(w))) *
                                               F.packed_width);
          }
        } else {
          isnull = (r[1] >> j) & 1ull;
          w = r[2 + j];
        }
        F.valid[j][o] = isnull ? 0 : 1;
        store_typed(F.vals[j], o, F.rtype[j], isnull ? 0 : w);
      }
      // aggregates
      const uint64_t* f = r + fo;
      const uint64_t rows = f[0];
      for (int a = 0; a < F.naggs; ++a) {
        const int oc = P.nkeys + a;
        const int vf = F.vfield[a];
        const uint64_t nulls = F.nfield[a] >= 0 ? f[F.nfield[a]] : 0;
        const uint64_t nn = rows - nulls;
        const int32_t rt = F.rtype[oc];
        uint8_t ok = 1;
        uint64_t w = 0;
        switch (F.func[a]) {
          case 0: w = rows; break;  // COUNT(*)
          case 1: w = nn; break;    // COUNT(col)
          case 2:                   // SUM
            if (nn == 0) ok = 0;
            else w = f[vf];
            break;
          case 5: {  // AVG = sum / non-null count, in double (ops/agg_internal.h:217-227)
            if (nn == 0) {
              ok = 0;
            } else {
              const double sum = (P.fkind[vf] == F_SUMF) ? __longlong_as_double(static_cast<long long>(f[vf]))
                                                          : static_cast<double>(static_cast<int64_t>(f[vf]));
              w = static_cast<uint64_t>(__double_as_longlong(sum / static_cast<double>(nn)));
            }
            break;
          }
          default: {  // MIN / MAX
            if (nn == 0) {
              ok = 0;
              break;
            }
            const uint8_t fk = P.fkind[vf];
            const uint64_t e = f[vf];
            if (fk == F_MINF) w = dec_f64_bits(~e);
            else if (fk == F_MAXF) w = dec_f64_bits(e);
            else if (fk == F_MINI) w = static_cast<uint64_t>(dec_i64(~e));
            else w = static_cast<uint64_t>(dec_i64(e));
            break;
          }
        }
        F.valid[oc][o] = ok;
        store_typed(F.vals[oc], o, rt, ok ? w : 0);
      }
    }
  }
}

int32_t agg_result_type(int32_t func, int32_t in) {
  switch (func) {
    case QEG_COUNT_STAR:
    case QEG_COUNT: return QEG_I64;
    case QEG_SUM: return in == QEG_F64 ? QEG_F64 : QEG_I64;
    case QEG_AVG: return QEG_F64;
    default: return in;
  }
}

uint64_t next_pow2(uint64_t v) {
  uint64_t c = 1;
  while (c < v) c <<= 1;
  return c;
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

void AggState::plan(const int32_t* col_types, int ncols, const uint32_t* key_cols, int nk,
                    const qeg_agg_spec* aggs_in, int na) {
  require(ncols > 0 && col_types != nullptr, "aggregate needs an input schema");
  require(na >= 1 && aggs_in != nullptr, "Aggregate needs >=1 aggregate");
  require(nk >= 0 && nk <= kMaxKeys, "GPU aggregate supports 0..8 key columns");
  require(na <= kMaxAggs, "GPU aggregate supports at most 32 aggregates");
  types.assign(col_types, col_types + ncols);
  for (int32_t t : types) require(t >= QEG_I32 && t <= QEG_STR, "unknown column type");
  keys.assign(key_cols, key_cols + nk);
  for (uint32_t k : keys) require(k < static_cast<uint32_t>(ncols), "key column index out of range");
  aggs.assign(aggs_in, aggs_in + na);
  mode = nk == 0 ? 0 : (nk == 1 ? 1 : 2);

  // Distinct value columns and their fields, grouped by column.
  val_cols.clear();
  fkind.assign(1, F_ROWS);
  std::vector<std::vector<uint8_t>> per_col;
  vfield.assign(na, -1);
  nfield.assign(na, -1);
  rtypes.clear();
  for (uint32_t k : keys) rtypes.push_back(types[k]);
  struct Want { int col; uint8_t kind; };
  std::vector<Want> wants;
  for (int a = 0; a < na; ++a) {
    const qeg_agg_spec& s = aggs[a];
    require(s.func >= QEG_COUNT_STAR && s.func <= QEG_AVG, "unknown aggregate function");
    if (s.func == QEG_COUNT_STAR) {
      rtypes.push_back(QEG_I64);
      continue;
    }
    require(s.input_col < static_cast<uint32_t>(ncols), "aggregate input column out of range");
    const int32_t in = types[s.input_col];
    if (in == QEG_STR && (s.func == QEG_SUM || s.func == QEG_AVG))
      require(false, s.func == QEG_SUM ? "SUM is not defined on STR (VARCHAR)"
                                       : "AVG is not defined on STR (VARCHAR)");
    rtypes.push_back(agg_result_type(s.func, in));
  }
  // Assign fields per distinct column.
  std::vector<int> colslot(ncols, -1);
  for (int a = 0; a < na; ++a) {
    const qeg_agg_spec& s = aggs[a];
    if (s.func == QEG_COUNT_STAR) continue;
    if (colslot[s.input_col] < 0) {
      require(static_cast<int>(val_cols.size()) < kMaxVals, "GPU aggregate supports at most 8 input columns");
      colslot[s.input_col] = static_cast<int>(val_cols.size());
      val_cols.push_back(s.input_col);
      per_col.emplace_back();
    }
    const int vc = colslot[s.input_col];
    const bool isf = types[s.input_col] == QEG_F64;
    uint8_t kind = F_NULLS;
    if (s.func == QEG_SUM || s.func == QEG_AVG) kind = isf ? F_SUMF : F_SUMI;
    if (s.func == QEG_MIN) kind = isf ? F_MINF : F_MINI;
    if (s.func == QEG_MAX) kind = isf ? F_MAXF : F_MAXI;
    auto& v = per_col[vc];
    if (std::find(v.begin(), v.end(), F_NULLS) == v.end()) v.insert(v.begin(), F_NULLS);
    if (kind != F_NULLS && std::find(v.begin(), v.end(), kind) == v.end()) v.push_back(kind);
  }
  // Fields of a column in kind order (NULLS, sums, MINs, MAXes) whatever the
  // order of the aggregates, so equal field sets share a specialised kernel.
  for (auto& v : per_col) std::sort(v.begin(), v.end());
  cfirst.assign(val_cols.size(), 0);
  cnf.assign(val_cols.size(), 0);
  for (size_t c = 0; c < val_cols.size(); ++c) {
    cfirst[c] = static_cast<int>(fkind.size());
    cnf[c] = static_cast<int>(per_col[c].size());
    for (uint8_t k : per_col[c]) fkind.push_back(k);
  }
  require(static_cast<int>(fkind.size()) <= kMaxFields, "too many aggregate state fields for the GPU path");
  for (int a = 0; a < na; ++a) {
    const qeg_agg_spec& s = aggs[a];
    if (s.func == QEG_COUNT_STAR) continue;
    const int vc = colslot[s.input_col];
    const bool isf = types[s.input_col] == QEG_F64;
    uint8_t kind = F_NULLS;
    if (s.func == QEG_SUM || s.func == QEG_AVG) kind = isf ? F_SUMF : F_SUMI;
    if (s.func == QEG_MIN) kind = isf ? F_MINF : F_MINI;
    if (s.func == QEG_MAX) kind = isf ? F_MAXF : F_MAXI;
    for (int k = 0; k < cnf[vc]; ++k) {
      if (fkind[cfirst[vc] + k] == F_NULLS) nfield[a] = cfirst[vc] + k;
      if (fkind[cfirst[vc] + k] == kind) vfield[a] = cfirst[vc] + k;
    }
  }
  nfields = static_cast<int>(fkind.size());
  row_words = (mode == 2 ? 2 + nk : 1) + nfields;
  // Two keys of at most 4 bytes fit one key word: such a GROUP BY runs as a
  // single-key one (private tables, sketch) while no batch has NULLs in
  // either column. 20M rows over 21k (I32, I32) groups took 7.1 ms through the
  // composite table, whose hot rows every warp updates with global
  // reductions. A strategy asked for by name keeps the composite table.
  auto small_key = [&](int j) {
    const int32_t t = types[keys[j]];
    return t == QEG_I32 || t == QEG_BOOL || t == QEG_STR;
  };
  packable = nk == 2 && cfg.strategy == QEG_AGG_AUTO && small_key(0) && small_key(1);
}

DevCol AggState::key_col(const std::vector<StagedCol>& staged, size_t j) const {
  DevCol c = staged[keys[j]].dev;
  c.bucket = (bucket_width > 0 && j + 1 == keys.size()) ? bucket_width : 0;
  if (packed && j == 0) {
    c.type1 = c.type;
    c.type = bucket_width > 0 ? kPackedKey : kPackedPair;
    c.all_valid = 1;
    c.validity = nullptr;
    c.data2 = staged[keys[1]].dev.data;
    c.code_map2 = staged[keys[1]].dev.code_map;
    c.type2 = staged[keys[1]].dev.type;
    c.bucket = bucket_width;
  }
  return c;
}

namespace {
// Smallest and largest value of an integer column without NULLs, as
// order-preserving encodings: out[0] = min, out[1] = max. Reads 32 bytes per
// access from the first aligned one on (one value per thread and step took 180
// us for 50M 8-byte times).
template <class T>
__global__ void __launch_bounds__(256) int_range_kernel(const T* __restrict__ v, uint64_t n, uint64_t head,
                                                        unsigned long long* out) {
  using V = Vec32<T>;
  const uint64_t at = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  const uint64_t step = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const uint64_t nv = (n - head) / V::kN;
  T lo = v[0], hi = v[0];
  for (uint64_t i = at; i < nv; i += 2 * step) {
    V a, b;
    const bool two = i + step < nv;
    a.load(v + head + i * V::kN);
    if (two) b.load(v + head + (i + step) * V::kN);
#pragma unroll
    for (int e = 0; e < V::kN; ++e) {
      const T x = a.at(e), y = two ? b.at(e) : x;
      lo = min(lo, min(x, y));
      hi = max(hi, max(x, y));
    }
  }
  for (uint64_t i = at; i < head + (n - head) % V::kN; i += step) {  // before and behind the aligned part
    const T x = v[i < head ? i : i + nv * V::kN];
    lo = min(lo, x);
    hi = max(hi, x);
  }
  int64_t mn = lo, mx = hi;
  for (int o = 16; o > 0; o >>= 1) {
    mn = min(mn, __shfl_down_sync(0xffffffffu, mn, o));
    mx = max(mx, __shfl_down_sync(0xffffffffu, mx, o));
  }
  __shared__ int64_t smn[8], smx[8];
  if ((threadIdx.x & 31) == 0) {
    smn[threadIdx.x >> 5] = mn;
    smx[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      mn = min(mn, smn[w]);
      mx = max(mx, smx[w]);
    }
    atomicMin(out + 0, static_cast<unsigned long long>(enc_i64(mn)));
    atomicMax(out + 1, static_cast<unsigned long long>(enc_i64(mx)));
  }
}

template <class T>
void launch_range(qeg_ctx* ctx, const void* data, uint64_t n, unsigned long long* out) {
  const uint64_t off = reinterpret_cast<uintptr_t>(data) % 32;
  const uint64_t head = std::min<uint64_t>(n, off ? (32 - off) / sizeof(T) : 0);
  int_range_kernel<T><<<grid_for(ctx, n, 256, 8), 256, 0, ctx->stream>>>(static_cast<const T*>(data), n, head, out);
  ctx->launches++;
}

void column_range(qeg_ctx* ctx, const DevCol& c, uint64_t n, unsigned long long* out) {
  if (c.type == kI32) launch_range<int32_t>(ctx, c.data, n, out);
  else launch_range<int64_t>(ctx, c.data, n, out);
}

// Packed rows -> composite rows: every occupied single-key row (and the key-0
// side row) is decoded into (partition key, bucket start) key words, or into
// its two 4-byte keys (width 0), and inserted into the new composite table with its fields.
__global__ void unpack_kernel(const AggK P, const uint64_t* __restrict__ old, uint64_t old_cap, int old_w,
                              int64_t width, int32_t key_type, int32_t time_type) {
  unsigned long long inserted = 0;
  const int fo = 2 + P.nkeys;
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < old_cap + 2;
       s += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t* src = old + s * old_w;
    uint64_t k;
    if (s < old_cap) {
      k = src[0];
      if (k == 0) continue;
    } else {
      if (src[1] == 0) continue;  // side rows: occupied when their row count is not zero
      if (s == old_cap + 1) {     // a NULL key cannot be packed
        atomicOr(P.err, kDevBadInput);
        continue;
      }
      k = 0;
    }
    uint64_t words[kMaxKeys] = {};
    if (width == 0) {  // two 4-byte keys
      words[0] = k >> 32;
      words[1] = k & 0xffffffffull;
      uint64_t* dst = global_rowN(P, words, 0, row_hashN(P, words, 0), inserted);
      if (!dst) {
        atomicOr(P.err, kDevSpillOverflow);
        continue;
      }
      for (int f = 0; f < P.nfields; ++f) dst[fo + f] = src[1 + f];
      continue;
    }
    const int32_t a = static_cast<int32_t>(static_cast<uint32_t>(k >> 32));
    words[0] = key_type == kI32 ? static_cast<uint64_t>(static_cast<uint32_t>(a))
                                : static_cast<uint64_t>(static_cast<int64_t>(a));
    const int64_t b = static_cast<int64_t>(static_cast<int32_t>(static_cast<uint32_t>(k))) * width;
    words[1] = time_type == kI32 ? static_cast<uint64_t>(static_cast<uint32_t>(static_cast<int32_t>(b)))
                                 : static_cast<uint64_t>(b);
    uint64_t* dst = global_rowN(P, words, 0, row_hashN(P, words, 0), inserted);
    if (!dst) {
      atomicOr(P.err, kDevSpillOverflow);
      continue;
    }
    for (int f = 0; f < P.nfields; ++f) dst[fo + f] = src[1 + f];
  }
  for (int o = 16; o > 0; o >>= 1) inserted += __shfl_down_sync(0xffffffffu, inserted, o);
  if ((threadIdx.x & 31) == 0 && inserted) atomicAdd(P.counters + 2, inserted);
}
}  // namespace

// The batch can keep (or start) the packed key: both key columns without
// NULLs, the key's values (an I64/TS key) and every bucket index of the time
// column within int32.
bool AggState::can_pack(const std::vector<StagedCol>& staged, uint64_t len) {
  if (!packable || staged.empty()) return false;
  const DevCol& a = staged[keys[0]].dev;
  const DevCol& t = staged[keys[1]].dev;
  if (!a.all_valid || !t.all_valid) return false;
  if (len == 0 || bucket_width == 0) return true;  // a pair of 4-byte keys always fits
  const bool wide_key = a.type != kI32;
  DevBuf mm(32, ctx->stream);
  const unsigned long long init[4] = {~0ull, 0ull, ~0ull, 0ull};
  QEG_CUDA(cudaMemcpyAsync(mm.get(), init, 32, cudaMemcpyHostToDevice, ctx->stream));
  column_range(ctx, t, len, mm.get<unsigned long long>());
  if (wide_key) column_range(ctx, a, len, mm.get<unsigned long long>() + 2);
  QEG_CUDA(cudaGetLastError());
  unsigned long long r[4];
  QEG_CUDA(cudaMemcpyAsync(r, mm.get(), 32, cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  if (wide_key && (dec_i64(r[2]) < INT32_MIN || dec_i64(r[3]) > INT32_MAX)) return false;
  const int64_t qmin = dec_i64(r[0]) / bucket_width, qmax = dec_i64(r[1]) / bucket_width;
  if (!table.get()) {
    pack_qmin = qmin;
    pack_qmax = qmax;
  }
  return qmin >= INT32_MIN && qmax <= INT32_MAX;
}

// Converts the packed single-key table into composite rows, after which the
// window or GROUP BY runs as an ordinary composite-key one. A single-key table
// fills to 0.85 before it grows, where runs of taken slots pass the probe limit
// even in small tables: the composite one is at most half full, and its rows
// are placed however far the search takes (as a grown table's are).
// The tail rows of a partitioned batch are single-key rows too: they join the
// table first.
void AggState::unpack() {
  merge_tails();
  tails.release();
  tails_cap = 0;
  pool.release();
  DevBuf old;
  old.swap(table);
  const uint64_t old_cap = cap;
  const int old_w = row_words;
  packed = false;
  mode = 2;
  row_words = 2 + static_cast<int>(keys.size()) + nfields;
  strategy = QEG_AGG_GLOBAL;
  smem_slots = 0;
  nhot = 0;
  alloc_table(std::max(old_cap, next_pow2(2 * (inserted + 1))));
  part_cap = static_cast<uint64_t>(ctx->sms) * 32 * 2 + 64;
  spill_parts.alloc(part_cap * row_words * 8, ctx->stream);
  QEG_CUDA(cudaMemsetAsync(counters.get<uint8_t>() + 16, 0, 8, ctx->stream));
  AggK P = kparams_base();
  P.probe_limit = static_cast<int>(std::min<uint64_t>(cap, 1u << 30));
  const unsigned g = grid_for(ctx, old_cap + 2, 256, 8);
  unpack_kernel<<<g, 256, 0, ctx->stream>>>(P, old.get<uint64_t>(), old_cap, old_w, bucket_width, types[keys[0]],
                                            types[keys[1]]);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
  uint64_t c[3];
  read_counters(c);
  check_device_error(ctx);
  inserted = c[2];
}

AggK AggState::kparams(const std::vector<StagedCol>& staged, const uint32_t* sel, uint64_t nrows,
                       uint64_t len) const {
  AggK P{};
  P.nkeys = static_cast<int>(keys.size());
  for (size_t j = 0; j < keys.size(); ++j) P.key[j] = key_col(staged, j);
  P.nvals = static_cast<int>(val_cols.size());
  for (size_t c = 0; c < val_cols.size(); ++c) P.val[c] = staged[val_cols[c]].dev;
  P.nfields = nfields;
  for (int f = 0; f < nfields; ++f) P.fkind[f] = fkind[f];
  set_field_columns(P);
  P.row_words = row_words;
  P.table = table.get<uint64_t>();
  P.cap = cap;
  P.sel = sel;
  P.nrows = nrows;
  P.len = len;
  P.smem_slots = smem_slots;  // (composite private tables)
  P.smem_insert = smem_insert;
  P.hot = hot_keys_dev.get<uint64_t>();
  P.nhot = nhot;
  P.probe_limit = probe_limit;
  P.spill_rows = spill_rows.get<uint32_t>();
  P.spill_cap = spill_cap;
  P.spill_parts = spill_parts.get<uint64_t>();
  P.part_cap = part_cap;
  P.counters = counters.get<unsigned long long>();
  if (mode == 1) {
    // Raise the table-full signal at 85% occupancy (counting the keys already in).
    const uint64_t at = static_cast<uint64_t>(0.85 * static_cast<double>(cap));
    P.full_flag = reinterpret_cast<uint32_t*>(P.counters + 4);
    P.full_at = at > inserted ? at - inserted : 1;
  }
  P.err = static_cast<uint32_t*>(ctx->dev_err.get());
  return P;
}

uint32_t AggState::field_spec(const AggK& P) const {
  // The launch's field set, NULL counts of columns without NULLs skipped.
  const int n = nfields - 1;
  if (n > 7) return kGenericSpec;
  uint32_t spec = static_cast<uint32_t>(n), counted = spec;
  for (int i = 1; i <= n; ++i) {
    const int col = P.fcol[i];
    if (col > 1) return kGenericSpec;
    const int kind = fkind[i];
    counted |= spec_field(i, kind, col);
    spec |= spec_field(i, kind == F_NULLS && P.val[col].all_valid ? 0 : kind, col);
  }
  // NULLs in one of two columns only: the field set that counts both.
  if (spec != counted && (counted == kSpecIntF64Nulls || counted == kSpecIntSumF64StatsNulls) &&
      spec != kSpecIntF64 && spec != kSpecIntSumF64Stats)
    return counted;
  return spec;
}

void AggState::set_field_columns(AggK& P) const {
  for (size_t c = 0; c < cfirst.size(); ++c)
    for (int k = 0; k < cnf[c]; ++k) P.fcol[cfirst[c] + k] = static_cast<uint8_t>(c);
}

// 1024-thread CTAs for the single-key private-table strategy (64M Zipf(1.1) rows
// over 100k keys, the largest tables: 1.72 ms, 2.82 with 512 threads; 1024
// slots: 1.68 and 1.71), 512 otherwise.
int AggState::block_threads() const {
  if (cfg.block_threads > 0) return cfg.block_threads;
  return (mode == 1 && (strategy == QEG_AGG_SMEM || strategy == QEG_AGG_PARTITIONED)) ? 1024 : 512;
}

void AggState::alloc_table(uint64_t new_cap) {
  cap = std::max<uint64_t>(new_cap, 1024);
  const uint64_t rows = (mode == 1) ? cap + 2 : (mode == 0 ? 1 : cap);
  table.alloc(rows * row_words * 8, ctx->stream);
  QEG_CUDA(cudaMemsetAsync(table.get(), 0, rows * row_words * 8, ctx->stream));
}

size_t AggState::smem_bytes(int block) const {
  return mode == 0 ? (1 + static_cast<size_t>(block / 32)) * (row_words | 1) * 8 : 0;
}

// Bit of column c's NULL count among the fields (0 when it has none).
uint32_t AggState::null_field(int c) const {
  return cnf[c] > 0 && fkind[cfirst[c]] == F_NULLS ? 1u << cfirst[c] : 0;
}

// Most slots of a private table (a power of two, at most 8192) that shared
// memory holds beside the kernel's static variables.
int AggState::priv_max_slots(uint32_t skip, bool ssum) const {
  int slots = 64;
  while (slots < 8192 &&
         priv_layout(fkind.data(), nfields, slots * 2, skip, kPrivReps, ssum).bytes + 1024 <= ctx->smem_optin)
    slots *= 2;
  return slots;
}

// Single key, private tables: 1024 threads per SM. The table has as many slots
// as the launch gives each CTA rows, within [256, smem_slots]: clearing and
// flushing a table that no CTA can fill costs a small launch more than its
// rows.
void AggState::launch_private1(const AggK& P0, uint64_t nrows) {
  AggK P = P0;
  void (*kern)(AggK, PrivK) = nullptr;
  const int nv = static_cast<int>(val_cols.size());
  const uint32_t spec = field_spec(P);
  auto pick = [&](auto ssum) -> void (*)(AggK, PrivK) {
    constexpr bool kS = decltype(ssum)::value;
    if (spec == kSpecIntF64) return agg_private_kernel<2, kSpecIntF64, kS>;
    if (spec == kSpecIntF64Nulls) return agg_private_kernel<2, kSpecIntF64Nulls, kS>;
    if (spec == kSpecF64) return agg_private_kernel<1, kSpecF64, kS>;
    if (spec == kSpecF64Nulls) return agg_private_kernel<1, kSpecF64Nulls, kS>;
    if (spec == kSpecCount) return agg_private_kernel<1, kSpecCount>;
    if (spec == kSpecIntSumF64Stats) return agg_private_kernel<2, kSpecIntSumF64Stats, kS>;
    if (spec == kSpecIntSumF64StatsNulls) return agg_private_kernel<2, kSpecIntSumF64StatsNulls, kS>;
    if (nv <= 1) return agg_private_kernel<1, kGenericSpec, kS>;
    if (nv <= 2) return agg_private_kernel<2, kGenericSpec, kS>;
    if (nv <= 4) return agg_private_kernel<4, kGenericSpec, kS>;
    return agg_private_kernel<8, kGenericSpec, kS>;
  };
  // F64 sums in shared memory (qeg_privagg.cuh) when the estimate puts the
  // global table beyond half of L2, as for the partitioned passes. A window's
  // groups come and go, so its tables hold most rows whatever the estimate.
  // (512M Zipf(1.1) rows over 64M keys, 25M groups: 32.5 ms with the sums at L2,
  // 30.7 here; 64M rows over 50k pairs of keys the other way round, 3.0 and 6.5.)
  const bool ssum = bucket_width == 0 && P.nhot == 0 && spec != kSpecCount &&
                    std::find(fkind.begin(), fkind.end(), F_SUMF) != fkind.end() &&
                    est_groups / kTargetLoad * row_words * 8.0 >= static_cast<double>(kPartMinTableBytes);
  kern = ssum ? pick(std::true_type{}) : pick(std::false_type{});
  const int block = block_threads();
  uint32_t skip = 0;
  for (int c = 0; c < nv; ++c)
    if (P.val[c].all_valid) skip |= null_field(c);
  const int most = std::min(smem_slots, priv_max_slots(skip, ssum));
  // A few thousand rows per CTA at least, so the flush stays small. A CTA of
  // fewer than 1024 threads shares its SM with others as far as their tables
  // (and the partial-row list) allow: 64M Zipf(1.1) rows over 100k keys, 1024
  // slots, 256 threads 4.6 ms with one CTA per SM, 1.8 now.
  const size_t full = priv_layout(fkind.data(), nfields, most, skip, kPrivReps, ssum).bytes;
  const uint64_t per_sm = std::max<uint64_t>(
      1, std::min<uint64_t>({static_cast<uint64_t>(1024 / block),
                             static_cast<uint64_t>(blocks_per_sm(reinterpret_cast<const void*>(kern), block, full)),
                             part_cap / (static_cast<uint64_t>(ctx->sms) * (most + 2))}));
  const uint64_t grid = std::max<uint64_t>(
      1, std::min<uint64_t>((nrows + 4095) / 4096, static_cast<uint64_t>(ctx->sms) * per_sm));
  int slots = 256;
  while (slots < most && static_cast<uint64_t>(slots) * grid < nrows) slots *= 2;
  if (P.nhot > 0) slots = smem_slots;  // preloaded
  slots = std::min(slots, most);
  PrivK A = priv_layout(fkind.data(), nfields, slots, skip, kPrivReps, ssum);
  priv_sums_for(A, grid);
  require(blocks_per_sm(reinterpret_cast<const void*>(kern), block, A.bytes) > 0,
          "aggregate kernel does not fit on an SM with this configuration");
  kern<<<(unsigned)grid, block, A.bytes, ctx->stream>>>(P, A);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
}

void AggState::launch_private(const AggK& P, uint64_t nrows) {
  void (*kern)(AggK) = nullptr;
  const int nv = static_cast<int>(val_cols.size());
  const uint32_t spec = field_spec(P);
  if (spec == kSpecIntF64) kern = agg2_private_kernel<2, kSpecIntF64>;
  else if (spec == kSpecIntF64Nulls) kern = agg2_private_kernel<2, kSpecIntF64Nulls>;
  else if (spec == kSpecF64) kern = agg2_private_kernel<1, kSpecF64>;
  else if (spec == kSpecF64Nulls) kern = agg2_private_kernel<1, kSpecF64Nulls>;
  else if (spec == kSpecCount) kern = agg2_private_kernel<1, kSpecCount>;
  else if (spec == kSpecIntSumF64Stats) kern = agg2_private_kernel<2, kSpecIntSumF64Stats>;
  else if (spec == kSpecIntSumF64StatsNulls) kern = agg2_private_kernel<2, kSpecIntSumF64StatsNulls>;
  else if (nv <= 1) kern = agg2_private_kernel<1, kGenericSpec>;
  else if (nv <= 2) kern = agg2_private_kernel<2, kGenericSpec>;
  else if (nv <= 4) kern = agg2_private_kernel<4, kGenericSpec>;
  else kern = agg2_private_kernel<8, kGenericSpec>;
  const int block = 512;
  const size_t sb = static_cast<size_t>(smem_slots) * (row_words | 1) * 8;
  const int per_sm = blocks_per_sm(reinterpret_cast<const void*>(kern), block, sb);
  require(per_sm > 0, "aggregate kernel does not fit on an SM with this configuration");
  // Each CTA walks one contiguous range; a few thousand rows at least.
  uint64_t grid = std::min<uint64_t>((nrows + 4095) / 4096, static_cast<uint64_t>(ctx->sms) * per_sm);
  if (grid == 0) grid = 1;
  kern<<<(unsigned)grid, block, sb, ctx->stream>>>(P);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
}

void AggState::launch(const AggK& P, uint64_t nrows) {
  if (mode == 2 && strategy == QEG_AGG_SMEM) {
    launch_private(P, nrows);
    return;
  }
  if (mode == 1)  // running insert count and table-full flag
    QEG_CUDA(cudaMemsetAsync(counters.get<uint8_t>() + 24, 0, 16, ctx->stream));
  if (mode == 1 && smem_slots > 0) {
    launch_private1(P, nrows);
    return;
  }
  const int block = block_threads();
  const size_t sb = smem_bytes(block);
  // Kernel variant: the mode and the number of value columns rounded up to 1,
  // 2, 4 or 8 (loops over value columns are unrolled to that count).
  void (*kern)(AggK) = nullptr;
  const int nv = static_cast<int>(val_cols.size());
#define QEG_AGG_VARIANT(M)                                       \
  (nv <= 1   ? agg_kernel<M, 1, kGenericSpec>                     \
   : nv <= 2 ? agg_kernel<M, 2, kGenericSpec>                     \
   : nv <= 4 ? agg_kernel<M, 4, kGenericSpec>                     \
             : agg_kernel<M, 8, kGenericSpec>)
#define QEG_AGG_SPEC(M)                                                       \
  (spec == kSpecIntF64        ? agg_kernel<M, 2, kSpecIntF64>                 \
   : spec == kSpecIntF64Nulls ? agg_kernel<M, 2, kSpecIntF64Nulls>            \
   : spec == kSpecF64         ? agg_kernel<M, 1, kSpecF64>                    \
   : spec == kSpecF64Nulls    ? agg_kernel<M, 1, kSpecF64Nulls>               \
   : spec == kSpecCount       ? agg_kernel<M, 1, kSpecCount>                  \
   : spec == kSpecIntSumF64Stats ? agg_kernel<M, 2, kSpecIntSumF64Stats>      \
   : spec == kSpecIntSumF64StatsNulls ? agg_kernel<M, 2, kSpecIntSumF64StatsNulls> \
                              : nullptr)
  const uint32_t spec = field_spec(P);
  if (mode == 0) kern = QEG_AGG_SPEC(0);
  else if (mode == 1) kern = QEG_AGG_SPEC(1);
  else kern = QEG_AGG_SPEC(2);
  if (kern == nullptr) {
    if (mode == 0) kern = QEG_AGG_VARIANT(0);
    else if (mode == 1) kern = QEG_AGG_VARIANT(1);
    else kern = QEG_AGG_VARIANT(2);
  }
#undef QEG_AGG_SPEC
#undef QEG_AGG_VARIANT
  const int per_sm = blocks_per_sm(reinterpret_cast<const void*>(kern), block, sb);
  require(per_sm > 0, "aggregate kernel does not fit on an SM with this configuration");
  // Each CTA should aggregate a few thousand rows at least, so clearing and
  // flushing its private table (which touches occupied rows only) stays small.
  const uint64_t min_rows_per_cta = 4096;
  uint64_t want = (nrows + min_rows_per_cta - 1) / min_rows_per_cta;
  uint64_t grid = std::min<uint64_t>(want, static_cast<uint64_t>(ctx->sms) * per_sm);
  if (grid == 0) grid = 1;
  kern<<<(unsigned)grid, block, sb, ctx->stream>>>(P);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
}

void AggState::read_counters(uint64_t out[3]) {
  QEG_CUDA(cudaMemcpyAsync(out, counters.get(), 24, cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
}

void AggState::grow(uint64_t new_cap) {
  DevBuf old;
  old.swap(table);
  const uint64_t old_cap = cap;
  alloc_table(new_cap);
  QEG_CUDA(cudaMemsetAsync(counters.get<uint8_t>() + 16, 0, 8, ctx->stream));
  std::vector<StagedCol> none;
  AggK P = kparams_base();
  const uint64_t n = (mode == 1) ? old_cap + 2 : old_cap;
  const unsigned g = grid_for(ctx, n, 256, 8);
  if (mode == 1) rehash_kernel<1><<<g, 256, 0, ctx->stream>>>(P, old.get<uint64_t>(), old_cap);
  else rehash_kernel<2><<<g, 256, 0, ctx->stream>>>(P, old.get<uint64_t>(), old_cap);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
  ++resizes;
}

AggK AggState::kparams_base() const {
  std::vector<StagedCol> dummy;
  AggK P{};
  P.nkeys = static_cast<int>(keys.size());
  P.nvals = static_cast<int>(val_cols.size());
  P.nfields = nfields;
  for (int f = 0; f < nfields; ++f) P.fkind[f] = fkind[f];
  set_field_columns(P);
  P.row_words = row_words;
  P.table = table.get<uint64_t>();
  P.cap = cap;
  P.probe_limit = probe_limit;
  P.counters = counters.get<unsigned long long>();
  P.err = static_cast<uint32_t*>(ctx->dev_err.get());
  return P;
}

void AggState::consume(const qeg_column* cols, int ncols, const uint32_t* sel, uint64_t sel_len) {
  require(!finished, "consume() after finish()");
  require(ncols == static_cast<int>(types.size()), "batch column count does not match the schema");
  require(cols != nullptr, "cols is NULL");
  const uint64_t len = cols[0].len;
  for (int c = 0; c < ncols; ++c) {
    require(cols[c].type == types[c], "batch column type does not match the schema");
    require(cols[c].len == len, "batch columns differ in length");
    require(cols[c].all_valid || cols[c].validity != nullptr,
            "column with all_valid=0 must carry a validity bitmap");
  }
  const uint64_t nrows = sel ? sel_len : len;
  require(len <= 0xffffffffull, "a batch holds at most 2^32-1 rows");
  std::vector<StagedCol> staged(ncols);
  for (uint32_t k : keys) stage_column(ctx, cols[k], staged[k]);
  for (uint32_t v : val_cols) stage_column(ctx, cols[v], staged[v]);
  DevBuf selbuf;
  const uint32_t* dsel = nullptr;
  stage_sel(ctx, sel, sel_len, selbuf, &dsel);
  if (!table.get()) first_consume(staged, nrows, len, dsel);
  else if (packed && !can_pack(staged, len)) unpack();
  if (nrows > spill_cap) {  // a later, larger batch: the spill list must hold all of it
    spill_cap = 0;
    spill_rows.alloc(nrows * 4, ctx->stream);
    spill_cap = nrows;
  }
  rows_seen += nrows;
  if (nrows == 0) return;
  fit_private(staged);

  if (strategy == QEG_AGG_PARTITIONED) {
    consume_partitioned(staged, nrows, len, dsel);
    return;
  }
  AggK P = kparams(staged, dsel, nrows, len);
  launch(P, nrows);
  settle(staged, len);
}

// After a pass: while rows were spilled (their key found no slot within the
// probe limit) or private-table rows could not be flushed, grow the global
// table and replay them.
void AggState::settle(const std::vector<StagedCol>& staged, uint64_t len) {
  uint64_t c[3];
  read_words_and_error(ctx, counters.get(), 3, c);  // one synchronisation
  inserted = c[2];
  uint64_t nspill = c[0], nparts = c[1];
  int rounds = 0;
  while (nspill > 0 || nparts > 0) {
    require(++rounds < 64, "aggregate table failed to converge after 64 resize rounds");
    // Copy the spill lists out of the way, grow the table, then replay.
    DevBuf rows_copy(std::max<uint64_t>(nspill, 1) * 4, ctx->stream), parts_copy(std::max<uint64_t>(nparts, 1) * row_words * 8, ctx->stream);
    if (nspill) QEG_CUDA(cudaMemcpyAsync(rows_copy.get(), spill_rows.get(), nspill * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    if (nparts) QEG_CUDA(cudaMemcpyAsync(parts_copy.get(), spill_parts.get(), nparts * row_words * 8, cudaMemcpyDeviceToDevice, ctx->stream));
    // Partial rows' keys are mostly among the spilled rows' too, so the larger
    // count is enough: with the sum of both, 16M rows of 3M groups announced as
    // 100k ended in 16.8M slots (6.9 ms), now in 8.4M (6.5).
    const uint64_t want = std::max<uint64_t>(cap * 2, next_pow2(2 * (inserted + std::max(nparts, nspill / 4))));
    grow(want);
    QEG_CUDA(cudaMemsetAsync(counters.get(), 0, 16, ctx->stream));
    if (nparts) {
      AggK Q = kparams_base();
      if (mode == 2)
        merge_parts_kernel<2><<<grid_for(ctx, nparts, 256, 8), 256, 0, ctx->stream>>>(Q, parts_copy.get<uint64_t>(),
                                                                                      nparts);
      else
        merge_parts_kernel<1><<<grid_for(ctx, nparts, 256, 8), 256, 0, ctx->stream>>>(Q, parts_copy.get<uint64_t>(),
                                                                                      nparts);
      ctx->launches++;
      QEG_CUDA(cudaGetLastError());
    }
    if (nspill) {
      AggK Q = kparams(staged, rows_copy.get<uint32_t>(), nspill, len);
      launch(Q, nspill);
    }
    read_words_and_error(ctx, counters.get(), 3, c);
    inserted = c[2];
    nspill = c[0];
    nparts = c[1];
  }
}

void AggState::first_consume(const std::vector<StagedCol>& staged, uint64_t nrows, uint64_t len,
                             const uint32_t* dsel) {
  // Two packable keys start packed when the batch allows. (Decided anew when an
  // earlier first batch was refused before there was a table.)
  if (packable) {
    packed = can_pack(staged, len);
    mode = packed ? 1 : 2;
    row_words = (packed ? 1 : 2 + static_cast<int>(keys.size())) + nfields;
  }
  // Sizing. QEG_SIZE_FIXED: the configured (or default) first capacity, grown on
  // overflow. QEG_SIZE_LEARNED: the estimator's group count (see qeg_estimate),
  // falling back to the row count bound when no estimate is available.
  uint64_t want;
  est_groups = 0;
  if (mode == 0) {
    want = 1;
  } else if (cfg.expected_groups > 0) {
    // The sketch still runs for its skew estimate (the private-table strategy
    // needs the heavy-hitter share) and, with hot_keys > 0, the heavy hitters.
    if (mode == 1 && (cfg.hot_keys > 0 || nrows >= kSketchMinRows)) estimate_groups(staged, nrows, len, dsel);
    want = static_cast<uint64_t>(static_cast<double>(cfg.expected_groups) / kTargetLoad) + 64;
    est_groups = static_cast<double>(cfg.expected_groups);
  } else if (cfg.sizing == QEG_SIZE_FIXED) {
    want = cfg.initial_capacity ? cfg.initial_capacity : (1ull << 20);
  } else if (nrows < kSketchMinRows) {
    // Too few rows for the sketch to pay for its round trip: the row count
    // bounds the group count, capped at the fixed default.
    want = std::min<uint64_t>(static_cast<uint64_t>(static_cast<double>(nrows) / kTargetLoad) + 64, 1ull << 20);
  } else {
    est_groups = estimate_groups(staged, nrows, len, dsel);
    // Head-room over the estimate keeps the probe short if it is low; an
    // estimate that is far too low is caught by overflow -> grow -> replay.
    want = static_cast<uint64_t>(std::max(kEstimateHeadroom * est_groups / kTargetLoad, 1024.0));
  }
  // Partitioned strategy: asked for, or chosen when the estimate puts the
  // global table far beyond L2, where every row that misses the private tables
  // costs its reductions on random lines: 512M Zipf(1.1) rows over 64M keys
  // take 14.1 ms partitioned and 30.7 ms through the private tables, 48M
  // uniform rows over 10M keys 3.3 ms and (global table alone) 8.2. Its global
  // table only takes the private tables' flushes, so it starts small.
  bool go_part = false;
  const double part_most = kPartMaxFill * part_table_slots(0) * static_cast<double>(1u << kPartMaxBits);
  if (mode == 1 && part_eligible(staged)) {
    // Asked for: partitioned unless the estimate exceeds what its 2^15
    // second-pass tables hold (every partition would overflow into the global
    // table one by one: 2.6 s for 512M rows over 64M uniform keys, against
    // 131 ms through the global table, which it then takes).
    if (cfg.strategy == QEG_AGG_PARTITIONED)
      go_part = !(est_groups > part_most);
    else if (cfg.strategy == QEG_AGG_AUTO && nrows >= kPartMinRows && est_groups > 0 &&
             est_groups / kTargetLoad * row_words * 8.0 >= static_cast<double>(kPartMinTableBytes) &&
             est_groups <= part_most)
      go_part = true;  // (more groups than 2^15 second-pass tables hold: the global table)
  }
  // Heavy hitters: asked for, or for a partitioned pass whose column has a
  // head worth a table of its own (each row's lookup costs more than it saves
  // below that).
  heavy_candidates.clear();
  if (mode == 1 && nrows > 0 && est_groups > 0 &&
      (cfg.hot_keys > 0 ? go_part || est_groups > 1024 : go_part && hot_share >= kPartMinHotShare))
    find_heavy(staged, nrows, len, dsel);
  if (go_part) want = next_pow2(2ull * ctx->sms * (2048 + 2));
  alloc_table(want);
  counters.alloc(64, ctx->stream);
  QEG_CUDA(cudaMemsetAsync(counters.get(), 0, 64, ctx->stream));
  // The spill list holds every row of a batch and the partial-row list every
  // private-table slot of every resident CTA, so neither can overflow.
  spill_cap = std::max<uint64_t>(1u << 16, nrows);
  spill_rows.alloc(spill_cap * 4, ctx->stream);

  // Strategy.
  strategy = go_part ? QEG_AGG_SMEM : (cfg.strategy == QEG_AGG_PARTITIONED ? QEG_AGG_AUTO : cfg.strategy);
  // Composite keys: CTA-private tables with periodic flushes when asked for,
  // the global table alone otherwise. (On the 200M-trade (sym, minute) window
  // the private tables measured slower, 39.3 vs 35.3 ms: the ~10k live groups
  // of a minute do not fit a CTA's table, while they do fit L2.)
  if (mode == 2) strategy = cfg.strategy == QEG_AGG_SMEM ? QEG_AGG_SMEM : QEG_AGG_GLOBAL;
  if (mode == 0) strategy = QEG_AGG_SMEM;
  // The largest private table that fits beside the kernel's static variables.
  uint32_t skip = 0;
  for (size_t c = 0; c < val_cols.size(); ++c)
    if (!staged.empty() && staged[val_cols[c]].dev.all_valid) skip |= null_field(static_cast<int>(c));
  const int slots = priv_max_slots(skip);
  if (strategy == QEG_AGG_AUTO) {
    // Private tables pay off when a CTA sees each key many times: few groups
    // (all fit), a heavy head of the key distribution, or keys clustered in
    // time (a window's buckets).
    strategy = (est_groups > 0 && est_groups > 128.0 * 1024 && hot_share < 0.3 && !(packed && bucket_width > 0))
                   ? QEG_AGG_GLOBAL
                   : QEG_AGG_SMEM;
  }
  nhot = 0;
  if (strategy == QEG_AGG_SMEM && mode == 1) {
    // First-come private tables as large as shared memory allows: on a heavy
    // head the hot keys arrive first and keep their slots. Preloading the
    // sketch's heavy hitters into a read-only table is an option
    // (hot_keys > 0).
    // The partitioned strategy preloads the heavy hitters (when the sketch
    // found any) into a read-only 4096-slot table: which rows reach the pool
    // must not depend on the order rows arrive in, so a sizing pass can count
    // them. (256M Zipf rows over 64M keys: 8.2 ms with 2048 slots, 7.7 with
    // 4096, about as many as fit beside two values' fields.)
    const bool preload = !heavy_candidates.empty() && (go_part || (cfg.hot_keys > 0 && est_groups > 1024));
    smem_slots = cfg.smem_slots > 0 ? static_cast<int>(next_pow2(cfg.smem_slots))
                                    : go_part ? (preload ? 4096 : 64)
                                              : (preload ? 1024 : slots);
    smem_slots = std::min(std::max(smem_slots, 64), slots);
    smem_insert = go_part ? 0 : 1;
    if (preload) {
      preload_hot();
      smem_insert = 0;
    }
  } else if (strategy == QEG_AGG_SMEM && mode == 2) {
    // Two 512-thread CTAs per SM, each with its table.
    const size_t row_bytes = static_cast<size_t>(row_words | 1) * 8;
    int fit = 1;
    while (static_cast<size_t>(fit) * 2 * row_bytes <= ctx->smem_optin / 2 - 2048) fit *= 2;
    smem_slots = cfg.smem_slots > 0 ? static_cast<int>(next_pow2(cfg.smem_slots)) : 1024;
    smem_slots = std::max(64, std::min(smem_slots, fit));
    smem_insert = 1;
  } else {
    smem_slots = 0;
  }
  // At most 2 private tables per SM (1024 threads in all, so more of smaller
  // CTAs, each with fewer slots); the composite tables run more CTAs.
  const int tables = mode == 1 ? std::max(2, std::min(1024 / block_threads(), 16384 / (smem_slots + 2))) : 32;
  part_cap = static_cast<uint64_t>(ctx->sms) * tables * (smem_slots + 2) + 64;
  spill_parts.alloc(part_cap * row_words * 8, ctx->stream);
  if (go_part && smem_slots > 0) setup_partitioned(nrows);
}

// Uploads the heavy hitters' table for smem_slots slots.
void AggState::preload_hot() {
  const int want = cfg.hot_keys > 0 ? cfg.hot_keys : smem_slots;
  const std::vector<uint64_t> hot = hot_table(std::min(want, smem_slots * 17 / 20), smem_slots, &nhot);
  hot_keys_dev.alloc(hot.size() * 8, ctx->stream);
  QEG_CUDA(cudaMemcpyAsync(hot_keys_dev.get(), hot.data(), hot.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
}

// The private tables that keep their size from batch to batch (partitioned
// passes, preloaded heavy hitters) were laid out for the first batch's fields:
// a batch whose values have NULLs needs their counts too, and may not fit with
// as many slots. It gets fewer, and a heavy hitters' table of that size.
void AggState::fit_private(const std::vector<StagedCol>& staged) {
  if (mode != 1 || (strategy != QEG_AGG_PARTITIONED && nhot == 0)) return;
  uint32_t skip = 0;
  for (size_t c = 0; c < val_cols.size(); ++c)
    if (staged[val_cols[c]].dev.all_valid) skip |= null_field(static_cast<int>(c));
  const int most = priv_max_slots(skip);
  if (smem_slots <= most) return;
  smem_slots = most;
  if (nhot > 0) preload_hot();
}

bool AggState::part_eligible(const std::vector<StagedCol>& staged) const {
  return mode == 1 && bucket_width == 0 && staged.size() == types.size();
}

// Slots of a second-pass table: two CTAs per SM.
int AggState::part_table_slots(uint32_t skip) const {
  int slots = 64;
  while (slots < 8192 &&
         priv_layout(fkind.data(), nfields, slots + 64, skip, 0).bytes + (slots + 64) * 2 + 1536 <= ctx->smem_optin / 2)
    slots += 64;
  return slots;
}

void AggState::setup_partitioned(uint64_t nrows) {
  // Without an estimate the row count bounds the group count.
  const double g = est_groups > 0 ? est_groups : std::max<double>(1.0, static_cast<double>(nrows));
  int bits = static_cast<int>(std::ceil(std::log2(std::max(2.0, g / (kPartFill * part_table_slots(0))))));
  if (const char* e = std::getenv("QEG_AGG_PART_BITS")) bits = std::atoi(e);
  // At most 2^15 partitions: the sizing pass keeps a 32-bit counter per
  // partition in shared memory.
  part_bits = std::max(1, std::min(bits, kPartMaxBits));
  strategy = QEG_AGG_PARTITIONED;
}

// The heavy hitters' table: S key words in which each of the first `want`
// candidates (most frequent first) lies in one of its two pairs of slots
// (hot_slot), then the slots of the kPrivReps most frequent ones (S: none).
// Built by moving earlier keys to their other pair; a key that finds no place
// is left out. Key word 0 has a row of its own.
std::vector<uint64_t> AggState::hot_table(int want, int S, int* count) const {
  std::vector<uint64_t> t(static_cast<size_t>(S) + kPrivReps, 0);
  auto find = [&](uint64_t k, uint64_t what) {  // slot of k's pairs that holds `what`
    const uint64_t h = key_hash1(k);
    const uint32_t p = hot_pair1(h, S), q = hot_pair2(h, S);
    for (uint32_t s : {p, p + 1, q, q + 1})
      if (t[s] == what) return static_cast<int>(s);
    return -1;
  };
  int n = 0;
  std::vector<std::pair<uint32_t, uint64_t>> undo;
  for (uint64_t c : heavy_candidates) {
    if (n >= want) break;
    if (c == 0 || find(c, c) >= 0) continue;  // (listed twice)
    undo.clear();
    uint64_t k = c;
    uint32_t pair = hot_pair1(key_hash1(k), S);
    bool placed = false;
    for (int step = 0; step < 64 && !placed; ++step) {
      const int free_slot = find(k, 0);
      if (free_slot >= 0) {
        t[free_slot] = k;
        placed = true;
        break;
      }
      const uint32_t s = pair + ((step >> 1) & 1);  // displace one key of the pair
      undo.emplace_back(s, t[s]);
      std::swap(k, t[s]);
      const uint64_t h = key_hash1(k);  // it goes to its other pair
      pair = pair == hot_pair1(h, S) ? hot_pair2(h, S) : hot_pair1(h, S);
    }
    if (placed) ++n;
    else
      for (size_t i = undo.size(); i-- > 0;) t[undo[i].first] = undo[i].second;
  }
  int r = 0;
  for (uint64_t c : heavy_candidates) {
    if (r == kPrivReps) break;
    const int s = c != 0 ? find(c, c) : -1;
    if (s >= 0) t[S + r++] = static_cast<uint64_t>(s);
  }
  for (; r < kPrivReps; ++r) t[S + r] = S;
  *count = n;
  return t;
}

namespace {
// The partitioned kernels of a field set.
struct PartKernels {
  void (*pass1)(AggK, PrivK, PoolK);
  void (*agg)(AggK, PrivK, PoolK, PartB);
  void (*insert)(AggK, PoolK, const uint32_t*, uint32_t, const uint32_t*, uint64_t);
  int words;
};
template <int NV, uint32_t SPEC, bool MASK>
PartKernels part_kernels_of() {
  return PartKernels{part_pass1_kernel<NV, SPEC, MASK>, part_agg_kernel<NV, SPEC, MASK>,
                     pool_insert_kernel<NV, SPEC, MASK>, pool_words<NV, MASK>()};
}
PartKernels part_kernels(uint32_t spec, int nv, bool nulls) {
  if (spec == kSpecIntF64) return part_kernels_of<2, kSpecIntF64, true>();
  if (spec == kSpecIntF64Nulls) return part_kernels_of<2, kSpecIntF64Nulls, true>();
  if (spec == kSpecIntSumF64Stats) return part_kernels_of<2, kSpecIntSumF64Stats, true>();
  if (spec == kSpecIntSumF64StatsNulls) return part_kernels_of<2, kSpecIntSumF64StatsNulls, true>();
  if (spec == kSpecF64) return part_kernels_of<1, kSpecF64, false>();
  if (spec == kSpecF64Nulls) return part_kernels_of<1, kSpecF64Nulls, true>();
  if (spec == kSpecCount) return part_kernels_of<1, kSpecCount, false>();
  if (nv <= 1) return nulls ? part_kernels_of<1, kGenericSpec, true>() : part_kernels_of<1, kGenericSpec, false>();
  if (nv <= 2) return part_kernels_of<2, kGenericSpec, true>();
  if (nv <= 4) return part_kernels_of<4, kGenericSpec, true>();
  return part_kernels_of<8, kGenericSpec, true>();
}
}  // namespace

// One batch through the partitioned passes: the sizing pass counts the rows
// of every partition that will go to the pool, a scan turns the counts into
// exact regions, the first pass aggregates the heavy hitters in the private
// tables and appends every other row to its region, the second pass
// aggregates each partition in shared memory.
void AggState::consume_partitioned(const std::vector<StagedCol>& staged, uint64_t nrows, uint64_t len,
                                   const uint32_t* dsel) {
  if (ntails) merge_tails();  // an earlier batch's groups join the global table
  const uint64_t np = 1ull << part_bits;
  AggK P = kparams(staged, dsel, nrows, len);
  const int nv = static_cast<int>(val_cols.size());
  uint32_t skip = 0;
  bool nulls = false;
  for (int c = 0; c < nv; ++c) {
    if (P.val[c].all_valid) skip |= null_field(c);
    else nulls = true;
  }
  const PartKernels kern = part_kernels(field_spec(P), nv, nulls);
  PoolK Q{};
  Q.shift = 64 - part_bits;
  if (part_words.bytes() < ((2 + kCursorWords) * np + 1) * 4)
    part_words.alloc(((2 + kCursorWords) * np + 1) * 4, ctx->stream);
  Q.hist = part_words.get<uint32_t>();
  Q.cursor = Q.hist + np;
  Q.off = Q.cursor + np * kCursorWords;
  QEG_CUDA(cudaMemsetAsync(Q.hist, 0, np * 4, ctx->stream));
  {
    const size_t sb = static_cast<size_t>(smem_slots) * 8 + np * 4;
    constexpr int kHistRows = 8;
    const int per_sm = blocks_per_sm(reinterpret_cast<const void*>(part_hist_kernel<kHistRows>), 1024, sb);
    require(per_sm > 0, "partition sizing kernel does not fit on an SM");
    const uint64_t grid = std::max<uint64_t>(
        1, std::min<uint64_t>((nrows + 65535) / 65536, static_cast<uint64_t>(ctx->sms) * per_sm));
    part_hist_kernel<kHistRows><<<(unsigned)grid, 1024, sb, ctx->stream>>>(P, Q, smem_slots);
    unsigned long long* total = counters.get<unsigned long long>() + 6;
    part_scan_kernel<<<1, 1024, 0, ctx->stream>>>(Q, total);
    ctx->launches += 2;
    QEG_CUDA(cudaGetLastError());
    uint64_t pooled = 0;
    read_words_and_error(ctx, total, 1, &pooled);
    Q.total = pooled;
  }
  // The pool takes 16 bytes or more per row that is not a heavy hitter's. An
  // input that would otherwise go to the private tables and the global one
  // does not depend on that memory: without it the batch goes there.
  try {
    const size_t pool_bytes = std::max<uint64_t>(Q.total, 1) * kern.words * 8;
    if (pool.bytes() < pool_bytes) pool.alloc(pool_bytes, ctx->stream);
  } catch (const Error& e) {
    if (e.code != QEG_ERR_OOM) throw;
    launch(P, nrows);
    settle(staged, len);
    return;
  }
  Q.rows = pool.get<uint64_t>();
  {
    PrivK A = priv_layout(fkind.data(), nfields, smem_slots, skip, kPrivReps);
    const int per_sm = blocks_per_sm(reinterpret_cast<const void*>(kern.pass1), 1024, A.bytes);
    require(per_sm > 0, "partitioned first pass does not fit on an SM");
    const uint64_t grid = std::max<uint64_t>(
        1, std::min<uint64_t>((nrows + 8191) / 8192, static_cast<uint64_t>(ctx->sms) * std::min(per_sm, 2)));
    priv_sums_for(A, grid);
    kern.pass1<<<(unsigned)grid, 1024, A.bytes, ctx->stream>>>(P, A, Q);
    ctx->launches++;
    QEG_CUDA(cudaGetLastError());
  }
  settle(staged, len);
  // ---- second pass ----
  P = kparams_base();
  for (int c = 0; c < nv; ++c) P.val[c].type = types[val_cols[c]] == QEG_F64 ? QEG_F64 : QEG_I64;
  PrivK A = priv_layout(fkind.data(), nfields, part_table_slots(skip), skip, 0);
  const size_t sb = A.bytes + static_cast<size_t>(A.slots) * 2;
  const int per_sm = blocks_per_sm(reinterpret_cast<const void*>(kern.agg), 512, sb);
  require(per_sm > 0, "partitioned aggregate kernel does not fit on an SM");
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(np, static_cast<uint64_t>(ctx->sms) * per_sm));
  priv_sums_for(A, grid);
  if (!part_counters.get()) part_counters.alloc(16, ctx->stream);
  if (part_failed.bytes() < np * 4) part_failed.alloc(np * 4, ctx->stream);
  PartB B{};
  B.counters = part_counters.get<unsigned long long>();
  B.failed = part_failed.get<uint32_t>();
  uint64_t cnt[2] = {0, 0};
  uint64_t want_tails = tails_cap ? tails_cap : static_cast<uint64_t>(std::max(1.25 * est_groups, 4096.0));
  for (int round = 0;; ++round) {
    require(round < 4, "partitioned aggregate: tail buffer sizing failed");
    // (Taken after the first pass: beside the pool it made the allocator's
    // blocks fit the next call worse, 256M Zipf rows 9.98 -> 10.72 ms.)
    try {
      if (tails_cap < want_tails) alloc_tails(want_tails);
    } catch (const Error& e) {
      if (e.code != QEG_ERR_OOM) throw;
      // No room for tail rows: every partition's rows go to the global table.
      std::vector<uint32_t> all(np);
      for (uint32_t i = 0; i < np; ++i) all[i] = i;
      QEG_CUDA(cudaMemcpyAsync(part_failed.get(), all.data(), np * 4, cudaMemcpyHostToDevice, ctx->stream));
      QEG_CUDA(cudaStreamSynchronize(ctx->stream));
      cnt[0] = 0;
      cnt[1] = np;
      break;
    }
    B.tails = tails.get<uint64_t>();
    B.tails_cap = tails_cap;
    QEG_CUDA(cudaMemsetAsync(part_counters.get(), 0, 16, ctx->stream));
    kern.agg<<<grid, 512, sb, ctx->stream>>>(P, A, Q, B);
    ctx->launches++;
    QEG_CUDA(cudaGetLastError());
    read_words_and_error(ctx, part_counters.get(), 2, cnt);
    if (cnt[0] <= tails_cap) break;
    // More groups than the tail buffer holds: size it to the count and re-run
    // (the pass only reads the pool).
    want_tails = cnt[0] + cnt[0] / 8 + 4096;
  }
  ntails = cnt[0];
  // Two empty rows after the tails: the finalize pass reads a single-key
  // table's side rows there.
  if (tails_cap) QEG_CUDA(cudaMemsetAsync(tails.get<uint64_t>() + ntails * row_words, 0, 2 * row_words * 8, ctx->stream));
  // Partitions whose groups did not fit their table: rows into the global
  // table, which grows until all have a place.
  const uint32_t nfailed = static_cast<uint32_t>(std::min<uint64_t>(cnt[1], np));
  if (nfailed == 0) return;
  DevBuf list;
  uint64_t nlist = 0;
  for (int round = 0; round == 0 || nlist > 0; ++round) {
    require(round < 64, "aggregate table failed to converge after 64 resize rounds");
    QEG_CUDA(cudaMemsetAsync(counters.get(), 0, 8, ctx->stream));
    P = kparams_base();
    for (int c = 0; c < nv; ++c) P.val[c].type = types[val_cols[c]] == QEG_F64 ? QEG_F64 : QEG_I64;
    P.spill_rows = spill_rows.get<uint32_t>();
    P.spill_cap = spill_cap;
    const unsigned g = round == 0 ? std::min<unsigned>(nfailed, ctx->sms * 4u) : grid_for(ctx, nlist, 512, 4);
    kern.insert<<<g, 512, 0, ctx->stream>>>(P, Q, part_failed.get<uint32_t>(), nfailed, list.get<uint32_t>(), nlist);
    ctx->launches++;
    QEG_CUDA(cudaGetLastError());
    uint64_t c[3];
    read_words_and_error(ctx, counters.get(), 3, c);
    inserted = c[2];
    nlist = c[0];
    if (nlist == 0) break;
    list.alloc(nlist * 4, ctx->stream);
    QEG_CUDA(cudaMemcpyAsync(list.get(), spill_rows.get(), nlist * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    grow(std::max<uint64_t>(cap * 2, next_pow2(2 * (inserted + nlist / 4))));
  }
  QEG_CUDA(cudaMemsetAsync(counters.get(), 0, 16, ctx->stream));
}

// Room for `rows` tail rows and the two empty ones behind them.
void AggState::alloc_tails(uint64_t rows) {
  tails_cap = 0;
  tails.alloc((rows + 2) * row_words * 8, ctx->stream);
  tails_cap = rows;
}

// The launch's blocks of F64 sums, one per CTA.
void AggState::priv_sums_for(PrivK& A, uint64_t grid) {
  if (priv_sums.bytes() < A.sum_bytes * grid) priv_sums.alloc(A.sum_bytes * grid, ctx->stream);
  A.sums = priv_sums.get<uint8_t>();
}

// Moves the tail rows into the global table (grown to hold them).
void AggState::merge_tails() {
  if (ntails == 0) return;
  const uint64_t need = next_pow2(2 * (inserted + ntails));
  if (cap < need) grow(need);
  AggK Q = kparams_base();
  merge_parts_kernel<1><<<grid_for(ctx, ntails, 256, 8), 256, 0, ctx->stream>>>(Q, tails.get<uint64_t>(), ntails);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
  uint64_t c[3];
  read_counters(c);
  check_device_error(ctx);
  inserted = c[2];
  ntails = 0;
}

void AggState::finish(uint64_t* nrows_out) {
  if (finished) {
    *nrows_out = nout;
    return;
  }
  if (!table.get()) {
    // Nothing consumed: set up an empty table so the global case emits its row.
    std::vector<StagedCol> none;
    first_consume(none, 0, 0, nullptr);
  }
  const uint64_t out_cap = (mode == 0) ? 1 : std::max<uint64_t>(inserted + 2 + ntails, 1);
  const int ncolsout = static_cast<int>(keys.size() + aggs.size());
  // One allocation for all output columns.
  const size_t val_bytes = (out_cap * 8 + 255) / 256 * 256, ok_bytes = (out_cap + 255) / 256 * 256;
  out_slab.alloc((val_bytes + ok_bytes) * ncolsout, ctx->stream);
  out_vals.assign(ncolsout, nullptr);
  out_valid.assign(ncolsout, nullptr);
  FinK F{};
  F.naggs = static_cast<int>(aggs.size());
  for (int c = 0; c < ncolsout; ++c) {
    out_vals[c] = out_slab.get<uint8_t>() + val_bytes * c;
    out_valid[c] = out_slab.get<uint8_t>() + val_bytes * ncolsout + ok_bytes * c;
    F.vals[c] = out_vals[c];
    F.valid[c] = out_valid[c];
    F.rtype[c] = rtypes[c];
  }
  for (size_t a = 0; a < aggs.size(); ++a) {
    F.func[a] = aggs[a].func;
    F.vfield[a] = vfield[a];
    F.nfield[a] = nfield[a];
  }
  F.out_count = counters.get<unsigned long long>() + 5;
  QEG_CUDA(cudaMemsetAsync(F.out_count, 0, 8, ctx->stream));
  F.out_cap = out_cap;
  F.packed_width = packed ? bucket_width : 0;
  F.packed_pair = packed && bucket_width == 0;
  AggK P = kparams_base();
  if (mode == 1 && ntails > 0) {
    // Partitioned strategy: the tail rows first, each merged into the global
    // table instead when its key is there too; then the global table.
    AggK T = P;
    T.table = tails.get<uint64_t>();
    T.cap = ntails;
    FinK FT = F;
    FT.merge_table = table.get<uint64_t>();
    FT.merge_cap = cap;
    finalize_kernel<1><<<grid_for(ctx, ntails + 2, 1024, 2), 1024, 0, ctx->stream>>>(T, FT);
    ctx->launches++;
    QEG_CUDA(cudaGetLastError());
  }
  const uint64_t total = (mode == 0) ? 1 : (mode == 1 ? cap + 2 : cap);
  const unsigned g = grid_for(ctx, total, 1024, 2);
  if (mode == 0) finalize_kernel<0><<<g, 1024, 0, ctx->stream>>>(P, F);
  else if (mode == 1) finalize_kernel<1><<<g, 1024, 0, ctx->stream>>>(P, F);
  else finalize_kernel<2><<<g, 1024, 0, ctx->stream>>>(P, F);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
  read_words_and_error(ctx, F.out_count, 1, &nout);  // one synchronisation
  finished = true;
  *nrows_out = nout;
}

void AggState::fetch(uint64_t first, uint64_t count, const qeg_out_column* outs) {
  require(finished, "fetch() before finish()");
  require(first <= nout && count <= nout - first, "fetch range outside the result");
  require(outs != nullptr, "outs is NULL");
  std::vector<FetchCol> cols;
  for (size_t c = 0; c < out_vals.size(); ++c)
    cols.push_back(FetchCol{out_vals[c], out_valid[c], type_width(rtypes[c])});
  fetch_columns(ctx, cols.data(), static_cast<int>(cols.size()), first, count, outs);
}

}  // namespace qeg

using qeg::AggState;

struct qeg_agg {
  AggState st;
};

extern "C" {

qeg_status qeg_agg_create(qeg_ctx* ctx, const int32_t* col_types, int ncols, const uint32_t* key_cols,
                          int nkeys, const qeg_agg_spec* aggs, int naggs, const qeg_agg_config* cfg,
                          qeg_agg** out) {
  return qeg::guarded(ctx, [&] {
    qeg::require(ctx != nullptr && out != nullptr, "ctx/out is NULL");
    QEG_CUDA(cudaSetDevice(ctx->device));
    auto a = std::make_unique<qeg_agg>();
    a->st.ctx = ctx;
    if (cfg) a->st.cfg = *cfg;
    const int bt = a->st.cfg.block_threads;
    qeg::require(bt == 0 || (bt >= 32 && bt <= 1024 && bt % 32 == 0),
                 "block_threads must be 0 or a multiple of 32 in [32, 1024]");
    a->st.plan(col_types, ncols, key_cols, nkeys, aggs, naggs);
    *out = a.release();
  });
}

qeg_status qeg_window_create(qeg_ctx* ctx, const int32_t* col_types, int ncols, const uint32_t* key_cols,
                             int nkeys, uint32_t time_col, int64_t width, const qeg_agg_spec* aggs, int naggs,
                             const qeg_agg_config* cfg, qeg_agg** out) {
  return qeg::guarded(ctx, [&] {
    qeg::require(ctx != nullptr && out != nullptr, "ctx/out is NULL");
    qeg::require(ncols > 0 && col_types != nullptr, "window needs an input schema");
    qeg::require(nkeys >= 0 && (nkeys == 0 || key_cols != nullptr), "key_cols is NULL");
    qeg::require(nkeys + 1 <= qeg::kMaxKeys, "GPU window supports at most 7 partition keys");
    qeg::require(naggs >= 1 && aggs != nullptr, "Window needs >=1 aggregate");
    qeg::require(time_col < static_cast<uint32_t>(ncols), "window time column out of range");
    for (int k = 0; k < nkeys; ++k) {
      qeg::require(key_cols[k] < static_cast<uint32_t>(ncols), "window key column out of range");
      qeg::require(col_types[key_cols[k]] != QEG_STR,
                   "Window: STR partition keys are not supported (out of grammar)");
    }
    for (int a = 0; a < naggs; ++a)
      if (aggs[a].func != QEG_COUNT_STAR && aggs[a].input_col < static_cast<uint32_t>(ncols))
        qeg::require(col_types[aggs[a].input_col] != QEG_STR,
                     "Window: STR aggregate inputs are not supported (out of grammar)");
    const int32_t tt = col_types[time_col];
    qeg::require(tt == QEG_I32 || tt == QEG_I64 || tt == QEG_TS, "Window: time column must be I32/I64/TS");
    qeg::require(width > 0, "Window: tumbling width W must be > 0");
    std::vector<uint32_t> k(key_cols, key_cols + nkeys);
    k.push_back(time_col);
    QEG_CUDA(cudaSetDevice(ctx->device));
    auto a = std::make_unique<qeg_agg>();
    a->st.ctx = ctx;
    if (cfg) a->st.cfg = *cfg;
    const int bt = a->st.cfg.block_threads;
    qeg::require(bt == 0 || (bt >= 32 && bt <= 1024 && bt % 32 == 0),
                 "block_threads must be 0 or a multiple of 32 in [32, 1024]");
    a->st.plan(col_types, ncols, k.data(), nkeys + 1, aggs, naggs);
    a->st.bucket_width = width;
    const int32_t kt = nkeys == 1 ? col_types[key_cols[0]] : -1;
    a->st.packable = kt == QEG_I32 || kt == QEG_I64 || kt == QEG_TS;
    *out = a.release();
  });
}

qeg_status qeg_agg_consume(qeg_agg* agg, const qeg_column* cols, int ncols, const uint32_t* sel,
                           uint64_t sel_len) {
  qeg::NvtxRange nvtx_range("qeg_agg_consume");
  qeg_ctx* ctx = agg ? agg->st.ctx : nullptr;
  return qeg::guarded(ctx, [&] {
    qeg::require(agg != nullptr, "agg is NULL");
    QEG_CUDA(cudaSetDevice(ctx->device));
    agg->st.consume(cols, ncols, sel, sel_len);
  });
}

qeg_status qeg_agg_finish(qeg_agg* agg, uint64_t* num_rows) {
  qeg::NvtxRange nvtx_range("qeg_agg_finish");
  qeg_ctx* ctx = agg ? agg->st.ctx : nullptr;
  return qeg::guarded(ctx, [&] {
    qeg::require(agg != nullptr && num_rows != nullptr, "agg/num_rows is NULL");
    QEG_CUDA(cudaSetDevice(ctx->device));
    agg->st.finish(num_rows);
  });
}

qeg_status qeg_agg_result_types(const qeg_agg* agg, int32_t* types) {
  qeg_ctx* ctx = agg ? agg->st.ctx : nullptr;
  return qeg::guarded(ctx, [&] {
    qeg::require(agg != nullptr && types != nullptr, "agg/types is NULL");
    for (size_t c = 0; c < agg->st.rtypes.size(); ++c) types[c] = agg->st.rtypes[c];
  });
}

qeg_status qeg_agg_fetch(qeg_agg* agg, uint64_t first, uint64_t count, const qeg_out_column* outs) {
  qeg::NvtxRange nvtx_range("qeg_agg_fetch");
  qeg_ctx* ctx = agg ? agg->st.ctx : nullptr;
  return qeg::guarded(ctx, [&] {
    qeg::require(agg != nullptr, "agg is NULL");
    QEG_CUDA(cudaSetDevice(ctx->device));
    agg->st.fetch(first, count, outs);
  });
}

qeg_status qeg_agg_stats(const qeg_agg* agg, uint64_t* capacity, uint32_t* resizes, int32_t* strategy,
                         int32_t* hot_keys, double* est_groups) {
  qeg_ctx* ctx = agg ? agg->st.ctx : nullptr;
  return qeg::guarded(ctx, [&] {
    qeg::require(agg != nullptr, "agg is NULL");
    if (capacity) *capacity = agg->st.cap;
    if (resizes) *resizes = agg->st.resizes;
    if (strategy) *strategy = agg->st.strategy;
    if (hot_keys) *hot_keys = agg->st.nhot;
    if (est_groups) *est_groups = agg->st.est_groups;
  });
}

void qeg_agg_destroy(qeg_agg* agg) {
  if (!agg) return;
  cudaSetDevice(agg->st.ctx->device);
  delete agg;
}

}  // extern "C"
