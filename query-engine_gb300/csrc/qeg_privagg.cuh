// qeg_privagg.cuh -- CTA-private GROUP BY tables in shared memory whose rows
// are updated lane by lane with shared-memory reductions.
#pragma once

#include "qeg_agg.h"
#include "qeg_device.cuh"
#include "qeg_warpagg.cuh"

namespace qeg {

// ---------------------------------------------------------------------------
// Layout (dynamic shared memory): [slots] key words, then one array per
// aggregate field over all rows, then a replica number per slot. Rows are the
// slots, a row for key word 0, a row for the NULL key, and 32 replica rows
// (one per lane) for each of up to kPrivReps hot slots. Row and NULL counts
// are 32-bit (a CTA sees fewer than 2^32 rows), other fields 64-bit.
// F64 sums live in a block of global memory of the CTA's own, which stays in
// L2: shared memory has no F64 add, and its compare-and-swap loop costs 1986
// clocks per 32 rows spread over 8 words, 348 over 64 and 103 over 512 (32
// warps of an SM at once), while a reduction at L2 costs 70-95 clocks of L2
// throughput whatever the spread, and no time of the SM. 64-bit integer sums
// are added as two 32-bit halves with a carry: the 64-bit shared add is such
// a loop too (352 clocks over 8 words, 32-bit adds take 3).
// Where most rows miss the private tables anyway and update a global table far
// beyond L2, those reductions are what bounds the launch (about 50 G/s there),
// and the hits' sums must not add to them: SSUM tables keep the F64 sums in
// shared memory, in fewer slots.
// ---------------------------------------------------------------------------
constexpr int kPrivReps = 16;

struct PrivK {
  int slots;  // power of two, a multiple of 4
  int rows;   // slots + 2 + 32 replica rows per replicated slot
  uint32_t foff[kMaxFields];  // byte offset of each field's array (F64 sums: in the CTA's global block)
  uint32_t rep_off;           // u8 per slot row (slots + 2): replica number, 0 = none
  uint32_t bytes;             // whole table, a multiple of 16
  uint32_t skip;              // fields without an array
  uint32_t sum_bytes;         // F64 sums per CTA, a multiple of 16
  uint8_t* sums;              // the launch's blocks, one per CTA
};

// Lays out a table of `slots` slots for the given fields. `skip` has a bit for
// every field that no row of the launch changes (NULL counts of columns
// without NULLs): these have no array; `reps` is the number of slots that may
// have replica rows; `ssum` puts F64 sums into shared memory too.
inline PrivK priv_layout(const uint8_t* fkind, int nfields, int slots, uint32_t skip, int reps, bool ssum = false) {
  PrivK A{};
  A.slots = slots;
  A.rows = slots + 2 + 32 * reps;
  uint32_t at = static_cast<uint32_t>(slots) * 8;
  for (int pass = 0; pass < 2; ++pass)  // 8-byte fields first
    for (int f = 0; f < nfields; ++f) {
      const uint32_t size = fkind[f] <= F_NULLS ? 4 : 8;
      if ((fkind[f] == F_SUMF && !ssum) || (size == 4) != (pass == 1) || ((skip >> f) & 1u)) continue;
      A.foff[f] = at;
      at += size * static_cast<uint32_t>(A.rows);
    }
  for (int f = 0; f < nfields; ++f)
    if (fkind[f] == F_SUMF && !ssum) {
      A.foff[f] = A.sum_bytes;
      A.sum_bytes += 8 * static_cast<uint32_t>(A.rows);
    }
  A.skip = skip;
  A.rep_off = at;
  at += static_cast<uint32_t>(slots + 2);
  A.bytes = (at + 15) / 16 * 16;
  A.sum_bytes = (A.sum_bytes + 15) / 16 * 16;
  return A;
}

// A CTA's table: its shared-memory address and its block of F64 sums.
struct PrivT {
  uint32_t base;
  uint8_t* sums;
};

// Slot of key word k (nonzero) in the private table, found or claimed, or -1:
// its four-slot bucket is full. Slots are tried in the order s ^ 0..3 from the
// home slot and filled in that order, so the first empty one ends the search.
__device__ __forceinline__ int priv_slot(uint64_t* keys, int slots, uint64_t k, uint64_t h) {
  const uint32_t s0 = static_cast<uint32_t>(h >> 32) & static_cast<uint32_t>(slots - 1);
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) {
    const uint32_t s = s0 ^ j;
    unsigned long long cur = *reinterpret_cast<const volatile unsigned long long*>(keys + s);
    if (cur == k) return static_cast<int>(s);
    if (cur == 0) {
      cur = atomicCAS(reinterpret_cast<unsigned long long*>(keys + s), 0ull, static_cast<unsigned long long>(k));
      if (cur == 0 || cur == k) return static_cast<int>(s);
    }
  }
  return -1;
}

// Read-only table of heavy hitters: a key lies in one of two pairs of slots
// (first slot of each), loaded 16 bytes at a time, without a search. The slot
// that holds key word k (nonzero), or -1. (Single slots would fill to 0.45 at
// most, pairs to 0.85: 3480 keys in 4096 slots, 7.77 -> 7.71 ms for 256M Zipf
// rows.)
__host__ __device__ __forceinline__ uint32_t hot_pair1(uint64_t h, int slots) {
  return static_cast<uint32_t>(h >> 32) & static_cast<uint32_t>(slots - 2);
}
__host__ __device__ __forceinline__ uint32_t hot_pair2(uint64_t h, int slots) {
  return static_cast<uint32_t>(h >> 46) & static_cast<uint32_t>(slots - 2);
}
__device__ __forceinline__ int hot_slot(const uint64_t* keys, int slots, uint64_t k, uint64_t h) {
  const int p = static_cast<int>(hot_pair1(h, slots)), q = static_cast<int>(hot_pair2(h, slots));
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(keys + p);
  const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(keys + q);
  int s = -1;
  if (b.y == k) s = q + 1;
  if (b.x == k) s = q;
  if (a.y == k) s = p + 1;
  if (a.x == k) s = p;
  return s;
}

// Merges one contribution x into field f (of kind `kind`) of private row `row`.
template <bool SSUM = false>
__device__ __forceinline__ void priv_red(const PrivT& T, const PrivK& A, int f, uint8_t kind, int row, uint64_t x) {
  if (!x) return;  // zero is the identity of every field
  if (kind == F_SUMF && !SSUM) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(T.sums + A.foff[f] + static_cast<uint32_t>(row) * 8u),
                 "d"(__longlong_as_double(static_cast<long long>(x)))
                 : "memory");
    return;
  }
  const uint32_t a = T.base + A.foff[f] + static_cast<uint32_t>(row) * (kind <= F_NULLS ? 4u : 8u);
  if (kind == F_SUMF) {
    asm volatile("red.shared.add.f64 [%0], %1;" ::"r"(a), "d"(__longlong_as_double(static_cast<long long>(x))) : "memory");
  } else if (kind <= F_NULLS) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(static_cast<uint32_t>(x)) : "memory");
  } else if (kind == F_SUMI) {
    const uint32_t lo = static_cast<uint32_t>(x);
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(lo) : "memory");
    const uint32_t hi = static_cast<uint32_t>(x >> 32) + (old + lo < old ? 1u : 0u);
    if (hi) asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a + 4), "r"(hi) : "memory");
  } else {
    asm volatile("red.shared.max.u64 [%0], %1;" ::"r"(a), "l"(x) : "memory");
  }
}

template <bool SSUM = false>
__device__ __forceinline__ uint64_t priv_load(const PrivT& T, const PrivK& A, int f, uint8_t kind, int row) {
  uint64_t v;
  if (kind == F_SUMF && !SSUM) {  // from L2, where the reductions land
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
                 : "=l"(v)
                 : "l"(T.sums + A.foff[f] + static_cast<uint32_t>(row) * 8u)
                 : "memory");
    return v;
  }
  const uint32_t a = T.base + A.foff[f] + static_cast<uint32_t>(row) * (kind <= F_NULLS ? 4u : 8u);
  if (kind <= F_NULLS) {
    uint32_t w;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(a) : "memory");
    return w;
  }
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}

template <bool SSUM = false>
__device__ __forceinline__ void priv_clear(const PrivT& T, const PrivK& A, int f, uint8_t kind, int row) {
  if (kind == F_SUMF && !SSUM) {
    *reinterpret_cast<volatile uint64_t*>(T.sums + A.foff[f] + static_cast<uint32_t>(row) * 8u) = 0;
    return;
  }
  const uint32_t a = T.base + A.foff[f] + static_cast<uint32_t>(row) * (kind <= F_NULLS ? 4u : 8u);
  if (kind <= F_NULLS) asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(0u) : "memory");
  else asm volatile("st.shared.u64 [%0], %1;" ::"r"(a), "l"(0ull) : "memory");
}

// Zeroes the CTA's table; a barrier must follow.
__device__ __forceinline__ PrivT priv_init(uint64_t* sm, const PrivK& A) {
  const PrivT T{static_cast<uint32_t>(__cvta_generic_to_shared(sm)),
                A.sums + static_cast<size_t>(blockIdx.x) * A.sum_bytes};
  for (uint32_t i = threadIdx.x; i < A.bytes / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(sm)[i] = make_uint4(0, 0, 0, 0);
  for (uint32_t i = threadIdx.x; i < A.sum_bytes / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(T.sums)[i] = make_uint4(0, 0, 0, 0);
  return T;
}

// Adds one input row to private row `row`.
template <uint32_t SPEC, int NV, bool SSUM = false>
__device__ __forceinline__ void priv_apply(const PrivT& T, const PrivK& A, int row, const uint8_t* fkind,
                                           const uint8_t* fcol, int nfields, const bool (&vv)[kMaxVals],
                                           const uint64_t (&vb)[kMaxVals]) {
  priv_red<SSUM>(T, A, 0, F_ROWS, row, 1);
  if constexpr (SPEC != kGenericSpec) {
#pragma unroll
    for (int i = 1; i <= spec_n(SPEC); ++i) {
      const uint8_t kind = static_cast<uint8_t>(spec_kind(SPEC, i));
      const int col = spec_col(SPEC, i) < NV ? spec_col(SPEC, i) : 0;
      if (kind != 0) priv_red<SSUM>(T, A, i, kind, row, field_contrib(kind, vv[col], vb[col]));
    }
  } else {
#pragma unroll 1
    for (int i = 1; i < nfields; ++i) {
      const uint8_t kind = fkind[i];
      bool v = false;
      uint64_t b = 0;
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        if (j == fcol[i]) {
          v = vv[j];
          b = vb[j];
        }
      }
      const uint64_t x = field_contrib(kind, v, b);
      if (x) priv_red<SSUM>(T, A, i, kind, row, x);
    }
  }
}

// Adds one input row to the field block `f` of a global table row.
template <uint32_t SPEC, int NV>
__device__ __forceinline__ void global_apply(uint64_t* f, const uint8_t* fkind, const uint8_t* fcol, int nfields,
                                             const bool (&vv)[kMaxVals], const uint64_t (&vb)[kMaxVals]) {
  field_red<kRowGlobal>(f, F_ROWS, 1);
  if constexpr (SPEC != kGenericSpec) {
#pragma unroll
    for (int i = 1; i <= spec_n(SPEC); ++i) {
      const uint8_t kind = static_cast<uint8_t>(spec_kind(SPEC, i));
      const int col = spec_col(SPEC, i) < NV ? spec_col(SPEC, i) : 0;
      if (kind != 0) field_red<kRowGlobal>(f + i, kind, field_contrib(kind, vv[col], vb[col]));
    }
  } else {
#pragma unroll 1
    for (int i = 1; i < nfields; ++i) {
      const uint8_t kind = fkind[i];
      bool v = false;
      uint64_t b = 0;
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        if (j == fcol[i]) {
          v = vv[j];
          b = vb[j];
        }
      }
      field_red<kRowGlobal>(f + i, kind, field_contrib(kind, v, b));
    }
  }
}

// Gives the slots that several lanes of a warp hit at once a row per lane:
// lanes on one word serialise (an F64 reduction over one word costs 231
// clocks per warp, over a word per lane 54).
// All lanes call it; `slot` is -1 where the lane has none. At most kPrivReps
// slots get replicas until the next flush. Two warps may give a slot two
// replica sets at once: both are folded back, the later one is used.
__device__ __forceinline__ void priv_promote(int slot, uint8_t* rep, uint16_t* rslot, unsigned* nrep, unsigned lane) {
  const unsigned peers = __match_any_sync(0xffffffffu, slot >= 0 ? static_cast<unsigned>(slot) : (0x80000000u | lane));
  if (slot >= 0 && __popc(peers) >= 3 && __ffs(peers) - 1 == static_cast<int>(lane) && rep[slot] == 0 &&
      *reinterpret_cast<volatile unsigned*>(nrep) < kPrivReps) {
    const unsigned id = atomicAdd(nrep, 1u);
    if (id < kPrivReps) {
      rslot[id] = static_cast<uint16_t>(slot);
      rep[slot] = static_cast<uint8_t>(id + 1);
    }
  }
  __syncwarp();
}

// Adds the replica rows to their slots' rows and clears them. All threads of
// the CTA call it, after a barrier; priv_fence() must follow before the slots'
// rows are read.
template <bool SSUM = false>
__device__ __forceinline__ void priv_fold(const PrivT& T, const PrivK& A, const uint16_t* rslot, unsigned nrep,
                                          const uint8_t* fkind, int nfields) {
  const int n = static_cast<int>(min(nrep, static_cast<unsigned>(kPrivReps))) * 32;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int row = A.slots + 2 + i, slot = rslot[i >> 5];
    for (int f = 0; f < nfields; ++f) {
      if ((A.skip >> f) & 1u) continue;
      const uint8_t kind = fkind[f];
      priv_red<SSUM>(T, A, f, kind, slot, priv_load<SSUM>(T, A, f, kind, row));
      priv_clear<SSUM>(T, A, f, kind, row);
    }
  }
}

// Barrier after which every thread of the CTA sees every earlier update of
// the table (the F64 sums' reductions are performed at L2).
__device__ __forceinline__ void priv_fence() {
  __threadfence();
  __syncthreads();
}

}  // namespace qeg
