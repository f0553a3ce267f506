// qeg_sketch.cu -- on-device sketch of a key column: HyperLogLog registers,
// a count-min sketch and heavy-hitter candidates over a strided sample. The
// sketch is the input of the distinct-group estimator that sizes the GROUP BY
// table and picks its strategy (the reference sizes by growth only,
// ops/hashtable.h:83-94; results never depend on the estimate, because an
// overflowing table is grown and the affected rows replayed).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "qeg_agg.h"
#include "qeg_mlp.h"

namespace qeg {

namespace {

constexpr int kHllP = 14;
constexpr int kHllM = 1 << kHllP;
constexpr int kCmsDepth = 4;
constexpr int kCmsWidth = 2048;
constexpr int kCandLocal = 1024;
constexpr int kCandGlobal = 8192;
constexpr int kSampleBlock = 256;

// What the host needs of a sketch: whole numbers, from which it computes the
// features, and the network's outputs for them.
struct SketchOut {
  uint32_t hist[66];             // registers by value (the last: padding)
  unsigned long long top[12];    // sum of the 2^i largest candidate estimates
  unsigned long long f2;         // sum of squares of the first count-min row
  unsigned long long rows, nulls;
  float net[2];
};

struct SketchK {
  DevCol key;
  const uint32_t* sel;
  uint64_t nrows, len;
  uint64_t stride;   // rows between the starts of consecutive sample blocks
  uint64_t nblocks;  // sample blocks
  uint32_t* hll;     // kHllM
  uint32_t* cms;     // kCmsDepth * kCmsWidth
  unsigned long long* cand_key;  // kCandGlobal
  unsigned long long* cand_cnt;  // kCandGlobal
  unsigned long long* stats;     // [0] sampled rows, [1] sampled nulls
  unsigned int* done;            // CTAs that have merged their part
  SketchOut* out;
  const __nv_bfloat16* net;      // estimator weights, or nullptr
  float log_rows, log_total, sampled;  // features 75..77 (known before the sample is read)
  uint32_t* err;
};

__device__ __forceinline__ uint64_t sketch_hash(uint64_t w) { return mix64(w ^ 0x243F6A8885A308D3ull); }

// The registers and the sketch take 140 KB of shared memory, so one CTA runs
// per SM: kSketchThreads of them, several sample blocks at a time, hide the
// latency of the loads and shared-memory atomics (256 threads: 67 us for 1M
// sampled rows).
constexpr int kSketchThreads = 1024;

// The merged sketch's host part, by the last CTA: register histogram,
// candidates ranked by their count-min estimates, features, network. On the
// host this took up to 0.3 ms (225 KB copied, 8192 candidates sorted, and the
// network as a round trip of its own); here it adds 10 to 25 us to the launch.
__device__ void sketch_finish(const SketchK& P, uint32_t* sh) {
  uint32_t* ranked = sh;                                     // kCandGlobal
  __nv_bfloat16* w = reinterpret_cast<__nv_bfloat16*>(sh + kCandGlobal);  // kParams
  uint32_t* cms = sh + kHllM;                                // kCmsDepth * kCmsWidth
  static_assert(kCandGlobal * 4 + kParams * 2 <= kHllM * 4, "candidates and weights take the registers' place");
  __shared__ uint32_t hist[66], nranked;
  __shared__ unsigned long long top[12], f2;
  __shared__ float f[kIn], h1[kHid], h2[kHid];
  const unsigned tid = threadIdx.x, lane = tid & 31u;
  if (tid < 66) hist[tid] = 0;
  if (tid < 12) top[tid] = 0;
  if (tid == 0) {
    nranked = 0;
    f2 = 0;
  }
  if (P.net)
    for (unsigned i = tid; i < kParams; i += blockDim.x) w[i] = P.net[i];
  for (unsigned i = tid; i < kCmsDepth * kCmsWidth; i += blockDim.x) cms[i] = __ldcg(P.cms + i);
  __syncthreads();
  for (unsigned i = tid; i < kHllM; i += blockDim.x) {  // (kHllM is a multiple of the block)
    const uint32_t r = min(__ldcg(P.hll + i), 64u);
    const unsigned same = __match_any_sync(0xffffffffu, r);
    if (static_cast<unsigned>(__ffs(same)) == lane + 1) atomicAdd(&hist[r], static_cast<unsigned>(__popc(same)));
  }
  unsigned long long sq = 0;
  for (unsigned c = tid; c < kCmsWidth; c += blockDim.x) sq += static_cast<unsigned long long>(cms[c]) * cms[c];
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
  if (lane == 0) atomicAdd(&f2, sq);
  for (unsigned i = tid; i < kCandGlobal; i += blockDim.x) {
    const unsigned long long kk = __ldcg(P.cand_key + i);
    if (!kk) continue;
    const uint64_t h = sketch_hash(kk - 1);
    uint32_t best = UINT32_MAX;
#pragma unroll
    for (int d = 0; d < kCmsDepth; ++d) {
      const uint32_t c = static_cast<uint32_t>(mix64(h + 0x9E3779B97F4A7C15ull * (d + 1)) >> 40) & (kCmsWidth - 1);
      best = min(best, cms[d * kCmsWidth + c]);
    }
    ranked[atomicAdd(&nranked, 1u)] = best;
  }
  __syncthreads();
  // Descending bitonic sort, padded with zeros to a power of two. A thread
  // holds 8 neighbours, a warp 256: steps within them are exchanges of
  // registers and lanes, the wider ones go through shared memory (step by step
  // there, 8192 candidates took 45 us).
  const unsigned n = nranked;
  unsigned size = 256;
  while (size < n) size *= 2;
  for (unsigned i = n + tid; i < size; i += blockDim.x) ranked[i] = 0;
  __syncthreads();
  for (unsigned k = 2; k <= size; k <<= 1) {
    for (unsigned j = k >> 1; j >= 256; j >>= 1) {
      for (unsigned q = tid; q < size / 2; q += blockDim.x) {
        const unsigned i = 2 * q - (q & (j - 1)), x = i + j;
        const uint32_t a = ranked[i], b = ranked[x];
        if ((i & k) == 0 ? a < b : a > b) {
          ranked[i] = b;
          ranked[x] = a;
        }
      }
      __syncthreads();
    }
    if (tid * 8 < size) {  // whole warps: size is a multiple of 256
      uint32_t v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = ranked[tid * 8 + e];
      for (unsigned j = min(k >> 1, 128u); j >= 8; j >>= 1) {
        const bool larger = ((tid * 8 & k) == 0) == ((tid * 8 & j) == 0);  // this end takes the larger one
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v[e], j / 8);
          v[e] = larger ? max(v[e], o) : min(v[e], o);
        }
      }
#pragma unroll
      for (unsigned j = 4; j >= 1; j >>= 1) {
        if (j >= k) continue;
#pragma unroll
        for (unsigned e = 0; e < 8; ++e) {
          if (e & j) continue;
          const uint32_t lo = min(v[e], v[e | j]), hi = max(v[e], v[e | j]);
          const bool down = ((tid * 8 + e) & k) == 0;
          v[e] = down ? hi : lo;
          v[e | j] = down ? lo : hi;
        }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ranked[tid * 8 + e] = v[e];
    }
    __syncthreads();
  }
  // The estimate at position j counts toward every prefix longer than j:
  // bucket bitlength(j) and above (the same for 32 aligned positions from 32 on).
  for (unsigned j = tid; j < 2048 && j - lane < size; j += blockDim.x) {
    const int b = j == 0 ? 0 : 32 - __clz(j);
    unsigned long long v = ranked[j];
    if (j < 32) {
      atomicAdd(&top[b], v);
    } else {
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) atomicAdd(&top[b], v);
    }
  }
  __syncthreads();
  if (tid == 0)
    for (int i = 1; i < 12; ++i) top[i] += top[i - 1];
  __syncthreads();
  const unsigned long long rows = __ldcg(P.stats), nulls = __ldcg(P.stats + 1);
  if (P.net) {
    // Features as the host computes them (sketch_features).
    const double nonnull = static_cast<double>(rows) - static_cast<double>(nulls);
    if (tid < kIn) {
      float v = 0;
      if (tid < 64) {
        v = static_cast<float>(hist[tid]) / kHllM;
        if (tid == 63) v += static_cast<float>(hist[64]) / kHllM;
      } else if (tid < 74) {
        v = nonnull > 0 ? static_cast<float>(fmin(1.0, static_cast<double>(top[tid - 64]) / nonnull)) : 0.f;
      } else if (tid == 74) {
        v = nonnull > 0 ? static_cast<float>(static_cast<double>(f2) / (nonnull * nonnull)) : 0.f;
      } else if (tid == 75) {
        v = P.log_rows;
      } else if (tid == 76) {
        v = P.log_total;
      } else if (tid == 77) {
        v = P.sampled;
      } else if (tid == 78) {
        v = rows ? static_cast<float>(static_cast<double>(nulls) / static_cast<double>(rows)) : 0.f;
      } else if (nonnull > 0) {
        double sum = 0;
        for (int r = 0; r <= 64; ++r) sum += hist[r] * ldexp(1.0, -r);
        const double m = kHllM;
        double e = (0.7213 / (1.0 + 1.079 / m)) * m * m / sum;
        if (e <= 2.5 * m && hist[0] > 0) e = m * log(m / hist[0]);
        v = static_cast<float>(fmin(1.0, e / nonnull));
      }
      f[tid] = v;
    }
    __syncthreads();
    if (tid < kHid) {
      float acc = __bfloat162float(w[kOffB1 + tid]);
      for (int i = 0; i < kIn; ++i) acc = fmaf(f[i], __bfloat162float(w[kOffW1 + tid * kIn + i]), acc);
      h1[tid] = fmaxf(acc, 0.f);
    }
    __syncthreads();
    if (tid < kHid) {
      float acc = __bfloat162float(w[kOffB2 + tid]);
      for (int i = 0; i < kHid; ++i) acc = fmaf(h1[i], __bfloat162float(w[kOffW2 + tid * kHid + i]), acc);
      h2[tid] = fmaxf(acc, 0.f);
    }
    __syncthreads();
    if (tid < kOut) {
      float acc = __bfloat162float(w[kOffB3 + tid]);
      for (int i = 0; i < kHid; ++i) acc = fmaf(h2[i], __bfloat162float(w[kOffW3 + tid * kHid + i]), acc);
      P.out->net[tid] = acc;
    }
  }
  if (tid < 66) P.out->hist[tid] = hist[tid];
  if (tid < 12) P.out->top[tid] = top[tid];
  if (tid == 0) {
    P.out->f2 = f2;
    P.out->rows = rows;
    P.out->nulls = nulls;
  }
}

__global__ void __launch_bounds__(kSketchThreads) sketch_kernel(const SketchK P) {
  extern __shared__ uint32_t sh[];
  uint32_t* hll = sh;                                  // kHllM
  uint32_t* cms = hll + kHllM;                         // kCmsDepth * kCmsWidth
  unsigned long long* ck = reinterpret_cast<unsigned long long*>(cms + kCmsDepth * kCmsWidth);
  uint32_t* cc = reinterpret_cast<uint32_t*>(ck + kCandLocal);
  for (int i = threadIdx.x; i < kHllM + kCmsDepth * kCmsWidth; i += blockDim.x) sh[i] = 0;
  for (int i = threadIdx.x; i < kCandLocal; i += blockDim.x) {
    ck[i] = 0;
    cc[i] = 0;
  }
  __shared__ unsigned long long s_rows, s_nulls;
  if (threadIdx.x == 0) s_rows = s_nulls = 0;
  __syncthreads();
  unsigned long long rows = 0, nulls = 0;
  constexpr int kBlocks = kSketchThreads / kSampleBlock;  // sample blocks per CTA at a time
  for (uint64_t b = blockIdx.x * static_cast<uint64_t>(kBlocks) + threadIdx.x / kSampleBlock; b < P.nblocks;
       b += gridDim.x * static_cast<uint64_t>(kBlocks)) {
    const uint64_t i = b * P.stride + threadIdx.x % kSampleBlock;
    if (i >= P.nrows) continue;
    uint64_t p = i;
    if (P.sel) {
      p = P.sel[i];
      if (p >= P.len) {
        atomicOr(P.err, kDevBadInput);
        continue;
      }
    }
    ++rows;
    if (!col_valid(P.key, p)) {
      ++nulls;
      continue;
    }
    const uint64_t w = key_word(P.key, p);
    const uint64_t h = sketch_hash(w);
    const uint32_t idx = static_cast<uint32_t>(h >> (64 - kHllP));
    const uint64_t rest = (h << kHllP) | (1ull << (kHllP - 1));
    const uint32_t rho = static_cast<uint32_t>(__clzll(static_cast<long long>(rest))) + 1;
    atomicMax(&hll[idx], rho);
#pragma unroll
    for (int d = 0; d < kCmsDepth; ++d) {
      const uint32_t c = static_cast<uint32_t>(mix64(h + 0x9E3779B97F4A7C15ull * (d + 1)) >> 40) & (kCmsWidth - 1);
      atomicAdd(&cms[d * kCmsWidth + c], 1u);
    }
    // First-come candidate table: a key seen early and often stays resident.
    uint32_t s = static_cast<uint32_t>(h) & (kCandLocal - 1);
    const unsigned long long kk = w + 1;  // 0 marks an empty candidate slot
    for (int t = 0; t < 8; ++t) {
      unsigned long long cur = ck[s];
      if (cur == 0) cur = atomicCAS(&ck[s], 0ull, kk);
      if (cur == 0 || cur == kk) {
        atomicAdd(&cc[s], 1u);
        break;
      }
      s = (s + 1) & (kCandLocal - 1);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    rows += __shfl_down_sync(0xffffffffu, rows, o);
    nulls += __shfl_down_sync(0xffffffffu, nulls, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&s_rows, rows);
    atomicAdd(&s_nulls, nulls);
  }
  __syncthreads();
  // Every CTA starts at its own place: all of them adding to the same words in
  // the same order would queue up at the L2.
  const unsigned turn = blockIdx.x * 1664u;
  for (int k = threadIdx.x; k < kHllM; k += blockDim.x) {
    const unsigned i = (k + turn) & (kHllM - 1);
    if (hll[i]) atomicMax(&P.hll[i], hll[i]);
  }
  for (int k = threadIdx.x; k < kCmsDepth * kCmsWidth; k += blockDim.x) {
    const unsigned i = (k + turn) & (kCmsDepth * kCmsWidth - 1);
    if (cms[i]) atomicAdd(&P.cms[i], cms[i]);
  }
  for (int i = threadIdx.x; i < kCandLocal; i += blockDim.x) {
    if (cc[i] < 2) continue;
    const unsigned long long kk = ck[i];
    uint32_t s = static_cast<uint32_t>(mix64(kk)) & (kCandGlobal - 1);
    for (int t = 0; t < 32; ++t) {
      unsigned long long cur = atomicCAS(&P.cand_key[s], 0ull, kk);
      if (cur == 0 || cur == kk) {
        atomicAdd(&P.cand_cnt[s], static_cast<unsigned long long>(cc[i]));
        break;
      }
      s = (s + 1) & (kCandGlobal - 1);
    }
  }
  if (threadIdx.x == 0) {
    atomicAdd(&P.stats[0], s_rows);
    atomicAdd(&P.stats[1], s_nulls);
  }
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(P.done, 1u) + 1 == gridDim.x;
  __syncthreads();
  if (!last) return;
  __threadfence();
  sketch_finish(P, sh);
}

// Exact counts of the sampled keys (the heavy-hitter candidates of a GROUP BY
// are the sample's most frequent keys): a linear-probing table of key words
// (0 = empty; key word 0 has a side row in the aggregation and is skipped)
// and counts, over the same strided sample blocks as sketch_kernel.
constexpr int kHeavyBins = 4096;

struct HeavyK {
  DevCol key;
  const uint32_t* sel;
  uint64_t nrows, len, stride, nblocks;
  unsigned long long* keys;  // [cap]
  unsigned int* cnt;         // [cap]
  uint64_t cap;              // power of two, >= 2 x the sampled rows
  unsigned int* hist;        // [kHeavyBins] keys per count (the last bin: >= kHeavyBins - 1)
  unsigned long long* out;   // [2 * out_cap] (key, count) of the kept keys
  unsigned int* nout;
  uint32_t out_cap, min_count;
  uint32_t* err;
};

__global__ void __launch_bounds__(kSampleBlock) heavy_count_kernel(const HeavyK P) {
  for (uint64_t b = blockIdx.x; b < P.nblocks; b += gridDim.x) {
    const uint64_t i = b * P.stride + threadIdx.x;
    if (i >= P.nrows) continue;
    uint64_t p = i;
    if (P.sel) {
      p = P.sel[i];
      if (p >= P.len) continue;  // reported by sketch_kernel
    }
    if (!col_valid(P.key, p)) continue;
    const uint64_t w = key_word(P.key, p);
    if (w == 0) continue;
    uint64_t s = mix64(w ^ 0x3C6EF372FE94F82Bull) & (P.cap - 1);
    for (uint64_t t = 0; t < P.cap; ++t) {  // at most half full: ends at a free slot
      unsigned long long cur = P.keys[s];
      if (cur == 0) cur = atomicCAS(P.keys + s, 0ull, static_cast<unsigned long long>(w));
      if (cur == 0 || cur == w) {
        atomicAdd(P.cnt + s, 1u);
        break;
      }
      s = (s + 1) & (P.cap - 1);
    }
  }
}

__global__ void heavy_hist_kernel(const HeavyK P) {
  __shared__ unsigned int h[kHeavyBins];
  for (int b = threadIdx.x; b < kHeavyBins; b += blockDim.x) h[b] = 0;
  __syncthreads();
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < P.cap; s += (uint64_t)gridDim.x * blockDim.x) {
    const unsigned int c = P.cnt[s];
    if (c) atomicAdd(&h[min(c, kHeavyBins - 1u)], 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < kHeavyBins; b += blockDim.x)
    if (h[b]) atomicAdd(P.hist + b, h[b]);
}

__global__ void heavy_compact_kernel(const HeavyK P) {
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < P.cap; s += (uint64_t)gridDim.x * blockDim.x) {
    const unsigned int c = P.cnt[s];
    if (c < P.min_count) continue;
    const unsigned int o = atomicAdd(P.nout, 1u);
    if (o < P.out_cap) {
      P.out[2 * o] = P.keys[s];
      P.out[2 * o + 1] = c;
    }
  }
}

// HyperLogLog estimate from the number of registers of each value.
double hll_estimate(const uint32_t (&regs)[66]) {
  const double m = kHllM;
  double sum = 0;
  for (int r = 0; r <= 64; ++r) sum += regs[r] * std::ldexp(1.0, -r);
  const uint32_t zeros = regs[0];
  const double alpha = 0.7213 / (1.0 + 1.079 / m);
  double e = alpha * m * m / sum;
  if (e <= 2.5 * m && zeros > 0) e = m * std::log(m / zeros);  // linear counting
  return e;
}

// Sample blocks of kSampleBlock rows, `stride` rows apart, of about
// `sample_target` rows in all.
void sample_blocks(uint64_t nrows, uint64_t sample_target, uint64_t& stride, uint64_t& nblocks) {
  const uint64_t target_blocks = std::max<uint64_t>(1, sample_target / kSampleBlock);
  stride = kSampleBlock;
  nblocks = (nrows + kSampleBlock - 1) / kSampleBlock;
  if (nblocks > target_blocks) {
    stride = ((nrows / target_blocks) / kSampleBlock) * kSampleBlock;
    if (stride < kSampleBlock) stride = kSampleBlock;
    nblocks = (nrows + stride - 1) / stride;
  }
}

}  // namespace

void sketch_key_column(qeg_ctx* ctx, const DevCol& key, const uint32_t* sel, uint64_t nrows, uint64_t len,
                       uint64_t sample_target, SketchResult& out) {
  out = SketchResult{};
  out.total_rows = static_cast<double>(nrows);
  uint64_t stride, nblocks;
  sample_blocks(nrows, sample_target, stride, nblocks);
  // Rows of the sample blocks: all but the last are whole.
  uint64_t sampled = 0;
  if (nblocks > 0) {
    const uint64_t whole = nrows >= kSampleBlock ? std::min(nblocks, (nrows - kSampleBlock) / stride + 1) : 0;
    sampled = whole * kSampleBlock + (whole < nblocks ? nrows - whole * stride : 0);
  }
  SketchOut o{};
  o.hist[0] = kHllM;  // (no rows: an empty sketch)
  out.have_net = false;
  const double log_rows = std::log2(1.0 + static_cast<double>(sampled)) / 32.0;
  const double log_total = std::log2(1.0 + out.total_rows) / 32.0;
  const double share = out.total_rows > 0 ? static_cast<double>(sampled) / out.total_rows : 1.0;
  if (nblocks > 0) {
    const size_t words = kHllM + kCmsDepth * kCmsWidth;
    static_assert(sizeof(SketchOut) % 8 == 0, "copied in words");
    const size_t head = words * 4 + kCandGlobal * 16 + 24;
    DevBuf buf(head + sizeof(SketchOut), ctx->stream);
    QEG_CUDA(cudaMemsetAsync(buf.get(), 0, head, ctx->stream));
    SketchK P{};
    P.key = key;
    P.sel = sel;
    P.nrows = nrows;
    P.len = len;
    P.stride = stride;
    P.nblocks = nblocks;
    P.hll = buf.get<uint32_t>();
    P.cms = P.hll + kHllM;
    P.cand_key = reinterpret_cast<unsigned long long*>(P.cms + kCmsDepth * kCmsWidth);
    P.cand_cnt = P.cand_key + kCandGlobal;
    P.stats = P.cand_cnt + kCandGlobal;
    P.done = reinterpret_cast<unsigned int*>(P.stats + 2);
    P.out = reinterpret_cast<SketchOut*>(P.stats + 3);
    P.net = ctx->mlp && ctx->mlp->loaded ? ctx->mlp->wbf.get<__nv_bfloat16>() : nullptr;
    P.log_rows = static_cast<float>(log_rows);
    P.log_total = static_cast<float>(log_total);
    P.sampled = static_cast<float>(share);
    P.err = static_cast<uint32_t*>(ctx->dev_err.get());
    const size_t sb = words * 4 + kCandLocal * 12;
    raise_dynamic_smem(reinterpret_cast<const void*>(sketch_kernel), sb);
    constexpr uint64_t kPer = kSketchThreads / kSampleBlock;
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>((nblocks + kPer - 1) / kPer, ctx->sms));
    sketch_kernel<<<grid, kSketchThreads, sb, ctx->stream>>>(P);
    ctx->launches++;
    QEG_CUDA(cudaGetLastError());
    read_words_and_error(ctx, P.out, sizeof(SketchOut) / 8, reinterpret_cast<uint64_t*>(&o));
    out.have_net = P.net != nullptr;
    out.net[0] = o.net[0];
    out.net[1] = o.net[1];
  }

  out.sample_rows = static_cast<double>(o.rows);
  const double nulls = static_cast<double>(o.nulls);
  out.null_frac = out.sample_rows > 0 ? nulls / out.sample_rows : 0;
  const double nonnull = out.sample_rows - nulls;
  out.hll_estimate = nonnull > 0 ? hll_estimate(o.hist) : 0;

  // Features: 64 normalised HLL register-value bins, then 16 frequency features.
  float* f = out.features;
  for (int i = 0; i < kSketchFeatures; ++i) f[i] = 0;
  for (uint32_t r = 0; r <= 64; ++r) f[std::min<uint32_t>(r, 63)] += static_cast<float>(o.hist[r]) / kHllM;
  for (int i = 0; i < 12; ++i)
    out.top_share[i] = nonnull > 0 ? std::min(1.0, static_cast<double>(o.top[i]) / nonnull) : 0;
  for (int i = 0; i < 10; ++i) f[64 + i] = static_cast<float>(out.top_share[i]);
  f[74] = nonnull > 0 ? static_cast<float>(static_cast<double>(o.f2) / (nonnull * nonnull)) : 0.f;
  f[75] = static_cast<float>(log_rows);
  f[76] = static_cast<float>(log_total);
  f[77] = static_cast<float>(share);
  f[78] = static_cast<float>(out.null_frac);
  f[79] = nonnull > 0 ? static_cast<float>(std::min(1.0, out.hll_estimate / nonnull)) : 0.f;
}

// Heavy hitters: the sample's `want` most frequent keys, by exact counts.
std::vector<uint64_t> sample_heavy(qeg_ctx* ctx, const DevCol& key, const uint32_t* sel, uint64_t nrows, uint64_t len,
                                   uint64_t sample_target, int want) {
  std::vector<uint64_t> out;
  uint64_t stride, nblocks;
  sample_blocks(nrows, sample_target, stride, nblocks);
  if (nblocks == 0) return out;
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(nblocks, ctx->sms * 8ull));
  HeavyK H{};
  H.key = key;
  H.sel = sel;
  H.nrows = nrows;
  H.len = len;
  H.stride = stride;
  H.nblocks = nblocks;
  H.cap = 1;
  while (H.cap < 2 * nblocks * kSampleBlock) H.cap <<= 1;
  H.out_cap = static_cast<uint32_t>(4 * want);
  const size_t head = H.cap * 12 + kHeavyBins * 4 + 16;
  DevBuf hb(head + static_cast<size_t>(H.out_cap) * 16, ctx->stream);
  QEG_CUDA(cudaMemsetAsync(hb.get(), 0, head, ctx->stream));
  H.keys = hb.get<unsigned long long>();
  H.cnt = reinterpret_cast<unsigned int*>(H.keys + H.cap);
  H.hist = H.cnt + H.cap;
  H.nout = H.hist + kHeavyBins;
  H.out = reinterpret_cast<unsigned long long*>(hb.get<uint8_t>() + head);
  H.err = static_cast<uint32_t*>(ctx->dev_err.get());
  heavy_count_kernel<<<grid, kSampleBlock, 0, ctx->stream>>>(H);
  heavy_hist_kernel<<<grid_for(ctx, H.cap, 256, 4), 256, 0, ctx->stream>>>(H);
  std::vector<uint32_t> hist(kHeavyBins);
  QEG_CUDA(cudaMemcpyAsync(hist.data(), H.hist, kHeavyBins * 4, cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  // The smallest count threshold that keeps at most out_cap keys (whole bins
  // only, so the kept set does not depend on the order of the atomics; the
  // top bin holds at most sample/(kHeavyBins-1) keys, fewer than out_cap).
  uint64_t kept = 0;
  uint32_t c = kHeavyBins - 1;
  while (c > 1 && kept + hist[c] <= H.out_cap) kept += hist[c--];
  if (c == 1 && kept + hist[1] <= H.out_cap) c = 0;
  H.min_count = c + 1;
  heavy_compact_kernel<<<grid_for(ctx, H.cap, 256, 4), 256, 0, ctx->stream>>>(H);
  ctx->launches += 3;
  QEG_CUDA(cudaGetLastError());
  uint32_t n = 0;
  QEG_CUDA(cudaMemcpyAsync(&n, H.nout, 4, cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  n = std::min(n, H.out_cap);
  std::vector<unsigned long long> kc(2 * static_cast<size_t>(n));
  if (n) {
    QEG_CUDA(cudaMemcpyAsync(kc.data(), H.out, kc.size() * 8, cudaMemcpyDeviceToHost, ctx->stream));
    QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  std::vector<std::pair<uint64_t, uint64_t>> top(n);
  for (uint32_t i = 0; i < n; ++i) top[i] = {kc[2 * i + 1], kc[2 * i]};
  std::sort(top.begin(), top.end(), [](const auto& a, const auto& b) {
    return a.first != b.first ? a.first > b.first : a.second < b.second;
  });
  const size_t nh = std::min<size_t>(top.size(), static_cast<size_t>(want));
  for (size_t i = 0; i < nh; ++i) out.push_back(top[i].second);
  return out;
}

// ---------------------------------------------------------------------------
// Batched sketch: one CTA per query of a batch (qeg_batch.cu). The CTA walks
// the query's whole sample (the same strided 256-row sample blocks as
// sketch_key_column), builds HyperLogLog registers, the count-min sketch and a
// first-come candidate table in shared memory, and computes the 80 features
// itself, so planning a batch costs one launch and one small copy back.
// ---------------------------------------------------------------------------
namespace {

constexpr int kBSThreads = 1024;
constexpr int kBSCand = 2048;

struct BatchSketchOut {
  float f[kSketchFeatures];
  double hll, rows, nulls;
  double top[12];
};

struct BatchSketchK {
  DevCol key;
  const uint64_t* offs;  // nq + 1 row offsets
  uint64_t sample_target;
  BatchSketchOut* out;
};

__global__ void __launch_bounds__(kBSThreads) batch_sketch_kernel(const BatchSketchK P) {
  extern __shared__ uint32_t sh[];
  uint32_t* hll = sh;                                                   // kHllM
  uint32_t* cms = hll + kHllM;                                          // kCmsDepth * kCmsWidth
  unsigned long long* ck = reinterpret_cast<unsigned long long*>(cms + kCmsDepth * kCmsWidth);  // kBSCand
  uint32_t* cc = reinterpret_cast<uint32_t*>(ck + kBSCand);             // kBSCand
  __shared__ unsigned long long s_rows, s_nulls;
  __shared__ uint32_t s_hist[64];
  __shared__ unsigned long long s_bucket[12];
  __shared__ double s_sum, s_f2;
  __shared__ uint32_t s_zeros;
  const int tid = threadIdx.x;
  for (int i = tid; i < kHllM + kCmsDepth * kCmsWidth; i += blockDim.x) sh[i] = 0;
  for (int i = tid; i < kBSCand; i += blockDim.x) {
    ck[i] = 0;
    cc[i] = 0;
  }
  if (tid < 64) s_hist[tid] = 0;
  if (tid < 12) s_bucket[tid] = 0;
  if (tid == 0) {
    s_rows = s_nulls = 0;
    s_sum = s_f2 = 0;
    s_zeros = 0;
  }
  __syncthreads();

  const uint64_t base = P.offs[blockIdx.x];
  const uint64_t n = P.offs[blockIdx.x + 1] - base;
  const uint64_t target_blocks = P.sample_target / kSampleBlock > 0 ? P.sample_target / kSampleBlock : 1;
  uint64_t stride = kSampleBlock;
  uint64_t nblocks = (n + kSampleBlock - 1) / kSampleBlock;
  if (nblocks > target_blocks) {
    stride = ((n / target_blocks) / kSampleBlock) * kSampleBlock;
    if (stride < kSampleBlock) stride = kSampleBlock;
    nblocks = (n + stride - 1) / stride;
  }
  unsigned long long rows = 0, nulls = 0;
  for (uint64_t j = tid; j < nblocks * kSampleBlock; j += blockDim.x) {
    const uint64_t i = (j / kSampleBlock) * stride + (j % kSampleBlock);
    if (i >= n) continue;
    const uint64_t p = base + i;
    ++rows;
    if (!col_valid(P.key, p)) {
      ++nulls;
      continue;
    }
    const uint64_t w = key_word(P.key, p);
    const uint64_t h = sketch_hash(w);
    const uint32_t idx = static_cast<uint32_t>(h >> (64 - kHllP));
    const uint64_t rest = (h << kHllP) | (1ull << (kHllP - 1));
    const uint32_t rho = static_cast<uint32_t>(__clzll(static_cast<long long>(rest))) + 1;
    atomicMax(&hll[idx], rho);
#pragma unroll
    for (int d = 0; d < kCmsDepth; ++d) {
      const uint32_t c = static_cast<uint32_t>(mix64(h + 0x9E3779B97F4A7C15ull * (d + 1)) >> 40) & (kCmsWidth - 1);
      atomicAdd(&cms[d * kCmsWidth + c], 1u);
    }
    uint32_t s = static_cast<uint32_t>(h) & (kBSCand - 1);
    const unsigned long long kk = w + 1;
    for (int t = 0; t < 8; ++t) {
      unsigned long long cur = ck[s];
      if (cur == 0) cur = atomicCAS(&ck[s], 0ull, kk);
      if (cur == 0 || cur == kk) {
        atomicAdd(&cc[s], 1u);
        break;
      }
      s = (s + 1) & (kBSCand - 1);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    rows += __shfl_down_sync(0xffffffffu, rows, o);
    nulls += __shfl_down_sync(0xffffffffu, nulls, o);
  }
  if ((tid & 31) == 0) {
    atomicAdd(&s_rows, rows);
    atomicAdd(&s_nulls, nulls);
  }
  __syncthreads();

  // Register histogram, HyperLogLog sum and zero count, F2 of CMS row 0.
  double hsum = 0, f2 = 0;
  uint32_t zeros = 0;
  for (int i = tid; i < kHllM; i += blockDim.x) {
    const uint32_t r = hll[i];
    atomicAdd(&s_hist[r < 63 ? r : 63], 1u);
    hsum += ldexp(1.0, -static_cast<int>(r));
    zeros += r == 0;
  }
  for (int c = tid; c < kCmsWidth; c += blockDim.x) {
    const double v = cms[c];
    f2 += v * v;
  }
  for (int o = 16; o > 0; o >>= 1) {
    hsum += __shfl_down_sync(0xffffffffu, hsum, o);
    f2 += __shfl_down_sync(0xffffffffu, f2, o);
    zeros += __shfl_down_sync(0xffffffffu, zeros, o);
  }
  if ((tid & 31) == 0) {
    atomicAdd(&s_sum, hsum);
    atomicAdd(&s_f2, f2);
    atomicAdd(&s_zeros, zeros);
  }
  // Count-min estimate of every candidate seen at least twice (0 otherwise),
  // into cc, then a descending bitonic sort of those estimates.
  for (int i = tid; i < kBSCand; i += blockDim.x) {
    uint32_t est = 0;
    if (cc[i] >= 2) {
      const uint64_t h = sketch_hash(ck[i] - 1);
      est = UINT32_MAX;
#pragma unroll
      for (int d = 0; d < kCmsDepth; ++d) {
        const uint32_t c = static_cast<uint32_t>(mix64(h + 0x9E3779B97F4A7C15ull * (d + 1)) >> 40) & (kCmsWidth - 1);
        est = min(est, cms[d * kCmsWidth + c]);
      }
    }
    cc[i] = est;
  }
  __syncthreads();
  for (int k = 2; k <= kBSCand; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < kBSCand; i += blockDim.x) {
        const int x = i ^ j;
        if (x > i) {
          const uint32_t a = cc[i], b = cc[x];
          if (((i & k) == 0) ? (a < b) : (a > b)) {
            cc[i] = b;
            cc[x] = a;
          }
        }
      }
      __syncthreads();
    }
  }
  // Sum of the top 2^b estimates: the estimate at sorted position j counts
  // toward every prefix longer than j, i.e. bucket bitlength(j) and above.
  for (int j = tid; j < kBSCand; j += blockDim.x) {
    const int b = j == 0 ? 0 : 32 - __clz(j);
    if (b < 12 && cc[j]) atomicAdd(&s_bucket[b], static_cast<unsigned long long>(cc[j]));
  }
  __syncthreads();
  if (tid == 0) {
    BatchSketchOut& o = P.out[blockIdx.x];
    const double srows = static_cast<double>(s_rows), snulls = static_cast<double>(s_nulls);
    const double nonnull = srows - snulls;
    const double m = kHllM;
    double e = (0.7213 / (1.0 + 1.079 / m)) * m * m / s_sum;
    if (e <= 2.5 * m && s_zeros > 0) e = m * log(m / s_zeros);
    o.hll = nonnull > 0 ? e : 0;
    o.rows = srows;
    o.nulls = snulls;
    for (int i = 0; i < kSketchFeatures; ++i) o.f[i] = 0;
    for (int r = 0; r < 64; ++r) o.f[r] = static_cast<float>(s_hist[r]) / kHllM;
    double cum = 0;
    for (int i = 0; i < 12; ++i) {
      cum += static_cast<double>(s_bucket[i]);
      o.top[i] = nonnull > 0 ? fmin(1.0, cum / nonnull) : 0;
    }
    for (int i = 0; i < 10; ++i) o.f[64 + i] = static_cast<float>(o.top[i]);
    o.f[74] = nonnull > 0 ? static_cast<float>(s_f2 / (nonnull * nonnull)) : 0.f;
    o.f[75] = static_cast<float>(log2(1.0 + srows) / 32.0);
    o.f[76] = static_cast<float>(log2(1.0 + static_cast<double>(n)) / 32.0);
    o.f[77] = n > 0 ? static_cast<float>(srows / static_cast<double>(n)) : 1.f;
    o.f[78] = srows > 0 ? static_cast<float>(snulls / srows) : 0.f;
    o.f[79] = nonnull > 0 ? static_cast<float>(fmin(1.0, o.hll / nonnull)) : 0.f;
  }
}

}  // namespace

void batch_sketch(qeg_ctx* ctx, const DevCol& key, const uint64_t* d_offsets, const std::vector<uint64_t>& offsets,
                  uint64_t sample_target, std::vector<SketchResult>& out) {
  const uint32_t nq = static_cast<uint32_t>(offsets.size() - 1);
  out.assign(nq, SketchResult{});
  if (nq == 0) return;
  DevBuf buf(static_cast<size_t>(nq) * sizeof(BatchSketchOut), ctx->stream);
  BatchSketchK P{};
  P.key = key;
  P.offs = d_offsets;
  P.sample_target = sample_target;
  P.out = buf.get<BatchSketchOut>();
  const size_t sb = (kHllM + kCmsDepth * kCmsWidth) * 4 + kBSCand * 12;
  raise_dynamic_smem(reinterpret_cast<const void*>(batch_sketch_kernel), sb);
  batch_sketch_kernel<<<nq, kBSThreads, sb, ctx->stream>>>(P);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
  std::vector<BatchSketchOut> h(nq);
  QEG_CUDA(cudaMemcpyAsync(h.data(), buf.get(), nq * sizeof(BatchSketchOut), cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  check_device_error(ctx);
  for (uint32_t q = 0; q < nq; ++q) {
    SketchResult& r = out[q];
    std::copy(h[q].f, h[q].f + kSketchFeatures, r.features);
    r.hll_estimate = h[q].hll;
    r.sample_rows = h[q].rows;
    r.total_rows = static_cast<double>(offsets[q + 1] - offsets[q]);
    r.null_frac = h[q].rows > 0 ? h[q].nulls / h[q].rows : 0;
    for (int i = 0; i < 12; ++i) r.top_share[i] = h[q].top[i];
  }
}

double classic_estimate(const SketchResult& s) {
  // Distinct count of the sample from HyperLogLog, scaled to the population by
  // inverting E[d_sample] = D (1 - (1 - 1/D)^m) (a uniform-frequency model),
  // plus the NULL group. Skewed data breaks the uniform model; that is what the
  // learned estimator corrects.
  const double nonnull_rows = s.total_rows * (1.0 - s.null_frac);
  const double m = s.sample_rows * (1.0 - s.null_frac);
  double d = s.hll_estimate;
  if (m <= 0) return s.null_frac > 0 ? 1.0 : 0.0;
  if (s.sample_rows < s.total_rows && d > 0) {
    if (d >= m * 0.999) {
      d = nonnull_rows;  // every sampled row distinct: assume all distinct
    } else {
      double lo = d, hi = std::max(d, nonnull_rows);
      for (int it = 0; it < 100; ++it) {
        const double mid = 0.5 * (lo + hi);
        const double e = mid * (1.0 - std::exp(m * std::log1p(-1.0 / std::max(mid, 1.0 + 1e-9))));
        if (e < d) lo = mid;
        else hi = mid;
      }
      d = 0.5 * (lo + hi);
    }
  }
  d = std::min(d, nonnull_rows);
  return d + (s.null_frac > 0 ? 1.0 : 0.0);
}

double AggState::estimate_groups(const std::vector<StagedCol>& staged, uint64_t nrows, uint64_t len,
                                 const uint32_t* dsel) {
  if (mode != 1 || nrows == 0) {
    // Composite keys: bounded by the row count (grown on overflow).
    return static_cast<double>(std::min<uint64_t>(std::max<uint64_t>(nrows, 1), 1ull << 22));
  }
  SketchResult s;
  if (packed && bucket_width > 0) {
    // A packed window's (partition key, bucket) words are clustered by time,
    // which a strided sample cannot extrapolate: estimate the partition key's
    // distinct count instead and multiply by the buckets the time range
    // spans (at most one group per row).
    sketch_key_column(ctx, staged[keys[0]].dev, dsel, nrows, len, 1u << 20, s);
    double keys_est = 0, share = 0;
    if (!learned_estimate(ctx, s, &keys_est, &share)) keys_est = classic_estimate(s);
    hot_share = 0;
    const double buckets = static_cast<double>(pack_qmax - pack_qmin + 1);
    return std::max(1.0, std::min(static_cast<double>(nrows), std::max(keys_est, 1.0) * buckets));
  }
  sketch_key_column(ctx, key_col(staged, 0), dsel, nrows, len, 1u << 20, s);
  double groups = 0, share = 0;
  if (learned_estimate(ctx, s, &groups, &share)) {
    hot_share = share;
  } else {
    groups = classic_estimate(s);
    hot_share = s.top_share[11];
  }
  return std::max(groups, 1.0);
}

// The most frequent keys of a sample of the batch, most frequent first.
void AggState::find_heavy(const std::vector<StagedCol>& staged, uint64_t nrows, uint64_t len, const uint32_t* dsel) {
  heavy_candidates = sample_heavy(ctx, key_col(staged, 0), dsel, nrows, len, 1u << 20, 4096);
}

}  // namespace qeg
