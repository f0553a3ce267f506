// qeg_ctx.cu -- context, staging of host inputs, result fetch, device error word.
#include <mutex>

#include "qeg_internal.h"

thread_local std::string g_qeg_tls_err;

namespace qeg {

namespace {

// Output columns of one fetch (qeg::fetch_columns): at most every key and
// aggregate of a GROUP BY.
struct FetchK {
  const uint8_t* vals[kMaxFetchCols];
  const uint8_t* valid[kMaxFetchCols];
  uint8_t* dst[kMaxFetchCols];      // nullptr: the values go by a copy of their own, or are not wanted
  uint64_t* words[kMaxFetchCols];   // nullptr: no validity words wanted
  uint32_t* null_flags;          // page-locked host memory, one per column, zeroed: 1 when it holds a NULL
  uint64_t count;
  uint8_t width[kMaxFetchCols];
  uint8_t unit[kMaxFetchCols];  // bytes per copied element: 16, or at most the width, as both ends are aligned
};

// Copies `n` elements of type T.
template <typename T>
__device__ __forceinline__ void copy_elems(uint8_t* dst, const uint8_t* src, uint64_t n, uint64_t i, uint64_t step) {
#pragma unroll 4
  for (; i < n; i += step) reinterpret_cast<T*>(dst)[i] = __ldg(reinterpret_cast<const T*>(src) + i);
}

// One launch for a whole fetch, blockIdx.y = column: packs one byte per row (1
// = valid) into 64-bit validity words, LSB-first (core/validity.h:21-40;
// padding bits of the last word set, core/validity.h:53-58), and copies the
// values. Small results are bound by the launch and the synchronisation that
// follows, so the columns share both; large ones by the copy (16-byte loads
// and stores where both ends allow). Per column a copy, an allocation, a
// memset, a pack kernel, two more copies and a synchronisation took 45-55 us
// (fetch of 6 small columns: 290 us into device buffers, 330 us into host
// arrays); packing with one thread per word read the valid bytes 64 apart
// (35 us per 16.6M-row column), a warp per word reads them side by side.
__global__ void __launch_bounds__(256) fetch_kernel(const FetchK P) {
  const int c = blockIdx.y;
  const uint64_t n = P.count;
  const unsigned lane = threadIdx.x & 31u;
  uint64_t* words = P.words[c];
  const uint8_t* valid = P.valid[c];
  const uint64_t nw = (n + 63) / 64;
  bool nulls = false;
  constexpr int kU = 4;  // words per warp and step, their loads independent
  for (uint64_t w0 = (blockIdx.x * 8ull + (threadIdx.x >> 5)) * kU; w0 < nw; w0 += gridDim.x * 8ull * kU) {
    bool lo[kU], hi[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t r = (w0 + u) * 64 + lane;
      lo[u] = r >= n || valid[r] != 0;
      hi[u] = r + 32 >= n || valid[r + 32] != 0;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t bits = __ballot_sync(0xffffffffu, lo[u]) |
                            (static_cast<uint64_t>(__ballot_sync(0xffffffffu, hi[u])) << 32);
      if (w0 + u < nw) {
        nulls |= bits != ~0ull;
        if (words && lane == 0) words[w0 + u] = bits;
      }
    }
  }
  if (nulls && lane == 0) P.null_flags[c] = 1u;
  uint8_t* dst = P.dst[c];
  if (!dst) return;
  const uint8_t* src = P.vals[c];
  const uint64_t i = blockIdx.x * 256ull + threadIdx.x, step = gridDim.x * 256ull;
  const uint64_t bytes = n * P.width[c];
  const int unit = P.unit[c];
  if (unit == 16) {
    copy_elems<uint4>(dst, src, bytes / 16, i, step);
    for (uint64_t b = bytes / 16 * 16 + i; b < bytes; b += step) dst[b] = src[b];
  } else if (unit == 8) {
    copy_elems<uint64_t>(dst, src, bytes / 8, i, step);
  } else if (unit == 4) {
    copy_elems<uint32_t>(dst, src, bytes / 4, i, step);
  } else {
    copy_elems<uint8_t>(dst, src, bytes, i, step);
  }
}

// One thread waits, with the bounded wait every composite-key table uses, on
// a row state word that is claimed and never published.
__global__ void stuck_claim_kernel(uint64_t* word, int polls, uint32_t* err) {
  *word = kRowClaimed;
  __threadfence();
  wait_published(word, kRowClaimed, polls, err);
}

}  // namespace

void stage_column(qeg_ctx* ctx, const qeg_column& c, StagedCol& out) {
  require(c.type >= QEG_I32 && c.type <= QEG_STR, "unknown column type");
  out.len = c.len;
  out.dev.type = c.type;
  out.dev.all_valid = (c.all_valid || c.validity == nullptr) ? 1 : 0;
  const size_t w = type_width(c.type);
  if (c.len == 0) {
    out.dev.data = nullptr;
    out.dev.validity = nullptr;
  } else if (is_device_ptr(c.data)) {
    out.dev.data = c.data;
  } else {
    require(c.data != nullptr, "column data is NULL");
    out.data.alloc(c.len * w, ctx->stream);
    QEG_CUDA(cudaMemcpyAsync(out.data.get(), c.data, c.len * w, cudaMemcpyHostToDevice, ctx->stream));
    out.dev.data = out.data.get();
  }
  if (!out.dev.all_valid && c.len > 0) {
    const size_t vb = ((c.len + 63) / 64) * 8;
    if (is_device_ptr(c.validity)) {
      out.dev.validity = c.validity;
    } else {
      out.validity.alloc(vb, ctx->stream);
      QEG_CUDA(cudaMemcpyAsync(out.validity.get(), c.validity, vb, cudaMemcpyHostToDevice, ctx->stream));
      out.dev.validity = out.validity.get<uint64_t>();
    }
  } else {
    out.dev.validity = nullptr;
  }
  out.dev.code_map = nullptr;
  if (c.type == QEG_STR && c.code_map != nullptr && c.code_map_len > 0) {
    if (is_device_ptr(c.code_map)) {
      out.dev.code_map = c.code_map;
    } else {
      out.code_map.alloc(c.code_map_len * 4, ctx->stream);
      QEG_CUDA(cudaMemcpyAsync(out.code_map.get(), c.code_map, c.code_map_len * 4,
                               cudaMemcpyHostToDevice, ctx->stream));
      out.dev.code_map = out.code_map.get<int32_t>();
    }
  }
}

void stage_sel(qeg_ctx* ctx, const uint32_t* sel, uint64_t n, DevBuf& buf, const uint32_t** dev) {
  if (sel == nullptr || n == 0) {
    *dev = nullptr;
    return;
  }
  if (is_device_ptr(sel)) {
    *dev = sel;
    return;
  }
  buf.alloc(n * 4, ctx->stream);
  QEG_CUDA(cudaMemcpyAsync(buf.get(), sel, n * 4, cudaMemcpyHostToDevice, ctx->stream));
  *dev = buf.get<uint32_t>();
}

void check_device_error(qeg_ctx* ctx) {
  uint32_t e = 0;
  QEG_CUDA(cudaMemcpyAsync(&e, ctx->dev_err.get(), 4, cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  raise_device_error(ctx, e);
}

void read_words_and_error(qeg_ctx* ctx, const void* dev_words, size_t nwords, uint64_t* out) {
  uint8_t* pin = static_cast<uint8_t*>(ctx->pinned_in.reserve(nwords * 8 + 16));
  if (nwords)
    QEG_CUDA(cudaMemcpyAsync(pin + 16, dev_words, nwords * 8, cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaMemcpyAsync(pin, ctx->dev_err.get(), 4, cudaMemcpyDeviceToHost, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  uint32_t e;
  std::memcpy(&e, pin, 4);
  if (nwords) std::memcpy(out, pin + 16, nwords * 8);
  raise_device_error(ctx, e);
}

namespace {
// The shared-memory attribute belongs to the function (for every thread of the
// process), so it is only ever raised: the largest size set so far is kept
// per (device, kernel), and a request for more raises it. A launch of `smem`
// bytes after its own request therefore always fits, whatever other threads
// request meanwhile. The occupancy answers are cached per (device, kernel,
// block, shared bytes).
struct SmemAttr {
  const void* kern;
  int dev;
  size_t smem;
};
struct SmemOcc {
  const void* kern;
  int dev, block;
  size_t smem;
  int per_sm;
};
std::mutex g_smem_mu;
std::vector<SmemAttr> g_smem_attrs;
std::vector<SmemOcc> g_smem_occs;

void raise_locked(const void* kern, int dev, size_t smem) {
  if (smem <= 48 * 1024) return;
  SmemAttr* a = nullptr;
  for (SmemAttr& x : g_smem_attrs)
    if (x.kern == kern && x.dev == dev) a = &x;
  if (a && a->smem >= smem) return;
  QEG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  if (a) a->smem = smem;
  else g_smem_attrs.push_back(SmemAttr{kern, dev, smem});
}
}  // namespace

void raise_dynamic_smem(const void* kern, size_t smem) {
  int dev = 0;
  QEG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(g_smem_mu);
  raise_locked(kern, dev, smem);
}

int blocks_per_sm(const void* kern, int block, size_t smem) {
  int dev = 0;
  QEG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(g_smem_mu);
  raise_locked(kern, dev, smem);
  for (const SmemOcc& o : g_smem_occs)
    if (o.kern == kern && o.dev == dev && o.block == block && o.smem == smem) return o.per_sm;
  int per_sm = 0;
  QEG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem));
  g_smem_occs.push_back(SmemOcc{kern, dev, block, smem, per_sm});
  return per_sm;
}

void raise_device_error(qeg_ctx* ctx, uint32_t e) {
  if (e == kDevOk) return;
  QEG_CUDA(cudaMemsetAsync(ctx->dev_err.get(), 0, 4, ctx->stream));
  if (e & kDevSpinTimeout)
    throw Error(QEG_ERR_TIMEOUT, "a bounded device-side wait ran out (slot publication)");
  if (e & kDevBadInput)
    throw Error(QEG_ERR_INVALID, "an input index (selection or dictionary code) is out of range");
  throw Error(QEG_ERR_CUDA, "device error word " + std::to_string(e));
}

void fetch_columns(qeg_ctx* ctx, const FetchCol* cols, int ncols, uint64_t first, uint64_t count,
                   const qeg_out_column* outs) {
  require(ncols <= kMaxFetchCols, "too many output columns in one fetch");
  if (count == 0) {
    for (int c = 0; c < ncols; ++c)
      if (outs[c].all_valid) *outs[c].all_valid = 1;
    return;
  }
  const uint64_t nw = (count + 63) / 64;
  const size_t flag_bytes = static_cast<size_t>(kMaxFetchCols) * 4;
  // Where each column's values and words go. Host destinations of a small
  // result are written by the kernel into the context's page-locked buffer
  // and copied from there by the host (no device-to-host copy commands); those
  // of a large one by a copy per array, at the host link's speed when the
  // destination is page-locked. The line: a copy command into pageable memory
  // costs about 10 us of host time whatever its size, the host's own copy of
  // kSmallFetch bytes about as much in all.
  constexpr size_t kSmallFetch = 256 << 10;
  // Device words go straight to the caller when they are 8-byte aligned.
  // Memory of another device than the context's goes by copies.
  std::vector<bool> dev_data(ncols), dev_words(ncols), copy_words(ncols), far_data(ncols);
  size_t host_bytes = 0;
  for (int c = 0; c < ncols; ++c) {
    dev_data[c] = outs[c].data && is_device_ptr(outs[c].data);
    dev_words[c] = outs[c].validity && is_device_ptr(outs[c].validity);
    far_data[c] = dev_data[c] && !kernel_reaches(outs[c].data, ctx->device);
    if (outs[c].data && !dev_data[c]) host_bytes += (count * cols[c].width + 15) / 16 * 16;
    if (outs[c].validity && !dev_words[c]) host_bytes += (nw * 8 + 15) / 16 * 16;
  }
  const bool small = host_bytes <= kSmallFetch;
  bool any_copy = false;
  for (int c = 0; c < ncols; ++c) {
    copy_words[c] = outs[c].validity &&
                    (dev_words[c] ? reinterpret_cast<uintptr_t>(outs[c].validity) % 8 != 0 ||
                                        !kernel_reaches(outs[c].validity, ctx->device)
                                  : !small);
    any_copy = any_copy || copy_words[c];
  }
  uint8_t* pin = static_cast<uint8_t*>(ctx->pinned_in.reserve(flag_bytes + (small ? host_bytes : 0)));
  std::memset(pin, 0, flag_bytes);
  DevBuf staged;  // validity words that go by a copy
  if (any_copy) staged.alloc(nw * 8 * ncols, ctx->stream);
  FetchK P{};
  P.count = count;
  P.null_flags = reinterpret_cast<uint32_t*>(pin);
  std::vector<uint8_t*> pin_data(ncols, nullptr), pin_words(ncols, nullptr);
  uint8_t* at = pin + flag_bytes;
  for (int c = 0; c < ncols; ++c) {
    const size_t bytes = count * cols[c].width;
    P.vals[c] = static_cast<const uint8_t*>(cols[c].vals) + first * cols[c].width;
    P.valid[c] = cols[c].valid + first;
    P.width[c] = static_cast<uint8_t>(cols[c].width);
    if (dev_data[c] && !far_data[c]) {
      P.dst[c] = static_cast<uint8_t*>(outs[c].data);
    } else if (outs[c].data && !dev_data[c] && small) {
      P.dst[c] = pin_data[c] = at;
      at += (bytes + 15) / 16 * 16;
    } else if (outs[c].data) {
      QEG_CUDA(cudaMemcpyAsync(outs[c].data, P.vals[c], bytes, cudaMemcpyDefault, ctx->stream));
    }
    if (copy_words[c]) {
      P.words[c] = staged.get<uint64_t>() + nw * c;
    } else if (dev_words[c]) {
      P.words[c] = outs[c].validity;
    } else if (outs[c].validity) {
      pin_words[c] = at;
      P.words[c] = reinterpret_cast<uint64_t*>(at);
      at += (nw * 8 + 15) / 16 * 16;
    }
    const uintptr_t ends = reinterpret_cast<uintptr_t>(P.vals[c]) | reinterpret_cast<uintptr_t>(P.dst[c]);
    P.unit[c] = ends % 16 == 0 ? 16 : ends % cols[c].width == 0 ? P.width[c] : 1;
  }
  // About 1024 rows per block, at most eight blocks per SM over all columns.
  const uint64_t gx = std::min<uint64_t>((count + 1023) / 1024,
                                         std::max<uint64_t>(1, static_cast<uint64_t>(ctx->sms) * 8 / ncols));
  fetch_kernel<<<dim3(static_cast<unsigned>(gx), static_cast<unsigned>(ncols)), 256, 0, ctx->stream>>>(P);
  ctx->launches++;
  QEG_CUDA(cudaGetLastError());
  for (int c = 0; c < ncols; ++c)
    if (copy_words[c])
      QEG_CUDA(cudaMemcpyAsync(outs[c].validity, P.words[c], nw * 8, cudaMemcpyDefault, ctx->stream));
  QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  for (int c = 0; c < ncols; ++c) {
    if (pin_data[c]) std::memcpy(outs[c].data, pin_data[c], count * cols[c].width);
    if (pin_words[c]) std::memcpy(outs[c].validity, pin_words[c], nw * 8);
    if (outs[c].all_valid) *outs[c].all_valid = P.null_flags[c] ? 0 : 1;
  }
}

void fetch_column(qeg_ctx* ctx, const void* dev_vals, const uint8_t* dev_valid, size_t width,
                  uint64_t first, uint64_t count, const qeg_out_column& out) {
  const FetchCol col{dev_vals, dev_valid, width};
  fetch_columns(ctx, &col, 1, first, count, &out);
}

}  // namespace qeg

extern "C" {

qeg_status qeg_ctx_create(int device, qeg_ctx** out) {
  return qeg::guarded(nullptr, [&] {
    qeg::require(out != nullptr, "out is NULL");
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
      cudaGetLastError();
      throw qeg::Error(QEG_ERR_NO_DEVICE, "no CUDA device available");
    }
    qeg::require(device >= 0 && device < n, "device index out of range");
    QEG_CUDA(cudaSetDevice(device));
    auto c = std::make_unique<qeg_ctx>();
    c->device = device;
    cudaDeviceProp p{};
    QEG_CUDA(cudaGetDeviceProperties(&p, device));
    c->sms = p.multiProcessorCount;
    c->smem_optin = p.sharedMemPerBlockOptin;
    QEG_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
    // QEG_L2_FETCH_BYTES (32..128): the largest L2 fetch from DRAM on an L2
    // miss, a limit of this process's CUDA context (for measuring random
    // table reads; unset leaves the context's default).
    if (const char* e = std::getenv("QEG_L2_FETCH_BYTES")) {
      const size_t v = static_cast<size_t>(std::atoi(e));
      if (v >= 32 && v <= 128) QEG_CUDA(cudaDeviceSetLimit(cudaLimitMaxL2FetchGranularity, v));
    }
    // Keep freed stream-ordered allocations cached in this process's pool, so a
    // query's tables and scratch are re-used instead of re-mapped every call.
    cudaMemPool_t pool;
    QEG_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
    uint64_t keep = UINT64_MAX;
    QEG_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    c->dev_err.alloc(64, c->stream);
    QEG_CUDA(cudaMemsetAsync(c->dev_err.get(), 0, 64, c->stream));
    QEG_CUDA(cudaStreamSynchronize(c->stream));
    qeg::load_default_weights(c.get());
    *out = c.release();
  });
}

void qeg_ctx_destroy(qeg_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  // Every buffer owned by the context is freed on its stream: release them
  // all while the stream still exists, then destroy it.
  ctx->dev_err.release();
  ctx->mlp.reset();
  cudaStreamSynchronize(ctx->stream);
  cudaStreamDestroy(ctx->stream);
  if (ctx->side) {
    cudaStreamSynchronize(ctx->side);
    cudaStreamDestroy(ctx->side);
    cudaEventDestroy(ctx->side_in);
    cudaEventDestroy(ctx->side_out);
  }
  delete ctx;
}

const char* qeg_last_error(const qeg_ctx* ctx) {
  return ctx ? ctx->err.c_str() : g_qeg_tls_err.c_str();
}

void* qeg_ctx_stream(qeg_ctx* ctx) { return ctx ? static_cast<void*>(ctx->stream) : nullptr; }

qeg_status qeg_ctx_synchronize(qeg_ctx* ctx) {
  return qeg::guarded(ctx, [&] {
    qeg::require(ctx != nullptr, "ctx is NULL");
    qeg::check_device_error(ctx);
  });
}

uint64_t qeg_ctx_kernel_launches(const qeg_ctx* ctx) { return ctx ? ctx->launches : 0; }

qeg_status qeg_host_alloc(uint64_t bytes, void** out) {
  return qeg::guarded(nullptr, [&] {
    qeg::require(out != nullptr, "out is NULL");
    *out = nullptr;
    if (bytes == 0) return;
    const cudaError_t e = cudaHostAlloc(out, bytes, cudaHostAllocPortable);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *out = nullptr;
      throw qeg::Error(QEG_ERR_OOM, std::string("page-locked host allocation: ") + cudaGetErrorString(e));
    }
  });
}

void qeg_host_free(void* p) {
  if (p) cudaFreeHost(p);
}

qeg_status qeg_dev_alloc(qeg_ctx* ctx, uint64_t bytes, void** out) {
  return qeg::guarded(ctx, [&] {
    qeg::require(ctx != nullptr && out != nullptr, "ctx/out is NULL");
    *out = nullptr;
    if (bytes == 0) return;
    QEG_CUDA(cudaSetDevice(ctx->device));
    const cudaError_t e = cudaMalloc(out, bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *out = nullptr;
      throw qeg::Error(QEG_ERR_OOM, std::string("device allocation: ") + cudaGetErrorString(e));
    }
  });
}

qeg_status qeg_dev_upload(qeg_ctx* ctx, void* dst, const void* src, uint64_t bytes) {
  return qeg::guarded(ctx, [&] {
    qeg::require(ctx != nullptr, "ctx is NULL");
    if (bytes == 0) return;
    qeg::require(dst != nullptr && src != nullptr, "dst/src is NULL");
    qeg::require(qeg::is_device_ptr(dst), "upload destination is not device memory");
    QEG_CUDA(cudaSetDevice(ctx->device));
    QEG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
    QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  });
}

qeg_status qeg_dev_download(qeg_ctx* ctx, void* dst, const void* src, uint64_t bytes) {
  return qeg::guarded(ctx, [&] {
    qeg::require(ctx != nullptr, "ctx is NULL");
    if (bytes == 0) return;
    qeg::require(dst != nullptr && src != nullptr, "dst/src is NULL");
    qeg::require(qeg::is_device_ptr(src), "download source is not device memory");
    QEG_CUDA(cudaSetDevice(ctx->device));
    QEG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    QEG_CUDA(cudaStreamSynchronize(ctx->stream));
  });
}

void qeg_dev_free(void* p) {
  if (p) cudaFree(p);
}

qeg_status qeg_ctx_check_bounded_wait(qeg_ctx* ctx, int32_t polls) {
  return qeg::guarded(ctx, [&] {
    qeg::require(ctx != nullptr, "ctx is NULL");
    qeg::require(polls >= 0 && polls <= (1 << 20), "polls must lie in [0, 2^20]");
    qeg::DevBuf word(8, ctx->stream);
    qeg::stuck_claim_kernel<<<1, 1, 0, ctx->stream>>>(word.get<uint64_t>(), polls, ctx->dev_err.get<uint32_t>());
    ctx->launches++;
    QEG_CUDA(cudaGetLastError());
    qeg::check_device_error(ctx);
  });
}

}  // extern "C"
