// Loading a dense weight: host memory -> NVFP4 codes, DEVICE-layout scales and bias on the GPU in one call, where the reference uploads and
// prepares a weight (WeightPrep, thinfer-core/src/backend/mod.rs:65-90, thinfer-core/src/ops/weight_prep.rs:86-163).
#include <algorithm>

#include "context.h"

using namespace tnf;

namespace {
// Staging that stays for the next load. With a budget, which may be planned to the byte, every load makes and frees its own.
constexpr uint64_t kKeptStaging = 160u << 20;

struct Staging {
  tnf_ctx* ctx;
  uint64_t id = 0;
  bool kept = false;  // the context's, taken until this goes
  explicit Staging(tnf_ctx* c) : ctx(c) {}
  int32_t make(uint64_t bytes, uint8_t** p) {
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (!ctx->budget && bytes <= kKeptStaging && !ctx->load_busy) {
      if (bytes > ctx->load_stage_bytes) {
        if (ctx->load_stage_id) free_locked(ctx, ctx->load_stage_id);
        ctx->load_stage_id = ctx->load_stage_bytes = 0;
        const int32_t st = alloc_locked(ctx, bytes, TNF_CAT_STAGING, &ctx->load_stage_id);
        if (st != TNF_OK) return st;
        ctx->load_stage_bytes = bytes;
      }
      ctx->load_busy = kept = true;
      id = ctx->load_stage_id;
    } else {
      const int32_t st = alloc_locked(ctx, bytes, TNF_CAT_STAGING, &id);
      if (st != TNF_OK) return st;
    }
    *p = static_cast<uint8_t*>(ctx->bufs.at(id).ptr);
    return TNF_OK;
  }
  ~Staging() {
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (kept) ctx->load_busy = false;
    else if (id) free_locked(ctx, id);
  }
};
}  // namespace

extern "C" int32_t tnf_load_weight(tnf_ctx* ctx, const void* w_host, int32_t src_dtype, uint32_t n, uint32_t k, const uint16_t* bias_host,
                                   uint64_t* codes_id, uint64_t* scales_id, uint64_t* bias_id, float* global_scale) {
  if (!ctx || !w_host || !codes_id || !scales_id || !global_scale || (bias_host && !bias_id) || n == 0 || k == 0 || k % 32 != 0 ||
      (src_dtype != TNF_DTYPE_F32 && src_dtype != TNF_DTYPE_BF16)) {
    set_error("tnf_load_weight: null argument, or n=%u k=%u (k %% 32 == 0) dtype=%d", n, k, src_dtype);
    return TNF_ERR_INVALID_ARGUMENT;
  }
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
  const uint64_t src_bytes = uint64_t(n) * k * (src_dtype == TNF_DTYPE_BF16 ? 2 : 4);
  const uint64_t bytes[3] = {uint64_t(n) * (k / 2), sf_device_bytes(n, k), std::max<uint64_t>(uint64_t(n) * 2, 16)};
  const int made = bias_host ? 3 : 2;
  uint64_t ids[3] = {0, 0, 0};
  uint8_t* ptr[3] = {nullptr, nullptr, nullptr};
  int32_t st = TNF_OK;
  {
    Staging staging(ctx);
    uint8_t* src = nullptr;
    st = staging.make(src_bytes, &src);
    if (st == TNF_OK) {
      std::lock_guard<std::mutex> lk(ctx->mu);
      for (int i = 0; i < made && st == TNF_OK; ++i) {
        st = alloc_locked(ctx, bytes[i], TNF_CAT_WEIGHTS, &ids[i]);
        if (st == TNF_OK) ptr[i] = static_cast<uint8_t*>(ctx->bufs.at(ids[i]).ptr);
      }
    }
    if (st == TNF_OK) {
      if (bias_host) e = cudaMemcpyAsync(ptr[2], bias_host, uint64_t(n) * 2, cudaMemcpyHostToDevice, ctx->compute);
      if (e == cudaSuccess) e = write_host(ctx, src, static_cast<const uint8_t*>(w_host), src_bytes);  // waits: the bias has been read, too
      if (e != cudaSuccess) st = cuda_fail(e, "tnf_load_weight copy");
      else st = quantize_own_scale(ctx, src, src_dtype, n, k, true, ptr[0], ptr[1], global_scale);  // waits: the staging is free again
    }
  }
  if (st != TNF_OK) {
    std::lock_guard<std::mutex> lk(ctx->mu);
    for (uint64_t id : ids)
      if (id) free_locked(ctx, id);
    return st;
  }
  *codes_id = ids[0];
  *scales_id = ids[1];
  if (bias_id) *bias_id = ids[2];
  return TNF_OK;
}
