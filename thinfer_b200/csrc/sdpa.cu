// Joint scaled-dot-product attention between the linears of a DiT block (op_sdpa, thinfer-core/src/ops/sdpa.rs:10-47;
// call site thinfer-models/src/qwen_image/dit.rs:618-655: full attention over [txt ++ img], has_mask = 0, D = 128):
// out = softmax(Q K^T * scale) V per (batch, head), bf16 in and out, f32 softmax statistics and accumulation.
//
// Flash-attention tiling, 128 query rows x 128 keys a tile, both products on the tensor cores (tcgen05.mma kind::f16),
// scores, probabilities and running outputs in TMEM, TWO softmax groups per CTA with nothing between them: each has a score
// tile S_g, a running output O_g and a reference maximum of its own, so that one group's exponentials run under the
// other's two products. One persistent CTA per SM; an item of its work is one of two shapes:
//   rows mode   256 query rows of one (head, batch): group g has rows 128g .. 128g+127 and all key tiles
//   keys mode   128 query rows: group g has the key tiles of parity g; the two outputs are joined at the end
// With so few blocks of 128 query rows that SMs would idle, a cluster of CTAs takes a block in keys mode, a share of the key tiles
// each, and joins the outputs through distributed shared memory (kSplit; sdpa_split in rules.h).
// Rows mode reads K and V once for 256 rows; keys mode halves an item's time, which fills the chip when there are few rows
// and shortens the last wave (sdpa_plan in rules.h says which item is which). The loads and the first scores of an item run under the
// previous one's last products and output.
//   TMEM columns 0-127 S_0, 128-255 S_1 (f32), 256-383 O_0, 384-511 O_1 (f32). P_g (bf16 pairs, 64 columns) takes the place
//   of S_g: a thread has its score row in registers before it writes the first probability.
//   warp 0      TMA: the Q tiles once, then K tiles into a two-stage ring ([128 rows x 64 bf16] boxes with 128-byte swizzle
//               straight out of the [B, S, H, D] tensors: a head is a 256-byte column window); warp 2 the same for V;
//   warp 1      one elected thread issues, for the groups in turn, O_g += P_g V_j and at once S_g = Q_g K_j'^T of the
//               group's next tile. The tensor pipe runs them in order: S_g may overwrite P_g without a wait, and a finished
//               S_g says that O_g is complete as well. Q, K: shared memory, K-major; P: tensor memory; V as it lies in
//               memory (keys x d: an MN-major B operand, no transpose pass). O_g += P_g V starts when 96 of the tile's
//               128 probabilities are written;
//   warps 4-11  the softmax groups, one query row per thread (TMEM lane = row): the row's scores to registers in one round
//               trip, p = exp2(s * scale * log2e - m), f32 row sum, bf16 pairs to P_g. m is the row maximum of the group's
//               first tile. Later tiles have no pass over the scores for their maximum: the row sum of the first 96 keys (and
//               the maximum of the last 32) tells whether a probability can have passed 2^10; only then, before anything is
//               written, is the maximum taken, m moved, O_g rescaled (tcgen05.ld / mul / tcgen05.st) and the tile redone.
// The reference's kernel is the same recurrence one key at a time in f32 (m' = max(m, s); o = o * exp(m - m') +
// exp(s - m') v; l likewise); here it runs a tile at a time, p is rounded to bf16 for the tensor cores, and exp is
// exp2 with the scale folded in: the result agrees with the f32 recurrence to bf16 rounding (tests: relative
// Frobenius error <= 4e-3 against the restated reference).
// Keys past s_k in the last tile get p = 0; query rows past s_q are computed and not stored. Every mbarrier wait is
// bounded; a wait that gives up sets the context's status word and the kernel returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdint>
#include <mutex>

#include "../../include/thinfer_nvfp4.h"
#include "context.h"
#include "epilogue.cuh"
#include "internal.h"
#include "ptx.cuh"
#include "quant_dev.cuh"

namespace tnf {

namespace at {
constexpr int kThreads = 384;          // Q/K loader, MMA issuer, V loader, a spare warp, two softmax groups of four warps
constexpr uint32_t kD = 128;           // head dimension
constexpr uint32_t kRows = 128;        // query rows per group, keys per tile
constexpr uint32_t kSub = 128 * 128;   // one [128 rows x 64 bf16] swizzled box: 16 KB
constexpr uint32_t kTile = 2 * kSub;   // [128 x 128] bf16
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kOCol = 256;        // O_g at kOCol + 128 g; S_g (and P_g in its first 64 columns) at 128 g
constexpr uint32_t kSplitK = 6;        // P V starts when kSplitK * 16 probabilities of every row are written
constexpr float kLazy = 10.0f;         // m moves when a score may exceed it by more than this (exp2 domain) ...
constexpr float kLazySum = 1024.0f;    // ... which a sum of probabilities above 2^kLazy shows
constexpr uint32_t kSmemBytes = 1024 + 6 * kTile + 512 + 512 + 2048;  // Q x 2 | K x 2 | V x 2 | barriers | quantiser table | row statistics
}  // namespace at

struct SdpaParams {
  uint16_t* out;        // bf16 [b, s_q, h_q, 128], or null when only the NVFP4 copy is wanted
  uint8_t* q_codes;     // NVFP4 copy of the output as an [b * s_q, h_q * 128] operand: codes ...
  uint8_t* q_scales;    // ... and DEVICE-layout scales; null when not asked for
  float q_global, q_inv_t;
  uint32_t q_k_atoms;
  uint32_t* status;
  long long wait_limit;
  uint32_t s_q, s_k, h_q, h_kv;
  SdpaPlan plan;
  uint32_t split;       // CTAs of a cluster that share an item's keys (kSplit)
  uint32_t wide_out;    // out starts on a 32-byte boundary
  float scale_log2;     // scale * log2(e)
};

// MN-major operand, 128-byte swizzle: rows of 128 bytes hold 64 consecutive MN elements of one K index, 8-row (K)
// groups are 1024 bytes apart (SBO), the next 64 MN elements start `lbo_bytes` further (LBO).
__device__ __forceinline__ uint64_t make_desc_mn_sw128(uint32_t saddr, uint32_t lbo_bytes) {
  return uint64_t((saddr & 0x3FFFFu) >> 4) | (uint64_t(lbo_bytes >> 4) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
         (uint64_t(2) << 61);
}
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: the A operand (bf16, two K elements per 32-bit column, lane = row) comes from tensor memory.
__device__ __forceinline__ void tc_mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// Work item `it` of the persistent loop.
struct SdpaItem {
  bool keys_mode;
  uint32_t bb, hq, hkv, q_first, tiles, units;
  uint32_t tile0 = 0, end;  // first key tile of this CTA, key tiles of the sequence
  // rank, split: this CTA's share of the keys
  __device__ __forceinline__ SdpaItem(const SdpaParams& p, uint32_t it, uint32_t rank = 0u, uint32_t split = 1u) {
    const SdpaSlot slot = sdpa_slot(p.plan, it);
    keys_mode = slot.keys_mode != 0u;
    bb = slot.pair / p.h_q;
    hq = slot.pair - bb * p.h_q;
    hkv = (hq * p.h_kv) / p.h_q;
    q_first = slot.q_first;  // first query row within the sequence
    end = tiles = (p.s_k + at::kRows - 1u) / at::kRows;
    if (split > 1u) {
      tile0 = rank * tiles / split;
      tiles = (rank + 1u) * tiles / split - tile0;
    }
    units = keys_mode ? tiles : tiles * 2u;  // (key tile, group) pairs in the order the MMAs are issued
  }
};

// Joins the outputs of a cluster. Every CTA has its rows' joint O of its two groups, as factor-free sums for its own reference maximum;
// 16-column unit u goes to CTA u * split / 8, which gets it from all CTAs with their maxima and sums of probabilities, adds them up in
// the order of the ranks and stores. The units travel as f32 into the K and V stages, whose last reader is done once every CTA has
// passed the first barrier; [unit][4 columns][row] keeps the accesses of a warp contiguous.
__device__ __forceinline__ uint32_t split_owner(uint32_t unit, uint32_t split) { return unit * split / 8u; }
__device__ __forceinline__ uint32_t split_first(uint32_t rank, uint32_t split) { return (rank * 8u + split - 1u) / split; }  // first unit
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void st_cluster_v2(uint32_t addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ float4 ld_shared_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_shared_v2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __noinline__ void split_output(const SdpaParams& p, const SdpaItem& item, uint32_t rank, uint32_t split, uint32_t sQ, uint32_t sK,
                                          const float* lut, uint32_t lane_addr, uint32_t g, uint32_t row, bool own, bool other, float m_own, float l_own,
                                          float m_o, float l_o) {
  using namespace at;
  constexpr uint32_t kUnit = 16u * kRows * 4u;  // bytes of a unit
  const uint32_t per = (8u + split - 1u) / split;  // units of a CTA, at most
  const float m = fmaxf(own ? m_own : -INFINITY, other ? m_o : -INFINITY);
  const float e_own = own ? ex2(m_own - m) : 0.0f, e_other = other ? ex2(m_o - m) : 0.0f;
  const float l = (own ? l_own * e_own : 0.0f) + (other ? l_o * e_other : 0.0f);
  tc_fence_before();
  cluster_arrive();
  cluster_wait();  // every CTA's products are complete: K, V and Q may be overwritten
  tc_fence_after();
  for (uint32_t u = g * 4u; u < g * 4u + 4u; ++u) {
    uint32_t a[16], b[16];
    if (own) tmem_ld_32x32b_x16(lane_addr + kOCol + g * 128u + u * 16u, a);
    if (other) tmem_ld_32x32b_x16(lane_addr + kOCol + (g ^ 1u) * 128u + u * 16u, b);
    tmem_ld_wait();
    const uint32_t to = split_owner(u, split);
    const uint32_t dst = mapa_cluster(sK + ((rank * per + u - split_first(to, split)) * kUnit) + row * 16u, to);
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      float v[4];
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        v[i] = (own ? __uint_as_float(a[q * 4 + i]) * e_own : 0.0f) + (other ? __uint_as_float(b[q * 4 + i]) * e_other : 0.0f);
      st_cluster_v4(dst + q * kRows * 16u, v[0], v[1], v[2], v[3]);
    }
  }
  for (uint32_t to = g; to < split; to += 2u) st_cluster_v2(mapa_cluster(sQ + (rank * kRows + row) * 8u, to), m, l);
  cluster_arrive();
  cluster_wait();
  const uint32_t q_in_seq = item.q_first + row;
  if (q_in_seq >= p.s_q) return;
  float m_all = -INFINITY, l_all = 0.0f, f[8];
  for (uint32_t r = 0; r < split; ++r) m_all = fmaxf(m_all, ld_shared_v2(sQ + (r * kRows + row) * 8u).x);
#pragma unroll
  for (uint32_t r = 0; r < 8; ++r)
    if (r < split) {
      const float2 s = ld_shared_v2(sQ + (r * kRows + row) * 8u);
      f[r] = ex2(s.x - m_all);
      l_all += s.y * f[r];
    }
  const float inv = 1.0f / l_all;
  const uint64_t grow = uint64_t(item.bb) * p.s_q + q_in_seq;  // row of the [b * s_q, h_q * 128] matrix
  const uint32_t first = split_first(rank, split), units = split_first(rank + 1u, split) - first;
  for (uint32_t i = g; i < units; i += 2u) {
    float o[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) o[c] = 0.0f;
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r)
      if (r < split)
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
          const float4 v = ld_shared_v4(sK + (r * per + i) * kUnit + q * kRows * 16u + row * 16u);
          o[q * 4] = fmaf(v.x, f[r], o[q * 4]);
          o[q * 4 + 1] = fmaf(v.y, f[r], o[q * 4 + 1]);
          o[q * 4 + 2] = fmaf(v.z, f[r], o[q * 4 + 2]);
          o[q * 4 + 3] = fmaf(v.w, f[r], o[q * 4 + 3]);
        }
    uint32_t w[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) w[c] = pack_bf16x2(o[2 * c] * inv, o[2 * c + 1] * inv);
    const uint32_t u = first + i;
    if (p.out) {
      uint16_t* dst = p.out + (grow * p.h_q + item.hq) * kD + u * 16u;
      if (p.wide_out) {
        st_global_v8(dst, w);
      } else {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
    if (p.q_codes) {  // as in the kernel's own output, a block at a time
      uint32_t lo, hi;
      const uint32_t sc = quant_block16_bf16(w, lut, p.q_inv_t, lo, hi);
      *reinterpret_cast<uint2*>(p.q_codes + grow * (uint64_t(p.h_q) * 64u) + item.hq * 64u + u * 8u) = make_uint2(lo, hi);
      p.q_scales[((grow >> 7) * p.q_k_atoms + item.hq * 2u + (u >> 2)) * 512u + (grow & 31u) * 16u + ((grow & 127u) >> 5) * 4u + (u & 3u)] = uint8_t(sc);
    }
  }
}

// kSplit: a cluster of p.split CTAs takes one item, 128 query rows in keys mode, a share of the key tiles each, and joins the outputs
// through distributed shared memory: for calls whose blocks of query rows leave SMs idle.
template <bool kSplit>
__global__ void __launch_bounds__(at::kThreads, 1)
    sdpa_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const SdpaParams p) {
  using namespace at;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t sQ = smem_base, sK = sQ + 2 * kTile, sV = sK + 2 * kTile, sBar = sV + 2 * kTile;
  const uint32_t q_full = sBar, k_full = sBar + 8, k_empty = sBar + 24, v_full = sBar + 40, v_empty = sBar + 56;
  const uint32_t s_full = sBar + 72, p_part = sBar + 88, p_full = sBar + 104, o_full = sBar + 120;
  const uint32_t q_empty = sBar + 136, tmem_holder = sBar + 144;
  volatile uint32_t* tmem_holder_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_holder - smem_base));
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_holder + 8u - smem_base));
  float* inv_d_lut = reinterpret_cast<float*>(smem_gen + (sBar + 512u - smem_base));  // the activation quantiser's table
  float* m_part = reinterpret_cast<float*>(smem_gen + (sBar + 1024u - smem_base));    // keys mode: [2 groups][128 rows]
  float* l_part = m_part + 256;

  // the warp index as a warp-uniform value: the role branches and the MMA descriptors then live in uniform registers
  // (score MMAs alone: 593 cycles a tile against 617)
  const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31u;
  const uint32_t rank = kSplit ? cluster_ctarank() : 0u, split = kSplit ? p.split : 1u;
  const uint32_t it_first = kSplit ? blockIdx.x / split : sdpa_first(p.plan, blockIdx.x);
  auto next_item = [&](uint32_t it) { return kSplit ? p.plan.items : sdpa_next(p.plan, blockIdx.x, it); };
  const SdpaItem first(p, it_first, rank, split);  // before the wait for the previous kernel: its divisions cost nothing there
  const uint32_t last_valid = p.s_k - ((p.s_k - 1u) / kRows) * kRows;  // keys of the last tile
  const long long wait_limit = p.wait_limit > 0 ? p.wait_limit : kDefaultWaitLimitCycles;

  if (tid == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (uint32_t i = 0; i < 2; ++i) {
      mbar_init(k_full + 8 * i, 1);
      mbar_init(k_empty + 8 * i, 1);
      mbar_init(v_full + 8 * i, 1);
      mbar_init(v_empty + 8 * i, 1);
      mbar_init(s_full + 8 * i, 1);
      mbar_init(p_part + 8 * i, 4);  // a group's four warps
      mbar_init(p_full + 8 * i, 4);
      mbar_init(o_full + 8 * i, 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
  }
  if (p.q_codes) fill_inv_scale_lut(inv_d_lut, p.q_global, tid, kThreads);
  if (warp == 1) {
    tmem_alloc(tmem_holder, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_holder_gen, 0);
  pdl_launch_dependents();
  pdl_wait();  // Q, K and V are the previous kernels' outputs

  // The CTA's key tiles, counted over all its items, travel through ring stage n % 2 of K and V.
  if (warp == 0) {
    // ---------------- Q and K loader ----------------
    uint32_t n = 0, q_use = 0;
    bool ok = true;
    for (uint32_t it = it_first; it < p.plan.items && ok; it = next_item(it)) {
      const SdpaItem w = it == it_first ? first : SdpaItem(p, it);
      if (q_use > 0 && !mbar_wait_warp(q_empty, (q_use - 1u) & 1u, abort_flag, kStatusProducerTimeout, wait_limit)) break;
      ++q_use;
      const uint32_t q_row0 = w.bb * p.s_q + w.q_first, k_row0 = w.bb * p.s_k;
      if (elect_one()) {
        const uint32_t q_tiles = w.keys_mode ? 1u : 2u;
        mbar_arrive_expect_tx(q_full, q_tiles * kTile);
        for (uint32_t g = 0; g < q_tiles; ++g) {
          tma_load_2d(sQ + g * kTile, &map_q, q_full, int32_t(w.hq * kD), int32_t(q_row0 + g * kRows));
          tma_load_2d(sQ + g * kTile + kSub, &map_q, q_full, int32_t(w.hq * kD + 64), int32_t(q_row0 + g * kRows));
        }
      }
      __syncwarp();
      for (uint32_t j = 0; j < w.tiles; ++j, ++n) {
        const uint32_t st = n & 1u, use = n >> 1;
        if (use > 0 && !mbar_wait_warp(k_empty + 8 * st, (use - 1u) & 1u, abort_flag, kStatusProducerTimeout, wait_limit)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_arrive_expect_tx(k_full + 8 * st, kTile);
          tma_load_2d(sK + st * kTile, &map_k, k_full + 8 * st, int32_t(w.hkv * kD), int32_t(k_row0 + (w.tile0 + j) * kRows));
          tma_load_2d(sK + st * kTile + kSub, &map_k, k_full + 8 * st, int32_t(w.hkv * kD + 64), int32_t(k_row0 + (w.tile0 + j) * kRows));
        }
        __syncwarp();
      }
    }
  } else if (warp == 2) {
    // ---------------- V loader (its ring frees later than K's: a warp of its own, so that K never waits behind V) ----------------
    uint32_t n = 0;
    bool ok = true;
    for (uint32_t it = it_first; it < p.plan.items && ok; it = next_item(it)) {
      const SdpaItem w = it == it_first ? first : SdpaItem(p, it);
      const uint32_t k_row0 = w.bb * p.s_k;
      for (uint32_t j = 0; j < w.tiles; ++j, ++n) {
        const uint32_t st = n & 1u, use = n >> 1;
        if (use > 0 && !mbar_wait_warp(v_empty + 8 * st, (use - 1u) & 1u, abort_flag, kStatusProducerTimeout, wait_limit)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_arrive_expect_tx(v_full + 8 * st, kTile);
          tma_load_2d(sV + st * kTile, &map_v, v_full + 8 * st, int32_t(w.hkv * kD), int32_t(k_row0 + (w.tile0 + j) * kRows));
          tma_load_2d(sV + st * kTile + kSub, &map_v, v_full + 8 * st, int32_t(w.hkv * kD + 64), int32_t(k_row0 + (w.tile0 + j) * kRows));
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    constexpr uint32_t idesc_qk = make_idesc_bf16(kRows, kRows);            // A and B K-major
    constexpr uint32_t idesc_pv = make_idesc_bf16(kRows, kD) | (1u << 16);  // B (V) MN-major
    // descriptor words of the first tile; the loops only add to the low word's start address
    const uint64_t k_desc = make_desc_sw128(sK), v_desc = make_desc_mn_sw128(sV, kSub);
    const uint32_t k_hi = uint32_t(k_desc >> 32), v_hi = uint32_t(v_desc >> 32);
    const uint32_t q_lo0 = uint32_t(make_desc_sw128(sQ)), k_lo0 = uint32_t(k_desc), v_lo0 = uint32_t(v_desc);
    uint32_t n0 = 0, q_use = 0, used0 = 0, used1 = 0;  // key tiles, items and each group's tiles of the items before
    bool ok = true;
    for (uint32_t it = it_first; it < p.plan.items && ok; it = next_item(it)) {
      const SdpaItem w = it == it_first ? first : SdpaItem(p, it);
      const uint32_t tiles = w.tiles, units = w.units;
      auto tile_of = [&](uint32_t u) { return w.keys_mode ? u : u >> 1; };  // unit u = (key tile, group u & 1)
      auto wait_k = [&](uint32_t u) -> bool {
        const uint32_t n = n0 + tile_of(u);
        return mbar_wait_warp(k_full + 8 * (n & 1u), (n >> 1) & 1u, abort_flag, kStatusMmaTimeout, wait_limit);
      };
      auto wait_v = [&](uint32_t u) -> bool {
        const uint32_t n = n0 + tile_of(u);
        return mbar_wait_warp(v_full + 8 * (n & 1u), (n >> 1) & 1u, abort_flag, kStatusMmaTimeout, wait_limit);
      };
      auto issue_s = [&](uint32_t u) {  // one elected lane
        const uint32_t g = u & 1u, st = (n0 + tile_of(u)) & 1u;
        const uint32_t q_lo = q_lo0 + (w.keys_mode ? 0u : g) * (kTile >> 4), k_lo = k_lo0 + st * (kTile >> 4);
#pragma unroll
        for (uint32_t kk = 0; kk < 8; ++kk) {
          const uint32_t off = ((kk >> 2) * kSub + (kk & 3u) * 32u) >> 4;
          tc_mma_bf16(tmem_base + g * 128u, (uint64_t(k_hi) << 32) | (q_lo + off), (uint64_t(k_hi) << 32) | (k_lo + off), idesc_qk, kk != 0u);
        }
        tc_commit(s_full + 8 * g);
        if (w.keys_mode || g) tc_commit(k_empty + 8 * st);  // the tile's last reader
        if (u + 1u == units) tc_commit(q_empty);                           // the item's last scores
      };
      // Waits take about 100 cycles each even when their phase is long over: V of the next unit and K of the scores that this
      // unit issues at its end are waited for where this warp is idle, between the two parts of a unit's P V, not on the way
      // from a finished P to the next scores. K of the unit after that would be too early: in keys mode its stage has only just
      // been freed. So has V's of the next unit there: keys mode waits for V when its unit begins, after this unit's scores
      // have been issued (us, waiting here against there, K and V of 16 heads from HBM: 414 x 15764 x 16 135 / 104; from L2:
      // 700 x 8000 x 24 74 / 62, 700 x 2000 x 24 19.6 / 19.8).
      auto wait_loads = [&](uint32_t u) { return (w.keys_mode || u + 1u >= units || wait_v(u + 1u)) && (u + 2u >= units || wait_k(u + 2u)); };
      ok = mbar_wait_warp(q_full, q_use & 1u, abort_flag, kStatusMmaTimeout, wait_limit);
      ++q_use;
      for (uint32_t u = 0; u < 2u && u < units && ok; ++u) {
        ok = wait_k(u);
        tc_fence_after();
        if (ok && elect_one()) issue_s(u);
        __syncwarp();
      }
      ok = ok && wait_v(0);
      for (uint32_t u = 0; u < units && ok; ++u) {
        const uint32_t g = u & 1u, j = tile_of(u), st = (n0 + j) & 1u;
        const uint32_t use = w.keys_mode ? u >> 1 : j, parity = ((g ? used1 : used0) + use) & 1u;
        const uint32_t k_steps = w.tile0 + j + 1u == w.end ? (last_valid + 15u) >> 4 : 8u;  // 16 keys each: those past s_k are left out
        const bool next = u + 2u < units;
        const uint32_t v_lo = v_lo0 + st * (kTile >> 4), d_o = tmem_base + kOCol + g * 128u, a_p = tmem_base + g * 128u;
        ok = (!w.keys_mode || u == 0u || wait_v(u)) && mbar_wait_warp(p_part + 8 * g, parity, abort_flag, kStatusMmaTimeout, wait_limit);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (uint32_t kk = 0; kk < kSplitK; ++kk)  // P's packed columns 8kk.. in TMEM, V rows 16kk..
            if (kk < k_steps)
              tc_mma_bf16_ts(d_o, a_p + kk * 8u, (uint64_t(v_hi) << 32) | (v_lo + kk * (2048u >> 4)), idesc_pv, (use | kk) != 0u);
        }
        __syncwarp();
        ok = wait_loads(u) && mbar_wait_warp(p_full + 8 * g, parity, abort_flag, kStatusMmaTimeout, wait_limit);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (uint32_t kk = kSplitK; kk < 8; ++kk)
            if (kk < k_steps)
              tc_mma_bf16_ts(d_o, a_p + kk * 8u, (uint64_t(v_hi) << 32) | (v_lo + kk * (2048u >> 4)), idesc_pv, 1u);
          if (w.keys_mode || g) tc_commit(v_empty + 8 * st);
          if (next) issue_s(u + 2u);
          else tc_commit(o_full + 8 * g);  // the group's last product
        }
        __syncwarp();
      }
      if (kSplit) break;
      n0 += tiles;
      used0 += w.keys_mode ? (tiles + 1u) >> 1 : tiles;
      used1 += w.keys_mode ? tiles >> 1 : tiles;
    }
  } else if (warp >= 4) {
    // ---------------- softmax: two groups, one query row per thread ----------------
    const uint32_t g = (warp - 4u) >> 2, quarter = warp & 3u, row = quarter * 32u + lane;
    const uint32_t lane_addr = tmem_base + ((quarter * 32u) << 16);
    const uint32_t s_addr = lane_addr + g * 128u, o_addr = lane_addr + kOCol + g * 128u;
    uint32_t s0[32], s1[32], s2[32], s3[32];
    uint32_t seen = 0, done = 0;  // key tiles and items of this group so far
    bool ok = true;               // once a wait has given up every later one does at once; the barriers of all items are still met
    for (uint32_t it = it_first; it < p.plan.items; it = next_item(it)) {
      const SdpaItem item(p, it, rank, split);  // its divisions run while the first scores are on their way
      const bool keys_mode = kSplit || item.keys_mode;
      // below every finite score, so that a first tile of scores of -inf weighs nothing and a later tile moves m
      float m_ref = -3.402823466e38f, l = 0.0f;
      uint32_t use = 0;
      const uint32_t j_step = keys_mode ? 2u : 1u;
      for (uint32_t j = (keys_mode ? g : 0u) + (kSplit ? item.tile0 : 0u); (kSplit ? j < item.tile0 + item.tiles : j * kRows < p.s_k) && ok;
           j += j_step, ++use, ++seen) {
        const uint32_t valid = min(kRows, p.s_k - j * kRows);  // keys of this tile that exist
        // S_g complete; the pipe ran O_g += P_g V of the tile before in front of it, so O_g is complete too
        if (!mbar_wait_warp(s_full + 8 * g, seen & 1u, abort_flag, kStatusEpilogueTimeout, wait_limit)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // the whole score row goes to registers in one round trip (four loads in flight, one wait)
        tmem_ld_32x32b_x32(s_addr, s0);
        tmem_ld_32x32b_x32(s_addr + 32u, s1);
        tmem_ld_32x32b_x32(s_addr + 64u, s2);
        tmem_ld_32x32b_x32(s_addr + 96u, s3);
        tmem_ld_wait();
        // keys that do not exist weigh nothing: 2^(-inf). Masked here and not per chunk: the exponentials of a tile then are one
        // block without branches, which the compiler can interleave
        auto mask = [&]() {
          if (valid < kRows) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (uint32_t(i) >= valid) s0[i] = 0xFF800000u;
              if (32u + uint32_t(i) >= valid) s1[i] = 0xFF800000u;
              if (64u + uint32_t(i) >= valid) s2[i] = 0xFF800000u;
              if (96u + uint32_t(i) >= valid) s3[i] = 0xFF800000u;
            }
          }
        };
        mask();
        auto chunk_max = [&](const uint32_t(&c)[32]) -> float {
          float a = -INFINITY, b = -INFINITY, d = -INFINITY, e = -INFINITY;
#pragma unroll
          for (int i = 0; i < 32; i += 8) {  // three-input maxima: 16 instructions for 32 values
            a = max3(a, __uint_as_float(c[i]), __uint_as_float(c[i + 1]));
            b = max3(b, __uint_as_float(c[i + 2]), __uint_as_float(c[i + 3]));
            d = max3(d, __uint_as_float(c[i + 4]), __uint_as_float(c[i + 5]));
            e = max3(e, __uint_as_float(c[i + 6]), __uint_as_float(c[i + 7]));
          }
          return fmaxf(fmaxf(a, b), fmaxf(d, e));
        };
        uint64_t l01, l23;
        // p = exp2(s * scale_log2 - m) of 32 keys: row sum in f32, P as bf16 pairs (two per 32-bit column, key 2i in the low half)
        auto exps = [&](uint32_t(&c)[32], uint32_t(&w)[16]) {
          const uint64_t sc2 = pack2(p.scale_log2, p.scale_log2), nm2 = pack2(-m_ref, -m_ref);
#pragma unroll
          for (int i = 0; i < 32; i += 2) {  // the scale and the shift for two scores in one packed FMA
            float x0, x1;
            unpack2(fma2(pack2u(c[i], c[i + 1]), sc2, nm2), x0, x1);
            c[i] = __float_as_uint(ex2(x0));
            c[i + 1] = __float_as_uint(ex2(x1));
          }
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            l01 = add2(l01, pack2u(c[i], c[i + 1]));
            l23 = add2(l23, pack2u(c[i + 2], c[i + 3]));
          }
#pragma unroll
          for (int i = 0; i < 16; ++i)
            w[i] = pack_bf16x2(__uint_as_float(c[2 * i]), __uint_as_float(c[2 * i + 1]));
        };
        auto sum4 = [&]() -> float {
          float a, b, c, d;
          unpack2(l01, a, b);
          unpack2(l23, c, d);
          return (a + b) + (c + d);
        };
        uint32_t w0[16], w1[16], w2[16];
        const float top3 = chunk_max(s3) * p.scale_log2;  // scale > 0: the maximum commutes with it
        bool bad = use == 0;     // this row's m has to be taken from the scores
        bool redo = use == 0;    // ... or some row's of this warp
#pragma unroll 1
        while (true) {
          if (redo) {
            const float mx = fmaxf(fmaxf(fmaxf(chunk_max(s0), chunk_max(s1)), chunk_max(s2)) * p.scale_log2, top3);
            float alpha = 1.0f;
            if (bad && mx > m_ref) {
              alpha = ex2(m_ref - mx);
              l *= alpha;
              m_ref = mx;
            }
            if (use > 0) {  // O_g is rescaled before this tile's product, which waits for the arrivals below
              uint32_t o8[8];
#pragma unroll 1
              for (uint32_t c = 0; c < kD; c += 8u) {
                tmem_ld_32x32b_x8(o_addr + c, o8);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i) o8[i] = __float_as_uint(__uint_as_float(o8[i]) * alpha);
                tmem_st_32x32b_x8(o_addr + c, o8);
              }
            }
          }
          l01 = l23 = pack2(0.0f, 0.0f);
          exps(s0, w0);
          exps(s1, w1);
          exps(s2, w2);
          if (redo) break;
          bad = !(sum4() <= kLazySum) || !(top3 - m_ref <= kLazy);  // NaN counts as too large
          redo = __any_sync(0xFFFFFFFFu, bad);
          if (!redo) break;
          tmem_ld_32x32b_x32(s_addr, s0);  // rare: the scores again (nothing has been written over them yet)
          tmem_ld_32x32b_x32(s_addr + 32u, s1);
          tmem_ld_32x32b_x32(s_addr + 64u, s2);
          tmem_ld_wait();
          mask();
        }
        tmem_st_32x32b_x16(s_addr, w0);
        tmem_st_32x32b_x16(s_addr + 16u, w1);
        tmem_st_32x32b_x16(s_addr + 32u, w2);
        tmem_st_wait();
        tc_fence_before();  // this thread's TMEM reads and writes are ordered before the arrival below
        __syncwarp();
        if (lane == 0) mbar_arrive(p_part + 8 * g);
        exps(s3, w0);
        tmem_st_32x32b_x16(s_addr + 48u, w0);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + 8 * g);
        l += sum4();
      }
      // ---------------- O / l -> global ----------------
      // rows mode: a group stores its own rows, all columns. Keys mode: group g stores columns 64g .. 64g+63 of the joint rows,
      // O = (O_0 2^(m_0 - m) + O_1 2^(m_1 - m)) / (l_0 2^(m_0 - m) + l_1 2^(m_1 - m)).
      if (ok && use > 0) ok = mbar_wait_warp(o_full + 8 * g, done++ & 1u, abort_flag, kStatusEpilogueTimeout, wait_limit);
      float f_own = 1.0f / l, f_other = 0.0f;
      const bool other = keys_mode && (g == 1u || (kSplit ? item.tiles > 1u : p.s_k > kRows));  // the other group has seen a tile
      if (keys_mode) {
        m_part[g * 128u + row] = m_ref;
        l_part[g * 128u + row] = l;
        tc_fence_before();
        // the eight softmax warps; every one of them gets here, whatever happened. Each has waited for its group's O by now.
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (other) {
          const float m_o = m_part[(g ^ 1u) * 128u + row], l_o = l_part[(g ^ 1u) * 128u + row];
          const float m = use > 0 ? fmaxf(m_ref, m_o) : m_o;
          const float e_own = use > 0 ? ex2(m_ref - m) : 0.0f, e_other = ex2(m_o - m);
          const float inv = 1.0f / (use > 0 ? l * e_own + l_o * e_other : l_o * e_other);
          f_own = e_own * inv;
          f_other = e_other * inv;
        }
      }
      if constexpr (kSplit) {
        split_output(p, item, rank, split, sQ, sK, inv_d_lut, lane_addr, g, row, use > 0, other, m_ref, l, m_part[(g ^ 1u) * 128u + row],
                     l_part[(g ^ 1u) * 128u + row]);
        break;
      }
      tc_fence_after();
      if (ok && __all_sync(0xFFFFFFFFu, *abort_flag == 0u)) {
        const uint32_t q_in_seq = item.q_first + (keys_mode ? 0u : g * kRows) + row;
        const bool store = q_in_seq < p.s_q;
        const uint64_t grow = uint64_t(item.bb) * p.s_q + q_in_seq;  // row of the [b * s_q, h_q * 128] matrix
        uint16_t* dst = p.out ? p.out + (grow * p.h_q + item.hq) * kD : nullptr;
        const uint32_t c_first = keys_mode ? g * 2u : 0u, c_end = keys_mode ? g * 2u + 2u : 4u;  // 32-column chunks
        uint32_t sc4 = 0;  // the four block scales of 64 columns: one word of the scale layout
#pragma unroll 1
        for (uint32_t c2 = c_first; c2 < c_end; ++c2) {
          if (use > 0) {
            tmem_ld_32x32b_x32(o_addr + c2 * 32u, s0);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) s0[i] = __float_as_uint(__uint_as_float(s0[i]) * f_own);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) s0[i] = 0u;
          }
          if (other) {
            tmem_ld_32x32b_x32(lane_addr + kOCol + (g ^ 1u) * 128u + c2 * 32u, s1);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) s0[i] = __float_as_uint(fmaf(__uint_as_float(s1[i]), f_other, __uint_as_float(s0[i])));
          }
          if (store) {
            uint32_t w[16];  // 32 columns as bf16 pairs
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(s0[2 * i]), __uint_as_float(s0[2 * i + 1]));
            if (dst) {
              if (p.wide_out) {  // whole 32-byte sectors: the rows of a warp are far apart, half sectors would cost two writes each
                st_global_v8(dst + c2 * 32u, &w[0]);
                st_global_v8(dst + c2 * 32u + 16u, &w[8]);
              } else {
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q)
                  *reinterpret_cast<uint4*>(dst + c2 * 32u + q * 8u) = make_uint4(w[q * 4], w[q * 4 + 1], w[q * 4 + 2], w[q * 4 + 3]);
              }
            }
            if (p.q_codes) {
              // the out-projection's activation quantiser, on the bf16-rounded values: two 16-column blocks per 32 columns,
              // 8 code bytes each; the same bits tnf_quantize_act makes of the bf16 output
              uint32_t codes[4];
              if ((c2 & 1u) == 0u) sc4 = 0;
#pragma unroll
              for (uint32_t blk = 0; blk < 2; ++blk) {
                const uint32_t w8[8] = {w[blk * 8], w[blk * 8 + 1], w[blk * 8 + 2], w[blk * 8 + 3], w[blk * 8 + 4], w[blk * 8 + 5], w[blk * 8 + 6], w[blk * 8 + 7]};
                const uint32_t sc = quant_block16_bf16(w8, inv_d_lut, p.q_inv_t, codes[blk * 2], codes[blk * 2 + 1]);
                sc4 |= sc << (8u * ((c2 & 1u) * 2u + blk));
              }
              *reinterpret_cast<uint4*>(p.q_codes + grow * (uint64_t(p.h_q) * 64u) + item.hq * 64u + c2 * 16u) =
                  make_uint4(codes[0], codes[1], codes[2], codes[3]);
              // blocks hq*8 + 4 * half .. +3 of the row: one 4-byte word of atom hq*2 + half (the launcher has cleared the padding)
              if (c2 & 1u)
                *reinterpret_cast<uint32_t*>(p.q_scales + ((grow >> 7) * p.q_k_atoms + item.hq * 2u + (c2 >> 1)) * 512u + (grow & 31u) * 16u + ((grow & 127u) >> 5) * 4u) = sc4;
            }
          }
        }
      }
      if (keys_mode) {  // the other group's rows may be overwritten by its next item: not before this group has read them
        tc_fence_before();
        asm volatile("bar.sync 1, 256;" ::: "memory");
      }
    }
  }
  if (kSplit && warp < 4u) {  // the warps without rows: split_output has the others'
    cluster_arrive();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0u)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies and MMAs in flight retire
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
  if (tid == 0 && *abort_flag != 0u) atomicCAS(p.status, 0u, *abort_flag);
}

}  // namespace tnf

using namespace tnf;

extern "C" int32_t tnf_sdpa(tnf_ctx* ctx, const tnf_sdpa_args* a) {
  if (!ctx || !a) {
    set_error("tnf_sdpa: null context or args");
    return TNF_ERR_INVALID_ARGUMENT;
  }
  if (a->b == 0 || a->s_q == 0 || a->s_k == 0 || a->h_q == 0 || a->h_kv == 0 || a->d != at::kD || a->h_q % a->h_kv != 0 ||
      !(a->scale > 0.0f) || a->mask_mode != 0 || (a->flags & ~uint32_t(TNF_SDPA_OUT_NVFP4 | TNF_SDPA_NO_BF16_OUT)) ||
      ((a->flags & TNF_SDPA_NO_BF16_OUT) && !(a->flags & TNF_SDPA_OUT_NVFP4)) || ((a->flags & TNF_SDPA_OUT_NVFP4) && !(a->out_global > 0.0f))) {
    set_error("tnf_sdpa: b=%u s_q=%u s_k=%u h_q=%u h_kv=%u d=%u scale=%g mask_mode=%u (d must be 128, h_kv must divide h_q, "
              "scale > 0, mask_mode 0; flags 0x%x: NO_BF16_OUT needs OUT_NVFP4, which needs out_global > 0)", a->b, a->s_q, a->s_k, a->h_q, a->h_kv,
              a->d, a->scale, a->mask_mode, a->flags);
    return TNF_ERR_INVALID_ARGUMENT;
  }
  const uint64_t q_rows = uint64_t(a->b) * a->s_q, k_rows = uint64_t(a->b) * a->s_k;
  if (q_rows >= (1ull << 31) || k_rows >= (1ull << 31) || a->h_q > 65535u || a->b > 65535u) {
    set_error("tnf_sdpa: problem too large (b * s_q and b * s_k below 2^31, h_q and b up to 65535)");
    return TNF_ERR_INVALID_ARGUMENT;
  }
  int32_t st = TNF_OK;
  const uint64_t q_cols = uint64_t(a->h_q) * at::kD, kv_cols = uint64_t(a->h_kv) * at::kD;
  // leading dimensions in elements: q, k and v may be column windows of one wider matrix (the fused QKV output)
  const uint64_t q_ld = a->q_ld ? a->q_ld : q_cols, kv_ld = a->kv_ld ? a->kv_ld : kv_cols;
  if (q_ld < q_cols || kv_ld < kv_cols || q_ld % 8 != 0 || kv_ld % 8 != 0) {
    set_error("tnf_sdpa: q_ld %llu / kv_ld %llu must cover the heads (%llu / %llu elements) and be multiples of 8",
              (unsigned long long)q_ld, (unsigned long long)kv_ld, (unsigned long long)q_cols, (unsigned long long)kv_cols);
    return TNF_ERR_INVALID_ARGUMENT;
  }
  uint8_t* q = resolve(ctx, a->q, ((q_rows - 1) * q_ld + q_cols) * 2, "q", &st);
  if (!q) return st;
  uint8_t* k = resolve(ctx, a->k, ((k_rows - 1) * kv_ld + kv_cols) * 2, "k", &st);
  if (!k) return st;
  uint8_t* v = resolve(ctx, a->v, ((k_rows - 1) * kv_ld + kv_cols) * 2, "v", &st);
  if (!v) return st;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15u) {
    set_error("tnf_sdpa: q, k and v must start on 16-byte boundaries");
    return TNF_ERR_INVALID_ARGUMENT;
  }
  uint8_t* out = nullptr;
  if (!(a->flags & TNF_SDPA_NO_BF16_OUT)) {
    out = resolve(ctx, a->out, q_rows * q_cols * 2, "out", &st);
    if (!out) return st;
  }
  uint8_t *q_codes = nullptr, *q_scales = nullptr;
  if (a->flags & TNF_SDPA_OUT_NVFP4) {  // the out-projection's A operand: [b * s_q, h_q * 128] codes + DEVICE scales
    q_codes = resolve(ctx, a->out_codes, q_rows * (q_cols / 2), "out_codes", &st);
    if (!q_codes) return st;
    q_scales = resolve(ctx, a->out_scales, sf_device_bytes(uint32_t(q_rows), uint32_t(q_cols)), "out_scales", &st);
    if (!q_scales) return st;
  }
  if (cudaSetDevice(ctx->device) != cudaSuccess) return cuda_fail(cudaGetLastError(), "cudaSetDevice");
  CUtensorMap mq, mk, mv;  // [rows, heads * 128] bf16, boxes of 64 columns x 128 rows, 128-byte swizzle
  if (!get_map(ctx, MapSpec{q, 2, q_cols, q_rows, q_ld * 2, 64, 128, 128}, &mq) ||
      !get_map(ctx, MapSpec{k, 2, kv_cols, k_rows, kv_ld * 2, 64, 128, 128}, &mk) ||
      !get_map(ctx, MapSpec{v, 2, kv_cols, k_rows, kv_ld * 2, 64, 128, 128}, &mv))
    return TNF_ERR_INVALID_ARGUMENT;
  SdpaParams p{};
  p.out = reinterpret_cast<uint16_t*>(out);
  p.wide_out = reinterpret_cast<uintptr_t>(out) % 32u == 0 ? 1u : 0u;
  if (q_codes) {
    p.q_codes = q_codes;
    p.q_scales = q_scales;
    p.q_global = a->out_global;
    p.q_inv_t = 1.0f / (6.0f * a->out_global);
    p.q_k_atoms = sf_k_atoms(uint32_t(q_cols));
    // benign (zero) scales where the kernel writes none: the K-padding atoms of every row block, and the rows of the
    // last 128-row block past the matrix
    const uint32_t used_atoms = uint32_t(q_cols / 64), row_blocks = uint32_t((q_rows + 127u) / 128u);
    if (used_atoms < p.q_k_atoms) {
      cudaError_t e = cudaMemset2DAsync(q_scales + uint64_t(used_atoms) * 512u, uint64_t(p.q_k_atoms) * 512u, 0,
                                        uint64_t(p.q_k_atoms - used_atoms) * 512u, row_blocks, ctx->compute);
      if (e != cudaSuccess) return cuda_fail(e, "out_scales padding clear");
    }
    if (q_rows % 128u != 0) {
      cudaError_t e = cudaMemsetAsync(q_scales + uint64_t(row_blocks - 1u) * p.q_k_atoms * 512u, 0, uint64_t(p.q_k_atoms) * 512u, ctx->compute);
      if (e != cudaSuccess) return cuda_fail(e, "out_scales last block clear");
    }
  }
  p.status = ctx->dwords;
  p.wait_limit = ctx->wait_limit_cycles;
  p.s_q = a->s_q; p.s_k = a->s_k; p.h_q = a->h_q; p.h_kv = a->h_kv;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  const uint64_t pairs = uint64_t(a->h_q) * a->b;
  uint32_t split = 1u;
  {
    // One thread prepares a device; another's first call waits for the attributes and the whole table, so that the same call takes
    // the same kernel whoever comes first. What failed is tried again by the next call.
    static std::mutex mu;
    static bool ready[kMaxDevices + 1] = {};       // the last entry: devices past the table, prepared by every call
    static int clusters[kMaxDevices + 1][9] = {};  // clusters of 2 .. 8 CTAs that fit the device at once
    const int dev = ctx->device < kMaxDevices ? ctx->device : kMaxDevices;
    std::lock_guard<std::mutex> lk(mu);
    if (!ready[dev]) {
      cudaError_t e = cudaFuncSetAttribute(sdpa_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(at::kSmemBytes));
      if (e == cudaSuccess) e = cudaFuncSetAttribute(sdpa_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(at::kSmemBytes));
      if (e != cudaSuccess) return cuda_fail(e, "sdpa kernel attribute");
      max_clusters(sdpa_kernel<true>, at::kThreads, at::kSmemBytes, ctx->sm_count, clusters[dev]);
      ready[dev] = dev < kMaxDevices;
    }
    split = sdpa_split(pairs * ((uint64_t(a->s_q) + 127u) / 128u), a->s_k, clusters[dev]);
  }
  if (split > 1u) {
    sdpa_split_plan(a->s_q, pairs, &p.plan);
  } else if (!sdpa_plan(a->s_q, pairs, uint32_t(ctx->sm_count), &p.plan)) {
    set_error("tnf_sdpa: problem too large (b=%u s_q=%u h_q=%u: more than 2^31 work items)", a->b, a->s_q, a->h_q);
    return TNF_ERR_INVALID_ARGUMENT;
  }
  p.split = split;
  cudaError_t e = split > 1u ? launch_pdl_cluster(sdpa_kernel<true>, dim3(p.plan.items * split), dim3(at::kThreads), split, at::kSmemBytes, ctx->compute, mq, mk, mv, p)
                             : launch_pdl(sdpa_kernel<false>, dim3(p.plan.ctas), dim3(at::kThreads), at::kSmemBytes, ctx->compute, mq, mk, mv, p);
  if (e != cudaSuccess) return cuda_fail(e, "sdpa launch");
  return TNF_OK;
}
