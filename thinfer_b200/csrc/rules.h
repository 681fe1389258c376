// Index rules that kernels and launchers share and a CPU test compiles: no CUDA header in here.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TNF_HD __host__ __device__
#else
#define TNF_HD
#endif

namespace tnf {

// 128-row block of an operand's block scales that holds `row`; the last block there is for rows past the operand. A tile that
// hangs over the end of W copies that block once more: those columns are not stored, and the layout has nothing behind it.
TNF_HD inline uint32_t sf_row_block(uint32_t row, uint32_t rows) {
  const uint32_t last = (rows - 1u) >> 7, block = row >> 7;
  return block < last ? block : last;
}

// Width of the 1-CTA GEMM's 128-row tiles. 256 only when such tiles still fill the SMs and W has columns for more than half of
// one; 128-wide tiles also double-buffer the accumulator; with so few tiles that half the SMs would idle, 64-wide ones: a CTA's
// time is what it has to pull in (its A tile and its share of W) and what it writes out, and both shrink with the tile.
TNF_HD inline uint32_t tile_n_rule(uint32_t m, uint32_t n, uint32_t sms) {
  const uint64_t tm = (uint64_t(m) + 127u) / 128u;
  if (n > 128u && tm * ((uint64_t(n) + 255u) / 256u) >= sms) return 256u;
  return tm * ((uint64_t(n) + 127u) / 128u) * 2u <= sms ? 64u : 128u;
}

}  // namespace tnf
