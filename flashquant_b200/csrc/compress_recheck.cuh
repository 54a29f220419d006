// One arithmetic for the codes and signs, whichever kernel makes them.  Included by compress.cu.
//
// A code whose coordinate lies within a rounding of a boundary may fall on either side of it, and
// where its key holds a tenth of a row's softmax weight the two choices differ by percents of that
// row.  So that a vector's bytes do not depend on how many vectors a call carries, the kernels decide alike:
// the norm is summed in the order of compress_coop_kernel (of compress_kernel where a call has
// kCoopMaxTiles tiles or more), and a coordinate within kNearBoundary of a boundary, or a
// projection within kNearZero |x| of zero, is computed again by the split-fp16 `mma.sync` chain of
// those two kernels (the order of plane_mma and reg_mma_group).
//
// kNearBoundary: over 2 10^9 codes of N(0,1) vectors with and without outlier channels, all types, two
// of the kernels disagreed only within 6.0e-8 of a boundary; four times that.  About 0.2 % of the vectors have
// such a coordinate.  kNearZero: they disagreed only within 5.9e-8 |x| of zero; four times that, 0.02 %.
#pragma once

namespace fq {

constexpr float kNearBoundary = 0x1p-22f;
constexpr float kNearZero = 0x1p-22f;

// y is in cell idx of the table sb (15 boundaries, padded with +inf): next to an edge of it?
__device__ __forceinline__ bool near_boundary(float y, int idx, const float* sb) {
  return (sb[idx] - y <= kNearBoundary) | ((idx > 0) & (y - sb[idx > 0 ? idx - 1 : 0] <= kNearBoundary));
}

__device__ __forceinline__ void split_words(float2 v, uint32_t& hi, uint32_t& lo) {
  __half h0, l0, h1, l1;
  split_hi_lo(v.x, h0, l0);
  split_hi_lo(v.y, h1, l1);
  hi = pack_h2(h0, h1);
  lo = pack_h2(l0, l1);
}

// Where element (k, n) of a right operand lies: rows of m are the columns n (m[n][k]), the matrix as it
// is (m[k][n]), or the even / odd columns in m / m2.
enum : int { kMatRows = 0, kMatCols = 1, kMatSplit = 2 };

// sum_k a[row][k] B[k][n] for row = lane / 4 (n_rows of them, D floats each) and the columns
// n = col0 + 2 (lane % 4), + 1; a whole warp.  (A loop and not unrolled: it is rarely run, so its
// instructions come from memory.)
template <int D, int kMat>
__device__ __forceinline__ float2 recheck_columns(const float* a, int n_rows, const float* m,
                                                  const float* m2, int col0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n = col0 + g;
  float hi[4] = {0.f, 0.f, 0.f, 0.f}, co[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int ks = 0; ks < D / 16; ++ks) {
    uint32_t ah[2], al[2], bh[2], bl[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = 16 * ks + 8 * i + 2 * t;
      float2 x = make_float2(0.f, 0.f), y;
      if (g < n_rows) x = *reinterpret_cast<const float2*>(a + g * D + k);
      if constexpr (kMat == kMatRows) {
        y = *reinterpret_cast<const float2*>(m + n * D + k);
      } else if constexpr (kMat == kMatCols) {
        y = make_float2(m[k * D + n], m[(k + 1) * D + n]);
      } else {
        const float* s = ((n & 1) ? m2 : m) + (n >> 1);
        y = make_float2(s[k * (D / 2)], s[(k + 1) * (D / 2)]);
      }
      split_words(x, ah[i], al[i]);
      split_words(y, bh[i], bl[i]);
    }
    mma_f16(hi, ah[0], 0u, ah[1], 0u, bh[0], bh[1]);
    mma_f16(co, ah[0], 0u, ah[1], 0u, bl[0], bl[1]);
    mma_f16(co, al[0], 0u, al[1], 0u, bh[0], bh[1]);
  }
  return make_float2(fmaf(co[0], kLoUnscale, hi[0]), fmaf(co[1], kLoUnscale, hi[1]));
}

}  // namespace fq
