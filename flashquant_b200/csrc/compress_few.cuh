// A few vectors (a decode step appends one token per sequence): fp32 FMAs with the matrices read
// straight from L2 into registers.  Included by compress.cu.
//
// Such a call is bound by latency: the 16-row tensor-core kernel spends 7 us on 32 tokens, nearly all
// of it turning the fp32 matrix into fp16 planes in shared memory before the first product.
// Here a CTA takes kFewVecs vectors of one source, a warp = eight output columns (rows of Pi, a row per
// load instruction) or a thread = four columns and 1/16 of k, and every global load of the kernel - the vectors and all matrices of
// the chain - is issued before the first use of any of them, so one trip to L2 is the whole wait.
// An fp32 FMA contraction of these few vectors is a few hundred cycles.
//
// kTwoStage: source 0 goes through the two-stage quantiser (x_tilde, gamma, signs).
#pragma once

namespace fq {

constexpr int kFewVecs = 4;
// One wave: two CTAs on each of 148 SMs.  Above it the CTA-per-tile kernel is faster, as every CTA reads the
// 64 KB of its matrix from the L2.  Time per call in us, keys and values of n tokens x 8 heads (the
// CTA-per-tile kernel in brackets): n = 1: 3.8 (6.8), 32: 4.9 (7.5), 73: 6.7 (7.6), 100: 8.8 (7.6); two-stage
// 6.4 (13.2), 8.5 (14.1), 12.0 (14.2), 15.8 (14.2); head_dim 64 3.2 (4.7), 3.7 (5.2), 3.9 (5.2), 4.5 (5.3).
// (The recheck is about 0.7 us of 32 tokens and 1.3 us of 73: some CTA of the call has one.)
constexpr int64_t kFewMaxVectors = 1184;

template <int D, int DT, bool kTwoStage>
__global__ void __launch_bounds__(kFewVecs* D, kTwoStage ? 1 : 2)
    compress_few_kernel(CompressArgs p) {
  using T = typename Elem<DT>::type;
  constexpr int kThreads = kFewVecs * D;
  constexpr int kLenA = D / 32, kLenB = D / 16, kQuads = D / 4;
  constexpr int kWarpsPerVec = D / 32;
  __shared__ __align__(16) float xs[kFewVecs][D];
  __shared__ __align__(16) float xr[kFewVecs][D];  // the vectors as they came
  __shared__ float s_nrm[kFewVecs];
  __shared__ __align__(16) float red[16][kFewVecs][D];
  __shared__ float part[kThreads / 32];
  __shared__ float s_bnd[16], s_cent[16];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s = blockIdx.y;
  const bool two_stage = kTwoStage && s == 0;
  const uint32_t n_vec = uint32_t(p.n_tokens * p.heads), heads = uint32_t(p.heads);
  // owner maps: (vector r, column j) with j along the lanes, and (column ja, vector sl)
  const int r = tid / D, j = tid % D;
  const int ja = tid >> 2, sl = tid & 3;
  const int c4 = tid % kQuads, ks = tid / kQuads;

  // ---- every load of the kernel ---------------------------------------------------------------
  const uint32_t v = blockIdx.x * kFewVecs + r;
  float x = 0.f;
  if (v < n_vec) {
    const uint32_t tok = v / heads;
    x = to_f32(static_cast<const T*>(p.src[s])[int64_t(tok) * p.token_stride + int64_t(v - tok * heads) * D + j]);
  }
  // where vector i of the CTA goes: -1 nowhere
  auto slot_of = [&](int i, int& head) -> int64_t {
    const uint32_t vec = blockIdx.x * kFewVecs + i;
    head = 0;
    if (vec >= n_vec) return -1;
    const uint32_t tok = vec / heads;
    head = int(vec - tok * heads);
    if (p.slots) {
      const int64_t slot = p.slot64 ? static_cast<const int64_t*>(p.slots)[tok]
                                    : int64_t(static_cast<const int32_t*>(p.slots)[tok]);
      return slot < p.num_slots ? slot : -1;
    }
    return p.seg_len ? segment_row(p, tok) : int64_t(tok);
  };
  int head_r, head_sl;
  const int64_t slot_r = slot_of(r, head_r);     // of the vector this thread owns by (r, j)
  const int64_t slot_sl = slot_of(sl, head_sl);  // ... by (ja, sl)
  const float* mat_a = s && p.mat_a1 ? p.mat_a1 : p.mat_a;
  const float* mat_b = s && p.mat_b1 ? p.mat_b1 : p.mat_b;
  float4 fwd[8], mid[kTwoStage ? kLenB : 1], sgn[kTwoStage ? 8 : 1];
  // rows 8*warp .. +7 of a matrix, the lane's D/32 columns of each: one line per load, whatever the row
  auto load_rows = [&](const float* m, float4* f) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float* src = m + (8 * warp + i) * D + lane * kLenA;
      if constexpr (kLenA == 4) {
        f[i] = *reinterpret_cast<const float4*>(src);
      } else {
        const float2 h = *reinterpret_cast<const float2*>(src);
        f[i] = make_float4(h.x, h.y, 0.f, 0.f);
      }
    }
  };
  if (p.rot_split) {
    // columns 4*c4 .. of [even | odd] of Pi^T, rows ks*kLenB ..
    const float* m = (c4 < kQuads / 2 ? mat_a : mat_b) + 4 * (c4 % (kQuads / 2));
#pragma unroll
    for (int i = 0; i < kLenB; ++i)
      fwd[i] = *reinterpret_cast<const float4*>(m + (ks * kLenB + i) * (D / 2));
  } else {
    load_rows(mat_a, fwd);
  }
  if constexpr (kTwoStage) {
    if (two_stage) {
#pragma unroll
      for (int i = 0; i < kLenB; ++i)
        mid[i] = *reinterpret_cast<const float4*>(p.mat_a + (ks * kLenB + i) * D + 4 * c4);
      load_rows(p.qjl, sgn);
    }
  }
  if (tid < 16) {
    s_bnd[tid] = tid < p.nb[s] ? p.bnd[s][tid] : __int_as_float(0x7f800000);
    s_cent[tid] = two_stage && tid <= p.nb[0] ? p.cent0[tid] : 0.f;
  }

  // sum over the D threads of a vector, to all of them
  auto vector_sum = [&](float a) {
    a = warp_sum(a);
    if (lane == 0) part[warp] = a;
    __syncthreads();
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarpsPerVec; ++w) sum += part[r * kWarpsPerVec + w];
    return sum;
  };
  // sum_k xs[sl][k] m[ja][k]: every lane has its share of k for the warp's eight columns and the
  // four vectors; the 32 sums are reduced by halving, lane l keeps sum l
  auto product_rows = [&](const float4* m) {
    float acc[8 * kFewVecs];
#pragma unroll
    for (int i = 0; i < kFewVecs; ++i) {
      float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < kLenA; ++q) a[q] = xs[i][lane * kLenA + q];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float sum = fmaf(a[1], m[c].y, a[0] * m[c].x);
        if constexpr (kLenA == 4) sum = fmaf(a[3], m[c].w, fmaf(a[2], m[c].z, sum));
        acc[c * kFewVecs + i] = sum;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const float keep = up ? acc[i + o] : acc[i], give = up ? acc[i] : acc[i + o];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    return acc[0];
  };
  // red[ks][i][4*c4 ..] = partial of sum_k xs[i][k] m[k][4*c4 ..]
  auto product_cols = [&](const float4* m) {
#pragma unroll
    for (int i = 0; i < kFewVecs; ++i) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < kLenB; ++q) {
        const float a = xs[i][ks * kLenB + q];
        acc.x = fmaf(a, m[q].x, acc.x);
        acc.y = fmaf(a, m[q].y, acc.y);
        acc.z = fmaf(a, m[q].z, acc.z);
        acc.w = fmaf(a, m[q].w, acc.w);
      }
      *reinterpret_cast<float4*>(&red[ks][i][4 * c4]) = acc;
    }
  };
  auto gather = [&](int col) {
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < 16; ++q) sum += red[q][r][col];
    return sum;
  };

  // ---- norm (summed as compress_coop_kernel does), x_hat ------------------------------------------
  xr[r][j] = x;
  __syncthreads();
  float ss = 0.f;
#pragma unroll
  for (int q = 0; q < kLenA; ++q) ss = fmaf(xr[r][lane * kLenA + q], xr[r][lane * kLenA + q], ss);
  const float nrm = sqrtf(warp_sum(ss));
  xs[r][j] = x * (1.f / (nrm + 1e-10f));
  if (j == 0) {
    s_nrm[r] = nrm;
    if (slot_r >= 0)
      *reinterpret_cast<float*>(p.norm[s] + slot_r * p.norm_row_stride + head_r * 4) = nrm;
  }
  __syncthreads();

  // ---- y = x_hat Pi^T, codes; the centroid vector replaces x_hat --------------------------------
  int idx;
  float y;
  if (p.rot_split) {
    product_cols(fwd);
    __syncthreads();
    y = gather((j >> 1) + (j & 1) * (D / 2));
  } else {
    y = product_rows(fwd);
  }
  idx = bucketize15(y, s_bnd);
  // (a zero vector's coordinates are zero in any arithmetic)
  const bool near = near_boundary(y, idx, s_bnd) && s_nrm[p.rot_split ? r : sl] > 0.f;
  if (const uint32_t lanes = __ballot_sync(0xffffffffu, near)) {
    if (p.rot_split) {
      const int col0 = j - lane;  // the warp's 32 columns of vector r, eight at a time
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        if (!(lanes >> (8 * c) & 0xffu)) continue;
        const float2 f = recheck_columns<D, kMatSplit>(xs[r], 1, mat_a, mat_b, col0 + 8 * c);
        const float f0 = __shfl_sync(0xffffffffu, f.x, (lane & 7) >> 1);
        const float f1 = __shfl_sync(0xffffffffu, f.y, (lane & 7) >> 1);
        if (lane >> 3 == c) idx = bucketize15((lane & 1) ? f1 : f0, s_bnd);
      }
    } else {
      const float2 f = recheck_columns<D, kMatRows>(xs[0], kFewVecs, mat_a, nullptr, 8 * warp);
      const float f0 = __shfl_sync(0xffffffffu, f.x, 4 * sl + (lane >> 3));
      const float f1 = __shfl_sync(0xffffffffu, f.y, 4 * sl + (lane >> 3));
      idx = bucketize15((lane >> 2 & 1) ? f1 : f0, s_bnd);
    }
  }
  if (p.rot_split) {
    // a warp holds 32 consecutive columns of vector r: eight lanes make a word
    uint32_t w = uint32_t(idx) << (8 * ((j >> 1) & 3) + ((j & 1) ? 0 : 4));
    w |= __shfl_xor_sync(0xffffffffu, w, 1);
    w |= __shfl_xor_sync(0xffffffffu, w, 2);
    w |= __shfl_xor_sync(0xffffffffu, w, 4);
    if ((lane & 7) == 0 && slot_r >= 0)
      store_code_word(p.code[s] + slot_r * p.code_row_stride + int64_t(head_r) * p.code_head_stride + j / 2, w);
  } else {
    // a warp holds columns 8*warp .. 8*warp+7 of every vector, column = lane / 4
    uint32_t w = uint32_t(idx) << (8 * (lane >> 3) + ((ja & 1) ? 0 : 4));
    w |= __shfl_xor_sync(0xffffffffu, w, 4);
    w |= __shfl_xor_sync(0xffffffffu, w, 8);
    w |= __shfl_xor_sync(0xffffffffu, w, 16);
    if (lane < 4 && slot_sl >= 0)
      store_code_word(p.code[s] + slot_sl * p.code_row_stride + int64_t(head_sl) * p.code_head_stride + 4 * warp,
                      w);
    if constexpr (kTwoStage) {
      __syncthreads();  // x_hat has been read
      xs[sl][ja] = s_cent[idx];
    }
  }

  if constexpr (kTwoStage) {
    if (!two_stage) return;
    // ---- x_tilde = (c[code] Pi) n, residual, gamma ----------------------------------------------
    __syncthreads();
    product_cols(mid);
    __syncthreads();
    const float res = x - gather(j) * nrm;
    xs[r][j] = res;
    const float gam = sqrtf(vector_sum(res * res));  // (its barrier also publishes the residual)
    if (j == 0 && slot_r >= 0)
      *reinterpret_cast<float*>(p.gam + slot_r * p.gam_row_stride + head_r * 4) = gam;
    // ---- sign(r S^T): bit j%8 of byte j/8 is 1 for a projection >= 0; a warp makes one byte ------
    const float proj = product_rows(sgn);
    uint32_t b = proj >= 0.f ? 1u << (lane >> 2) : 0u;
    b |= __shfl_xor_sync(0xffffffffu, b, 4);
    b |= __shfl_xor_sync(0xffffffffu, b, 8);
    b |= __shfl_xor_sync(0xffffffffu, b, 16);
    if (__syncthreads_or(fabsf(proj) <= kNearZero * s_nrm[sl] && s_nrm[sl] > 0.f)) {
      // the chain from the codes on, eight columns a warp (the residual has been read)
      const int g = lane >> 2, col = 8 * warp + 2 * (lane & 3);
      xs[sl][ja] = s_cent[idx];
      __syncthreads();
      float2 f = recheck_columns<D, kMatCols>(&xs[0][0], kFewVecs, p.mat_a, nullptr, 8 * warp);
      if (g < kFewVecs)
        *reinterpret_cast<float2*>(&red[0][g][col]) =
            make_float2(fmaf(-f.x, s_nrm[g], xr[g][col]), fmaf(-f.y, s_nrm[g], xr[g][col + 1]));
      __syncthreads();
      f = recheck_columns<D, kMatRows>(&red[0][0][0], kFewVecs, p.qjl, nullptr, 8 * warp);
      b = ((f.x >= 0.f ? 1u : 0u) | (f.y >= 0.f ? 2u : 0u)) << (2 * (lane & 3));
      b |= __shfl_xor_sync(0xffffffffu, b, 1);
      b |= __shfl_xor_sync(0xffffffffu, b, 2);
      b = __shfl_sync(0xffffffffu, b, 4 * (lane & 3));  // lane i < 4: of vector i
    }
    if (lane < 4 && slot_sl >= 0)
      p.sign[slot_sl * p.sign_row_stride + head_sl * (D / 8) + warp] = uint8_t(b);
  }
}

template <int D, int DT, bool kTwoStage>
static int launch_compress_few(const CompressArgs& a, int64_t n_vec, cudaStream_t stream) {
  const dim3 grid(unsigned((n_vec + kFewVecs - 1) / kFewVecs), unsigned(a.n_src));
  compress_few_kernel<D, DT, kTwoStage><<<grid, kFewVecs * D, 0, stream>>>(a);
  return check_launch("compress kernel launch");
}

}  // namespace fq
