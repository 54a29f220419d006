// One query token per sequence over a contiguous cache: a CTA of 16 warps takes a slice of the 16-token
// tiles of ONE (sequence, KV head).  Included by paged_decode.cu, whose tile arithmetic (fast_keys /
// fast_back) it shares.
//
// Such a call is bound by latency: 4 sequences of 4000 tokens are 17 MB, 2.6 us of memory time.  So every CTA
// rotates the few query rows of its pair itself (64 KB of Pi from the L2, no kernel of its own for it), its
// first tiles are on their way meanwhile, a warp reads its tiles from memory straight into registers one
// tile ahead (a head's 16 tokens are 1 KB of consecutive bytes: nothing to stage), the 16 warps merge in
// shared memory, and the launch that rotates back merges the slices.
//
// Measured, attention call, against the 128-row query tile (32 / 8 heads): 1 x 20 tokens 22 -> 14 us, 4 x 4000
// 48 -> 20 us, 8 x 16384 220 -> 56 us (2.5 TB/s; one dependent chain per warp and tile bounds it).
#pragma once

#include "decode_direct.cuh"

namespace fq {

constexpr int kDirThreads = 512;
struct DirectSmem {
  static constexpr uint32_t kLut = 0;                    // 256 x (32 lanes K | 32 lanes V); at the end
  static constexpr uint32_t kOut = 0;                    //   [16 warps][8 columns][128] f32
  static constexpr uint32_t kCent = 65536;
  static constexpr uint32_t kX = kCent + kCentBytes;     // [8][128] f32 query rows
  static constexpr uint32_t kQ = kX + 8 * 128 * 4;       // [8][128] f16 rotated rows
  static constexpr uint32_t kMl = kQ + 8 * 128 * 2;      // [16 warps][8 columns] (m, l)
  static constexpr uint32_t kBytes = kMl + 16 * 8 * 8;
};

struct DirectTile {
  FastRaw k;
  uint2 v[4];
  float nk_lo, nk_hi, nv_lo, nv_hi;
};

template <typename TQ, bool KPRMT, bool PSPLIT>
__global__ void __launch_bounds__(kDirThreads, 1) decode_direct_kernel(DirectArgs p) {
  using S = DirectSmem;
  constexpr int D = 128;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int slice = blockIdx.x, head = blockIdx.y, seq = blockIdx.z;
  const int group = p.hq / p.hkv;  // columns in use (<= 8)
  const int64_t rows = int64_t(p.seqs) * p.hq, row0 = int64_t(seq) * p.hq + head * group;
  const int len = p.nkv;
  const int tiles = (len + 15) >> 4;
  const int t0 = int(int64_t(tiles) * slice / p.n_splits);
  const int t1 = int(int64_t(tiles) * (slice + 1) / p.n_splits);

  // ---- a tile's codes and norms, memory -> registers ------------------------------------------------
  // K: rows g, g+8, bytes 16t..; V: tokens 2t, 2t+1, 2t+8, 2t+9, bytes 8g..; norms of rows g, g+8.
  // Nothing is read beyond the last token.
  const int64_t first = (int64_t(seq) * p.hkv + head) * p.kv_stride;
  const uint8_t* k_lane = p.k_codes + first * 64 + 16 * t;
  const uint8_t* v_lane = p.v_codes + first * 64 + 8 * g;
  const float* kn = p.k_norms + first;
  const float* vn = p.v_norms + first;
  auto load = [&](int tile, DirectTile& x) {
    const int at = tile * 16, last = len - 1;
    auto row = [&](int r) { return min(at + r, last); };
    auto k16 = [&](int r) { return *reinterpret_cast<const uint4*>(k_lane + int64_t(r) * 64); };
    auto v8 = [&](int r) { return *reinterpret_cast<const uint2*>(v_lane + int64_t(r) * 64); };
    const int lo = row(g), hi = row(g + 8);
    x.k.ka = k16(lo);
    x.k.kb = k16(hi);
    x.nk_lo = kn[lo]; x.nk_hi = kn[hi];
    x.nv_lo = vn[lo]; x.nv_hi = vn[hi];
    x.v[0] = v8(row(2 * t));
    x.v[1] = v8(row(2 * t + 1));
    x.v[2] = v8(row(2 * t + 8));
    x.v[3] = v8(row(2 * t + 9));
  };
  DirectTile cur;
  int tile = t0 + warp;
  if (tile < t1) load(tile, cur);

  // ---- query rows, centroids; q_rot = round(q Pi^T) -------------------------------------------------
  float4 pi[8];
  const int j = tid >> 2, sl = tid & 3;  // output coordinate; chunks sl, sl + 4, .. of four k
#pragma unroll
  for (int i = 0; i < 8; ++i)
    pi[i] = reinterpret_cast<const float4*>(p.rotation + j * D + 4 * sl)[4 * i];
  float* xs = reinterpret_cast<float*>(smem + S::kX);
  __half* qs = reinterpret_cast<__half*>(smem + S::kQ);
  const TQ* q = static_cast<const TQ*>(p.q) + row0 * D;
  for (int i = tid; i < group * D; i += kDirThreads) xs[i] = to_f32(q[i]);
  uint32_t* record = p.status + kScaleCacheOffset / 4;
  if (warp == 1) {
    const int i = lane & 15;
    float c = 0.f;
    if (lane < 16) { if (i < p.nck) c = p.cent_k[i]; } else { if (i < p.ncv) c = p.cent_v[i]; }
    stage_centroids(smem + S::kCent, c, p.nck, p.ncv, record, lane);
  }
  __syncthreads();
  for (int r = 0; r < group; ++r) {
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(xs + r * D + 4 * sl + 16 * i);
      acc = fmaf(a.x, pi[i].x, acc);
      acc = fmaf(a.y, pi[i].y, acc);
      acc = fmaf(a.z, pi[i].z, acc);
      acc = fmaf(a.w, pi[i].w, acc);
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    if (sl == 0) qs[r * D + j] = __float2half_rn(to_f32(from_f32<TQ>(acc)));
  }
  scale_centroid_tables(smem + S::kCent, p.nck, p.ncv, tid,
                        slice + head + seq == 0 ? record : nullptr);
  const unsigned short* cs = reinterpret_cast<const unsigned short*>(smem + S::kCent);
  for (int i = tid; i < 256 * 32; i += kDirThreads) {
    const int e = i >> 5, l = i & 31;
    const uint32_t hi = e >> 4, lo = e & 15;
    // entries as in paged_decode_fast_kernel
    *reinterpret_cast<uint32_t*>(smem + e * kLutStride + l * 4) =
        KPRMT ? uint32_t(cs[lo]) | (uint32_t(cs[hi]) << 16) : uint32_t(cs[hi]) | (uint32_t(cs[lo]) << 16);
    *reinterpret_cast<uint32_t*>(smem + e * kLutStride + 128 + l * 4) =
        uint32_t(cs[16 + lo]) | (uint32_t(cs[16 + hi]) << 16);
  }
  __syncthreads();

  FastWarp w;
  w.lut = smem_u32(smem);
  w.laneK = w.laneN = w.laneV = 0u;
  w.lane4 = uint32_t(lane) * 4;
  w.tab[0] = w.tab[1] = w.tab[2] = w.tab[3] = 0u;
  if constexpr (KPRMT) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t h = cs[i];
      const uint32_t lo8 = (h & 0xffu) << (8 * (i & 3)), hi8 = (h >> 8) << (8 * (i & 3));
      if (i < 4) { w.tab[0] |= lo8; w.tab[2] |= hi8; } else { w.tab[1] |= lo8; w.tab[3] |= hi8; }
    }
  }
  const float beta_k = reinterpret_cast<const float*>(smem + S::kCent + 192)[0];
  const float beta_v = reinterpret_cast<const float*>(smem + S::kCent + 192)[1];
  const float k_scale_log2 = p.scale_log2 * beta_k;
  const int my_col = PSPLIT ? (g & 3) : g;
  const bool col_ok = my_col < group;
  uint32_t qf[8][2];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    uint2 v = *reinterpret_cast<const uint2*>(qs + (col_ok ? my_col : 0) * D + 32 * t + 4 * s);
    if constexpr (KPRMT) {  // the byte-permute path delivers (odd, even) pairs
      v.x = prmt(v.x, v.x, 0x1032);
      v.y = prmt(v.y, v.y, 0x1032);
    }
    qf[s][0] = col_ok ? v.x : 0u;
    qf[s][1] = col_ok ? v.y : 0u;
  }
  float m_run[2] = {kNegBig, kNegBig}, l_run[2] = {0.f, 0.f};
  float oacc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) oacc[i][c] = 0.f;

#pragma unroll 1
  while (tile < t1) {
    FastMid mid;
    mid.nk_lo = cur.nk_lo; mid.nk_hi = cur.nk_hi;
    mid.nv_lo = cur.nv_lo; mid.nv_hi = cur.nv_hi;
    fast_keys<KPRMT>(w, cur.k, qf, mid);
    fast_pair_values(cur.v[0], cur.v[1], cur.v[2], cur.v[3], mid);
    const int n_valid = len - tile * 16;
    tile += kDirThreads / 32;
    if (tile < t1) load(tile, cur);  // under the softmax and the value product
    if (n_valid >= 16)
      fast_back<false, PSPLIT>(w, mid, g, t >= 2, 16, 16, k_scale_log2, oacc, m_run, l_run);
    else
      fast_back<true, PSPLIT>(w, mid, g, t >= 2, n_valid, n_valid, k_scale_log2, oacc, m_run, l_run);
  }

  // ---- the warps' rows meet in shared memory --------------------------------------------------------
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], o);
    l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], o);
  }
  if constexpr (PSPLIT) {  // second-term accumulators of lanes t+2 join those of lanes t
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) oacc[i][c] += __shfl_xor_sync(0xffffffffu, oacc[i][c], 2);
  }
  __syncthreads();  // nobody reads the look-up table any more
  float* out = reinterpret_cast<float*>(smem + S::kOut);
  float2* ml = reinterpret_cast<float2*>(smem + S::kMl);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int col = 2 * t + c;
    if (col >= group || (PSPLIT && t >= 2)) continue;
    float* row = out + (warp * 8 + col) * D;
#pragma unroll
    for (int i = 0; i < 8; ++i)  // cache byte b = 8g + i -> coordinates 2b, 2b + 1
      *reinterpret_cast<float2*>(row + 2 * (8 * g + i)) = make_float2(oacc[i][c], oacc[i][2 + c]);
    if (g == 0) ml[warp * 8 + col] = make_float2(m_run[c], l_run[c]);
  }
  __syncthreads();
  float* part = p.part + (int64_t(slice) * rows + row0) * (D + kPartPad);
  const float unscale = beta_v / float(1 << int(kPScaleLog2));  // the value table is c / beta_v
  for (int i = tid; i < group * D; i += kDirThreads) {
    const int col = i >> 7, d = i & 127;
    float m = kNegBig;
#pragma unroll
    for (int u = 0; u < 16; ++u) m = fmaxf(m, ml[u * 8 + col].x);
    float o = 0.f, l = 0.f;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const float2 x = ml[u * 8 + col];
      const float a = fast_exp2(x.x - m);  // a warp without a tile: 2^-big, and its row is 0
      o = fmaf(a, out[(u * 8 + col) * D + d], o);
      l = fmaf(a, x.y, l);
    }
    float* dst = part + col * (D + kPartPad);
    dst[d] = o * unscale;
    if (d == 0) *reinterpret_cast<float2*>(dst + D) = make_float2(m, l);
  }
}

template <typename TQ, bool KPRMT, bool PSPLIT>
static int launch_decode_direct_t(const DirectArgs& a, cudaStream_t stream) {
  auto kern = decode_direct_kernel<TQ, KPRMT, PSPLIT>;
  static thread_local int configured_device = -1;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(FQ_ERR_CUDA, "cudaGetDevice failed");
  if (configured_device != dev) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(DirectSmem::kBytes));
    if (e != cudaSuccess)
      return fail(FQ_ERR_CUDA, "decode: shared memory opt-in of %u bytes refused: %s",
                  DirectSmem::kBytes, cudaGetErrorString(e));
    configured_device = dev;
  }
  kern<<<dim3(a.n_splits, a.hkv, a.seqs), kDirThreads, DirectSmem::kBytes, stream>>>(a);
  return check_launch("decode kernel launch");
}

template <typename TQ>
static int launch_decode_direct_q(const DirectArgs& a, cudaStream_t stream) {
  const bool split = a.hq / a.hkv <= 4;  // two-term weights ride in the idle columns
  if (a.nck <= 8)
    return split ? launch_decode_direct_t<TQ, true, true>(a, stream)
                 : launch_decode_direct_t<TQ, true, false>(a, stream);
  return split ? launch_decode_direct_t<TQ, false, true>(a, stream)
               : launch_decode_direct_t<TQ, false, false>(a, stream);
}

int launch_decode_direct(const DirectArgs& a, int dtype, cudaStream_t stream) {
  return dtype == FQ_BF16 ? launch_decode_direct_q<__nv_bfloat16>(a, stream)
                          : launch_decode_direct_q<__half>(a, stream);
}

}  // namespace fq
