// Many vectors of head_dim 128: the products on tcgen05 with 128-vector tiles.  Included by compress.cu.
//
// The element-wise work around the products bounds the compressor (about 28 instructions per
// coordinate: split into fp16 terms, bucketize, pack), and the warp-per-tile kernel could not overlap it
// with its own `mma.sync` chain: 8 warps per SM, tensor pipe 35 % busy.  Here the products leave the
// warps altogether.  A CTA of 512 threads is two groups of 256; a group owns a tile of 128
// vectors of one source, two threads per vector (64 coordinates each):
//   load -> |x| -> x_hat as hi / lo' fp16 planes -> TMEM (A operand, 2 x 64 columns)
//   24 MMAs 128x128x16 against the resident hi / lo' planes of the matrix -> D (128 columns)
//   D -> registers -> codes; two-stage keys go round twice more (codes -> centroids -> x_tilde ->
//   residual -> signs) with the vector kept in registers.
// While one group waits for its products or its loads the other computes.  The arithmetic is that of
// the other kernels: hi lo' + lo' hi is accumulated first, and the first hi hi MMA scales that sum by 2^-11
// (scale-input-d), so one accumulator does.
//
// Codes and signs next to a decision are left to the arithmetic of the 16-row kernels (compress_recheck.cuh): a
// group notes such vectors and computes them again, 16 at a time, when its items are done.  (As a
// call inside the loop it cost 24 us of 262 144 vectors in spilled registers.)
//
// Measured (per call): 8192 tokens x 8 heads, two-stage keys: 143 -> 63 us; 262 144 vectors of one source
// 127 -> 69 us (1.3 TB/s); 8000 vectors 14 -> 11.7 us.  Of the 69 us the order of the sum of squares takes 2,
// the distances to the boundaries 5, the recheck 3.  Two-stage fp32 input spills 32 bytes.
#pragma once

namespace fq {

constexpr int kTileThreads = 512;
constexpr int kTileGroup = 256;
constexpr int kTileVecs = 128;
constexpr uint32_t kTileSlab = 128 * 16;        // one 8-element k chunk of 128 matrix rows
constexpr uint32_t kTilePlane = 128 * 128 * 2;  // one fp16 plane of a matrix, [k chunk][row][16 B]
constexpr int kTileLd = 128 + 8;                // halves per row of a recheck's left operand
constexpr uint32_t kTileXch = 2 * 16 * kTileLd * 2;
constexpr int kTileList = 512;   // vectors a group can note; if there are more, it rechecks all of its own

template <bool QJL>
struct TileSmem {
  static constexpr uint32_t kMats = QJL ? 3 : 1;
  static constexpr uint32_t kBnd = kMats * 2 * kTilePlane;  // [2][16] f32
  static constexpr uint32_t kCent = kBnd + 32 * 4;          // [16] hi | lo' << 16
  static constexpr uint32_t kPart = kCent + 16 * 4;         // [2 groups][|x|^2, gamma^2][2 halves][128]
  // per group: [16][128] partial sums of |x|^2; in a recheck the left operand's hi and lo' rows
  static constexpr uint32_t kXch = kPart + 2 * 2 * 2 * 128 * 4;
  static constexpr uint32_t kList = kXch + 2 * kTileXch;  // [2 groups][kTileList] vectors noted for a recheck
  static constexpr uint32_t kBar = kList + 2 * kTileList * 8;
  static constexpr uint32_t kBytes = kBar + 32;
};
static_assert(TileSmem<true>::kBytes <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kTileGroup) : "memory");
}
__device__ __forceinline__ float min_abs(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// D = A[tmem] * B[smem] + D * 2^-11
__device__ __forceinline__ void umma_ts_scale11(bool leader, uint32_t d_tmem, uint32_t a_tmem,
                                                uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "setp.ne.b32 q, %4, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, 11;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(uint32_t(leader))
      : "memory");
}

// D = A B with A (hi, lo' planes at a_tmem, a_tmem + 64) and the matrix planes at shared address b
__device__ __forceinline__ void tile_product(bool leader, uint32_t d_tmem, uint32_t a_tmem, uint32_t b) {
  constexpr uint32_t kIdesc = umma_idesc(128, 128, false);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
    umma_ts(leader, d_tmem, a_tmem + 64 + 8 * ks, smem_desc(b + 2 * ks * kTileSlab, kTileSlab, 128),
            kIdesc, ks > 0);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
    umma_ts(leader, d_tmem, a_tmem + 8 * ks,
            smem_desc(b + kTilePlane + 2 * ks * kTileSlab, kTileSlab, 128), kIdesc, true);
  umma_ts_scale11(leader, d_tmem, a_tmem, smem_desc(b, kTileSlab, 128), kIdesc);
#pragma unroll
  for (int ks = 1; ks < 8; ++ks)
    umma_ts(leader, d_tmem, a_tmem + 8 * ks, smem_desc(b + 2 * ks * kTileSlab, kTileSlab, 128), kIdesc,
            true);
}

// Two coordinates times s as packed hi and lo' words; s_lo = 2048 s, so that
// lo' = fp16(2048 v - 2048 hi) has the one rounding it should have (2048 v is v with another exponent).
__device__ __forceinline__ void split_pair(uint64_t x, uint64_t s, uint64_t s_lo, uint32_t& hi,
                                           uint32_t& lo) {
  const float2 v = f2_unpack(f2_mul(x, s));
  hi = pack_half2(v.x, v.y);
  const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  const float2 l = f2_unpack(f2_fma(f2_pack(h.x, h.y), f2_pack(-kLoScale, -kLoScale), f2_mul(x, s_lo)));
  lo = pack_half2(l.x, l.y);
}

// A thread's 64 coordinates as they were loaded: words of two 16-bit values, or of one float.
template <int DT>
struct TileRaw {
  static constexpr int kWords = DT == FQ_F32 ? 64 : 32;
  uint32_t w[kWords];
  __device__ __forceinline__ uint64_t pair(int i) const {
    if constexpr (DT == FQ_F32) {
      return f2_pack(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
    } else if constexpr (DT == FQ_BF16) {
      return f2_pack(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      return f2_pack(f.x, f.y);
    }
  }
  // the same, not to be kept unpacked for a later use of pair(i) (64 registers)
  __device__ __forceinline__ float2 once(int i) const {
    TileRaw r;
    constexpr int kPer = DT == FQ_F32 ? 2 : 1;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      r.w[k] = w[kPer * i + k];
      if constexpr (DT != FQ_F32) asm volatile("" : "+r"(r.w[k]));
    }
    return f2_unpack(r.pair(0));
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = 0u;
  }
  // 16-bit sources need only be aligned to four elements
  __device__ __forceinline__ void load(const void* src, bool wide) {
    if (wide) {
#pragma unroll
      for (int i = 0; i < kWords / 4; ++i) {
        const uint4 v = reinterpret_cast<const uint4*>(src)[i];
        w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kWords / 2; ++i) {
        const uint2 v = reinterpret_cast<const uint2*>(src)[i];
        w[2 * i] = v.x; w[2 * i + 1] = v.y;
      }
    }
  }
};

// 4 * index of y in the boundary table at `sb`; b3, b7, b11 are the table's entries.  `least`: smallest
// distance to a boundary (the two around y are among the four it is compared with)
__device__ __forceinline__ uint32_t bucket_offset(float y, const unsigned char* sb, float b3, float b7,
                                                  float b11, float& least) {
  const float d7 = y - b7, d3 = y - (d7 > 0.f ? b11 : b3);
  uint32_t off = d7 > 0.f ? 32u : 0u;
  off += d3 > 0.f ? 16u : 0u;
  const float d1 = y - *reinterpret_cast<const float*>(sb + off + 4);
  off += d1 > 0.f ? 8u : 0u;
  const float d0 = y - *reinterpret_cast<const float*>(sb + off);
  off += d0 > 0.f ? 4u : 0u;
  least = min_abs(min_abs(least, d7, d3), d1, d0);
  return off;
}
// code byte of two offsets: even coordinate << 4 | odd coordinate
__device__ __forceinline__ uint32_t code_byte(uint32_t even, uint32_t odd) {
  return (even << 2) | (odd >> 2);
}

// Stage a matrix as hi / lo' operand planes, plane[n][k] = get(n, k).  kRows: a row is contiguous in k, so a
// warp takes 8 rows x 32 k (whole lines; its stores cover all banks), else n runs along the lanes.  (One row
// per lane and 512 bytes between lanes took 9 us per matrix: every load touched 32 lines.)
template <bool kRows, typename Get>
__device__ __forceinline__ void stage_planes(unsigned char* dst, int tid, Get get) {
#pragma unroll 2
  for (int i = tid; i < 128 * 16; i += kTileThreads) {
    const int n = kRows ? (i & 7) | ((i >> 5 & 15) << 3) : i & 127;
    const int c = kRows ? (i >> 3 & 3) | (i >> 9 << 2) : i >> 7;
    float v[8];
    get(n, 8 * c, v);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      split_pair(f2_pack(v[2 * k], v[2 * k + 1]), f2_pack(1.f, 1.f), f2_pack(kLoScale, kLoScale), hi[k],
                 lo[k]);
    unsigned char* at = dst + c * kTileSlab + n * 16;
    *reinterpret_cast<uint4*>(at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(at + kTilePlane) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}
__device__ __forceinline__ void load_row8(const float* src, float (&v)[8]) {
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = src[k];
  }
}

template <int DT, bool QJL>
__global__ void __launch_bounds__(kTileThreads, 1) compress_tile_kernel(CompressArgs p) {
  using T = typename Elem<DT>::type;
  using S = TileSmem<QJL>;
  constexpr int D = 128;
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBar);
  uint32_t* holder = reinterpret_cast<uint32_t*>(smem + S::kBar + 16);
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int group = warp >> 3;
  const int half = (warp >> 2) & 1;            // coordinates 64 half ..
  const int row = (warp & 3) * 32 + lane;      // vector of the tile = TMEM lane

  const uint32_t n_vec = uint32_t(p.n_tokens * p.heads), heads = uint32_t(p.heads);
  const uint32_t n_tiles = (n_vec + kTileVecs - 1) / kTileVecs;
  const uint32_t n_items = n_tiles * uint32_t(p.n_src);  // all tiles of source 0, then of source 1
  const uint32_t stride = 2 * gridDim.x;
  uint32_t item = blockIdx.x + uint32_t(group) * gridDim.x;

  bool wide = true;
  if constexpr (DT != FQ_F32)
    wide = (p.token_stride & 7) == 0 && ((reinterpret_cast<uintptr_t>(p.src[0]) |
                                          reinterpret_cast<uintptr_t>(p.src[p.n_src - 1])) & 15) == 0;
  // row that token tok goes to, below 0 for none
  auto row_of = [&](uint32_t tok) -> int64_t {
    if (!p.slots) return p.seg_len ? segment_row(p, tok) : int64_t(tok);
    const int64_t slot = p.slot64 ? reinterpret_cast<const int64_t*>(p.slots)[tok]
                                  : int64_t(reinterpret_cast<const int32_t*>(p.slots)[tok]);
    return slot < p.num_slots ? slot : -1;
  };
  // the thread's vector of work item `it`
  TileRaw<DT> raw;
  int64_t slot = -1;
  int head = 0;
  auto fetch = [&](uint32_t it) {
    const int s = it >= n_tiles;
    const uint32_t vec = (s ? it - n_tiles : it) * kTileVecs + row;
    slot = -1;
    head = 0;
    if (it >= n_items || vec >= n_vec) {
      raw.clear();
      return;
    }
    const uint32_t tok = vec / heads;
    head = int(vec - tok * heads);
    raw.load(static_cast<const T*>(p.src[s]) + int64_t(tok) * p.token_stride + head * D + 64 * half,
             wide);
    slot = row_of(tok);
  };
  fetch(item);  // on its way while the matrices are laid out

  if (warp == 0) tmem_alloc(holder, 512);
  if (tid == 0) {
    mbar_init(bars, 1);
    mbar_init(bars + 1, 1);
    mbar_fence_init();
  }
  if (tid < 2) reinterpret_cast<uint32_t*>(smem + S::kBar + 20)[tid] = 0;
  if (p.rot_split) {
    stage_planes<false>(smem, tid, [&](int n, int k0, float (&v)[8]) {
      const float* src = ((n & 1) ? p.mat_b : p.mat_a) + k0 * (D / 2) + (n >> 1);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = src[k * (D / 2)];
    });
  } else {
    stage_planes<true>(smem, tid, [&](int n, int k0, float (&v)[8]) { load_row8(p.mat_a + n * D + k0, v); });
  }
  if constexpr (QJL) {
    stage_planes<false>(smem + 2 * kTilePlane, tid, [&](int n, int k0, float (&v)[8]) {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = p.mat_a[(k0 + k) * D + n];
    });
    stage_planes<true>(smem + 4 * kTilePlane, tid,
                       [&](int n, int k0, float (&v)[8]) { load_row8(p.qjl + n * D + k0, v); });
  }
  if (tid < 32) {
    const int s = tid >> 4, i = tid & 15;
    const int src = s < p.n_src ? s : 0;
    reinterpret_cast<float*>(smem + S::kBnd)[tid] =
        i < p.nb[src] ? p.bnd[src][i] : __int_as_float(0x7f800000);
  }
  if (QJL && tid >= 32 && tid < 48) {
    const int i = tid - 32;
    __half h, l;
    split_hi_lo(i <= p.nb[0] ? p.cent0[i] : 0.f, h, l);
    reinterpret_cast<uint32_t*>(smem + S::kCent)[i] = pack_h2(h, l);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_relinquish();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(holder);

  const uint32_t d_tmem = tmem + 256 * group, a_tmem = d_tmem + 128;
  const uint32_t lane_base = uint32_t(warp & 3) << 21;  // this warp's 32 TMEM lanes
  const uint32_t d_mine = d_tmem + lane_base + 64 * half;
  const uint32_t a_mine = a_tmem + lane_base + 32 * half;
  const uint32_t planes = smem_u32(smem);
  float* part = reinterpret_cast<float*>(smem + S::kPart) + group * 512 + row;
  float* xch = reinterpret_cast<float*>(smem + S::kXch + group * kTileXch) + row;
  uint2* list = reinterpret_cast<uint2*>(smem + S::kList) + group * kTileList;  // vector | source << 31, |x|
  uint32_t* listed = reinterpret_cast<uint32_t*>(smem + S::kBar + 20) + group;
  uint64_t* bar = bars + group;
  uint32_t parity = 0;
  bool dead = false;

  // A is in TMEM: one warp of the group issues the product with matrix m, all wait for it.  A wait that
  // runs out is not repeated; the rows then get NaN for a norm.
  auto product = [&](int m) {
    tc_wait_st();
    tc_fence_before();
    group_sync(group);
    if ((warp & 7) == 0) {
      tc_fence_after();
      const bool leader = elect_one();
      tile_product(leader, d_tmem, a_tmem, planes + m * 2 * kTilePlane);
      umma_commit_if(leader, bar);
    }
  };
  auto await = [&]() {
    if (!dead) dead = !mbar_wait(bar, parity);
    parity ^= 1u;
    __syncwarp();
    tc_fence_after();
  };

  // This row of the item, if `near`: into the list.
  auto note = [&](bool near, int s, float nrm) {
    const uint32_t rows = __ballot_sync(0xffffffffu, near);
    if (rows == 0) return;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(listed, uint32_t(__popc(rows)));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(rows & ((1u << lane) - 1));
    if (near && at < kTileList) {
      const uint32_t vec = (item - (s ? n_tiles : 0u)) * kTileVecs + row;
      list[at] = make_uint2(vec | uint32_t(s) << 31, __float_as_uint(nrm));
    }
  };
  // The group's list, 16 vectors at a time, by the arithmetic of compress_coop_kernel: a warp has 16 columns.
  auto work_off = [&]() {
    group_sync(group);
    uint32_t n = *const_cast<volatile uint32_t*>(listed);
    const uint32_t first = blockIdx.x + uint32_t(group) * gridDim.x;
    const bool all = n > kTileList;
    if (all) n = (n_items - first + stride - 1) / stride * kTileVecs;
    const int wg = warp & 7, g = lane >> 2, t = lane & 3;
    const int j = lane >> 3, r8 = lane & 7;  // ldmatrix: lanes 8j .. give the rows of matrix j
    __half* a_hi = reinterpret_cast<__half*>(smem + S::kXch + group * kTileXch);
    __half* a_lo = a_hi + 16 * kTileLd;
    float* gpart = reinterpret_cast<float*>(smem + S::kPart) + group * 512;  // [8 warps][16]
    const uint32_t a_lane = smem_u32(a_hi + ((j & 1) * 8 + r8) * kTileLd + 8 * (j >> 1));
    const uint32_t b_lane = planes + (j >> 1) * kTilePlane + (j & 1) * kTileSlab + (16 * wg + r8) * 16;
    auto chain = [&](int m, float(&acc)[2][4]) {
      float hi[2][4] = {}, co[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t xh[4], xl[4], b[4];
        ldmatrix_x4(xh, a_lane + 32 * ks);
        ldmatrix_x4(xl, a_lane + 32 * kTileLd + 32 * ks);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          ldmatrix_x4(b, b_lane + m * 2 * kTilePlane + 2 * ks * kTileSlab + i * 128);
          mma_f16(hi[i], xh[0], xh[1], xh[2], xh[3], b[0], b[1]);
          mma_f16(co[i], xh[0], xh[1], xh[2], xh[3], b[2], b[3]);
          mma_f16(co[i], xl[0], xl[1], xl[2], xl[3], b[0], b[1]);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = fmaf(co[i][c], kLoUnscale, hi[i][c]);
    };
    // entry e of the list (zeros beyond the last): source, its vector's elements, destination row and head
    struct Entry {
      int s, head;
      float nrm;
      const T* x;
      int64_t slot;
    };
    auto entry = [&](uint32_t e) {
      Entry v{0, 0, 0.f, nullptr, -1};
      if (e >= n) return v;
      uint32_t vec;
      if (all) {
        const uint32_t it = first + e / kTileVecs * stride;
        v.s = it >= n_tiles;
        vec = (v.s ? it - n_tiles : it) * kTileVecs + e % kTileVecs;
        if (vec >= n_vec) return v;
      } else {
        const uint2 w = list[e];
        v.s = int(w.x >> 31);
        vec = w.x & 0x7fffffffu;
        v.nrm = __uint_as_float(w.y);
      }
      const uint32_t tok = vec / heads;
      v.slot = row_of(tok);
      if (v.slot < 0) return v;
      v.head = int(vec - tok * heads);
      if (all) v.nrm = *reinterpret_cast<const float*>(p.norm[v.s] + v.slot * p.norm_row_stride + v.head * 4);
      v.x = static_cast<const T*>(p.src[v.s]) + int64_t(tok) * p.token_stride + v.head * D;
      return v;
    };
    auto store_planes = [&](int r, int col, float2 v) {
      uint32_t hi, lo;
      split_words(v, hi, lo);
      *reinterpret_cast<uint32_t*>(a_hi + r * kTileLd + col) = hi;
      *reinterpret_cast<uint32_t*>(a_lo + r * kTileLd + col) = lo;
    };
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += 16) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const Entry v = entry(base + wg + 8 * i);
        const float inv = 1.f / (v.nrm + 1e-10f);
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        if (v.x) load4(v.x + 4 * lane, x);
        store_planes(wg + 8 * i, 4 * lane, make_float2(x[0] * inv, x[1] * inv));
        store_planes(wg + 8 * i, 4 * lane + 2, make_float2(x[2] * inv, x[3] * inv));
      }
      group_sync(group);
      const Entry to[2] = {entry(base + g), entry(base + g + 8)};
      float acc[2][4];
      chain(0, acc);
      uint32_t off[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float* sb = reinterpret_cast<const float*>(smem + S::kBnd) + 16 * to[k].s;
          off[i][2 * k] = 4 * bucketize15(acc[i][2 * k], sb);
          off[i][2 * k + 1] = 4 * bucketize15(acc[i][2 * k + 1], sb);
          uint32_t w = code_byte(off[i][2 * k], off[i][2 * k + 1]) << (8 * t);
          w |= __shfl_xor_sync(0xffffffffu, w, 1);
          w |= __shfl_xor_sync(0xffffffffu, w, 2);
          if (t == 0 && to[k].slot >= 0)
            store_code_word(p.code[to[k].s] + to[k].slot * p.code_row_stride +
                                int64_t(to[k].head) * p.code_head_stride + 8 * wg + 4 * i, w);
        }
      group_sync(group);
      if constexpr (QJL) {
        const unsigned char* cent = smem + S::kCent;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint32_t e = *reinterpret_cast<const uint32_t*>(cent + off[i][2 * k]);
            const uint32_t o = *reinterpret_cast<const uint32_t*>(cent + off[i][2 * k + 1]);
            const int at = (g + 8 * k) * kTileLd + 16 * wg + 8 * i + 2 * t;
            *reinterpret_cast<uint32_t*>(a_hi + at) = prmt(e, o, 0x5410);
            *reinterpret_cast<uint32_t*>(a_lo + at) = prmt(e, o, 0x7632);
          }
        group_sync(group);
        chain(1, acc);
        group_sync(group);
        float ss[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int col = 16 * wg + 8 * i + 2 * t;
            const float2 f = to[k].x ? load_pair(to[k].x + col) : make_float2(0.f, 0.f);
            const float2 r = make_float2(fmaf(-acc[i][2 * k], to[k].nrm, f.x),
                                         fmaf(-acc[i][2 * k + 1], to[k].nrm, f.y));
            ss[k] = fmaf(r.x, r.x, fmaf(r.y, r.y, ss[k]));
            store_planes(g + 8 * k, col, r);
          }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], 1);
          ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], 2);
          if (t == 0) gpart[16 * wg + g + 8 * k] = ss[k];
        }
        group_sync(group);
        chain(2, acc);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint32_t b = 0u;
#pragma unroll
          for (int i = 0; i < 2; ++i)
            b |= ((acc[i][2 * k] >= 0.f ? 1u : 0u) | (acc[i][2 * k + 1] >= 0.f ? 2u : 0u)) << (8 * i + 2 * t);
          b |= __shfl_xor_sync(0xffffffffu, b, 1);
          b |= __shfl_xor_sync(0xffffffffu, b, 2);
          if (t == 0 && to[k].slot >= 0 && to[k].s == 0) {
            *reinterpret_cast<uint16_t*>(p.sign + to[k].slot * p.sign_row_stride + to[k].head * (D / 8) +
                                         2 * wg) = uint16_t(b);
            if (wg == 0) {
              float sum = 0.f;
#pragma unroll
              for (int w = 0; w < 8; ++w) sum += gpart[16 * w + g + 8 * k];
              *reinterpret_cast<float*>(p.gam + to[k].slot * p.gam_row_stride + to[k].head * 4) = sqrtf(sum);
            }
          }
        }
        group_sync(group);
      }
    }
  };

#pragma unroll 1
  for (; item < n_items; item += stride) {
    const int s = item >= n_tiles;
    const bool two_stage = QJL && s == 0;
    const unsigned char* sb = smem + S::kBnd + 64 * s;
    const int64_t slot_now = slot;
    const int head_now = head;

    // ---- |x| over both halves, in the order of the 16-row kernel that was made for such a call ------
    if (p.sum_by_quads) {
      // compress_kernel: four sums t over the k-steps 0 .. 7, columns 2t, 2t+1, 2t+8, 2t+9 of each
      float q[4] = {0.f, 0.f, 0.f, 0.f};
      auto add = [&]() {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 a = raw.once(8 * ks + t), b = raw.once(8 * ks + 4 + t);
            q[t] = fmaf(a.x, a.x, fmaf(a.y, a.y, fmaf(b.x, b.x, fmaf(b.y, b.y, q[t]))));
          }
      };
      if (half == 0) {
        add();
#pragma unroll
        for (int t = 0; t < 4; ++t) xch[128 * t] = q[t];
      }
      group_sync(group);
      if (half == 1) {
#pragma unroll
        for (int t = 0; t < 4; ++t) q[t] = xch[128 * t];
        add();
        part[0] = (q[0] + q[1]) + (q[2] + q[3]);
      }
    } else {
      // compress_coop_kernel: 32 sums of four, then halving
      float q[16];
#pragma unroll
      for (int l = 0; l < 16; ++l) {
        const float2 a = raw.once(2 * l), b = raw.once(2 * l + 1);
        q[l] = fmaf(b.y, b.y, fmaf(b.x, b.x, fmaf(a.y, a.y, a.x * a.x)));
      }
      if (half == 1) {
#pragma unroll
        for (int l = 0; l < 16; ++l) xch[128 * l] = q[l];
      }
      group_sync(group);
      if (half == 0) {
#pragma unroll
        for (int l = 0; l < 16; ++l) q[l] += xch[128 * l];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
          for (int l = 0; l < o; ++l) q[l] += q[l + o];
        part[0] = q[0];
      }
    }
    group_sync(group);
    // ---- x_hat as hi / lo' planes ----------------------------------------------------------------
    const float nrm = sqrtf(part[0]);
    // one reciprocal per vector instead of a division per coordinate: x_hat may differ from
    // x / (n + 1e-10) in the last bit, far inside the rounding of the contraction
    const float inv = 1.f / (nrm + 1e-10f);
    {
      const uint64_t sc = f2_pack(inv, inv), sc_lo = f2_pack(inv * kLoScale, inv * kLoScale);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) split_pair(raw.pair(16 * c + i), sc, sc_lo, hi[i], lo[i]);
        tmem_st16_async(a_mine + 16 * c, hi);
        tmem_st16_async(a_mine + 64 + 16 * c, lo);
      }
    }
    if (!two_stage) fetch(item + stride);  // under the product and the rest of this item
    product(0);
    await();

    // ---- codes --------------------------------------------------------------------------------------
    const float b3 = reinterpret_cast<const float*>(sb)[3], b7 = reinterpret_cast<const float*>(sb)[7],
                b11 = reinterpret_cast<const float*>(sb)[11];
    float least = 1.f;
    uint8_t* dst = p.code[s] + slot_now * p.code_row_stride + int64_t(head_now) * p.code_head_stride +
                   32 * half;
    uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
    for (int c = 0; c < 4; ++c) {  // 16 coordinates each
      uint32_t y[16];
      tmem_ld16_async(d_mine + 16 * c, y);
      tc_wait_ld(y);
      uint32_t off[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) off[i] = bucket_offset(__uint_as_float(y[i]), sb, b3, b7, b11, least);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        w[2 * c + (i >> 2)] |= code_byte(off[2 * i], off[2 * i + 1]) << (8 * (i & 3));
      if constexpr (QJL) {
        if (two_stage) {  // the centroids are the next product's A (the last one is done with it)
          uint32_t a[8], b[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t e = *reinterpret_cast<const uint32_t*>(smem + S::kCent + off[2 * i]);
            const uint32_t o = *reinterpret_cast<const uint32_t*>(smem + S::kCent + off[2 * i + 1]);
            a[i] = prmt(e, o, 0x5410);
            b[i] = prmt(e, o, 0x7632);
          }
          tmem_st8_async(a_mine + 8 * c, a);
          tmem_st8_async(a_mine + 64 + 8 * c, b);
        }
      }
    }
    // (a zero vector's coordinates are zero in any arithmetic)
    note(least <= kNearBoundary && nrm > 0.f && slot_now >= 0, s, nrm);
    if (slot_now >= 0) {
      if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) store_code_word(dst + 4 * i, w[i]);
      }
    }
    if (half == 0 && slot_now >= 0)
      *reinterpret_cast<float*>(p.norm[s] + slot_now * p.norm_row_stride + head_now * 4) =
          dead ? __int_as_float(0x7fc00000) : nrm;

    if constexpr (QJL) {
      if (two_stage) {
        // ---- x_tilde = (c[code] Pi) n, r = x - x_tilde, gamma = |r|; r / n is the last left operand --
        product(1);
        await();
        float rs0 = 0.f, rs1 = 0.f;
        const uint64_t neg_n = f2_pack(-nrm, -nrm);
        const uint64_t sc = f2_pack(inv, inv), sc_lo = f2_pack(inv * kLoScale, inv * kLoScale);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t y[16], hi[8], lo[8];
          tmem_ld16_async(d_mine + 16 * c, y);
          tc_wait_ld(y);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t yy = f2_pack(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1]));
            const uint64_t r = f2_fma(yy, neg_n, raw.pair(8 * c + i));
            const float2 f = f2_unpack(r);
            rs0 = fmaf(f.x, f.x, rs0);
            rs1 = fmaf(f.y, f.y, rs1);
            split_pair(r, sc, sc_lo, hi[i], lo[i]);
          }
          tmem_st8_async(a_mine + 8 * c, hi);
          tmem_st8_async(a_mine + 64 + 8 * c, lo);
        }
        part[256 + 128 * half] = rs0 + rs1;
        fetch(item + stride);
        product(2);
        // ---- sign(r S^T): bit j%8 of byte j/8 is 1 for a projection >= 0 ----------------------------
        await();
        if (half == 0 && slot_now >= 0)
          *reinterpret_cast<float*>(p.gam + slot_now * p.gam_row_stride + head_now * 4) =
              dead ? __int_as_float(0x7fc00000) : sqrtf(part[256] + part[384]);
        uint32_t* sign = reinterpret_cast<uint32_t*>(p.sign + slot_now * p.sign_row_stride +
                                                     head_now * (D / 8) + 8 * half);
        least = 1.f;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t y[32], w = 0u;
          tmem_ld32_async(d_mine + 32 * c, y);
          tc_wait_ld(y);
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            w |= __uint_as_float(y[i]) >= 0.f ? 1u << i : 0u;
            least = fminf(least, fabsf(__uint_as_float(y[i])));
          }
          if (slot_now >= 0) sign[c] = w;
        }
        note(least <= kNearZero && nrm > 0.f && slot_now >= 0, s, nrm);
      }
    }
  }
  work_off();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

template <int DT, bool QJL>
static int launch_compress_tile(CompressArgs a, int64_t n_vec, bool sum_by_quads, int sm_count,
                                cudaStream_t stream) {
  a.sum_by_quads = sum_by_quads;
  using S = TileSmem<QJL>;
  auto kern = compress_tile_kernel<DT, QJL>;
  static thread_local int configured_device = -1;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(FQ_ERR_CUDA, "cudaGetDevice failed");
  if (configured_device != dev) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(S::kBytes));
    if (e != cudaSuccess)
      return fail(FQ_ERR_CUDA, "compress: shared memory opt-in of %u bytes refused: %s", S::kBytes,
                  cudaGetErrorString(e));
    configured_device = dev;
  }
  const int64_t items = (n_vec + kTileVecs - 1) / kTileVecs * a.n_src;
  const int grid = int(items < sm_count ? items : sm_count);
  kern<<<grid, kTileThreads, S::kBytes, stream>>>(a);
  return check_launch("compress kernel launch");
}

}  // namespace fq
