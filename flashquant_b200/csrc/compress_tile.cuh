// Many vectors of head_dim 128: the products on tcgen05 with 128-vector tiles.  Included by compress.cu.
//
// The element-wise work around the products bounds the compressor (about 22 instructions per
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
// Measured (per call): 8192 tokens x 8 heads, two-stage keys: 144 -> 56 us; 262 144 vectors of one source
// 124 -> 56 us (1.5 TB/s); 8000 vectors 13.3 -> 8.3 us.  At 262 144 vectors the schedulers issue in 46 % of
// the cycles (27 M warp instructions); the rest is the two groups meeting in the same phase, and the 32
// lines that every 16-byte load of a row per thread touches (load/store wavefronts 51 % of peak).
#pragma once

namespace fq {

constexpr int kTileThreads = 512;
constexpr int kTileGroup = 256;
constexpr int kTileVecs = 128;
constexpr uint32_t kTileSlab = 128 * 16;        // one 8-element k chunk of 128 matrix rows
constexpr uint32_t kTilePlane = 128 * 128 * 2;  // one fp16 plane of a matrix, [k chunk][row][16 B]

template <bool QJL>
struct TileSmem {
  static constexpr uint32_t kMats = QJL ? 3 : 1;
  static constexpr uint32_t kBnd = kMats * 2 * kTilePlane;  // [2][16] f32
  static constexpr uint32_t kCent = kBnd + 32 * 4;          // [16] hi | lo' << 16
  static constexpr uint32_t kPart = kCent + 16 * 4;         // [2 groups][|x|^2, gamma^2][2 halves][128]
  static constexpr uint32_t kBar = kPart + 2 * 2 * 2 * 128 * 4;
  static constexpr uint32_t kBytes = kBar + 32;
};

__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kTileGroup) : "memory");
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

// 4 * index of y in the boundary table at `sb`; b3, b7, b11 are the table's entries
__device__ __forceinline__ uint32_t bucket_offset(float y, const unsigned char* sb, float b3, float b7,
                                                  float b11) {
  const bool up = y > b7;
  uint32_t off = up ? 32u : 0u;
  off += y > (up ? b11 : b3) ? 16u : 0u;
  off += y > *reinterpret_cast<const float*>(sb + off + 4) ? 8u : 0u;
  off += y > *reinterpret_cast<const float*>(sb + off) ? 4u : 0u;
  return off;
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
    if (p.slots) {
      slot = p.slot64 ? reinterpret_cast<const int64_t*>(p.slots)[tok]
                      : int64_t(reinterpret_cast<const int32_t*>(p.slots)[tok]);
      if (slot >= p.num_slots) slot = -1;
    } else {
      slot = p.seg_len ? segment_row(p, tok) : int64_t(tok);
    }
  };
  fetch(item);  // on its way while the matrices are laid out

  if (warp == 0) tmem_alloc(holder, 512);
  if (tid == 0) {
    mbar_init(bars, 1);
    mbar_init(bars + 1, 1);
    mbar_fence_init();
  }
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

#pragma unroll 1
  for (; item < n_items; item += stride) {
    const int s = item >= n_tiles;
    const bool two_stage = QJL && s == 0;
    const unsigned char* sb = smem + S::kBnd + 64 * s;
    const int64_t slot_now = slot;
    const int head_now = head;

    // ---- |x| over both halves, x_hat as hi / lo' planes --------------------------------------------
    float ss0 = 0.f, ss1 = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float2 f = f2_unpack(raw.pair(i));
      ss0 = fmaf(f.x, f.x, ss0);
      ss1 = fmaf(f.y, f.y, ss1);
    }
    part[128 * half] = ss0 + ss1;
    group_sync(group);
    const float nrm = sqrtf(part[0] + part[128]);
    // one reciprocal per vector instead of a division per coordinate: x_hat may differ from
    // x / (n + 1e-10) in the last bit, far inside the rounding of the contraction
    const float inv = 1.f / (nrm + 1e-10f);
    {
      const uint64_t sc = f2_pack(inv, inv), sc_lo = f2_pack(inv * kLoScale, inv * kLoScale);
      uint32_t hi[32], lo[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) split_pair(raw.pair(i), sc, sc_lo, hi[i], lo[i]);
      tmem_st32_async(a_mine, hi);
      tmem_st32_async(a_mine + 64, lo);
    }
    if (!two_stage) fetch(item + stride);  // under the product and the rest of this item
    product(0);
    await();

    // ---- codes --------------------------------------------------------------------------------------
    const float b3 = reinterpret_cast<const float*>(sb)[3], b7 = reinterpret_cast<const float*>(sb)[7],
                b11 = reinterpret_cast<const float*>(sb)[11];
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
      for (int i = 0; i < 16; ++i) off[i] = bucket_offset(__uint_as_float(y[i]), sb, b3, b7, b11);
      // byte = even coordinate << 4 | odd coordinate; off = 4 * index
#pragma unroll
      for (int i = 0; i < 8; ++i)
        w[2 * c + (i >> 2)] |= ((off[2 * i] << 2) | (off[2 * i + 1] >> 2)) << (8 * (i & 3));
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
    if (slot_now >= 0) {
      if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
      } else if ((reinterpret_cast<uintptr_t>(dst) & 3) == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) reinterpret_cast<uint32_t*>(dst)[i] = w[i];
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) reinterpret_cast<uint16_t*>(dst)[i] = uint16_t(w[i >> 1] >> (16 * (i & 1)));
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
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t y[32], w = 0u;
          tmem_ld32_async(d_mine + 32 * c, y);
          tc_wait_ld(y);
#pragma unroll
          for (int i = 0; i < 32; ++i) w |= __uint_as_float(y[i]) >= 0.f ? 1u << i : 0u;
          if (slot_now >= 0) sign[c] = w;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

template <int DT, bool QJL>
static int launch_compress_tile(const CompressArgs& a, int64_t n_vec, int sm_count, cudaStream_t stream) {
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
