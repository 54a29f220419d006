// Fused TQ4 attention for many query rows: warp-specialised tcgen05 kernel, both rotations inside.
// Included by prefill.cu.
//
// A CTA owns TWO tiles of 128 query rows that attend over the same keys - two heads of a KV group
// at the same positions, or (odd groups) 256 consecutive positions of one head - and walks the keys in
// tiles of 64 tokens:
//   warps 0-3, 4-7    softmax of tile 0 / 1, one thread per row: reads its row of S from TMEM into
//                     registers and hands S back at once, applies |k| and the scale, the lazily
//                     raised reference exponent, writes the fp16 weights p |v| 2^8 to TMEM as the A
//                     operand of the value product;
//   warps 8-11/12-15  turn key / value codes into fp16 operand tiles in shared memory (global ->
//                     registers two tiles ahead -> look-up or byte permute -> store), once for both
//                     query tiles;
//   warp 16 / 17      issues the MMAs of tile 0 / 1: S_t = Q_t K^T and O_t += P_t V.  (One warp for
//                     both took them in a fixed order, and a tile whose weights were ready
//                     waited for the other's: 2.9 ms.)
// TMEM: S_0 S_1 (64 columns each), P_0 P_1 (32 each), Q_0 (64), O_0 O_1 (128 each).  Nothing in the
// loop is a block-wide barrier.
//
// The query rotation round(q Pi^T) is the kernel's first MMA and the back-rotation o Pi its last:
// as kernels of their own they moved every query and output row through memory twice and took
// 0.6 ms at 4 x 8192 tokens.  Both keep fp32-level accuracy on fp16 operands: a row is scaled by a power of two
// to [1, 2) and split in two fp16 terms (a query needs one: bf16 and fp16 fit), so is 8 Pi, and every
// product but lo x lo, 2^-22 of the row, is accumulated in fp32.  attention_prep_kernel writes the two
// planes of 8 Pi in the operand layout.
//
// Per 64 tokens the pair costs 1024 cycles of MMA, 1024 of exponentials (16 per cycle and SM) and
// about 1450 of shared-memory bandwidth (MMA operand reads 768: Q_0 comes from TMEM; operand stores
// 256, look-ups 128, norms 288), which bounds it.  Measured at 4 x 8192 tokens, 32 / 8 heads: 5.8 ms with one
// query tile per 256-thread CTA and block-wide barriers; 2.75 ms with this split on tiles of 128
// tokens, where the weights lay over the scores, so that softmax and MMA of a tile took turns.
#pragma once

namespace fq {

constexpr int kPpThreads = 640;
constexpr int kPpN = 64;                        // keys per tile
constexpr int kPpSlots = 3;                     // key and value operand rings
constexpr int kPpNorms = 8;                     // norm ring, see the key warps
constexpr uint32_t kPpTile = 128 * 128 * 2;     // operand tile of 128 rows
constexpr uint32_t kPpHalf = kPpTile / 2;       // ... of 64 keys or values
constexpr uint32_t kPpSlab = 128 * 16;          // one 8-element chunk of 128 rows
constexpr uint32_t kPpSlabKV = kPpN * 16;
constexpr float kPpPiScale = 8.f;               // planes hold 8 Pi

struct PairSmem {
  static constexpr uint32_t kQ = 0;                                  // Q_1; output staging of tile 1
  static constexpr uint32_t kK = kQ + kPpTile;                       // key ring ...
  static constexpr uint32_t kV = kK + kPpSlots * kPpHalf;            // ... and value ring; before and
  static constexpr uint32_t kPi = kK;                                //   after the loop the planes and
  static constexpr uint32_t kA0 = kPi + 2 * kPpTile;                 //   the query rows of tile 0
  static constexpr uint32_t kLut = kV + kPpSlots * kPpHalf;          // 256 x (32 lanes K | 32 lanes V)
  static constexpr uint32_t kNorm = kLut + 256 * 256;                // [8][nk | lv | vs][64]
  static constexpr uint32_t kRow = kNorm + kPpNorms * 3 * kPpN * 4;  // [2][128] query row scales
  static constexpr uint32_t kBar = kRow + 2 * 128 * 4;
  static constexpr uint32_t kBytes = kBar + 512;
};
static_assert(2 * kPpSlots * kPpHalf == 3 * kPpTile, "planes and query rows fit the rings");
static_assert(PairSmem::kBytes <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ ulonglong2 lds_f2x2(uint32_t a) {  // four consecutive floats
  ulonglong2 r;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(r.x), "=l"(r.y) : "r"(a));
  return r;
}

// power of two that brings x to [1, 2) (1 for zero; x finite)
__device__ __forceinline__ float pow2_to_one(float x) {
  const uint32_t e = (__float_as_uint(x) >> 23) & 0xffu;
  return e == 0u || e > 253u ? 1.f : __uint_as_float((254u - e) << 23);
}
__device__ __forceinline__ float max_abs2(uint32_t bf16x2) {
  return fmaxf(fabsf(__uint_as_float(bf16x2 << 16)), fabsf(__uint_as_float(bf16x2 & 0xffff0000u)));
}

// The scale search and the planes of 8 Pi for the launch that follows: block 0 finds (or finds again)
// beta_k, beta_v; blocks 1 .. 4 and 5 .. 8 split the two rotations into fp16 terms in the MMA operand
// layout, [8-column chunk][row][16 B], hi plane then lo plane.
__global__ void __launch_bounds__(kScaleThreads) attention_prep_kernel(
    const float* __restrict__ cent_k, int nck, const float* __restrict__ cent_v, int ncv,
    uint32_t* __restrict__ cache, const float* __restrict__ rot_a, const float* __restrict__ rot_b,
    unsigned char* __restrict__ planes) {
  __shared__ __align__(16) unsigned char cent[kCentBytes];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (blockIdx.x > 0) {
    const int m = (blockIdx.x - 1) >> 2, i = ((blockIdx.x - 1) & 3) * kScaleThreads + tid;
    const int row = i >> 4, chunk = i & 15;
    const float* src = (m ? rot_b : rot_a) + row * 128 + chunk * 8;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float a = src[2 * k] * kPpPiScale, b = src[2 * k + 1] * kPpPiScale;
      const __half2 h = __floats2half2_rn(a, b);
      hi[k] = *reinterpret_cast<const uint32_t*>(&h);
      lo[k] = pack_half2(a - __low2float(h), b - __high2float(h));
    }
    unsigned char* dst = planes + m * (2 * kPpTile) + chunk * kPpSlab + row * 16;
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + kPpTile) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    return;
  }
  if (warp == 1) {
    const int i = lane & 15;
    float c = 0.f;
    if (lane < 16) { if (i < nck) c = cent_k[i]; } else { if (i < ncv) c = cent_v[i]; }
    stage_centroids(cent, c, nck, ncv, cache, lane);
  }
  __syncthreads();
  scale_centroid_tables(cent, nck, ncv, tid, cache);
}

// T: the queries' and outputs' type
template <typename T, bool PAGED>
__global__ void __launch_bounds__(kPpThreads, 1) prefill_pair_kernel(PrefillArgs p) {
  using S = PairSmem;
  constexpr int D = 128;
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr uint32_t kIdescS = umma_idesc(128, kPpN, false);
  constexpr uint32_t kIdescO = umma_idesc(128, D, true);
  constexpr uint32_t kIdescQ = umma_idesc(128, D, false);
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBar);
  uint64_t* k_full = bars;          // [3] key tile stored (128 arrivals)
  uint64_t* k_empty = bars + 3;     // [3] its products are complete (one commit per query tile)
  uint64_t* v_full = bars + 6;      // [3]
  uint64_t* v_empty = bars + 9;     // [3]
  uint64_t* norm_full = bars + 12;  // [8] norms of a tile stored (128 arrivals)
  uint64_t* s_full = bars + 20;     // [2] scores of query tile t complete
  uint64_t* s_free = bars + 22;     // [2] ... and read (4 warps)
  uint64_t* p_full = bars + 24;     // [2] weights of query tile t stored (4 warps)
  uint64_t* o_done = bars + 26;     // [2] value product of query tile t complete
  uint64_t* planes = bars + 28;     // planes of Pi landed (prologue, epilogue)
  uint64_t* rows_in = bars + 29;    // [2] operand rows of tile t stored (4 warps: rotated Q, split O)
  uint64_t* turned = bars + 31;     // [2] a rotation of tile t is complete (prologue, epilogue)
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 33);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int b = blockIdx.y;
  const int group = p.hq / p.hkv;
  const bool two_heads = (group & 1) == 0;
  const int rows_per_cta = two_heads ? 128 : 256;
  // the query tiles with the most keys go first: they are the slowest grid dimension
  const int m_base = (int(gridDim.z) - 1 - int(blockIdx.z)) * rows_per_cta;
  const int head0 = two_heads ? 2 * int(blockIdx.x) : int(blockIdx.x);
  const int hkv = head0 / group;

  // this sequence's query tokens and keys; ctx keys precede the first query token
  int q_first = 0, q_len = p.nq, kv_len = p.nkv, ctx = 0;
  bool clamped = false;
  if constexpr (PAGED) {
    q_first = p.cu_q[b];
    q_len = p.cu_q[b + 1] - q_first;
    kv_len = p.seq_lens[b];
    const int64_t room = p.bt_stride * int64_t(p.block_size);  // keys a block-table row can name
    if (kv_len > room) {
      kv_len = int(room);
      clamped = true;
    }
    ctx = kv_len - q_len;
    // a chunk outside the query tokens is not touched; one longer than the grid covers is cut
    const bool outside = q_first < 0 || q_len < 0 || int64_t(q_first) + q_len > p.total_q;
    if ((outside || q_len > int(gridDim.z) * rows_per_cta) && m_base == 0 && tid == 0 && p.status)
      atomicOr(p.status, FQ_DEV_BAD_LENGTH);
    if (outside || m_base >= q_len) return;  // the grid is sized for the longest chunk
  }
  const int left = q_len - m_base;
  const int all_rows = left < rows_per_cta ? left : rows_per_cta;
  int kv_end = kv_len;
  if (p.causal && ctx + m_base + all_rows < kv_end) kv_end = ctx + m_base + all_rows;
  if (kv_end < 0) kv_end = 0;
  const int n_tiles = (kv_end + kPpN - 1) / kPpN;
  auto tile_m0 = [&](int t) { return two_heads ? m_base : m_base + 128 * t; };
  auto tile_head = [&](int t) { return two_heads ? head0 + t : head0; };
  // row of q and out that query row r of tile t is
  auto io_row = [&](int t, int r) {
    return PAGED ? int64_t(q_first + tile_m0(t) + r) * p.hq + tile_head(t)
                 : (int64_t(b) * p.hq + tile_head(t)) * p.nq + tile_m0(t) + r;
  };

  // ---- set-up -----------------------------------------------------------------------------------
  if (tid == 0) {
    for (int i = 0; i < kPpSlots; ++i) {
      mbar_init(k_full + i, 128);
      mbar_init(k_empty + i, 2);
      mbar_init(v_full + i, 128);
      mbar_init(v_empty + i, 2);
    }
    for (int i = 0; i < kPpNorms; ++i) mbar_init(norm_full + i, 128);
    for (int i = 0; i < 2; ++i) {
      mbar_init(s_full + i, 1);
      mbar_init(s_free + i, 4);
      mbar_init(p_full + i, 4);
      mbar_init(o_done + i, 1);
      mbar_init(rows_in + i, 4);
      mbar_init(turned + i, 1);
    }
    mbar_init(planes, 1);
    mbar_fence_init();
    if (n_tiles > 0) {
      mbar_expect_tx(planes, 2 * kPpTile);
      bulk_g2s(smem + S::kPi, p.planes_q, kPpTile, planes);
      bulk_g2s(smem + S::kPi + kPpTile, p.planes_q + kPpTile, kPpTile, planes);
    }
  }
  if (warp == 0) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  // query rows -> fp16 operand tiles [k-chunk][row][16 B]; a bf16 row scaled to [1, 2)
  for (int i = tid; i < 2 * 128 * 16; i += kPpThreads) {  // (16 lanes share a row)
    const int t = i >> 11, r = (i >> 4) & 127, kc = i & 15;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (tile_m0(t) + r < q_len)
      v = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.q_src) + io_row(t, r) * D + kc * 8);
    if constexpr (kBf16) {
      float mx = fmaxf(fmaxf(max_abs2(v.x), max_abs2(v.y)), fmaxf(max_abs2(v.z), max_abs2(v.w)));
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float sc = pow2_to_one(mx);
      if (kc == 0) reinterpret_cast<float*>(smem + S::kRow)[t * 128 + r] = 1.f / sc;
      auto half2_of = [&](uint32_t w) {
        return pack_half2(__uint_as_float(w << 16) * sc, __uint_as_float(w & 0xffff0000u) * sc);
      };
      v = make_uint4(half2_of(v.x), half2_of(v.y), half2_of(v.z), half2_of(v.w));
    }
    *reinterpret_cast<uint4*>(smem + (t ? S::kQ : S::kA0) + kc * kPpSlab + r * 16) = v;
  }
  // tables of fp16(c / beta): beta_k folds into the score scale, beta_v into the weights.  Entry e (a
  // cache byte): 32 copies of the keys' pair, then 32 of the values', so that lane l reads bank l
  const float beta_k = p.scales[0], beta_v = p.scales[1];
  const float rbk = 1.f / beta_k, rbv = 1.f / beta_v;
  for (int i = tid; i < 256 * 16; i += kPpThreads) {
    const int e = i >> 4, hi = e >> 4, lo = e & 15;
    const bool is_v = (i & 8) != 0;
    const float* c = is_v ? p.cent_v : p.cent_k;
    const int n = is_v ? p.ncv : p.nck;
    const float rb = is_v ? rbv : rbk;
    const uint32_t v = pack_half2(hi < n ? c[hi] * rb : 0.f, lo < n ? c[lo] * rb : 0.f);
    *reinterpret_cast<uint4*>(smem + S::kLut + i * 16) = make_uint4(v, v, v, v);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_holder, 0);
  const uint32_t tm_p = tmem + 128, tm_q0 = tmem + 192, tm_o = tmem + 256;
  bool dead = false;

  if (warp >= 16) {
    // ---- MMA issue, a warp per query tile ----------------------------------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    const int t = warp - 16;
    if (t < 2 && n_tiles > 0) {
      const bool leader = elect_one();
      const uint32_t base = smem_u32(smem);
      const uint32_t q_rows = base + (t ? S::kQ : S::kA0);
      const uint32_t my_s = tmem + 64 * t, my_p = tm_p + 32 * t, my_o = tm_o + 128 * t;
      auto wait = [&](uint64_t* bar, uint32_t phase) {
        if (!dead) dead = !mbar_wait_warp(bar, phase & 1, kDefaultWaitNs);
        tc_fence_after();
        return !dead;
      };
      auto scores = [&](int j) {
        const uint32_t k = base + S::kK + (j % kPpSlots) * kPpHalf;
        if (t == 0) {
#pragma unroll
          for (int s = 0; s < D / 16; ++s)
            umma_ts(leader, my_s, tm_q0 + 8 * s, smem_desc(k + 2 * s * kPpSlabKV, kPpSlabKV, 128),
                    kIdescS, s > 0);
        } else {
#pragma unroll
          for (int s = 0; s < D / 16; ++s)
            umma_ss(leader, my_s, smem_desc(q_rows + 2 * s * kPpSlab, kPpSlab, 128),
                    smem_desc(k + 2 * s * kPpSlabKV, kPpSlabKV, 128), kIdescS, s > 0);
        }
        umma_commit_if(leader, s_full + t);
        umma_commit_if(leader, k_empty + j % kPpSlots);
      };
      auto values = [&](int j) {
        const uint32_t v = base + S::kV + (j % kPpSlots) * kPpHalf;
#pragma unroll
        for (int s = 0; s < kPpN / 16; ++s)
          umma_ts(leader, my_o, my_p + 8 * s, smem_desc(v + s * 256, 128, kPpSlabKV), kIdescO,
                  j > 0 || s > 0);
        umma_commit_if(leader, o_done + t);
        umma_commit_if(leader, v_empty + j % kPpSlots);
      };
      // q Pi^T: the query rows on both planes, into O_t.  (Here and in o Pi the small terms go first:
      // the accumulator is rounded at its full size only while the large ones are added.)
      if (wait(planes, 0)) {
#pragma unroll
        for (int s = 0; s < 2 * D / 16; ++s)
          umma_ss(leader, my_o, smem_desc(q_rows + 2 * (s & 7) * kPpSlab, kPpSlab, 128),
                  smem_desc(base + S::kPi + (s < 8 ? kPpTile : 0) + 2 * (s & 7) * kPpSlab, kPpSlab, 128),
                  kIdescQ, s > 0);
        umma_commit_if(leader, turned + t);
      }
      if (wait(rows_in + t, 0) && wait(k_full, 0)) scores(0);
#pragma unroll 1
      for (int j = 0; j < n_tiles && !dead; ++j) {
        // the next tile's scores as soon as this tile's have been read
        const int n = j + 1;
        if (n < n_tiles && wait(k_full + n % kPpSlots, n / kPpSlots) && wait(s_free + t, j)) scores(n);
        if (wait(v_full + j % kPpSlots, j / kPpSlots) && wait(p_full + t, j)) values(j);
      }
      // o Pi: the rows' second terms on the hi plane, their first (both over S, P and Q_0) on the lo
      // and then the hi plane
      if (wait(planes, 1) && wait(rows_in + t, 1)) {
#pragma unroll
        for (int s = 0; s < 3 * D / 16; ++s)
          umma_ts(leader, my_o, tmem + 128 * t + (s < 8 ? 64 : 0) + 8 * (s & 7),
                  smem_desc(base + S::kPi + (s >> 3 == 1 ? kPpTile : 0) + (s & 7) * 256, 128, kPpSlab),
                  kIdescO, s > 0);
        umma_commit_if(leader, turned + t);
      }
      if (dead && leader && p.status) atomicOr(p.status, FQ_DEV_WAIT_TIMEOUT);
    }
  } else if (warp >= 8) {
    // ---- codes -> operand tiles; warps 8-11 keys, 12-15 values ---------------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    const bool is_k = warp < 12;
    const int dt = (tid - 256) & 127, dw = dt >> 5;
    uint64_t* full = is_k ? k_full : v_full;
    uint64_t* empty = is_k ? k_empty : v_empty;
    // Lane = (quarter q of a token's 64 code bytes, token of eight): the 16-byte loads of a warp
    // cover 512 contiguous bytes, its stores 128 contiguous bytes per eight lanes.
    const int q4 = lane >> 3, tok8 = 8 * dw + (lane & 7);  // + 32 * i: token of load i
    const int row_bytes = p.hkv * (D + 8), plane_v = p.hkv * (D / 2 + 4);
    const int64_t kv_row0 = PAGED ? 0 : (int64_t(b) * p.hkv + hkv) * p.kv_stride;
    const uint8_t* codes = PAGED ? p.kv_cache + (is_k ? 0 : plane_v) + hkv * (D / 2) + 16 * q4
                                 : (is_k ? p.k_packed : p.v_packed) + kv_row0 * (D / 2) + 16 * q4;
    bool bad_page = false;
    // cache row of a token (token index in the contiguous form), -1 past the end
    auto row_of = [&](int t) -> int {
      if (t >= kv_end) return -1;
      if constexpr (!PAGED) return t;
      const int page = t / p.block_size;
      int64_t phys = p.block_table[int64_t(b) * p.bt_stride + page];
      if (phys < 0 || phys >= p.num_blocks) {  // reported, not followed
        phys = 0;
        bad_page = true;
      }
      return int(phys * p.block_size + (t - page * p.block_size));
    };
    // key warps: threads 0-63 bring |k| of the tile's tokens, 64-127 |v|
    struct Rows {
      int code[2], norm;
    };
    auto rows_of = [&](int j) {
      Rows r;
#pragma unroll
      for (int i = 0; i < 2; ++i) r.code[i] = row_of(j * kPpN + 32 * i + tok8);
      r.norm = is_k ? row_of(j * kPpN + (dt & 63)) : -1;
      return r;
    };
    struct Raw {
      uint4 w[2];
      float norm;
    };
    auto load = [&](const Rows& r) {
      Raw x;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        x.w[i] = make_uint4(0u, 0u, 0u, 0u);
        if (r.code[i] >= 0)
          x.w[i] = __ldg(reinterpret_cast<const uint4*>(
              codes + int64_t(r.code[i]) * (PAGED ? row_bytes : D / 2)));
      }
      x.norm = 0.f;
      if (r.norm >= 0) {
        if constexpr (PAGED)
          x.norm = *reinterpret_cast<const float*>(p.kv_cache + int64_t(r.norm) * row_bytes +
                                                   (dt < 64 ? 0 : plane_v) + p.hkv * (D / 2) + 4 * hkv);
        else
          x.norm = (dt < 64 ? p.k_norms : p.v_norms)[kv_row0 + r.norm];
      }
      return x;
    };
    // 8-entry key table in registers: low and high bytes of the fp16 centroids
    uint32_t tl0 = 0, tl1 = 0, th0 = 0, th1 = 0;
    const bool by_permute = is_k && p.nck <= 8;
    if (by_permute) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t h =
            uint32_t(__half_as_ushort(__float2half_rn(i < p.nck ? p.cent_k[i] * rbk : 0.f)));
        const uint32_t lo8 = (h & 0xffu) << (8 * (i & 3)), hi8 = (h >> 8) << (8 * (i & 3));
        if (i < 4) { tl0 |= lo8; th0 |= hi8; } else { tl1 |= lo8; th1 |= hi8; }
      }
    }
    const unsigned char* lut = smem + S::kLut + (is_k ? 0 : 128);
    const uint32_t lane4 = 4 * lane;
    auto look = [&](uint32_t w, uint32_t sel) {  // (byte of w) * 256 + lane4 in one permute
      return *reinterpret_cast<const uint32_t*>(lut + prmt(w, lane4, sel));
    };
    auto permuted = [&](uint32_t w) {
      // nibbles of w, low to high: odd0, even0, odd1, even1, ...
      const uint32_t la = prmt(tl0, tl1, w), ha = prmt(th0, th1, w);
      const uint32_t lb = prmt(tl0, tl1, w >> 16), hb = prmt(th0, th1, w >> 16);
      return make_uint4(prmt(la, ha, 0x4051), prmt(la, ha, 0x6273), prmt(lb, hb, 0x4051),
                        prmt(lb, hb, 0x6273));
    };
    Raw cur = load(rows_of(0)), nxt = load(rows_of(1));
    Rows rows = rows_of(2);
    // the rings hold the planes and query rows of the first rotation until it is done
    if (n_tiles > 0 && !(mbar_wait_warp(turned, 0, kDefaultWaitNs) &&
                         mbar_wait_warp(turned + 1, 0, kDefaultWaitNs)))
      dead = true;
    const float norm_scale = dt < 64 ? p.scale_log2 * beta_k : 256.f * beta_v;
#pragma unroll 1
    for (int j = 0; j < n_tiles && !dead; ++j) {
      const int slot = j % kPpSlots;
      if (j >= kPpSlots && !mbar_wait_warp(empty + slot, (j / kPpSlots - 1) & 1, kDefaultWaitNs)) {
        dead = true;
        break;
      }
      if (is_k) {
        // Norm slot j % 8 held tile j - 8.  The wait above saw the scores of tile j - 3 complete;
        // they were issued after the softmax had read the scores of tile j - 4, hence was through
        // with tile j - 5 and its norms.
        float* ns = reinterpret_cast<float*>(smem + S::kNorm) + (j % kPpNorms) * (3 * kPpN) + (dt & 63);
        if (dt < 64) {
          ns[0] = cur.norm * norm_scale;
        } else {
          ns[kPpN] = fmaxf(fast_log2(cur.norm), -40.f);
          ns[2 * kPpN] = cur.norm * norm_scale;
        }
        mbar_arrive(norm_full + j % kPpNorms);
      }
      unsigned char* dst = smem + (is_k ? S::kK : S::kV) + slot * kPpHalf + 4 * q4 * kPpSlabKV + tok8 * 16;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t w[4] = {cur.w[i].x, cur.w[i].y, cur.w[i].z, cur.w[i].w};
        uint4 o[4];
        if (by_permute) {
#pragma unroll
          for (int c = 0; c < 4; ++c) o[c] = permuted(w[c]);
        } else {  // all sixteen look-ups before the first store
#pragma unroll
          for (int c = 0; c < 4; ++c)
            o[c] = make_uint4(look(w[c], 0x5504), look(w[c], 0x5514), look(w[c], 0x5524),
                              look(w[c], 0x5534));
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(dst + c * kPpSlabKV + i * 512) = o[c];
      }
      fence_async_smem();
      mbar_arrive(full + slot);
      cur = nxt;
      nxt = load(rows);        // tile j + 2
      rows = rows_of(j + 3);
    }
    if (dead && lane == 0 && p.status) atomicOr(p.status, FQ_DEV_WAIT_TIMEOUT);
    if constexpr (PAGED) {
      if ((bad_page || clamped) && p.status) atomicOr(p.status, FQ_DEV_BAD_BLOCK_INDEX);
    }
  } else {
    // ---- softmax of query tile t, one thread per row -------------------------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
    const int t = warp >> 2, row = tid & 127;
    const int m0 = tile_m0(t);
    const int q_pos = m0 + row;
    const uint32_t lane_sel = uint32_t((warp & 3) * 32) << 16;
    const uint32_t my_s = tmem + 64 * t + lane_sel, my_p = tm_p + 32 * t + lane_sel;
    const uint32_t my_o = tm_o + 128 * t + lane_sel;
    // ---- the rotated query row: round to the query's type, then fp16 --------------------------------
    if (n_tiles > 0) {
      if (!mbar_wait_warp(turned + t, 0, kDefaultWaitNs)) dead = true;
      tc_fence_after();
      float unscale = 1.f / kPpPiScale;
      if constexpr (kBf16) unscale *= reinterpret_cast<const float*>(smem + S::kRow)[t * 128 + row];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32], h[16];
        tmem_ld32_async(my_o + 32 * c, r);
        tc_wait_ld(r);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          h[i] = pack_half2(to_f32(from_f32<T>(__uint_as_float(r[2 * i]) * unscale)),
                            to_f32(from_f32<T>(__uint_as_float(r[2 * i + 1]) * unscale)));
        if (t == 0) {
          tmem_st16_async(tm_q0 + lane_sel + 16 * c, h);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(smem + S::kQ + (4 * c + i) * kPpSlab + row * 16) =
                make_uint4(h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
        }
      }
      if (t == 0) tc_wait_st(); else fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(rows_in + t);
    }
    float m_run = -INFINITY;
    uint64_t l2 = 0;  // (0, 0)
    // one key tile; masked: it reaches past the end of the keys or the row's causal limit
    auto tile = [&](int j, auto masked) {
      const uint32_t norms = smem_u32(smem + S::kNorm) + (j % kPpNorms) * (3 * kPpN * 4);
      uint64_t s2[kPpN / 2];
      {
        uint32_t r[2][32];
#pragma unroll
        for (int c = 0; c < 2; ++c) tmem_ld32_async(my_s + 32 * c, r[c]);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tc_wait_ld(r[c]);
#pragma unroll
          for (int i = 0; i < 16; ++i)
            s2[16 * c + i] = f2_pack(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1]));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free + t);  // the next tile's scores may come
      // logit * log2e = s |k| scale; the exponent that bounds the weights adds log2 |v|
      const int lim = [&] {
        if constexpr (!decltype(masked)::value) return kPpN;
        int n = kv_end - j * kPpN;
        if (p.causal && q_pos + ctx + 1 - j * kPpN < n) n = q_pos + ctx + 1 - j * kPpN;
        return n;
      }();
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int c = 0; c < kPpN / 4; ++c) {
        const ulonglong2 nk = lds_f2x2(norms + 16 * c), lv = lds_f2x2(norms + kPpN * 4 + 16 * c);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint64_t v = f2_mul(s2[2 * c + u], u ? nk.y : nk.x);
          if constexpr (decltype(masked)::value) {
            const float2 f = f2_unpack(v);
            v = f2_pack(4 * c + 2 * u < lim ? f.x : -INFINITY, 4 * c + 2 * u + 1 < lim ? f.y : -INFINITY);
          }
          s2[2 * c + u] = v;
          const float2 e = f2_unpack(f2_add(v, u ? lv.y : lv.x));
          mx0 = fmaxf(mx0, e.x);
          mx1 = fmaxf(mx1, e.y);
        }
      }
      const float mx = fmaxf(mx0, mx1);
      // The reference exponent m only has to stay within kPfMaxSlack bits of the running maximum
      // (weights then stay below 2^14 in fp16), so O, which lives in TMEM across all tiles, is
      // rescaled only when some row of the warp outgrows it by more than that.
      const bool grew = mx > m_run + kPfMaxSlack;
      if (__any_sync(0xffffffffu, grew)) {
        const float m_new = grew ? mx : m_run;
        const float alpha = (m_run == -INFINITY || !grew) ? 1.f : fast_exp2(m_run - m_new);
        if (j > 0) {
          if (!mbar_wait_warp(o_done + t, (j - 1) & 1, kDefaultWaitNs)) dead = true;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 8; ++c) {
            uint32_t r[16];
            tmem_ld16_async(my_o + 16 * c, r);
            tc_wait_ld(r);
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st16_async(my_o + 16 * c, r);
          }
          tc_wait_st();
        }
        l2 = f2_mul(l2, f2_pack(alpha, alpha));
        m_run = m_new;
      }
      // p = 2^(logit log2e - m) feeds the denominator; the weight that meets the value codes is
      // p |v| 2^8, two per TMEM column
      const float neg = m_run == -INFINITY ? 0.f : -m_run;
      const uint64_t neg2 = f2_pack(neg, neg);
      uint32_t w[32];
#pragma unroll
      for (int c = 0; c < kPpN / 4; ++c) {
        const ulonglong2 vs = lds_f2x2(norms + 2 * kPpN * 4 + 16 * c);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float2 d = f2_unpack(f2_add(s2[2 * c + u], neg2));
          const uint64_t pe = f2_pack(fast_exp2(d.x), fast_exp2(d.y));
          l2 = f2_add(l2, pe);
          float2 wf = f2_unpack(f2_mul(pe, u ? vs.y : vs.x));
          if constexpr (decltype(masked)::value) {  // (the norm of a masked token need not be finite)
            if (d.x == -INFINITY) wf.x = 0.f;
            if (d.y == -INFINITY) wf.y = 0.f;
          }
          w[2 * c + u] = pack_half2(wf.x, wf.y);
        }
      }
      // the previous weights have been read
      if (j > 0 && !mbar_wait_warp(o_done + t, (j - 1) & 1, kDefaultWaitNs)) dead = true;
      tc_fence_after();
      tmem_st32_async(my_p, w);
      tc_wait_st();
    };
#pragma unroll 1
    for (int j = 0; j < n_tiles && !dead; ++j) {
      if (!mbar_wait_warp(norm_full + j % kPpNorms, (j / kPpNorms) & 1, kDefaultWaitNs) ||
          !mbar_wait_warp(s_full + t, j & 1, kDefaultWaitNs)) {
        dead = true;
        break;
      }
      tc_fence_after();
      const bool whole = (j + 1) * kPpN <= kv_end && (!p.causal || (j + 1) * kPpN <= m0 + ctx + 1);
      if (whole) tile(j, std::false_type{}); else tile(j, std::true_type{});
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + t);
    }
    // ---- epilogue: normalise, round where the reference does, o Pi ------------------------------------
    if (n_tiles > 0 && !dead && !mbar_wait_warp(o_done + t, (n_tiles - 1) & 1, kDefaultWaitNs)) dead = true;
    tc_fence_after();
    // both tiles are through: S, P and Q_0 of either may be overwritten, and so may the rings
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (tid == 0 && n_tiles > 0) {
      fence_proxy_async();
      mbar_expect_tx(planes, 2 * kPpTile);
      bulk_g2s(smem + S::kPi, p.planes_o, kPpTile, planes);
      bulk_g2s(smem + S::kPi + kPpTile, p.planes_o + kPpTile, kPpTile, planes);
    }
    const float2 lf = f2_unpack(l2);
    const float l_row = lf.x + lf.y;
    const float inv = l_row > 0.f ? 1.f / (l_row * 256.f) : 0.f;
    float unscale = 1.f / kPpPiScale;
    if (n_tiles > 0) {
      auto entry = [&](uint32_t bits) {
        float o = __uint_as_float(bits) * inv;
        // the reference's attention over de-quantised pages returns rows of the activation
        // type, which it then rotates (src/flashquant/vllm/impl.py:477-509): round here too
        if constexpr (PAGED) o = to_f32(from_f32<T>(o));
        return o;
      };
      float mx = 0.f;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        tmem_ld32_async(my_o + 32 * c, r);
        tc_wait_ld(r);
#pragma unroll
        for (int i = 0; i < 32; ++i) mx = fmaxf(mx, fabsf(entry(r[i])));
      }
      const float sc = pow2_to_one(mx);
      unscale /= sc;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {  // hi terms to columns 0-63 of the tile's half, lo terms to 64-127
        uint32_t r[32], hi[16], lo[16];
        tmem_ld32_async(my_o + 32 * c, r);
        tc_wait_ld(r);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = entry(r[2 * i]) * sc, o = entry(r[2 * i + 1]) * sc;
          const __half2 h = __floats2half2_rn(a, o);
          hi[i] = *reinterpret_cast<const uint32_t*>(&h);
          lo[i] = pack_half2(a - __low2float(h), o - __high2float(h));
        }
        tmem_st16_async(tmem + 128 * t + lane_sel + 16 * c, hi);
        tmem_st16_async(tmem + 128 * t + lane_sel + 64 + 16 * c, lo);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(rows_in + t);
      if (!mbar_wait_warp(turned + t, 1, kDefaultWaitNs)) dead = true;
      tc_fence_after();
    }
    if (dead && lane == 0 && p.status) atomicOr(p.status, FQ_DEV_WAIT_TIMEOUT);
    // ---- out rows through shared memory (16-byte units, rotated by the row), then 256 bytes per row ----
    unsigned char* stage = smem + (t ? S::kQ : S::kLut);
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t r[32];
      if (n_tiles > 0 && !dead) {
        tmem_ld32_async(my_o + 32 * c, r);  // whole warps: the load is warp-collective
        tc_wait_ld(r);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = 0u;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        __align__(16) T o[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = from_f32<T>(__uint_as_float(r[8 * i + k]) * unscale);
        *reinterpret_cast<uint4*>(stage + row * 256 + (((4 * c + i) ^ (row & 15)) * 16)) =
            *reinterpret_cast<const uint4*>(o);
      }
    }
    __syncwarp();  // a warp copies the 32 rows it stored
    const int r0 = (warp & 3) * 32;
#pragma unroll 4
    for (int i = 0; i < 16; ++i) {
      const int r = r0 + 2 * i + (lane >> 4), u = lane & 15;
      const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 256 + ((u ^ (r & 15)) * 16));
      if (m0 + r < q_len)
        *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + io_row(t, r) * D + 8 * u) = v;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace fq
