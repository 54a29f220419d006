// Fused TQ4 attention for many query rows: warp-specialised tcgen05 kernel.  Included by prefill.cu.
//
// A CTA owns TWO tiles of 128 query rows that attend over the same keys - two heads of a KV group
// at the same positions, or (odd groups) 256 consecutive positions of one head - and walks the keys in
// tiles of 128 tokens:
//   warps 0-3, 4-7  softmax of tile 0 / 1, one thread per row: reads its row of S from TMEM,
//                   applies |k| and the scale, the lazily raised reference exponent, writes the
//                   fp16 weights p |v| 2^8 over S as the A operand of the value product;
//   warps 8-11      turn codes into fp16 operand tiles in shared memory (global -> registers one
//                   tile ahead -> look-up / byte permute -> store): once for both query tiles;
//   warp 12         issues every MMA: S_t = Q_t K^T (operands in shared memory) and
//                   O_t += P_t V (P from TMEM).
// The two query tiles take turns on the tensor pipe: while softmax 0 runs, the pipe works on
// tile 1.  TMEM: S_0 S_1 (128 columns each, P over S), O_0 O_1.  Nothing in the loop is a
// block-wide barrier.
//
// Why this split: per 128 tokens the pair costs 2048 cycles of MMA, 2048 of exponentials (16
// per cycle and SM), and about 2900 of shared-memory bandwidth (MMA operand reads 1536, operand
// stores 512, look-ups 256, norms 768), which is what bounds it.  The earlier one-tile CTA, whose
// 256 threads did all of it between three block barriers, de-quantised every tile for 128 rows only
// and needed 5.8 ms at 4 x 8192 tokens, 32 / 8 heads.
#pragma once

namespace fq {

constexpr int kPpThreads = 512;
constexpr int kPpN = 128;                       // keys per tile
constexpr int kPpVSlots = 3;                    // value operand ring, 64 tokens per slot
constexpr uint32_t kPpTile = 128 * 128 * 2;     // operand tile of 128 rows
constexpr uint32_t kPpHalf = kPpTile / 2;
constexpr uint32_t kPpSlab = 128 * 16;          // one 8-element chunk of 128 rows
constexpr uint32_t kPpSlabV = 64 * 16;
constexpr int kPpKCopies = 8;                   // key table copies (16-level keys only)

struct PairSmem {
  static constexpr uint32_t kQ = 0;                                  // two query tiles
  static constexpr uint32_t kK = kQ + 2 * kPpTile;                   // two key tiles
  static constexpr uint32_t kV = kK + 2 * kPpTile;                   // three value halves
  static constexpr uint32_t kLutV = kV + kPpVSlots * kPpHalf;        // 256 entries x 32 lanes
  static constexpr uint32_t kLutK = kLutV + 256 * 128;               // 256 entries x 8 copies
  static constexpr uint32_t kNorm = kLutK + 256 * 4 * kPpKCopies;    // [3][nk | lv | vs][128]
  static constexpr uint32_t kBar = kNorm + 3 * 3 * kPpN * 4;
  static constexpr uint32_t kBytes = kBar + 256;
};
static_assert(PairSmem::kBytes <= 227 * 1024, "shared memory of one CTA");

// ---- packed fp32 pairs ------------------------------------------------------------------------
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ ulonglong2 lds_f2x2(uint32_t a) {  // four consecutive floats
  ulonglong2 r;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(r.x), "=l"(r.y) : "r"(a));
  return r;
}

// 32 columns of this warp's 32 TMEM lanes, without waiting for them
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32_async(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31])
      : "memory");
}
// The loads of this thread have delivered: the registers pass through the wait, so that nothing
// that reads them is scheduled before it.
__device__ __forceinline__ void tc_wait_ld(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]),
                 "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                 "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]),
                 "+r"(r[31])::"memory");
}
__device__ __forceinline__ void tc_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// MMA issue by a converged warp: every lane computes the same operands - the descriptors then live in
// uniform registers, where the instruction wants them - and `leader` (one lane) issues.  Inside
// an `if (lane == 0)` every MMA moved its operands over from vector registers: 250 cycles each
// instead of a few, which starved the tensor pipe.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok));
  return ok != 0;
}
// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void umma_ss(bool leader, uint32_t d_tmem, uint64_t a_desc,
                                        uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(uint32_t(accumulate)), "r"(uint32_t(leader))
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: A holds two consecutive k per 32-bit column
__device__ __forceinline__ void umma_ts(bool leader, uint32_t d_tmem, uint32_t a_tmem,
                                        uint64_t b_desc, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(uint32_t(accumulate)), "r"(uint32_t(leader))
      : "memory");
}
// all MMAs that `leader` has issued arrive on the barrier when they have completed
__device__ __forceinline__ void umma_commit_if(bool leader, uint64_t* bar) {
  asm volatile(
      "{\n\t"
      ".reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n" ::"r"(smem_u32(bar)),
      "r"(uint32_t(leader))
      : "memory");
}

template <bool PAGED>
__global__ void __launch_bounds__(kPpThreads, 1) prefill_pair_kernel(PrefillArgs p) {
  using S = PairSmem;
  constexpr int D = 128;
  constexpr uint32_t kIdescS = umma_idesc(128, kPpN, false);
  constexpr uint32_t kIdescO = umma_idesc(128, D, true);
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBar);
  uint64_t* k_full = bars;          // [2] key tile stored (128 arrivals)
  uint64_t* k_empty = bars + 2;     // [2] its products are complete
  uint64_t* v_full = bars + 4;      // [3]
  uint64_t* v_empty = bars + 7;     // [3]
  uint64_t* norm_full = bars + 10;  // [3] norms of a tile stored (128 arrivals)
  uint64_t* s_full = bars + 13;     // [2] scores of query tile t complete
  uint64_t* p_full = bars + 15;     // [2] weights of query tile t stored (4 warps)
  uint64_t* o_done = bars + 17;     // [2] value product of query tile t complete
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 19);

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
  auto tile_rows = [&](int t) {
    const int r = q_len - tile_m0(t);
    return r < 0 ? 0 : (r < 128 ? r : 128);
  };

  // ---- set-up -----------------------------------------------------------------------------------
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(k_full + i, 128);
      mbar_init(k_empty + i, 1);
      mbar_init(s_full + i, 1);
      mbar_init(p_full + i, 4);
      mbar_init(o_done + i, 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(v_full + i, 128);
      mbar_init(v_empty + i, 1);
      mbar_init(norm_full + i, 128);
    }
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  // tables of fp16(c / beta): beta_k folds into the score scale, beta_v into the weights
  const float beta_k = p.scales[0], beta_v = p.scales[1];
  const float rbk = 1.f / beta_k, rbv = 1.f / beta_v;
  const bool k_by_permute = p.nck <= 8;
  // 16-level keys with the values' own table (the same centroids, hence the same beta): one table
  const bool same_table =
      p.nck == p.ncv && beta_k == beta_v &&
      __all_sync(0xffffffffu, lane >= p.nck || p.cent_k[lane & 15] == p.cent_v[lane & 15]);
  {
    const int e = tid >> 1;  // two threads per entry, 16 copies each
    const int hi = e >> 4, lo = e & 15;
    const uint32_t v = pack_half2(hi < p.ncv ? p.cent_v[hi] * rbv : 0.f,
                                  lo < p.ncv ? p.cent_v[lo] * rbv : 0.f);
    uint4* dst = reinterpret_cast<uint4*>(smem + S::kLutV + e * 128 + (tid & 1) * 64);
    const uint4 v4 = make_uint4(v, v, v, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = v4;
    if (!k_by_permute && !same_table) {
      const uint32_t k = pack_half2(hi < p.nck ? p.cent_k[hi] * rbk : 0.f,
                                    lo < p.nck ? p.cent_k[lo] * rbk : 0.f);
      *reinterpret_cast<uint4*>(smem + S::kLutK + e * (4 * kPpKCopies) + (tid & 1) * 16) =
          make_uint4(k, k, k, k);
    }
  }
  // query tiles -> [k-chunk][row][16 B]
  for (int i = tid; i < 2 * 128 * 16; i += kPpThreads) {
    const int t = i >> 11, r = (i >> 4) & 127, kc = i & 15;
    const int m0 = tile_m0(t), head = two_heads ? head0 + t : head0;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (m0 + r < q_len) {
      const __half* src = PAGED ? p.q_rot + (int64_t(q_first + m0 + r) * p.hq + head) * D
                                : p.q_rot + ((int64_t(b) * p.hq + head) * p.nq + m0 + r) * D;
      v = *reinterpret_cast<const uint4*>(src + kc * 8);
    }
    *reinterpret_cast<uint4*>(smem + S::kQ + t * kPpTile + kc * kPpSlab + r * 16) = v;
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_holder, 0);
  bool dead = false, bad_page = false;

  if (warp >= 12) {
    // ---- MMA issue --------------------------------------------------------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 12 && n_tiles > 0) {
      const bool leader = elect_one();
      const uint32_t qa = smem_u32(smem + S::kQ), ka = smem_u32(smem + S::kK), va = smem_u32(smem + S::kV);
      auto scores = [&](int t, int j) {
        const uint32_t q = qa + t * kPpTile, k = ka + (j & 1) * kPpTile;
#pragma unroll
        for (int s = 0; s < D / 16; ++s)
          umma_ss(leader, tmem + 128 * t, smem_desc(q + 2 * s * kPpSlab, kPpSlab, 128),
                   smem_desc(k + 2 * s * kPpSlab, kPpSlab, 128), kIdescS, s > 0);
        umma_commit_if(leader, s_full + t);
      };
      auto values = [&](int t, int j) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t v = va + ((2 * j + h) % kPpVSlots) * kPpHalf;
#pragma unroll
          for (int s = 0; s < 4; ++s)
            umma_ts(leader, tmem + 256 + 128 * t, tmem + 128 * t + 32 * h + 8 * s,
                        smem_desc(v + s * 256, 128, kPpSlabV), kIdescO, j > 0 || h > 0 || s > 0);
        }
        umma_commit_if(leader, o_done + t);
      };
      // weights of query tile t and values of key tile j are there
      auto wait_values = [&](int t, int j) {
        bool ok = mbar_wait_warp(p_full + t, j & 1, kDefaultWaitNs);
        if (t == 0) {
          const int h0 = 2 * j, h1 = 2 * j + 1;
          ok = ok && mbar_wait_warp(v_full + h0 % kPpVSlots, (h0 / kPpVSlots) & 1, kDefaultWaitNs) &&
               mbar_wait_warp(v_full + h1 % kPpVSlots, (h1 / kPpVSlots) & 1, kDefaultWaitNs);
        }
        tc_fence_after();
        return ok;
      };
      auto free_values = [&](int j) {
        umma_commit_if(leader, v_empty + (2 * j) % kPpVSlots);
        umma_commit_if(leader, v_empty + (2 * j + 1) % kPpVSlots);
      };
#pragma unroll 1
      for (int j = 0; j < n_tiles && !dead; ++j) {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j > 0 && !dead) {
            dead = !wait_values(t, j - 1);
            if (!dead) values(t, j - 1);
          }
          if (t == 0 && !dead) {
            dead = !mbar_wait_warp(k_full + (j & 1), (j >> 1) & 1, kDefaultWaitNs);
            tc_fence_after();
          }
          if (!dead) scores(t, j);
        }
        if (dead) break;
        umma_commit_if(leader, k_empty + (j & 1));
        if (j > 0) free_values(j - 1);
      }
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (dead) break;
        dead = !wait_values(t, n_tiles - 1);
        if (!dead) values(t, n_tiles - 1);
      }
      if (dead && leader && p.status) atomicOr(p.status, FQ_DEV_WAIT_TIMEOUT);
    }
  } else if (warp >= 8) {
    // ---- codes -> operand tiles ----------------------------------------------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    const int dt = tid - 256, dw = warp - 8;
    const float k_scale = p.scale_log2 * beta_k, v_scale = 256.f * beta_v;
    // 8-entry key table in registers: low and high bytes of the fp16 centroids
    uint32_t tl0 = 0, tl1 = 0, th0 = 0, th1 = 0;
    if (k_by_permute) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t h =
            uint32_t(__half_as_ushort(__float2half_rn(i < p.nck ? p.cent_k[i] * rbk : 0.f)));
        const uint32_t lo8 = (h & 0xffu) << (8 * (i & 3)), hi8 = (h >> 8) << (8 * (i & 3));
        if (i < 4) { tl0 |= lo8; th0 |= hi8; } else { tl1 |= lo8; th1 |= hi8; }
      }
    }
    // Lane = (quarter q of a token's 64 code bytes, token of eight): the 16-byte loads of a warp
    // cover 512 contiguous bytes, its stores 128 contiguous bytes per eight lanes.
    const int q4 = lane >> 3, tok8 = 8 * dw + (lane & 7);  // + 32 * i: token of load i
    const int row_bytes = p.hkv * (D + 8);
    const int64_t kv_row0 = PAGED ? 0 : (int64_t(b) * p.hkv + hkv) * p.kv_stride;
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
    struct Rows {
      int code[4], norm;
    };
    auto rows_of = [&](int j, Rows& r) {
#pragma unroll
      for (int i = 0; i < 4; ++i) r.code[i] = row_of(j * kPpN + 32 * i + tok8);
      r.norm = row_of(j * kPpN + dt);
    };
    auto load_codes = [&](const Rows& r, bool is_k, uint4 (&reg)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        reg[i] = make_uint4(0u, 0u, 0u, 0u);
        if (r.code[i] >= 0) {
          const uint8_t* src;
          if constexpr (PAGED)
            src = p.kv_cache + int64_t(r.code[i]) * row_bytes +
                  (is_k ? 0 : p.hkv * (D / 2 + 4)) + hkv * (D / 2);
          else
            src = (is_k ? p.k_packed : p.v_packed) + (kv_row0 + r.code[i]) * (D / 2);
          reg[i] = __ldg(reinterpret_cast<const uint4*>(src) + q4);
        }
      }
    };
    auto load_norms = [&](const Rows& r, float& nk, float& nv) {
      nk = nv = 0.f;
      if (r.norm < 0) return;
      if constexpr (PAGED) {
        const uint8_t* src = p.kv_cache + int64_t(r.norm) * row_bytes + p.hkv * (D / 2) + 4 * hkv;
        nk = *reinterpret_cast<const float*>(src);
        nv = *reinterpret_cast<const float*>(src + p.hkv * (D / 2 + 4));
      } else {
        nk = p.k_norms[kv_row0 + r.norm];
        nv = p.v_norms[kv_row0 + r.norm];
      }
    };
    const uint32_t lut_v = smem_u32(smem + S::kLutV) + 4 * lane;
    const uint32_t lut_k = same_table ? lut_v
                                      : smem_u32(smem + S::kLutK) + 4 * (lane & (kPpKCopies - 1));
    const uint32_t k_shift = same_table ? 7u : 5u;  // bytes per key table entry, log2
    auto lut = [&](uint32_t base, uint32_t shift, uint32_t byte) {
      uint32_t v;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(base + (byte << shift)));
      return v;
    };
    auto by_table = [&](uint32_t base, uint32_t shift, uint32_t w) {
      return make_uint4(lut(base, shift, w & 0xff), lut(base, shift, (w >> 8) & 0xff),
                        lut(base, shift, (w >> 16) & 0xff), lut(base, shift, w >> 24));
    };
    auto by_permute = [&](uint32_t w) {
      // nibbles of w, low to high: odd0, even0, odd1, even1, ...
      const uint32_t la = prmt(tl0, tl1, w), ha = prmt(th0, th1, w);
      const uint32_t lb = prmt(tl0, tl1, w >> 16), hb = prmt(th0, th1, w >> 16);
      return make_uint4(prmt(la, ha, 0x4051), prmt(la, ha, 0x6273), prmt(lb, hb, 0x4051),
                        prmt(lb, hb, 0x6273));
    };
    Rows cur, nxt;
    uint4 kreg[4], vreg[4];
    float nk = 0.f, nv = 0.f;
    rows_of(0, cur);
    load_codes(cur, true, kreg);
    load_norms(cur, nk, nv);
    load_codes(cur, false, vreg);
    rows_of(1, nxt);
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      // ---- keys (and all norms) of tile j ----------------------------------------------------------
      if (j >= 2 && !mbar_wait(k_empty + (j & 1), ((j >> 1) - 1) & 1)) { dead = true; break; }
      // (norm slot j % 3 was read by the softmax of tile j - 3, which the scores of tile j - 2,
      // complete by the wait above, came after)
      float* ns = reinterpret_cast<float*>(smem + S::kNorm) + (j % 3) * 3 * kPpN + dt;
      ns[0] = nk * k_scale;
      ns[kPpN] = fmaxf(fast_log2(nv), -40.f);
      ns[2 * kPpN] = nv * v_scale;
      mbar_arrive(norm_full + j % 3);
      unsigned char* kdst = smem + S::kK + (j & 1) * kPpTile + 4 * q4 * kPpSlab + tok8 * 16;
      auto store_keys = [&](auto expand) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t w[4] = {kreg[i].x, kreg[i].y, kreg[i].z, kreg[i].w};
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(kdst + c * kPpSlab + i * 512) = expand(w[c]);
        }
      };
      if (k_by_permute) store_keys(by_permute);
      else store_keys([&](uint32_t w) { return by_table(lut_k, k_shift, w); });
      fence_async_smem();
      mbar_arrive(k_full + (j & 1));
      const bool more = j + 1 < n_tiles;
      if (more) {
        load_codes(nxt, true, kreg);
        load_norms(nxt, nk, nv);
      }
      // ---- values, 64 tokens at a time ---------------------------------------------------------------
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = 2 * j + h, slot = n % kPpVSlots;
        if (n >= kPpVSlots && !mbar_wait(v_empty + slot, (n / kPpVSlots - 1) & 1)) { dead = true; break; }
        unsigned char* vdst = smem + S::kV + slot * kPpHalf + 4 * q4 * kPpSlabV + tok8 * 16;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 r = vreg[2 * h + i];
          const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(vdst + c * kPpSlabV + i * 512) = by_table(lut_v, 7u, w[c]);
        }
        fence_async_smem();
        mbar_arrive(v_full + slot);
      }
      if (dead) break;
      if (more) {
        load_codes(nxt, false, vreg);
        cur = nxt;
        rows_of(j + 2, nxt);
      }
    }
    if (dead && dt == 0 && p.status) atomicOr(p.status, FQ_DEV_WAIT_TIMEOUT);
    if constexpr (PAGED) {
      if ((bad_page || clamped) && p.status) atomicOr(p.status, FQ_DEV_BAD_BLOCK_INDEX);
    }
  } else {
    // ---- softmax of query tile t, one thread per row -------------------------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    const int t = warp >> 2, row = tid & 127;
    const int m0 = tile_m0(t), rows = tile_rows(t);
    const int q_pos = m0 + row;
    const uint32_t lane_sel = uint32_t((warp & 3) * 32) << 16;
    const uint32_t tm_s = tmem + 128 * t + lane_sel, tm_o = tmem + 256 + 128 * t + lane_sel;
    float m_run = -INFINITY;
    uint64_t l2 = 0;  // (0, 0)
    // one key tile; masked: it reaches past the end of the keys or the row's causal limit
    auto tile = [&](int j, auto masked) {
      const uint32_t norms = smem_u32(smem + S::kNorm) + (j % 3) * (3 * kPpN * 4);
      uint64_t s2[kPpN / 2];
      {
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32_async(tm_s + 32 * c, r[c]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tc_wait_ld(r[c]);
#pragma unroll
          for (int i = 0; i < 16; ++i)
            s2[16 * c + i] = f2_pack(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1]));
        }
      }
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
          if (!mbar_wait(o_done + t, (j - 1) & 1)) dead = true;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld32_async(tm_o + 32 * c, r);
            tc_wait_ld(r);
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st32_async(tm_o + 32 * c, r);
          }
          tc_wait_st();
        }
        l2 = f2_mul(l2, f2_pack(alpha, alpha));
        m_run = m_new;
      }
      // p = 2^(logit log2e - m) feeds the denominator; the weight that meets the value codes is
      // p |v| 2^8, two per TMEM column, over the scores
      const float neg = m_run == -INFINITY ? 0.f : -m_run;
      const uint64_t neg2 = f2_pack(neg, neg);
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        uint32_t w[32];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const ulonglong2 vs = lds_f2x2(norms + 2 * kPpN * 4 + 16 * (16 * hc + c));
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float2 d = f2_unpack(f2_add(s2[32 * hc + 2 * c + u], neg2));
            const uint64_t pe = f2_pack(fast_exp2(d.x), fast_exp2(d.y));
            l2 = f2_add(l2, pe);
            const float2 wf = f2_unpack(f2_mul(pe, u ? vs.y : vs.x));
            w[2 * c + u] = pack_half2(wf.x, wf.y);
          }
        }
        tmem_st32_async(tm_s + 32 * hc, w);
      }
      tc_wait_st();
    };
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      if (!mbar_wait_warp(norm_full + j % 3, (j / 3) & 1, kDefaultWaitNs) ||
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
    // ---- epilogue: normalise, round, store the rotated-space row -----------------------------------
    if (n_tiles > 0 && !dead && !mbar_wait_warp(o_done + t, (n_tiles - 1) & 1, kDefaultWaitNs)) dead = true;
    dead = __any_sync(0xffffffffu, dead);
    tc_fence_after();
    if (dead && lane == 0 && p.status) atomicOr(p.status, FQ_DEV_WAIT_TIMEOUT);
    const float2 lf = f2_unpack(l2);
    const float l_row = lf.x + lf.y;
    const float inv = l_row > 0.f ? 1.f / (l_row * 256.f) : 0.f;
    const int head = two_heads ? head0 + t : head0;
    const int64_t row_global = PAGED ? int64_t(q_first + q_pos) * p.hq + head
                                     : (int64_t(b) * p.hq + head) * p.nq + q_pos;
    float* dst = p.o_rot + row_global * D;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t r[32];
      if (n_tiles > 0 && !dead) {
        tmem_ld32_async(tm_o + 32 * c, r);  // whole warps: the load is warp-collective
        tc_wait_ld(r);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = 0u;
      }
      if (row < rows) {
        float o[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          o[i] = __uint_as_float(r[i]) * inv;
          // the reference's attention over de-quantised pages returns rows of the activation
          // type, which it then rotates (src/flashquant/vllm/impl.py:477-509): round here too
          if (p.round_out == FQ_BF16) o[i] = __bfloat162float(__float2bfloat16_rn(o[i]));
          if (p.round_out == FQ_F16) o[i] = __half2float(__float2half_rn(o[i]));
        }
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<float4*>(dst + 32 * c + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
      }
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
