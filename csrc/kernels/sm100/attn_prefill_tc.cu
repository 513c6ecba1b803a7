// Causal prefill attention over the paged KV cache on the 5th-generation tensor cores (tcgen05 + TMEM), head_dim 128.
//
// The reference's prefill attention is a flash kernel on mma.sync tiles (kernels/m1/m1_attn.cu:120-410, 64-row query
// tiles, K/V through cp.async).  Here a query tile is 128 rows = (128 / gq) consecutive tokens x the gq query heads of
// one KV head (GQA: the heads of a group share every K/V byte), the native M of tcgen05.mma.  A CTA owns two tiles and
// walks the sequence in blocks of 128 keys (one tile where that leaves every CTA an SM of its own).  Warps 0-3 / 4-7 are
// the softmax of tile 0 / 1 (thread = row), warp 8 issues the MMAs, warp 9 fetches K and V by TMA (a 16-token page of one
// head is 16 contiguous rows of 256 bytes; the 128-byte swizzle is the tensor map's).  Per tile and block:
//   S (128 x 128, fp32, TMEM)  = Q (smem) x K^T (smem, K-major)                        8 MMAs of k = 16
//   P = exp2((S - m) scale)    bf16, written over S in TMEM (tcgen05.st), the A operand of
//   O (128 x 128, fp32, TMEM) += P (TMEM) x V (smem, MN-major)                         8 MMAs of k = 16
// O stays in TMEM; a warp reads and scales it in the blocks in which one of its rows has a new maximum, after P, when the
// scores' registers are free.  Exponents are taken against the running maximum itself: scaling only after it had grown by
// 2^8 was 4 % faster, but leaves a row's heaviest probabilities anywhere in a binade instead of at its top, where bf16
// rounds best, and 2048 rows after 6144 tokens were 2.35e-3 from 64 bits instead of 2.30e-3.  The tensor core works on one
// tile while the other is in its softmax; S(j + 1) follows P V(j) of the same tile in issue order, so S may overwrite P, and
// a finished S implies a finished O.
//
// What bounds it: at long contexts the softmax's issue slots (some 4.5 instructions a score: 1150 cycles a block of two
// tiles) beside 2048 cycles of MMA at the nominal rate, and the last wave of CTAs (one per SM); short ones the chain of
// launch, first copies, one block and output, for which Q comes by asynchronous copies (4 us sooner than load by load) and
// the first two blocks of K and V are under way before it is there.  The kernel before had one tile of 128 threads per CTA,
// S and P through registers and shared memory, O in registers and the copies in the same threads.  64 q / 8 kv heads,
// before -> now: 2048 rows after 6144 tokens 1050 -> 500 us (960 TFLOP/s), after 8000 1322 -> 568, from 0 181 -> 102; 256
// rows after 8000 256 -> 122, from 0 13.2 -> 10.9; 64 rows from 0 7.2 -> 7.4.
// Every wait is bounded; expiry sets the status word and the CTA leaves through the normal exit (TMEM is released).
#include <cuda.h>

#include "common.cuh"

namespace b2 {
namespace {

constexpr int HD = 128;
constexpr int BK = 128;                // keys per block
constexpr int kPfThreads = 320;
constexpr int kSmsP = 148;
constexpr int SM_Q = 0, SM_K = 65536, SM_V = 131072;       // two 32 KB tiles of Q, two stages of K, two of V
constexpr int SM_PF_BYTES = 196608 + 1024;                 // + slack for the 1024-byte alignment of the swizzle pattern

struct PfArgs {
  const bf16* q;          // [T][hq * 128]
  const int* bt;          // block-table row of the sequence
  bf16* out;              // [T][hq * 128]
  int T, pos0, hq, hkv, n_pages, bt_len;
  float scale_log2;
  int* status;
};

__device__ __forceinline__ void pf_mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool pf_mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// K-major operand, 128-byte swizzle: rows 128 B apart, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t pf_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D fp32, A / B bf16, A K-major, B K-major or (b_mn) MN-major, N / 8 and M / 16.
__host__ __device__ constexpr uint32_t pf_idesc(int m, int n, bool b_mn = false) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// MN-major operand, 128-byte swizzle: 64 elements of the MN dimension are contiguous (128 B); successive k rows are
// 128 B apart, 8-row groups `sbo` bytes apart, the next 64 MN elements `lbo` bytes away.
__device__ __forceinline__ uint64_t pf_desc_mn(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(lbo >> 4) << 16;
  d |= (uint64_t)(sbo >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void pf_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void pf_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void pf_tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void pf_tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16-byte asynchronous copy; `valid` false writes zeros (source size 0) without touching the source.
__device__ __forceinline__ void pf_cp16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
// 2^x on the special-function unit; 2^-inf = 0
__device__ __forceinline__ float pf_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pf_pack(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Bounded wait of a warp (about two seconds); the vote brings the lanes back together for the .aligned instructions that
// follow.
__device__ __forceinline__ bool pf_wait_warp(uint32_t bar, uint32_t parity) {
  bool ok = true;
  if (!pf_mbar_try(bar, parity)) {
    uint64_t t0 = 0;
    for (unsigned it = 1; !pf_mbar_try(bar, parity); ++it) {
      if ((it & 255u) == 0u) {
        const uint64_t t = globaltimer_ns();
        if (!t0) t0 = t;
        else if (t - t0 > 2000000000ull) { ok = false; break; }
      }
    }
  }
  return __all_sync(0xffffffffu, ok) != 0;
}
__device__ __forceinline__ void pf_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void pf_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pf_tma(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void pf_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void pf_tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void pf_tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
        "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
        "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void pf_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
}  // namespace

// TILES: query tiles of a CTA, 1 or 2.
template <int TILES>
__global__ void __launch_bounds__(kPfThreads, 1) attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_kv, const PfArgs a) {
  extern __shared__ __align__(1024) uint8_t pf_smem[];
  __shared__ __align__(8) uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], o_final[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_failed;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t base = (smem_u32(pf_smem) + 1023u) & ~1023u;
  const int gq = a.hq / a.hkv;
  const int tt = 128 / gq;                                   // tokens per tile
  const int per = TILES * tt;                                // tokens per CTA
  const int kvh = blockIdx.y;
  const int tok0 = ((a.T + per - 1) / per - 1 - (int)blockIdx.x) * per;     // longest first
  const int n_tok = min(per, a.T - tok0);
  constexpr int last = TILES - 1;                            // the last tile (it may have no tokens)
  const int kv_len = a.pos0 + tok0 + n_tok;
  const int nb = (kv_len + BK - 1) / BK;

  // K / V pages of one block by warp 9: lane = (page of the block, 64-dim half); false = a wait for a free stage gave up
  auto fetch_block = [&](int j) -> bool {
    const int st = j & 1;
    const int pi = j * 8 + (lane >> 1);
    const bool on = lane < 16 && pi * 16 < kv_len;
    int page = 0;
    if (on) {
      page = pi < a.bt_len ? __ldg(a.bt + pi) : -1;
      if (page < 0 || page >= a.n_pages) { atomicExch(a.status, (int)B2_ERR_BOUNDS); page = 0; }
    }
    const uint32_t bytes = (uint32_t)min(8, (kv_len - j * BK + 15) / 16) * 4096u;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const uint32_t full = smem_u32(which ? &v_full[st] : &k_full[st]), empty = smem_u32(which ? &v_empty[st] : &k_empty[st]);
      if (j >= 2 && !pf_wait_warp(empty, (uint32_t)((j >> 1) - 1) & 1u)) return false;
      if (lane == 0) pf_expect(full, bytes);
      __syncwarp();
      if (on)
        pf_tma(base + (which ? SM_V : SM_K) + st * 32768 + (lane & 1) * 16384 + (lane >> 1) * 2048, &map_kv, (lane & 1) * 64,
               ((page * 2 + which) * a.hkv + kvh) * 16, full);
      __syncwarp();
    }
    return true;
  };
  if (warp == 9) {
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_kv) : "memory");
      for (int i = 0; i < 2; ++i) {
        pf_mbar_init(smem_u32(&k_full[i]), 1);
        pf_mbar_init(smem_u32(&k_empty[i]), 1);
        pf_mbar_init(smem_u32(&v_full[i]), 1);
        pf_mbar_init(smem_u32(&v_empty[i]), 1);
        pf_mbar_init(smem_u32(&s_full[i]), 1);
        pf_mbar_init(smem_u32(&p_ready[i]), 4);
        pf_mbar_init(smem_u32(&o_final[i]), 1);
      }
      s_failed = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    pdl_wait();
    for (int j = 0; j < 2 && j < nb; ++j) fetch_block(j);    // both stages are free: no wait
  } else {
    if (warp == 8) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    if (warp < 8) {
      // ---- Q tiles: 128 rows x 256 B -> two swizzled 64-dim halves each; rows past the chunk are zero.  Asynchronous
      // copies: one latency for all of a thread
      const int lg = __ffs(gq) - 1;                          // gq divides 128
#pragma unroll
      for (int i = 0; i < 8 * TILES; ++i) {
        const int e = i * 256 + tid;
        const int tl = e >> 11, r = (e >> 4) & 127, c = e & 15;
        const int t = r >> lg, h = r & (gq - 1);
        const int tok = tl * tt + t;
        const bool ok = tok < n_tok;
        pf_cp16(base + SM_Q + tl * 32768 + (c >> 3) * 16384 + r * 128 + (((c & 7) ^ (r & 7)) << 4),
                a.q + ((size_t)(tok0 + (ok ? tok : 0)) * a.hq + (size_t)kvh * gq + h) * HD + c * 8, ok);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  if (warp == 9) {
    // ---------------- K / V pages ----------------
    for (int j = 2; j < nb; ++j)
      if (!fetch_block(j)) { s_failed = 1; break; }
  } else if (warp == 8) {
    // ---------------- MMA issuer ----------------
    constexpr uint32_t idesc_s = pf_idesc(128, BK), idesc_o = pf_idesc(128, HD, true);
    auto issue_s = [&](int t, int st) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint64_t dq = pf_desc(base + SM_Q + t * 32768 + h * 16384), dk = pf_desc(base + SM_K + st * 32768 + h * 16384);
#pragma unroll
        for (int k = 0; k < 4; ++k) pf_mma(tmem + (uint32_t)t * 128u, dq + 2 * k, dk + 2 * k, idesc_s, (h | k) ? 1u : 0u);
      }
      pf_commit(smem_u32(&s_full[t]));
    };
    bool ok = pf_wait_warp(smem_u32(&k_full[0]), 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok && lane == 0) {
      issue_s(0, 0);
      if (TILES == 2) issue_s(1, 0);
      pf_commit(smem_u32(&k_empty[0]));
    }
    __syncwarp();
    for (int j = 0; j < nb && ok; ++j) {
      const int st = j & 1, sn = st ^ 1;
      ok = pf_wait_warp(smem_u32(&v_full[st]), (uint32_t)(j >> 1) & 1u);
#pragma unroll
      for (int t = 0; t < TILES; ++t) {
        ok = ok && pf_wait_warp(smem_u32(&p_ready[t]), (uint32_t)j & 1u);
        if (t == 0 && j + 1 < nb) ok = ok && pf_wait_warp(smem_u32(&k_full[sn]), (uint32_t)((j + 1) >> 1) & 1u);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (lane == 0) {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            pf_mma_ts(tmem + 256u + (uint32_t)t * 128u, tmem + (uint32_t)t * 128u + (uint32_t)k * 8u,
                      pf_desc_mn(base + SM_V + st * 32768 + k * 2048, 16384, 1024), idesc_o, (j || k) ? 1u : 0u);
          if (j == nb - 1) pf_commit(smem_u32(&o_final[t]));
          if (t == last && j + 2 < nb) pf_commit(smem_u32(&v_empty[st]));   // no arrival is left for after the last wait
          if (j + 1 < nb) {
            issue_s(t, sn);
            if (t == last) pf_commit(smem_u32(&k_empty[sn]));
          }
        }
        __syncwarp();
      }
    }
    if (!ok) s_failed = 1;
  } else if ((warp >> 2) <= last) {
    // ---------------- softmax of tile t: thread = row = TMEM lane ----------------
    const int t = warp >> 2;
    const int row = tid & 127;
    const int rt = t * tt + row / gq, rh = row % gq;
    const bool row_valid = rt < n_tok;
    const int limit = a.pos0 + tok0 + rt;                    // last key this row may see
    const uint32_t trow = tmem + ((uint32_t)(warp & 3) << 21);
    const uint32_t ts = trow + (uint32_t)t * 128u, to = trow + 256u + (uint32_t)t * 128u;
    float m_ref = -INFINITY, l_run = 0.f;
    bool ok = true;
#pragma unroll 1
    for (int j = 0; j < nb; ++j) {
      if (!pf_wait_warp(smem_u32(&s_full[t]), (uint32_t)j & 1u)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[BK];
      {
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) pf_tmem_ld32_issue(ts + (uint32_t)c * 32u, r[c]);
        pf_tmem_wait();
#pragma unroll
        for (int i = 0; i < BK; ++i) s[i] = __uint_as_float(r[i >> 5][i & 31]);
      }
      const int kb = j * BK;
      if (!row_valid || kb + BK - 1 > limit) {
#pragma unroll
        for (int i = 0; i < BK; ++i)
          if (!row_valid || kb + i > limit) s[i] = -INFINITY;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < BK; i += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) mx4[u] = fmaxf(mx4[u], s[i + u]);
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // p = 2^((s - m) scale) against the row's running maximum; a new maximum scales what the row has so far
      const bool grow = j > 0 && mx > m_ref;
      const float corr = grow ? pf_ex2((m_ref - mx) * a.scale_log2) : 1.f;
      m_ref = fmaxf(m_ref, mx);
      const float moff = m_ref == -INFINITY ? 0.f : -m_ref * a.scale_log2;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float p0 = pf_ex2(fmaf(s[c * 32 + i], a.scale_log2, moff)), p1 = pf_ex2(fmaf(s[c * 32 + i + 1], a.scale_log2, moff));
          const float p2 = pf_ex2(fmaf(s[c * 32 + i + 2], a.scale_log2, moff)), p3 = pf_ex2(fmaf(s[c * 32 + i + 3], a.scale_log2, moff));
          sum4[0] += p0; sum4[1] += p1; sum4[2] += p2; sum4[3] += p3;
          pk[i >> 1] = pf_pack(p0, p1);
          pk[(i >> 1) + 1] = pf_pack(p2, p3);
        }
        pf_tmem_st16(ts + (uint32_t)c * 16u, pk);
      }
      l_run = l_run * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
      if (__any_sync(0xffffffffu, grow)) {
        uint32_t r[4][32];                                   // the scores' registers are free again
#pragma unroll
        for (int c = 0; c < 4; ++c) pf_tmem_ld32_issue(to + (uint32_t)c * 32u, r[c]);
        pf_tmem_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[c][i] = __float_as_uint(__uint_as_float(r[c][i]) * corr);
          pf_tmem_st32(to + (uint32_t)c * 32u, r[c]);
        }
      }
      if (t == 0 && j == nb - 1 && (kv_len & (BK - 1))) {
        // the V rows past the context are zero (P is zero there, but zero times whatever the page holds need not be)
        if (!pf_wait_warp(smem_u32(&v_full[j & 1]), (uint32_t)(j >> 1) & 1u)) { ok = false; break; }
        const int r0 = kv_len & (BK - 1);
        for (int e = tid; e < (BK - r0) * 16; e += 128) {
          const int r = r0 + (e >> 4), c = e & 15;
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(base + SM_V + (j & 1) * 32768 + (c >> 3) * 16384 + r * 128 + (c & 7) * 16), "r"(0) : "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      pf_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) pf_arrive(smem_u32(&p_ready[t]));
    }
    if (ok && pf_wait_warp(smem_u32(&o_final[t]), 0)) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      bf16* dst = a.out + ((size_t)(tok0 + (row_valid ? rt : 0)) * a.hq + (size_t)kvh * gq + rh) * HD;
      uint32_t r[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) pf_tmem_ld32_issue(to + (uint32_t)c * 32u, r[c]);
      pf_tmem_wait();
      if (row_valid) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pf_pack(__uint_as_float(r[c][i]) * inv, __uint_as_float(r[c][i + 1]) * inv);
            w.y = pf_pack(__uint_as_float(r[c][i + 2]) * inv, __uint_as_float(r[c][i + 3]) * inv);
            w.z = pf_pack(__uint_as_float(r[c][i + 4]) * inv, __uint_as_float(r[c][i + 5]) * inv);
            w.w = pf_pack(__uint_as_float(r[c][i + 6]) * inv, __uint_as_float(r[c][i + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + i) = w;
          }
      }
    } else {
      s_failed = 1;
    }
  }
  pdl_launch_dependents();
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_failed) {
    if (tid == 0 && a.status) atomicExch(a.status, (int)B2_ERR_TIMEOUT);
    const uint64_t t_end = globaltimer_ns() + 2000000ull;    // copies still in flight get a bounded time to land
    while (globaltimer_ns() < t_end) { }
  }
  if (warp == 8) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

}  // namespace b2

using namespace b2;

typedef CUresult (*PfEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Causal attention of a prefill chunk: q [T][hq * 128] at positions pos0 .. pos0 + T - 1 of one sequence whose block
// table row is `bt` (bt_len entries); the KV pool already holds the chunk's own K / V.  head_dim 128, gq = hq / hkv
// a divisor of 128.
B2_API int b2_attn_prefill_tc(const void* q, const void* kv_pool, const int* bt, int bt_len, void* out, int T, int pos0, int hq, int hkv,
                              int n_pages, float scale, int* status, cudaStream_t stream) {
  if (T <= 0 || hq <= 0 || hkv <= 0 || hq % hkv || 128 % (hq / hkv) || !status) return B2_ERR_ARG;
  static PfEncode enc = nullptr;
  if (!enc) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) return B2_ERR_LAUNCH;
    for (auto kern : {attn_prefill_tc_kernel<1>, attn_prefill_tc_kernel<2>})
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_PF_BYTES) != cudaSuccess) return B2_ERR_LAUNCH;
    enc = reinterpret_cast<PfEncode>(f);
  }
  // the pool as a matrix of 256-byte rows: row ((page * 2 + K|V) * hkv + head) * 16 + token; boxes of half a page slab
  CUtensorMap map;
  cuuint64_t dims[2] = {(cuuint64_t)HD, (cuuint64_t)n_pages * 2 * hkv * 16};
  cuuint64_t strides[1] = {HD * 2};
  cuuint32_t box[2] = {64, 16}, estr[2] = {1, 1};
  if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(kv_pool), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return B2_ERR_LAUNCH;
  PfArgs a;
  a.q = static_cast<const bf16*>(q);
  a.bt = bt;
  a.bt_len = bt_len;
  a.out = static_cast<bf16*>(out);
  a.T = T; a.pos0 = pos0; a.hq = hq; a.hkv = hkv; a.n_pages = n_pages;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.status = status;
  const int tt = 128 / (hq / hkv);
  // Two tiles share a CTA's K and V and fill each other's waits; while the CTAs of one tile each are at most one per SM,
  // they are done sooner on their own (64 q / 8 kv heads, 64 rows from 0 9.2 -> 7.6 us, 256 rows after 300 20.0 -> 17.4).
  const int tiles = (long)((T + tt - 1) / tt) * hkv <= kSmsP ? 1 : 2, per = tiles * tt;
  const dim3 grid((unsigned)((T + per - 1) / per), (unsigned)hkv, 1);
  if (tiles == 1) attn_prefill_tc_kernel<1><<<grid, kPfThreads, SM_PF_BYTES, stream>>>(map, a);
  else attn_prefill_tc_kernel<2><<<grid, kPfThreads, SM_PF_BYTES, stream>>>(map, a);
  return cudaGetLastError() == cudaSuccess ? B2_OK : B2_ERR_LAUNCH;
}
