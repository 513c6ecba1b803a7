// Mixed-bit weight GEMM on the 5th-generation tensor cores for 9 .. 256 token rows (batched decode, big verify blocks,
// prefill chunks): y[tok][row] = sum_k W[row][k] x[tok][k], W stored as 2/3/4-bit codes in the FM layout of the GEMV.
//
// The weights are the M operand (128 rows per tile), the tokens the N operand, so one tcgen05.mma covers 128 weight
// rows x all tokens x 16 k.  The A operand is taken from TMEM: the FM layout's lane fragments are the lane fragments of
// tcgen05.st.16x256b, so a dequantiser warp turns its words into fp16 weights and stores them to TMEM directly, without
// a pass through shared memory.  The work is the list of (128-row tile, 128-k batch) units, tile by tile; CTA c takes
// the contiguous range [c U / G, (c + 1) U / G) of it, so every SM has the same share for every shape.  Per CTA:
//   warp 0       bulk copies of the packed weights (four 32-row panels a unit) into a ring of shared-memory stages; they do
//                not depend on the previous kernel and start before the dependency wait
//   warp 1       its first lane issues tcgen05.mma (kind f16, A in TMEM, B in shared memory, fp32 accumulator in TMEM)
//   warp 2       TMA: fp16 activation tiles [tokens][64 k] (128-byte swizzle)
//   warps 4-11   epilogue (store, residual + next-norm statistics, SwiGLU, fp32, argmax partials as in the GEMV): two
//                warps per 32 TMEM lanes, half of the tokens each; accumulators are double-buffered up to 128 tokens
//   warps 12-23  dequantisers: three sets of four warps (one 32-row panel each) take the units in turn
// A tile that several CTAs share (at most its first and last tile of a CTA) meets in scratch memory; the CTA that
// arrives last adds the parts in k order.  The cuts depend on (n, k) only: a row's bits do not depend on the number of
// rows that travel with it.  Every wait is bounded; on expiry the CTA sets B2_ERR_TIMEOUT, frees its TMEM and returns.
// Replaces dequant_kt_kernel + cuBLAS and w4_gemm_kernel / w4h_bt_kernel of the reference
// (kernels/m1/m1_model.cu:1875-1895, kernels/src/w4_gemv.cu, w4h.cu) for every m above the GEMV's range.
//
// What bounds it: up to about 64 tokens the pace of the issuing warps (some 650 cycles a unit; two units are one pipeline
// step there, one barrier round for sixteen MMAs), beyond that the MMAs (256 tokens: 1024 cycles a unit at the nominal
// rate) and, above 128 tokens, the epilogue of a tile, since only one such accumulator fits TMEM.  The earlier kernel wrote
// fp16 tiles to shared memory from a register ring and cut k into equal slices (80 tiles x 2 slices = two waves of 148).
// 4 bits, graph replays over weights larger than L2, before -> now: 16 tokens qkv 55 -> 21 us, o 49 -> 19, gate_up 105 ->
// 56, down 94 -> 37, lm_head 303 -> 141; 256 tokens qkv 215 -> 46, o 211 -> 48, gate_up 222 -> 120 (1120 TFLOP/s), down
// 268 -> 79, lm_head 655 -> 327 (1220 TFLOP/s).
#include <cuda.h>

#include "common.cuh"
#include "wq_frag.cuh"

namespace b2 {

struct WqMmArgs {
  const uint8_t* wq; int n, k, m;
  int bits, group;
  int ctas;                   // b2_wq_mm_ctas(n, k)
  int n_pad;                  // token rows of the fp16 activation buffer: b2_wq_mm_npad(m)
  int per;                    // units of a pipeline step: 2 up to 64 tokens, else 1
  int raw_stages, bufs;       // shared-memory stages of packed weights; operand buffers (weights in TMEM, activations in shared memory)
  int epi;
  bf16* y; long ldy;
  const bf16* resid; long ldr;
  float* ss_out; int ss_ld;
  float* yf;
  float* amax_val; int* amax_idx; int n_valid;
  float* scratch; unsigned* counters;
  int* status;
};

namespace {

enum { EPI_STORE = 0, EPI_RESID = 1, EPI_SWIGLU = 2, EPI_F32 = 3, EPI_ARGMAX = 4 };
constexpr int BM = 128, BKS = 64;                // BKS: width of one 128-byte swizzle atom in fp16 elements
constexpr int kMmThreads = 768;                  // 24 warps: weights, MMA, activations, spare, 8 epilogue, 12 dequantisers
constexpr int kEpiWarp0 = 4, kEpiWarps = 8, kDqWarp0 = 12, kDqSets = 3;
constexpr int kMaxRaw = 16, kMaxBuf = 4;
constexpr int kTmemColsM = 512;

__device__ __forceinline__ void mbar_arrive_m(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d_m(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D fp32, A and B fp16 (format 0), both K-major
__host__ __device__ constexpr uint32_t idesc_f16(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_m(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16_m(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// 16 TMEM lanes x 64 columns: register 4 s + i of lane (g, t) goes to lane g + 8 (i >> 1), column 8 s + 2 t + (i & 1)
__device__ __forceinline__ void tmem_st_frag(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x8.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
        "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
        "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ uint32_t hfma2_u(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// Position in a ring of `n` stages: stage index and the parity of the phase that is filled (or freed) there.  Advanced by
// additions: a division by a run-time count costs some 200 cycles of latency, and the MMA issuer has 300 a unit.
struct RingPos {
  int s = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next(int n, int by = 1) {
    s += by;
    while (s >= n) { s -= n; ph ^= 1u; }
  }
};

// fp16 weights of one 16-row block x 128 k from the lane's FM words, in the register order of tmem_st_frag.
// code = (1024 + c code) / c - 1024 / c (exact), weight = code * scale - zero * scale with zero * scale formed in fp16
// (one rounding of the product, as an fp32 product rounded once would give).
template <int BITS, int GROUP>
__device__ __forceinline__ void dequant_frag(const WFrag<BITS, GROUP>& f, uint32_t (&out)[32]) {
  constexpr int GPB = 128 / GROUP;
#pragma unroll
  for (int gi = 0; gi < GPB; ++gi) {
    const __half2 z0 = *reinterpret_cast<const __half2*>(&f.sz[gi][0]), z1 = *reinterpret_cast<const __half2*>(&f.sz[gi][1]);
    const __half2 s0h = __low2half2(z0), s1h = __low2half2(z1);
    const __half2 b0h = __hneg2(__hmul2(__high2half2(z0), s0h)), b1h = __hneg2(__hmul2(__high2half2(z1), s1h));
    const uint32_t sc0 = *reinterpret_cast<const uint32_t*>(&s0h), sc1 = *reinterpret_cast<const uint32_t*>(&s1h);
    const uint32_t bi0 = *reinterpret_cast<const uint32_t*>(&b0h), bi1 = *reinterpret_cast<const uint32_t*>(&b1h);
#pragma unroll
    for (int s8 = 0; s8 < 8 / GPB; ++s8) {
      const int s = gi * (8 / GPB) + s8;
      uint32_t a[4];
      extract<BITS, GROUP>(f, s, a);
      // fp16 bit patterns of (1 / c, -1024 / c); c = 1, 16 (4 bits); 1, 4 and 16, 64 on odd steps (2 and 3 bits)
      const uint32_t m0 = (BITS != 4 && (s & 1)) ? 0x2C002C00u : 0x3C003C00u, a0 = (BITS != 4 && (s & 1)) ? 0xD400D400u : 0xE400E400u;
      const uint32_t m1 = BITS == 4 ? 0x2C002C00u : ((s & 1) ? 0x24002400u : 0x34003400u);
      const uint32_t a1 = BITS == 4 ? 0xD400D400u : ((s & 1) ? 0xCC00CC00u : 0xDC00DC00u);
      out[4 * s + 0] = hfma2_u(hfma2_u(a[0], m0, a0), sc0, bi0);     // row g, slots 0, 1
      out[4 * s + 1] = hfma2_u(hfma2_u(a[2], m1, a1), sc0, bi0);     // row g, slots 2, 3
      out[4 * s + 2] = hfma2_u(hfma2_u(a[1], m0, a0), sc1, bi1);     // row g + 8
      out[4 * s + 3] = hfma2_u(hfma2_u(a[3], m1, a1), sc1, bi1);
    }
  }
}

// Epilogue of one output value per lane (row) and token; `part` = 32-row panel of the warp.
template <int EPI>
__device__ __forceinline__ void mm_emit(const WqMmArgs& a, float val, int tok, int row, bool row_ok, int part, int npan, int lane) {
  if (EPI == EPI_STORE) {
    if (row_ok) a.y[(size_t)tok * a.ldy + row] = __float2bfloat16_rn(val);
  } else if (EPI == EPI_F32) {
    if (row_ok) a.yf[(size_t)tok * a.ldy + row] = val;
  } else if (EPI == EPI_RESID) {
    float sq = 0.f;
    if (row_ok) {
      const bf16 hb = __float2bfloat16_rn(val + __bfloat162float(a.resid[(size_t)tok * a.ldr + row]));
      a.y[(size_t)tok * a.ldy + row] = hb;
      const float hf = __bfloat162float(hb);
      sq = hf * hf;
    }
    sq = warp_sum(sq);
    if (lane == 0 && a.ss_out && part < npan) a.ss_out[(size_t)part * a.ss_ld + tok] = sq;
  } else if (EPI == EPI_SWIGLU) {
    const float up = __shfl_down_sync(0xffffffffu, val, 8);
    if ((lane & 8) == 0 && row_ok)
      a.y[(size_t)tok * a.ldy + (size_t)part * 16 + (lane >> 4) * 8 + (lane & 7)] = __float2bfloat16_rn(silu_f(bf16_round(val)) * bf16_round(up));
  } else {
    if (a.yf && row_ok) a.yf[(size_t)tok * a.ldy + row] = val;
    float best = (row_ok && row < a.n_valid) ? val : -INFINITY;
    int bi = (row_ok && row < a.n_valid) ? row : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0 && part < npan) { a.amax_val[(size_t)part * a.ss_ld + tok] = best; a.amax_idx[(size_t)part * a.ss_ld + tok] = bi; }
  }
}
template <int EPI>
__device__ __forceinline__ void mm_emit16(const WqMmArgs& a, const float (&v)[16], int c0, int c1, int row, bool row_ok, int part, int npan, int lane) {
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (c0 + i < c1) mm_emit<EPI>(a, v[i], c0 + i, row, row_ok, part, npan, lane);
}

}  // namespace

template <int BITS, int GROUP>
__global__ void __launch_bounds__(kMmThreads, 1) wq_mm_kernel(const __grid_constant__ CUtensorMap map_x, const WqMmArgs a) {
  using R = Ring<BITS, GROUP, 2>;
  constexpr int GPB = 128 / GROUP;
  constexpr int RAW = 4 * R::BLK;                     // packed weights of one unit
  extern __shared__ __align__(1024) uint8_t smem_m[];
  // one pair of barriers per operand buffer (four dequantiser warps and one TMA arrive; one commit frees both operands)
  __shared__ __align__(8) uint64_t raw_full[kMaxRaw], raw_empty[kMaxRaw], op_full[kMaxBuf], op_empty[kMaxBuf], d_full[2], d_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_failed;
  __shared__ unsigned s_prev;

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int RS = a.raw_stages;
  const uint32_t x_sub = (uint32_t)a.n_pad * BKS * 2;
  const int P = a.per, NB = a.bufs;
  const uint32_t x_step = (uint32_t)P * 2 * x_sub, raw_step = (uint32_t)(P * RAW);
  const uint32_t x_ring = (smem_u32(smem_m) + 1023u) & ~1023u;                     // [NB][P][2 halves of k][n_pad rows][128 B]
  const uint32_t raw_ring = x_ring + (uint32_t)NB * x_step;                        // [RS][4 panels][P][block]
  uint8_t* raw_ptr = smem_m + (raw_ring - smem_u32(smem_m));
  const int nbat = a.k / 128, npan = a.n / 32;
  const int tiles = (a.n + BM - 1) / BM;
  const long U = (long)tiles * nbat;
  const long lo = U * blockIdx.x / a.ctas;
  const int nu = (int)(U * (blockIdx.x + 1) / a.ctas - lo);                        // units of this CTA
  const int tile0 = (int)(lo / nbat), kb0 = (int)(lo - (long)tile0 * nbat);
  const int nd = a.n_pad <= 128 ? 2 : 1;                                           // accumulators

  if (threadIdx.x == 0) {
    for (int i = 0; i < RS; ++i) { mbar_init(smem_u32(&raw_full[i]), 1); mbar_init(smem_u32(&raw_empty[i]), 4); }
    for (int i = 0; i < NB; ++i) { mbar_init(smem_u32(&op_full[i]), 5); mbar_init(smem_u32(&op_empty[i]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&d_full[i]), 1); mbar_init(smem_u32(&d_empty[i]), kEpiWarps); }
    s_failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kTmemColsM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_slot;
  const uint32_t tmem_d0 = tmem_base + (uint32_t)(NB * P) * 64;

  if (warp == 0) {
    // ---------------- packed weights ----------------
    // lane p < 4 copies panel p of every step
    int left = nbat - kb0, tile = tile0;
    const uint8_t* src = a.wq + ((size_t)min(tile * 4 + (lane & 3), npan - 1) * nbat + kb0) * R::BLK;
    uint32_t full = smem_u32(&raw_full[0]), empty = smem_u32(&raw_empty[0]), dst = raw_ring + (uint32_t)((lane & 3) * P * R::BLK);
    uint32_t ph = 1;
    for (int i = 0, st = 0, s = 0; i < nu; ++st) {
      const int cnt = min(P, min(left, nu - i));
      if (st >= RS && !mbar_wait_warp(empty, ph)) { atomicExch(&s_failed, 1); break; }
      if (lane == 0) mbar_expect_tx(full, (uint32_t)(cnt * RAW));
      __syncwarp();
      if (lane < 4) bulk_g2s(dst, src, (uint32_t)(cnt * R::BLK), full);
      i += cnt;
      src += cnt * R::BLK;
      left -= cnt;
      if (left == 0) {               // a ragged last tile repeats the last panel; its rows are never stored
        left = nbat;
        ++tile;
        src = a.wq + (size_t)min(tile * 4 + (lane & 3), npan - 1) * nbat * R::BLK;
      }
      full += 8; empty += 8; dst += raw_step;
      if (++s == RS) { s = 0; ph ^= 1u; full -= RS * 8; empty -= RS * 8; dst -= RS * raw_step; }
    }
  } else if (warp == 2) {
    // ---------------- activation tiles by TMA (written by the previous kernel) ----------------
    if (lane == 0) {
      pdl_wait();
      pdl_launch_dependents();
      int kb = kb0;
      RingPos r;
      for (int i = 0, st = 0; i < nu; ++st, r.next(NB)) {
        const int cnt = min(P, min(nbat - kb, nu - i));
        if (st >= NB && !mbar_wait_quick(smem_u32(&op_empty[r.s]), r.ph ^ 1u)) { atomicExch(&s_failed, 1); break; }
        const uint32_t bar = smem_u32(&op_full[r.s]);
        mbar_expect_tx(bar, (uint32_t)cnt * 2 * x_sub);
        for (int h = 0; h < 2 * cnt; ++h) tma_load_2d_m(x_ring + r.s * x_step + h * x_sub, &map_x, kb * 128 + h * BKS, 0, bar);
        i += cnt;
        kb += cnt;
        if (kb == nbat) kb = 0;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // The whole warp runs the loop and its first lane issues: addresses then stay in uniform registers, which tcgen05.mma
    // takes its operands from (under `if (lane == 0)` around the loop an MMA took 70 cycles to issue, 1050 a unit).
    const uint32_t idesc = idesc_f16(BM, a.n_pad);
    const uint64_t dx_base = desc_sw128(x_ring);            // the address field counts 16 bytes
    const uint32_t dx_half = x_sub >> 4, dx_step = x_step >> 4, ta_step = (uint32_t)P * 64;
    const uint32_t full0 = smem_u32(&op_full[0]), empty0 = smem_u32(&op_empty[0]), wrap = (uint32_t)NB * 8;
    uint32_t off = 0, ph = 0, ta = tmem_base;
    uint64_t dx = dx_base;
    RingPos d;
    bool ok = true;
    int kb = kb0;
    for (int left = nu, frag = 0; left > 0 && ok; ++frag, d.next(nd)) {
      int cnt = min(nbat - kb, left);
      left -= cnt;
      kb = 0;
      if (frag >= nd && !mbar_wait_warp(smem_u32(&d_empty[d.s]), d.ph ^ 1u)) { ok = false; break; }
      const uint32_t td = tmem_d0 + (uint32_t)(d.s * a.n_pad);
      uint32_t acc = 0;
      while (cnt > 0) {
        const int c = min(P, cnt);
        cnt -= c;
        if (!mbar_wait_warp(full0 + off, ph)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t dh = dx + dx_half, dy = dh + dx_half, dz = dy + dx_half;
        if (lane == 0) {
          umma_f16(td, ta, dx, idesc, acc);
#pragma unroll
          for (int q = 1; q < 4; ++q) umma_f16(td, ta + q * 8, dx + 2 * q, idesc, 1u);
#pragma unroll
          for (int q = 0; q < 4; ++q) umma_f16(td, ta + 32 + q * 8, dh + 2 * q, idesc, 1u);
          if (c == 2) {
#pragma unroll
            for (int q = 0; q < 4; ++q) umma_f16(td, ta + 64 + q * 8, dy + 2 * q, idesc, 1u);
#pragma unroll
            for (int q = 0; q < 4; ++q) umma_f16(td, ta + 96 + q * 8, dz + 2 * q, idesc, 1u);
          }
          umma_commit_m(empty0 + off);
          if (cnt == 0) umma_commit_m(smem_u32(&d_full[d.s]));
        }
        __syncwarp();
        acc = 1u;
        off += 8; ta += ta_step; dx += dx_step;
        if (off == wrap) { off = 0; ta = tmem_base; dx = dx_base; ph ^= 1u; }
      }
    }
    if (!ok) s_failed = 1;
  } else if (warp >= kDqWarp0) {
    // ---------------- dequantisers: panel warp % 4 of every third unit ----------------
    const int p = warp & 3;
    const int set = (warp - kDqWarp0) >> 2;
    RingPos rw, rb;
    rw.next(RS, set);
    rb.next(NB, set);
    int kb = kb0, st = 0, turn = 0;
    for (int i = 0; i < nu; ++st) {
      const int cnt = min(P, min(nbat - kb, nu - i));
      i += cnt;
      kb += cnt;
      if (kb == nbat) kb = 0;
      const bool mine = turn == set;                        // the sets take the steps in turn
      if (++turn == kDqSets) turn = 0;
      if (!mine) continue;
      if (!mbar_wait_warp(smem_u32(&raw_full[rw.s]), rw.ph)) { atomicExch(&s_failed, 1); break; }
      bool ok = true;
      const uint8_t* blk = raw_ptr + rw.s * raw_step + p * P * R::BLK;
      for (int c = 0; c < cnt; ++c, blk += R::BLK) {
        WFrag<BITS, GROUP> f[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) load_frag_smem<BITS, GROUP>(f[r], blk + r * R::W_BATCH, blk + 2 * R::W_BATCH + r * GPB * 64, lane);
        if (c == cnt - 1) {
          __syncwarp();
          if (lane == 0) mbar_arrive_m(smem_u32(&raw_empty[rw.s]));
        }
        if (c == 0 && st >= NB) {                           // the packed words are in registers before this wait
          ok = mbar_wait_warp(smem_u32(&op_empty[rb.s]), rb.ph ^ 1u);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (!ok) break;
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          uint32_t w[32];
          dequant_frag<BITS, GROUP>(f[r], w);
          tmem_st_frag(tmem_base + ((uint32_t)(p * 32 + r * 16) << 16) + (uint32_t)((rb.s * P + c) * 64), w);
        }
      }
      if (!ok) { atomicExch(&s_failed, 1); break; }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_m(smem_u32(&op_full[rb.s]));
      rw.next(RS, kDqSets);
      rb.next(NB, kDqSets);
    }
  } else if (warp >= kEpiWarp0) {
    // ---------------- epilogue: TMEM lanes 32 (warp % 4), token half (warp - 4) / 4 ----------------
    pdl_wait();                                           // the residual comes from, and the scratch was used by, earlier kernels
    const int lane_base = (warp & 3) * 32, rit = lane_base + lane;
    const int half = ((a.n_pad / 2) + 15) & ~15;
    const int t0 = ((warp - kEpiWarp0) >> 2) * half, t1 = min(a.m, t0 + half);
    const size_t slot_sz = (size_t)a.n_pad * BM;
    int i = 0, tile = tile0, kb = kb0;
    bool dead = false;                                    // a wait gave up: no more waits or stores, but every barrier is kept
    RingPos d;
    for (int frag = 0; i < nu; ++frag, d.next(nd)) {
      const int db = d.s;
      const int len = min(nbat - kb, nu - i);
      const bool whole = len == nbat;
      if (!dead && !mbar_wait_warp(smem_u32(&d_full[db]), d.ph)) { dead = true; atomicExch(&s_failed, 1); }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t trow = tmem_d0 + ((uint32_t)lane_base << 16) + (uint32_t)(db * a.n_pad);
      const int row = tile * BM + rit, part = tile * 4 + (warp & 3);
      const bool row_ok = row < a.n;
      bool emit = whole && !dead;
      const float* parts = nullptr;
      int c_first = 0, c_last = 0;
      bool first_slot = false;
      if (!whole) {
        float* mine = a.scratch + (2 * (size_t)blockIdx.x + (frag ? 1 : 0)) * slot_sz + rit;
        for (int c0 = t0; c0 < t1 && !dead; c0 += 16) {
          uint32_t r[16];
          tmem_ld16_m(trow + (uint32_t)c0, r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c0 + j < t1) mine[(size_t)(c0 + j) * BM] = __uint_as_float(r[j]);
          __syncwarp();
        }
        __threadfence();
        c_first = (int)((((long)tile * nbat + 1) * a.ctas - 1) / U);
        c_last = (int)((((long)tile + 1) * nbat * a.ctas - 1) / U);
        first_slot = (int)(U * c_first / a.ctas / nbat) != tile;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (warp == kEpiWarp0 && lane == 0) s_prev = s_failed ? 0xffffffffu : atomicInc(a.counters + tile, (unsigned)(c_last - c_first));
        asm volatile("bar.sync 1, 256;" ::: "memory");
        emit = !dead && s_prev == (unsigned)(c_last - c_first);
        if (emit) __threadfence();
        parts = a.scratch + rit;
      }
      if (emit) {
        for (int c0 = t0; c0 < t1; c0 += 16) {
          float v[16];
          if (whole) {
            uint32_t r[16];
            tmem_ld16_m(trow + (uint32_t)c0, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = 0.f;
            // k order, two parts' loads in flight.  A CTA's slot 0 holds the tile it starts in, slot 1 the tile it ends
            // in, so only the first part can be in a slot 1.
            for (int c = c_first; c <= c_last; c += 2) {
              const float* q = parts + (2 * (size_t)c + (c == c_first && first_slot ? 1 : 0)) * slot_sz;
              const float* q1 = parts + 2 * (size_t)(c + 1) * slot_sz;
              float pv[16], pw[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) pv[j] = c0 + j < t1 ? __ldcg(q + (size_t)(c0 + j) * BM) : 0.f;
#pragma unroll
              for (int j = 0; j < 16; ++j) pw[j] = c0 + j < t1 && c < c_last ? __ldcg(q1 + (size_t)(c0 + j) * BM) : 0.f;
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] += pv[j];
              if (c < c_last) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += pw[j];
              }
            }
          }
          switch (a.epi) {
            case EPI_STORE: mm_emit16<EPI_STORE>(a, v, c0, t1, row, row_ok, part, npan, lane); break;
            case EPI_RESID: mm_emit16<EPI_RESID>(a, v, c0, t1, row, row_ok, part, npan, lane); break;
            case EPI_SWIGLU: mm_emit16<EPI_SWIGLU>(a, v, c0, t1, row, row_ok, part, npan, lane); break;
            case EPI_F32: mm_emit16<EPI_F32>(a, v, c0, t1, row, row_ok, part, npan, lane); break;
            default: mm_emit16<EPI_ARGMAX>(a, v, c0, t1, row, row_ok, part, npan, lane); break;
          }
          __syncwarp();                                   // single lanes store in there; the next tcgen05.ld is .aligned
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_m(smem_u32(&d_empty[db]));
      i += len;
      kb = 0;
      ++tile;
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_failed) {
    if (threadIdx.x == 0 && a.status) atomicExch(a.status, (int)B2_ERR_TIMEOUT);
    // copies still in flight get a bounded time to land before the CTA's shared memory is released
    const uint64_t t_end = globaltimer_ns() + 2000000ull;
    while (globaltimer_ns() < t_end) { }
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColsM) : "memory");
  }
}

// x (bf16 [m][ldx], optionally RMS-normalised with statistics left by the previous epilogue) -> fp16 [n_pad][k], rows
// >= m zero.  One CTA per output row.
__global__ void __launch_bounds__(256) wq_mm_xprep_kernel(const bf16* __restrict__ x, long ldx, int m, int k, const float* __restrict__ ss_in,
                                                          int ss_parts, int ss_ld, const bf16* __restrict__ norm_w, float eps,
                                                          __half* __restrict__ out) {
  __shared__ float s_inv;
  pdl_wait();
  pdl_launch_dependents();
  const int tok = blockIdx.x;
  __half* o = out + (size_t)tok * k;
  if (tok >= m) {
    for (int i = threadIdx.x * 8; i < k; i += 256 * 8) *reinterpret_cast<uint4*>(o + i) = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  float inv = 1.f;
  if (norm_w) {
    if (threadIdx.x < 32) {
      float s = 0.f;
      for (int p = threadIdx.x; p < ss_parts; p += 32) s += ss_in[(size_t)p * ss_ld + tok];
      s = warp_sum(s);
      if (threadIdx.x == 0) s_inv = rsqrtf(s / (float)k + eps);
    }
    __syncthreads();
    inv = s_inv;
  }
  for (int i = threadIdx.x * 8; i < k; i += 256 * 8) {
    const uint4 raw = *reinterpret_cast<const uint4*>(x + (size_t)tok * ldx + i);
    const bf16* xb = reinterpret_cast<const bf16*>(&raw);
    __align__(16) __half hv[8];
    if (norm_w) {
      const uint4 wr = *reinterpret_cast<const uint4*>(norm_w + i);
      const bf16* wb = reinterpret_cast<const bf16*>(&wr);
#pragma unroll
      for (int j = 0; j < 8; ++j) hv[j] = __float2half_rn(bf16_round(__bfloat162float(xb[j]) * inv * __bfloat162float(wb[j])));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) hv[j] = __float2half_rn(__bfloat162float(xb[j]));
    }
    *reinterpret_cast<uint4*>(o + i) = *reinterpret_cast<const uint4*>(hv);
  }
}

}  // namespace b2

using namespace b2;

typedef CUresult (*EncodeTiledFnM)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFnM encode_fn_m() {
  static EncodeTiledFnM fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFnM>(p);
  }
  return fn;
}

// CTAs of a linear, a function of the shape only: one per SM of a 148-SM part, at least kMinUnitsM units each (a unit
// takes 0.2 us, the hand-over of a shared tile 3 and more), but a tile of fewer units has a CTA of its own (5120 x 256 at 16
// rows: 6.5 us, 12.7 with tiles put together; the kernel before 8.2).
static const int kMmCtas = 148, kMinUnitsM = 6;
B2_API int b2_wq_mm_ctas(int n, int k) {
  const long tiles = (n + BM - 1) / BM, U = tiles * (k / 128);
  const long c = U / kMinUnitsM > tiles ? U / kMinUnitsM : tiles;
  return (int)(c > kMmCtas ? kMmCtas : c);
}
B2_API int b2_wq_mm_npad(int m) { return m <= 16 ? 16 : (m + 15) / 16 * 16; }
// Partial tiles: two slots per CTA.
B2_API long b2_wq_mm_scratch_floats(int n, int k, int n_pad) { return 2L * b2_wq_mm_ctas(n, k) * n_pad * BM; }

// x16: caller-provided fp16 [n_pad][k] staging buffer (16-byte aligned).  pro_norm: ss_in / norm_w given.
B2_API int b2_wq_mm(const WqMmArgs* args, const bf16* x, long ldx, const float* ss_in, int ss_parts, int ss_ld, const bf16* norm_w,
                    float eps, __half* x16, cudaStream_t st) {
  WqMmArgs a = *args;
  if (a.n <= 0 || a.n % 32 || a.k % 128 || a.m < 1 || a.m > 256 || (a.bits != 2 && a.bits != 3 && a.bits != 4) ||
      (a.group != 64 && a.group != 128) || !x || !x16 || (ldx % 8))
    return B2_ERR_ARG;
  a.n_pad = b2_wq_mm_npad(a.m);
  a.ctas = b2_wq_mm_ctas(a.n, a.k);
  if ((a.epi == EPI_RESID || a.epi == EPI_ARGMAX) && a.m > a.ss_ld) return B2_ERR_ARG;
  if (!a.scratch || !a.counters) return B2_ERR_ARG;
  // TMEM holds bufs x 64 columns of weights and the accumulators; shared memory the activation tiles and about 64 KB of
  // packed weights (what is left above 160 tokens, whose activation tiles are large)
  const int raw = 8 * (a.bits == 3 ? 768 : (a.bits == 4 ? 1024 : 512)) + 8 * (128 / a.group) * 64;
  const int x_sub = a.n_pad * BKS * 2;
  // A step of two units halves the issuing warps' cost per unit; its three buffers take 384 TMEM columns, which leaves two
  // accumulators of 64 tokens.  With four buffers a dequantiser set uses a buffer every third time only: that its wait for
  // the commit of step st - 4 cannot take the phase of st - 8 for it rests on the commits of one thread arriving in order, of
  // which it saw st - 7 a whole dequantisation earlier.  Three buffers there: 5120 x 25600 at 72 tokens 44 -> 48 us, else equal.
  a.per = a.n_pad <= 64 ? 2 : 1;
  a.bufs = a.n_pad <= 64 ? 3 : (a.n_pad <= 160 ? 4 : 3);
  const int left = 220 * 1024 - a.bufs * a.per * 2 * x_sub;
  a.raw_stages = (left < 80 * 1024 ? left : 80 * 1024) / (a.per * raw);
  if (a.raw_stages > kMaxRaw) a.raw_stages = kMaxRaw;
  // A multiple of the dequantiser sets: a stage is then always read by the same set, which has seen its previous phase
  // complete before it waits for the next (a parity wait must not come a phase early).
  a.raw_stages -= a.raw_stages % kDqSets;
  if (a.raw_stages < kDqSets) return B2_ERR_ARG;
  EncodeTiledFnM fn = encode_fn_m();
  if (!fn) return B2_ERR_LAUNCH;
  CUtensorMap mx;
  cuuint64_t dims[2] = {(cuuint64_t)a.k, (cuuint64_t)a.n_pad};
  cuuint64_t strides[1] = {(cuuint64_t)a.k * 2};
  cuuint32_t box[2] = {(cuuint32_t)BKS, (cuuint32_t)a.n_pad};
  cuuint32_t estr[2] = {1, 1};
  if (fn(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x16, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return B2_ERR_LAUNCH;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.n_pad); cfg.blockDim = dim3(256); cfg.stream = st; cfg.attrs = at; cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, wq_mm_xprep_kernel, x, ldx, a.m, a.k, ss_in, ss_parts, ss_ld, norm_w, eps, x16) != cudaSuccess)
      return B2_ERR_LAUNCH;
  }
  const size_t smem = (size_t)a.bufs * a.per * 2 * x_sub + (size_t)a.raw_stages * a.per * raw + 1024;
  void (*kern)(const CUtensorMap, const WqMmArgs) = nullptr;
  if (a.bits == 4) kern = a.group == 128 ? wq_mm_kernel<4, 128> : wq_mm_kernel<4, 64>;
  else if (a.bits == 3) kern = a.group == 128 ? wq_mm_kernel<3, 128> : wq_mm_kernel<3, 64>;
  else kern = a.group == 128 ? wq_mm_kernel<2, 128> : wq_mm_kernel<2, 64>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024) != cudaSuccess) return B2_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)a.ctas, 1, 1);
  cfg.blockDim = dim3(kMmThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, mx, a) == cudaSuccess ? B2_OK : B2_ERR_LAUNCH;
}
