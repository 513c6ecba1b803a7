// Mixed 2/3/4-bit dequant GEMV for one to eight token rows (decode, small verify blocks), sm_100a; more rows run in
// chunks of eight.  Same weight layout, arithmetic per group and epilogues as wq_gemv.cu, whose kernel stays for the
// tensor-parallel push epilogue and for matrices beyond the schedule here (b2_wq_gemv8_takes).
//
// Work: the units (32-row panel, 128-k batch) of the matrix.  k is cut into equal slices of at most 5120 inputs, so that
// a CTA's activations fit its shared memory at eight rows, and every slice has the same number of CTAs; CTA c of a slice
// takes the c-th share of the slice's units in panel order, its sixteen warps consecutive shares of that.  A panel
// segment inside one warp is finished by that warp; one that several warps share meets in shared memory, one that several
// CTAs or slices share in scratch memory, where the last arriver adds the parts in (slice, CTA) order.  Matrices of one
// slice with at least eight panels per CTA are cut at panels and need no scratch.  Cuts and orders depend on (n, k) only,
// so a row's bits do not depend on the rows that travel with it.
//
// One CTA of 16 warps per SM at full registers.  (64 registers and half of the shared memory, so that the next linear's
// CTAs could prefetch beside this one, measured slower: four 32B layers and the head at one row 747 us, 420 in this form
// with its slices of k -- the early CTAs keep the attention kernels between the linears off the SMs.)
//
// What bounds it: large matrices the inner loop (the logic pipe takes two cycles an instruction and scheduler, some 110 of
// them a unit, and 16 half-precision MMAs of 8) and, at 4 bits, DRAM; small ones the fixed 4 us of launch, staging and
// hand-over.  The kernel of wq_gemv.cu staged every row of a CTA's slice and summed every row's parts one after the
// other, and its shared memory left one CTA of eight warps per SM from five rows on.  4 bits, graph replays over weights
// larger than L2, before -> now: one row gate_up 36 -> 28 us, lm_head 82 -> 72 (floor 63), down 25 -> 19, qkv 14.0 ->
// 11.5, o 13.6 -> 10.7, 4096 x 1024 7.2 -> 3.9; eight rows gate_up 101 -> 35, lm_head 199 -> 78, down 191 -> 26, qkv
// 64 -> 16, o 79 -> 15.
#include "wq_frag.cuh"
#include "wq_gemv.cuh"

namespace b2 {

struct Gemv8Plan {
  int slices, per_slice;         // functions of (n, k): slices of k, CTAs per slice
  int panel_cut;
  int fmax;                      // most CTAs that share a segment
  int xb;                        // batches of the longest slice
  int nst;                       // ring stages per warp
};

namespace {

constexpr int kW8 = 16, kT8 = kW8 * 32;

__device__ __forceinline__ int slice_base(int s, int nbat, int S) { return s * nbat / S; }

}  // namespace

// ONE: a single row (columns other than the token's are not scaled); otherwise two to eight rows.
template <int BITS, int GROUP, bool ONE>
__global__ void __launch_bounds__(kT8, 1) wq_gemv8_kernel(const WqGemvArgs a, const Gemv8Plan p) {
  constexpr int GPB = 128 / GROUP;
  constexpr int MP = ONE ? 1 : 8;
  using R = Ring<BITS, GROUP, 2>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int m = ONE ? 1 : a.m;
  const int npan = a.n >> 5, nbat = a.k >> 7, S = p.slices;
  const unsigned G = (unsigned)p.per_slice;
  const int slice = (int)(blockIdx.x / G);
  const unsigned cta = blockIdx.x - (unsigned)slice * G;
  const int base = slice_base(slice, nbat, S), len = slice_base(slice + 1, nbat, S) - base;   // batches of this slice
  const unsigned U = (unsigned)npan * (unsigned)len;                                          // its units
  const int NST = p.nst;
  const int XST = p.xb * 128 + 16;               // halfs per staged row (row pitch = 32 B mod 128 B)

  // shared memory: [16 rings][barriers][1/rms][16 x 2 partial tiles][group sums][activations]
  const uint32_t ring_u = smem_u32(smem_raw) + (uint32_t)(warp * NST * R::BLK);
  const uint8_t* ring = smem_raw + (size_t)warp * NST * R::BLK;
  uint8_t* after = smem_raw + (size_t)kW8 * NST * R::BLK;
  const uint32_t bars_u = smem_u32(after) + (uint32_t)(warp * NST * 8);
  float* inv_rms = reinterpret_cast<float*>(after + kW8 * NST * 8);
  float* tiles = inv_rms + 8;                                              // [16][2][m][32]
  float2* gsum = reinterpret_cast<float2*>(tiles + (size_t)kW8 * 2 * m * 32);   // [xb * GPB][MP]
  __half* xs = reinterpret_cast<__half*>(gsum + (((size_t)p.xb * GPB * MP + 1) & ~(size_t)1));  // [m][XST]
  auto tile_of = [&](int w, int which) { return tiles + (size_t)((w * 2 + which) * m) * 32; };

  // ranges of units: CTA [lo, hi), warp [wlo, whi); unit u = batch u % len of panel u / len
  const unsigned lo = p.panel_cut ? (unsigned)npan * cta / G * (unsigned)len : U * cta / G;
  const unsigned hi = p.panel_cut ? (unsigned)npan * (cta + 1) / G * (unsigned)len : U * (cta + 1) / G;
  const unsigned nu = hi - lo;
  auto warp_lo = [&](int w) { return lo + (unsigned)w * nu / kW8; };
  auto warp_of = [&](unsigned u) { return (int)(((u - lo + 1) * kW8 - 1) / nu); };
  const unsigned wlo = warp_lo(warp), whi = warp_lo(warp + 1);

  if (lane == 0) {
    for (int i = 0; i < NST; ++i) mbar_init(bars_u + i * 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  // weights do not depend on the previous kernel: fill the ring before the dependency wait
  const int wpan = (int)(wlo / (unsigned)len), wb = (int)(wlo - (unsigned)wpan * (unsigned)len);
  // producer (lane 0): source of the next unit, units left in its panel and in this warp's range
  const uint8_t* psrc = a.wq + ((size_t)wpan * nbat + base + wb) * R::BLK;
  int pseg = len - wb, pleft = (int)(whi - wlo);
  uint32_t pdst = ring_u, pbar = bars_u;
  auto issue = [&]() {
    mbar_expect_tx(pbar, (uint32_t)R::BLK);
    bulk_g2s(pdst, psrc, (uint32_t)R::BLK, pbar);
    pdst += R::BLK;
    pbar += 8;
    if (pbar == bars_u + NST * 8) { pbar = bars_u; pdst = ring_u; }
    psrc += R::BLK;
    --pleft;
    if (--pseg == 0) {           // on to the slice's batches of the next panel
      psrc += (size_t)(nbat - len) * R::BLK;
      pseg = len;
    }
  };
  if (lane == 0) {
    for (int i = 0; i < NST && pleft > 0; ++i) issue();
  }
  __syncwarp();
  const int nvec = len * 16, total = nvec * m;
  auto item = [&](int i, int& tok, int& v) { tok = ONE ? 0 : i / nvec; v = i - tok * nvec; };
  uint4 pre[2], prw[2];
  pdl_wait();                      // nothing but packed weights is read before this
  pdl_launch_dependents();

  // ---- stage the activations of the slice: fp16(x / c) and the per-group sums ----
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = (int)threadIdx.x + j * kT8;
    pre[j] = prw[j] = make_uint4(0u, 0u, 0u, 0u);
    if (i < total) {
      int tok, v;
      item(i, tok, v);
      pre[j] = *reinterpret_cast<const uint4*>(a.x + (size_t)tok * a.ldx + base * 128 + v * 8);
      if (a.pro == PRO_NORM) prw[j] = *reinterpret_cast<const uint4*>(a.norm_w + base * 128 + v * 8);
    }
  }
  if (a.pro == PRO_NORM) {
    if (warp < m) {
      // partial sums are fetched eight at a time so that their latencies overlap; the order of the adds is fixed
      float s = 0.f;
      for (int p0 = lane; p0 < a.ss_parts; p0 += 256) {
        float pv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int q = p0 + 32 * i;
          pv[i] = q < a.ss_parts ? a.ss_in[(size_t)q * a.ss_ld + warp] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) s += pv[i];
      }
      s = warp_sum(s);
      if (lane == 0) inv_rms[warp] = rsqrtf(s / (float)a.k + a.eps);
    }
    __syncthreads();
  }
  for (int i0 = 0; i0 < total; i0 += 2 * kT8) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int i = i0 + j * kT8 + (int)threadIdx.x;
      const bool act = i < total;
      float ssum = 0.f, xsum = 0.f;
      int tok = 0, v = 0;
      if (act) {
        item(i, tok, v);
        const uint4 raw = pre[j];
        const bf16* xb = reinterpret_cast<const bf16*>(&raw);
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __bfloat162float(xb[e]);
        if (a.pro == PRO_NORM) {
          const uint4 wr = prw[j];
          const bf16* wb = reinterpret_cast<const bf16*>(&wr);
          const float ir = inv_rms[tok];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = bf16_round(f[e] * ir * __bfloat162float(wb[e]));
        }
        __align__(16) __half h[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float cinv, c;
          slot_scale<BITS>((v * 8 + e) & 127, cinv, c);
          h[e] = __float2half_rn(f[e] * cinv);
          const float hf = __half2float(h[e]);
          ssum += hf;
          xsum += hf * c;
        }
        *reinterpret_cast<uint4*>(xs + (size_t)tok * XST + v * 8) = *reinterpret_cast<const uint4*>(h);
      }
      // reduce over the GROUP / 8 lanes that cover one group (fixed xor tree)
#pragma unroll
      for (int o = GROUP / 16; o > 0; o >>= 1) {
        ssum += __shfl_xor_sync(0xffffffffu, ssum, o);
        xsum += __shfl_xor_sync(0xffffffffu, xsum, o);
      }
      if (act && (lane % (GROUP / 8)) == 0) gsum[((v * 8) / GROUP) * MP + tok] = make_float2(1024.f * ssum, xsum);
      const int in = i + 2 * kT8;
      if (in < total) {
        int tk, vn;
        item(in, tk, vn);
        pre[j] = *reinterpret_cast<const uint4*>(a.x + (size_t)tk * a.ldx + base * 128 + vn * 8);
        if (a.pro == PRO_NORM) prw[j] = *reinterpret_cast<const uint4*>(a.norm_w + base * 128 + vn * 8);
      }
    }
  }
  __syncthreads();

  // Epilogue of one panel: v[tok] of row pan * 32 + lane.
  auto epilogue = [&](int pan, const float (&v)[MP]) {
    const int row = pan * 32 + lane;
    if (a.epi == EPI_STORE) {
#pragma unroll
      for (int tok = 0; tok < MP; ++tok)
        if (tok < m) a.y[(size_t)tok * a.ldy + row] = __float2bfloat16_rn(v[tok]);
    } else if (a.epi == EPI_F32) {
#pragma unroll
      for (int tok = 0; tok < MP; ++tok)
        if (tok < m) a.yf[(size_t)tok * a.ldy + row] = v[tok];
    } else if (a.epi == EPI_RESID) {
      float rs[MP];
#pragma unroll
      for (int tok = 0; tok < MP; ++tok) rs[tok] = tok < m ? __bfloat162float(a.resid[(size_t)tok * a.ldr + row]) : 0.f;
#pragma unroll
      for (int tok = 0; tok < MP; ++tok) {
        if (tok < m) {
          const bf16 hb = __float2bfloat16_rn(v[tok] + rs[tok]);
          a.y[(size_t)tok * a.ldy + row] = hb;
          const float hf = __bfloat162float(hb);
          const float sq = warp_sum(hf * hf);
          if (lane == 0 && a.ss_out) a.ss_out[(size_t)pan * a.ss_ld + tok] = sq;
        }
      }
    } else if (a.epi == EPI_SWIGLU) {
      // lanes 0-7 / 16-23 hold gate rows, lanes 8-15 / 24-31 the matching up rows
#pragma unroll
      for (int tok = 0; tok < MP; ++tok) {
        if (tok < m) {
          const float up = __shfl_down_sync(0xffffffffu, v[tok], 8);
          if ((lane & 8) == 0)
            a.y[(size_t)tok * a.ldy + (size_t)pan * 16 + (lane >> 4) * 8 + (lane & 7)] =
                __float2bfloat16_rn(silu_f(bf16_round(v[tok])) * bf16_round(up));
        }
      }
    } else if (a.epi == EPI_ARGMAX) {
#pragma unroll
      for (int tok = 0; tok < MP; ++tok) {
        if (tok < m) {
          if (a.yf) a.yf[(size_t)tok * a.ldy + row] = v[tok];
          float best = row < a.n_valid ? v[tok] : -INFINITY;
          int bi = row < a.n_valid ? row : 0x7fffffff;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
          }
          if (lane == 0) {
            a.amax_val[(size_t)pan * a.ss_ld + tok] = best;
            a.amax_idx[(size_t)pan * a.ss_ld + tok] = bi;
          }
        }
      }
    }
  };
  // This CTA's part of panel `pan` is complete in v: the epilogue if that is the whole panel, else the hand-over through
  // scratch.
  auto finish = [&](int pan, bool whole, float (&v)[MP]) {
    if (whole && S == 1) { epilogue(pan, v); return; }
    // lane l: CTAs of slice l that share the panel.  The CTA of unit u is the last whose range begins at or before it.
    int first = 0, cnt = 0;
    if (lane < S) {
      const unsigned ll = (unsigned)(slice_base(lane + 1, nbat, S) - slice_base(lane, nbat, S)), Ul = (unsigned)npan * ll;
      first = (int)((((unsigned)pan * ll + 1u) * G - 1u) / Ul);
      cnt = (int)((((unsigned)pan + 1u) * ll * G - 1u) / Ul) - first + 1;
    }
    const int my_first = __shfl_sync(0xffffffffu, first, slice);
    int nparts = cnt;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nparts += __shfl_xor_sync(0xffffffffu, nparts, o);
    const size_t tsz = (size_t)m * 32;
    float* mine = a.scratch + (((size_t)slice * npan + pan) * p.fmax + ((int)cta - my_first)) * tsz + lane;
#pragma unroll
    for (int tok = 0; tok < MP; ++tok)
      if (tok < m) mine[tok * 32] = v[tok];
    __threadfence();
    __syncwarp();
    unsigned prev = 0;
    if (lane == 0) prev = atomicInc(a.counters + pan, (unsigned)nparts - 1u);
    prev = __shfl_sync(0xffffffffu, prev, 0);
    if (prev != (unsigned)nparts - 1u) return;
    __threadfence();
#pragma unroll
    for (int tok = 0; tok < MP; ++tok) v[tok] = 0.f;
    constexpr int FL = ONE ? 16 : 2;              // parts in flight
    int es = 0, ef = 0, ecnt = __shfl_sync(0xffffffffu, cnt, 0);
    for (int p0 = 0; p0 < nparts; p0 += FL) {
      float pv[FL][MP];
#pragma unroll
      for (int i = 0; i < FL; ++i) {
        const bool on = p0 + i < nparts;
        const float* q = a.scratch + (((size_t)es * npan + pan) * p.fmax + ef) * tsz + lane;
#pragma unroll
        for (int tok = 0; tok < MP; ++tok) pv[i][tok] = on && tok < m ? __ldcg(q + tok * 32) : 0.f;
        if (on && ++ef == ecnt) {
          ef = 0;
          if (es + 1 < S) ++es;
          ecnt = __shfl_sync(0xffffffffu, cnt, es);
        }
      }
#pragma unroll
      for (int i = 0; i < FL; ++i)
#pragma unroll
        for (int tok = 0; tok < MP; ++tok)
          if (p0 + i < nparts) v[tok] += pv[i][tok];
    }
    epilogue(pan, v);
  };

  // ---- main loop over this warp's units ----
  const uint8_t* cptr = ring;
  uint32_t cbar = bars_u, cph = 0;
  bool failed = false;
  const bool tok_ok = g < m;
  int pan = wpan, b0 = wb;
  for (unsigned u = wlo; u < whi && !failed; ++pan, b0 = 0) {
    // one fragment: the units of this panel inside [u, whi)
    const unsigned seg0 = (unsigned)pan * (unsigned)len, seg1 = seg0 + (unsigned)len;
    const int cnt = (int)(min(seg1, whi) - u);
    const __half* xrow = xs + (size_t)(ONE ? 0 : (tok_ok ? g : 0)) * XST + b0 * 128 + t * 4;
    const float2* gs = gsum + (size_t)(b0 * GPB) * MP + (ONE ? 0 : 2 * t);
    u += (unsigned)cnt;
    float y[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) y[r][i] = 0.f;
#pragma unroll 1
    for (int i = 0; i < cnt; ++i) {
      if (!mbar_wait_warp(cbar, cph)) {           // voted: the mma below are .aligned
        if (a.status && lane == 0) atomicExch(a.status, (int)B2_ERR_TIMEOUT);
        failed = true;
        break;
      }
      WFrag<BITS, GROUP> cf[2];
#pragma unroll
      for (int r = 0; r < 2; ++r)
        load_frag_smem<BITS, GROUP>(cf[r], cptr + r * R::W_BATCH, cptr + 2 * R::W_BATCH + r * GPB * 64, lane);
#pragma unroll
      for (int gg = 0; gg < GPB; ++gg) {
        // accumulators start at -1024 * sum(x / c) of the group, so the mma result is sum(code * x) directly
        const float2 q0 = gs[gg * MP], q1 = ONE ? q0 : gs[gg * MP + 1];
        float acc[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          acc[r][0] = -q0.x; acc[r][1] = -q1.x;
          acc[r][2] = -q0.x; acc[r][3] = -q1.x;
        }
#pragma unroll
        for (int s8 = 0; s8 < 8 / GPB; ++s8) {
          const int st = gg * (8 / GPB) + s8;
          uint2 bf = make_uint2(0u, 0u);
          if (tok_ok) bf = *reinterpret_cast<const uint2*>(xrow + st * 16);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            uint32_t af[4];
            extract<BITS, GROUP>(cf[r], st, af);
            mma_f16_16816(acc[r], af, bf.x, bf.y);
          }
        }
        // y += scale * (acc - zero * sum(x))
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float2 s0 = __half22float2(*reinterpret_cast<const __half2*>(&cf[r].sz[gg][0]));
          const float2 s1 = __half22float2(*reinterpret_cast<const __half2*>(&cf[r].sz[gg][1]));
          y[r][0] = fmaf(s0.x, fmaf(-s0.y, q0.y, acc[r][0]), y[r][0]);
          y[r][2] = fmaf(s1.x, fmaf(-s1.y, q0.y, acc[r][2]), y[r][2]);
          if (!ONE) {
            y[r][1] = fmaf(s0.x, fmaf(-s0.y, q1.y, acc[r][1]), y[r][1]);
            y[r][3] = fmaf(s1.x, fmaf(-s1.y, q1.y, acc[r][3]), y[r][3]);
          }
        }
      }
      xrow += 128;
      gs += GPB * MP;
      cptr += R::BLK;
      cbar += 8;
      if (cbar == bars_u + NST * 8) { cbar = bars_u; cptr = ring; cph ^= 1u; }
      __syncwarp();                               // the stage is free again
      if (lane == 0 && pleft > 0) issue();
      __syncwarp();
    }
    if (failed) break;
    // fragment layout -> tile [tok][32 rows]; the first fragment of a warp has its own tile, the others use the second
    const bool head = max(seg0, lo) <= wlo;       // the segment's part in this CTA starts before or with this warp
    const bool alone = max(seg0, lo) >= wlo && min(seg1, hi) <= whi;              // ... and lies in this warp entirely
    float* tile = tile_of(warp, head && !alone ? 0 : 1);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int tok = 2 * t;
      if (tok < m) { tile[tok * 32 + r * 16 + g] = y[r][0]; tile[tok * 32 + r * 16 + g + 8] = y[r][2]; }
      if (!ONE && tok + 1 < m) { tile[(tok + 1) * 32 + r * 16 + g] = y[r][1]; tile[(tok + 1) * 32 + r * 16 + g + 8] = y[r][3]; }
    }
    __syncwarp();
    if (alone) {
      float v[MP];
#pragma unroll
      for (int tok = 0; tok < MP; ++tok) v[tok] = tok < m ? tile[tok * 32 + lane] : 0.f;
      __syncwarp();
      finish(pan, seg0 >= lo && seg1 <= hi, v);
    }
  }
  const bool any_failed = __syncthreads_or(failed ? 1 : 0) != 0;
  if (any_failed) {
    // copies still in flight get a bounded time to land before the CTA's shared memory is released
    const uint64_t t_end = globaltimer_ns() + 2000000ull;
    while (globaltimer_ns() < t_end) { }
    return;
  }
  // ---- segments that several warps share: segment j of the CTA is added up by warp j % 16 ----
  for (int pn = (int)(lo / (unsigned)len) + warp; (unsigned)pn * (unsigned)len < hi; pn += kW8) {
    const unsigned seg0 = (unsigned)pn * (unsigned)len, seg1 = seg0 + (unsigned)len;
    const unsigned a0 = max(seg0, lo), a1 = min(seg1, hi);
    const int wa = warp_of(a0), wz = warp_of(a1 - 1u);
    if (wa == wz) continue;
    float v[MP];
#pragma unroll
    for (int tok = 0; tok < MP; ++tok) v[tok] = 0.f;
    for (int w = wa; w <= wz; ++w) {
      if (warp_lo(w) == warp_lo(w + 1)) continue;                                 // a warp without units
      const float* tile = tile_of(w, a0 <= warp_lo(w) ? 0 : 1);
#pragma unroll
      for (int tok = 0; tok < MP; ++tok)
        if (tok < m) v[tok] += tile[tok * 32 + lane];
    }
    finish(pn, seg0 >= lo && seg1 <= hi, v);
  }
}

static Gemv8Plan g8_plan(int n, int k) {
  Gemv8Plan p = {};
  const long npan = n / 32, nbat = k / 128;
  p.slices = (int)((nbat + 39) / 40);
  long G = npan * nbat / kW8;                     // at least one unit per warp
  G = G > 148 ? 148 : G;
  p.per_slice = (int)(G / p.slices < 1 ? 1 : G / p.slices);
  p.panel_cut = p.slices == 1 && npan >= 8L * p.per_slice;
  p.xb = (int)((nbat + p.slices - 1) / p.slices);
  const long per = npan * (nbat / p.slices) / p.per_slice;      // units of a CTA, at least
  p.fmax = p.panel_cut ? 1 : (int)((p.xb + per - 1) / (per < 1 ? 1 : per) + 1);
  return p;
}

template <int BITS, int GROUP, bool ONE>
static int g8_launch(const WqGemvArgs& a, Gemv8Plan p, cudaStream_t st) {
  using R = Ring<BITS, GROUP, 2>;
  constexpr int GPB = 128 / GROUP, MP = ONE ? 1 : 8;
  // Rings of 6.5 KB a warp, 104 KB an SM: 4.4 KB and 8.7 KB measured 10 and 1 % slower.
  const size_t rest = 32 + (size_t)kW8 * 2 * a.m * 32 * 4 + (((size_t)p.xb * GPB * MP + 1) & ~(size_t)1) * 8 + (size_t)a.m * (p.xb * 128 + 16) * 2;
  auto total = [&](int nst) { return (size_t)kW8 * nst * (R::BLK + 8) + rest; };
  p.nst = 6656 / R::BLK;
  while (total(p.nst) > 220 * 1024 && p.nst > 2) --p.nst;
  const size_t smem = total(p.nst);
  if (smem > 220 * 1024) return B2_ERR_ARG;
  auto kern = wq_gemv8_kernel<BITS, GROUP, ONE>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) return B2_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.slices * p.per_slice), 1, 1);
  cfg.blockDim = dim3(kT8, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, a, p) == cudaSuccess ? B2_OK : B2_ERR_LAUNCH;
}

}  // namespace b2

using namespace b2;

// Scratch floats of b2_wq_gemv8 (per chunk of eight rows; chunks run one after the other).
B2_API long b2_wq_gemv8_scratch_floats(int n, int k, int m) {
  const Gemv8Plan p = g8_plan(n, k);
  if (p.panel_cut) return 0;
  return (long)p.slices * (n / 32) * p.fmax * (m < 8 ? m : 8) * 32;
}

// Whether b2_wq_gemv8 takes a matrix: unit numbers times CTAs fit 32 bits, and the hand-over has a lane for every slice
// (k up to 163840).  b2_wq_gemv has neither limit there.  A matter of (n, k) only.
B2_API int b2_wq_gemv8_takes(int n, int k) {
  return (double)(n / 32) * (double)(k / 128) * 148.0 < 4.0e9 && g8_plan(n, k).slices <= 32;
}

// The GEMV of *args (fields vworkers, fmax and tp are not read, ks and rb do not matter) for 1 .. 32 rows, eight at a time.  `counters`
// holds n / 32 self-resetting words, `scratch` b2_wq_gemv8_scratch_floats(n, k, m) floats.
B2_API int b2_wq_gemv8(const WqGemvArgs* args, cudaStream_t stream) {
  const WqGemvArgs& a = *args;
  if (a.n <= 0 || a.k <= 0 || a.m <= 0 || a.m > 32 || a.n % 32 || a.k % 128) return B2_ERR_ARG;
  if (a.group != 64 && a.group != 128) return B2_ERR_ARG;
  if (a.ks < 1 || a.ks > kMaxKs || a.k / 128 % a.ks || (a.rb != 2 && a.rb != 4)) return B2_ERR_ARG;   // a linear that the other kernel takes
  if (!a.scratch || !a.counters || a.epi == EPI_TP_RESID) return B2_ERR_ARG;
  if ((a.ldx % 8) || (reinterpret_cast<uintptr_t>(a.x) & 15)) return B2_ERR_ARG;
  if (!b2_wq_gemv8_takes(a.n, a.k)) return B2_ERR_ARG;
  const Gemv8Plan p = g8_plan(a.n, a.k);
  for (int t0 = 0; t0 < a.m; t0 += 8) {
    WqGemvArgs c = a;
    c.m = a.m - t0 < 8 ? a.m - t0 : 8;
    c.x = a.x + (long)t0 * a.ldx;
    if (a.ss_in) c.ss_in = a.ss_in + t0;
    if (a.y) c.y = a.y + (long)t0 * a.ldy;
    if (a.yf) c.yf = a.yf + (long)t0 * a.ldy;
    if (a.resid) c.resid = a.resid + (long)t0 * a.ldr;
    if (a.ss_out) c.ss_out = a.ss_out + t0;
    if (a.amax_val) { c.amax_val = a.amax_val + t0; c.amax_idx = a.amax_idx + t0; }
    int rc = B2_ERR_ARG;
    const bool one = c.m == 1;
    switch (a.bits * 1000 + a.group) {
      case 4128: rc = one ? g8_launch<4, 128, true>(c, p, stream) : g8_launch<4, 128, false>(c, p, stream); break;
      case 4064: rc = one ? g8_launch<4, 64, true>(c, p, stream) : g8_launch<4, 64, false>(c, p, stream); break;
      case 3128: rc = one ? g8_launch<3, 128, true>(c, p, stream) : g8_launch<3, 128, false>(c, p, stream); break;
      case 3064: rc = one ? g8_launch<3, 64, true>(c, p, stream) : g8_launch<3, 64, false>(c, p, stream); break;
      case 2128: rc = one ? g8_launch<2, 128, true>(c, p, stream) : g8_launch<2, 128, false>(c, p, stream); break;
      case 2064: rc = one ? g8_launch<2, 64, true>(c, p, stream) : g8_launch<2, 64, false>(c, p, stream); break;
    }
    if (rc != B2_OK) return rc;
  }
  return B2_OK;
}
