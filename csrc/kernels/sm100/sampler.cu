// Device-side sampling and speculative acceptance.
//
// One rule decides every sampled token (reference: kernels/m1/m1_model.cu:796-818): the token at absolute position n
// of a sequence with seed s is InvCDF_q(u(s, n)), where q is the filtered distribution (temperature, top-k, top-p,
// min-p) of that position's logits and u is the first uniform of Philox4x32-10 keyed by s at counter n.  Because the
// draw depends only on (seed, position, logits), a verify block samples every row exactly as a plain decode step would,
// so "a draft is accepted iff it equals the target's own sample" gives the plain sampling distribution and, with a
// seed, the same tokens with or without speculation and at any batch size.
//
// Implementation: a cluster of CTAs per row (eight, fewer where many rows fill the chip anyway), each with its share of
// the row in shared memory.  Keys are the
// order-preserving integer images of the logits; top-k, top-p and the final inverse-CDF walk are radix descents over
// 8-bit digits (4 passes each) with 256-bin histograms of counts or probability mass, summed over the cluster through
// distributed shared memory; ties are broken by ascending token index.  Every sum is over integers, so the result does
// not depend on how a row is cut.
// Replaces samp_pos / samp_hist / samp_fast and accept_greedy / accept_sampled / bv_accept (m1_model.cu:476-579,
// 1099-1452, 1536).
#include "common.cuh"

namespace b2 {

struct SampleArgs {
  const float* logits; long ld; int vocab;      // [rows][ld], first `vocab` columns are valid
  const float* temperature;                      // per row; <= 0 means greedy
  const int* top_k;                              // per row; <= 0 means off
  const float* top_p;                            // per row; >= 1 means off
  const float* min_p;                            // per row; <= 0 means off
  const unsigned long long* seed;                // per row
  const int* position;                           // per row: absolute position of the token being sampled
  int* out;                                      // [rows]
};

namespace {

constexpr int kThreads = 1024;

__device__ __forceinline__ uint32_t key_of(float x) {      // larger float -> larger key
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// Philox4x32-10, returns the first 32-bit output for (key = seed, counter = ctr).
__device__ uint32_t philox_first(unsigned long long seed, unsigned long long ctr) {
  uint32_t c0 = (uint32_t)ctr, c1 = (uint32_t)(ctr >> 32), c2 = 0, c3 = 0;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
  return c0;
}

// Probability masses are fixed point (exp of a non-positive number times 2^31, so one mass fits 32 bits): integer sums
// do not depend on the order of the additions, so every threshold of the sampler is exactly reproducible.  A histogram
// bin is a (low, high) pair of 32-bit words: 32-bit shared-memory integer atomics are single instructions, where float
// and 64-bit ones are compare-and-swap loops; the carry into the high word is a second, rare, atomic.
__device__ __forceinline__ unsigned long long mass_of(float xv, float mx, float inv_t) {
  return (unsigned long long)(__expf((xv - mx) * inv_t) * 2147483648.f);
}
struct Hist { uint32_t lo[256], hi[256]; };
__device__ __forceinline__ void hist_add(Hist& h, uint32_t dig, unsigned long long v) {
  const uint32_t lo = (uint32_t)v;
  uint32_t hi = (uint32_t)(v >> 32);
  if (lo) { const uint32_t old = atomicAdd(&h.lo[dig], lo); hi += (old + lo < old) ? 1u : 0u; }
  if (hi) atomicAdd(&h.hi[dig], hi);
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
constexpr int kMaxCl = 8;              // most CTAs per row
constexpr int kSmsS = 148;
constexpr int kListCap = 2048;         // survivors of the filters that a CTA keeps apart
constexpr int kCacheBytes = 160 * 1024;

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
template <int CL>
__device__ __forceinline__ void cluster_sync() {
  if (CL == 1) { __syncthreads(); return; }
  __syncwarp();                      // single lanes store just before; the barrier is .aligned
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t rank) {      // the same variable in CTA `rank`
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ uint32_t peer_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long peer_u64(uint32_t a) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}

// One CTA's share of a row and the shared memory of the cluster exchange.  Exchanged variables exist twice and are used
// in turn (`turn`): a CTA overwrites its copy only two exchanges later, after a cluster barrier that every reader of the
// old value has passed.
struct Share {
  const float* x;            // values lo .. lo + n - 1 of the row, in shared memory when they fit
  int lo, n;
  const float* lv; const int* li; int ln;       // survivors of the filters (values, row indices) once collected; ln < 0: none
  Hist* hist;                // [2]
  unsigned long long* xch;   // [2]
  unsigned long long* warp64;  // [kThreads / 32]
  int* pick;                 // [1]
  unsigned long long* pickv; // [2]
  int turn;
};

// f(value, row index, valid) for every element of the share, the same number of calls on every thread of the CTA (so f
// may use warp-wide primitives).
template <typename F>
__device__ __forceinline__ void scan_share(const Share& s, F f) {
  if (s.ln >= 0) {
    for (int base = 0; base < s.ln; base += kThreads) {
      const int i = base + (int)threadIdx.x;
      const bool v = i < s.ln;
      f(v ? s.lv[i] : 0.f, v ? s.li[i] : 0, v);
    }
    return;
  }
#pragma unroll 4
  for (int base = 0; base < s.n; base += kThreads) {
    const int i = base + (int)threadIdx.x;
    const bool v = i < s.n;
    f(v ? s.x[i] : 0.f, s.lo + i, v);
  }
}

enum ClOp { CL_SUM, CL_MAX, CL_MIN };
// Reduction of one 64-bit value per thread over the CTA and the cluster; every thread gets the result.
template <ClOp OP, int CL>
__device__ unsigned long long cluster_reduce(Share& s, unsigned long long v) {
  auto comb = [](unsigned long long a, unsigned long long b) -> unsigned long long {
    if (OP == CL_SUM) return a + b;
    if (OP == CL_MIN) return a < b ? a : b;
    return a > b ? a : b;
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = comb(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) s.warp64[threadIdx.x >> 5] = v;
  __syncthreads();
  const int t = s.turn;
  s.turn ^= 1;
  if (threadIdx.x < 32) {
    v = s.warp64[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = comb(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) s.xch[t] = v;
  }
  cluster_sync<CL>();
  v = peer_u64(peer_addr(&s.xch[t], 0));
#pragma unroll
  for (uint32_t r = 1; r < CL; ++r) v = comb(v, peer_u64(peer_addr(&s.xch[t], r)));
  return v;
}

// Radix descent: finds the largest key prefix such that the mass of all elements with a strictly larger key is
// <= target (mass = probability or count).  On return *above = mass strictly above the final key.
// `keep_min`: elements with key < keep_min are ignored.
template <bool COUNT, int CL>
__device__ uint32_t radix_descend(Share& s, float mx, float inv_t, uint32_t keep_min, unsigned long long target,
                                  unsigned long long* above_out) {
  uint32_t prefix = 0, mask = 0;
  unsigned long long above = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int shift = 24; shift >= 0; shift -= 8) {
    const int t = s.turn;
    s.turn ^= 1;
    Hist& hist = s.hist[t];
    if (threadIdx.x < 256) { hist.lo[threadIdx.x] = 0; hist.hi[threadIdx.x] = 0; }
    __syncthreads();
    // Logits crowd into a few digits at the upper levels, where one shared-memory atomic per element would serialise
    // the warp: lanes that share a digit with at least seven others are summed in registers first and their leader
    // adds once; the rest add for themselves.
    scan_share(s, [&](float xv, int, bool valid) {
      const uint32_t k = key_of(xv);
      const bool on = valid && k >= keep_min && (k & mask) == prefix;
      if (!__any_sync(0xffffffffu, on)) return;
      const uint32_t dig = on ? (k >> shift) & 255u : 0xFFFFFFFFu;
      const unsigned long long v = !on ? 0ull : (COUNT ? 1ull : mass_of(xv, mx, inv_t));
      const unsigned peers = __match_any_sync(0xffffffffu, dig);
      const bool big = on && __popc(peers) >= 8;
      unsigned pending = __ballot_sync(0xffffffffu, big);
      while (pending) {
        const int leader = __ffs(pending) - 1;
        const unsigned grp = __shfl_sync(0xffffffffu, peers, leader);
        const unsigned long long sum = COUNT ? (unsigned long long)__popc(grp) : warp_sum_u64(((grp >> lane) & 1u) ? v : 0ull);
        if (lane == leader) hist_add(hist, dig, sum);
        pending &= ~grp;
      }
      if (on && !big) hist_add(hist, dig, v);
    });
    cluster_sync<CL>();
    // the row's digit d, walked from high to low, is the first with above + mass(digits >= d) > target (0 if none):
    // thread i < 256 takes digit 255 - i, so the running masses are prefix sums over the threads
    unsigned long long h = 0, inc = 0;
    if (threadIdx.x < 256) {
      const int d = 255 - (int)threadIdx.x;
#pragma unroll
      for (uint32_t r = 0; r < CL; ++r) {
        const uint32_t lo = peer_u32(peer_addr(&hist.lo[d], r)), hi = peer_u32(peer_addr(&hist.hi[d], r));
        h += ((unsigned long long)hi << 32) | lo;
      }
      inc = h;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long p = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += p;
      }
      if (lane == 31) s.warp64[warp] = inc;
    }
    if (threadIdx.x == 0) *s.pick = 255;
    __syncthreads();
    if (threadIdx.x < 256) {
      inc += above;
      for (int w = 0; w < warp; ++w) inc += s.warp64[w];
      const bool past = inc > target;
      if (past && threadIdx.x < 255) atomicMin(s.pick, (int)threadIdx.x);
    }
    __syncthreads();
    const int pick = *s.pick;
    if ((int)threadIdx.x == pick) s.pickv[t] = inc - h;
    __syncthreads();
    above = s.pickv[t];
    prefix |= (uint32_t)(255 - pick) << shift;
    mask |= 255u << shift;
  }
  *above_out = above;
  return prefix;
}

// The maximum of a row and its lowest index; NaNs are passed over.
struct Best {
  float v = -INFINITY;
  int i = 0x7fffffff;
  __device__ __forceinline__ void see(float x, int at) {
    if (x > v || (x == v && at < i)) { v = x; i = at; }
  }
  // As one integer that grows with the value and falls with the index (-0 counts as +0).
  __device__ __forceinline__ unsigned long long packed() const { return ((unsigned long long)key_of(v + 0.f) << 32) | (0xffffffffu - (uint32_t)i); }
};
__device__ __forceinline__ float packed_value(unsigned long long p) {
  const uint32_t k = (uint32_t)(p >> 32);
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
__device__ __forceinline__ int packed_index(unsigned long long p) { return (int)(0xffffffffu - (uint32_t)p); }

// Elements x[0 .. n) of a row (index lo on) as this thread sees them, four at a time where the alignment allows it; kept
// in `cache` if that is given.
__device__ __forceinline__ void load_share(const float* x, int n, int lo, float* cache, Best& b) {
  int i0 = 0;
  if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    const int n4 = n >> 2;
#pragma unroll 4
    for (int i = threadIdx.x; i < n4; i += kThreads) {
      const float4 v = reinterpret_cast<const float4*>(x)[i];
      if (cache) reinterpret_cast<float4*>(cache)[i] = v;
      const int at = lo + 4 * i;
      b.see(v.x, at); b.see(v.y, at + 1); b.see(v.z, at + 2); b.see(v.w, at + 3);
    }
    i0 = 4 * n4;
  }
  for (int i = i0 + threadIdx.x; i < n; i += kThreads) {
    const float v = x[i];
    if (cache) cache[i] = v;
    b.see(v, lo + i);
  }
}

}  // namespace

// Determinism: counts and fixed-point masses are integers, so every histogram, threshold and the final walk are
// independent of the order in which threads add; equal keys are ordered by token index.
//
// What bounds it: about fifteen passes over the row.  With one CTA per row (the earlier kernel) a pass moved 600 KB of
// logits from L2 through a single SM and walked its 256 bins serially on every thread: 518 us for 16 rows of 151936
// logits.  Here a row is read from memory once, a pass costs 19 values per thread plus a cluster barrier, and passes
// after top-k or min-p touch the survivors only: 92 us.  A greedy row is the load and one exchange (1 row 6.9 -> 4.3 us).
// CACHED: the share is in shared memory (known at compile time, so that the passes use shared-memory loads).
template <int CL, bool CACHED>
__global__ void __launch_bounds__(kThreads) sample_rows_kernel(const SampleArgs a, int share, int solo) {
  extern __shared__ __align__(16) float cache[];
  __shared__ Hist hist[2];
  __shared__ unsigned long long xch[2], warp64[kThreads / 32], pickv[2];
  __shared__ float list_v[kListCap];
  __shared__ int list_i[kListCap];
  __shared__ int s_pick, s_list;
  pdl_wait();
  pdl_launch_dependents();
  const int row = blockIdx.x / CL;
  const int rank = CL == 1 ? 0 : (int)cluster_rank();
  Share s;
  s.lo = min(rank * share, a.vocab);
  s.n = min(share, a.vocab - s.lo);
  s.ln = -1; s.lv = list_v; s.li = list_i;
  s.hist = hist; s.xch = xch; s.warp64 = warp64; s.pick = &s_pick; s.pickv = pickv;
  s.turn = 0;
  const float* gx = a.logits + (size_t)row * a.ld + s.lo;
  if (CACHED) s.x = cache;
  else s.x = gx;
  const float T = a.temperature ? a.temperature[row] : 0.f;
  const int topk = a.top_k ? a.top_k[row] : 0;
  const bool greedy = T <= 0.f || topk == 1;
  Best best;
  if (solo && greedy) {              // the first CTA alone; the others make room
    if (rank == 0) {
      load_share(gx, a.vocab, 0, nullptr, best);
      const unsigned long long top = cluster_reduce<CL_MAX, 1>(s, best.packed());
      if (threadIdx.x == 0) a.out[row] = packed_index(top);
    }
    return;
  }
  load_share(gx, s.n, s.lo, CACHED ? cache : nullptr, best);
  const unsigned long long top = cluster_reduce<CL_MAX, CL>(s, best.packed());         // its barriers also publish `cache` to the CTA
  const float mx = packed_value(top);
  if (greedy) {
    if (rank == 0 && threadIdx.x == 0) a.out[row] = packed_index(top);
    cluster_sync<CL>();              // no CTA leaves while another still reads its shared memory
    return;
  }
  const float inv_t = 1.f / T;
  uint32_t keep_min = 0;          // smallest key that survives the filters
  // min-p: p >= min_p * p_max  <=>  x >= mx + T * ln(min_p)
  const float minp = a.min_p ? a.min_p[row] : 0.f;
  if (minp > 0.f) keep_min = max(keep_min, key_of(mx + T * __logf(minp)));
  // top-k: key of the k-th largest logit (ties at the threshold are all kept; the index rule orders them)
  if (topk > 1 && topk < a.vocab) {
    unsigned long long above;
    const uint32_t kth = radix_descend<true, CL>(s, mx, inv_t, 0u, (unsigned long long)(topk - 1), &above);
    keep_min = max(keep_min, kth);
  }
  if (keep_min > 0) {                // later passes read this CTA's survivors only, if there is room for them
    if (threadIdx.x == 0) s_list = 0;
    __syncthreads();
    scan_share(s, [&](float xv, int i, bool valid) {
      if (valid && key_of(xv) >= keep_min) {
        const int at = atomicAdd(&s_list, 1);
        if (at < kListCap) { list_v[at] = xv; list_i[at] = i; }
      }
    });
    __syncthreads();
    if (s_list <= kListCap) s.ln = s_list;
  }
  auto mass_left = [&]() {           // mass of what is left
    unsigned long long z = 0;
    scan_share(s, [&](float xv, int, bool valid) { if (valid && key_of(xv) >= keep_min) z += mass_of(xv, mx, inv_t); });
    return cluster_reduce<CL_SUM, CL>(s, z);
  };
  // top-p over what is left: smallest descending prefix whose mass reaches top_p * Z
  const float topp = a.top_p ? a.top_p[row] : 1.f;
  if (topp < 1.f) {
    const unsigned long long z = mass_left();
    unsigned long long above;
    const uint32_t cut = radix_descend<false, CL>(s, mx, inv_t, keep_min, (unsigned long long)((double)topp * (double)z), &above);
    keep_min = max(keep_min, cut);
  }
  // draw
  const unsigned long long z = mass_left();                  // at least 2^31: the maximum always survives the filters
  const uint32_t r = philox_first(a.seed ? a.seed[row] : 0ull, (unsigned long long)(a.position ? a.position[row] : 0));
  const double u = ((double)(r >> 8) + 0.5) * (1.0 / 16777216.0);
  unsigned long long target = (unsigned long long)(u * (double)z);
  if (z > 0 && target >= z) target = z - 1;
  unsigned long long above;
  const uint32_t key = radix_descend<false, CL>(s, mx, inv_t, keep_min, target, &above);
  // among the tokens that share the final key, walk by ascending index: the `want`-th of them wins
  const unsigned long long w = mass_of(__uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key), mx, inv_t);
  const unsigned long long rank64 = w > 0 && target > above ? (target - above) / w : 0ull;
  const int nth = (int)(rank64 > 1000000000ull ? 1000000000ull : rank64);
  unsigned long long same = 0;
  scan_share(s, [&](float xv, int, bool valid) { same += valid && key_of(xv) == key ? 1u : 0u; });
  const int cnt = (int)cluster_reduce<CL_SUM, CL>(s, same);
  if (cnt == 0) {                                            // rounding pushed the walk past the last bin: take the mode
    if (rank == 0 && threadIdx.x == 0) a.out[row] = packed_index(top);
  } else if (cnt == 1) {                                     // the usual case: one token owns the key
    scan_share(s, [&](float xv, int i, bool valid) { if (valid && key_of(xv) == key) a.out[row] = i; });
  } else {
    // smallest index I with (number of equal-key tokens at index <= I) == want + 1, by bisection over the index range
    const int want = min(nth, cnt - 1);
    int lo = 0, hi = a.vocab - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      unsigned long long c = 0;
      scan_share(s, [&](float xv, int i, bool valid) { c += valid && i <= mid && key_of(xv) == key ? 1u : 0u; });
      c = cluster_reduce<CL_SUM, CL>(s, c);
      if ((int)c >= want + 1) hi = mid; else lo = mid + 1;
    }
    if (rank == 0 && threadIdx.x == 0) a.out[row] = lo;
  }
  cluster_sync<CL>();                // no CTA leaves while another still reads its shared memory
}

// Longest-prefix acceptance for one or more verify blocks.  Block b covers rows [row0[b], row0[b] + cnt[b]): row 0 is
// the bonus token, rows 1.. are drafts.  target[r] is the model's own token (argmax or sample) after row r.
// Draft j + 1 is accepted iff it equals target[j].  Emits the accepted drafts followed by the target's next token.
__global__ void spec_accept_kernel(const int* __restrict__ ids, const int* __restrict__ target, const int* __restrict__ row0,
                                   const int* __restrict__ cnt, int n_blocks, int* __restrict__ n_emitted,
                                   int* __restrict__ emitted, int emitted_ld) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_blocks) return;
  const int r0 = row0[b], c = cnt[b];
  int acc = 0;
  while (acc + 1 < c && ids[r0 + acc + 1] == target[r0 + acc]) ++acc;
  for (int j = 0; j < acc; ++j) emitted[(size_t)b * emitted_ld + j] = ids[r0 + j + 1];
  emitted[(size_t)b * emitted_ld + acc] = target[r0 + acc];
  n_emitted[b] = acc + 1;
}

}  // namespace b2

using namespace b2;

template <int CL, bool CACHED>
static int sample_launch(const SampleArgs& a, int rows, int share, int solo, cudaStream_t st) {
  auto kern = sample_rows_kernel<CL, CACHED>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kCacheBytes) != cudaSuccess) return B2_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)rows * CL); cfg.blockDim = dim3(kThreads); cfg.stream = st;
  cfg.dynamicSmemBytes = CACHED ? (size_t)share * 4 : 0;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = CL; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = CL == 1 ? 1 : 2;
  return cudaLaunchKernelEx(&cfg, kern, a, share, solo) == cudaSuccess ? B2_OK : B2_ERR_LAUNCH;
}

B2_API int b2_sample_rows(const SampleArgs* a, int rows, cudaStream_t st) {
  if (!a || rows <= 0 || a->vocab <= 0 || !a->logits || !a->out) return B2_ERR_ARG;
  // CTAs per row: eight, or fewer where a share would have fewer values than threads (1000 logits, greedy: 4.4 -> 2.7 us),
  // or where eight would not all be resident at once (two per SM, by their shared memory) and fewer still are.  Where they
  // come in waves all the same, a greedy row, which is one short pass, is left to one CTA.  128 rows, always eight -> by
  // this rule: greedy 151936 logits 44 -> 21 us (one CTA per row 13), 32000 28 -> 6 (5); top-p 32000 193 -> 96 (164).
  auto share_of = [&](int c) { return ((a->vocab + c - 1) / c + 3) & ~3; };   // multiple of four: shares keep the row's alignment
  auto two = [&](int c) { return (long)share_of(c) * 4 <= 88 * 1024; };
  auto waves = [&](int c) { return (long)rows * c > (two(c) ? 2L : 1L) * kSmsS; };
  int cl = kMaxCl;
  while (cl > 1 && (share_of(cl) < kThreads || (waves(cl) && two(cl / 2)))) cl /= 2;
  const int solo = waves(cl);
  const int share = share_of(cl);
  if (cl == 4) return sample_launch<4, true>(*a, rows, share, solo, st);
  if (cl == 2) return sample_launch<2, true>(*a, rows, share, solo, st);
  if (cl == 1) return sample_launch<1, true>(*a, rows, share, solo, st);
  return (long)share * 4 <= kCacheBytes ? sample_launch<8, true>(*a, rows, share, solo, st) : sample_launch<8, false>(*a, rows, share, solo, st);
}

B2_API int b2_spec_accept(const int* ids, const int* target, const int* row0, const int* cnt, int n_blocks, int* n_emitted,
                          int* emitted, int emitted_ld, cudaStream_t st) {
  if (n_blocks <= 0 || emitted_ld < 1) return B2_ERR_ARG;
  spec_accept_kernel<<<(n_blocks + 63) / 64, 64, 0, st>>>(ids, target, row0, cnt, n_blocks, n_emitted, emitted, emitted_ld);
  return cudaGetLastError() == cudaSuccess ? B2_OK : B2_ERR_LAUNCH;
}
