// kernels_pcg.cu -- resident PCG: a whole solve in one cooperative launch of one block per SM whose rows'
// vectors stay in shared memory from the set-up to the end.
//
// Each block owns a contiguous range of 32-row slices.  An SpMV is cut into units of one slice's every T-th
// entry (T warps share a slice, so a small system still fills the SM's warps and a large one divides evenly
// over them); the units' partial products meet in shared memory, where one thread per row adds them in order
// and makes the row's recurrences.  Only the vector that other rows gather (m, or p) is in global memory.
//
// The grid's reductions (exchange) have one counter: every block stores its sums, arrives with one acquire-release
// atomic, polls the counter and then adds all blocks' sums itself, in the same order, so the totals and the scalars
// made from them are the same bits everywhere and no block waits for another to combine or to announce them: one
// trip through L2 where counted groups, their sums and a release word take three.
//
// Measured on a GB300 (us per iteration of a whole solve on the FP16 copy, against the earlier kernel of 256-row
// virtual blocks with all vectors in global memory and counted group barriers): 1.02M-tet beam 11.4 (21.3), 192k-tet
// bar 5.0 (12.6), 64-cube batch of 1.9M tets 35 (53).  Cycles of a beam iteration: SpMV 10,000, exchange 5,000, row
// recurrences 4,600.  Taking units and recurrences from one queue, so that neither waits for the other's last warp, was
// slower on the beam (756 against 662 us a solve): the recurrences' chains of shared-memory loads stretch behind the
// gathers.

#include <cuda_fp16.h>

#include <algorithm>

#include "pcg_common.cuh"

namespace ssim_gb {
namespace {

constexpr int kMaxBlocks = 192;  // blocks of a resident launch (one per SM), a multiple of 32

struct GridExchange {
  unsigned long long* count;  // arrivals since the launch (zeroed before it)
  double* words;              // [2][4][kMaxBlocks] the blocks' sums of each value, double-buffered
  unsigned int extra;         // arrivals waited for beyond the grid (test hook: every wait runs out)
  long long spin_limit;
};

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void arrive_acq_rel(unsigned long long* p) {
  unsigned long long old;
  asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(old) : "l"(p) : "memory");
}

// shared memory of the exchanges
struct ExchangeShared {
  double own[4];  // this block's sums
  double tot[4];  // totals over the blocks
  int fail;
};

__device__ __forceinline__ double warp_add(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// An exchange has two parts; every thread of the block calls each.  GB300's FP64 unit takes a warp's addition every
// 64 cycles and adds no faster with more of them in flight, so each value's sums run in a warp of their own (there
// are four units an SM).
//
// exchange_wait number k (0, 1, ... in a launch), after a block-wide barrier that follows the block's partials
// sh[v * stride + i], i < np: warps 0 .. NV - 1 sum one value each (in FP64, lane-strided, then a shuffle tree), warp
// 0 stores the sums, arrives and polls.  The closing block-wide barrier releases the others: they see the global
// writes that any block made before the exchange.  false in every thread of a block whose wait ran out.  NV = 0: the
// barrier alone.  (Measured on 152 blocks of 1024 threads with a global write each before it: 3,115 cycles for the
// arrival and the wait, 1,906 of them the release's fence; polling 152 blocks' words {value, flag} instead, in one
// place or in a mailbox per block, 6,700 to 7,700: strong loads of many addresses are slow.)
template <typename S, int NV>
__device__ __forceinline__ bool exchange_wait(const GridExchange& gx, unsigned long long k, const S* sh, int stride,
                                              int np, ExchangeShared& xs) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if constexpr (NV > 0) {
    if (warp < NV) {
      double v = 0.0;
      for (int i = lane; i < np; i += 32) v += (double)sh[warp * stride + i];
      v = warp_add(v);
      if (lane == 0) xs.own[warp] = v;
      bar_sync(1, 32 * NV);
    }
  }
  if (warp == 0) {
    if (lane < NV) gx.words[((k & 1) * 4 + lane) * kMaxBlocks + blockIdx.x] = xs.own[lane];
    __syncwarp();
    if (lane == 0) {
      const unsigned long long target = (k + 1) * (unsigned long long)(gridDim.x + gx.extra);
      arrive_acq_rel(gx.count);
      long long n = 0;
      while (ld_acquire(gx.count) < target) {
        if (++n > gx.spin_limit) {
          xs.fail = 1;
          break;
        }
      }
    }
  }
  __syncthreads();
  return xs.fail == 0;
}
// exchange_total: warps 0 .. NV - 1 add one value's words of all blocks and warp 0's lane 0 hands the totals to epi; a
// block-wide barrier has to follow before another thread reads what epi wrote.  The other warps pass straight
// through.  Words of exchange k are overwritten by exchange k + 2, which no block reaches before every block arrived
// at k + 1, after its reads of k.
template <int NV, typename EPI>
__device__ __forceinline__ void exchange_total(const GridExchange& gx, unsigned long long k, ExchangeShared& xs,
                                               EPI&& epi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp >= NV) return;
  const double* w = gx.words + ((k & 1) * 4 + warp) * kMaxBlocks;
  double v[kMaxBlocks / 32];
#pragma unroll
  for (int j = 0; j < kMaxBlocks / 32; ++j) v[j] = lane + 32 * j < (int)gridDim.x ? __ldcg(w + lane + 32 * j) : 0.0;
  double t = v[0];
#pragma unroll
  for (int j = 1; j < kMaxBlocks / 32; ++j)
    if (32 * j < (int)gridDim.x) t += v[j];
  t = warp_add(t);
  if (lane == 0) xs.tot[warp] = t;
  if constexpr (NV > 1) bar_sync(2, 32 * NV);
  if (threadIdx.x == 0) {
    double tot[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) tot[c] = xs.tot[c];
    epi(tot);
  }
}
// the whole exchange, partials to totals
template <typename S, int NV, typename EPI>
__device__ __forceinline__ bool exchange(const GridExchange& gx, unsigned long long k, const S* sh, int stride, int np,
                                         ExchangeShared& xs, EPI&& epi) {
  __syncthreads();
  if (!exchange_wait<S, NV>(gx, k, sh, stride, np, xs)) return false;
  exchange_total<NV>(gx, k, xs, epi);
  __syncthreads();
  return true;
}
__device__ __forceinline__ bool exchange_barrier(const GridExchange& gx, unsigned long long k, ExchangeShared& xs) {
  __syncthreads();
  return exchange_wait<float, 0>(gx, k, nullptr, 0, 0, xs);
}

// The scalars of a solve, one copy per block (the same bits in each): Chronopoulos-Gear's
//   beta = g / g_old,  den = d - beta g / alpha_old,  alpha = g / den   (first: 0, d, g / d)
// from g = (r, u), d = (w, u), with the reciprocals of the last step kept: ig = 1 / g_old, ia = 1 / alpha_old.  The
// correction is (g ig)(g ia): both factors have the size of a ratio or of d, where g g ig ia would leave the range of FP64
// for residuals beyond 1e77 or below 1e-81.
struct Scalars {
  double ig, ia, g, den, rr, rr0, tol2, alpha, beta;
  int iters, done, status;
};

__device__ __forceinline__ bool positive(double x) {  // x > 0, by its bits (a comparison costs the FP64 unit 64 cycles)
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ bool is_finite(double x) {
  return ((__double_as_longlong(x) >> 52) & 0x7ff) != 0x7ff;
}

// one thread, after the dots: stop tests on the residual of the current x (first: relative to this one), then the step
// lengths.  rr and tol2 are not negative, so they compare as integers.  FP32STEP: alpha and beta are used in FP32, so a
// reciprocal to 2^-45 (FP32's, improved by one Newton step) is enough for alpha.  This chain is what a small system's
// iteration waits for: about 700 cycles against 2,000 with comparisons, two divisions and the next step's reciprocals.
template <bool FP32STEP>
__device__ __forceinline__ void step_scalars(Scalars& s, bool first, double g, double d, double rr, double rtol,
                                             int max_iters) {
  if (first) {
    s.rr0 = rr;
    s.tol2 = rtol * rtol * rr;
    s.iters = s.done = s.status = 0;
    s.alpha = s.beta = 0.0;
  }
  s.rr = rr;
  if (!is_finite(rr)) {
    s.done = 1;
    s.status = 2;
    return;
  }
  if (__double_as_longlong(rr) <= __double_as_longlong(s.tol2) || is_zero(g) || s.iters >= max_iters) {
    s.done = 1;
    return;
  }
  double den = d, beta = 0.0;
  if (s.iters > 0) {
    beta = g * s.ig;
    den = fma(-beta, g * s.ia, d);
  }
  if (!positive(den)) {  // breakdown: not SPD along p (or non-finite)
    s.done = 1;
    s.status = 1;
    return;
  }
  if constexpr (FP32STEP) {
    const float df = (float)den;
    if (df > 1e-30f && df < 1e30f) {
      const double r = (double)(1.f / df);
      s.alpha = g * fma(r, fma(-den, r, 1.0), r);
    } else {
      s.alpha = g / den;
    }
  } else {
    s.alpha = g / den;
  }
  s.beta = beta;
  s.g = g;
  s.den = den;
  s.iters += 1;
}
// one thread, any time before the next step_scalars: the reciprocals it will use
__device__ __forceinline__ void next_reciprocals(Scalars& s) {
  s.ig = 1.0 / s.g;
  s.ia = s.den * s.ig;
}
// the solve's scalars for the host
__device__ __forceinline__ void publish_scalars(const Scalars& s, DevScalars* o) {
  o->rr = s.rr;
  o->rr0 = s.rr0;
  o->tol2 = s.tol2;
  o->alpha = s.alpha;
  o->beta = s.beta;
  o->iters = s.iters;
  o->done = s.done;
  o->status = s.status;
}

// One unit of y = A x on the symmetric store: slice s's upper slots part, part + T, ... and lower slots
// T - 1 - part, ... (the two run against each other, so the parts get equal shares), two slots in flight.
template <typename S>
__device__ __forceinline__ void sym_unit(const SellMatrix& A, const S* __restrict__ vals, int s, int lane, int part,
                                         int T, const V4<S>* x, S& a0, S& a1, S& a2) {
  const int ub = A.sl_off[s], Wu = (A.sl_off[s + 1] - ub) >> 5;
  const int lb = A.lo_off[s], Wl = (A.lo_off[s + 1] - lb) >> 5;
  a0 = a1 = a2 = S(0);
  for (int k = part; k < Wu; k += 2 * T) {
    const bool two = k + T < Wu;
    const int q0 = ub + 32 * k + lane, q1 = two ? q0 + 32 * T : q0;
    const int c0 = A.sl_col[q0], c1 = A.sl_col[q1];
    const S *p0 = vals + sell_base(q0), *p1 = vals + sell_base(q1);
    S v[9], w[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) v[m] = p0[32 * m];
#pragma unroll
    for (int m = 0; m < 9; ++m) w[m] = two ? p1[32 * m] : S(0);
    const V4<S> x0 = x[c0], x1 = x[c1];
    a0 += v[0] * x0.x + v[1] * x0.y + v[2] * x0.z;
    a1 += v[3] * x0.x + v[4] * x0.y + v[5] * x0.z;
    a2 += v[6] * x0.x + v[7] * x0.y + v[8] * x0.z;
    if (two) {
      a0 += w[0] * x1.x + w[1] * x1.y + w[2] * x1.z;
      a1 += w[3] * x1.x + w[4] * x1.y + w[5] * x1.z;
      a2 += w[6] * x1.x + w[7] * x1.y + w[8] * x1.z;
    }
  }
  for (int k = T - 1 - part; k < Wl; k += 2 * T) {
    const bool two = k + T < Wl;
    const int i0 = lb + 32 * k + lane, i1 = two ? i0 + 32 * T : i0;
    const int c0 = A.lo_col[i0], c1 = A.lo_col[i1];
    const S *p0 = vals + sell_base(A.lo_src[i0]), *p1 = vals + sell_base(A.lo_src[i1]);
    S v[9], w[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) v[m] = p0[32 * m];
#pragma unroll
    for (int m = 0; m < 9; ++m) w[m] = two ? p1[32 * m] : S(0);
    const V4<S> x0 = x[c0], x1 = x[c1];
    a0 += v[0] * x0.x + v[3] * x0.y + v[6] * x0.z;
    a1 += v[1] * x0.x + v[4] * x0.y + v[7] * x0.z;
    a2 += v[2] * x0.x + v[5] * x0.y + v[8] * x0.z;
    if (two) {
      a0 += w[0] * x1.x + w[3] * x1.y + w[6] * x1.z;
      a1 += w[1] * x1.x + w[4] * x1.y + w[7] * x1.z;
      a2 += w[2] * x1.x + w[5] * x1.y + w[8] * x1.z;
    }
  }
}

// ------------------------------------------------------------------ FP16 copy, pipelined
// How a resident solve is laid out (resident_plan): the grid, T, how many of a block's slices keep their
// vectors in shared memory, how many slices one pass covers, and whether the block's matrix entries fit too.
struct HalfPlan {
  int grid, T, spc, res, tile, cached;  // spc: most slices of a block; res, tile in slices
  int cache_entries;                    // most entries of a block (when cached)
  int packed;                           // 16-bit columns (HalfMatrix vs = 2)
  int keep;                             // slices whose entries L2 is asked to keep; -1: no hints
  size_t smem;
};

constexpr int HT = 1024;        // threads of a block
constexpr int kHalfState = 27;  // FP32 values of a row kept on chip: x r p s z w (18), 1/scale (3), M (6)

__device__ __forceinline__ float2 unpack_h2(unsigned int w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }

__device__ __forceinline__ void half_fma(const uint4& p, uint16_t h8, const float4& xv, float& a0, float& a1, float& a2) {
  const float2 f01 = unpack_h2(p.x), f23 = unpack_h2(p.y), f45 = unpack_h2(p.z), f67 = unpack_h2(p.w);
  const float f8 = __half2float(__ushort_as_half(h8));
  a0 = fmaf(f23.x, xv.z, fmaf(f01.y, xv.y, fmaf(f01.x, xv.x, a0)));
  a1 = fmaf(f45.y, xv.z, fmaf(f45.x, xv.y, fmaf(f23.y, xv.x, a1)));
  a2 = fmaf(f8, xv.z, fmaf(f67.y, xv.y, fmaf(f67.x, xv.x, a2)));
}

// loads with an L2 replacement priority (HINT), or plain ones
template <bool HINT>
__device__ __forceinline__ uint4 ld_hint(const uint4* p, unsigned long long pol) {
  if constexpr (HINT) {
    uint4 v;
    asm("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p), "l"(pol));
    return v;
  } else {
    return *p;
  }
}
template <bool HINT>
__device__ __forceinline__ uint16_t ld_hint(const uint16_t* p, unsigned long long pol) {
  if constexpr (HINT) {
    uint16_t v;
    asm("ld.global.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
    return v;
  } else {
    return *p;
  }
}
template <bool HINT>
__device__ __forceinline__ int ld_hint(const int* p, unsigned long long pol) {
  if constexpr (HINT) {
    int v;
    asm("ld.global.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
  } else {
    return *p;
  }
}

// Entries k0, k0 + T, ... of a slice of width W (col / v8 / v1: its first entry, this lane): four at a time with all
// their loads in flight.  The kernel is bound by the instructions it issues (59% of the issue slots in a first
// version with run-time strides and a predicate per entry), so T is a compile-time stride (immediate offsets) and
// only a unit's ragged end tests the width.  PACKED: the ninth value and the column's distance from the slice's first row
// share a word, 20 bytes and two loads an entry instead of 22 and three (32-bit columns are kept for patterns that reach
// further than 2^15 rows).  Whole solves: 1.02M-tet beam 662 -> 652 us, 192k-tet bar 283 -> 279, 64-cube batch 1,734 ->
// 1,648, where the entries come from DRAM.
template <int T, bool HINT, bool PACKED>
__device__ __forceinline__ void half_unit(const int* col, const uint4* v8, const uint16_t* v1, int W, int k0, int row0,
                                          const float4* x, unsigned long long pol, float& a0, float& a1, float& a2) {
  const int* words = PACKED ? reinterpret_cast<const int*>(v1) + 32 * k0 : nullptr;
  v8 += 32 * k0;
  if constexpr (!PACKED) {
    col += 32 * k0;
    v1 += 32 * k0;
  }
  // column and ninth value of the entry at o
  auto load_ch = [&](int o, int& c, uint16_t& h) {
    if constexpr (PACKED) {
      const int w = ld_hint<HINT>(words + o, pol);
      c = row0 + (w >> 16);
      h = (uint16_t)w;
    } else {
      c = ld_hint<HINT>(col + o, pol);
      h = ld_hint<HINT>(v1 + o, pol);
    }
  };
  int n = W - k0;  // entries 0, T, ... < n remain
  for (; n > 3 * T; n -= 4 * T) {
    int c[4];
    uint4 p[4];
    uint16_t h[4];
    float4 xv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) load_ch(32 * T * j, c[j], h[j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = ld_hint<HINT>(v8 + 32 * T * j, pol);
#pragma unroll
    for (int j = 0; j < 4; ++j) xv[j] = x[c[j]];
#pragma unroll
    for (int j = 0; j < 4; ++j) half_fma(p[j], h[j], xv[j], a0, a1, a2);
    v8 += 128 * T;
    if constexpr (PACKED) {
      words += 128 * T;
    } else {
      col += 128 * T;
      v1 += 128 * T;
    }
  }
  if (n > 0) {  // one to three entries: the missing ones repeat the first with a zero vector
    const int o1 = n > T ? 32 * T : 0, o2 = n > 2 * T ? 64 * T : 0;
    int c0, c1, c2;
    uint16_t h0, h1, h2;
    load_ch(0, c0, h0);
    load_ch(o1, c1, h1);
    load_ch(o2, c2, h2);
    const uint4 p0 = ld_hint<HINT>(v8, pol), p1 = ld_hint<HINT>(v8 + o1, pol), p2 = ld_hint<HINT>(v8 + o2, pol);
    const float4 x0 = x[c0];
    float4 x1 = x[c1], x2 = x[c2];
    if (n <= T) x1 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n <= 2 * T) x2 = make_float4(0.f, 0.f, 0.f, 0.f);
    half_fma(p0, h0, x0, a0, a1, a2);
    half_fma(p1, h1, x1, a0, a1, a2);
    half_fma(p2, h2, x2, a0, a1, a2);
  }
}

// Pipelined PCG on the FP16 copy (Ghysels & Vanroose, Parallel Computing 40(7), 2014), in the copy's scaled
// space, as one launch: the set-up (x = 0, r~ = S (sign b), u0 = M r~), the iterations, x unscaled and, when
// a.check is set, the solve's check on the FP32 symmetric store: g . x, |x|^2, |sign b - K x|^2 and |b|^2.
// With u = M r, w = A u, m = M w, s = A p, z = A M s (M per vertex, so u and M s are formed where needed):
//   prologue:  w = A u0, m_0 = M w;       partials (r, u), (w, u), (r, r)                -> exchange
//   phase k:   n = A m_k;  z = n + beta z,  s = w + beta s,  p = M r + beta p;
//              x += alpha p,  r -= alpha s,  w -= alpha z;  m_{k+1} = M w;  partials    -> exchange
// One exchange per iteration both sums the dots and orders m's writes.  The scalars (step_scalars) and the stop
// rule are Chronopoulos-Gear's; the third dot is (r, r) of the unscaled residual.  In FP32 the recursive residual
// drifts from the true one with the iterations and the condition number, so after pipe_iters iterations the
// solve continues as Chronopoulos-Gear PCG from the same state (w = A u recomputed, two exchanges a round).
// CACHED: the block's matrix entries are in shared memory too.  HINT: they are loaded with L2 priorities (pl.keep).
template <bool CACHED, int T, bool HINT, bool PACKED>
__global__ void __launch_bounds__(HT, 1)
    resident_half_kernel(HalfMatrix H, const float4* __restrict__ dinv, float4* x, float4* r, float4* z, float4* p,
                         float4* sv, float4* w, float4* m, HalfSolveArgs a, HalfPlan pl, Reduce red, GridExchange gx) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ ExchangeShared xs;
  __shared__ Scalars sc;
  __shared__ float s_ab[2];  // alpha, beta
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nv = H.nv, nsl = (nv + 31) >> 5;
  constexpr int lt = T == 8 ? 3 : 2;
  static_assert(T == 1 << lt, "T is 4 or 8");
  constexpr int VS = PACKED ? 2 : 1;
  const int s0 = (int)((long long)blockIdx.x * nsl / gridDim.x), ns = (int)((long long)(blockIdx.x + 1) * nsl / gridDim.x) - s0;
  const int RS = 32 * pl.res, PR = 32 * pl.tile;
  // shared memory: cached matrix entries (16-byte values first), row state, unit partials, per-slice dots, offsets
  uint4* c8 = reinterpret_cast<uint4*>(smem);
  float* st = reinterpret_cast<float*>(smem + (size_t)16 * pl.cache_entries);
  float* pb = st + (size_t)kHalfState * RS;
  float* shw = pb + (size_t)3 * T * PR;
  int* off = reinterpret_cast<int*>(shw + 4 * pl.spc);
  // the cached entries' columns and ninth values: one word (PACKED), or 4-byte columns and then 2-byte values
  int* ccol = off + pl.spc + 1;
  uint16_t* c1 = reinterpret_cast<uint16_t*>(PACKED ? ccol : ccol + pl.cache_entries);
  if (tid == 0) xs.fail = 0;
  for (int i = tid; i <= ns; i += HT) off[i] = H.off[s0 + i];
  __syncthreads();
  const int e0 = off[0];
  if constexpr (CACHED) {
    const int ne = off[ns] - e0;
    for (int i = tid; i < ne; i += HT) {
      c8[i] = H.v8[e0 + i];
      if constexpr (PACKED) {
        ccol[i] = reinterpret_cast<const int*>(H.v1)[e0 + i];
      } else {
        ccol[i] = H.col[e0 + i];
        c1[i] = H.v1[e0 + i];
      }
    }
  }
  unsigned long long nx = 0;  // exchanges so far
  unsigned long long pol_keep = 0, pol_pass = 0;
  if constexpr (HINT) {
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_keep));
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_pass));
  }

  // products of the slices t0 .. t1 - 1 into the unit partials
  auto spmv = [&](const float4* v, int t0, int t1) {
    const int nu = (t1 - t0) << lt;
    // warps count down: the low ones, which form the scalars meanwhile, get the round that is not full
    for (int i = HT / 32 - 1 - warp; i < nu; i += HT / 32) {
      const int b = off[t0 + (i >> lt)], W = (off[t0 + (i >> lt) + 1] - b) >> 5;
      float a0 = 0.f, a1 = 0.f, a2 = 0.f;
      if constexpr (CACHED)
        half_unit<T, false, PACKED>(ccol + (b - e0) + lane, c8 + (b - e0) + lane, c1 + VS * (b - e0 + lane), W, i & (T - 1),
                                    32 * (s0 + t0 + (i >> lt)), v, 0, a0, a1, a2);
      else
        half_unit<T, HINT, PACKED>(H.col + b + lane, H.v8 + b + lane, H.v1 + (size_t)VS * (b + lane), W, i & (T - 1),
                                   32 * (s0 + t0 + (i >> lt)), v, t0 + (i >> lt) < pl.keep ? pol_keep : pol_pass, a0, a1,
                                   a2);
      float* o = pb + (size_t)3 * (i & (T - 1)) * PR + 32 * (i >> lt) + lane;
      o[0] = a0;
      o[PR] = a1;
      o[2 * PR] = a2;
    }
  };
  auto product = [&](int l, int t0, float& n0, float& n1, float& n2) {  // the row's product from its T partials
    const float* o = pb + (l - 32 * t0);
    n0 = o[0];
    n1 = o[PR];
    n2 = o[2 * PR];
#pragma unroll
    for (int q = 1; q < T; ++q) {
      o += 3 * (size_t)PR;
      n0 += o[0];
      n1 += o[PR];
      n2 += o[2 * PR];
    }
  };
  // component f of row l's state: shared memory for the first RS rows, the vectors in global memory beyond
  auto ld3 = [&](int f, const float4* g, int l, int u, float (&v)[3]) {
    if (l < RS) {
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = st[(size_t)(f + c) * RS + l];
    } else {
      const float4 t = g[u];
      v[0] = t.x;
      v[1] = t.y;
      v[2] = t.z;
    }
  };
  auto st3 = [&](int f, float4* g, int l, int u, const float (&v)[3]) {
    if (l < RS) {
#pragma unroll
      for (int c = 0; c < 3; ++c) st[(size_t)(f + c) * RS + l] = v[c];
    } else {
      g[u] = make_float4(v[0], v[1], v[2], 0.f);
    }
  };
  constexpr int FX = 0, FR = 3, FP = 6, FS = 9, FZ = 12, FW = 15, FI = 18, FM = 21;
  auto ldm = [&](int l, int u, float (&d)[6]) {
    if (l < RS) {
#pragma unroll
      for (int c = 0; c < 6; ++c) d[c] = st[(size_t)(FM + c) * RS + l];
    } else {
      const float4 d0 = dinv[3 * (size_t)u], d1 = dinv[3 * (size_t)u + 1], d2 = dinv[3 * (size_t)u + 2];
      d[0] = d0.x;
      d[1] = d0.y;
      d[2] = d0.z;
      d[3] = d1.y;
      d[4] = d1.z;
      d[5] = d2.z;
    }
  };
  auto mul = [](const float (&d)[6], const float (&v)[3], float (&o)[3]) {  // the symmetric 3x3 block-Jacobi rows
    o[0] = d[0] * v[0] + d[1] * v[1] + d[2] * v[2];
    o[1] = d[1] * v[0] + d[3] * v[1] + d[4] * v[2];
    o[2] = d[2] * v[0] + d[4] * v[1] + d[5] * v[2];
  };
  // the three dots of a 32-row slice, summed in FP32 within the warp: the first two levels split the values over
  // the lanes (6 shuffles instead of 15)
  auto dots = [&](int l, float d0, float d1, float d2) {
    const bool hi = lane & 16, odd = lane & 8;
    float u = hi ? d2 : d0, v = hi ? 0.f : d1;
    u += __shfl_xor_sync(0xffffffffu, hi ? d0 : d2, 16);
    v += __shfl_xor_sync(0xffffffffu, hi ? d1 : 0.f, 16);
    float t = odd ? v : u;
    t += __shfl_xor_sync(0xffffffffu, odd ? u : v, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((lane & 7) == 0 && lane < 24) shw[(lane >> 3) * pl.spc + (l >> 5)] = t;
  };
  auto unscaled2 = [](const float (&rv)[3], const float (&is)[3]) {
    const float t0 = rv[0] * is[0], t1 = rv[1] * is[1], t2 = rv[2] * is[2];
    return t0 * t0 + t1 * t1 + t2 * t2;
  };

  // set-up
  const double sg = a.negate ? -1.0 : 1.0;
  for (int l = tid; l < 32 * ns; l += HT) {
    const int u = 32 * s0 + l;
    if (u >= nv) continue;
    const float4 s4 = H.scale[u];
    const float rv[3] = {(float)(sg * a.b[3 * (size_t)u]) * s4.x, (float)(sg * a.b[3 * (size_t)u + 1]) * s4.y,
                         (float)(sg * a.b[3 * (size_t)u + 2]) * s4.z};
    const float zero[3] = {0.f, 0.f, 0.f};
    const float4 d0 = dinv[3 * (size_t)u], d1 = dinv[3 * (size_t)u + 1], d2 = dinv[3 * (size_t)u + 2];
    const float d[6] = {d0.x, d0.y, d0.z, d1.y, d1.z, d2.z};
    if (l < RS) {
      const float4 i4 = H.iscale[u];
      const float is[3] = {i4.x, i4.y, i4.z};
#pragma unroll
      for (int c = 0; c < 3; ++c) st[(size_t)(FI + c) * RS + l] = is[c];
#pragma unroll
      for (int c = 0; c < 6; ++c) st[(size_t)(FM + c) * RS + l] = d[c];
    }
    st3(FX, x, l, u, zero);
    st3(FR, r, l, u, rv);
    st3(FP, p, l, u, zero);
    st3(FS, sv, l, u, zero);
    st3(FZ, z, l, u, zero);
    float uv[3];
    mul(d, rv, uv);
    m[(size_t)nv + u] = make_float4(uv[0], uv[1], uv[2], 0.f);  // u0 in the second half of m
  }
  bool ok = exchange_barrier(gx, nx++, xs);
  // prologue
  if (ok) {
    for (int t0 = 0; t0 < ns; t0 += pl.tile) {
      const int t1 = min(ns, t0 + pl.tile);
      spmv(m + nv, t0, t1);
      __syncthreads();
      for (int l = 32 * t0 + tid; l < 32 * t1; l += HT) {
        const int u = 32 * s0 + l;
        float e0d = 0.f, e1d = 0.f, e2d = 0.f;
        if (u < nv) {
          float n[3], rv[3], is[3], d[6], uv[3], mv[3];
          product(l, t0, n[0], n[1], n[2]);
          ld3(FR, r, l, u, rv);
          ld3(FI, H.iscale, l, u, is);
          ldm(l, u, d);
          mul(d, rv, uv);
          mul(d, n, mv);
          st3(FW, w, l, u, n);
          m[u] = make_float4(mv[0], mv[1], mv[2], 0.f);
          e0d = rv[0] * uv[0] + rv[1] * uv[1] + rv[2] * uv[2];
          e1d = n[0] * uv[0] + n[1] * uv[1] + n[2] * uv[2];
          e2d = unscaled2(rv, is);
        }
        dots(l, e0d, e1d, e2d);
      }
      if (t1 < ns) __syncthreads();
    }
  }
  for (int k = 0; ok; ++k) {
    const bool first = k == 0;
    __syncthreads();
    ok = exchange_wait<float, 3>(gx, nx, shw, pl.spc, ns, xs);
    if (!ok) break;
    exchange_total<3>(gx, nx++, xs, [&](const double(&t)[3]) {
      step_scalars<true>(sc, first, t[0], t[1], t[2], a.rtol, a.max_iters);
      s_ab[0] = (float)sc.alpha;
      s_ab[1] = (float)sc.beta;
    });
    // the scalars are made while the other warps start on n = A m, which does not need them
    const bool pipe = k < a.pipe_iters;
    const float4* mk = m + (size_t)(k & 1) * nv;
    float4* mn = m + (size_t)((k + 1) & 1) * nv;
    if (pipe) spmv(mk, 0, min(ns, pl.tile));
    __syncthreads();
    if (sc.done) break;
    if (tid == HT - 32) next_reciprocals(sc);
    const float alpha = s_ab[0], beta = s_ab[1];
    if (!pipe) {
      // Chronopoulos-Gear: p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = M r; then w = A u
      for (int l = tid; l < 32 * ns; l += HT) {
        const int u = 32 * s0 + l;
        if (u >= nv) continue;
        float rv[3], wv[3], pv[3], ss[3], xv[3], d[6], uv[3];
        ld3(FR, r, l, u, rv);
        ld3(FW, w, l, u, wv);
        ld3(FP, p, l, u, pv);
        ld3(FS, sv, l, u, ss);
        ld3(FX, x, l, u, xv);
        ldm(l, u, d);
        mul(d, rv, uv);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          pv[c] = uv[c] + beta * pv[c];
          ss[c] = wv[c] + beta * ss[c];
          xv[c] += alpha * pv[c];
          rv[c] -= alpha * ss[c];
        }
        st3(FP, p, l, u, pv);
        st3(FS, sv, l, u, ss);
        st3(FX, x, l, u, xv);
        st3(FR, r, l, u, rv);
        mul(d, rv, uv);
        mn[u] = make_float4(uv[0], uv[1], uv[2], 0.f);
      }
      ok = exchange_barrier(gx, nx++, xs);
      if (!ok) break;
    }
    for (int t0 = 0; t0 < ns; t0 += pl.tile) {
      const int t1 = min(ns, t0 + pl.tile);
      if (!pipe || t0 > 0) {
        spmv(pipe ? mk : mn, t0, t1);
        __syncthreads();
      }
      for (int l = 32 * t0 + tid; l < 32 * t1; l += HT) {
        const int u = 32 * s0 + l;
        float e0d = 0.f, e1d = 0.f, e2d = 0.f;
        if (u < nv) {
          float n[3], rv[3], wv[3], d[6], uv[3], is[3];
          product(l, t0, n[0], n[1], n[2]);
          ld3(FR, r, l, u, rv);
          ldm(l, u, d);
          if (pipe) {
            float v[3], q[3];
            ld3(FW, w, l, u, wv);
            ld3(FZ, z, l, u, v);
#pragma unroll
            for (int c = 0; c < 3; ++c) n[c] += beta * v[c];  // z
            st3(FZ, z, l, u, n);
            ld3(FS, sv, l, u, v);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              v[c] = wv[c] + beta * v[c];  // s
              wv[c] -= alpha * n[c];
            }
            st3(FS, sv, l, u, v);
            st3(FW, w, l, u, wv);
            mul(d, rv, uv);
            ld3(FP, p, l, u, q);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              q[c] = uv[c] + beta * q[c];  // p
              rv[c] -= alpha * v[c];
            }
            st3(FP, p, l, u, q);
            st3(FR, r, l, u, rv);
            ld3(FX, x, l, u, v);
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c] += alpha * q[c];
            st3(FX, x, l, u, v);
            mul(d, wv, v);
            mn[u] = make_float4(v[0], v[1], v[2], 0.f);
          } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) wv[c] = n[c];
            st3(FW, w, l, u, wv);
          }
          mul(d, rv, uv);
          ld3(FI, H.iscale, l, u, is);
          e0d = rv[0] * uv[0] + rv[1] * uv[1] + rv[2] * uv[2];
          e1d = wv[0] * uv[0] + wv[1] * uv[1] + wv[2] * uv[2];
          e2d = unscaled2(rv, is);
        }
        dots(l, e0d, e1d, e2d);
      }
      if (t1 < ns) __syncthreads();
    }
  }
  // x = S x~ (own rows)
  for (int l = tid; l < 32 * ns; l += HT) {
    const int u = 32 * s0 + l;
    if (u >= nv) continue;
    float xv[3];
    ld3(FX, x, l, u, xv);
    const float4 s4 = H.scale[u];
    x[u] = make_float4(xv[0] * s4.x, xv[1] * s4.y, xv[2] * s4.z, 0.f);
  }
  if (ok && blockIdx.x == 0 && tid == 0) publish_scalars(sc, red.sc);
  // the check on the FP32 values: every block's x is final after the exchange; the slices' dots go to the row
  // state's memory (no longer needed) in FP64
  if (ok && a.check) ok = exchange_barrier(gx, nx++, xs);
  if (ok && a.check) {
    double q[4] = {0, 0, 0, 0};
    for (int t0 = 0; t0 < ns; t0 += pl.tile) {
      const int t1 = min(ns, t0 + pl.tile), nu = (t1 - t0) << lt;
      for (int i = warp; i < nu; i += HT / 32) {
        const int ls = t0 + (i >> lt), part = i & (T - 1);
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        if (32 * (s0 + ls) + lane < nv) sym_unit<float>(a.A32, a.vals32, s0 + ls, lane, part, T, x, a0, a1, a2);
        float* o = pb + (size_t)3 * part * PR + 32 * (ls - t0) + lane;
        o[0] = a0;
        o[PR] = a1;
        o[2 * PR] = a2;
      }
      __syncthreads();
      for (int l = 32 * t0 + tid; l < 32 * t1; l += HT) {
        const int u = 32 * s0 + l;
        if (u >= nv) continue;
        float n0, n1, n2;
        product(l, t0, n0, n1, n2);
        const float4 dv = x[u];
        const double g0 = a.b[3 * (size_t)u], g1 = a.b[3 * (size_t)u + 1], g2 = a.b[3 * (size_t)u + 2];
        const double x0 = dv.x, x1 = dv.y, x2 = dv.z;
        q[0] += g0 * x0 + g1 * x1 + g2 * x2;
        q[1] += x0 * x0 + x1 * x1 + x2 * x2;
        const double q0 = sg * g0 - (double)n0, q1 = sg * g1 - (double)n1, q2 = sg * g2 - (double)n2;
        q[2] += q0 * q0 + q1 * q1 + q2 * q2;
        q[3] += g0 * g0 + g1 * g1 + g2 * g2;
      }
      __syncthreads();
    }
    // per-warp sums to shared memory (the unit partials' space: at least 3 * 32 * 4 * 8 values)
    double* shq = reinterpret_cast<double*>(pb);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const double t = warp_add(q[c]);
      if (lane == 0) shq[32 * c + warp] = t;
    }
    ok = exchange<double, 4>(gx, nx++, shq, 32, HT / 32, xs, [&](const double(&t)[4]) {
      if (blockIdx.x == 0) {
        red.sc->gd = t[0];
        red.sc->dnorm2 = t[1];
        red.sc->true_rr = t[2];
        red.sc->true_bb = t[3];
      }
    });
  }
  if (!ok && tid == 0) atomicExch(&red.sc->wait_failed, 1);
}

// ------------------------------------------------------------------ FP64
struct Plan64 {
  int grid, T, spc, cached;
  int cache_entries;  // most entries of a block (when cached)
  size_t smem;
};

constexpr int DT = 512;        // threads of a block
constexpr int kState64 = 27;   // FP64 values of a row kept on chip: x r p s z w u (21), M (6)

// PCG in FP64 on the symmetric store, the whole solve in one launch with the set-up and, with a.check, g . x and |x|^2
// at its end: Chronopoulos-Gear (as cgcg_persistent_kernel), after pipe_iters pipelined iterations (as
// resident_half_kernel, in the unscaled space) that save one of its two exchanges.  GB300 has two FP64 lanes an SM and
// clock, so the work is laid out for them: any four warps fill the units, a lone warp fills one; the row recurrences
// run a thread per dof (15 operations deep instead of 57), M r is carried in place of being formed twice, and T
// partial products cost T - 1 additions, so T is 4 only where a block has fewer than four slices.  With CACHED the
// block's rows of the matrix, lower triangle included, are copied to shared memory once a solve.  Bound by the
// exchanges on small systems and by the FP64 units (135 operations a row in the product) beyond a few thousand rows.
template <bool CACHED, int T>
__global__ void __launch_bounds__(DT, 1)
    resident64_kernel(SellMatrix A, const double* __restrict__ vals, const double4_32a* __restrict__ dinv, double4_32a* x,
                      double4_32a* m, Solve64Args a, Plan64 pl, Reduce red, GridExchange gx) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ ExchangeShared xs;
  __shared__ Scalars sc;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nv = A.nv, nsl = (nv + 31) >> 5;
  const int s0 = (int)((long long)blockIdx.x * nsl / gridDim.x), ns = (int)((long long)(blockIdx.x + 1) * nsl / gridDim.x) - s0;
  const int RS = 32 * pl.spc, nd = 96 * ns;  // row stride of the state; dofs of this block (padding rows included)
  constexpr int lt = T == 4 ? 2 : 1;
  static_assert(T == 1 << lt, "T is 2 or 4");
  double* cv = reinterpret_cast<double*>(smem);  // cached values: entry e (a multiple of 32) at 9 e + 32 c + lane
  double* st = cv + (size_t)9 * pl.cache_entries;
  double* pb = st + (size_t)kState64 * RS;       // unit partials
  double* sh = pb + (size_t)3 * T * RS;          // 3 x DT partial dots
  int* cc = reinterpret_cast<int*>(sh + 3 * DT);
  double *X = st, *R = st + 3 * RS, *P = st + 6 * RS, *S = st + 9 * RS, *Z = st + 12 * RS, *W = st + 15 * RS,
         *U = st + 18 * RS, *M = st + 21 * RS;
  if (tid == 0) xs.fail = 0;
  if constexpr (CACHED) {
    for (int ls = warp; ls < ns; ls += DT / 32) {
      const int s = s0 + ls, ub = A.sl_off[s], lb = A.lo_off[s];
      const int Wu = (A.sl_off[s + 1] - ub) >> 5, Wl = (A.lo_off[s + 1] - lb) >> 5;
      const int e0 = (ub - A.sl_off[s0]) + (lb - A.lo_off[s0]);
      for (int k = 0; k < Wu + Wl; ++k) {
        const bool up = k < Wu;
        const int q = up ? ub + 32 * k + lane : A.lo_src[lb + 32 * (k - Wu) + lane];
        // padding columns name the entry's own row, which may lie past the last vertex
        cc[e0 + 32 * k + lane] = min(up ? A.sl_col[q] : A.lo_col[lb + 32 * (k - Wu) + lane], nv - 1);
        const double* src = vals + sell_base(q);
        double* dst = cv + (size_t)9 * (e0 + 32 * k) + lane;
#pragma unroll
        for (int c = 0; c < 9; ++c) dst[32 * c] = src[32 * (up ? c : 3 * (c % 3) + c / 3)];
      }
    }
  }

  auto spmv = [&](const double4_32a* v) {
    for (int i = DT / 32 - 1 - warp; i < (ns << lt); i += DT / 32) {
      const int ls = i >> lt, part = i & (T - 1), s = s0 + ls;
      double a0 = 0, a1 = 0, a2 = 0;
      if constexpr (CACHED) {
        const int e0 = (A.sl_off[s] - A.sl_off[s0]) + (A.lo_off[s] - A.lo_off[s0]);
        const int n = ((A.sl_off[s + 1] - A.sl_off[s]) + (A.lo_off[s + 1] - A.lo_off[s])) >> 5;
        const double* pv = cv + (size_t)9 * e0 + lane;
        for (int k = part; k < n; k += 2 * T) {
          const bool two = k + T < n;
          const int k1 = two ? k + T : k;
          const double4_32a x0 = v[cc[e0 + 32 * k + lane]];
          double4_32a x1 = v[cc[e0 + 32 * k1 + lane]];
          const double *p0 = pv + 288 * k, *p1 = pv + 288 * k1;
          a0 = fma(p0[64], x0.z, fma(p0[32], x0.y, fma(p0[0], x0.x, a0)));
          a1 = fma(p0[160], x0.z, fma(p0[128], x0.y, fma(p0[96], x0.x, a1)));
          a2 = fma(p0[256], x0.z, fma(p0[224], x0.y, fma(p0[192], x0.x, a2)));
          if (two) {
            a0 = fma(p1[64], x1.z, fma(p1[32], x1.y, fma(p1[0], x1.x, a0)));
            a1 = fma(p1[160], x1.z, fma(p1[128], x1.y, fma(p1[96], x1.x, a1)));
            a2 = fma(p1[256], x1.z, fma(p1[224], x1.y, fma(p1[192], x1.x, a2)));
          }
        }
      } else if (32 * s + lane < nv) {
        sym_unit<double>(A, vals, s, lane, part, T, v, a0, a1, a2);
      }
      double* o = pb + (size_t)3 * part * RS + 32 * ls + lane;
      o[0] = a0;
      o[RS] = a1;
      o[2 * RS] = a2;
    }
  };
  // dof j of the block: component j / (32 ns) of row j % (32 ns), so that a warp's threads share the component
  auto dof = [&](int j, int& c, int& l) {
    const int n = 32 * ns;
    c = (j >= n) + (j >= 2 * n);
    l = j - c * n;
  };
  auto product = [&](int c, int l) {
    const double* o = pb + (size_t)c * RS + l;
    double t = o[0];
#pragma unroll
    for (int q = 1; q < T; ++q) t += o[(size_t)3 * q * RS];
    return t;
  };
  // component c of the symmetric M v; M holds the rows' (00, 01, 02, 11, 12, 22)
  auto precond = [&](const double* v, int c, int l) {
    const int i0 = c, i1 = c == 0 ? 1 : c + 2, i2 = c == 0 ? 2 : c + 3;
    return fma(M[(size_t)i2 * RS + l], v[2 * RS + l], fma(M[(size_t)i1 * RS + l], v[RS + l], M[(size_t)i0 * RS + l] * v[l]));
  };
  auto put = [&](double4_32a* g, int u, int c, double v) { reinterpret_cast<double*>(g + u)[c] = v; };

  // set-up
  const double sg = a.negate ? -1.0 : 1.0;
  for (int l = tid; l < 32 * ns; l += DT) {
    const int u = 32 * s0 + l;
    double4_32a d0 = mk4<double>(0, 0, 0), d1 = d0, d2 = d0;
    if (u < nv) {
      d0 = dinv[3 * (size_t)u];
      d1 = dinv[3 * (size_t)u + 1];
      d2 = dinv[3 * (size_t)u + 2];
    }
    const double d[6] = {d0.x, d0.y, d0.z, d1.y, d1.z, d2.z};
#pragma unroll
    for (int c = 0; c < 6; ++c) M[(size_t)c * RS + l] = d[c];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      R[c * RS + l] = u < nv ? sg * a.b[3 * (size_t)u + c] : 0.0;
      X[c * RS + l] = P[c * RS + l] = S[c * RS + l] = Z[c * RS + l] = 0.0;
    }
  }
  __syncthreads();
  for (int j = tid; j < nd; j += DT) {
    int c, l;
    dof(j, c, l);
    const double u0 = precond(R, c, l);
    U[c * RS + l] = u0;
    if (32 * s0 + l < nv) put(m + nv, 32 * s0 + l, c, u0);  // u0 in the second half of m
  }
  unsigned long long nx = 0;
  bool ok = exchange_barrier(gx, nx++, xs);
  const int np = min(DT, nd);
  auto store_dots = [&](double d0, double d1, double d2) {
    sh[tid] = d0;
    sh[DT + tid] = d1;
    sh[2 * DT + tid] = d2;
  };
  if (ok) {  // prologue: w = A u0, m_0 = M w
    spmv(m + nv);
    __syncthreads();
    for (int j = tid; j < nd; j += DT) {
      int c, l;
      dof(j, c, l);
      W[c * RS + l] = product(c, l);
    }
    __syncthreads();
    double d0 = 0, d1 = 0, d2 = 0;
    for (int j = tid; j < nd; j += DT) {
      int c, l;
      dof(j, c, l);
      const double r = R[c * RS + l], u = U[c * RS + l];
      d0 = fma(r, u, d0);
      d1 = fma(W[c * RS + l], u, d1);
      d2 = fma(r, r, d2);
      if (a.pipe_iters > 0 && 32 * s0 + l < nv) put(m, 32 * s0 + l, c, precond(W, c, l));
    }
    store_dots(d0, d1, d2);
  }
  for (int k = 0; ok; ++k) {
    const bool first = k == 0;
    __syncthreads();
    ok = exchange_wait<double, 3>(gx, nx, sh, DT, np, xs);
    if (!ok) break;
    exchange_total<3>(gx, nx++, xs, [&](const double(&t)[3]) {
      step_scalars<false>(sc, first, t[0], t[1], t[2], a.rtol, a.max_iters);
    });
    const bool pipe = k < a.pipe_iters;
    const double4_32a* mk = m + (size_t)(k & 1) * nv;
    double4_32a* mn = m + (size_t)((k + 1) & 1) * nv;
    if (pipe) spmv(mk);  // n = A m while the scalars are made
    __syncthreads();
    if (sc.done) break;
    if (tid == DT - 32) next_reciprocals(sc);
    const double alpha = sc.alpha, beta = sc.beta;
    double d0 = 0, d1 = 0, d2 = 0;
    for (int j = tid; j < nd; j += DT) {
      int c, l;
      dof(j, c, l);
      const int i = c * RS + l;
      const double w = W[i], p = fma(beta, P[i], U[i]), s = fma(beta, S[i], w);
      P[i] = p;
      S[i] = s;
      X[i] = fma(alpha, p, X[i]);
      R[i] = fma(-alpha, s, R[i]);
      if (pipe) {
        const double z = fma(beta, Z[i], product(c, l));
        Z[i] = z;
        W[i] = fma(-alpha, z, w);
      }
    }
    __syncthreads();
    for (int j = tid; j < nd; j += DT) {
      int c, l;
      dof(j, c, l);
      const int i = c * RS + l;
      const double u = precond(R, c, l);
      U[i] = u;
      if (pipe) {
        const double r = R[i];
        d0 = fma(r, u, d0);
        d1 = fma(W[i], u, d1);
        d2 = fma(r, r, d2);
      }
      if (32 * s0 + l < nv) put(mn, 32 * s0 + l, c, pipe ? precond(W, c, l) : u);
    }
    if (!pipe) {  // Chronopoulos-Gear: w = A u after every block's u is there
      ok = exchange_barrier(gx, nx++, xs);
      if (!ok) break;
      spmv(mn);
      __syncthreads();
      for (int j = tid; j < nd; j += DT) {
        int c, l;
        dof(j, c, l);
        const int i = c * RS + l;
        const double r = R[i], u = U[i], w = product(c, l);
        W[i] = w;
        d0 = fma(r, u, d0);
        d1 = fma(w, u, d1);
        d2 = fma(r, r, d2);
      }
    }
    store_dots(d0, d1, d2);
  }
  __syncthreads();
  double q[2] = {0, 0};
  for (int l = tid; l < 32 * ns; l += DT) {
    const int u = 32 * s0 + l;
    if (u >= nv) continue;
    const double x0 = X[l], x1 = X[RS + l], x2 = X[2 * RS + l];
    x[u] = mk4<double>(x0, x1, x2);
    if (a.check) {
      q[0] = fma(a.b[3 * (size_t)u + 2], x2, fma(a.b[3 * (size_t)u + 1], x1, fma(a.b[3 * (size_t)u], x0, q[0])));
      q[1] = fma(x2, x2, fma(x1, x1, fma(x0, x0, q[1])));
    }
  }
  if (ok && blockIdx.x == 0 && tid == 0) publish_scalars(sc, red.sc);
  if (ok && a.check) {
    sh[tid] = q[0];
    sh[DT + tid] = q[1];
    ok = exchange<double, 2>(gx, nx++, sh, DT, min(DT, 32 * ns), xs, [&](const double(&t)[2]) {
      if (blockIdx.x == 0) {
        red.sc->gd = t[0];
        red.sc->dnorm2 = t[1];
      }
    });
  }
  if (!ok && tid == 0) atomicExch(&red.sc->wait_failed, 1);
}

size_t smem64(const Plan64& p) {
  const size_t rs = (size_t)32 * p.spc;
  return 8 * ((size_t)9 * p.cache_entries + kState64 * rs + 3 * p.T * rs + 3 * DT) + 4 * (size_t)p.cache_entries + 64;
}

constexpr size_t kSmemReserve = 8 * 1024;  // static shared memory and the 1 KB a block costs

size_t half_smem(const HalfPlan& p) {
  const size_t f = (size_t)kHalfState * 32 * p.res + (size_t)3 * p.T * 32 * p.tile + 4 * (size_t)p.spc;
  return (size_t)16 * p.cache_entries + 4 * f + 4 * ((size_t)p.spc + 1) +
         (p.packed ? 4 : 6) * (size_t)p.cache_entries + 64;
}

}  // namespace

size_t resident_sync_bytes() { return 128 + (size_t)2 * 4 * kMaxBlocks * sizeof(double); }

// first slice of block c's part of nsl slices over g blocks
static int part_begin(int c, int nsl, int g) { return (int)((long long)c * nsl / g); }

static GridExchange grid_exchange(const ResidentSync& rs, cudaStream_t st) {
  SSIM_CUDA(cudaMemsetAsync(rs.mem, 0, sizeof(unsigned long long), st));
  return GridExchange{reinterpret_cast<unsigned long long*>(rs.mem), reinterpret_cast<double*>(rs.mem + 128),
                      (unsigned int)rs.extra, rs.spin_limit > 0 ? rs.spin_limit : (1LL << 21)};
}

// 20 or 22 bytes an entry against the double-buffered m and the vectors of the rows that are not on chip
static HalfPlan l2_hints(HalfPlan p, int nv, const int32_t* off, size_t l2) {
  const double matrix = (p.packed ? 20.0 : 22.0) * off[div_up(nv, 32)];
  const double other = 32.0 * nv + 176.0 * nv * (p.spc - p.res) / std::max(p.spc, 1);
  if (p.grid > 0 && matrix + other > 0.8 * (double)l2)
    p.keep = (int)(p.spc * std::min(1.0, std::max(0.0, 0.6 * (double)l2 - other) / matrix));
  return p;
}

// Layout of a resident solve on the FP16 copy (host arithmetic only; off: the copy's slice offsets).
//  T: 4 warps a slice (a 15-entry slice is four entries a unit: all of a unit's loads in flight at once), 8 where a
//  block has fewer than 8 slices (small systems: fewer dependent rounds).
//  The vectors of all rows stay on chip while they and one pass over the block's slices fit (1,408 rows a block,
//  214,000 on 152 SMs); beyond, passes of 32 slices and the rows that fit.  The matrix entries too
//  where the block's part of them fits (about 70,000 rows): an iteration then reads nothing but the gathered
//  vector from L2.
//  L2 hints where what an iteration cycles through does not fit (table: 22-byte entries): swept in order, an LRU-like cache then keeps nothing.
//  The entries of the first slices of every block are loaded with evict_last, the others with evict_first.  Measured on
//  batches of cubes, 126 MB of L2 (matrix / other bytes, MB; Newton iterations, ms): 77 / 8 6.43 without and 6.77 with
//  60 MB kept; 92 / 17 10.1, 8.87 with 60; 108 / 28 15.1, 12.9 with 50; 118 / 35 18.0, 15.4 with 40; 157 / 60 22.7, 20.3
//  with 20; 250 / 122 36.9, 36.6.  So: hints above 0.8 of L2, 0.6 of L2 less the other bytes kept.
static HalfPlan half_plan(int nv, int packed, const int32_t* off, int nsm, size_t smem_max, size_t l2, int max_blocks) {
  HalfPlan p{};
  p.packed = packed;
  p.keep = -1;
  const int nsl = div_up(nv, 32);
  p.grid = std::max(1, std::min(std::min(nsm, kMaxBlocks), nsl));
  if (max_blocks > 0) p.grid = std::min(p.grid, max_blocks);
  for (int c = 0; c < p.grid; ++c) p.spc = std::max(p.spc, part_begin(c + 1, nsl, p.grid) - part_begin(c, nsl, p.grid));
  p.T = 4;
  p.res = p.tile = p.spc;
  if (half_smem(p) > smem_max) {
    p.tile = 32;
    p.res = 0;
    const size_t base = half_smem(p);
    const size_t row = (size_t)4 * kHalfState * 32;
    p.res = base < smem_max ? (int)std::min<size_t>((size_t)p.spc, (smem_max - base) / row) : 0;
    if (base > smem_max) p.grid = 0;
    return l2_hints(p, nv, off, l2);
  }
  HalfPlan q = p;
  for (int c = 0; c < p.grid; ++c)
    q.cache_entries = std::max(q.cache_entries, off[part_begin(c + 1, nsl, p.grid)] - off[part_begin(c, nsl, p.grid)]);
  q.cached = 1;
  if (p.spc < 8) q.T = 8;
  return half_smem(q) <= smem_max ? q : l2_hints(p, nv, off, l2);
}

// properties of the current device that a resident launch needs; false without cooperative launches
static bool resident_device(int& nsm, size_t& smem_max, size_t& l2) {
  int dev = 0, coop = 0, smax = 0, l2b = 0;
  SSIM_CUDA(cudaGetDevice(&dev));
  SSIM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  SSIM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  SSIM_CUDA(cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  SSIM_CUDA(cudaDeviceGetAttribute(&l2b, cudaDevAttrL2CacheSize, dev));
  smem_max = (size_t)smax - kSmemReserve;
  l2 = (size_t)l2b;
  return coop != 0;
}
// The limit on dynamic shared memory belongs to the kernel in its context, and handles launch from any thread: every call
// sets the same value, the device's most, and never this handle's size.
static bool resident_fits(const void* fn, int threads, size_t smem, size_t smem_max) {
  int per_sm = 0;
  SSIM_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
  SSIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
  return per_sm >= 1;
}

bool launch_pcg_half_resident(const HalfMatrix& H, const int32_t* off_host, const float4* dinv16, float4* x, float4* r,
                              float4* z, float4* p, float4* sv, float4* w, float4* m, const HalfSolveArgs& pa,
                              const Reduce& red, const ResidentSync& rs, int max_blocks, cudaStream_t st) {
  if (H.nv <= 0) return true;
  int nsm = 0;
  size_t smem_max = 0, l2 = 0;
  if (!resident_device(nsm, smem_max, l2)) return false;
  HalfPlan pl = half_plan(H.nv, H.vs == 2, off_host, nsm, smem_max, l2, max_blocks);
  if (pl.grid < 1) return false;
  pl.smem = half_smem(pl);
  auto kernel = [&](auto P) {
    constexpr bool k = decltype(P)::value;
    return pl.keep >= 0 ? (const void*)resident_half_kernel<false, 4, true, k>
           : !pl.cached ? (const void*)resident_half_kernel<false, 4, false, k>
           : pl.T == 4  ? (const void*)resident_half_kernel<true, 4, false, k>
                        : (const void*)resident_half_kernel<true, 8, false, k>;
  };
  const void* fn = pl.packed ? kernel(std::true_type{}) : kernel(std::false_type{});
  if (!resident_fits(fn, HT, pl.smem, smem_max)) return false;
  GridExchange gx = grid_exchange(rs, st);
  HalfMatrix h = H;
  HalfSolveArgs ha = pa;
  Reduce rd = red;
  void* args[] = {(void*)&h, (void*)&dinv16, (void*)&x,  (void*)&r,  (void*)&z,  (void*)&p,  (void*)&sv,
                  (void*)&w, (void*)&m,      (void*)&ha, (void*)&pl, (void*)&rd, (void*)&gx};
  SSIM_CUDA(cudaLaunchCooperativeKernel(fn, dim3(pl.grid), dim3(HT), args, pl.smem, st));
  after_launch("pcg_half_resident");
  return true;
}

// Layout of a resident FP64 solve: all rows' vectors on chip or none (25 slices a block, 121,600 rows on 152 SMs), the
// matrix entries too where they fit (four slices of 15 entries a row, 19,000 rows).  grid 0: does not fit.
static Plan64 plan64(int nv, const int32_t* sl_off, const int32_t* lo_off, int nsm, size_t smem_max, int max_blocks) {
  Plan64 p{};
  const int nsl = div_up(nv, 32);
  p.grid = std::max(1, std::min(std::min(nsm, kMaxBlocks), nsl));
  if (max_blocks > 0) p.grid = std::min(p.grid, max_blocks);
  Plan64 q{};
  for (int c = 0; c < p.grid; ++c) {
    const int a = part_begin(c, nsl, p.grid), b = part_begin(c + 1, nsl, p.grid);
    p.spc = std::max(p.spc, b - a);
    q.cache_entries = std::max(q.cache_entries, (sl_off[b] - sl_off[a]) + (lo_off[b] - lo_off[a]));
  }
  p.T = p.spc < 4 ? 4 : 2;
  q.grid = p.grid;
  q.spc = p.spc;
  q.T = p.T;
  q.cached = 1;
  if (smem64(q) <= smem_max) return q;
  p.T = 2;
  if (smem64(p) > smem_max) p.grid = 0;
  return p;
}

bool launch_pcg64_resident(const SellMatrix& A, const int32_t* sl_off, const int32_t* lo_off, const double* vals,
                           const double4_32a* dinv, double4_32a* x, const std::function<double4_32a*()>& scratch,
                           const Solve64Args& sa, const Reduce& red,
                           const ResidentSync& rs, int max_blocks, cudaStream_t st) {
  if (A.nv <= 0) return true;
  int nsm = 0;
  size_t smem_max = 0, l2 = 0;
  if (!resident_device(nsm, smem_max, l2)) return false;
  Plan64 pl = plan64(A.nv, sl_off, lo_off, nsm, smem_max, max_blocks);
  if (pl.grid < 1) return false;
  pl.smem = smem64(pl);
  const void* fn = !pl.cached   ? (const void*)resident64_kernel<false, 2>
                   : pl.T == 2 ? (const void*)resident64_kernel<true, 2>
                               : (const void*)resident64_kernel<true, 4>;
  if (!resident_fits(fn, DT, pl.smem, smem_max)) return false;
  double4_32a* m = scratch();
  GridExchange gx = grid_exchange(rs, st);
  SellMatrix a = A;
  Solve64Args s = sa;
  Reduce rd = red;
  void* args[] = {(void*)&a, (void*)&vals, (void*)&dinv, (void*)&x,  (void*)&m,
                  (void*)&s, (void*)&pl,   (void*)&rd,   (void*)&gx};
  SSIM_CUDA(cudaLaunchCooperativeKernel(fn, dim3(pl.grid), dim3(DT), args, pl.smem, st));
  after_launch("pcg64_resident");
  return true;
}

}  // namespace ssim_gb
