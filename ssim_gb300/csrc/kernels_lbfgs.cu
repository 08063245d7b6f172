// kernels_lbfgs.cu -- the L-BFGS two-loop recursion and curvature pair with every coefficient kept in device
// memory, so an L-BFGS iteration needs no host round trip until its line-search trial has been evaluated.
//
// The recursion is the textbook one (Nocedal & Wright, Algorithm 7.4): first loop a_i = rho_i s_i.q,
// q -= a_i y_i (newest pair first); z = H0 q; second loop b_i = rho_i y_i.z, z += (a_i - b_i) s_i (oldest
// first); d = -z.  Each pass kernel applies the previous step's update and forms the next step's dot in one
// sweep over the vectors; the last block to finish writes the coefficient, which the next launch reads.
#include "kernels.cuh"

namespace ssim_gb {
namespace {

constexpr int LB = 256;

// Per-vertex arithmetic is in S (FP32 in mixed precision: GB300's FP64 pipe is narrow, and a float<->double
// conversion costs an FP64 slot); partial sums go to FP64 at the warp level and the grid sums are FP64.
template <typename S>
__device__ __forceinline__ S dot3(const V4<S>& a, const V4<S>& b) {
  return a.x * b.x + a.y * b.y + a.z * b.z;
}

// vout = scale * (vin + c w), c = csign (cA - cB) read from device memory (w == null: no update; vin == null:
// the FP64 gradient g is the input); then out = rho * (a . vout) when a != null
template <typename S>
__global__ void __launch_bounds__(LB)
    lbfgs_pass_kernel(int nv, const V4<S>* vin, const double* __restrict__ g, V4<S>* vout, const V4<S>* __restrict__ w,
                      const double* __restrict__ cA, const double* __restrict__ cB, double csign,
                      const double* __restrict__ scale_ptr, double scale, const V4<S>* __restrict__ a, double rho,
                      double* __restrict__ out, Reduce red) {
  __shared__ double shred[LB / 32][1];
  const int u = blockIdx.x * LB + threadIdx.x;
  S part[1] = {S(0)};
  if (u < nv) {
    V4<S> x;
    if (vin != nullptr)
      x = vin[u];
    else
      x = mk4<S>((S)g[3 * u], (S)g[3 * u + 1], (S)g[3 * u + 2]);
    if (w != nullptr) {
      const S c = (S)(csign * (cA[0] - (cB != nullptr ? cB[0] : 0.0)));
      const V4<S> wv = w[u];
      x.x += c * wv.x;
      x.y += c * wv.y;
      x.z += c * wv.z;
    }
    const S sc = (S)(scale_ptr != nullptr ? scale_ptr[0] : scale);
    const V4<S> r = mk4<S>(sc * x.x, sc * x.y, sc * x.z);
    vout[u] = r;
    if (a != nullptr) part[0] = dot3<S>(a[u], r);
  }
  if (a == nullptr) return;
  double v1[1];
  block_sum_s<1, LB, S>(part, v1, shred);
  double tot[1];
  if (grid_sum_last<1, LB>(v1, red.partials, red.counter, tot)) out[0] = rho * tot[0];
}

// d = -(z + c w), g . d and |d|^2 into the scalars (c = cA - cB; w == null: none); d may be z
template <typename S>
__global__ void __launch_bounds__(LB)
    lbfgs_final_kernel(int nv, const V4<S>* z, const V4<S>* __restrict__ w, const double* __restrict__ cA,
                       const double* __restrict__ cB, const double* __restrict__ g, V4<S>* d, Reduce red) {
  __shared__ double shred[LB / 32][2];
  const int u = blockIdx.x * LB + threadIdx.x;
  S part[2] = {S(0), S(0)};
  if (u < nv) {
    V4<S> x = z[u];
    if (w != nullptr) {
      const S c = (S)(cA[0] - (cB != nullptr ? cB[0] : 0.0));
      const V4<S> wv = w[u];
      x.x += c * wv.x;
      x.y += c * wv.y;
      x.z += c * wv.z;
    }
    const V4<S> dv = mk4<S>(-x.x, -x.y, -x.z);
    d[u] = dv;
    const V4<S> gv = mk4<S>((S)g[3 * u], (S)g[3 * u + 1], (S)g[3 * u + 2]);
    part[0] = dot3<S>(gv, dv);
    part[1] = dot3<S>(dv, dv);
  }
  double v2[2];
  block_sum_s<2, LB, S>(part, v2, shred);
  double tot[2];
  if (grid_sum_last<2, LB>(v2, red.partials, red.counter, tot)) {
    red.sc->gd = tot[0];
    red.sc->dnorm2 = tot[1];
  }
}

// the curvature pair of a trial point: s = alpha d, y = g_new - g_old (differenced in FP64, then rounded);
// s . y and y . y into the scalars
template <typename S>
__global__ void __launch_bounds__(LB)
    lbfgs_pair_kernel(int nv, double alpha, const V4<S>* __restrict__ d, const double* __restrict__ gnew,
                      const double* __restrict__ gold, V4<S>* __restrict__ sv, V4<S>* __restrict__ yv, Reduce red) {
  __shared__ double shred[LB / 32][2];
  const int u = blockIdx.x * LB + threadIdx.x;
  S part[2] = {S(0), S(0)};
  if (u < nv) {
    const V4<S> dv = d[u];
    const S a = (S)alpha;
    const V4<S> s = mk4<S>(a * dv.x, a * dv.y, a * dv.z);
    const V4<S> y = mk4<S>((S)(gnew[3 * u] - gold[3 * u]), (S)(gnew[3 * u + 1] - gold[3 * u + 1]),
                           (S)(gnew[3 * u + 2] - gold[3 * u + 2]));
    sv[u] = s;
    yv[u] = y;
    part[0] = dot3<S>(s, y);
    part[1] = dot3<S>(y, y);
  }
  double v2[2];
  block_sum_s<2, LB, S>(part, v2, shred);
  double tot[2];
  if (grid_sum_last<2, LB>(v2, red.partials, red.counter, tot)) {
    red.sc->pair_sy = tot[0];
    red.sc->pair_yy = tot[1];
  }
}

// accept a step: u += alpha d (FP64 state), g_old = g_new
template <typename S>
__global__ void __launch_bounds__(LB)
    lbfgs_accept_kernel(int nv, double alpha, const V4<S>* __restrict__ d, double* __restrict__ u,
                        const double* __restrict__ gnew, double* __restrict__ gold) {
  const int v = blockIdx.x * LB + threadIdx.x;
  if (v >= nv) return;
  const V4<S> dv = d[v];
  u[3 * v] += alpha * (double)dv.x;
  u[3 * v + 1] += alpha * (double)dv.y;
  u[3 * v + 2] += alpha * (double)dv.z;
  gold[3 * v] = gnew[3 * v];
  gold[3 * v + 1] = gnew[3 * v + 1];
  gold[3 * v + 2] = gnew[3 * v + 2];
}

// ---------------------------------------------------------------- compact form
// The same L-BFGS matrix in the compact representation of Byrd, Nocedal & Schnabel (Math. Prog. 63, 1994;
// Nocedal & Wright eq. 7.24): H g = gamma g + S p - gamma Y q with q = R^-1 (S^T g) and
// p = R^-T ((D + gamma Y^T Y) q - gamma Y^T g), R the upper triangle of S^T Y in age order, D its diagonal.
// One pass forms S^T g, Y^T g and the newest pair's column of S^T Y and Y^T Y (all vectors read once); the
// last block solves the small triangular systems; a second pass forms d = -H g.

// the exchanges of sums of N values (a power of two up to 32) over a warp: each halves the values a lane still carries (N - 1
// additions instead of 5 N); what is left is summed over the lanes that differ in the bits from 32 / N up and belongs to the
// value those bits name, lowest first
template <int N, typename S>
__device__ __forceinline__ S warp_transpose_sum(const S (&v)[N]) {
  if constexpr (N == 1) {
    return v[0];
  } else {
    constexpr int o = N / 2;  // values kept; the lanes' distance at this level is 16 for the first one
    const int lane = threadIdx.x & 31;
    S w[o];
    constexpr int dist = N == 32 ? 1 : N == 16 ? 2 : N == 8 ? 4 : N == 4 ? 8 : 16;
    const bool hi = lane & dist;
#pragma unroll
    for (int k = 0; k < o; ++k) {
      const S keep = hi ? v[2 * k + 1] : v[2 * k], give = hi ? v[2 * k] : v[2 * k + 1];
      w[k] = keep + __shfl_xor_sync(0xffffffffu, give, dist);
    }
    return warp_transpose_sum<o, S>(w);
  }
}

// per vertex: a_j = s_j.g, b_j = y_j.g, c_j = s_j.y_new, e_j = y_j.y_new (j in age order, oldest first);
// the last block keeps the new column in the slot-indexed S^T Y / Y^T Y tables and writes the coefficients.
// PG warps share 32 vertices, each taking 8 / PG of the pairs: 1 for large systems, 4 where the vertices are too few to
// occupy the SMs otherwise (in FP64 a thread's 96 products then cost 24).  In FP64 the kernel is bound by the FP64 units
// (a warp's operation every 64 cycles): the 32 sums take 31 additions a warp instead of 160, and the small triangular
// systems are solved by eight lanes with the diagonal's reciprocals instead of by one thread with 16 divisions.
// 9,225 vertices, FP64: 10.5 us (38.4 before).
template <typename S, int PG>
__global__ void __launch_bounds__(LB)
    lbfgs_multidot_kernel(int nv, const double* __restrict__ g, LbfgsHist<S> h, double* __restrict__ partials,
                          double* __restrict__ tab, unsigned int* counter) {
  constexpr int NV = 4 * kLbfgsMaxCompact, NP = kLbfgsMaxCompact / PG, NA = 4 * NP;
  constexpr int VB = LB / PG;  // vertices of a block at a time
  static_assert(NV == 32 && LB % NV == 0, "a lane per value");
  __shared__ double shred[LB / 32][NV];
  __shared__ bool am_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pg = warp % PG;
  S acc[NA];
#pragma unroll
  for (int k = 0; k < NA; ++k) acc[k] = S(0);
  // a grid of a few blocks per SM striding over the vertices: the block sums and the last block's sum
  // over the grid (NV values per block) stay short
  for (int u = blockIdx.x * VB + 32 * (warp / PG) + lane; u < nv; u += gridDim.x * VB) {
    const V4<S> gv = mk4<S>((S)g[3 * u], (S)g[3 * u + 1], (S)g[3 * u + 2]);
    const V4<S> yn = h.y[h.n - 1][u];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int j = NP * pg + i;
      if (j < h.n) {
        const V4<S> sv = h.s[j][u], yv = h.y[j][u];
        acc[4 * i + 0] += dot3<S>(sv, gv);
        acc[4 * i + 1] += dot3<S>(yv, gv);
        acc[4 * i + 2] += dot3<S>(sv, yn);
        acc[4 * i + 3] += dot3<S>(yv, yn);
      }
    }
  }
  // block sums (FP32 within a warp, FP64 across warps), then the grid sum in FP64 by the last block
  {
    S x = warp_transpose_sum<NA, S>(acc);
#pragma unroll
    for (int o = 16 / NA; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    // the lanes' bits, lowest distance first, name the value: level by level the low bit of the index
    int k = 0;
#pragma unroll
    for (int b = 0; (1 << b) < NA; ++b) {
      constexpr int first = NA == 32 ? 0 : NA == 16 ? 1 : 2;
      k |= ((lane >> (first + b)) & 1) << b;
    }
    if (NA == 32 || (lane & ((32 / NA) - 1)) == 0) shred[warp][NA * pg + k] = (double)x;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double b = 0;
    const int own = threadIdx.x / NA;  // the warps that carry this value
#pragma unroll
    for (int w = 0; w < LB / 32 / PG; ++w) b += shred[PG * w + own][threadIdx.x];
    partials[(size_t)blockIdx.x * NV + threadIdx.x] = b;
  }
  __syncthreads();  // orders the partials before thread 0's release
  if (threadIdx.x == 0) am_last = (atom_inc_acq_rel_gpu(counter) == gridDim.x - 1);
  __syncthreads();
  if (!am_last) return;
  // LB / NV groups of threads each sum every (LB / NV)-th block's partials (four chains), then the groups in order
  double tot = 0;  // lane k of warp 0: value k
  {
    constexpr int G = LB / NV;
    const int k = threadIdx.x % NV, grp = threadIdx.x / NV;
    double t[4] = {0, 0, 0, 0};
    for (int b = grp; b < (int)gridDim.x; b += 4 * G) {
      double v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = b + i * G < (int)gridDim.x ? __ldcg(partials + (size_t)(b + i * G) * NV + k) : 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (b + i * G < (int)gridDim.x) t[i] += v[i];
    }
    shred[grp][k] = (t[0] + t[1]) + (t[2] + t[3]);
    __syncthreads();
    if (threadIdx.x >= NV) return;
#pragma unroll
    for (int q = 0; q < G; ++q) tot += shred[q][threadIdx.x];
  }
  if (threadIdx.x == 0) *counter = 0;
  // tables: tab[0 .. M*M) = S^T Y by slot (row s-slot, column y-slot), tab[M*M .. 2 M*M) = Y^T Y by slot;
  // coefficients written to tab[2 M*M ..): p (age order), q (age order), gamma.  Lane j < n works on row j.
  constexpr int M = kLbfgsMaxCompact;
  double* SY = tab;
  double* YY = tab + M * M;
  double* out = tab + 2 * M * M;
  const int n = h.n, sn = h.slot[n - 1], j = lane < n ? lane : n - 1;
  int sj = 0;
#pragma unroll
  for (int i = 0; i < M; ++i) sj = i == j ? h.slot[i] : sj;
  const double aj = __shfl_sync(0xffffffffu, tot, 4 * j), bj = __shfl_sync(0xffffffffu, tot, 4 * j + 1);
  const double cj = __shfl_sync(0xffffffffu, tot, 4 * j + 2), ej = __shfl_sync(0xffffffffu, tot, 4 * j + 3);
  if (lane < n) {
    SY[sj * M + sn] = cj;
    YY[sj * M + sn] = ej;
    YY[sn * M + sj] = ej;
  }
  __syncwarp();
  double sy[M], yy[M], syt[M];  // row j of S^T Y and Y^T Y, column j of S^T Y, in age order
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const bool in = i < n;
    const int si = h.slot[i];
    sy[i] = in ? SY[sj * M + si] : 0.0;
    syt[i] = in ? SY[si * M + sj] : 0.0;
    yy[i] = in ? YY[sj * M + si] : 0.0;
  }
  double djj = 0, dyy = 0;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    djj = i == j ? sy[i] : djj;
    dyy = i == j ? yy[i] : dyy;
  }
  const double inv = 1.0 / djj;
  const double gamma = __shfl_sync(0xffffffffu, djj / dyy, n - 1);
  // R q = a, R[j][k] = s_j.y_k (k >= j): the newest first, each solved value leaving the rows before it
  double r = aj, q = 0, t = -gamma * bj;
#pragma unroll
  for (int k = M - 1; k >= 0; --k) {
    if (k < n) {
      const double qk = __shfl_sync(0xffffffffu, r * inv, k);
      if (j == k) q = qk;
      if (j < k) r -= sy[k] * qk;
      t += gamma * yy[k] * qk;  // t = (D + gamma Y^T Y) q - gamma b, less the diagonal
    }
  }
  t += djj * q;
  double p = 0;  // R^T p = t, the oldest first
#pragma unroll
  for (int k = 0; k < M; ++k) {
    if (k < n) {
      const double pk = __shfl_sync(0xffffffffu, t * inv, k);
      if (j == k) p = pk;
      if (j > k) t -= syt[k] * pk;
    }
  }
  if (lane < n) {
    out[j] = p;
    out[M + j] = -gamma * q;
  }
  if (lane == 0) out[2 * M] = gamma;
}

// d = -(gamma g + sum_j p_j s_j + sum_j q'_j y_j) (coefficients from the multidot pass; gamma_host when
// h.n == 0), g . d and |d|^2 into the scalars.  L = 1: a thread per vertex; L = 4: four lanes a vertex, three of them a
// component each, for systems that leave FP64 units idle (a thread's 51 FP64 operations at m = 8, 64 cycles each for a
// warp, become 17): FP64, 9,225 vertices 10.9 -> 7.1 us.  The border is the multidot's
// (twice as many warps as that leave the units two rounds of a thread per vertex).
template <typename S, int L>
__global__ void __launch_bounds__(LB)
    lbfgs_combine_kernel(int nv, const double* __restrict__ g, LbfgsHist<S> h, const double* __restrict__ coef,
                         double gamma_host, V4<S>* __restrict__ d, Reduce red) {
  constexpr int M = kLbfgsMaxCompact;
  __shared__ double shred[LB / 32][2];
  __shared__ S cs[2 * M + 1];
  if (threadIdx.x < 2 * M + 1) {
    const int k = threadIdx.x;
    const bool used = k == 2 * M || (k < M ? k < h.n : k - M < h.n);
    cs[k] = used ? (S)(k == 2 * M && h.n == 0 ? gamma_host : coef[k]) : S(0);
  }
  __syncthreads();
  const int i = blockIdx.x * LB + threadIdx.x, u = i / L;
  S part[2] = {S(0), S(0)};
  if (u < nv) {
    const S gm = cs[2 * M];
    if constexpr (L == 1) {
      const V4<S> gv = mk4<S>((S)g[3 * u], (S)g[3 * u + 1], (S)g[3 * u + 2]);
      S x = gm * gv.x, y = gm * gv.y, z = gm * gv.z;
#pragma unroll
      for (int j = 0; j < M; ++j) {
        if (j < h.n) {
          const V4<S> sv = h.s[j][u], yv = h.y[j][u];
          const S a = cs[j], b = cs[M + j];
          x += a * sv.x + b * yv.x;
          y += a * sv.y + b * yv.y;
          z += a * sv.z + b * yv.z;
        }
      }
      const V4<S> dv = mk4<S>(-x, -y, -z);
      d[u] = dv;
      part[0] = dot3<S>(gv, dv);
      part[1] = dot3<S>(dv, dv);
    } else {
      const int q = i % L;
      const S gq = q < 3 ? (S)g[3 * (size_t)u + q] : S(0);
      S x = gm * gq;
      const size_t c = 4 * (size_t)u + q;
#pragma unroll
      for (int j = 0; j < M; ++j)
        if (j < h.n)
          x += cs[j] * reinterpret_cast<const S*>(h.s[j])[c] + cs[M + j] * reinterpret_cast<const S*>(h.y[j])[c];
      x = q < 3 ? -x : S(0);
      reinterpret_cast<S*>(d)[c] = x;
      part[0] = gq * x;
      part[1] = x * x;
    }
  }
  double v2[2];
  block_sum_s<2, LB, S>(part, v2, shred);
  double tot[2];
  if (grid_sum_last<2, LB>(v2, red.partials, red.counter, tot)) {
    red.sc->gd = tot[0];
    red.sc->dnorm2 = tot[1];
  }
}

}  // namespace

// 2 blocks per SM (each thread then sums several vertices in FP32 before the block sums); with four warps to 32 vertices
// where blocks of 64 vertices are no more than that
constexpr int kMultidotGroups = 4;
static void multidot_shape(int nv, int& grid, int& groups) {
  int dev = 0, nsm = 0;
  SSIM_CUDA(cudaGetDevice(&dev));
  SSIM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int most = 2 * std::max(nsm, 1), small = div_up(nv, LB / kMultidotGroups);
  groups = small <= most ? kMultidotGroups : 1;
  grid = groups == 1 ? std::max(1, std::min(div_up(nv, LB), most)) : std::max(1, small);
}

template <typename S>
void launch_lbfgs_multidot(int nv, const double* g, const LbfgsHist<S>& h, double* partials, double* tab,
                           unsigned int* counter, cudaStream_t st) {
  int grid, groups;
  multidot_shape(nv, grid, groups);
  if (groups == 1)
    lbfgs_multidot_kernel<S, 1><<<grid, LB, 0, st>>>(nv, g, h, partials, tab, counter);
  else
    lbfgs_multidot_kernel<S, kMultidotGroups><<<grid, LB, 0, st>>>(nv, g, h, partials, tab, counter);
  after_launch("lbfgs_multidot");
}

template <typename S>
void launch_lbfgs_combine(int nv, const double* g, const LbfgsHist<S>& h, const double* coef, double gamma_host,
                          V4<S>* d, const Reduce& red, cudaStream_t st) {
  int grid, groups;
  multidot_shape(nv, grid, groups);
  if (sizeof(S) == 8 && groups > 1)
    lbfgs_combine_kernel<S, 4><<<div_up(4LL * nv, LB), LB, 0, st>>>(nv, g, h, coef, gamma_host, d, red);
  else
    lbfgs_combine_kernel<S, 1><<<div_up(nv, LB), LB, 0, st>>>(nv, g, h, coef, gamma_host, d, red);
  after_launch("lbfgs_combine");
}

int lbfgs_multidot_partials(int nv) {
  int grid, groups;
  multidot_shape(nv, grid, groups);
  return grid * 4 * kLbfgsMaxCompact;
}

template <typename S>
void launch_lbfgs_pass(int nv, const V4<S>* vin, const double* g, V4<S>* vout, const V4<S>* w, const double* cA,
                       const double* cB, double csign, const double* scale_ptr, double scale, const V4<S>* a,
                       double rho, double* out, const Reduce& red, cudaStream_t st) {
  lbfgs_pass_kernel<S><<<div_up(nv, LB), LB, 0, st>>>(nv, vin, g, vout, w, cA, cB, csign, scale_ptr, scale, a, rho,
                                                      out, red);
  after_launch("lbfgs_pass");
}

template <typename S>
void launch_lbfgs_final(int nv, const V4<S>* z, const V4<S>* w, const double* cA, const double* cB, const double* g,
                        V4<S>* d, const Reduce& red, cudaStream_t st) {
  lbfgs_final_kernel<S><<<div_up(nv, LB), LB, 0, st>>>(nv, z, w, cA, cB, g, d, red);
  after_launch("lbfgs_final");
}

template <typename S>
void launch_lbfgs_pair(int nv, double alpha, const V4<S>* d, const double* gnew, const double* gold, V4<S>* sv,
                       V4<S>* yv, const Reduce& red, cudaStream_t st) {
  lbfgs_pair_kernel<S><<<div_up(nv, LB), LB, 0, st>>>(nv, alpha, d, gnew, gold, sv, yv, red);
  after_launch("lbfgs_pair");
}

template <typename S>
void launch_lbfgs_accept(int nv, double alpha, const V4<S>* d, double* u, const double* gnew, double* gold,
                         cudaStream_t st) {
  lbfgs_accept_kernel<S><<<div_up(nv, LB), LB, 0, st>>>(nv, alpha, d, u, gnew, gold);
  after_launch("lbfgs_accept");
}

#define SSIM_LBFGS_INST(S)                                                                                         \
  template void launch_lbfgs_multidot<S>(int, const double*, const LbfgsHist<S>&, double*, double*, unsigned int*, \
                                         cudaStream_t);                                                           \
  template void launch_lbfgs_combine<S>(int, const double*, const LbfgsHist<S>&, const double*, double, V4<S>*,   \
                                        const Reduce&, cudaStream_t);                                             \
  template void launch_lbfgs_pass<S>(int, const V4<S>*, const double*, V4<S>*, const V4<S>*, const double*,       \
                                     const double*, double, const double*, double, const V4<S>*, double, double*, \
                                     const Reduce&, cudaStream_t);                                                \
  template void launch_lbfgs_final<S>(int, const V4<S>*, const V4<S>*, const double*, const double*,             \
                                      const double*, V4<S>*, const Reduce&, cudaStream_t);                        \
  template void launch_lbfgs_pair<S>(int, double, const V4<S>*, const double*, const double*, V4<S>*, V4<S>*,     \
                                     const Reduce&, cudaStream_t);                                                \
  template void launch_lbfgs_accept<S>(int, double, const V4<S>*, double*, const double*, double*, cudaStream_t);

SSIM_LBFGS_INST(float)
SSIM_LBFGS_INST(double)

}  // namespace ssim_gb
