// Eigenpairs of the real symmetric tridiagonal T = tridiag(e, d, e).
//
// Eigenvalues (DSTEBZ, external/LAPACK/zheevx.f:490, range 'I'): one CTA of T
// threads per requested eigenvalue index, multisection on the Sturm count (2 T
// points per step, the interval shrinks 2 T + 1 times) from the Gershgorin
// interval; stop when the width is below max(abstol, pivmin,
// 2 ulp max(|lo|,|hi|)) exactly as DSTEBZ's bisection test.
//
// Eigenvectors (DSTEIN, zheevx.f:496): inverse iteration with the shifted
// tridiagonal factored by Gaussian elimination with partial pivoting, at
// most five iterations, growth test sqrt(0.1/n) plus two extra iterations,
// unit 2-norm with the largest component positive; pivots below eps ||T|| become
// that (a shift can meet an eigenvalue exactly beside couplings of 1e-170, whose
// reciprocals as pivots overflowed the vector).  Eigenvalues closer than
// CLUSTER_REL * ||T|| form a cluster: its shifts are separated by 10 ulp
// (DSTEIN's perturbation) and its vectors are Gram-Schmidt orthogonalised
// against the earlier members inside the iteration.  Residual loss of
// orthogonality between well-separated vectors is removed afterwards by a
// Cholesky-QR pass on the complex vectors (see solve.cu).
#include "handle.cuh"
#include "sturm.cuh"

#include <algorithm>
#include <cmath>

namespace {

constexpr double CLUSTER_REL = 1e-9;

// scal[0] = gl, [1] = gu, [2] = pivmin, [3] = tnorm; de[i] = (d[i], e[i-1]^2)
__global__ void k_tridiag_prep(int n, const double* d, const double* e, double2* de, double* scal) {
  __shared__ double s_lo[256], s_hi[256], s_e2[256], s_nrm[256];
  double lo = 1e300, hi = -1e300, em = 0.0, nm = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double ea = (i > 0) ? fabs(e[i - 1]) : 0.0;
    const double eb = (i < n - 1) ? fabs(e[i]) : 0.0;
    lo = fmin(lo, d[i] - ea - eb);
    hi = fmax(hi, d[i] + ea + eb);
    nm = fmax(nm, fabs(d[i]) + ea + eb);
    const double e2 = (i > 0) ? e[i - 1] * e[i - 1] : 0.0;
    de[i] = make_double2(d[i], e2);
    em = fmax(em, e2);
  }
  s_lo[threadIdx.x] = lo; s_hi[threadIdx.x] = hi; s_e2[threadIdx.x] = em; s_nrm[threadIdx.x] = nm;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      s_lo[threadIdx.x] = fmin(s_lo[threadIdx.x], s_lo[threadIdx.x + o]);
      s_hi[threadIdx.x] = fmax(s_hi[threadIdx.x], s_hi[threadIdx.x + o]);
      s_e2[threadIdx.x] = fmax(s_e2[threadIdx.x], s_e2[threadIdx.x + o]);
      s_nrm[threadIdx.x] = fmax(s_nrm[threadIdx.x], s_nrm[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double safemin = 2.2250738585072014e-308;
    const double ulp = 2.220446049250313e-16;
    const double pivmin = safemin * fmax(1.0, s_e2[0]);
    const double tnorm = fmax(fabs(s_lo[0]), fabs(s_hi[0]));
    const double fudge = 2.1;
    scal[0] = s_lo[0] - fudge * tnorm * ulp * n - fudge * 2.0 * pivmin;
    scal[1] = s_hi[0] + fudge * tnorm * ulp * n + fudge * 2.0 * pivmin;
    scal[2] = pivmin;
    scal[3] = s_nrm[0];
  }
}

// One CTA per eigenvalue index; its threads' points (tid and tid + T) are a step's.
__global__ void k_stebz(int n, const double2* de, const double* scal, int k, double abstol, double* w,
                        int* status) {
  __shared__ int s_first[2][32];
  const int j = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
  const double pivmin = scal[2];
  const double ulp = 2.220446049250313e-16;
  const double atol = abstol > 0.0 ? abstol : ulp * scal[3];
  const bool minors = scal[3] < 0x1p38;
  double lo = scal[0], hi = scal[1];
  bool conv = false;
  for (int it = 0; it < 200; ++it) {
    const double width = hi - lo;
    const double tol = fmax(fmax(atol, pivmin), 2.0 * ulp * fmax(fabs(lo), fabs(hi)));
    if (width <= tol) { conv = true; break; }
    const double step = width / (NPT * T + 1);
    double x[NPT];
    int cnt[NPT];
#pragma unroll
    for (int r = 0; r < NPT; ++r) x[r] = fmin(lo + (tid + r * T + 1) * step, hi);
    sturm_count(n, de, x, pivmin, minors, cnt);
    // the first point with at least j + 1 eigenvalues below it (NPT T: none)
    int mine = NPT * T;
#pragma unroll
    for (int r = NPT - 1; r >= 0; --r) {
      const unsigned ball = __ballot_sync(0xffffffffu, cnt[r] >= j + 1);
      if (ball) mine = r * T + 32 * warp + __ffs(ball) - 1;
    }
    if (lane == 0) s_first[it & 1][warp] = mine;
    __syncthreads();
    int f = NPT * T;
    for (int q = 0; q < T / 32; ++q) f = min(f, s_first[it & 1][q]);
    const double l0 = lo;
    if (f > 0) lo = fmin(l0 + f * step, hi);
    if (f < NPT * T) hi = fmin(l0 + (f + 1) * step, hi);
    if (!(hi > lo)) { conv = true; break; }
  }
  if (tid == 0) {
    w[j] = 0.5 * (lo + hi);
    if (!conv) atomicAdd(&status[ST_STEBZ], 1);
  }
}

// cluster starts: cl[j] = 1 if j starts a cluster
__global__ void k_clusters(int k, const double* w, const double* scal, int* cl) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= k) return;
  const double tol = CLUSTER_REL * fmax(scal[3], 1e-300);
  cl[j] = (j == 0) || (w[j] - w[j - 1] > tol);
}

__device__ __forceinline__ double urand(unsigned long long a, unsigned long long b) {
  unsigned long long z = a * 0x9E3779B97F4A7C15ull + b * 0xBF58476D1CE4E5B9ull + 0x94D049BB133111EBull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return ((double)(z >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0;
}

// One thread per cluster.  Work arrays are interleaved by eigenvalue index
// (element i of slot j at [i*k + j]) so that neighbouring threads touch
// neighbouring addresses.  Y (interleaved too) receives the vectors.  The
// factorisation stores the pivots' reciprocals, so the solves' dependency
// chains hold only multiply-adds; the loops are unrolled so that loads run
// ahead of the recurrences.
__global__ void k_stein(int n, const double* __restrict__ d, const double* __restrict__ e,
                        const double* __restrict__ scal, int k, const double* __restrict__ w,
                        const int* __restrict__ cl, double* __restrict__ ua, double* __restrict__ ub,
                        double* __restrict__ uf, double* __restrict__ um, double* __restrict__ Yi,
                        int* status) {
  const int j0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (j0 >= k || !cl[j0]) return;
  int j1 = j0 + 1;
  while (j1 < k && !cl[j1]) ++j1;
  const double eps = 1.1102230246251565e-16;
  const double tnorm = scal[3];
  const double dtpcrt = sqrt(0.1 / n);
  const double pert = fmax(eps * tnorm, 1e-300);
  double xprev = 0.0;
  for (int j = j0; j < j1; ++j) {
    double lam = w[j];
    if (j > j0) {
      const double pertol = 10.0 * fabs(eps * lam);
      if (lam - xprev < pertol) lam = xprev + pertol;
    }
    xprev = lam;
    // factor T - lam I (slot j); ua holds 1/pivot
    double a = d[0] - lam, b = (n > 1) ? e[0] : 0.0;
    double ulast = 0.0;
#pragma unroll 4
    for (int i = 0; i < n - 1; ++i) {
      const double c = e[i], dd = d[i + 1] - lam, ee = (i + 1 < n - 1) ? e[i + 1] : 0.0;
      const size_t o = (size_t)i * k + j;
      if (fabs(a) >= fabs(c)) {
        const double aa = (fabs(a) < pert) ? copysign(pert, a) : a;
        const double ra = 1.0 / aa;
        ua[o] = ra; ub[o] = b; uf[o] = 0.0;
        const double m = c * ra;
        um[o] = m;
        a = dd - m * b;
        b = ee;
      } else {
        const double rc = 1.0 / ((fabs(c) < pert) ? copysign(pert, c) : c);
        ua[o] = rc; ub[o] = dd; uf[o] = ee;
        const double m = a * rc;
        um[o] = -m - 2.0;  // encodes a swap (a multiplier |m| <= 1 never reaches below -1)
        a = b - m * dd;
        b = -m * ee;
      }
    }
    {
      const size_t o = (size_t)(n - 1) * k + j;
      const double aa = (fabs(a) < pert) ? copysign(pert, a) : a;
      ua[o] = 1.0 / aa;
      ub[o] = 0.0; uf[o] = 0.0; um[o] = 0.0;
      ulast = fabs(aa);
    }
    for (int i = 0; i < n; ++i) Yi[(size_t)i * k + j] = urand(j + 1, i + 1);
    int nrmchk = 0;
    bool conv = false;
    for (int its = 0; its < 5; ++its) {
      // scale the right-hand side: ||x||_1 = n ||T|| max(eps, |u_last|)
      double s1 = 0.0;
#pragma unroll 8
      for (int i = 0; i < n; ++i) s1 += fabs(Yi[(size_t)i * k + j]);
      const double scl = (s1 > 0.0) ? n * tnorm * fmax(eps, ulast) / s1 : 1.0;
      // forward elimination on the right-hand side
      double cur = Yi[j] * scl;
#pragma unroll 4
      for (int i = 0; i < n - 1; ++i) {
        const size_t o = (size_t)i * k + j;
        const double nx = Yi[o + k] * scl;
        const double m = um[o];
        if (m < -1.0) {  // swapped
          Yi[o] = nx;
          cur = cur + (m + 2.0) * nx;
        } else {
          Yi[o] = cur;
          cur = nx - m * cur;
        }
      }
      // back substitution with the stored reciprocals
      double x2 = 0.0, x1 = cur * ua[(size_t)(n - 1) * k + j];
      Yi[(size_t)(n - 1) * k + j] = x1;
      double nrm = fabs(x1);
#pragma unroll 4
      for (int i = n - 2; i >= 0; --i) {
        const size_t o = (size_t)i * k + j;
        const double x = (Yi[o] - ub[o] * x1 - uf[o] * x2) * ua[o];
        Yi[o] = x;
        nrm = fmax(nrm, fabs(x));
        x2 = x1;
        x1 = x;
      }
      // orthogonalise against the earlier members of the cluster
      if (j > j0) {
        for (int q = j0; q < j; ++q) {
          double dot = 0.0;
          for (int i = 0; i < n; ++i) dot += Yi[(size_t)i * k + q] * Yi[(size_t)i * k + j];
          for (int i = 0; i < n; ++i) Yi[(size_t)i * k + j] -= dot * Yi[(size_t)i * k + q];
        }
        nrm = 0.0;
        for (int i = 0; i < n; ++i) nrm = fmax(nrm, fabs(Yi[(size_t)i * k + j]));
      }
      if (!(nrm >= dtpcrt)) {
        if (nrm > 0.0 && nrm < 1e-200) {
          for (int i = 0; i < n; ++i) Yi[(size_t)i * k + j] *= 1e200;
        }
        continue;
      }
      ++nrmchk;
      if (nrmchk >= 3) { conv = true; break; }
    }
    if (!conv) atomicAdd(&status[ST_STEIN], 1);
    // normalise: unit 2-norm, largest component positive
    double s2 = 0.0, big = 0.0;
    int ib = 0;
    for (int i = 0; i < n; ++i) {
      const double v = Yi[(size_t)i * k + j];
      s2 += v * v;
      if (fabs(v) > big) { big = fabs(v); ib = i; }
    }
    double sc = (s2 > 0.0) ? 1.0 / sqrt(s2) : 0.0;
    if (Yi[(size_t)ib * k + j] < 0.0) sc = -sc;
    for (int i = 0; i < n; ++i) Yi[(size_t)i * k + j] *= sc;
  }
}

// The same inverse iteration with the factor and the working vector of one
// eigenvector in shared memory (40 n bytes): one warp per cluster, lane 0
// runs the recurrences (factorisation, forward elimination, back
// substitution) at shared-memory latency, the warp shares the element-wise
// passes.  The finished vectors go to Yi (interleaved as in k_stein) because
// later members of a cluster are orthogonalised against them.  The recurrences
// are what it takes its time for: SCH rows at a time are loaded before any of them
// is stored (a load does not pass a store that may alias it) and swaps are
// selections.  k = 200, n = 1964: 639 -> 394 us; k = 20, n = 316: 108 -> 69 us.
constexpr int SCH = 8;
constexpr size_t STEIN_SMEM = 200 * 1024;  // most dynamic shared memory (order 5120)
__global__ void __launch_bounds__(32) k_stein_smem(int n, const double* __restrict__ d,
                                                   const double* __restrict__ e,
                                                   const double* __restrict__ scal, int k,
                                                   const double* __restrict__ w,
                                                   const int* __restrict__ cl, double* Yi,
                                                   int* status) {
  extern __shared__ double sm[];
  double* ra = sm;          // 1 / pivot
  double* rb = ra + n;      // first superdiagonal of U
  double* rf = rb + n;      // second superdiagonal (fill-in from swaps)
  double* rm = rf + n;      // multiplier (swap encoded as -m-2)
  double* y = rm + n;       // working vector
  const int j0 = blockIdx.x;
  const int lane = threadIdx.x;
  if (!cl[j0]) return;
  int j1 = j0 + 1;
  while (j1 < k && !cl[j1]) ++j1;
  const double eps = 1.1102230246251565e-16;
  const double tnorm = scal[3];
  const double dtpcrt = sqrt(0.1 / n);
  const double pert = fmax(eps * tnorm, 1e-300);
  double xprev = 0.0;
  for (int j = j0; j < j1; ++j) {
    double lam = w[j];
    if (j > j0) {
      const double pertol = 10.0 * fabs(eps * lam);
      if (lam - xprev < pertol) lam = xprev + pertol;
    }
    xprev = lam;
    __shared__ double s_ulast;
    if (lane == 0) {
      double a = d[0] - lam, b = (n > 1) ? e[0] : 0.0;
      auto row = [&](int i, double c, double dd, double ee) {
        const bool sw = !(fabs(a) >= fabs(c));
        double piv = sw ? c : a;
        if (fabs(piv) < pert) piv = copysign(pert, piv);
        const double r = 1.0 / piv, m = (sw ? a : c) * r;
        ra[i] = r;
        rb[i] = sw ? dd : b;
        rf[i] = sw ? ee : 0.0;
        rm[i] = sw ? -m - 2.0 : m;
        a = (sw ? b : dd) - m * (sw ? dd : b);
        b = sw ? -m * ee : ee;
      };
      int i = 0;
      for (; i + SCH < n - 1; i += SCH) {
        double ev[SCH + 1], dv[SCH];
#pragma unroll
        for (int u = 0; u < SCH; ++u) { ev[u] = e[i + u]; dv[u] = d[i + u + 1] - lam; }
        ev[SCH] = e[i + SCH];
#pragma unroll
        for (int u = 0; u < SCH; ++u) row(i + u, ev[u], dv[u], ev[u + 1]);
      }
      for (; i < n - 1; ++i) row(i, e[i], d[i + 1] - lam, (i + 1 < n - 1) ? e[i + 1] : 0.0);
      const double aa = (fabs(a) < pert) ? copysign(pert, a) : a;
      ra[n - 1] = 1.0 / aa;
      rb[n - 1] = 0.0; rf[n - 1] = 0.0; rm[n - 1] = 0.0;
      s_ulast = fabs(aa);
    }
    for (int i = lane; i < n; i += 32) y[i] = urand(j + 1, i + 1);
    __syncwarp();
    const double ulast = s_ulast;
    int nrmchk = 0;
    bool conv = false;
    for (int its = 0; its < 5; ++its) {
      double s1 = 0.0;
      for (int i = lane; i < n; i += 32) s1 += fabs(y[i]);
      for (int o = 16; o > 0; o >>= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      const double scl = (s1 > 0.0) ? n * tnorm * fmax(eps, ulast) / s1 : 1.0;
      if (lane == 0) {
        // forward elimination; a swapped row keeps the next entry and goes on with
        // cur + (m + 2) next, the others keep cur and go on with next - m cur
        double cur = y[0] * scl;
        auto fwd = [&](double m, double nx) {
          const bool sw = m < -1.0;
          const double kept = sw ? nx : cur;
          cur = fma(sw ? m + 2.0 : -m, kept, sw ? cur : nx);
          return kept;
        };
        int i = 0;
        for (; i + SCH <= n - 1; i += SCH) {
          double mv[SCH], yv[SCH];
#pragma unroll
          for (int u = 0; u < SCH; ++u) { mv[u] = rm[i + u]; yv[u] = y[i + u + 1] * scl; }
#pragma unroll
          for (int u = 0; u < SCH; ++u) y[i + u] = fwd(mv[u], yv[u]);
        }
        for (; i < n - 1; ++i) y[i] = fwd(rm[i], y[i + 1] * scl);
        // back substitution: the reciprocal pivot goes into the factors first, so a
        // row adds one multiply-add to the chain
        double x2 = 0.0, x1 = cur * ra[n - 1];
        y[n - 1] = x1;
        auto bwd = [&](double p, double b, double f, double c) {
          const double x = fma(-(b * p), x1, fma(-(f * p), x2, c * p));
          x2 = x1;
          x1 = x;
          return x;
        };
        i = n - 2;
        for (; i - SCH + 1 >= 0; i -= SCH) {
          double pv[SCH], bv[SCH], fv[SCH], yv[SCH];
#pragma unroll
          for (int u = 0; u < SCH; ++u) {
            pv[u] = ra[i - u]; bv[u] = rb[i - u]; fv[u] = rf[i - u]; yv[u] = y[i - u];
          }
#pragma unroll
          for (int u = 0; u < SCH; ++u) y[i - u] = bwd(pv[u], bv[u], fv[u], yv[u]);
        }
        for (; i >= 0; --i) y[i] = bwd(ra[i], rb[i], rf[i], y[i]);
      }
      __syncwarp();
      for (int q = j0; q < j; ++q) {
        double dot = 0.0;
        for (int i = lane; i < n; i += 32) dot += Yi[(size_t)i * k + q] * y[i];
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        for (int i = lane; i < n; i += 32) y[i] -= dot * Yi[(size_t)i * k + q];
        __syncwarp();
      }
      double nrm = 0.0;
      for (int i = lane; i < n; i += 32) nrm = fmax(nrm, fabs(y[i]));
      for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
      if (!(nrm >= dtpcrt)) {
        if (nrm > 0.0 && nrm < 1e-200)
          for (int i = lane; i < n; i += 32) y[i] *= 1e200;
        __syncwarp();
        continue;
      }
      ++nrmchk;
      if (nrmchk >= 3) { conv = true; break; }
    }
    if (!conv && lane == 0) atomicAdd(&status[ST_STEIN], 1);
    // normalise: unit 2-norm, largest component positive (lowest index on ties)
    double s2 = 0.0, big = -1.0;
    int ib = 0;
    for (int i = lane; i < n; i += 32) {
      const double v = y[i];
      s2 += v * v;
      if (fabs(v) > big) { big = fabs(v); ib = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      const double ob = __shfl_xor_sync(0xffffffffu, big, o);
      const int oi = __shfl_xor_sync(0xffffffffu, ib, o);
      if (ob > big || (ob == big && oi < ib)) { big = ob; ib = oi; }
    }
    double sc = (s2 > 0.0) ? 1.0 / sqrt(s2) : 0.0;
    if (y[ib] < 0.0) sc = -sc;
    for (int i = lane; i < n; i += 32) Yi[(size_t)i * k + j] = y[i] * sc;
    __syncwarp();
  }
}

// Z(i, j) = Yi[i*k + j] (interleaved real -> column-major complex, ld ldz)
__global__ void k_y_to_z(int n, int k, const double* Yi, cplx* Z, long long ldz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= n || j >= k) return;
  Z[i + ldz * j] = cmk(Yi[(size_t)i * k + j], 0.0);
}

}  // namespace

// Lowest k eigenvalues into w, eigenvectors as complex columns of Z (n x k).
// scratch: de (2n), scal (8), 4*n*k doubles for the factors, n*k for Yi; 16-byte aligned.
int tridiag_eig(excfv_handle* h, int n, int k, double abstol, const double* d, const double* e,
                double* w, cplx* Z, long long ldz, double* scratch, int* iscratch) {
  cudaStream_t s = h->stream;
  double2* de = reinterpret_cast<double2*>(scratch);
  double* scal = scratch + 2 * (size_t)n;
  double* ua = scal + 8;
  double* ub = ua + (size_t)n * k;
  double* uf = ub + (size_t)n * k;
  double* um = uf + (size_t)n * k;
  double* Yi = um + (size_t)n * k;
  k_tridiag_prep<<<1, 256, 0, s>>>(n, d, e, de, scal); count_launch();
  CUDA_TRY(cudaGetLastError());
  // Threads per eigenvalue: a pass narrows the interval 2 T + 1 times and takes n
  // times the larger of one warp's latency, about 22 clocks, and 16 issue slots per
  // warp of an SM quarter (two points of three double-precision operations of two
  // slots each, signs and loads); the T with the shortest product of passes (for 50
  // bits) and step.
  const int sms = (h->grid_ctas > 0) ? h->grid_ctas : h->nsm;
  int T = 32;
  double best = 1e300;
  for (int t = 32; t <= 256; t *= 2) {
    const double warps = (double)((k + sms - 1) / sms) * t / 128.0;
    const double est = std::ceil(50.0 / std::log2(NPT * t + 1.0)) * std::max(22.0, 16.0 * warps);
    if (est < best) { best = est; T = t; }
  }
  k_stebz<<<k, T, 0, s>>>(n, de, scal, k, abstol, w, h->ws.status); count_launch();
  CUDA_TRY(cudaGetLastError());
  k_clusters<<<(k + 127) / 128, 128, 0, s>>>(k, w, scal, iscratch); count_launch();
  CUDA_TRY(cudaGetLastError());
  const size_t sbytes = 40 * (size_t)n;
  if (sbytes <= STEIN_SMEM) {
    CUDA_TRY(raise_smem_limit(k_stein_smem, STEIN_SMEM));
    k_stein_smem<<<k, 32, sbytes, s>>>(n, d, e, scal, k, w, iscratch, Yi, h->ws.status); count_launch();
  } else {
    k_stein<<<(k + 31) / 32, 32, 0, s>>>(n, d, e, scal, k, w, iscratch, ua, ub, uf, um, Yi,
                                         h->ws.status); count_launch();
  }
  CUDA_TRY(cudaGetLastError());
  k_y_to_z<<<dim3((n + 255) / 256, k), 256, 0, s>>>(n, k, Yi, Z, ldz); count_launch();
  CUDA_TRY(cudaGetLastError());
  return EXCFV_OK;
}

size_t tridiag_eig_scratch_doubles(int n, int k) { return 2 * (size_t)n + 8 + 5 * (size_t)n * k; }
