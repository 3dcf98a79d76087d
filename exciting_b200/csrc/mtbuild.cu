// The per-SCF-iteration muffin-tin Hamiltonian and radial overlaps on the
// device: hmlint = mt_kin + mt_pot (src/src_eigensystem/hmlint.f90:14-58,
// mt_kin.f90:64-230, mt_pot.f90:131-311) and olprad (olprad.f90:30-143),
// written straight into the handle's aa / loa / lolo / oalo / ololo / h1aa.
//
// Every radial integral of the reference is the spline integral of
// fderiv(-1) (src/src_lib/fderiv.f90 with spline.f90) over the species'
// mesh, a linear functional of the integrand: integral = sum_r w_r f(r), with
// weights w fixed by the mesh (the transpose of the spline rule, one
// tridiagonal solve per species on the host).  So the build is
//   radial integrals   of the potential: one thread per integral, a weighted
//                      sum over r of products of radial functions with r^2
//                      and the potential's lm; the few kinetic and overlap
//                      integrals (with the ZORA factor 1/(1 - a V_00 y00)):
//                      one warp per integral;
//   Gaunt contraction  one thread per matrix element: aa(f1, f3) = kinetic
//                      (same lm) + sum_lm2 gntyry(lm1, lm2, lm3) haa(lm2),
//                      the same for loa and lolo.
// The Gaunt coefficient gntyry(lm1, lm2, lm3) = integral of conj(Y_lm1) R_lm2
// Y_lm3 (R the real harmonics, lm2 up to lmaxvr) comes from Gauss-Legendre
// quadrature in cos(theta) of the Y_lm of specfun.cuh at phi = 0 (the phi
// integral is 2 pi delta(m1 = m2 + m3)); the nodes by Newton's method on the
// Legendre recurrence.  It vanishes unless |m2| = |m1 - m3|, so the table
// holds one real number per (lm1, lm3, l2), and the contraction runs over l2.
//
// What the build costs (8 atoms, lmaxmat 10, lmaxvr 8, 300 mesh points, host
// copies of the blocks wanted): the full complex table formed on the host and
// uploaded (19 MB) took 30 of the call's 38 ms; formed on the device in its
// compact form (1 MB) it takes 7.6 us.  The call now takes 1.6 ms, most of it
// the copy of the blocks (7.5 MB) into pageable host memory; of its 0.2 ms of
// kernels the potential integrals are 0.16 ms.
#include <cmath>
#include <vector>

#include "handle.cuh"
#include "specfun.cuh"

namespace {

constexpr double Y00C = 0.28209479177387814347;
constexpr double ALPHA_FS = 1.0 / 137.03599911;

// ---- host: spline integral weights -------------------------------------
// The integral of fderiv(-1) over the whole mesh for one integrand f: the
// spline coefficients by the recurrences of spline.f90, then the sum of the
// per-interval cubic integrals.
double spline_integral(int n, const double* x, const double* f, std::vector<double>& c1,
                       std::vector<double>& c2, std::vector<double>& c3, std::vector<double>& w) {
  for (int i = 0; i < n - 1; ++i) {
    w[i] = 1.0 / (x[i + 1] - x[i]);
    c1[i] = w[i] * (f[i + 1] - f[i]);
  }
  c2[0] = 1.0;
  c3[0] = (c1[1] - c1[0]) / (x[2] - x[0]);
  double t1 = (x[1] - x[0]) * w[1];
  double t2 = t1 * c2[0];
  double t3 = 1.0 / (2.0 * (t1 + 1.0));
  c2[1] = t3;
  double t4 = 3.0 * (c1[1] - c1[0]) * w[1] - t2 * c3[0];
  c3[1] = t4;
  for (int i = 2; i < n - 1; ++i) {
    t1 = (x[i] - x[i - 1]) * w[i];
    t2 = t1 * t3;
    t3 = 1.0 / (2.0 * t1 + 2.0 - t2);
    c2[i] = t3;
    t4 = 3.0 * (c1[i] - c1[i - 1]) * w[i] - t2 * t4;
    c3[i] = t4;
  }
  c2[n - 1] = 1.0;
  t1 = (c1[n - 2] - c1[n - 3]) / (x[n - 1] - x[n - 3]);
  c3[n - 1] = t1;
  for (int i = n - 2; i >= 1; --i) {
    t1 = c3[i] - t1 * c2[i + 1];
    c3[i] = t1;
  }
  for (int i = 0; i < n; ++i) c2[i] *= c3[i];
  double g = 0.0;
  for (int i = 0; i < n - 1; ++i) {
    const double d3 = (1.0 / 3.0) * (c2[i + 1] - c2[i]) * w[i];
    const double dx = x[i + 1] - x[i];
    const double d1 = c1[i] - (c2[i] + d3 * dx) * dx;
    g += (((0.25 * d3 * dx + (1.0 / 3.0) * c2[i]) * dx + 0.5 * d1) * dx + f[i]) * dx;
  }
  return g;
}

// Weights w_j with integral(f) = sum_j w_j f_j: the transpose of the rule
// above.  The integral is the trapezoidal sum minus sum_i h_i^3 (c_i +
// c_{i+1}) / 12, with the second coefficients c from a tridiagonal system
//   h_{i-1}/h_i c_{i-1} + 2 (h_{i-1}/h_i + 1) c_i + c_{i+1} = 3 (s_i - s_{i-1}) / h_i
// (s_i the divided differences) between end values from the first and last
// three points; so w = trapezoid - B^T M^-T v / 12, one solve with M^T.
void spline_weights(int n, const double* x, double* wout) {
  std::vector<double> h(n), v(n, 0.0), g(n), cp(n), y(n);
  for (int i = 0; i < n; ++i) wout[i] = 0.0;
  for (int i = 0; i < n - 1; ++i) {
    h[i] = x[i + 1] - x[i];
    wout[i] += 0.5 * h[i];
    wout[i + 1] += 0.5 * h[i];
    const double q = h[i] * h[i] * h[i] / 12.0;
    v[i] += q;
    v[i + 1] += q;
  }
  // M^T y = v: row j of M^T holds M(j-1, j), M(j, j), M(j+1, j); rows 0 and
  // n-1 of M are unit rows, so y_1 .. y_{n-2} solve the inner system alone
  auto sub = [&](int i) { return h[i - 1] / h[i]; };                       // M(i, i-1)
  auto dia = [&](int i) { return 2.0 * (h[i - 1] / h[i] + 1.0); };         // M(i, i)
  for (int j = 1; j <= n - 2; ++j) {
    const double lo = (j > 1) ? 1.0 : 0.0;                                  // M(j-1, j)
    const double up = (j < n - 2) ? sub(j + 1) : 0.0;                       // M(j+1, j)
    const double m = dia(j) - (j > 1 ? lo * cp[j - 1] : 0.0);
    cp[j] = up / m;
    g[j] = (v[j] - (j > 1 ? lo * g[j - 1] : 0.0)) / m;
  }
  for (int j = n - 2; j >= 1; --j) y[j] = g[j] - (j < n - 2 ? cp[j] * y[j + 1] : 0.0);
  y[0] = v[0] - sub(1) * y[1];
  y[n - 1] = v[n - 1] - y[n - 2];
  // w -= B^T y, row by row of the right-hand side
  auto slope = [&](int i, double c) {  // c times the divided difference s_i
    wout[i] -= -c / h[i];
    wout[i + 1] -= c / h[i];
  };
  const double e0 = y[0] / (x[2] - x[0]), e1 = y[n - 1] / (x[n - 1] - x[n - 3]);
  slope(1, e0);
  slope(0, -e0);
  slope(n - 2, e1);
  slope(n - 3, -e1);
  for (int i = 1; i <= n - 2; ++i) {
    const double c = 3.0 * y[i] / h[i];
    slope(i, c);
    slope(i - 1, -c);
  }
}

// ---- host: Gaunt table ---------------------------------------------------
void gauss_legendre(int n, std::vector<double>& xq, std::vector<double>& wq) {
  xq.assign(n, 0.0);
  wq.assign(n, 0.0);
  for (int i = 0; i < n; ++i) {
    double z = cos(M_PI * (i + 0.75) / (n + 0.5));
    for (int it = 0; it < 100; ++it) {
      double p0 = 1.0, p1 = z;
      for (int k = 2; k <= n; ++k) {
        const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      const double dp = n * (z * p1 - p0) / (z * z - 1.0);
      const double dz = p1 / dp;
      z -= dz;
      if (fabs(dz) < 1e-16) {
        xq[i] = z;
        wq[i] = 2.0 / ((1.0 - z * z) * dp * dp);
        break;
      }
      xq[i] = z;
      wq[i] = 2.0 / ((1.0 - z * z) * dp * dp);
    }
  }
}

// Quadrature nodes of the Gaunt coefficients for l1, l3 <= lg: weights times 2 pi,
// then Y_lm (real at phi = 0) of every node, lm up to max(lg, lmaxvr).
int gaunt_nodes(int lg, int lmaxvr) { return (2 * lg + lmaxvr) / 2 + 2; }
void gaunt_node_values(int lg, int lmaxvr, double* out) {
  const int L = std::max(lg, lmaxvr), lmL = (L + 1) * (L + 1);
  const int nq = gaunt_nodes(lg, lmaxvr);
  std::vector<double> xq, wq;
  gauss_legendre(nq, xq, wq);
  std::vector<cplx> y(lmL);
  for (int q = 0; q < nq; ++q) {
    sf_ylm(L, acos(xq[q]), 0.0, y.data(), 1);
    out[q] = wq[q];
    for (int lm = 0; lm < lmL; ++lm) out[nq + (size_t)q * lmL + lm] = y[lm].x;
  }
}

// ---- device ------------------------------------------------------------------
struct MtArgs {
  int natmtot, lmaxmat, lmaxapw, apwordmax, nlomax, lmvr, nrmtmax, maxaa, maxnlo;
  const int* idxis;     // (natmtot)
  const int* nrmt;      // (nspecies)
  const int* apword;    // (lmaxapw+1, nspecies)
  const int* nlorb;     // (nspecies)
  const int* lorbl;     // (nspecies, nlomax): species fastest
  const double* wts;    // (nrmtmax, nspecies) spline-integral weights times r^2
  const double* spr;    // (nrmtmax, nspecies)
  const double* apwfr;  // (nrmtmax, 2, apwordmax, lmaxapw+1, natmtot)
  const double* lofr;   // (nrmtmax, 2, nlomax, natmtot)
  const double* veff;   // (lmvr, nrmtmax, natmtot)
  double a;             // ZORA: alpha^2 / 2 (0 without valence relativity)
  int lmaxvr, nspecies;
  int lg;               // largest l of the APWs and local orbitals
  const double* gnt;    // (lmaxvr+1, (lg+1)^2, (lg+1)^2): integral conj(Y_lm1) Y_(l2, m1-m3) Y_lm3
};

__device__ __forceinline__ int l_of(int lm) {
  int l = (int)sqrtf((float)lm);
  while ((l + 1) * (l + 1) <= lm) ++l;
  while (l * l > lm) --l;
  return l;
}

// gnt(l2, lm3, lm1) from the quadrature nodes y (gaunt_node_values), one
// thread per entry; exact zeros by the triangle rule and parity
__global__ void k_gaunt(int lg, int lmaxvr, int nq, const double* __restrict__ y, double* __restrict__ gnt) {
  const int lmg = (lg + 1) * (lg + 1);
  const int L = max(lg, lmaxvr), lmL = (L + 1) * (L + 1);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)lmg * lmg * (lmaxvr + 1)) return;
  const int l2 = (int)(t % (lmaxvr + 1));
  const int lm3 = (int)((t / (lmaxvr + 1)) % lmg);
  const int lm1 = (int)(t / ((long long)(lmaxvr + 1) * lmg));
  const int l1 = l_of(lm1), l3 = l_of(lm3);
  const int m2 = (lm1 - l1 * (l1 + 1)) - (lm3 - l3 * (l3 + 1));
  double s = 0.0;
  if (abs(m2) <= l2 && !((l1 + l2 + l3) & 1) && l1 <= l2 + l3 && l2 <= l1 + l3 && l3 <= l1 + l2) {
    const int lm2 = l2 * (l2 + 1) + m2;
    for (int q = 0; q < nq; ++q) {
      const double* yq = y + nq + (size_t)q * lmL;
      s += y[q] * yq[lm1] * yq[lm2] * yq[lm3];
    }
    s *= 2.0 * M_PI;
  }
  gnt[t] = s;
}

// sum_lm2 gntyry(lm1, lm2, lm3) h(lm2).  With M = m1 - m3 and G = gnt(l2) only
// m2 = M, -M contribute: R_lm2 = (Y_lm2 + (-1)^m Y_l2,-m2)/sqrt 2 for m2 > 0,
// -i (Y_lm2 - (-1)^m Y_l2,-m2)/sqrt 2 for m2 < 0, Y_l2,0 for m2 = 0.
__device__ __forceinline__ cplx gaunt_sum(const MtArgs& m, int lm1, int l1, int lm3, int l3, const double* h) {
  const int lmg = (m.lg + 1) * (m.lg + 1);
  const int M = (lm1 - l1 * (l1 + 1)) - (lm3 - l3 * (l3 + 1)), am = abs(M);
  const double* g = m.gnt + ((size_t)lm1 * lmg + lm3) * (m.lmaxvr + 1);
  const double sg = (am & 1) ? -1.0 : 1.0, sh = sqrt(0.5);
  const double fx = (M > 0) ? sh : sh * sg;      // factor of h(l2, |M|)
  const double fy = (M > 0) ? sh * sg : -sh;     // factor of i h(l2, -|M|)
  cplx s = cmk(0.0, 0.0);
  int l2 = max(abs(l1 - l3), am);
  if ((l1 + l2 + l3) & 1) ++l2;
  for (; l2 <= min(m.lmaxvr, l1 + l3); l2 += 2) {
    const double G = g[l2];
    const int c = l2 * (l2 + 1);
    if (M == 0) {
      s.x += G * h[c];
    } else {
      s.x += fx * G * h[c + am];
      s.y += fy * G * h[c - am];
    }
  }
  return s;
}

__device__ __forceinline__ const double* apw(const MtArgs& m, int ias, int d, int io, int l) {
  return m.apwfr + (size_t)m.nrmtmax * (d + 2 * (io + (size_t)m.apwordmax * (l + (size_t)(m.lmaxapw + 1) * ias)));
}
__device__ __forceinline__ const double* lof(const MtArgs& m, int ias, int d, int ilo) {
  return m.lofr + (size_t)m.nrmtmax * (d + 2 * (ilo + (size_t)m.nlomax * ias));
}

// potential integrals sum_r w_r r^2 p1(r) p2(r) V_lm2(r), the three kinds in
// one launch (each alone leaves most SMs idle)
//   kind 0: (l1, io1, l3, io2, lm2) of two APWs
//   kind 1: (ilo, l3, io, lm2) of an LO and an APW
//   kind 2: (ilo1, ilo2, lm2) of two LOs
__global__ void k_mt_potint(MtArgs m, int per0, int per1, int per2, double* out0, double* out1, double* out2) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n0 = (long long)per0 * m.natmtot, n1 = (long long)per1 * m.natmtot,
                  n2 = (long long)per2 * m.natmtot;
  int kind = 0, per_atom = per0;
  double* out = out0;
  if (t >= n0) {
    t -= n0;
    kind = 1; per_atom = per1; out = out1;
    if (t >= n1) {
      t -= n1;
      kind = 2; per_atom = per2; out = out2;
      if (t >= n2) return;
    }
  }
  const int ias = (int)(t / per_atom);
  int q = (int)(t % per_atom);
  const int is = m.idxis[ias];
  const int lm2 = q % m.lmvr;
  q /= m.lmvr;
  const double *p1 = nullptr, *p2 = nullptr;
  const int L1 = m.lmaxmat + 1;
  if (kind == 0) {
    const int io2 = q % m.apwordmax; q /= m.apwordmax;
    const int l3 = q % L1; q /= L1;
    const int io1 = q % m.apwordmax; q /= m.apwordmax;
    const int l1 = q;
    if (io1 >= m.apword[l1 + (m.lmaxapw + 1) * is] || io2 >= m.apword[l3 + (m.lmaxapw + 1) * is]) {
      out[t] = 0.0;
      return;
    }
    p1 = apw(m, ias, 0, io1, l1);
    p2 = apw(m, ias, 0, io2, l3);
  } else if (kind == 1) {
    const int io = q % m.apwordmax; q /= m.apwordmax;
    const int l3 = q % L1; q /= L1;
    const int ilo = q;
    if (ilo >= m.nlorb[is] || io >= m.apword[l3 + (m.lmaxapw + 1) * is]) {
      out[t] = 0.0;
      return;
    }
    p1 = lof(m, ias, 0, ilo);
    p2 = apw(m, ias, 0, io, l3);
  } else {
    const int ilo2 = q % m.nlomax;
    const int ilo1 = q / m.nlomax;
    if (ilo1 >= m.nlorb[is] || ilo2 >= m.nlorb[is]) {
      out[t] = 0.0;
      return;
    }
    p1 = lof(m, ias, 0, ilo1);
    p2 = lof(m, ias, 0, ilo2);
  }
  const int nr = m.nrmt[is];
  const double* w = m.wts + (size_t)m.nrmtmax * is;
  const double* v = m.veff + (size_t)m.lmvr * m.nrmtmax * ias + lm2;
  double s = 0.0;
#pragma unroll 4
  for (int r = 0; r < nr; ++r) s += w[r] * p1[r] * p2[r] * v[(size_t)m.lmvr * r];
  out[t] = s;
}

// kinetic-type integrals sum_r w_r r^2 (1/2 p1' p2' f + 1/2 l(l+1) p1 p2 f / r^2),
// f = rm (kinetic, mode 0) or a rm^2 (IORA* h1, mode 1), rm = 1/(1 - a V_00 y00)
//   kind 0: (l, io1, io2); kind 1: (ilo, io) with l = lorbl(ilo); kind 2: (ilo1, ilo2), equal l
// and the plain overlaps sum_r w_r r^2 p1 p2 (mode 2; kinds 1 and 2).
// All the wanted (kind, mode) sets in one launch, a warp per integral: there
// are only a few hundred of each, so with a thread per integral the launches
// took 104 us apiece, a serial loop over the mesh with a division in it.
struct RadSet {
  int kind, mode, per_atom;
  double* out;
};
struct RadSets {
  int n;
  RadSet s[8];
};
__global__ void k_mt_radint(MtArgs m, RadSets sets) {
  long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  int q0 = 0;
  while (q0 < sets.n && t >= (long long)sets.s[q0].per_atom * m.natmtot) {
    t -= (long long)sets.s[q0].per_atom * m.natmtot;
    ++q0;
  }
  if (q0 == sets.n) return;
  const int kind = sets.s[q0].kind, mode = sets.s[q0].mode, per_atom = sets.s[q0].per_atom;
  double* out = sets.s[q0].out;
  const int ias = (int)(t / per_atom);
  int q = (int)(t % per_atom);
  const int is = m.idxis[ias];
  const int L1 = m.lmaxmat + 1;
  const double *p1 = nullptr, *d1 = nullptr, *p2 = nullptr, *d2 = nullptr;
  int l = 0;
  if (kind == 0) {
    const int io2 = q % m.apwordmax; q /= m.apwordmax;
    const int io1 = q % m.apwordmax;
    l = q / m.apwordmax;
    if (l >= L1 || io1 >= m.apword[l + (m.lmaxapw + 1) * is] || io2 >= m.apword[l + (m.lmaxapw + 1) * is]) {
      out[t] = 0.0;
      return;
    }
    p1 = apw(m, ias, 0, io1, l); d1 = apw(m, ias, 1, io1, l);
    p2 = apw(m, ias, 0, io2, l); d2 = apw(m, ias, 1, io2, l);
  } else if (kind == 1) {
    const int io = q % m.apwordmax;
    const int ilo = q / m.apwordmax;
    if (ilo >= m.nlorb[is]) { out[t] = 0.0; return; }
    l = m.lorbl[is + m.nspecies * ilo];
    if (l > m.lmaxapw || io >= m.apword[l + (m.lmaxapw + 1) * is]) { out[t] = 0.0; return; }
    p1 = apw(m, ias, 0, io, l); d1 = apw(m, ias, 1, io, l);
    p2 = lof(m, ias, 0, ilo); d2 = lof(m, ias, 1, ilo);
  } else {
    const int ilo2 = q % m.nlomax;
    const int ilo1 = q / m.nlomax;
    if (ilo1 >= m.nlorb[is] || ilo2 >= m.nlorb[is]) { out[t] = 0.0; return; }
    l = m.lorbl[is + m.nspecies * ilo1];
    if (m.lorbl[is + m.nspecies * ilo2] != l) { out[t] = 0.0; return; }
    p1 = lof(m, ias, 0, ilo1); d1 = lof(m, ias, 1, ilo1);
    p2 = lof(m, ias, 0, ilo2); d2 = lof(m, ias, 1, ilo2);
  }
  const int nr = m.nrmt[is];
  const double* w = m.wts + (size_t)m.nrmtmax * is;
  const double* r_ = m.spr + (size_t)m.nrmtmax * is;
  const double* v00 = m.veff + (size_t)m.lmvr * m.nrmtmax * ias;
  const double ll = (double)l * (l + 1);
  double s = 0.0;
  for (int r = lane; r < nr; r += 32) {
    if (mode == 2) {
      s += w[r] * p1[r] * p2[r];
      continue;
    }
    const double rm = 1.0 / (1.0 - m.a * v00[(size_t)m.lmvr * r] * Y00C);
    const double f = (mode == 0) ? rm : m.a * rm * rm;
    const double rr = r_[r];
    s += w[r] * (0.5 * d1[r] * d2[r] * f + 0.5 * ll * p1[r] * p2[r] * f / (rr * rr));
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[t] = s;
}

// aa(f1, f3, ias) = kinetic (same lm) + sum_lm2 gnt(lm1, lm2, lm3) haa(l1, io1, l3, io2, lm2)
__global__ void k_mt_aa(MtArgs m, const int* flist, const double* haa, const double* kaa, cplx* aa) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)m.maxaa * m.maxaa * m.natmtot) return;
  const int f1 = (int)(t % m.maxaa);
  const int f3 = (int)((t / m.maxaa) % m.maxaa);
  const int ias = (int)(t / ((long long)m.maxaa * m.maxaa));
  const int is = m.idxis[ias];
  const int c1 = flist[f1 + m.maxaa * is], c3 = flist[f3 + m.maxaa * is];
  if (c1 < 0 || c3 < 0) { aa[t] = cmk(0.0, 0.0); return; }
  const int lm1 = c1 / m.apwordmax, io1 = c1 % m.apwordmax;
  const int lm3 = c3 / m.apwordmax, io2 = c3 % m.apwordmax;
  const int l1 = l_of(lm1), l3 = l_of(lm3);
  const int L1 = m.lmaxmat + 1;
  double kin = 0.0;
  if (lm1 == lm3 && kaa) kin = kaa[((size_t)ias * L1 + l1) * m.apwordmax * m.apwordmax + io1 * m.apwordmax + io2];
  const double* h = haa + ((((size_t)ias * L1 + l1) * m.apwordmax + io1) * L1 + l3) * m.apwordmax * m.lmvr +
                    (size_t)io2 * m.lmvr;
  cplx s = gaunt_sum(m, lm1, l1, lm3, l3, h);
  s.x += kin;
  aa[t] = s;
}

// loa(j, f, ias): LO function j = (ilo, lm1) of the atom against APW f
__global__ void k_mt_loa(MtArgs m, const int* flist, const int* lo_lm, const int* lo_ilo,
                         const double* halo, const double* kalo, cplx* loa) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)m.maxnlo * m.maxaa * m.natmtot) return;
  const int j = (int)(t % m.maxnlo);
  const int f = (int)((t / m.maxnlo) % m.maxaa);
  const int ias = (int)(t / ((long long)m.maxnlo * m.maxaa));
  const int is = m.idxis[ias];
  const int lm1 = lo_lm[j + m.maxnlo * ias], ilo = lo_ilo[j + m.maxnlo * ias];
  const int c3 = flist[f + m.maxaa * is];
  if (lm1 < 0 || ilo < 0 || c3 < 0) { loa[t] = cmk(0.0, 0.0); return; }
  const int lm3 = c3 / m.apwordmax, io = c3 % m.apwordmax;
  const int l1 = l_of(lm1), l3 = l_of(lm3);
  const int L1 = m.lmaxmat + 1;
  double kin = 0.0;
  if (lm1 == lm3 && kalo) kin = kalo[((size_t)ias * m.nlomax + ilo) * m.apwordmax + io];
  const double* h = halo + ((((size_t)ias * m.nlomax + ilo) * L1 + l3) * m.apwordmax + io) * m.lmvr;
  cplx s = gaunt_sum(m, lm1, l1, lm3, l3, h);
  s.x += kin;
  loa[t] = s;
}

// lolo(j1, j3, ias)
__global__ void k_mt_lolo(MtArgs m, const int* lo_lm, const int* lo_ilo, const double* hlolo,
                          const double* klolo, cplx* lolo) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)m.maxnlo * m.maxnlo * m.natmtot) return;
  const int j1 = (int)(t % m.maxnlo);
  const int j3 = (int)((t / m.maxnlo) % m.maxnlo);
  const int ias = (int)(t / ((long long)m.maxnlo * m.maxnlo));
  const int lm1 = lo_lm[j1 + m.maxnlo * ias], ilo1 = lo_ilo[j1 + m.maxnlo * ias];
  const int lm3 = lo_lm[j3 + m.maxnlo * ias], ilo2 = lo_ilo[j3 + m.maxnlo * ias];
  if (lm1 < 0 || ilo1 < 0 || lm3 < 0 || ilo2 < 0) { lolo[t] = cmk(0.0, 0.0); return; }
  double kin = 0.0;
  if (lm1 == lm3 && klolo) kin = klolo[((size_t)ias * m.nlomax + ilo1) * m.nlomax + ilo2];
  const double* h = hlolo + (((size_t)ias * m.nlomax + ilo1) * m.nlomax + ilo2) * m.lmvr;
  cplx s = gaunt_sum(m, lm1, l_of(lm1), lm3, l_of(lm3), h);
  s.x += kin;
  lolo[t] = s;
}

// oalo(io, ilo, ias) = olap + h1 and ololo(ilo1, ilo2, ias) likewise (IORA* folded in),
// h1aa(io1, io2, l, ias) from the per-(l, io1, io2) integrals
__global__ void k_mt_olp(MtArgs m, const double* oalo_r, const double* h1loa_r, const double* ololo_r,
                         const double* h1lolo_r, const double* h1aa_r, double* oalo, double* ololo, double* h1aa,
                         int h1on) {
  const int ias = blockIdx.x;
  const int L1 = m.lmaxmat + 1;
  for (int e = threadIdx.x; e < m.apwordmax * m.nlomax; e += blockDim.x) {
    const int io = e % m.apwordmax, ilo = e / m.apwordmax;
    const size_t src = ((size_t)ias * m.nlomax + ilo) * m.apwordmax + io;
    oalo[io + (size_t)m.apwordmax * (ilo + (size_t)m.nlomax * ias)] = oalo_r[src] + (h1on ? h1loa_r[src] : 0.0);
  }
  for (int e = threadIdx.x; e < m.nlomax * m.nlomax; e += blockDim.x) {
    const int i1 = e % m.nlomax, i2 = e / m.nlomax;
    const size_t src = ((size_t)ias * m.nlomax + i1) * m.nlomax + i2;
    ololo[i1 + (size_t)m.nlomax * (i2 + (size_t)m.nlomax * ias)] = ololo_r[src] + (h1on ? h1lolo_r[src] : 0.0);
  }
  if (h1on && h1aa)
    for (int e = threadIdx.x; e < m.apwordmax * m.apwordmax * (m.lmaxapw + 1); e += blockDim.x) {
      const int io1 = e % m.apwordmax, io2 = (e / m.apwordmax) % m.apwordmax, l = e / (m.apwordmax * m.apwordmax);
      h1aa[io1 + (size_t)m.apwordmax * (io2 + (size_t)m.apwordmax * (l + (size_t)(m.lmaxapw + 1) * ias))] =
          (l < L1) ? h1aa_r[(((size_t)ias * L1 + l) * m.apwordmax + io1) * m.apwordmax + io2] : 0.0;
    }
}

}  // namespace

// mt_kin (kinetic) + mt_pot of the field `pot` (host, veffmt's layout; NULL:
// veffmt) into dst_aa / dst_loa / dst_lolo (device, the handle's block
// layouts), and with `olp` olprad into the handle's oalo / ololo / h1 terms;
// the host copies (nullable) receive aa, loa, lolo (complex) and oalo, ololo
// (real, without the IORA* terms) in the reference layouts.
static int mt_build(excfv_handle* h, const excfv_mtrad* r, const double* pot, bool kinetic, bool olp,
                    cplx* dst_aa, cplx* dst_loa, cplx* dst_lolo, double* aa_out, double* loa_out,
                    double* lolo_out, double* oalo_out, double* ololo_out) {
  DevStatic& st = h->st;
  const int* nlorb_h = st.h_nlorb.data();
  const int* lorbl_h = st.h_lorbl.data();
  if (r->lmaxvr < 0 || r->lmaxvr > SPECFUN_LMAX || r->nrmtmax < 3 || !r->nrmt || !r->spr || !r->apwfr ||
      (!pot && !r->veffmt) || (kinetic && !r->veffmt) || (st.nlotot > 0 && !r->lofr)) {
    excfv_set_error("muffin-tin build: missing or inconsistent radial data");
    return EXCFV_ERR_ARG;
  }
  if (!pot) pot = r->veffmt;
  cudaStream_t s = h->stream;
  const int lmvr = (r->lmaxvr + 1) * (r->lmaxvr + 1);
  const int nlomax = std::max(st.nlomax, 1);
  const int L1 = st.lmaxmat + 1;
  // host: spline weights (times r^2) per species, the Gaunt quadrature nodes
  // and the species' local-orbital lists, in one block for one upload
  int lg = st.lmaxmat;
  for (int is = 0; is < st.nspecies; ++is)
    for (int ilo = 0; ilo < nlorb_h[is]; ++ilo) lg = std::max(lg, lorbl_h[ilo + (size_t)nlomax * is]);
  const int lmg = (lg + 1) * (lg + 1), lmL = std::max(lmg, lmvr), nq = gaunt_nodes(lg, r->lmaxvr);
  const size_t nr2 = (size_t)r->nrmtmax, N = st.natmtot;
  const size_t n_mesh = nr2 * st.nspecies, n_node = (size_t)nq * (lmL + 1);
  const size_t n_int = ((size_t)(2 + nlomax) * st.nspecies + 1) / 2;  // ints, in doubles
  std::vector<double> pack(2 * n_mesh + n_node + n_int, 0.0);
  double* wts = pack.data();
  int* ints = reinterpret_cast<int*>(pack.data() + 2 * n_mesh + n_node);
  for (int is = 0; is < st.nspecies; ++is) {
    const int nr = r->nrmt[is];
    if (nr < 3 || nr > r->nrmtmax) {
      excfv_set_error("excfv_hmlint: species %d has %d mesh points (need 3..nrmtmax)", is + 1, nr);
      return EXCFV_ERR_ARG;
    }
    const double* x = r->spr + nr2 * is;
    spline_weights(nr, x, wts + nr2 * is);
    for (int i = 0; i < nr; ++i) wts[nr2 * is + i] *= x[i] * x[i];
    ints[is] = nr;
    ints[st.nspecies + is] = nlorb_h[is];
    for (int ilo = 0; ilo < nlorb_h[is]; ++ilo)
      ints[(2 + ilo) * st.nspecies + is] = lorbl_h[ilo + (size_t)nlomax * is];
  }
  std::copy(r->spr, r->spr + n_mesh, pack.begin() + n_mesh);
  gaunt_node_values(lg, r->lmaxvr, pack.data() + 2 * n_mesh);
  // device: inputs and integrals in the handle's scratch
  const int A = st.apwordmax;
  const int per_aa = L1 * A * L1 * A * lmvr, per_loa = nlomax * L1 * A * lmvr, per_lolo = nlomax * nlomax * lmvr;
  const int per_kaa = L1 * A * A, per_kalo = nlomax * A, per_klolo = nlomax * nlomax;
  const size_t n_apw = nr2 * 2 * A * (st.lmaxapw + 1) * N, n_lo = nr2 * 2 * nlomax * N, n_v = (size_t)lmvr * nr2 * N;
  const size_t n_gnt = (size_t)lmg * lmg * (r->lmaxvr + 1);
  size_t total = 0;
  auto take = [&](size_t n) { const size_t at = total; total += (n + 31) / 32 * 32; return at; };
  const size_t o_pack = take(pack.size()), o_apw = take(n_apw), o_lo = take(n_lo), o_v = take(n_v),
               o_gnt = take(n_gnt), o_haa = take(per_aa * N), o_halo = take(per_loa * N),
               o_hlolo = take(per_lolo * N), o_kaa = take(per_kaa * N), o_kalo = take(per_kalo * N),
               o_klolo = take(per_klolo * N), o_oalo = take(per_kalo * N), o_ololo = take(per_klolo * N),
               o_h1aa = take(per_kaa * N), o_h1loa = take(per_kalo * N), o_h1lolo = take(per_klolo * N);
  void* base = nullptr;
  int rc = handle_scratch(h, sizeof(double) * total, &base);
  if (rc) return rc;
  double* D = static_cast<double*>(base);
  double *haa = D + o_haa, *halo = D + o_halo, *hlolo = D + o_hlolo, *kaa = D + o_kaa, *kalo = D + o_kalo,
         *klolo = D + o_klolo, *oalo_r = D + o_oalo, *ololo_r = D + o_ololo, *h1aa_r = D + o_h1aa,
         *h1loa_r = D + o_h1loa, *h1lolo_r = D + o_h1lolo;
  MtArgs m;
  m.natmtot = st.natmtot; m.lmaxmat = st.lmaxmat; m.lmaxapw = st.lmaxapw; m.apwordmax = st.apwordmax;
  m.nlomax = nlomax; m.lmvr = lmvr; m.nrmtmax = r->nrmtmax; m.maxaa = st.maxaa; m.maxnlo = std::max(st.maxnlo, 1);
  m.a = (st.vrel != 0) ? 0.5 * ALPHA_FS * ALPHA_FS : 0.0;
  m.lmaxvr = r->lmaxvr; m.lg = lg; m.nspecies = st.nspecies;
  m.idxis = st.idxis; m.apword = st.apword;
  const int* d_ints = reinterpret_cast<const int*>(D + o_pack + 2 * n_mesh + n_node);
  m.nrmt = d_ints; m.nlorb = d_ints + st.nspecies; m.lorbl = d_ints + 2 * st.nspecies;
  m.wts = D + o_pack; m.spr = D + o_pack + n_mesh;
  m.apwfr = D + o_apw; m.lofr = D + o_lo; m.veff = D + o_v; m.gnt = D + o_gnt;
  auto copy_in = [&](size_t at, const double* src, size_t n) {
    return src ? cudaMemcpyAsync(D + at, src, sizeof(double) * n, cudaMemcpyHostToDevice, s)
               : cudaMemsetAsync(D + at, 0, sizeof(double) * n, s);
  };
  if (copy_in(o_pack, pack.data(), pack.size()) != cudaSuccess || copy_in(o_apw, r->apwfr, n_apw) != cudaSuccess ||
      copy_in(o_lo, r->lofr, n_lo) != cudaSuccess || copy_in(o_v, pot, n_v) != cudaSuccess) {
    excfv_set_error("muffin-tin build: upload failed");
    rc = EXCFV_ERR_CUDA;
    goto done;
  }
  {
    auto grid = [](long long n) { return (unsigned)((n + 127) / 128); };
    k_gaunt<<<grid((long long)n_gnt), 128, 0, s>>>(lg, r->lmaxvr, nq, D + o_pack + 2 * n_mesh, D + o_gnt);
    count_launch();
    RadSets sets;
    sets.n = 0;
    auto want = [&](int kind, int mode, int per, double* out) { sets.s[sets.n++] = RadSet{kind, mode, per, out}; };
    if (kinetic) {
      want(0, 0, per_kaa, kaa);
      want(1, 0, per_kalo, kalo);
      want(2, 0, per_klolo, klolo);
    }
    if (olp) {
      want(1, 2, per_kalo, oalo_r);
      want(2, 2, per_klolo, ololo_r);
    }
    if (olp && st.h1on) {
      want(0, 1, per_kaa, h1aa_r);
      want(1, 1, per_kalo, h1loa_r);
      want(2, 1, per_klolo, h1lolo_r);
    }
    long long nrad = 0;
    for (int q = 0; q < sets.n; ++q) nrad += (long long)sets.s[q].per_atom * N;
    if (nrad > 0) {
      k_mt_radint<<<grid(32 * nrad), 128, 0, s>>>(m, sets); count_launch();
    }
    k_mt_potint<<<grid((long long)(per_aa + per_loa + per_lolo) * N), 128, 0, s>>>(m, per_aa, per_loa, per_lolo, haa,
                                                                                   halo, hlolo);
    count_launch();
    // assembly into the static blocks
    const double* ka = kinetic ? kaa : nullptr;
    const double* kl = kinetic ? kalo : nullptr;
    const double* kll = kinetic ? klolo : nullptr;
    k_mt_aa<<<grid((long long)st.maxaa * st.maxaa * N), 128, 0, s>>>(m, st.flist, haa, ka, dst_aa);
    count_launch();
    if (st.maxnlo > 0) {
      k_mt_loa<<<grid((long long)st.maxnlo * st.maxaa * N), 128, 0, s>>>(m, st.flist, st.lo_lm, st.lo_ilo, halo,
                                                                          kl, dst_loa);
      count_launch();
      k_mt_lolo<<<grid((long long)st.maxnlo * st.maxnlo * N), 128, 0, s>>>(m, st.lo_lm, st.lo_ilo, hlolo, kll,
                                                                            dst_lolo);
      count_launch();
    }
    if (olp && (st.nlomax > 0 || st.h1on)) {
      k_mt_olp<<<st.natmtot, 128, 0, s>>>(m, oalo_r, h1loa_r, ololo_r, h1lolo_r, h1aa_r, st.oalo, st.ololo,
                                          st.h1aa, st.h1on);
      count_launch();
    }
    if (cudaGetLastError() != cudaSuccess) { rc = EXCFV_ERR_CUDA; goto done; }
    // optional host copies (reference layouts)
    if (aa_out) cudaMemcpyAsync(aa_out, dst_aa, sizeof(cplx) * st.maxaa * st.maxaa * N, cudaMemcpyDeviceToHost, s);
    if (loa_out && st.maxnlo > 0)
      cudaMemcpyAsync(loa_out, dst_loa, sizeof(cplx) * st.maxnlo * st.maxaa * N, cudaMemcpyDeviceToHost, s);
    if (lolo_out && st.maxnlo > 0)
      cudaMemcpyAsync(lolo_out, dst_lolo, sizeof(cplx) * st.maxnlo * st.maxnlo * N, cudaMemcpyDeviceToHost, s);
    std::vector<double> tmp;
    if (olp && (oalo_out || ololo_out) && st.nlomax > 0) {
      tmp.resize((size_t)(per_kalo + per_klolo) * N);
      cudaMemcpyAsync(tmp.data(), oalo_r, sizeof(double) * per_kalo * N, cudaMemcpyDeviceToHost, s);
      cudaMemcpyAsync(tmp.data() + per_kalo * N, ololo_r, sizeof(double) * per_klolo * N, cudaMemcpyDeviceToHost, s);
    }
    if (cudaStreamSynchronize(s) != cudaSuccess) { rc = EXCFV_ERR_CUDA; goto done; }
    if (!tmp.empty()) {
      for (size_t ias = 0; ias < N; ++ias) {
        for (int ilo = 0; ilo < st.nlomax; ++ilo)
          for (int io = 0; io < A; ++io)
            if (oalo_out)
              oalo_out[io + (size_t)A * (ilo + (size_t)st.nlomax * ias)] = tmp[(ias * nlomax + ilo) * A + io];
        for (int i1 = 0; i1 < st.nlomax; ++i1)
          for (int i2 = 0; i2 < st.nlomax; ++i2)
            if (ololo_out)
              ololo_out[i1 + (size_t)st.nlomax * (i2 + (size_t)st.nlomax * ias)] =
                  tmp[per_kalo * N + (ias * nlomax + i1) * nlomax + i2];
      }
    }
  }
done:
  cudaStreamSynchronize(s);
  if (rc == EXCFV_OK && olp && st.h1on) st.have_h1aa = true;
  return rc;
}

int stage_hmlint(excfv_handle* h, const excfv_mtrad* r, double* aa_out, double* loa_out, double* lolo_out,
                 double* oalo_out, double* ololo_out) {
  DevStatic& st = h->st;
  return mt_build(h, r, nullptr, true, true, st.aa, st.loa, st.lolo, aa_out, loa_out, lolo_out, oalo_out,
                  ololo_out);
}

// mt_pot of a field without the kinetic term and without olprad (the spin
// blocks of hmlint.f90:88-108) into the given device blocks
int stage_mt_field(excfv_handle* h, const excfv_mtrad* r, const double* field, cplx* aa, cplx* loa, cplx* lolo,
                   double* aa_out, double* loa_out, double* lolo_out) {
  return mt_build(h, r, field, false, false, aa, loa, lolo, aa_out, loa_out, lolo_out, nullptr, nullptr);
}

// The cubic spline of spline.f90 on the host: d1 = cf(1, :), the first
// derivative at each mesh point (fderiv(1)); returns the integral over the
// whole mesh (fderiv(-1) at the last point) of f.
double host_spline(int n, const double* x, const double* f, double* d1) {
  std::vector<double> c1(n), c2(n), c3(n), w(n);
  const double g = spline_integral(n, x, f, c1, c2, c3, w);
  if (d1) {
    // spline_integral leaves c1 = the divided differences and c2 = the second
    // coefficients; the first coefficients follow as in spline.f90
    for (int i = 0; i < n - 1; ++i) {
      const double d3 = (1.0 / 3.0) * (c2[i + 1] - c2[i]) * w[i];
      const double dx = x[i + 1] - x[i];
      d1[i] = c1[i] - (c2[i] + d3 * dx) * dx;
    }
    const double dxl = x[n - 1] - x[n - 2];
    const double d3l = (1.0 / 3.0) * (c2[n - 1] - c2[n - 2]) * w[n - 2];
    d1[n - 1] = d1[n - 2] + (2.0 * c2[n - 2] + 3.0 * d3l * dxl) * dxl;
  }
  return g;
}
