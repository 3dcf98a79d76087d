// The muffin-tin valence density of one k-point on the device: rhovalk
// (src/rhovalk.f90:56-203) for the spin-unpolarised ground state without
// second-variational vectors, with wavefmt (src/wavefmt.f90) inside.
//
//   c(io, lm, j)   = sum_G apwalm(G, io, lm, ias) evecfv(G, j)    (zdotu of wavefmt)
//                    one batched GEMM over the atoms, op(A) = apwalm^T
//   wf(lm, r, j)   = sum_io c(io, lm, j) u_io,l(r) + sum_ilo evecfv(ngp + idxlo, j) v_ilo(r)
//                    (wavefmt_add: a real or imaginary part below 1e-14 is dropped)
//   rfmt(tp, r)    = sum_j w_j |sum_lm zbshtvr(tp, lm) wf(lm, r, j)|^2
//   rhomt(lm, r)  += sum_tp rfshtvr(lm, tp) rfmt(tp, r)
// on the coarse radial mesh (every lradstep-th point), w_j = wkpt occsv
// (states with |w_j| <= epsocc skipped).  With second-variational vectors
// (collinear spin, rhovalk.f90:74-160) each spinor component of state j is
// sum_ist evecsv((ispn-1) nstfv + ist, j) wfmt(ist), which is linear in the
// coefficients: the first-variational coefficients (their parts below 1e-14
// dropped first, as wavefmt_add drops them) times the spin's rows of evecsv
// (entries with |Re| + |Im| <= epsocc dropped) by one GEMM, then the same
// kernels per spin, rhomt += up + dn and magmt += up - dn.  The densities on the
// covering points (k_rho_psi) go through a small buffer to the forward real
// transform (k_rho_sht); each rhomt entry has one owner, so k-points accumulate
// in stream order without atomics.  The non-collinear branch has one CTA per
// (coarse radial point, atom) that keeps both spinor components in shared memory.
#include <vector>

#include "handle.cuh"

namespace {

constexpr int JB = 16;         // states per chunk of the non-collinear kernel
constexpr int RHO_LMAX = 8;    // lmaxvr supported by the shared-memory transform
constexpr double WF_EPS = 1e-14;

struct RhoArgs {
  int natmtot, lmaxvr, lmmaxvr, lradstep, nrcmax, nrmtmax, apwordmax, nlomax, maxnlo, nst, ngp;
  const int* idxis;
  const int* nrmt;       // (nspecies)
  const int* apword;     // (lmaxapw+1, nspecies)
  int lmaxapw;
  const int* lo_lm;      // (maxnlo, natmtot)
  const int* lo_ilo;     // (maxnlo, natmtot)
  const int* lo_first;   // (natmtot) first global LO index, -1 none
  const int* lorbl;      // (nlomax, nspecies)
  const double* ucoarse; // (nrcmax, apwordmax, lmaxvr+1, natmtot)
  const double* vcoarse; // (nrcmax, nlomax, natmtot)
  const cplx* zb;        // (lmmaxvr, lmmaxvr): (tp, lm)
  const double* rf;      // (lmmaxvr, lmmaxvr): (lm, tp)
  // APW coefficients, ldc between states, cstride between atoms; the row of
  // (lm, io) is io + apwordmax * lm, or its packed index when fofl is given
  const cplx* coef;
  long long ldc, cstride;
  const int* fofl;       // nullable: DevStatic::fofl
  int lmmaxapw;
  int ias0;              // first atom of the launch (k_rho_ang, k_rho_psi)
  const cplx* evec;      // (nmatmax, nst)
  long long ldev;
  const cplx* locoef;    // nullable: LO coefficients (q + maxnlo ias, j) in place of evec's rows
  long long ldlo;
  int cut;               // apply wavefmt_add's cut-off to the coefficients
  const double* w;       // (nst) weights, 0 for skipped states
  double* rhomt;         // (lmmaxvr, nrmtmax, natmtot)
  double* magmt;         // nullable: += msign * the same density
  double msign;
};

// The densities on the covering points, rho(tp, r) = sum_j w_j |psi_j(tp, r)|^2.
// A state's value is a sum over the atom's radial functions b (an APW (l, io)
// or a local orbital) of u_b(r) g_b(tp, j), where g_b = sum_m zb(tp, lm)
// c(lm, io, j) does not depend on r; so the backward transform runs once per
// state (k_rho_ang) instead of once per state and radial point, and the radial
// part (k_rho_psi) is a real-by-complex product over about 22 functions instead
// of a complex one over (lmaxvr+1)^2 harmonics.
// 130 states, 150 radial points, 8 atoms, lmaxvr 8: 67 us and 134 us, against
// 3430 us for one CTA per radial point with a thread per covering point.

// gang(j, b, tp, ias - ias0) = sum_m zb(tp, lm) c: a thread per state keeps its 2l+1
// coefficients in registers and runs over the covering points of blockIdx.z's
// share; zb's rows of this l are broadcast from shared memory.
constexpr int ANG_T = 64;
__global__ void __launch_bounds__(ANG_T) k_rho_ang(RhoArgs a, cplx* __restrict__ gang) {
  constexpr int MM = 2 * RHO_LMAX + 1;
  __shared__ cplx sz[(RHO_LMAX + 1) * (RHO_LMAX + 1) * MM];
  const int L = a.lmmaxvr, L1 = a.lmaxvr + 1;
  const int nb = L1 * a.apwordmax + a.nlomax;
  const int b = blockIdx.y % nb, ias = a.ias0 + blockIdx.y / nb, is = a.idxis[ias];
  const int per = (L + gridDim.z - 1) / gridDim.z, t0 = blockIdx.z * per, t1 = min(L, t0 + per);
  const int j = blockIdx.x * ANG_T + threadIdx.x;
  const bool on = j < a.nst && a.w[j] != 0.0;  // skipped states may hold anything
  const bool apw = b < L1 * a.apwordmax;
  const int ilo = b - L1 * a.apwordmax, io = b % a.apwordmax;
  int l = b / a.apwordmax, nm = 0;
  if (apw) {
    if (io < a.apword[l + (a.lmaxapw + 1) * is]) nm = 2 * l + 1;
  } else if (a.lo_first[ias] >= 0) {
    l = a.lorbl[ilo + a.nlomax * is];
    if (l < L1) nm = 2 * l + 1;
  }
  for (int e = threadIdx.x; e < (t1 - t0) * nm; e += ANG_T)
    sz[(e / nm) * MM + e % nm] = a.zb[t0 + e / nm + L * (l * l + e % nm)];
  cplx c[MM];
#pragma unroll
  for (int m = 0; m < MM; ++m) {
    c[m] = cmk(0.0, 0.0);
    if (m < nm && on) {
      const int lm = l * l + m;
      if (apw) {
        const int row = a.fofl ? a.fofl[(size_t)(lm * a.apwordmax + io) + (size_t)a.lmmaxapw * a.apwordmax * is]
                               : io + a.apwordmax * lm;
        c[m] = a.coef[a.cstride * ias + row + a.ldc * j];
      } else {
        for (int q = 0; q < a.maxnlo; ++q)  // the function (ilo, lm) of the atom, if it has one
          if (a.lo_ilo[q + a.maxnlo * ias] == ilo && a.lo_lm[q + a.maxnlo * ias] == lm)
            c[m] = a.locoef ? a.locoef[(size_t)(q + a.maxnlo * ias) + (size_t)a.ldlo * j]
                            : a.evec[(size_t)(a.ngp + a.lo_first[ias] + q) + (size_t)a.ldev * j];
      }
      if (a.cut) {  // wavefmt_add: parts below the cut-off do not contribute
        if (fabs(c[m].x) < WF_EPS) c[m].x = 0.0;
        if (fabs(c[m].y) < WF_EPS) c[m].y = 0.0;
      }
    }
  }
  __syncthreads();
  if (j >= a.nst) return;
  for (int tp = t0; tp < t1; ++tp) {
    cplx v = cmk(0.0, 0.0);
#pragma unroll
    for (int m = 0; m < MM; ++m)
      if (m < nm) v = cadd(v, cmul(sz[(tp - t0) * MM + m], c[m]));
    gang[j + (size_t)a.nst * (b + (size_t)nb * (tp + (size_t)L * (ias - a.ias0)))] = v;
  }
}

// One covering point of one atom and PSI_R radial points per CTA.  g of a chunk
// of states is copied to shared memory; a lane owns radial points r, r+32, ...;
// a warp takes JT states at a time (g broadcast, u coalesced from L1), so each u
// or g loaded feeds JT or RK complex FMAs, and |psi|^2 stays in registers.
// Bound by FP64 FMAs.  STAGED false: more functions than shared memory holds for a
// warp's states; g is read where it is.
constexpr int RK = 4;    // radial points per lane
constexpr int JT = 4;    // states per warp step
constexpr int PSI_T = 256;
constexpr int PSI_R = 32 * RK;
constexpr size_t PSI_SMEM = 200 * 1024;  // most dynamic shared memory

template <bool STAGED>
__global__ void __launch_bounds__(PSI_T) k_rho_psi(RhoArgs a, int jc, const cplx* __restrict__ gang,
                                                   double* __restrict__ rtp) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int tp = blockIdx.x, ias = a.ias0 + blockIdx.y, r0 = blockIdx.z * PSI_R;
  const int nrc = (a.nrmt[a.idxis[ias]] + a.lradstep - 1) / a.lradstep;
  if (r0 >= nrc) return;
  const int L = a.lmmaxvr, L1 = a.lmaxvr + 1;
  const int na = L1 * a.apwordmax, nb = na + a.nlomax;  // (l, io), then local orbitals
  cplx* g = reinterpret_cast<cplx*>(dsm);               // [nb][jc]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double acc[RK];
#pragma unroll
  for (int k = 0; k < RK; ++k) acc[k] = 0.0;
  const cplx* gin = gang + (size_t)a.nst * nb * (tp + (size_t)L * blockIdx.y);
  for (int j0 = 0; j0 < a.nst; j0 += jc) {
    const int nj = min(jc, a.nst - j0);
    if constexpr (STAGED) {
      __syncthreads();
      for (int b = warp; b < nb; b += PSI_T / 32)
        for (int jj = lane; jj < jc; jj += 32) g[b * jc + jj] = (jj < nj) ? gin[j0 + jj + (size_t)a.nst * b] : cmk(0.0, 0.0);
      __syncthreads();
    }
    for (int jj = JT * warp; jj < nj; jj += JT * (PSI_T / 32)) {  // jc is a multiple of JT
      cplx psi[RK][JT];
#pragma unroll
      for (int k = 0; k < RK; ++k)
#pragma unroll
        for (int t = 0; t < JT; ++t) psi[k][t] = cmk(0.0, 0.0);
      auto add = [&](const double* ub, int b) {
        cplx gv[JT];
#pragma unroll
        for (int t = 0; t < JT; ++t) {
          if constexpr (STAGED) gv[t] = g[b * jc + jj + t];
          else gv[t] = (jj + t < nj) ? gin[j0 + jj + t + (size_t)a.nst * b] : cmk(0.0, 0.0);
        }
#pragma unroll
        for (int k = 0; k < RK; ++k) {
          const int r = r0 + lane + 32 * k;
          const double u = (r < nrc) ? __ldg(ub + r) : 0.0;
#pragma unroll
          for (int t = 0; t < JT; ++t) {
            psi[k][t].x = fma(u, gv[t].x, psi[k][t].x);
            psi[k][t].y = fma(u, gv[t].y, psi[k][t].y);
          }
        }
      };
      const double* ua = a.ucoarse + (size_t)a.nrcmax * na * ias;
#pragma unroll 2
      for (int b = 0; b < na; ++b) add(ua + (size_t)a.nrcmax * b, b);
      const double* va = a.vcoarse + (size_t)a.nrcmax * a.nlomax * ias;
      for (int b = na; b < nb; ++b) add(va + (size_t)a.nrcmax * (b - na), b);
#pragma unroll
      for (int t = 0; t < JT; ++t) {
        const double wj = (jj + t < nj) ? a.w[j0 + jj + t] : 0.0;
        if (wj == 0.0) continue;
#pragma unroll
        for (int k = 0; k < RK; ++k) acc[k] += wj * (psi[k][t].x * psi[k][t].x + psi[k][t].y * psi[k][t].y);
      }
    }
  }
  // the warps' states, in a fixed order
  __shared__ double red[PSI_T / 32][PSI_R];
#pragma unroll
  for (int k = 0; k < RK; ++k) red[warp][lane + 32 * k] = acc[k];
  __syncthreads();
  for (int r = tid; r < PSI_R && r0 + r < nrc; r += PSI_T) {
    double s = 0.0;
    for (int w = 0; w < PSI_T / 32; ++w) s += red[w][r];
    rtp[(size_t)(r0 + r) + (size_t)a.nrcmax * (tp + (size_t)L * ias)] = s;
  }
}

// rhomt(lm, r) += sum_tp rf(lm, tp) rho(tp, r), and magmt += msign times it
constexpr int SHT_R = 4;  // radial points per CTA
__global__ void k_rho_sht(RhoArgs a, const double* __restrict__ rtp) {
  __shared__ double sr[(RHO_LMAX + 1) * (RHO_LMAX + 1)][SHT_R];
  const int ias = blockIdx.y, r0 = blockIdx.x * SHT_R;
  const int is = a.idxis[ias];
  const int nrc = (a.nrmt[is] + a.lradstep - 1) / a.lradstep;
  if (r0 >= nrc) return;
  const int L = a.lmmaxvr;
  for (int e = threadIdx.x; e < L * SHT_R; e += blockDim.x) {
    const int rr = e % SHT_R, tp = e / SHT_R;
    sr[tp][rr] = (r0 + rr < nrc) ? rtp[(size_t)(r0 + rr) + (size_t)a.nrcmax * (tp + (size_t)L * ias)] : 0.0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < L * SHT_R; e += blockDim.x) {
    const int lm = e % L, rr = e / L;
    if (r0 + rr >= nrc) continue;
    double s = 0.0;
#pragma unroll 9
    for (int tp = 0; tp < L; ++tp) s += a.rf[lm + (size_t)L * tp] * sr[tp][rr];
    const size_t at = lm + (size_t)L * ((r0 + rr) * a.lradstep + (size_t)a.nrmtmax * ias);
    a.rhomt[at] += s;
    if (a.magmt) a.magmt[at] += a.msign * s;
  }
}

// elements of gang: the atoms are taken in groups that keep it in the L2 cache
// (64 MB), or one by one where one alone is larger
size_t rho_gang_elems(size_t nst, size_t nb, size_t L, size_t natmtot) {
  const size_t one = nst * nb * L;
  return std::min(one * natmtot, std::max(one, (size_t)(64 << 20) / sizeof(cplx)));
}

// the three kernels over all atoms
int rho_mt(excfv_handle* h, RhoArgs a) {
  cudaStream_t s = h->stream;
  cplx* gang = h->rho.gang;
  double* rtp = h->rho.rtp;
  const int nb = (a.lmaxvr + 1) * a.apwordmax + a.nlomax;
  const int L = a.lmmaxvr;
  // states per chunk: all of them where two CTAs then still share an SM
  int jc = (a.nst + JT - 1) / JT * JT;
  const size_t per = sizeof(cplx) * nb;
  const int fit = (int)(96 * 1024 / per);
  if (jc > fit) jc = std::max(JT, fit / 32 * 32);
  const bool staged = per * jc <= PSI_SMEM;
  const size_t smem = staged ? per * jc : 0;
  CUDA_TRY(raise_smem_limit(k_rho_psi<true>, PSI_SMEM));
  auto* psi = staged ? k_rho_psi<true> : k_rho_psi<false>;
  const size_t one = (size_t)a.nst * nb * L;
  // (k_rho_ang's grid has a row per function and atom, 65535 at most)
  const int group = (int)std::min<size_t>(std::min(a.natmtot, std::max(1, 65535 / nb)),
                                          std::max<size_t>(1, h->rho.gang_elems / one));
  const int nj = (a.nst + ANG_T - 1) / ANG_T;
  for (a.ias0 = 0; a.ias0 < a.natmtot; a.ias0 += group) {
    const int na = std::min(group, a.natmtot - a.ias0);
    // shares of the covering points: enough CTAs for every SM
    const int tz = std::min(L, std::max(1, 4 * h->nsm / (nj * nb * na)));
    k_rho_ang<<<dim3(nj, nb * na, tz), ANG_T, 0, s>>>(a, gang);
    count_launch();
    psi<<<dim3(L, na, (a.nrcmax + PSI_R - 1) / PSI_R), PSI_T, smem, s>>>(a, jc, gang, rtp);
    count_launch();
  }
  k_rho_sht<<<dim3((a.nrcmax + SHT_R - 1) / SHT_R, a.natmtot), 256, 0, s>>>(a, rtp);
  count_launch();
  CUDA_TRY(cudaGetLastError());
  return EXCFV_OK;
}

// The wavefunction's lm expansion at coarse point irc of atom ias for state
// j from coefficients cf (APW, per atom) and lo (LO rows), without cut-off.
__device__ __forceinline__ cplx wf_lm(const RhoArgs& a, const cplx* cf, const cplx* lo, int ias, int is, int irc,
                                      int lm, int j) {
  cplx v = cmk(0.0, 0.0);
  int l = 0;
  while ((l + 1) * (l + 1) <= lm) ++l;
  const int nap = a.apword[l + (a.lmaxapw + 1) * is];
  for (int io = 0; io < nap; ++io) {
    const cplx c = cf[(size_t)(io + a.apwordmax * lm) + (size_t)a.apwordmax * a.lmmaxvr * j];
    const double u = a.ucoarse[irc + (size_t)a.nrcmax * (io + (size_t)a.apwordmax * (l + (size_t)(a.lmaxvr + 1) * ias))];
    v.x += c.x * u;
    v.y += c.y * u;
  }
  if (a.lo_first[ias] >= 0)
    for (int q = 0; q < a.maxnlo; ++q) {
      if (a.lo_lm[q + a.maxnlo * ias] != lm) continue;
      const int ilo = a.lo_ilo[q + a.maxnlo * ias];
      const cplx c = lo[(size_t)(q + a.maxnlo * ias) + (size_t)a.ldlo * j];
      const double f = a.vcoarse[irc + (size_t)a.nrcmax * (ilo + (size_t)a.nlomax * ias)];
      v.x += c.x * f;
      v.y += c.y * f;
    }
  return v;
}

// The non-collinear density (rhovalk.f90:151-195, ncmag): both spinor
// components of each state at each covering point, z1 (a.coef, a.locoef)
// and z2 (cdn, ldn); sums of w |z1|^2, w |z2|^2, w Re(z1 z2*), w Im(z1 z2*),
// each taken back to real harmonics: rhomt += r1 + r2, magmt(1) += 2 r3,
// magmt(2) -= 2 r4, magmt(3) += r1 - r2.
__global__ void k_rho_mt_nc(RhoArgs a, const cplx* cdn, const cplx* ldn, double* magmt3) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int irc = blockIdx.x, ias = blockIdx.y;
  const int is = a.idxis[ias];
  const int nr = a.nrmt[is];
  const int nrc = (nr + a.lradstep - 1) / a.lradstep;
  if (irc >= nrc) return;
  const int L = a.lmmaxvr;
  cplx* zb = reinterpret_cast<cplx*>(dsm);      // L x L
  cplx* w1 = zb + L * L;                        // L x JB
  cplx* w2 = w1 + L * JB;                       // L x JB
  double* rfmt = reinterpret_cast<double*>(w2 + L * JB);  // 4 x L
  for (int e = threadIdx.x; e < L * L; e += blockDim.x) zb[e] = a.zb[e];
  double s1 = 0.0, s2 = 0.0, s3 = 0.0, s4 = 0.0;  // thread tp < L
  const size_t off = (size_t)a.apwordmax * L * a.nst * ias;
  for (int j0 = 0; j0 < a.nst; j0 += JB) {
    const int nj = min(JB, a.nst - j0);
    __syncthreads();
    for (int e = threadIdx.x; e < L * nj; e += blockDim.x) {
      const int lm = e % L, jj = e / L, j = j0 + jj;
      const bool on = a.w[j] != 0.0;
      w1[lm + L * jj] = on ? wf_lm(a, a.coef + off, a.locoef, ias, is, irc, lm, j) : cmk(0.0, 0.0);
      w2[lm + L * jj] = on ? wf_lm(a, cdn + off, ldn, ias, is, irc, lm, j) : cmk(0.0, 0.0);
    }
    __syncthreads();
    if (threadIdx.x < L) {
      const int tp = threadIdx.x;
      for (int jj = 0; jj < nj; ++jj) {
        const double wj = a.w[j0 + jj];
        if (wj == 0.0) continue;
        cplx z1 = cmk(0.0, 0.0), z2 = cmk(0.0, 0.0);
        for (int lm = 0; lm < L; ++lm) {
          const cplx y = zb[tp + L * lm];
          z1 = cadd(z1, cmul(y, w1[lm + L * jj]));
          z2 = cadd(z2, cmul(y, w2[lm + L * jj]));
        }
        s1 += wj * (z1.x * z1.x + z1.y * z1.y);
        s2 += wj * (z2.x * z2.x + z2.y * z2.y);
        s3 += wj * (z1.x * z2.x + z1.y * z2.y);   // Re(z1 conj(z2))
        s4 += wj * (z1.y * z2.x - z1.x * z2.y);   // Im(z1 conj(z2))
      }
    }
  }
  if (threadIdx.x < L) {
    rfmt[threadIdx.x] = s1;
    rfmt[L + threadIdx.x] = s2;
    rfmt[2 * L + threadIdx.x] = s3;
    rfmt[3 * L + threadIdx.x] = s4;
  }
  __syncthreads();
  if (threadIdx.x < L) {
    const int lm = threadIdx.x;
    double r[4] = {0.0, 0.0, 0.0, 0.0};
    for (int tp = 0; tp < L; ++tp) {
      const double f = a.rf[lm + (size_t)L * tp];
      for (int k = 0; k < 4; ++k) r[k] += f * rfmt[k * L + tp];
    }
    const size_t at = lm + (size_t)L * (irc * a.lradstep + (size_t)a.nrmtmax * ias);
    const size_t comp = (size_t)L * a.nrmtmax * a.natmtot;
    a.rhomt[at] += r[0] + r[1];
    magmt3[at] += 2.0 * r[2];
    magmt3[at + comp] -= 2.0 * r[3];
    magmt3[at + 2 * comp] += r[0] - r[1];
  }
}

// drop real and imaginary parts below the cut-off (wavefmt_add)
__global__ void k_rho_cut(long long n, cplx* c) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  cplx v = c[t];
  if (fabs(v.x) < WF_EPS) v.x = 0.0;
  if (fabs(v.y) < WF_EPS) v.y = 0.0;
  c[t] = v;
}

// LO rows of evecfv per atom, cut: lo(q + maxnlo ias, j)
__global__ void k_rho_gather_lo(int natmtot, int maxnlo, int nst, int ngp, const int* lo_lm, const int* lo_first,
                                const cplx* evec, long long ldev, cplx* lo) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long rows = (long long)maxnlo * natmtot;
  if (t >= rows * nst) return;
  const int r = (int)(t % rows), j = (int)(t / rows);
  const int ias = r / maxnlo, q = r % maxnlo;
  cplx v = cmk(0.0, 0.0);
  if (lo_first[ias] >= 0 && lo_lm[q + maxnlo * ias] >= 0) {
    v = evec[(size_t)(ngp + lo_first[ias] + q) + ldev * j];
    if (fabs(v.x) < WF_EPS) v.x = 0.0;
    if (fabs(v.y) < WF_EPS) v.y = 0.0;
  }
  lo[t] = v;
}

// one spin's rows of evecsv (ld 2n), entries with |Re| + |Im| <= epsocc dropped
__global__ void k_rho_esv(int n, int spin, const cplx* evecsv, double epsocc, cplx* esv) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n * 2 * n) return;
  const int ist = (int)(t % n), j = (int)(t / n);
  cplx v = evecsv[(size_t)(spin * n + ist) + (size_t)2 * n * j];
  if (fabs(v.x) + fabs(v.y) <= epsocc) v = cmk(0.0, 0.0);
  esv[t] = v;
}

}  // namespace

void free_rho(DevRho& r) {
  if (r.block.base) cudaFree(r.block.base);
  r = DevRho();
}

int stage_set_rho(excfv_handle* h, const excfv_rhoset* r) {
  DevStatic& st = h->st;
  {  // forgets the data but keeps their memory
    const Block keep = h->rho.block;
    h->rho = DevRho();
    h->rho.block = keep;
  }
  if (r->lmaxvr < 0 || r->lmaxvr > RHO_LMAX || r->lmaxvr > st.lmaxapw || r->lradstep < 1 || r->nrmtmax < 1 ||
      !r->nrmt || !r->apwfr || !r->zbshtvr || !r->rfshtvr || (st.nlotot > 0 && !r->lofr)) {
    excfv_set_error("excfv_set_rho: lmaxvr must be 0..%d and <= lmaxapw, lradstep >= 1, arrays given", RHO_LMAX);
    return EXCFV_ERR_ARG;
  }
  DevRho& d = h->rho;
  d.lmaxvr = r->lmaxvr;
  d.lmmaxvr = (r->lmaxvr + 1) * (r->lmaxvr + 1);
  d.lradstep = r->lradstep;
  d.nrmtmax = r->nrmtmax;
  int nrmax = 0;
  for (int is = 0; is < st.nspecies; ++is) {
    if (r->nrmt[is] < 1 || r->nrmt[is] > r->nrmtmax) {
      excfv_set_error("excfv_set_rho: nrmt of species %d outside 1..nrmtmax", is + 1);
      return EXCFV_ERR_ARG;
    }
    nrmax = std::max(nrmax, r->nrmt[is]);
  }
  d.nrcmax = (nrmax + r->lradstep - 1) / r->lradstep;
  const int nlomax = std::max(st.nlomax, 1);
  const int L1 = r->lmaxvr + 1;
  std::vector<int> first(st.natmtot, -1);
  for (int a = 0; a < st.natmtot && a < (int)st.h_lo_first.size(); ++a) first[a] = st.h_lo_first[a];
  // Radial functions on the coarse mesh (function values only).  k_rho_psi sums
  // over every slot of an atom, so the slots that its species does not have (and
  // orbitals above lmaxvr) are zeros here: the caller's arrays may hold anything
  // there, and a NaN times the slot's zero coefficient would be a NaN.
  std::vector<double> u((size_t)d.nrcmax * st.apwordmax * L1 * st.natmtot, 0.0);
  std::vector<double> v((size_t)d.nrcmax * nlomax * st.natmtot, 0.0);
  for (int ias = 0; ias < st.natmtot; ++ias) {
    const int is = st.h_idxis[ias];
    const int nrc = (r->nrmt[is] + r->lradstep - 1) / r->lradstep;
    for (int l = 0; l < L1; ++l)
      for (int io = 0; io < st.h_apword[l + (size_t)(st.lmaxapw + 1) * is]; ++io) {
        double* dst = &u[(size_t)d.nrcmax * (io + (size_t)st.apwordmax * (l + (size_t)L1 * ias))];
        const double* src =
            r->apwfr + (size_t)r->nrmtmax * (2 * (io + (size_t)st.apwordmax * (l + (size_t)(st.lmaxapw + 1) * ias)));
        for (int irc = 0; irc < nrc; ++irc) dst[irc] = src[(size_t)irc * r->lradstep];
      }
    for (int ilo = 0; st.nlotot > 0 && ilo < std::min(st.h_nlorb[is], st.nlomax); ++ilo) {
      if (st.h_lorbl[ilo + (size_t)nlomax * is] > r->lmaxvr) continue;
      double* dst = &v[(size_t)d.nrcmax * (ilo + (size_t)nlomax * ias)];
      const double* src = r->lofr + (size_t)r->nrmtmax * (2 * (ilo + (size_t)nlomax * ias));
      for (int irc = 0; irc < nrc; ++irc) dst[irc] = src[(size_t)irc * r->lradstep];
    }
  }
  const size_t L = d.lmmaxvr;
  d.ncoef = (size_t)st.apwordmax * L * std::max(st.nstfv, 1) * st.natmtot;
  d.gang_elems = rho_gang_elems((size_t)2 * std::max(st.nstfv, 1), L1 * st.apwordmax + nlomax, L, st.natmtot);
  const size_t nst = std::max(st.nstfv, 1), nlo = (size_t)std::max(st.maxnlo, 1) * st.natmtot;
  const int rc = set_arrays(d.block, h->stream, [&](auto&& put) {
    put(&d.nrmt, r->nrmt, st.nspecies);
    put(&d.ucoarse, u.data(), u.size());
    put(&d.vcoarse, v.data(), v.size());
    put(&d.zb, r->zbshtvr, L * L);
    put(&d.rf, r->rfshtvr, L * L);
    put(&d.lo_first, first.data(), st.natmtot);
    put(&d.lorbl, st.h_lorbl.data(), st.h_lorbl.size());
    put(&d.rhomt, nullptr, L * r->nrmtmax * st.natmtot);
    put(&d.magmt, nullptr, L * r->nrmtmax * st.natmtot);
    put(&d.magmt3, nullptr, 3 * L * r->nrmtmax * st.natmtot);
    put(&d.w, nullptr, 2 * nst);
    put(&d.rtp, nullptr, L * d.nrcmax * st.natmtot);
    put(&d.gang, nullptr, d.gang_elems);
    put(&d.coef, nullptr, d.ncoef);
    put(&d.coef2, nullptr, 2 * d.ncoef);
    put(&d.coef3, nullptr, 2 * d.ncoef);
    put(&d.lo1, nullptr, nlo * nst);
    put(&d.lo2, nullptr, 2 * nlo * nst);
    put(&d.lo3, nullptr, 2 * nlo * nst);
    put(&d.esv, nullptr, 2 * nst * nst);
  });
  if (rc) return rc;
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  d.basis = Basis(st);
  d.ready = true;
  return EXCFV_OK;
}

// Whether the coefficients come from the packed matching coefficients (ws.Apk,
// lm up to lmaxmat) instead of the reference layout.
bool rho_packed(const excfv_handle* h) { return h->rho.lmaxvr <= h->st.lmaxmat; }

// rhomt += the k-point's density; evec (ld ldev) on the device, weights on the
// host, the matching coefficients in ws.Apk or (!rho_packed) apwalm
int stage_rhovalk(excfv_handle* h, int ngp, int ngkmax, const cplx* apwalm, const cplx* evec, long long ldev,
                  const double* wocc, double epsocc) {
  DevStatic& st = h->st;
  DevRho& d = h->rho;
  cudaStream_t s = h->stream;
  const int L = d.lmmaxvr;
  // rhovalk.f90:74: states with |wkpt occsv| <= epsocc do not contribute; those
  // above the last one that does need no coefficients
  std::vector<double> w(st.nstfv);
  int nst = 0;
  for (int j = 0; j < st.nstfv; ++j) {
    w[j] = (fabs(wocc[j]) > epsocc) ? wocc[j] : 0.0;
    if (w[j] != 0.0) nst = j + 1;
  }
  if (nst == 0) return EXCFV_OK;
  CUDA_TRY(cudaMemcpyAsync(d.w, w.data(), sizeof(double) * nst, cudaMemcpyHostToDevice, s));
  const bool packed = rho_packed(h);
  // c(lm io, j, ias) = sum_G apwalm(G, io, lm, ias) evec(G, j): rows up to lmaxvr
  int M = st.apwordmax * L;
  if (packed) {
    M = 0;
    for (int is = 0; is < st.nspecies; ++is) {
      int rows = 0;
      for (int l = 0; l <= d.lmaxvr; ++l) rows += (2 * l + 1) * st.h_apword[l + (size_t)(st.lmaxapw + 1) * is];
      M = std::max(M, rows);
    }
  }
  ZgemmArgs z;
  z.m = M; z.n = nst; z.k = ngp;
  z.alpha = cmk(1.0, 0.0); z.beta = cmk(0.0, 0.0);
  if (packed) {
    z.A = h->ws.Apk; z.lda = (long long)st.natmtot * st.maxaa; z.strideA = st.maxaa;
  } else {
    z.A = apwalm; z.lda = ngkmax; z.strideA = (long long)ngkmax * st.apwordmax * st.lmmaxapw;
  }
  z.B = evec; z.ldb = ldev; z.strideB = 0;
  z.C = d.coef; z.ldc = M; z.strideC = (long long)M * nst;
  z.batch = st.natmtot; z.uplo_c = TRI_NONE; z.tri_a = TRI_NONE; z.tri_b = TRI_NONE;
  z.splitk = 1; z.part = nullptr; z.kdec = 0;
  bind_gemm_ctx(h);
  int rc;
  if (M > 0 && (rc = zgemm(s, packed ? OP_N : OP_T, OP_N, z))) return rc;
  RhoArgs a;
  a.ias0 = 0; a.natmtot = st.natmtot; a.lmaxvr = d.lmaxvr; a.lmmaxvr = L; a.lradstep = d.lradstep; a.nrcmax = d.nrcmax;
  a.nrmtmax = d.nrmtmax; a.apwordmax = st.apwordmax; a.nlomax = std::max(st.nlomax, 1);
  a.maxnlo = std::max(st.maxnlo, 1); a.nst = nst; a.ngp = ngp;
  a.idxis = st.idxis; a.nrmt = d.nrmt; a.apword = st.apword; a.lmaxapw = st.lmaxapw;
  a.lo_lm = st.lo_lm; a.lo_ilo = st.lo_ilo; a.lo_first = d.lo_first; a.lorbl = d.lorbl;
  a.ucoarse = d.ucoarse; a.vcoarse = d.vcoarse; a.zb = d.zb; a.rf = d.rf;
  a.coef = d.coef; a.ldc = M; a.cstride = (long long)M * nst;
  a.fofl = packed ? st.fofl : nullptr; a.lmmaxapw = st.lmmaxapw;
  a.evec = evec; a.ldev = ldev; a.w = d.w; a.rhomt = d.rhomt;
  a.locoef = nullptr; a.ldlo = 0; a.cut = 1; a.magmt = nullptr; a.msign = 0.0;
  return rho_mt(h, a);
}

// rhomt and magmt += the k-point's density with second-variational vectors
// evecsv (2 nstfv x 2 nstfv, device, ld 2 nstfv) for a collinear field; the
// weights wocc (2 nstfv) on the host
namespace {

// The first-variational coefficients of every state (wavefmt_add's cut-off
// applied), the LO rows, and the weights (0 below epsocc) for the branches
// with second-variational vectors; then RhoArgs for the coarse-mesh kernels.
int sv_prepare(excfv_handle* h, int ngp, int ngkmax, const cplx* apwalm, const cplx* evec, long long ldev,
               const double* wocc, double epsocc, RhoArgs& a) {
  DevStatic& st = h->st;
  DevRho& d = h->rho;
  cudaStream_t s = h->stream;
  const int n = st.nstfv, n2 = 2 * st.nstfv;
  const int L = d.lmmaxvr;
  const long long M = (long long)st.apwordmax * L;
  const int nlo1 = std::max(st.maxnlo, 1);
  const long long LM = (long long)nlo1 * st.natmtot;
  std::vector<double> w(n2);
  for (int j = 0; j < n2; ++j) w[j] = (fabs(wocc[j]) > epsocc) ? wocc[j] : 0.0;
  CUDA_TRY(cudaMemcpyAsync(d.w, w.data(), sizeof(double) * n2, cudaMemcpyHostToDevice, s));
  CUDA_TRY(cudaStreamSynchronize(s));  // w is a host temporary
  bind_gemm_ctx(h);
  int rc;
  ZgemmArgs z;
  z.m = (int)M; z.n = n; z.k = ngp;
  z.alpha = cmk(1.0, 0.0); z.beta = cmk(0.0, 0.0);
  z.A = apwalm; z.lda = ngkmax; z.strideA = (long long)ngkmax * st.apwordmax * st.lmmaxapw;
  z.B = evec; z.ldb = ldev; z.strideB = 0;
  z.C = d.coef; z.ldc = M; z.strideC = M * n;
  z.batch = st.natmtot; z.uplo_c = TRI_NONE; z.tri_a = TRI_NONE; z.tri_b = TRI_NONE;
  z.splitk = 1; z.part = nullptr; z.kdec = 0;
  if ((rc = zgemm(s, OP_T, OP_N, z))) return rc;
  const long long nc = M * n * st.natmtot;
  k_rho_cut<<<(unsigned)((nc + 255) / 256), 256, 0, s>>>(nc, d.coef);
  count_launch();
  k_rho_gather_lo<<<(unsigned)((LM * n + 255) / 256), 256, 0, s>>>(st.natmtot, nlo1, n, ngp, st.lo_lm,
                                                                    d.lo_first, evec, ldev, d.lo1);
  count_launch();
  CUDA_TRY(cudaGetLastError());
  a.ias0 = 0; a.natmtot = st.natmtot; a.lmaxvr = d.lmaxvr; a.lmmaxvr = L; a.lradstep = d.lradstep; a.nrcmax = d.nrcmax;
  a.nrmtmax = d.nrmtmax; a.apwordmax = st.apwordmax; a.nlomax = std::max(st.nlomax, 1);
  a.maxnlo = nlo1; a.nst = n2; a.ngp = ngp;
  a.idxis = st.idxis; a.nrmt = d.nrmt; a.apword = st.apword; a.lmaxapw = st.lmaxapw;
  a.lo_lm = st.lo_lm; a.lo_ilo = st.lo_ilo; a.lo_first = d.lo_first; a.lorbl = d.lorbl;
  a.ucoarse = d.ucoarse; a.vcoarse = d.vcoarse; a.zb = d.zb; a.rf = d.rf; a.coef = d.coef2;
  a.ldc = M; a.cstride = M * n2; a.fofl = nullptr; a.lmmaxapw = st.lmmaxapw;
  a.evec = evec; a.ldev = ldev; a.locoef = d.lo2; a.ldlo = LM; a.cut = 0;
  a.w = d.w; a.rhomt = d.rhomt; a.magmt = d.magmt; a.msign = 1.0;
  return EXCFV_OK;
}

// one spinor component's coefficients: cf = coef esv_spin (per atom), lo = lo1 esv_spin
int sv_spin(excfv_handle* h, int spin, const cplx* evecsv, double epsocc, cplx* cf, cplx* lo) {
  DevStatic& st = h->st;
  DevRho& d = h->rho;
  cudaStream_t s = h->stream;
  const int n = st.nstfv, n2 = 2 * st.nstfv;
  const long long M = (long long)st.apwordmax * d.lmmaxvr;
  const long long LM = (long long)std::max(st.maxnlo, 1) * st.natmtot;
  k_rho_esv<<<(unsigned)(((long long)n * n2 + 255) / 256), 256, 0, s>>>(n, spin, evecsv, epsocc, d.esv);
  count_launch();
  CUDA_TRY(cudaGetLastError());
  ZgemmArgs g;
  g.m = (int)M; g.n = n2; g.k = n;
  g.alpha = cmk(1.0, 0.0); g.beta = cmk(0.0, 0.0);
  g.A = d.coef; g.lda = M; g.strideA = M * n;
  g.B = d.esv; g.ldb = n; g.strideB = 0;
  g.C = cf; g.ldc = M; g.strideC = M * n2;
  g.batch = st.natmtot; g.uplo_c = TRI_NONE; g.tri_a = TRI_NONE; g.tri_b = TRI_NONE;
  g.splitk = 1; g.part = nullptr; g.kdec = 0;
  int rc;
  if ((rc = zgemm(s, OP_N, OP_N, g))) return rc;
  g.m = (int)LM; g.A = d.lo1; g.lda = LM; g.strideA = 0;
  g.C = lo; g.ldc = LM; g.strideC = 0; g.batch = 1;
  return zgemm(s, OP_N, OP_N, g);
}

size_t rho_nc_smem(int L) {
  return sizeof(cplx) * ((size_t)L * L + (size_t)2 * L * JB) + sizeof(double) * 4 * L;
}

}  // namespace

int stage_rhovalk_sv(excfv_handle* h, int ngp, int ngkmax, const cplx* apwalm, const cplx* evec, long long ldev,
                     const cplx* evecsv, const double* wocc, double epsocc) {
  DevRho& d = h->rho;
  RhoArgs a;
  int rc;
  if ((rc = sv_prepare(h, ngp, ngkmax, apwalm, evec, ldev, wocc, epsocc, a))) return rc;
  for (int spin = 0; spin < 2; ++spin) {
    if ((rc = sv_spin(h, spin, evecsv, epsocc, d.coef2, d.lo2))) return rc;
    a.msign = spin == 0 ? 1.0 : -1.0;
    if ((rc = rho_mt(h, a))) return rc;
  }
  return EXCFV_OK;
}

int stage_rhovalk_sv_nc(excfv_handle* h, int ngp, int ngkmax, const cplx* apwalm, const cplx* evec, long long ldev,
                        const cplx* evecsv, const double* wocc, double epsocc) {
  DevRho& d = h->rho;
  cudaStream_t s = h->stream;
  RhoArgs a;
  int rc;
  if ((rc = sv_prepare(h, ngp, ngkmax, apwalm, evec, ldev, wocc, epsocc, a))) return rc;
  if ((rc = sv_spin(h, 0, evecsv, epsocc, d.coef2, d.lo2)) || (rc = sv_spin(h, 1, evecsv, epsocc, d.coef3, d.lo3)))
    return rc;
  const size_t smem = rho_nc_smem(d.lmmaxvr);
  CUDA_TRY(raise_smem_limit(k_rho_mt_nc, rho_nc_smem((RHO_LMAX + 1) * (RHO_LMAX + 1))));
  dim3 grid(d.nrcmax, h->st.natmtot);
  k_rho_mt_nc<<<grid, 128, smem, s>>>(a, d.coef3, d.lo3, d.magmt3);
  count_launch();
  CUDA_TRY(cudaGetLastError());
  return EXCFV_OK;
}
