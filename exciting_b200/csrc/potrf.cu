// Cholesky factorisation O = U^H U (upper) and the inverse factor U^-1.
//
// ZHEGVX starts with ZPOTRF('U') on the overlap matrix
// (external/LAPACK/zhegvx.f:410).  Here it is blocked right-looking with a
// 64-wide panel: one CTA factors the diagonal block in shared memory and
// also inverts it; the row panel is then one GEMM with the inverted diagonal
// block, and the trailing update one upper-triangle GEMM.  The inverse
// factor U^-1 (used for the two-sided reduction and the back-transform) is
// built block column by block column from the inverted diagonal blocks:
//   Ui(0:j, j) = -Ui(0:j, 0:j) * U(0:j, j) * inv(U_jj).
// A non-positive pivot records its 1-based position in status[ST_POTRF]; the
// remaining panels then return immediately.
#include "handle.cuh"

namespace {

constexpr int NBP = 64;

// One CTA factors the b x b diagonal block (b <= 64) and inverts the factor: a
// right-looking elimination of [A | I] in steps of four columns, which leaves
// U = L^H in A and L^-1 = (U^-1)^H in the unit part.  Per step
//   the two pivot warps, a thread per active column (A's columns right of the step,
//   the unit part's up to it), each factor the 4 x 4 diagonal block redundantly in
//   registers and solve their own column's four entries;
//   --- barrier ---
//   the pivot warps update the four rows of the next step, each thread its own
//   column, and go on to the next diagonal block at once (a barrier of their own);
//   beside them the other 14 warps update the rows below, four rows at a time with
//   the four pivot rows
// so a step has one block barrier and takes the longer of the pivots' chain (four
// reciprocal square roots) and the update.  A 64-block takes 24 us and a 22-block
// 13; with all warps updating between two barriers it was 30 and 15, a column at a
// time with 1024 threads and ~260 barriers 57 us for either.
constexpr int LDB = 65;
constexpr int DT = 512;

// Cholesky of the Hermitian 4 x 4 block at A(j, j) (upper part read): u above
// the diagonal, r = 1 / U(k, k).  Returns 0, or the 1-based first pivot that
// is not positive.
__device__ __forceinline__ int chol4(const cplx* A, int j, cplx (&u)[4][4], double (&r)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int c = k; c < 4; ++c) u[k][c] = A[(j + k) * LDB + j + c];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double d = u[k][k].x;
    if (!(d > 0.0)) return k + 1;
    r[k] = rsqrt(d);
#pragma unroll
    for (int c = k; c < 4; ++c) u[k][c] = (c == k) ? cmk(d * r[k], 0.0) : cscale(u[k][c], r[k]);
#pragma unroll
    for (int k2 = k + 1; k2 < 4; ++k2)
#pragma unroll
      for (int c = k2; c < 4; ++c) u[k2][c] = csub(u[k2][c], cmulc(u[k][k2], u[k][c]));
  }
  return 0;
}

__device__ __forceinline__ void potrf_diag_block(int n, int kb, cplx* O, long long ld, cplx* Ui, int* status) {
  extern __shared__ __align__(16) unsigned char dsm[];
  cplx* A = reinterpret_cast<cplx*>(dsm);   // 64 x LDB, row-major [r][c]
  cplx* Y = A + NBP * LDB;                  // the unit part, L^-1 at the end
  __shared__ int s_fail[2];  // by the parity of the step: the pivot warps run ahead
  if (status[ST_POTRF] != 0) return;
  const int b = min(NBP, n - kb);
  const int lim = (b + 3) / 4 * 4;          // rows past b are padded with the identity
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int t = tid; t < NBP * NBP; t += DT) {
    const int r = t % NBP, c = t / NBP;  // coalesced along r
    cplx a = cmk(r == c ? 1.0 : 0.0, 0.0);
    Y[r * LDB + c] = a;
    if (r < b && c < b && r <= c) a = O[(kb + r) + ld * (kb + c)];
    if (r == c) a.y = 0.0;
    A[r * LDB + c] = a;
  }
  if (tid < 2) s_fail[tid] = 0;
  __syncthreads();
  for (int j = 0; j < lim; j += 4) {
    int& fail = s_fail[(j >> 2) & 1];
    cplx u[4][4], x[4];
    double r[4];
    // columns right of the step in A, then columns 0 .. j + 3 of the unit part
    const bool mineA = tid < 60 - j;
    cplx* col = mineA ? A + j + 4 + tid : Y + tid - (60 - j);
    if (tid < 64) {
      const int bad = chol4(A, j, u, r);
      if (bad) {
        if (tid == 0) fail = j + bad;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          x[k] = col[(j + k) * LDB];
#pragma unroll
          for (int q = 0; q < k; ++q) x[k] = csub(x[k], cmulc(u[q][k], x[q]));
          x[k] = cscale(x[k], r[k]);
          col[(j + k) * LDB] = x[k];
        }
      }
    }
    __syncthreads();  // the pivot rows are there, the rows from j + 4 on have the last step's update
    if (fail) {
      if (tid == 0 && fail <= b) atomicCAS(&status[ST_POTRF], 0, kb + fail);
      return;
    }
    // rows i of both parts: row -= sum_k conj(U(j+k, i)) (row j+k)
    if (tid < 64) {
      if (tid == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int c = k; c < 4; ++c) A[(j + k) * LDB + j + c] = u[k][c];
      }
      if (j + 4 < lim) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = j + 4 + q;
          cplx v = col[i * LDB];
#pragma unroll
          for (int k = 0; k < 4; ++k) v = csub(v, cmulc(A[(j + k) * LDB + i], x[k]));
          col[i * LDB] = v;
        }
      }
      asm volatile("bar.sync 1, 64;" ::: "memory");
    } else {
      const int i0 = j + 6 + warp;
      if (i0 < lim) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = lane + 32 * h;
          const bool inA = c >= j + 4;
          cplx* M = inA ? A : Y;
          if (c >= lim) continue;
          cplx pv[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) pv[k] = M[(j + k) * LDB + c];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + 14 * q;
            if (i >= lim || (inA && c < i)) continue;
            cplx v = M[i * LDB + c];
#pragma unroll
            for (int k = 0; k < 4; ++k) v = csub(v, cmulc(A[(j + k) * LDB + i], pv[k]));
            M[i * LDB + c] = v;
          }
        }
      }
    }
  }
  __syncthreads();
  for (int t = tid; t < NBP * NBP; t += DT) {
    const int r = t % NBP, c = t / NBP;
    if (r < b && c < b && r <= c) {
      O[(kb + r) + ld * (kb + c)] = A[r * LDB + c];
      Ui[(kb + r) + ld * (kb + c)] = cconj(Y[c * LDB + r]);
    }
  }
}

__global__ void __launch_bounds__(DT) k_potrf_diag(int n, int kb, cplx* O, long long ld, cplx* Ui,
                                                   int* status) {
  potrf_diag_block(n, kb, O, ld, Ui, status);
}

// Grouped form: CTA b factors diagonal block kb of problem b.
__global__ void __launch_bounds__(DT) k_potrf_diag_grouped(const PotrfProb* __restrict__ probs, int kb) {
  const PotrfProb p = probs[blockIdx.x];
  potrf_diag_block(p.n, kb, p.O, p.ld, p.Ui, p.status);
}

}  // namespace

int potrf_smem_bytes() { return (int)(2 * sizeof(cplx) * NBP * LDB); }
int potrf_block() { return NBP; }

int potrf_diag_grouped(cudaStream_t s, const PotrfProb* d_probs, int nprob, int kb) {
  if (nprob <= 0) return EXCFV_OK;
  const int smem = potrf_smem_bytes();
  CUDA_TRY(cudaFuncSetAttribute(k_potrf_diag_grouped, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_potrf_diag_grouped<<<nprob, DT, smem, s>>>(d_probs, kb); count_launch();
  CUDA_TRY(cudaGetLastError());
  return EXCFV_OK;
}

int potrf_upper(excfv_handle* h, int n, cplx* O, cplx* Ui, long long ld) {
  cudaStream_t s = h->stream;
  const cplx one = cmk(1.0, 0.0), mone = cmk(-1.0, 0.0);
  const int smem = (int)(2 * sizeof(cplx) * NBP * LDB);
  CUDA_TRY(cudaFuncSetAttribute(k_potrf_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  for (int kb = 0; kb < n; kb += NBP) {
    const int b = min(NBP, n - kb);
    k_potrf_diag<<<1, DT, smem, s>>>(n, kb, O, ld, Ui, h->ws.status); count_launch();
    CUDA_TRY(cudaGetLastError());
    const int rest = n - kb - b;
    if (rest <= 0) break;
    cplx* panel = O + kb + ld * (kb + b);
    // U(kb, rest) = inv(U_kk)^H A(kb, rest)   (in place: one row tile per CTA)
    int rc = zgemm1(s, OP_C, OP_N, b, rest, b, one, Ui + kb + ld * kb, ld, panel, ld,
                    cmk(0.0, 0.0), panel, ld, TRI_NONE, TRI_LOWER, TRI_NONE);
    if (rc) return rc;
    // A(rest, rest) -= U(kb, rest)^H U(kb, rest), upper triangle: an A^H B
    // product with K = 64 whose operand tiles a TMA ring brings three stages
    // ahead (zgemm_tma.cu), so the K loop is not bound by load latency
    const cplx* Pp[1] = {panel};
    cplx* Cp[1] = {O + (kb + b) + ld * (kb + b)};
    rc = zgemm_cn_tma(h, rest, rest, b, mone, Pp, ld, Pp, ld, one, Cp, ld, 1, TRI_UPPER);
    if (rc) return rc;
  }
  return EXCFV_OK;
}

// Ui = U^-1 (upper).  The diagonal NBP-blocks of Ui were written by
// k_potrf_diag; pairs of inverted blocks are merged level by level,
//   inv([[U11, U12], [0, U22]]) = [[X11, -X11 U12 X22], [0, X22]],
// with all pairs of one level in one batched GEMM (log2(n / NBP) levels).
// scratch: n x n complex.
int trtri_upper(excfv_handle* h, int n, const cplx* U, cplx* Ui, long long ld, cplx* scratch) {
  cudaStream_t s = h->stream;
  const cplx one = cmk(1.0, 0.0), mone = cmk(-1.0, 0.0), zero = cmk(0.0, 0.0);
  for (int bs = NBP; bs < n; bs *= 2) {
    const int nfull = n / (2 * bs);             // pairs whose second block is complete
    const int rem = n - nfull * 2 * bs;          // rows left after the full pairs
    // full pairs, batched
    if (nfull > 0) {
      const long long step = 2LL * bs * (ld + 1);
      ZgemmArgs g;
      g.m = bs; g.n = bs; g.k = bs; g.kdec = 0; g.alpha = one; g.beta = zero;
      g.A = U + ld * bs; g.lda = ld; g.strideA = step;              // U12
      g.B = Ui + bs * (ld + 1); g.ldb = ld; g.strideB = step;        // X22
      g.C = scratch; g.ldc = bs; g.strideC = (long long)bs * bs;     // T = U12 X22
      g.batch = nfull; g.uplo_c = TRI_NONE; g.tri_a = TRI_NONE; g.tri_b = TRI_UPPER;
      g.splitk = 1; g.part = nullptr;
      int rc = zgemm(s, OP_N, OP_N, g);
      if (rc) return rc;
      g.alpha = mone;
      g.A = Ui; g.strideA = step;                                    // X11
      g.B = scratch; g.ldb = bs; g.strideB = (long long)bs * bs;     // T
      g.C = Ui + ld * bs; g.ldc = ld; g.strideC = step;              // X12
      g.tri_a = TRI_UPPER; g.tri_b = TRI_NONE;
      rc = zgemm(s, OP_N, OP_N, g);
      if (rc) return rc;
    }
    // a trailing pair whose second block is shorter than bs
    if (rem > bs) {
      const int a0 = nfull * 2 * bs, d0 = a0 + bs, sd = n - d0;
      cplx* T = scratch + (size_t)nfull * bs * bs;
      int rc = zgemm1(s, OP_N, OP_N, bs, sd, sd, one, U + a0 + ld * d0, ld, Ui + d0 + ld * d0, ld,
                      zero, T, bs, TRI_NONE, TRI_NONE, TRI_UPPER);
      if (rc) return rc;
      rc = zgemm1(s, OP_N, OP_N, bs, sd, bs, mone, Ui + a0 + ld * a0, ld, T, bs, zero,
                  Ui + a0 + ld * d0, ld, TRI_NONE, TRI_UPPER, TRI_NONE);
      if (rc) return rc;
    }
  }
  return EXCFV_OK;
}
