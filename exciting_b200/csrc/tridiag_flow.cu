// The panel of the Householder tridiagonal reduction (tridiag.cu: NBT columns,
// then a rank-2 NBT update) as a dataflow between thread blocks, without grid
// barriers.
//
// The barrier form spends about 10 us per column whatever the block's size: two
// grid barriers with their fences, atomics that have to drain before them, loads
// that can start only after them.  Here every number that crosses thread blocks
// travels as a 32-byte word of four 64-bit pairs {32 bits of data, tag}, tag =
// column + 1: a complex number whose every part says which column it belongs to,
// so no ordering between the parts or with other words is needed (a 64-bit access
// is the unit that the memory model keeps whole; the word goes as one 256-bit
// access).  A reader polls the word itself, so one trip through L2 replaces store,
// fence, counter, poll and load, and sums have a fixed order.  Thread blocks have one of two roles:
//
//   owners   (NO blocks, MC chunks of 64 rows each): the panel's V and W rows and
//            the column x in shared memory.  For column c they publish x; publish
//            partial sums over their rows of V^H x, W^H x, |x|^2, diag(C)|x|^2 and
//            x^H C(:, c+1); derive the reflector from the totals (every owner from
//            the same words, hence the same bits); collect the parts of y = C22 x
//            for their rows, form w and the next column, which only needs
//            w(c+1) besides own rows.
//   workers  (the other blocks): fixed equal shares of the lower triangle's
//            64 x 16 (FP64) or 64 x 32 (complex64) tiles.  They take x, publish the
//            row part A x and the column part A^H x of their tiles and Re(x^H A x),
//            and know nothing of the reflector: v = e1 + scale x is applied by the
//            owners (C22 v = C(:, c+1) + scale C22 x).  A share that fits the ring
//            of tiles in shared memory is loaded once per panel; a larger one is
//            streamed by TMA each column, ahead of the consumers.  One warp of each
//            worker adds up some of the owners' partial sums, in the time the
//            products take.
//
// Words are double buffered by the parity of the column.  A word of column c is
// overwritten at column c + 2, by a writer that has seen data of column c + 1 which
// every reader of the old word sent after reading it (an owner sends x of column
// c + 1 only after every worker's Re(x^H A x) of column c; a worker's products of
// column c + 1 need x from owners that finished column c; the totals of a column
// need all owners' partial sums).  The words are zeroed before each reduction, and
// tags count from 1, so words of an earlier one are never taken.
//
// Every wait is bounded: it gives up when the time limit has passed or another
// wait of the launch has given up (status[ST_BARRIER]); all threads of a block then
// leave at their next block barrier, which carries the decision.
//
// Measured against the barrier form over the same columns (all panels of one solve,
// the last 320 columns and the updates apart): FP64 order 715 4.15 -> 2.45 ms, 1964
// 19.3 -> 11.6 ms; complex64 order 1901 17.8 -> 10.2 ms.  A column takes 6.0 us at
// order 700, 6.7 at 1450, 7.4 at 1600, from where a worker's tiles no longer all fit
// its ring, and 10.2 at 1964 (barrier form 10, 13.5, 13.5 and 14.8).  Of order 5028
// the columns below 3136 go from 39.0 to 29.6 ms; those above, with two chunks per
// owner and every tile from HBM, are slower than the barrier form's since that got
// its present inner loop (69.2 against 58.9 ms).
#include "tridiag_dev.cuh"

namespace {

constexpr int FT = 256;              // main threads (8 warps)
constexpr int FTOT = FT + 64;        // and an auxiliary and a producer warp
constexpr int NK = 2 * NBT + 2;      // values summed over the owners: S, T, (norm, dg), h
constexpr int RUNMAX = 12;           // runs (parts of one row of tiles) per worker
constexpr int FSTAGES = 12;          // most ring slots

struct __align__(32) word {
  unsigned long long v[4];
};

// loads a word; true when all four parts carry the tag
__device__ __forceinline__ void ldw(const word* p, unsigned long long (&v)[4]) {
  asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
               : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void stw(word* p, cplx z, unsigned tag) {
  const unsigned long long x = (unsigned long long)__double_as_longlong(z.x),
                           y = (unsigned long long)__double_as_longlong(z.y), t = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(t | (x & 0xffffffffull)),
               "l"(t | (x >> 32)), "l"(t | (y & 0xffffffffull)), "l"(t | (y >> 32))
               : "memory");
}

struct Waiter {
  int* status;
  long long limit_ns;
  bool bad;
};

// The rarely taken end of a poll round, out of line: true to give up.
__device__ __noinline__ bool poll_expired(int* status, long long limit_ns, long long& t0) {
  const long long t = gtimer();
  if (t0 == 0) t0 = t;
  if (*(volatile int*)&status[ST_BARRIER] != 0) return true;
  if (t - t0 > limit_ns) {
    atomicAdd(&status[ST_BARRIER], 1);
    return true;
  }
  return false;
}

// All lanes of a warp poll, each the words whose mask bit is set, until all of
// the warp's carry the tag; the others read 0 (their pointers must be readable).
// The warp stays together: lanes that left one by one ran everything up to the
// next shuffle one after another (2 us for a dozen lanes).
// Only the first `cnt` (the same in every lane) are loaded at all.
template <int N>
__device__ __forceinline__ void poll(const word* const (&ptr)[N], unsigned mask, unsigned tag, cplx (&val)[N],
                                     Waiter& w, int cnt = N) {
  unsigned it = 0;
  long long t0 = 0;
  for (;;) {
    unsigned long long v[N][4];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      if (q < cnt) ldw(ptr[q], v[q]);
      else v[q][0] = v[q][1] = v[q][2] = v[q][3] = 0;
    }
    unsigned diff = 0;  // any tag that does not match, over the wanted words
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const unsigned d = ((unsigned)(v[q][0] >> 32) ^ tag) | ((unsigned)(v[q][1] >> 32) ^ tag) |
                         ((unsigned)(v[q][2] >> 32) ^ tag) | ((unsigned)(v[q][3] >> 32) ^ tag);
      const bool on = mask >> q & 1u;
      diff |= on ? d : 0u;
      val[q].x = on ? __hiloint2double((int)v[q][1], (int)v[q][0]) : 0.0;
      val[q].y = on ? __hiloint2double((int)v[q][3], (int)v[q][2]) : 0.0;
    }
    if (__all_sync(0xffffffffu, diff == 0) || w.bad) return;
    if ((++it & 63u) == 0) {
      const bool over = poll_expired(w.status, w.limit_ns, t0);
      if (__any_sync(0xffffffffu, over)) w.bad = true;  // the same in every lane
    }
  }
}

// Block barriers that carry the decision to leave (true if any thread is bad).
__device__ __forceinline__ bool bar_main(bool bad) {
  unsigned r;
  asm volatile(
      "{ .reg .pred p, q; setp.ne.u32 q, %1, 0; bar.red.or.pred p, 1, %2, q; selp.u32 %0, 1, 0, p; }"
      : "=r"(r)
      : "r"(bad ? 1u : 0u), "n"(FT)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ bool bar_owner(bool bad) {
  unsigned r;
  asm volatile(
      "{ .reg .pred p, q; setp.ne.u32 q, %1, 0; bar.red.or.pred p, 2, %2, q; selp.u32 %0, 1, 0, p; }"
      : "=r"(r)
      : "r"(bad ? 1u : 0u), "n"(FT + 32)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void bar_sync_main() { asm volatile("bar.sync 1, %0;" ::"n"(FT) : "memory"); }

template <typename T2>
struct FlowArgs {
  int n;
  long long ld;
  T2* C;
  T2* VW;   // n x 2 NBT: [V | W] of the panel
  T2* WV;   // n x 2 NBT: [W | V]
  double* d;
  double* e;
  cplx* tau;
  int* status;
  int p, nbp, final_panel;
  int NO, NWT, NW;    // owners, worker blocks, workers with tiles
  int nt;             // 64-row blocks from row p
  int stages, ecap;   // ring slots, columns of x a worker may stage
  long long wait_ns;
  unsigned planted;
  // words (two buffers each, `*_par` words apart)
  word *X, *COL, *ROW, *VAV, *PART, *TOT, *RVW;
  long long x_par, col_par, row_par, vav_par, part_par, tot_par, rvw_par;
};

// Units (tiles of BC columns) of the lower 64 x 64 blocks in folded row order:
// row k of blocks is followed by row nt-1-k, then the middle one; row I has
// (I + 1) BPT units.
template <int BPT>
struct Fold {
  int nt, npair;
  long long P, U;
  __device__ explicit Fold(int nt_) : nt(nt_), npair(nt_ >> 1) {
    P = (long long)(nt + 1) * BPT;
    U = (long long)nt * (nt + 1) / 2 * BPT;
  }
  // row and first unit of the run that holds unit t, and the row's end
  __device__ void run_of(long long t, int& I, long long& rs, long long& re) const {
    if (t < npair * P) {
      const int k = (int)(t / P);
      const long long base = k * P, mid = base + (long long)(k + 1) * BPT;
      if (t < mid) { I = k; rs = base; re = mid; }
      else { I = nt - 1 - k; rs = mid; re = base + P; }
    } else {
      I = npair; rs = npair * P; re = rs + (long long)(npair + 1) * BPT;
    }
  }
  __device__ long long row_begin(int I) const {
    if (I < npair) return I * P;
    if ((nt & 1) && I == npair) return npair * P;
    const int k = nt - 1 - I;
    return k * P + (long long)(k + 1) * BPT;
  }
  __device__ int rank(int I) const {  // position of row I in the order
    if (I < npair) return 2 * I;
    if ((nt & 1) && I == npair) return 2 * npair;
    return 2 * (nt - 1 - I) + 1;
  }
};

// The worker that holds unit t when worker w has units [U w / NW, U (w+1) / NW).
__device__ __forceinline__ int worker_of(long long t, long long U, int NW) {
  return (int)(((t + 1) * NW - 1) / U);
}
__device__ __forceinline__ int col_at(int I, int j) {  // column part of block row I, column j
  return 32 * I * (I + 1) + j;
}

// ---------------------------------------------------------------------------
template <typename T2>
__device__ void flow_worker(const FlowArgs<T2>& a, const CUtensorMap* tmap, unsigned char* dsm, int w) {
  constexpr int BC = TILE_COLS<T2>, BPT = 64 / BC, SPU = BC / 16;  // 16-column groups per unit
  constexpr int TILE = RCH * BC;
  constexpr unsigned BYTES = TILE * sizeof(T2);
  __shared__ __align__(8) uint64_t s_full[FSTAGES], s_empty[FSTAGES];
  __shared__ int s_nrun, s_I[RUNMAX], s_b0[RUNMAX], s_b1[RUNMAX], s_off[RUNMAX];
  __shared__ cplx s_red[2][FT / 32][64];
  __shared__ double s_v[4];
  T2* ring = reinterpret_cast<T2*>(dsm);
  T2* sx = reinterpret_cast<T2*>(dsm + (size_t)a.stages * BYTES);   // x of the share's columns
  cplx* sxr = reinterpret_cast<cplx*>(sx + a.ecap);                  // x of the runs' rows
  int* s_map = reinterpret_cast<int*>(sxr + RUNMAX * 64);            // row of every staged entry
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Fold<BPT> F(a.nt);
  const bool has = w < a.NW;
  const long long u0 = has ? F.U * w / a.NW : 0, u1 = has ? F.U * (w + 1) / a.NW : 0;
  const int mine = (int)(u1 - u0);
  const bool resident = mine <= a.stages;
  if (tid == 0) {
    for (int q = 0; q < a.stages; ++q) {
      mbar_init(&s_full[q], 1);
      mbar_init(&s_empty[q], FT / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    int nr = 0, off = 0;
    for (long long t = u0; t < u1; ++nr) {
      int I;
      long long rs, re;
      F.run_of(t, I, rs, re);
      const long long e = min(re, u1);
      s_I[nr] = I;
      s_b0[nr] = (int)(t - rs);
      s_b1[nr] = (int)(e - rs);
      s_off[nr] = off;
      off += (int)(e - t) * BC;
      t = e;
    }
    s_nrun = nr;
  }
  __syncthreads();
  const int nrun = s_nrun;
  Waiter wt{a.status, a.wait_ns, false};

  if (warp == FT / 32 + 1) {  // ---- producer
    if (lane != 0 || !has) return;
    unsigned q = 0;
    const int rounds = resident ? 1 : a.nbp;
    bool ok = true;
    for (int i = 0; i < rounds && ok; ++i)
      for (int k = 0; k < nrun && ok; ++k)
        for (int b = s_b0[k]; b < s_b1[k]; ++b, ++q) {
          const unsigned slot = q % a.stages;
          if (q >= (unsigned)a.stages &&
              !mbar_wait_ok(&s_empty[slot], ((q / a.stages) - 1u) & 1u, a.status, a.wait_ns)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&s_full[slot], BYTES);
          tma_tile(ring + (size_t)slot * TILE, tmap, 2 * (a.p + s_I[k] * 64), a.p + b * BC, &s_full[slot]);
        }
    // every copy has landed before the block's shared memory can go
    for (unsigned s = 0; s < (unsigned)a.stages && s < q; ++s) {
      const unsigned uses = q / a.stages + (s < q % a.stages ? 1u : 0u);
      const long long t0 = gtimer();
      while (!mbar_try_wait(&s_full[s], (uses - 1u) & 1u))
        if (gtimer() - t0 > a.wait_ns) break;
    }
    return;
  }

  if (warp == FT / 32) {  // ---- auxiliary warp: totals of the owners' partial sums
    for (int i = 0; i < a.nbp; ++i) {
      const int c = a.p + i, par = c & 1;
      const unsigned tag = (unsigned)c + 1u;
      for (int q = w; q < 2 * i + 2; q += a.NWT) {
        const int k = q < i ? q : (q < 2 * i ? NBT + q - i : 2 * NBT + q - 2 * i);
        const word* base = a.PART + par * a.part_par + (long long)k * a.NO;
        cplx s = cmk(0.0, 0.0);
        for (int o = lane; o < a.NO + lane; o += 64) {
          const word* ptr[2] = {base + min(o, a.NO - 1), base + min(o + 32, a.NO - 1)};
          cplx v[2];
          poll(ptr, (o < a.NO ? 1u : 0u) | (o + 32 < a.NO ? 2u : 0u), tag, v, wt);
          s = cadd(s, cadd(v[0], v[1]));
        }
        if (wt.bad) return;
        s = warp_sum(s);
        if (lane == 0) stw(a.TOT + par * a.tot_par + k, s, tag);
      }
    }
    return;
  }
  if (!has) return;

  // ---- main threads
  const int rg = tid & 15, cq = tid >> 4;
  const int ecol = mine * BC, etot = ecol + nrun * 64;
  for (int k = 0; k < nrun; ++k) {
    const int nc = (s_b1[k] - s_b0[k]) * BC;
    for (int e = tid; e < nc; e += FT) s_map[s_off[k] + e] = s_b0[k] * BC + e;
    if (tid < 64) s_map[ecol + k * 64 + tid] = s_I[k] * 64 + tid;
  }
  bar_sync_main();
  const int nrel = a.n - a.p;
  int sl = 0;        // ring slot of the next unit, and how often the ring has wrapped (streaming)
  unsigned wrap = 0;
  for (int i = 0; i < a.nbp; ++i) {
    const int c = a.p + i, par = c & 1;
    const unsigned tag = (unsigned)c + 1u;
    const unsigned xtag = tag + (i == 0 ? a.planted : 0u);
    // x of the share's columns and rows; rows up to c + 1 carry no weight.  A
    // warp first polls one word per group of 32 entries: all threads polling
    // all their words would take the L2 bandwidth that others need.
    const word* X = a.X + par * a.x_par;
    for (int g0 = 0; g0 < etot; g0 += 32 * FT) {
      const int e = min(g0 + lane * FT + warp * 32 + 31, etot - 1);
      const bool grp = g0 + lane * FT + warp * 32 < etot;
      const int rel = grp ? s_map[e] : 0;
      const word* ptr[1] = {X + rel};
      cplx v[1];
      poll(ptr, (grp && rel > i + 1 && rel < nrel) ? 1u : 0u, xtag, v, wt);
    }
    for (int e0 = tid; e0 < etot + tid; e0 += 4 * FT) {
      const word* ptr[4];
      unsigned mask = 0;
      cplx v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = e0 + q * FT;
        const int rel = e < etot ? s_map[e] : 0;
        const bool need = e < etot && rel > i + 1 && rel < nrel;
        ptr[q] = X + (need ? rel : 0);
        if (need) mask |= 1u << q;
      }
      poll(ptr, mask, xtag, v, wt);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = e0 + q * FT;
        if (e < ecol) sx[e] = fromD<T2>(v[q]);
        else if (e < etot) sxr[e - ecol] = v[q];
      }
    }
    if (bar_main(wt.bad)) return;
    double vav = 0.0;
    if (resident) { sl = 0; wrap = 0; }
    for (int k = 0; k < nrun; ++k) {
      const int I = s_I[k], b0 = s_b0[k], nsub = (s_b1[k] - b0) * SPU, off = s_off[k];
      cplx rowp[4];
      T2 xr[4], rowf[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        rowp[u] = cmk(0.0, 0.0);
        rowf[u] = fromD<T2>(cmk(0.0, 0.0));
        xr[u] = fromD<T2>(sxr[k * 64 + rg + 16 * u]);
      }
      word* cw = a.COL + par * a.col_par + col_at(I, 0);
      for (int q0 = 0; q0 < nsub; q0 += 4) {
        T2 cp[4];
#pragma unroll
        for (int z = 0; z < 4; ++z) cp[z] = fromD<T2>(cmk(0.0, 0.0));
        const int nz = min(4, nsub - q0), nu = (nz + SPU - 1) / SPU;
        const T2* tl[4 / SPU];   // the units' tiles, at this thread's column
#pragma unroll
        for (int z = 0; z < 4 / SPU; ++z) {
          int q = sl + z;
          const unsigned ph = wrap + (q >= a.stages ? 1u : 0u);
          if (q >= a.stages) q -= a.stages;
          if (z < nu && (!resident || i == 0)) mbar_wait(&s_full[q], ph & 1u, a.status, a.wait_ns);
          tl[z] = ring + (size_t)q * TILE + cq * RCH;
        }
        const T2* xq = sx + off + q0 * 16 + cq;
        const int jt0 = b0 * BC + q0 * 16 - 64 * I;  // first column against the diagonal block
        if (jt0 + 64 <= 0 && nz == 4) {
#pragma unroll
          for (int z = 0; z < 4; ++z) {
            const T2 xj = xq[z * 16];
            const T2* tile = tl[z / SPU] + (z % SPU) * 16 * RCH;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const T2 av = tile[rg + 16 * u];
              if constexpr (sizeof(T2) == 16) {
                rowp[u].x = fma(av.x, xj.x, fma(-av.y, xj.y, rowp[u].x));
                rowp[u].y = fma(av.x, xj.y, fma(av.y, xj.x, rowp[u].y));
              } else {
                rowf[u].x = fmaf(av.x, xj.x, fmaf(-av.y, xj.y, rowf[u].x));
                rowf[u].y = fmaf(av.x, xj.y, fmaf(av.y, xj.x, rowf[u].y));
              }
              cp[z].x = mad(av.x, xr[u].x, mad(av.y, xr[u].y, cp[z].x));
              cp[z].y = mad(av.x, xr[u].y, mad(-av.y, xr[u].x, cp[z].y));
            }
          }
        } else {
          // at the diagonal (or the last, incomplete quad): row part r >= j,
          // column part r > j
#pragma unroll
          for (int z = 0; z < 4; ++z) {
            if (z >= nz) continue;
            const T2 xj = xq[z * 16];
            const T2* tile = tl[z / SPU] + (z % SPU) * 16 * RCH;
            const int jt = jt0 + z * 16 + cq;  // negative left of the diagonal block
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int rl = rg + 16 * u;
              const T2 av = tile[rl];
              if (rl >= jt) {
                if constexpr (sizeof(T2) == 16) {
                  rowp[u].x = fma(av.x, xj.x, fma(-av.y, xj.y, rowp[u].x));
                  rowp[u].y = fma(av.x, xj.y, fma(av.y, xj.x, rowp[u].y));
                } else {
                  rowf[u].x = fmaf(av.x, xj.x, fmaf(-av.y, xj.y, rowf[u].x));
                  rowf[u].y = fmaf(av.x, xj.y, fmaf(av.y, xj.x, rowf[u].y));
                }
              }
              if (rl > jt) {
                cp[z].x = mad(av.x, xr[u].x, mad(av.y, xr[u].y, cp[z].x));
                cp[z].y = mad(av.x, xr[u].y, mad(-av.y, xr[u].x, cp[z].y));
              }
            }
          }
        }
        if (!resident) {
          // the slots are refilled by the async proxy: order this thread's reads before it
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            for (int z = 0; z < nu; ++z) mbar_arrive(&s_empty[sl + z >= a.stages ? sl + z - a.stages : sl + z]);
        }
        sl += nu;
        if (sl >= a.stages) {
          sl -= a.stages;
          ++wrap;
        }
        const T2 kk = scatter_sum16(cp, lane);
        const int z = 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1);
        const int j = b0 * BC + (q0 + z) * 16 + cq;
        if ((lane & 3) == 0 && z < nz && j > i && j < nrel) stw(cw + j, toD(kk), tag);
        if constexpr (sizeof(T2) == 8) {  // FP32 row sums of at most 32 terms
          if ((q0 & 31) == 28 || q0 + 4 >= nsub) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              rowp[u] = cadd(rowp[u], toD(rowf[u]));
              rowf[u] = fromD<T2>(cmk(0.0, 0.0));
            }
          }
        }
      }
      // row sums: the two column groups of a warp, then the 8 warps
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        rowp[u].x += __shfl_xor_sync(0xffffffffu, rowp[u].x, 16);
        rowp[u].y += __shfl_xor_sync(0xffffffffu, rowp[u].y, 16);
      }
      if (lane < 16) {
#pragma unroll
        for (int u = 0; u < 4; ++u) s_red[k & 1][warp][rg + 16 * u] = rowp[u];
      }
      // two runs at a time: one barrier for both
      if (!(k & 1) && k + 1 < nrun) continue;
      bar_sync_main();
      if (tid < 64 * (1 + (k & 1))) {
        const int kk = (k & ~1) + (tid >> 6), r = tid & 63;
        cplx s = cmk(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < FT / 32; ++q) s = cadd(s, s_red[kk & 1][q][r]);
        const cplx x = sxr[kk * 64 + r];
        vav += x.x * s.x + x.y * s.y;
        const int rel = s_I[kk] * 64 + r;
        if (rel > i && rel < nrel) stw(a.ROW + par * a.row_par + 64LL * (w + F.rank(s_I[kk])) + r, s, tag);
      }
      if (k + 1 < nrun) bar_sync_main();  // s_red is free again
    }
    // Re(x^H A x) of the share: its row parts count twice, the diagonal is
    // taken off by the owners
    for (int o = 16; o > 0; o >>= 1) vav += __shfl_xor_sync(0xffffffffu, vav, o);
    if (lane == 0 && warp < 4) s_v[warp] = vav;
    bar_sync_main();  // also: sx and sxr are free for the next column
    if (tid == 0) stw(a.VAV + par * a.vav_par + w, cmk(2.0 * (s_v[0] + s_v[1] + s_v[2] + s_v[3]), 0.0), tag);
  }
}

// ---------------------------------------------------------------------------
// Chunk ch of owner o: block row o, then nt - 1 - o (the parts of y for a block
// row decrease with its index, so the pairs are equally long); -1 for none.
__device__ __forceinline__ int owner_block(int o, int ch, int nt) {
  if (ch == 0) return o;
  const int m = nt - 1 - o;
  return m > o ? m : -1;
}

template <typename T2, int MC>
struct OwnerSmem {
  T2 V[MC][NBT][RCH + 2];  // padded: a warp reads four columns of eight rows
  T2 W[MC][NBT][RCH + 2];
  cplx X[MC][RCH];         // the column's entries below c + 1
  double D[MC][RCH];       // real diagonal of C
};

template <typename T2, int MC>
__device__ void flow_owner(const FlowArgs<T2>& a, unsigned char* dsm, int o) {
  constexpr int BPT = 64 / TILE_COLS<T2>;
  OwnerSmem<T2, MC>& S = *reinterpret_cast<OwnerSmem<T2, MC>*>(dsm);
  __shared__ double s_red4[FT / 32][4];
  __shared__ cplx s_S[NBT], s_T[NBT], s_vc[NBT], s_wc[NBT];  // totals; row c+1 of V and W
  __shared__ cplx s_sv[NBT], s_tv[NBT];                       // V^H v, W^H v
  __shared__ cplx s_nd, s_h, s_al, s_wc1;                     // (norm, dg), x^H C e1, x(c+1), w(c+1)
  __shared__ double s_aw;                                     // alpha of w
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.n, nrel = n - a.p;
  const long long ld = a.ld;
  T2* __restrict__ C = a.C;
  const Fold<BPT> F(a.nt);
  Waiter wt{a.status, a.wait_ns, false};
  if (warp == FT / 32 + 1) return;

  // reflector of the current column from the totals: the same in every thread
  cplx tau, scale;
  double beta;
  auto reflector = [&]() {
    const cplx al = s_al;
    const double xn2 = s_nd.x;
    tau = scale = cmk(0.0, 0.0);
    if (xn2 == 0.0 && al.y == 0.0) {
      beta = al.x;
    } else {
      const double nrm = sqrt(al.x * al.x + al.y * al.y + xn2);
      beta = (al.x >= 0.0) ? -nrm : nrm;
      const double dr = al.x - beta, di = al.y;  // scale = 1 / (alpha - beta)
      const double rb = 1.0 / beta, rd = 1.0 / (dr * dr + di * di);
      tau = cmk(1.0 - al.x * rb, -al.y * rb);
      scale = cmk(dr * rd, -di * rd);
    }
  };

  if (warp == FT / 32) {  // ---- auxiliary warp: w(c+1) and alpha
    // y(c+1): the row parts of block row 0 and the column parts of all rows
    const long long rs0 = F.row_begin(0);
    const int w0 = worker_of(rs0, F.U, a.NW), nrow0 = worker_of(rs0 + BPT - 1, F.U, a.NW) - w0 + 1;
    const int ncon = nrow0 + a.nt, rofs0 = 64 * (w0 + F.rank(0));
    for (int i = 0; i < a.nbp; ++i) {
      const int c = a.p + i, par = c & 1, c1 = c + 1;
      const unsigned tag = (unsigned)c + 1u;
      const double c11 = ldT(C + c1 + ld * c1).x;
      if (bar_owner(wt.bad)) return;
      reflector();
      cplx q1 = cmk(0.0, 0.0);
      double ts = 0.0;
      if (lane < i) {
        q1 = cadd(cmul(s_vc[lane], s_tv[lane]), cmul(s_wc[lane], s_sv[lane]));
        ts = s_tv[lane].x * s_sv[lane].x + s_tv[lane].y * s_sv[lane].y;
      }
      q1 = warp_sum(q1);
      for (int s = 16; s > 0; s >>= 1) ts += __shfl_xor_sync(0xffffffffu, ts, s);
      cplx y = cmk(0.0, 0.0);
      double vav = 0.0;
      for (int q = lane; q < (max(ncon, a.NW) + 31) / 32 * 32; q += 128) {
        const word* ptr[8];
        unsigned mask = 0;
        cplx v[8];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int qq = q + 32 * h;
          const int I = qq - nrow0;
          ptr[h] = (qq < nrow0) ? a.ROW + par * a.row_par + rofs0 + 64 * qq + i + 1
                                : a.COL + par * a.col_par + col_at(min(I, a.nt - 1), i + 1);
          if (qq < ncon) mask |= 1u << h;
          ptr[4 + h] = a.VAV + par * a.vav_par + (qq < a.NW ? qq : 0);
          if (qq < a.NW) mask |= 1u << (4 + h);
        }
        poll(ptr, mask, tag, v, wt);
        y = cadd(y, cadd(cadd(v[0], v[1]), cadd(v[2], v[3])));
        vav += (v[4].x + v[5].x) + (v[6].x + v[7].x);
      }
      y = warp_sum(y);
      for (int s = 16; s > 0; s >>= 1) vav += __shfl_xor_sync(0xffffffffu, vav, s);
      if (lane == 0) {
        // v^H C v with v = e1 + scale x; alpha = -1/2 |tau|^2 (v^H C v - 2 Re(t^H s))
        const double vcv = c11 + 2.0 * (scale.x * s_h.x + scale.y * s_h.y) +
                           (scale.x * scale.x + scale.y * scale.y) * (vav - s_nd.y);
        const double aw = -0.5 * (tau.x * tau.x + tau.y * tau.y) * (vcv - 2.0 * ts);
        cplx wc = cadd(cmul(scale, y), cmk(c11, 0.0));
        wc = cmul(tau, csub(wc, q1));
        wc.x += aw;
        s_aw = aw;
        s_wc1 = wc;
        if (o == 0) {
          a.e[c] = beta;
          a.tau[c] = tau;
        }
      }
      if (bar_owner(wt.bad)) return;
    }
    return;
  }

  // ---- main threads: four per row
  const int rsub = tid & 3, rloc = tid >> 2;
  // rows that a reflector does not reach take part in the sums with weight zero
  for (int e = tid; e < MC * NBT * (RCH + 2); e += FT) {
    (&S.V[0][0][0])[e] = fromD<T2>(cmk(0.0, 0.0));
    (&S.W[0][0][0])[e] = fromD<T2>(cmk(0.0, 0.0));
  }
  bar_sync_main();
  cplx x[MC], cn[MC];  // current column, and C(:, c+1)
  int rel[MC];
#pragma unroll
  for (int ch = 0; ch < MC; ++ch) {
    const int blk = owner_block(o, ch, a.nt);
    rel[ch] = (blk >= 0 && blk * 64 + rloc < nrel) ? blk * 64 + rloc : -1;
    x[ch] = cn[ch] = cmk(0.0, 0.0);
    if (rel[ch] < 0) continue;
    const int r = a.p + rel[ch];
    x[ch] = ldT(C + r + ld * a.p);
    if (rel[ch] > 0) cn[ch] = ldT(C + r + ld * (a.p + 1));
    if (rsub == 0) S.D[ch][rloc] = ldT(C + r + ld * r).x;
    if (rel[ch] == 0 && rsub == 0) {
      a.d[a.p] = x[ch].x;
      stT(C + r + ld * a.p, cmk(x[ch].x, 0.0));
    }
    if (rel[ch] >= 1 && rsub == 0) stw(a.X + (a.p & 1) * a.x_par + rel[ch], x[ch], (unsigned)a.p + 1u);
  }
  __syncwarp();

  // where the parts of y for own rows are: nrow row parts, then the column parts
  // of this and all later block rows
  int nrow[MC], ncon[MC];
  long long rofs[MC];
#pragma unroll
  for (int ch = 0; ch < MC; ++ch) {
    const int I = owner_block(o, ch, a.nt);
    nrow[ch] = ncon[ch] = 0;
    rofs[ch] = 0;
    if (I < 0) continue;
    const long long rs = F.row_begin(I);
    const int w0 = worker_of(rs, F.U, a.NW), w1 = worker_of(rs + (long long)(I + 1) * BPT - 1, F.U, a.NW);
    nrow[ch] = w1 - w0 + 1;
    ncon[ch] = nrow[ch] + a.nt - I;
    rofs[ch] = 64LL * (w0 + F.rank(I));
  }

  for (int i = 0; i < a.nbp; ++i) {
    const int c = a.p + i, par = c & 1, c1 = c + 1;
    const unsigned tag = (unsigned)c + 1u;
    // partial sums over own rows below c + 1: |x|^2, diag(C)|x|^2 and x^H C(:, c+1)
    // by the rows' threads, then V^H x and W^H x with four threads per column
    {
      double part = 0.0;
#pragma unroll
      for (int ch = 0; ch < MC; ++ch) {
        const bool on = rel[ch] >= i + 2;
        const cplx xt = on ? x[ch] : cmk(0.0, 0.0);
        if (rsub == 0) S.X[ch][rloc] = xt;
        if (!on) continue;
        if (rsub == 0) part += cabs2(xt);
        else if (rsub == 1) part += S.D[ch][rloc] * cabs2(xt);
        else if (rsub == 2) part += xt.x * cn[ch].x + xt.y * cn[ch].y;   // conj(x) C(r, c+1)
        else part += xt.x * cn[ch].y - xt.y * cn[ch].x;
      }
      for (int s = 4; s < 32; s <<= 1) part += __shfl_xor_sync(0xffffffffu, part, s);
      if (lane < 4) s_red4[warp][lane] = part;
    }
    bar_sync_main();
    {
      const int j = (tid >> 2) & (NBT - 1);
      word* q = a.PART + par * a.part_par + (long long)(tid >> 2) * a.NO + o;
      cplx s = cmk(0.0, 0.0);
      if (j < i) {
#pragma unroll
        for (int ch = 0; ch < MC; ++ch) {
          const T2* M = (tid < 4 * NBT) ? S.V[ch][j] : S.W[ch][j];
          cplx sa[4];  // independent chains
#pragma unroll
          for (int k = 0; k < 4; ++k) sa[k] = cmk(0.0, 0.0);
#pragma unroll
          for (int t = 0; t < RCH / 4; t += 4)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const cplx mv = toD(M[rsub + 4 * (t + k)]), xv = S.X[ch][rsub + 4 * (t + k)];
              sa[k].x = fma(mv.x, xv.x, fma(mv.y, xv.y, sa[k].x));
              sa[k].y = fma(mv.x, xv.y, fma(-mv.y, xv.x, sa[k].y));
            }
          s = cadd(s, cadd(cadd(sa[0], sa[1]), cadd(sa[2], sa[3])));
        }
      }
      s = shfl4_sum(s);
      if (j < i && rsub == 0) stw(q, s, tag);
      if (tid >= FT - 4) {  // no column NBT - 1 is ever summed: these threads are free
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < FT / 32; ++w) v += s_red4[w][rsub];
        const double v1 = __shfl_xor_sync(0xf0000000u, v, 1);
        if (!(rsub & 1)) stw(a.PART + par * a.part_par + (long long)(2 * NBT + (rsub >> 1)) * a.NO + o, cmk(v, v1), tag);
      }
    }
    // totals, row c + 1 of V and W, x(c+1)
    {
      const word* b = nullptr;
      cplx* dst = nullptr;
      int k = tid;
      if (k < i) { b = a.TOT + par * a.tot_par + k; dst = &s_S[k]; }
      else if ((k -= i) < i) { b = a.TOT + par * a.tot_par + NBT + k; dst = &s_T[k]; }
      else if ((k -= i) < i) { b = a.RVW + par * a.rvw_par + k; dst = &s_vc[k]; }
      else if ((k -= i) < i) { b = a.RVW + par * a.rvw_par + NBT + k; dst = &s_wc[k]; }
      else if ((k -= i) == 0) { b = a.TOT + par * a.tot_par + 2 * NBT; dst = &s_nd; }
      else if (k == 1) { b = a.TOT + par * a.tot_par + 2 * NBT + 1; dst = &s_h; }
      else if (k == 2) { b = a.X + par * a.x_par + i + 1; dst = &s_al; }
      const word* ptr[1] = {b ? b : a.X};
      cplx v[1];
      poll(ptr, b ? 1u : 0u, tag, v, wt);
      if (b) *dst = v[0];
    }
    bar_sync_main();
    reflector();
    if (tid < i) {
      const cplx vc = s_vc[tid], wc = s_wc[tid];
      s_sv[tid] = cadd(cmul(scale, s_S[tid]), cconj(vc));
      s_tv[tid] = cadd(cmul(scale, s_T[tid]), cconj(wc));
    }
    if (bar_owner(wt.bad)) return;
    cplx q[MC], u[MC];
#pragma unroll
    for (int ch = 0; ch < MC; ++ch) {
      q[ch] = u[ch] = cmk(0.0, 0.0);
      const bool act = rel[ch] >= i + 1;
      if (act) {
        cplx q2 = cmk(0.0, 0.0), u2 = cmk(0.0, 0.0);
#pragma unroll 2
        for (int j = rsub; j < i; j += 4) {
          const cplx vj = toD(S.V[ch][j][rloc]), wj = toD(S.W[ch][j][rloc]);
          const cplx tj = s_tv[j], sj = s_sv[j], wc = s_wc[j], vc = s_vc[j];
          q[ch].x = fma(vj.x, tj.x, fma(-vj.y, tj.y, q[ch].x));
          q[ch].y = fma(vj.x, tj.y, fma(vj.y, tj.x, q[ch].y));
          q2.x = fma(wj.x, sj.x, fma(-wj.y, sj.y, q2.x));
          q2.y = fma(wj.x, sj.y, fma(wj.y, sj.x, q2.y));
          u[ch].x = fma(vj.x, wc.x, fma(vj.y, wc.y, u[ch].x));  // v conj(w)
          u[ch].y = fma(vj.y, wc.x, fma(-vj.x, wc.y, u[ch].y));
          u2.x = fma(wj.x, vc.x, fma(wj.y, vc.y, u2.x));
          u2.y = fma(wj.y, vc.x, fma(-wj.x, vc.y, u2.y));
        }
        q[ch] = cadd(q[ch], q2);
        u[ch] = cadd(u[ch], u2);
      }
      q[ch] = shfl4_sum(q[ch]);
      u[ch] = shfl4_sum(u[ch]);
    }
    cplx y[MC];
    // y = C22 x: row parts of the workers that share the block row, then the
    // column parts of this and all later block rows
#pragma unroll
    for (int ch = 0; ch < MC; ++ch) {
      y[ch] = cmk(0.0, 0.0);
      const int I = max(owner_block(o, ch, a.nt), 0), r0 = I * 64;
      // rows past the matrix or above the column poll a row of the block that is sent
      const bool act = rel[ch] >= i + 1;
      const int rmin = max(i + 1 - r0, 0), rmax = min(63, nrel - 1 - r0);
      const int rr = min(max(rloc, rmin), rmax);
      const word* rb = a.ROW + par * a.row_par + rofs[ch];
      const word* cb = a.COL + par * a.col_par + r0;
      // one word per part first (of the last row the warp has), as the workers do
      const int rlast = min(max(rloc | 7, rmin), rmax);
      for (int k = lane; k < ncon[ch] + lane; k += 32) {
        const int kk = min(k, ncon[ch] - 1);
        const word* ptr[1] = {(kk < nrow[ch] ? rb + 64 * kk : cb + col_at(I + kk - nrow[ch], 0)) + rlast};
        cplx v[1];
        poll(ptr, 1u, tag, v, wt);
      }
      for (int k = rsub; k < ncon[ch] + rsub; k += 32) {
        const word* ptr[8];
        unsigned mask = 0;
        cplx v[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const int kk = min(k + 4 * h, ncon[ch] - 1);
          ptr[h] = (kk < nrow[ch] ? rb + 64 * kk : cb + col_at(I + kk - nrow[ch], 0)) + rr;
          if (act && k + 4 * h < ncon[ch]) mask |= 1u << h;
        }
        poll(ptr, mask, tag, v, wt, (ncon[ch] - (k - rsub) + 3) >> 2);
        y[ch] = cadd(y[ch], cadd(cadd(cadd(v[0], v[1]), cadd(v[2], v[3])), cadd(cadd(v[4], v[5]), cadd(v[6], v[7]))));
      }
      y[ch] = shfl4_sum(y[ch]);
    }
    if (bar_owner(wt.bad)) return;
    const cplx wc1 = s_wc1;
    const double aw = s_aw;
    const bool upd = (i + 1 < a.nbp) || a.final_panel;  // column c+1 is updated here
#pragma unroll
    for (int ch = 0; ch < MC; ++ch) {
      if (rel[ch] < i + 1) continue;
      const int r = a.p + rel[ch];
      const cplx vr = (rel[ch] == i + 1) ? cmk(1.0, 0.0) : cmul(scale, x[ch]);
      const cplx yr = cadd(cmul(scale, y[ch]), cn[ch]);
      const cplx wr = cadd(cmul(tau, csub(yr, q[ch])), cscale(vr, aw));
      cplx xn = csub(csub(csub(cn[ch], u[ch]), cmul_cb(vr, wc1)), wr);
      if (rel[ch] == i + 1) xn.y = 0.0;
      if (i + 1 < a.nbp && rel[ch] >= i + 2 && rsub == 0) stw(a.X + (par ^ 1) * a.x_par + rel[ch], xn, tag + 1u);
      x[ch] = xn;
      if (i + 1 < a.nbp && rel[ch] >= i + 2) cn[ch] = ldT(C + r + ld * (c1 + 1));
      if (rsub == 0) {
        S.V[ch][i][rloc] = fromD<T2>(vr);
        S.W[ch][i][rloc] = fromD<T2>(wr);
        stT(C + r + ld * c, vr);
        if (upd && rel[ch] == i + 1) a.d[c1] = xn.x;
      } else if (rsub == 1) {
        stT(a.VW + r + ld * i, vr);
        stT(a.WV + r + ld * (NBT + i), vr);
      } else if (rsub == 2) {
        stT(a.VW + r + ld * (NBT + i), wr);
        stT(a.WV + r + ld * i, wr);
      }
    }
    __syncwarp();
    // row c + 2 of V and W for the next column
    if (i + 1 < a.nbp) {
#pragma unroll
      for (int ch = 0; ch < MC; ++ch)
        if (rel[ch] == i + 2)
          for (int j = rsub; j <= i; j += 4) {
            word* b = a.RVW + (par ^ 1) * a.rvw_par + j;
            stw(b, toD(S.V[ch][j][rloc]), tag + 1u);
            stw(b + NBT, toD(S.W[ch][j][rloc]), tag + 1u);
          }
    }
  }
}

template <typename T2, int MC>
__global__ void __launch_bounds__(FTOT, 1)
    k_tridiag_flow(FlowArgs<T2> a, const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(128) unsigned char dsm_raw[];
  const unsigned b0 = smem_u32(dsm_raw);
  unsigned char* dsm = dsm_raw + (((b0 + 127u) & ~127u) - b0);
  if ((int)blockIdx.x < a.NO) flow_owner<T2, MC>(a, dsm, blockIdx.x);
  else flow_worker<T2>(a, &tmap, dsm, (int)blockIdx.x - a.NO);
}

// Words of one reduction of order n with G blocks (two buffers each).
struct FlowLayout {
  long long x, col, row, vav, part, tot, rvw, total;
  FlowLayout(int n, int G) {
    const long long nt = (n + 63) / 64;
    x = 64 * nt;
    col = 64 * nt * (nt + 1) / 2;
    row = 64 * (G + nt);
    vav = G;
    part = (long long)NK * G;
    tot = NK;
    rvw = 2 * NBT;
    total = 2 * (x + col + row + vav + part + tot + rvw);
  }
};

constexpr size_t FLOW_SMEM = 198 * 1024;  // dynamic; the static part is 28 KB of the 227 KB

// Roles and shared memory of the panel from column p on G blocks; false where
// the panel does not suit the form.
template <typename T2, int MC>
bool flow_shape(int n, int p, int G, FlowArgs<T2>& a, size_t* smem) {
  constexpr int BC = TILE_COLS<T2>, BPT = 64 / BC;
  a.nt = (n - p + 63) / 64;
  a.NO = (a.nt + MC - 1) / MC;
  a.NWT = G - a.NO;
  // enough workers to leave the products the larger part of the GPU, and one
  // warp for each of the NK totals
  if (a.NWT < NK || a.NWT < G / 2) return false;
  const long long U = (long long)a.nt * (a.nt + 1) / 2 * BPT;
  a.NW = (int)std::min<long long>(a.NWT, U);
  const int units = (int)((U + a.NW - 1) / a.NW);
  if (2 * (units / ((a.nt + 1) * BPT) + 1) + 3 > RUNMAX || units > 128) return false;
  a.ecap = (units * BC + 15) / 16 * 16;
  const size_t fixed = (size_t)a.ecap * (sizeof(T2) + 4) + RUNMAX * 64 * (sizeof(cplx) + 4);
  const size_t tile = (size_t)RCH * BC * sizeof(T2);
  a.stages = (int)std::min<size_t>(FSTAGES, (FLOW_SMEM - 128 - fixed) / tile);
  a.stages = std::min(a.stages, std::max(units, 4));
  if (a.stages < 4) return false;
  *smem = std::max(fixed + a.stages * tile, sizeof(OwnerSmem<T2, MC>)) + 128;
  return *smem <= FLOW_SMEM + 128;
}

template <typename T2, int MC>
int flow_panel(excfv_handle* h, const CUtensorMap& tmap, FlowArgs<T2> a, int G, size_t smem) {
  CUDA_TRY(raise_smem_limit(k_tridiag_flow<T2, MC>, FLOW_SMEM + 128));
  void* args[] = {&a, const_cast<CUtensorMap*>(&tmap)};
  CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k_tridiag_flow<T2, MC>, dim3(G), dim3(FTOT), args, smem,
                                       h->stream));
  count_launch();
  return EXCFV_OK;
}

}  // namespace

// Bytes of the words for orders up to n.
size_t tridiag_flow_bytes(int n, int nsm) { return (size_t)FlowLayout(n, nsm).total * sizeof(word); }

// Whether G blocks are enough for the roles at all (of the smaller trailing blocks).
bool tridiag_flow_available(int G) { return G - 16 >= NK; }

// Zeroes the words of the reduction that begins (tags of an earlier one must
// not be taken).
int tridiag_flow_begin(excfv_handle* h, int n, int G) {
  CUDA_TRY(cudaMemsetAsync(h->ws.flow, 0, (size_t)FlowLayout(n, G).total * sizeof(word), h->stream));
  return EXCFV_OK;
}

// The panel of columns [p, p + nbp) of C on G blocks; 1 where it does not suit
// this form (nothing is launched), else 0 or an error.
template <typename T2>
int tridiag_flow_panel(excfv_handle* h, int n, int p, int nbp, int final_panel, T2* C, long long ld, T2* VW, T2* WV,
                       int G, long long wait_ns, unsigned planted) {
  Workspace& ws = h->ws;
  FlowArgs<T2> a;
  size_t smem = 0;
  // one chunk of rows per owner where that leaves two thirds of the GPU to the
  // workers, else two
  int mc = 0;
  const int nt = (n - p + 63) / 64;
  if (3 * nt <= G && flow_shape<T2, 1>(n, p, G, a, &smem)) mc = 1;
  else if (flow_shape<T2, 2>(n, p, G, a, &smem)) mc = 2;
  if (!mc) return 1;
  const FlowLayout L(n, G);
  word* b = reinterpret_cast<word*>(ws.flow);
  a.X = b; b += 2 * L.x; a.COL = b; b += 2 * L.col; a.ROW = b; b += 2 * L.row; a.VAV = b; b += 2 * L.vav;
  a.PART = b; b += 2 * L.part; a.TOT = b; b += 2 * L.tot; a.RVW = b;
  a.x_par = L.x; a.col_par = L.col; a.row_par = L.row; a.vav_par = L.vav; a.part_par = L.part; a.tot_par = L.tot;
  a.rvw_par = L.rvw;
  a.n = n; a.ld = ld; a.C = C; a.VW = VW; a.WV = WV; a.d = ws.d; a.e = ws.e; a.tau = ws.tau; a.status = ws.status;
  a.p = p; a.nbp = nbp; a.final_panel = final_panel; a.wait_ns = wait_ns; a.planted = planted;
  CUtensorMap tmap;
  if (int rc = make_tile_map(&tmap, C, n, ld)) return rc;
  return mc == 1 ? flow_panel<T2, 1>(h, tmap, a, G, smem) : flow_panel<T2, 2>(h, tmap, a, G, smem);
}

template int tridiag_flow_panel<double2>(excfv_handle*, int, int, int, int, double2*, long long, double2*, double2*,
                                         int, long long, unsigned);
template int tridiag_flow_panel<float2>(excfv_handle*, int, int, int, int, float2*, long long, float2*, float2*, int,
                                        long long, unsigned);
