// Device and host helpers shared by the panel kernels of the tridiagonal
// reduction (tridiag.cu, tridiag_flow.cu): storage conversions, bounded mbarrier
// waits, the tile loads of the trailing matrix by TMA.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include "handle.cuh"

namespace {

constexpr int NBT = 32;   // columns per panel
constexpr int RCH = 64;   // rows per chunk and per tile
// columns of one TMA tile of RCH rows (16 KB)
template <typename T2>
constexpr int TILE_COLS = (sizeof(T2) == 16) ? 16 : 32;

// Storage type T2 of C, V and W: double2 (FP64 form) or float2 (the precision
// form's complex64 copy).  Arithmetic is FP64 in both.
__device__ __forceinline__ cplx ldT(const double2* p) { return __ldcg(p); }
__device__ __forceinline__ cplx ldT(const float2* p) {
  const float2 v = __ldcg(p);
  return cmk((double)v.x, (double)v.y);
}
__device__ __forceinline__ void stT(double2* p, cplx v) { *p = v; }
__device__ __forceinline__ void stT(float2* p, cplx v) { *p = make_float2((float)v.x, (float)v.y); }
__device__ __forceinline__ cplx toD(double2 v) { return v; }
__device__ __forceinline__ cplx toD(float2 v) { return cmk((double)v.x, (double)v.y); }
template <typename T2> __device__ __forceinline__ T2 fromD(cplx v);
template <> __device__ __forceinline__ double2 fromD<double2>(cplx v) { return v; }
template <> __device__ __forceinline__ float2 fromD<float2>(cplx v) {
  return make_float2((float)v.x, (float)v.y);
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ long long gtimer() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ cplx ldc(const cplx* p) { return __ldcg(p); }
__device__ __forceinline__ double ldd(const double* p) { return __ldcg(p); }

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for a TMA tile; gives up (status[ST_BARRIER] set) after
// limit_ns or as soon as another wait of the launch has given up.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, unsigned parity, int* status,
                                          long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = gtimer();
  unsigned it = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++it & 63u) == 0) {
      if (*(volatile int*)&status[ST_BARRIER] != 0) return;
      if (gtimer() - t0 > limit_ns) {
        atomicAdd(&status[ST_BARRIER], 1);
        return;
      }
    }
  }
}
// Bounded wait that reports whether the phase completed.
__device__ __forceinline__ bool mbar_wait_ok(uint64_t* bar, unsigned parity, int* status,
                                             long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = gtimer();
  unsigned it = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++it & 63u) == 0) {
      if (*(volatile int*)&status[ST_BARRIER] != 0) return false;
      if (gtimer() - t0 > limit_ns) {
        atomicAdd(&status[ST_BARRIER], 1);
        return false;
      }
    }
  }
  return true;
}
// Before the producer leaves the kernel: every TMA copy it issued has landed
// (q copies issued round-robin over the slots), so no copy writes into the
// shared memory of a finished block.  Bounded by limit_ns per slot; this wait
// ignores the status word, since the copies land whether or not a wait of the
// launch gave up.
template <int STAGES>
__device__ __forceinline__ void drain_copies(uint64_t* full, unsigned q, long long limit_ns) {
  for (unsigned s = 0; s < (unsigned)STAGES && s < q; ++s) {
    const unsigned uses = q / STAGES + (s < q % STAGES ? 1u : 0u);
    const unsigned parity = (uses - 1u) & 1u;
    const long long t0 = gtimer();
    while (!mbar_try_wait(&full[s], parity))
      if (gtimer() - t0 > limit_ns) break;
  }
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 2-D tiled TMA load (no multicast) of one 64 x BC tile; x counts scalars
// (re and im separately) along the rows, y counts columns.
__device__ __forceinline__ void tma_tile(void* dst, const CUtensorMap* tm, int x, int y,
                                         uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ cplx shfl4_sum(cplx v) {
  v.x += __shfl_xor_sync(0xffffffffu, v.x, 1);
  v.y += __shfl_xor_sync(0xffffffffu, v.y, 1);
  v.x += __shfl_xor_sync(0xffffffffu, v.x, 2);
  v.y += __shfl_xor_sync(0xffffffffu, v.y, 2);
  return v;
}

__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }

// Sums of four column groups over the 16 lanes of a half warp, scattered: lane
// bits 3 and 2 select the group whose sum the lane ends up with.
template <typename T2>
__device__ __forceinline__ T2 scatter_sum16(const T2 (&cp)[4], int lane) {
  const bool h3 = (lane >> 3) & 1, h2 = (lane >> 2) & 1;
  const T2 s0 = h3 ? cp[0] : cp[2], s1 = h3 ? cp[1] : cp[3];
  T2 k0 = h3 ? cp[2] : cp[0], k1 = h3 ? cp[3] : cp[1];
  k0.x += __shfl_xor_sync(0xffffffffu, s0.x, 8);
  k0.y += __shfl_xor_sync(0xffffffffu, s0.y, 8);
  k1.x += __shfl_xor_sync(0xffffffffu, s1.x, 8);
  k1.y += __shfl_xor_sync(0xffffffffu, s1.y, 8);
  T2 kk = h2 ? k1 : k0;
  const T2 s2 = h2 ? k0 : k1;
  kk.x += __shfl_xor_sync(0xffffffffu, s2.x, 4);
  kk.y += __shfl_xor_sync(0xffffffffu, s2.y, 4);
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    kk.x += __shfl_xor_sync(0xffffffffu, kk.x, o);
    kk.y += __shfl_xor_sync(0xffffffffu, kk.y, o);
  }
  return kk;
}

// a * conj(b)
__device__ __forceinline__ cplx cmul_cb(cplx a, cplx b) {
  return cmk(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

__device__ __forceinline__ cplx warp_sum(cplx v) {
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point
inline PFN_cuTensorMapEncodeTiled_v12000 encode_tiled_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// Tensor map of the n x n matrix C (leading dimension ld) as real scalars:
// 2n rows of re/im pairs, n columns; tiles of 64 complex rows x BC columns.
template <typename T2>
int make_tile_map(CUtensorMap* tm, const T2* C, int n, long long ld) {
  auto fn = encode_tiled_fn();
  if (!fn) {
    excfv_set_error("cuTensorMapEncodeTiled is not available from the driver");
    return EXCFV_ERR_CUDA;
  }
  if ((reinterpret_cast<uintptr_t>(C) & 15) || ((ld * sizeof(T2)) & 15)) {
    excfv_set_error("tridiagonal reduction: matrix base or column stride not 16-byte aligned");
    return EXCFV_ERR_ARG;
  }
  const cuuint64_t dims[2] = {2ull * (cuuint64_t)n, (cuuint64_t)n};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(T2)};
  const cuuint32_t box[2] = {2u * RCH, (cuuint32_t)TILE_COLS<T2>};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUtensorMapDataType dt =
      (sizeof(T2) == 16) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const CUresult r = fn(tm, dt, 2, const_cast<T2*>(C), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    excfv_set_error("cuTensorMapEncodeTiled failed (%d) for n=%d ld=%lld", (int)r, n, ld);
    return EXCFV_ERR_CUDA;
  }
  return EXCFV_OK;
}

}  // namespace
