// Block-CSR SpMV, diagonal (block-Jacobi) preconditioner and GMRES (sm_100a).
//
// Replaces SparseProdUP_3D / SparseProd_NS_conv / SparseProd_LS
// (src/SparseProd.f90:4-60,167-242,128-161) and SparseGMRES_up /
// SparseGMRES_ns_conv / SparseGMRES_tem (src/SparseGMRES_NS.f90:4-369,
// src/SparseGMRES_NS_conv.f:1-406, src/SparseGMRES_tem.f90:1-256).
//
// SpMV: a group of lanes owns one CSR row.  The slot values of a row are
// contiguous (24/16/1 per slot), so the lanes of a group read four values each
// per slot (16 bytes in FP32, 32 in FP64) and the whole row streams with full
// sectors; the x gathers hit L2.  The preconditioner (exact 3x3 inverse of the velocity
// diagonal block, reciprocal diagonal for p / phi / T) is applied to the row
// result before the store, so one pass produces P^-1 A x.
//
// GMRES: one Arnoldi cycle follows the reference step by step (left
// preconditioning, the coefficients of modified Gram-Schmidt, Givens rotations,
// exit rule |e(k+1)| <= tol |P^-1 b| and k >= kspace_min, back-substitution,
// sol += sum y_j v_j).  The coefficients of a step come from one pass of dots
// and a triangular product (gm_orthog_kernel); the one-launch variant
// (gm_arnoldi_kernel) takes them one after another in the reference's "project
// off j-1, dot with j" order.  All scalars live on the device; every dot product
// is added in FP64 in an order fixed by the grid, so results are bit-identical
// from run to run.  The host only polls the "done" word once
// per batch of iterations, a batch behind the launches.
#include "ovs_internal.cuh"

#include <algorithm>
#include <vector>

#include <cooperative_groups.h>
#include <type_traits>
#include <math.h>
#include <string.h>

namespace cg = cooperative_groups;

namespace {

constexpr int SPMV_THREADS = 256;
// threads of a block row product: 64 but for FP64 matrices with vectors by fields
// (see spmv_block_warp)
template <typename TM, bool AOS>
__host__ __device__ constexpr int spmv_threads() { return AOS || sizeof(TM) == 4 ? 64 : SPMV_THREADS; }

template <typename T> __device__ __forceinline__ T ldm(const T* p) { return __ldcs(p); }

// Four matrix values.  FP64: one 32-byte load instead of two streaming ones of 16,
// evicted first from L2, where the Krylov basis is worth more.  FP32: no hint.
// NS+VOF product with vectors by nodes, and in brackets the whole iteration at
// k = 25, at 31K, 233K and 2.1M nodes:
//   FP64  two of 16, streaming     24.4 (49.2), 111 (202), 1113 us (1765)
//         one of 32                16.6 (51.3), 119 (199), 1035    (1687)
//         one of 32, evict first   20.7 (45.4), 107 (196), 1060    (1711)
//   FP32  one of 16, streaming     12.4 (37.7),  60 (127),  611    (972)
//         one of 16                10.5 (36.8),  69 (126),  576    (938)
__device__ __forceinline__ void ld4(const float* p, float v[4]) {
  asm("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
}
__device__ __forceinline__ void ld4(const double* p, double v[4]) {
  asm("ld.global.nc.L2::evict_first.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

// Accumulation precision of the SpMV: FP32 storage accumulates in FP32 on
// the mixed path (the inner solver of the refinement), FP64 otherwise.
// (FP64 accumulation and an FP64 work vector in Gram-Schmidt were measured on
// the 2.1M-node quench system: they converged in as many refinement cycles
// and ran slower, so the mixed path keeps everything in FP32 except the dots,
// Givens and the refinement residual.)
template <typename A, typename B, bool ACC64> struct AccT { using type = double; };
template <> struct AccT<float, float, false> { using type = float; };

// MODE 0: y = A x ; MODE 1: y = P^-1 A x ; MODE 2: y = b - A x
// Block systems: NG groups of 4 values per slot, one lane per group.
//   NS   (NG=4): groups rows u1,u2,u3,p over columns (u1,u2,u3,p)
//   NSVOF(NG=6): + row phi over (u1,u2,u3,phi), + column phi into (u1,u2,u3,p)
// The RPW = 32/NG rows of warp chunk `wglob` (all 32 lanes take part in
// the shuffles).
// AOS: x and y by nodes (x[node nf + field]), as the Krylov basis holds its
// vectors, instead of by fields: a slot's gathers fall into one or two sectors
// instead of one per field (FP32 66.0 -> 62.1 us at 233K nodes, 0.627 -> 0.597 ms
// at 2.1M).  The kernel waits for its loads (20 stalled warps per issue), so the
// warps in flight decide: blocks of 64 threads, whose places are refilled sooner
// than those of 256, gain 1 to 8% there and for FP32 matrices by fields, and lose
// 7% for FP64 by fields.  Times: ld4.  Its bytes with the preconditioner's at 6.45
// TB/s, at 233K and 2.1M nodes: FP64 110 and 1024 us, FP32 56 and 522; with the
// benchmark's system at 2.1M nodes it takes 1051 and 557, 97% and 94% of that rate.
// LIST: the warp chunks run over the row list rows[0, nrows) (local row
// indices; an index outside [0, N) is skipped) instead of rows 0..N-1;
// each listed row is computed exactly as in the full product.
template <int NG, typename TM, typename TX, typename TY, int MODE, bool ACC64, bool LIST = false, bool AOS = false>
__device__ __forceinline__ void spmv_block_warp(long wglob, int N, const int* __restrict__ rowptr,
                                                const int* __restrict__ colidx, const TM* __restrict__ vals,
                                                const TX* __restrict__ x, TY* __restrict__ y,
                                                const TM* __restrict__ pre, const double* __restrict__ b,
                                                const int* __restrict__ rows = nullptr, long nrows = 0) {
  using AT = typename AccT<TM, TX, ACC64>::type;
  constexpr int NV = 4 * NG, NFX = NG == 6 ? 5 : 4;
  constexpr int RPW = 32 / NG;  // rows per warp
  const int lane = threadIdx.x & 31;
  const int sub = lane / NG;
  const int g = lane - sub * NG;
  const long rowl = wglob * RPW + sub;
  bool active;
  int row;
  if constexpr (LIST) {
    const int rl = (sub < RPW && rowl < nrows) ? __ldg(rows + rowl) : -1;
    active = rl >= 0 && rl < N;
    row = active ? rl : 0;
  } else {
    active = sub < RPW && rowl < N;
    row = active ? (int)rowl : 0;
  }
  // column fields read by this lane's 4 values
  int cf0, cf1, cf2, cf3;
  if (NG == 6 && g == 5) { cf0 = cf1 = cf2 = cf3 = 4; }
  else { cf0 = 0; cf1 = 1; cf2 = 2; cf3 = (NG == 6 && g == 4) ? 4 : 3; }
  AT a0 = 0, a1 = 0, a2 = 0, a3 = 0;
  if (active) {
    const int s0 = __ldg(rowptr + row), s1 = __ldg(rowptr + row + 1);
    // lane g of the row gathers field g of x at the slot's column (NS+VOF:
    // u,v,w,p,phi in lanes 0-4) and the row's lanes exchange them by
    // shuffles: 4-5 gathers per slot instead of 4 per lane
    int s = s0;
    const unsigned gmask = ((1u << NG) - 1u) << (sub * NG);
    const int base = sub * NG;
    const TX* xg = x + (AOS ? (size_t)(g < NFX ? g : 0) : (size_t)(g < NFX ? g : 0) * N);
    constexpr int XS = AOS ? NFX : 1;   // stride between nodes
    // FP32 values: 4 slots in flight per lane (measured 0.63 vs 0.72 ms at
    // 2.1M nodes); FP64 values already move 32 bytes per lane and slot, and
    // run faster with 2
    if constexpr (sizeof(TM) == 4) {
      for (; s + 3 < s1; s += 4) {
        const int c0 = __ldg(colidx + s), c1 = __ldg(colidx + s + 1), c2 = __ldg(colidx + s + 2),
                  c3 = __ldg(colidx + s + 3);
        TM v[4], w[4], y[4], z[4];
        ld4(vals + (size_t)s * NV + 4 * g, v);
        ld4(vals + (size_t)(s + 1) * NV + 4 * g, w);
        ld4(vals + (size_t)(s + 2) * NV + 4 * g, y);
        ld4(vals + (size_t)(s + 3) * NV + 4 * g, z);
        const AT f0 = (AT)__ldg(xg + (size_t)c0 * XS), f1 = (AT)__ldg(xg + (size_t)c1 * XS), f2 = (AT)__ldg(xg + (size_t)c2 * XS), f3 = (AT)__ldg(xg + (size_t)c3 * XS);
        a0 += (AT)v[0] * __shfl_sync(gmask, f0, base + cf0); a1 += (AT)v[1] * __shfl_sync(gmask, f0, base + cf1);
        a2 += (AT)v[2] * __shfl_sync(gmask, f0, base + cf2); a3 += (AT)v[3] * __shfl_sync(gmask, f0, base + cf3);
        a0 += (AT)w[0] * __shfl_sync(gmask, f1, base + cf0); a1 += (AT)w[1] * __shfl_sync(gmask, f1, base + cf1);
        a2 += (AT)w[2] * __shfl_sync(gmask, f1, base + cf2); a3 += (AT)w[3] * __shfl_sync(gmask, f1, base + cf3);
        a0 += (AT)y[0] * __shfl_sync(gmask, f2, base + cf0); a1 += (AT)y[1] * __shfl_sync(gmask, f2, base + cf1);
        a2 += (AT)y[2] * __shfl_sync(gmask, f2, base + cf2); a3 += (AT)y[3] * __shfl_sync(gmask, f2, base + cf3);
        a0 += (AT)z[0] * __shfl_sync(gmask, f3, base + cf0); a1 += (AT)z[1] * __shfl_sync(gmask, f3, base + cf1);
        a2 += (AT)z[2] * __shfl_sync(gmask, f3, base + cf2); a3 += (AT)z[3] * __shfl_sync(gmask, f3, base + cf3);
      }
    }
    for (; s + 1 < s1; s += 2) {
      const int c0 = __ldg(colidx + s), c1 = __ldg(colidx + s + 1);
      TM v[4], w[4];
      ld4(vals + (size_t)s * NV + 4 * g, v);
      ld4(vals + (size_t)(s + 1) * NV + 4 * g, w);
      const AT f0 = (AT)__ldg(xg + (size_t)c0 * XS), f1 = (AT)__ldg(xg + (size_t)c1 * XS);
      a0 += (AT)v[0] * __shfl_sync(gmask, f0, base + cf0); a1 += (AT)v[1] * __shfl_sync(gmask, f0, base + cf1);
      a2 += (AT)v[2] * __shfl_sync(gmask, f0, base + cf2); a3 += (AT)v[3] * __shfl_sync(gmask, f0, base + cf3);
      a0 += (AT)w[0] * __shfl_sync(gmask, f1, base + cf0); a1 += (AT)w[1] * __shfl_sync(gmask, f1, base + cf1);
      a2 += (AT)w[2] * __shfl_sync(gmask, f1, base + cf2); a3 += (AT)w[3] * __shfl_sync(gmask, f1, base + cf3);
    }
    if (s < s1) {
      const int c0 = __ldg(colidx + s);
      TM v[4];
      ld4(vals + (size_t)s * NV + 4 * g, v);
      const AT f0 = (AT)__ldg(xg + (size_t)c0 * XS);
      a0 += (AT)v[0] * __shfl_sync(gmask, f0, base + cf0); a1 += (AT)v[1] * __shfl_sync(gmask, f0, base + cf1);
      a2 += (AT)v[2] * __shfl_sync(gmask, f0, base + cf2); a3 += (AT)v[3] * __shfl_sync(gmask, f0, base + cf3);
    }
  }
  const int base = sub * NG;
  AT yv;
  if (NG == 6) {
    // lane 5 of the group holds the phi-column contributions of rows u1,u2,u3,p
    const AT t0 = __shfl_sync(0xffffffffu, a0, (base + 5) & 31);
    const AT t1 = __shfl_sync(0xffffffffu, a1, (base + 5) & 31);
    const AT t2 = __shfl_sync(0xffffffffu, a2, (base + 5) & 31);
    const AT t3 = __shfl_sync(0xffffffffu, a3, (base + 5) & 31);
    const AT add = g == 0 ? t0 : (g == 1 ? t1 : (g == 2 ? t2 : (g == 3 ? t3 : (AT)0)));
    yv = ((a0 + a1) + (a2 + a3)) + add;
  } else {
    yv = (a0 + a1) + (a2 + a3);
  }
  const AT y0 = __shfl_sync(0xffffffffu, yv, base & 31);
  const AT y1 = __shfl_sync(0xffffffffu, yv, (base + 1) & 31);
  const AT y2 = __shfl_sync(0xffffffffu, yv, (base + 2) & 31);
  if (!active || g >= NG - (NG == 6 ? 1 : 0)) return;
  AT z = yv;
  if (MODE == 1) {
    if (g < 3) {
      const TM* B = pre + (size_t)row * 9 + 3 * g;
      z = (AT)B[0] * y0 + (AT)B[1] * y1 + (AT)B[2] * y2;
    } else if (g == 3) {
      z = yv * (AT)pre[(size_t)9 * N + row];
    } else {
      z = yv * (AT)pre[(size_t)10 * N + row];
    }
  } else if (MODE == 2) {
    z = (AT)b[(size_t)g * N + row] - yv;
  }
  y[AOS ? (size_t)row * NFX + g : (size_t)g * N + row] = (TY)z;
}

template <int NG, typename TM, typename TX, typename TY, int MODE, bool ACC64, bool AOS>
__global__ void __launch_bounds__(spmv_threads<TM, AOS>())
spmv_block_kernel(int N, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                  const TM* __restrict__ vals, const TX* __restrict__ x, TY* __restrict__ y,
                  const TM* __restrict__ pre, const double* __restrict__ b,
                  const int* __restrict__ done) {
  if (done && *done) return;
  const long wglob = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  spmv_block_warp<NG, TM, TX, TY, MODE, ACC64, false, AOS>(wglob, N, rowptr, colidx, vals, x, y, pre, b);
}

// the same product over a list of rows (a partition's interior or boundary
// rows, ovs_spmv_device_rows)
template <int NG, typename TM, typename TX, typename TY, int MODE>
__global__ void __launch_bounds__(SPMV_THREADS)
spmv_block_rows_kernel(int N, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                       const TM* __restrict__ vals, const TX* __restrict__ x, TY* __restrict__ y,
                       const TM* __restrict__ pre, const int* __restrict__ rows, int nrows) {
  const long wglob = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  spmv_block_warp<NG, TM, TX, TY, MODE, true, true>(wglob, N, rowptr, colidx, vals, x, y, pre, nullptr, rows,
                                                     nrows);
}

// scalar CSR (temperature): 8 lanes per row
template <typename TM, typename TX, typename TY, int MODE, bool ACC64, bool LIST = false>
__device__ __forceinline__ void spmv_scalar_warp(long wglob, int N, const int* __restrict__ rowptr,
                                                 const int* __restrict__ colidx, const TM* __restrict__ vals,
                                                 const TX* __restrict__ x, TY* __restrict__ y,
                                                 const TM* __restrict__ pre, const double* __restrict__ b,
                                                 const int* __restrict__ rows = nullptr, long nrows = 0) {
  using AT = typename AccT<TM, TX, ACC64>::type;
  const int lane = threadIdx.x & 31;
  const int sub = lane >> 3, k = lane & 7;
  const long rowl = wglob * 4 + sub;
  bool active;
  int row;
  if constexpr (LIST) {
    const int rl = rowl < nrows ? __ldg(rows + rowl) : -1;
    active = rl >= 0 && rl < N;
    row = active ? rl : 0;
  } else {
    active = rowl < N;
    row = active ? (int)rowl : 0;
  }
  AT a = 0;
  if (active) {
    const int s0 = __ldg(rowptr + row), s1 = __ldg(rowptr + row + 1);
    for (int s = s0 + k; s < s1; s += 8) a += (AT)ldm(vals + s) * (AT)__ldg(x + __ldg(colidx + s));
  }
  a += __shfl_xor_sync(0xffffffffu, a, 4);
  a += __shfl_xor_sync(0xffffffffu, a, 2);
  a += __shfl_xor_sync(0xffffffffu, a, 1);
  if (!active || k != 0) return;
  AT z = a;
  if (MODE == 1) z = a * (AT)pre[row];
  else if (MODE == 2) z = (AT)b[row] - a;
  y[row] = (TY)z;
}

template <typename TM, typename TX, typename TY, int MODE, bool ACC64>
__global__ void __launch_bounds__(SPMV_THREADS)
spmv_scalar_kernel(int N, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                   const TM* __restrict__ vals, const TX* __restrict__ x, TY* __restrict__ y,
                   const TM* __restrict__ pre, const double* __restrict__ b,
                   const int* __restrict__ done) {
  if (done && *done) return;
  const long wglob = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  spmv_scalar_warp<TM, TX, TY, MODE, ACC64>(wglob, N, rowptr, colidx, vals, x, y, pre, b);
}

template <typename TM, typename TX, typename TY, int MODE>
__global__ void __launch_bounds__(SPMV_THREADS)
spmv_scalar_rows_kernel(int N, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                        const TM* __restrict__ vals, const TX* __restrict__ x, TY* __restrict__ y,
                        const TM* __restrict__ pre, const int* __restrict__ rows, int nrows) {
  const long wglob = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  spmv_scalar_warp<TM, TX, TY, MODE, true, true>(wglob, N, rowptr, colidx, vals, x, y, pre, nullptr, rows, nrows);
}

// y = A x or P^-1 A x (MODE 0 / 1) on the listed rows only (FP64 vectors,
// FP64 accumulation as in the full FP64-vector product)
template <typename TM, int MODE>
int launch_spmv_rows(ovs_ctx* c, int sys, const TM* vals, const double* x, double* y, const TM* pre,
                     const int* rows, int nrows) {
  if (nrows <= 0) return OVS_OK;
  const int N = c->N;
  int rpw = sys == OVS_SYS_NS ? 8 : (sys == OVS_SYS_NSVOF ? 5 : 4);
  long warps = ((long)nrows + rpw - 1) / rpw;
  long blocks = (warps * 32 + SPMV_THREADS - 1) / SPMV_THREADS;
  if (sys == OVS_SYS_NS)
    spmv_block_rows_kernel<4, TM, double, double, MODE><<<(int)blocks, SPMV_THREADS, 0, c->stream>>>(
        N, c->rowptr, c->colidx, vals, x, y, pre, rows, nrows);
  else if (sys == OVS_SYS_NSVOF)
    spmv_block_rows_kernel<6, TM, double, double, MODE><<<(int)blocks, SPMV_THREADS, 0, c->stream>>>(
        N, c->rowptr, c->colidx, vals, x, y, pre, rows, nrows);
  else
    spmv_scalar_rows_kernel<TM, double, double, MODE><<<(int)blocks, SPMV_THREADS, 0, c->stream>>>(
        N, c->rowptr, c->colidx, vals, x, y, pre, rows, nrows);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  return OVS_OK;
}

template <typename TM, typename TX, typename TY, int MODE, bool ACC64 = true, bool AOS = false>
int launch_spmv(ovs_ctx* c, int sys, const TM* vals, const TX* x, TY* y, const TM* pre,
                const double* b, const int* done) {
  const int N = c->N;
  int rpw = sys == OVS_SYS_NS ? 8 : (sys == OVS_SYS_NSVOF ? 5 : 4);
  long warps = ((long)N + rpw - 1) / rpw;
  const int threads = sys != OVS_SYS_TEM ? spmv_threads<TM, AOS>() : SPMV_THREADS;
  long blocks = (warps * 32 + threads - 1) / threads;
  if (sys == OVS_SYS_NS)
    {
      spmv_block_kernel<4, TM, TX, TY, MODE, ACC64, AOS><<<(int)blocks, threads, 0, c->stream>>>(
          N, c->rowptr, c->colidx, vals, x, y, pre, b, done);
      ++c->launches;
    }
  else if (sys == OVS_SYS_NSVOF)
    {
      spmv_block_kernel<6, TM, TX, TY, MODE, ACC64, AOS><<<(int)blocks, threads, 0, c->stream>>>(
          N, c->rowptr, c->colidx, vals, x, y, pre, b, done);
      ++c->launches;
    }
  else
    {
      spmv_scalar_kernel<TM, TX, TY, MODE, ACC64><<<(int)blocks, threads, 0, c->stream>>>(
          N, c->rowptr, c->colidx, vals, x, y, pre, b, done);
      ++c->launches;
    }
  OVS_CUDA_TRY(cudaGetLastError());
  return OVS_OK;
}

// ------------------------------------------------------ preconditioner
// Diagonal block extraction (scan of each row for the diagonal, taken from
// the pattern) and inversion: SparseGMRES_NS.f90:53-121 (u: 3x3 inverse by
// cofactors, p: 1/M or 1 if M == 0), SparseGMRES_NS_conv.f:54-139 (phi:
// 1/LS or 0 if LS == 0), SparseGMRES_tem.f90:38-58 (1/M or 1).
template <typename TM>
__global__ void precond_setup_kernel(int N, int sys, const int* __restrict__ diag,
                                     const TM* __restrict__ vals, TM* __restrict__ pre) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int d = diag[i];
  if (sys == OVS_SYS_TEM) {
    double m = d >= 0 ? (double)vals[d] : 0.0;
    pre[i] = (TM)(m != 0.0 ? 1.0 / m : 1.0);
    return;
  }
  const int nv = sys == OVS_SYS_NS ? 16 : 24;
  double K[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, m = 0.0, ls = 0.0;
  if (d >= 0) {
    const TM* v = vals + (size_t)d * nv;
    K[0] = v[0]; K[1] = v[1]; K[2] = v[2];
    K[3] = v[4]; K[4] = v[5]; K[5] = v[6];
    K[6] = v[8]; K[7] = v[9]; K[8] = v[10];
    m = v[15];
    if (sys == OVS_SYS_NSVOF) ls = v[19];
  }
  const double b11 = K[4] * K[8] - K[7] * K[5];
  const double b12 = K[7] * K[2] - K[1] * K[8];
  const double b13 = K[1] * K[5] - K[2] * K[4];
  const double tmp2 = b11 * K[0] + b12 * K[3] + b13 * K[6];
  const double t = 1.0 / tmp2;
  TM* B = pre + (size_t)i * 9;
  B[0] = (TM)(b11 * t); B[1] = (TM)(b12 * t); B[2] = (TM)(b13 * t);
  B[3] = (TM)((K[5] * K[6] - K[3] * K[8]) * t);
  B[4] = (TM)((K[0] * K[8] - K[6] * K[2]) * t);
  B[5] = (TM)((K[3] * K[2] - K[0] * K[5]) * t);
  B[6] = (TM)((K[3] * K[7] - K[4] * K[6]) * t);
  B[7] = (TM)((K[6] * K[1] - K[0] * K[7]) * t);
  B[8] = (TM)((K[0] * K[4] - K[1] * K[3]) * t);
  pre[(size_t)9 * N + i] = (TM)(m == 0.0 ? 1.0 : 1.0 / m);
  if (sys == OVS_SYS_NSVOF) pre[(size_t)10 * N + i] = (TM)(ls == 0.0 ? 0.0 : 1.0 / ls);
}

// ------------------------------------------------ deterministic reductions
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    for (int k = 0; k < nw; ++k) r += sh[k];
  }
  __syncthreads();
  return r;  // valid in thread 0
}

// Finish a reduction: block partial -> gm->partials; the last block sums
// the partials in index order.  Returns true in thread 0 of the last block
// with the total in *total.
__device__ __forceinline__ bool finish_reduction(GmresDev* gm, double partial, double* total) {
  __shared__ double sh[32];
  __shared__ int is_last;
  if (threadIdx.x == 0) {
    gm->partials[blockIdx.x] = partial;
    __threadfence();
    const int t = atomicAdd(&gm->counter, 1);
    is_last = (t == (int)gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return false;
  __threadfence();
  double v = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) v += __ldcg(gm->partials + k);
  const double s = block_sum(v, sh);
  if (threadIdx.x == 0) {
    gm->counter = 0;
    *total = s;
    return true;
  }
  return false;
}

template <typename TV> __device__ __forceinline__ double dv(TV v) { return (double)v; }

// generic dot of two vectors (FP64 accumulate), result to gm->scal[k]
template <typename TA, typename TB>
__global__ void __launch_bounds__(OVS_RED_THREADS)
dot_kernel(const TA* __restrict__ a, const TB* __restrict__ b, size_t n, GmresDev* gm, int k) {
  __shared__ double sh[32];
  double s = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    s += dv(a[i]) * dv(b[i]);
  double part = block_sum(s, sh);
  double tot;
  if (finish_reduction(gm, part, &tot)) gm->scal[k] = tot;
}

// ---------------------------------------------------------------- GMRES
// v0 = P^-1 rhs (rhs FP64), ||v0||^2 -> unorm0, epsnrm, e(1)
template <typename TM, typename TV = double>
__global__ void __launch_bounds__(OVS_RED_THREADS)
gm_start_kernel(int N, int nf, int sys, const double* __restrict__ rhs, const TM* __restrict__ pre,
                TV* __restrict__ v0, double tol, GmresDev* gm, int raw) {  // v0: FP64 work vector
  __shared__ double sh[32];
  double s = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)N;
       i += (size_t)gridDim.x * blockDim.x) {
    if (raw) {   // rhs is already preconditioned
      for (int f = 0; f < nf; ++f) {
        const double z = rhs[(size_t)f * N + i];
        v0[i * nf + f] = (TV)z;
        s += z * z;
      }
    } else if (sys == OVS_SYS_TEM) {
      const double z = (double)pre[i] * rhs[i];
      v0[i] = (TV)z;
      s += z * z;
    } else {
      const double r0 = rhs[i], r1 = rhs[(size_t)N + i], r2 = rhs[2 * (size_t)N + i];
      const TM* B = pre + i * 9;
      const double z0 = (double)B[0] * r0 + (double)B[1] * r1 + (double)B[2] * r2;
      const double z1 = (double)B[3] * r0 + (double)B[4] * r1 + (double)B[5] * r2;
      const double z2 = (double)B[6] * r0 + (double)B[7] * r1 + (double)B[8] * r2;
      const double z3 = rhs[3 * (size_t)N + i] * (double)pre[(size_t)9 * N + i];
      TV* v = v0 + i * nf;
      v[0] = (TV)z0; v[1] = (TV)z1; v[2] = (TV)z2; v[3] = (TV)z3;
      s += z0 * z0 + z1 * z1 + z2 * z2 + z3 * z3;
      if (nf == 5) {
        const double z4 = rhs[4 * (size_t)N + i] * (double)pre[(size_t)10 * N + i];
        v[4] = (TV)z4;
        s += z4 * z4;
      }
    }
  }
  double part = block_sum(s, sh);
  double tot;
  if (finish_reduction(gm, part, &tot)) {
    const double un = sqrt(tot);
    gm->unorm0 = un;
    gm->epsnrm = tol * un;
    gm->e[0] = un;
    gm->sc[0] = 1.0;
    gm->iks = 0;
    gm->done = (un == 0.0) ? -1 : 0;
    gm->breakdown = (un == 0.0) ? 1 : 0;
    gm->converged = (un == 0.0) ? 1 : 0;
    gm->ercheck = un;
    gm->beta = 0.0;
  }
}

// Krylov vectors are stored with a padded leading dimension (multiple of
// 64 values) so every basis vector starts 256-byte aligned, by nodes (the nf
// values of a node side by side; start and update convert).  The product
// is written to its slot and orthogonalized there; dots are formed and added in
// FP64 for either precision.
inline size_t basis_ld(size_t n) { return (n + 63) & ~(size_t)63; }

__device__ __forceinline__ void ld4v(const float* p, double v[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ld4v(const double* p, double v[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void st4v(float* p, const double v[4]) {
  *reinterpret_cast<float4*>(p) = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
}
__device__ __forceinline__ void st4v(double* p, const double v[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// the first vector: v = w / unorm0 (SparseGMRES_NS.f90:159-160; later vectors
// stay unnormalized, see gm_orthog_kernel)
template <typename TV>
__global__ void __launch_bounds__(OVS_RED_THREADS)
gm_normalize_kernel(const double* w, TV* v, size_t n, const GmresDev* gm) {
  const double d = gm->unorm0;
  if (!(d != 0.0)) return;
  const size_t n4 = n >> 2, stride = (size_t)gridDim.x * blockDim.x;
  const size_t t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  for (size_t q = t0; q < n4; q += stride) {
    double a[4];
    ld4v(w + 4 * q, a);
    a[0] /= d; a[1] /= d; a[2] /= d; a[3] /= d;
    st4v(v + 4 * q, a);
  }
  for (size_t i = 4 * n4 + t0; i < n; i += stride) v[i] = (TV)(w[i] / d);
}

// H(k+1,k) = unorm, Givens rotations of column k (Hk[0..k) in, its rotated form
// out in Ho; cs, sn: the earlier rotations; ek: e(k)), e update, exit test
// (SparseGMRES_NS.f90:289-327); one thread.  The arrays do not overlap, so that
// the loads of several rotations go ahead of the chain.
__device__ void givens_step(GmresDev* gm, int k, double unorm, const double* __restrict__ Hk, double* __restrict__ Ho,
                            const double* __restrict__ cs, const double* __restrict__ sn, double ek) {
  const double epsnrm = gm->epsnrm;
  const int kmin = gm->kmin, kspace = gm->kspace;
  double cur = Hk[0];
#pragma unroll 8
  for (int jk = 1; jk <= k - 1; ++jk) {
    const double nxt = Hk[jk], c = cs[jk - 1], q = sn[jk - 1];
    Ho[jk - 1] = c * cur + q * nxt;
    cur = -q * cur + c * nxt;
  }
  const double a = cur, b = unorm;
  const double tmp = sqrt(a * a + b * b);
  if (tmp == 0.0) {
    // column k of H is zero (P^-1 A v_k has no component outside
    // v_1..v_{k-1}): the rotation would be 0/0 and the reference carries NaN
    // on; the cycle ends with the solution of the first k-1 columns
    gm->iks = k - 1;
    gm->ercheck = fabs(ek);
    gm->done = k;
    gm->converged = fabs(ek) <= epsnrm;
    gm->breakdown = 1;
    return;
  }
  const double c = a / tmp, sg = b / tmp;
  gm->cs[k - 1] = c;
  gm->sn[k - 1] = sg;
  Ho[k - 1] = tmp;
  gm->e[k - 1] = c * ek;   // e(k+1) was 0
  const double en = -sg * ek;
  gm->e[k] = en;
  const double er = fabs(en);
  gm->ercheck = er;
  gm->iks = k;
  const bool conv = (er <= epsnrm) && (k >= kmin);
  const bool brk = unorm == 0.0;  // exact breakdown; NaN propagates as in the reference
  if (conv || brk || k >= kspace) {
    gm->done = k;
    gm->converged = er <= epsnrm;
    gm->breakdown = brk;
  }
}

// One Arnoldi iteration k in a single cooperative launch (all blocks
// co-resident): w = P^-1 A v_k into basis slot k, the k+1 modified
// Gram-Schmidt steps of the reference order with one grid-wide barrier
// each, the normalization and the Givens update.  The Gram-Schmidt partial
// sums are double buffered, so one barrier per step suffices; every block
// adds the partials in the same order, so all see the same beta, and the
// result does not depend on timing.
template <typename TM, typename TV, int SYS, bool ACC64>
__global__ void __launch_bounds__(256)
gm_arnoldi_kernel(int N, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                  const TM* __restrict__ vals, const TM* __restrict__ pre, TV* V, size_t ld, size_t n,
                  int k, GmresDev* gm, double* part) {
  cg::grid_group grid = cg::this_grid();
  if (gm->done) return;
  __shared__ double sh[32];
  __shared__ double sbeta;
  const TV* vk = V + ld * (size_t)(k - 1);
  TV* w = V + ld * (size_t)k;
  // ---- w = P^-1 A v_k
  {
    constexpr int RPW = SYS == OVS_SYS_NS ? 8 : (SYS == OVS_SYS_NSVOF ? 5 : 4);
    const long nwarps = (long)gridDim.x * (blockDim.x >> 5);
    const long nchunks = ((long)N + RPW - 1) / RPW;
    for (long c = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nchunks; c += nwarps) {
      if constexpr (SYS == OVS_SYS_NS)
        spmv_block_warp<4, TM, TV, TV, 1, ACC64, false, true>(c, N, rowptr, colidx, vals, vk, w, pre, nullptr);
      else if constexpr (SYS == OVS_SYS_NSVOF)
        spmv_block_warp<6, TM, TV, TV, 1, ACC64, false, true>(c, N, rowptr, colidx, vals, vk, w, pre, nullptr);
      else
        spmv_scalar_warp<TM, TV, TV, 1, ACC64>(c, N, rowptr, colidx, vals, vk, w, pre, nullptr);
    }
  }
  grid.sync();
  // ---- modified Gram-Schmidt, SparseGMRES_NS.f90:246-287
  const size_t n4 = n >> 2, stride = (size_t)gridDim.x * blockDim.x;
  const size_t t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const int G = gridDim.x;
  double beta = 0.0;
  for (int j = 1; j <= k + 1; ++j) {
    const TV* vprev = j >= 2 ? V + ld * (size_t)(j - 2) : nullptr;
    const TV* vj = j <= k ? V + ld * (size_t)(j - 1) : nullptr;
    double sacc = 0.0;
    for (size_t q = t0; q < n4; q += stride) {
      double a[4], pv[4];
      ld4v(w + 4 * q, a);
      if (j >= 2) {
        ld4v(vprev + 4 * q, pv);
        a[0] = a[0] - beta * pv[0]; a[1] = a[1] - beta * pv[1];
        a[2] = a[2] - beta * pv[2]; a[3] = a[3] - beta * pv[3];
        st4v(w + 4 * q, a);
        if (sizeof(TV) == 4) ld4v(w + 4 * q, a);
      }
      if (vj) {
        ld4v(vj + 4 * q, pv);
        sacc += a[0] * pv[0] + a[1] * pv[1] + a[2] * pv[2] + a[3] * pv[3];
      } else {
        sacc += a[0] * a[0] + a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
      }
    }
    for (size_t i = 4 * n4 + t0; i < n; i += stride) {
      double a = (double)w[i];
      if (j >= 2) { a = a - beta * (double)vprev[i]; const TV ar = (TV)a; w[i] = ar; a = (double)ar; }
      sacc += a * (vj ? (double)vj[i] : a);
    }
    const double bp = block_sum(sacc, sh);
    double* pb = part + (size_t)(j & 1) * G;
    if (threadIdx.x == 0) pb[blockIdx.x] = bp;
    grid.sync();
    double v = 0.0;
    for (int b = threadIdx.x; b < G; b += blockDim.x) v += __ldcg(pb + b);
    const double tot = block_sum(v, sh);
    if (threadIdx.x == 0) sbeta = tot;
    __syncthreads();
    beta = sbeta;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      gm->H[(size_t)(k - 1) * (gm->kspace + 1) + (j - 1)] = beta;
      gm->beta = beta;
    }
    __syncthreads();
  }
  // ---- normalize (SparseGMRES_NS.f90:291-294) and the Givens update
  const double unorm = sqrt(beta);
  if (unorm != 0.0) {
    for (size_t q = t0; q < n4; q += stride) {
      double a[4];
      ld4v(w + 4 * q, a);
      a[0] /= unorm; a[1] /= unorm; a[2] /= unorm; a[3] /= unorm;
      st4v(w + 4 * q, a);
    }
    for (size_t i = 4 * n4 + t0; i < n; i += stride) w[i] = (TV)((double)w[i] / unorm);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    gm->sc[k] = 1.0;
    double* Hk = gm->H + (size_t)(k - 1) * (gm->kspace + 1);
    givens_step(gm, k, unorm, Hk, gm->y, gm->cs, gm->sn, gm->e[k - 1]);   // (y is free until the cycle ends)
    for (int j = 0; j < k; ++j) Hk[j] = gm->y[j];
  }
}

// ------------------------------------------------- Gram-Schmidt, one kernel
// The orthogonalization of Arnoldi step k (w = P^-1 A v_k, written to basis
// slot k by the SpMV launch before it) with the coefficients of modified
// Gram-Schmidt and one grid-wide barrier instead of one per coefficient.
// MGS takes h_j = v_j . (w - sum_{i<j} h_i v_i), that is
//   (I + L) h = V^T w,   L_ji = v_j . v_i (j > i),
// so V^T w and the new row of L (v_k . v_j) are all the reductions a step
// needs: the inverse compact WY form of MGS (Swirydowicz, Langou, Ananthan,
// Yang, Thomas, "Low synchronization Gram-Schmidt and generalized minimal
// residual algorithms", 2021).  T = (I + L)^-1 grows by a row per step.
//   phase A  every v_j is read once, for both dots (FP64 products and sums);
//   barrier  every block adds the partial dots in the same order and forms h;
//   phase B  w -= sum_j h_j v_j and the partial sums of |w|^2.
// What the step leaves over is done where nothing waits for it: block G, beside
// the others' phase A, finishes the step before (norm, Givens rotations, exit
// test) and adds the row of T that the next step will use (the newest two rows
// of the triangular solve are done directly); every other block adds the norm
// partials itself.  w stays unnormalized: gm->sc[j] = 1 / |w| belongs to slot j,
// and the product (linear in its vector), the dots and the coefficients carry
// it, which saves the barrier and the pass over w that a division would need.
// (FP32: the new vector takes the scale in FP64 and is rounded once.  With the
// scale rounded to FP32 first, all of it was off by up to 2^-25 from what h
// belongs to; the two conversions cost nothing, 126.7 us either way for an
// iteration at 1.2M values, 980 at 10.7M.)
// Each basis vector is read twice per step, as in MGS; the bound is that
// traffic (two vectors a step at 6.4 TB/s) for long vectors and the chain
// launch - dots - barrier - h - update for short ones.  One iteration at k = 25,
// product included, in FP64: 4.9K nodes 27 us ((u,p) system 22), 31K nodes 45, 233K
// nodes 0.196 ms, 2.1M nodes 1.71 ms; a step of a whole cycle of 50, host polls,
// start and update included: 31 (28), 52, 207 us and 1.76 ms.  With the leftovers
// in front of the barrier of their own step, the step of a cycle was 32 against 27,
// 61 against 58 and 232 against 227 us at the first three sizes when that was
// changed.
//
// A warp owns sub-chunks of 32 V values.  Phase A takes JG vectors at a
// time: all their loads in flight, 2 JG sums per lane, reduced over the
// lanes by halving (16 shuffles for 16 sums) into the warp's accumulators in
// shared memory.  With 32-byte loads (V = 4 in FP64, 8 in FP32) a sub-chunk
// takes all its vectors in turn, and phase B visits the sub-chunks in reverse, so
// that what phase A read last is still in L2; with shorter ones the sums over
// the lanes would cost more than that saves, and a group of vectors goes through
// all the warp's sub-chunks first (Gram-Schmidt at k = 25: 153K values 25 against
// 28 us; FP32, 1.2M values 64 against 66; FP64, 1.2M values 103 against 90 the
// other way round).  V = 1 for vectors that would not give every warp of the grid
// a sub-chunk of four; the groups of vectors are split over `js` shares of the
// warps (orth_split).
constexpr int ORTH_THREADS = 512;
constexpr int ORTH_WARPS = ORTH_THREADS / 32;
constexpr int JG = 8;

// V values at index i (a multiple of V), zero at and beyond n (plain loads: the
// slot being orthogonalized is rewritten by the same thread)
template <int V, typename TV>
__device__ __forceinline__ void orth_ld(const TV* p, size_t i, size_t n, TV (&x)[V]) {
  if (V >= 4 && i + V <= n) {
    if constexpr (V == 4 && sizeof(TV) == 8) {
      asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3]) : "l"(p + i));
    } else if constexpr (V == 8 && sizeof(TV) == 4) {
      asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7])
          : "l"(p + i));
    } else if constexpr (V == 4) {
      const float4 v = *reinterpret_cast<const float4*>(p + i);
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    }
    return;
  }
#pragma unroll
  for (int q = 0; q < V; ++q) x[q] = i + q < n ? p[i + q] : (TV)0;
}

// Sums over the 32 lanes of 2 JG = 16 values per lane: lane l (even) ends up
// with the sum of value 8 b4 + 4 b3 + 2 b2 + b1 (b the bits of l).
__device__ __forceinline__ double lanes_sum16(double (&p)[16], int lane) {
#pragma unroll
  for (int half = 8, off = 16; half >= 1; half >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double send = up ? p[i] : p[i + half], keep = up ? p[i + half] : p[i];
      p[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return p[0] + __shfl_xor_sync(0xffffffffu, p[0], 1);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// shared memory of a step: the warps' sums (2 kk each), a, g, g of the step
// before, h, h sc, sc
inline size_t orth_smem(int k) {
  const size_t kk = ((size_t)k + JG - 1) / JG * JG;
  return sizeof(double) * ((2 * ORTH_WARPS + 6) * kk + 2);
}

// four sums over the lanes at a time (their chains overlap)
__device__ __forceinline__ void warp_sum4(double (&v)[4]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] += __shfl_xor_sync(0xffffffffu, v[u], o);
}

// the sum of G values by one warp, all its loads in flight (G <= 160: one
// block per SM), the same on every block
__device__ __forceinline__ double warp_gather(const double* p, int G, int lane) {
  double s[5], t = 0.0;
#pragma unroll
  for (int u = 0; u < 5; ++u) s[u] = lane + 32 * u < G ? __ldcg(p + lane + 32 * u) : 0.0;
  for (int q = lane + 160; q < G; q += 32) t += __ldcg(p + q);
#pragma unroll
  for (int u = 0; u < 5; ++u) t += s[u];
  return warp_sum(t);
}

// part: partial norms (G) and dots with v_k (kspace) of step k and the step
// before, by the parity of k, then [2 k - 1][G] partial dots
__device__ __forceinline__ void orth_part(double* part, int k, int G, int ks, double*& nrm, double*& gsave) {
  nrm = part + (size_t)(k & 1) * (G + ks);
  gsave = nrm + G;
}

// What step k leaves over, by one block (sm: 12 k values of shared memory): the
// norm of slot k, the Givens rotations of column k and the exit test (one
// thread, its data staged in shared memory), and, by the other warps, row k - 1
// of T from the dots of v_k with the vectors before it.
__device__ void finish_step(GmresDev* gm, int k, double* part, int G, double* T, double* sm) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, ks = gm->kspace;
  double *acc = sm, *Hs = acc + 8 * k, *cs = Hs + k, *sn = cs + k, *Ho = sn + k, *nrm, *gk;
  orth_part(part, k, G, ks, nrm, gk);
  double* Hk = gm->H + (size_t)(k - 1) * (ks + 1);
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    Hs[j] = __ldcg(Hk + j);
    if (j < k - 1) { cs[j] = __ldcg(gm->cs + j); sn[j] = __ldcg(gm->sn + j); }
  }
  __shared__ double total;
  const double ek = threadIdx.x == 0 ? __ldcg(gm->e + (k - 1)) : 0.0;
  if (wid == 0) {
    const double t = warp_gather(nrm, G, lane);
    if (lane == 0) total = t;
  }
  __syncthreads();
  const int cols = k - 1, nt = blockDim.x - 32, parts = cols ? max(1, min(8, nt / cols)) : 0;
  if (threadIdx.x == 0) {
    const double unorm = sqrt(total);
    gm->beta = total;
    gm->sc[k] = unorm != 0.0 ? 1.0 / unorm : 1.0;
    givens_step(gm, k, unorm, Hs, Ho, cs, sn, ek);
  } else if (wid > 0) {
    // t_c = -(g_c + sum_{j>c} g_j T_jc), T's diagonal being 1; up to eight
    // threads share a column's sum
    for (int u = threadIdx.x - 32; u < cols * parts; u += nt) {
      const int q = u / cols, c = u - q * cols;
      double s = q == 0 ? __ldcg(gk + c) : 0.0;
#pragma unroll 4
      for (int j = c + 1 + q; j < cols; j += parts) s += __ldcg(gk + j) * __ldcg(T + (size_t)j * ks + c);
      acc[u] = s;
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += blockDim.x) Hk[j] = Ho[j];
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < parts; ++q) s += acc[q * cols + c];
    T[(size_t)(k - 1) * ks + c] = -s;
  }
}

// Step k by the blocks b < G of the grid (blockIdx G is finish_step's; it takes
// part in the barrier).
// part: partial norms (G) and dots with v_k (kspace) of step k and the step
// before, by the parity of k, then [2 k - 1][G] partial dots.
template <typename TV, int V>
__device__ __forceinline__ void orth_step(cg::grid_group& grid, TV* basis, size_t ld, size_t n, int k, int ks,
                                          GmresDev* gm, double* part, double* T, int nsc, int js, double* orth_sm) {
  __shared__ double sh[ORTH_WARPS];
  const int kk = (k + JG - 1) / JG * JG, ncol = 2 * k - 1;   // columns: k dots with w, k - 1 with v_k
  double* acc = orth_sm;                    // [ORTH_WARPS][2 kk]
  double* as = acc + 2 * ORTH_WARPS * kk;   // V^T w
  double* gs = as + kk;                     // v_k . v_j
  double* gp = gs + kk;                     // v_{k-1} . v_j
  double* hh = gp + kk;                     // the coefficients
  double* hs = hh + kk;                     // times the slots' scales
  double* sc = hs + kk;                     // the slots' scales
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int G = gridDim.x - 1, b = blockIdx.x, W = G * ORTH_WARPS;
  double *nrm, *gsave;
  orth_part(part, k, G, ks, nrm, gsave);
  double *nrm1, *gsave1;                    // of the step before
  orth_part(part, k - 1, G, ks, nrm1, gsave1);
  double* col = part + 2 * (G + ks);
  const int gw = wid * G + b;               // short vectors spread over the blocks first
  const TV* vk = basis + ld * (size_t)(k - 1);
  TV* w = basis + ld * (size_t)k;
  double* my = acc + 2 * kk * wid;
  for (int c = lane; c < 2 * kk; c += 32) my[c] = 0.0;
  // the scales and the older dots travel while phase A runs
  const int t = threadIdx.x;
  const double sct = t < k - 1 ? __ldcg(gm->sc + t) : 0.0, gpt = t < k - 2 ? __ldcg(gsave1 + t) : 0.0;
  if (wid == ORTH_WARPS - 1) {              // 1 / |v_k| from the norm partials
    const double u = k > 1 ? sqrt(warp_gather(nrm1, G, lane)) : 1.0;
    if (lane == 0) sc[k - 1] = u != 0.0 ? 1.0 / u : 1.0;
  }
  __syncwarp();
  // ---- phase A
  const int slot = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
  auto dots = [&](int j0, size_t i, const TV (&wv)[V], const TV (&kv)[V], double (&p)[2 * JG]) {
    TV x[JG][V];
#pragma unroll
    for (int u = 0; u < JG; ++u) orth_ld<V>(basis + ld * (size_t)min(j0 + u, k - 1), i, n, x[u]);
#pragma unroll
    for (int u = 0; u < JG; ++u) {
#pragma unroll
      for (int q = 0; q < V; ++q) {
        p[u] += (double)wv[q] * (double)x[u][q];
        p[JG + u] += (double)kv[q] * (double)x[u][q];
      }
    }
  };
  auto add = [&](int j0, double (&p)[2 * JG]) {
    const double s = lanes_sum16(p, lane);
    if (!(lane & 1)) my[(slot < JG ? 0 : kk - JG) + j0 + slot] += s;
  };
  if (V == 1 || (V == 4 && sizeof(TV) == 4)) {   // short vectors: a warp's sub-chunks inside a group, one sum over the lanes per group
    const int Wj = W / js, jj = gw % js, si0 = gw / js;   // Wj warps per share of the groups
    for (int j0 = jj * JG; j0 < k && si0 < min(Wj, nsc); j0 += js * JG) {
      double p[2 * JG] = {};
      for (long si = si0; si < nsc; si += Wj) {
        const size_t i = ((size_t)si * 32 + lane) * V;
        TV wv[V], kv[V];
        orth_ld<V>(w, i, n, wv);
        orth_ld<V>(vk, i, n, kv);
        dots(j0, i, wv, kv, p);
      }
      add(j0, p);
    }
  } else {
    for (long si = gw; si < nsc; si += W) {
      const size_t i = ((size_t)si * 32 + lane) * V;
      TV wv[V], kv[V];
      orth_ld<V>(w, i, n, wv);
      orth_ld<V>(vk, i, n, kv);
      for (int j0 = 0; j0 < k; j0 += JG) {
        double p[2 * JG] = {};
        dots(j0, i, wv, kv, p);
        add(j0, p);
      }
    }
  }
  if (t < k - 1) sc[t] = sct;
  if (t < k - 2) gp[t] = gpt;
  __syncthreads();
  for (int c = threadIdx.x; c < ncol; c += ORTH_THREADS) {
    const int o = c < k ? c : kk + c - k;
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < ORTH_WARPS; ++q) s += acc[2 * kk * q + o];
    col[(size_t)c * G + b] = s;
  }
  grid.sync();
  const int done = *(volatile int*)&gm->done;   // the step before may have ended the cycle
  // ---- the dots, added over the blocks in the same order everywhere (four
  // columns of a warp's share in flight)
  const double sk = sc[k - 1];
  for (int c0 = wid; c0 < ncol; c0 += 4 * ORTH_WARPS) {
    double s[4][5];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = min(c0 + u * ORTH_WARPS, ncol - 1);
#pragma unroll
      for (int v = 0; v < 5; ++v) s[u][v] = lane + 32 * v < G ? __ldcg(col + (size_t)c * G + lane + 32 * v) : 0.0;
    }
    double r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      r[u] = 0.0;
      for (int q = lane + 160; q < G; q += 32) r[u] += __ldcg(col + (size_t)min(c0 + u * ORTH_WARPS, ncol - 1) * G + q);
#pragma unroll
      for (int v = 0; v < 5; ++v) r[u] += s[u][v];
    }
    warp_sum4(r);
    if (lane < 4) {
      const double v = (lane & 2) ? ((lane & 1) ? r[3] : r[2]) : ((lane & 1) ? r[1] : r[0]);
      const int c = c0 + lane * ORTH_WARPS;
      if (c < k) as[c] = v * sk * sc[c];
      else if (c < ncol) gs[c - k] = v * sk * sc[c - k];
    }
  }
  if (done) return;
  __syncthreads();
  // ---- h = T V^T w for rows 0..k-3 of T; the last two rows are direct
  // (four rows of a warp's share in flight)
  for (int j0 = wid; j0 < k - 2; j0 += 4 * ORTH_WARPS) {
    double s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u * ORTH_WARPS;
      const bool in0 = j < k - 2 && lane < j, in1 = j < k - 2 && lane + 32 < j;
      const double* Tj = T + (size_t)j * ks + lane;
      const double x0 = in0 ? __ldcg(Tj) : 0.0, x1 = in1 ? __ldcg(Tj + 32) : 0.0;
      s[u] = (in0 ? x0 * as[lane] : 0.0) + (in1 ? x1 * as[lane + 32] : 0.0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u * ORTH_WARPS;
      if (j < k - 2)
        for (int c = lane + 64; c < j; c += 32) s[u] += __ldcg(T + (size_t)j * ks + c) * as[c];
    }
    warp_sum4(s);
    if (lane < 4) {
      const double v = (lane & 2) ? ((lane & 1) ? s[3] : s[2]) : ((lane & 1) ? s[1] : s[0]);
      const int j = j0 + lane * ORTH_WARPS;
      if (j < k - 2) {
        hh[j] = as[j] + v;
        hs[j] = hh[j] * sc[j];
      }
    }
  }
  __syncthreads();
  if (wid == 0) {
    double t1 = 0.0, t2 = 0.0;
    for (int j = lane; j < k - 2; j += 32) { t1 += gp[j] * hh[j]; t2 += gs[j] * hh[j]; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      t2 += __shfl_xor_sync(0xffffffffu, t2, o);
    }
    if (lane == 0) {
      if (k > 1) {
        const double h = as[k - 2] - t1;
        hh[k - 2] = h;
        hs[k - 2] = h * sc[k - 2];
        t2 += gs[k - 2] * h;
      }
      hh[k - 1] = as[k - 1] - t2;
      hs[k - 1] = hh[k - 1] * sk;
    }
  }
  __syncthreads();
  if (b == 0) {   // for finish_step and the next step
    for (int j = threadIdx.x; j < k; j += ORTH_THREADS) {
      gm->H[(size_t)(k - 1) * (ks + 1) + j] = hh[j];
      if (j < k - 1) gsave[j] = gs[j];
    }
  }
  // ---- phase B: the update and its norm
  double na = 0.0;
  const int cnt = gw < nsc ? (nsc - gw + W - 1) / W : 0;
  auto update = [&](auto nb, int r) {   // sub-chunks r, r - 1, .. of the warp's, their loads in flight together
    constexpr int NB = decltype(nb)::value, JB = V == 1 ? 2 * JG : JG;
    size_t i[NB];
    TV wv[NB][V];
#pragma unroll
    for (int m = 0; m < NB; ++m) {
      i[m] = ((size_t)(gw + (long)(r - m) * W) * 32 + lane) * V;
      orth_ld<V>(w, i[m], n, wv[m]);
#pragma unroll
      for (int q = 0; q < V; ++q) wv[m][q] = (TV)((double)wv[m][q] * sk);   // the coefficients' own sk, not its FP32 rounding
    }
    for (int j0 = 0; j0 < k; j0 += JB) {
      TV x[NB][JB][V];
#pragma unroll
      for (int m = 0; m < NB; ++m)
#pragma unroll
        for (int u = 0; u < JB; ++u) orth_ld<V>(basis + ld * (size_t)min(j0 + u, k - 1), i[m], n, x[m][u]);
#pragma unroll
      for (int u = 0; u < JB; ++u) {
        const TV h = j0 + u < k ? (TV)hs[j0 + u] : (TV)0;
#pragma unroll
        for (int m = 0; m < NB; ++m)
#pragma unroll
          for (int q = 0; q < V; ++q) wv[m][q] = fma(-h, x[m][u][q], wv[m][q]);
      }
    }
#pragma unroll
    for (int m = 0; m < NB; ++m) {
      if (V >= 4 && i[m] + V <= n) {
#pragma unroll
        for (int q = 0; q + 4 <= V; q += 4) {
          const double d[4] = {(double)wv[m][q], (double)wv[m][q + 1], (double)wv[m][q + 2], (double)wv[m][q + 3]};
          st4v(w + i[m] + q, d);
        }
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (i[m] + q < n) w[i[m] + q] = wv[m][q];
      }
#pragma unroll
      for (int q = 0; q < V; ++q) na += (double)wv[m][q] * (double)wv[m][q];
    }
  };
  int r = cnt - 1;
  if constexpr (V == 1 && sizeof(TV) == 4)
    for (; r >= 1; r -= 2) update(std::integral_constant<int, 2>(), r);
  for (; r >= 0; --r) update(std::integral_constant<int, 1>(), r);
  na = warp_sum(na);
  if (lane == 0) sh[wid] = na;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < ORTH_WARPS; ++q) s += sh[q];
    nrm[b] = s;
  }
}

// one step per launch (after the SpMV that wrote slot k)
template <typename TV, int V>
__global__ void __launch_bounds__(ORTH_THREADS, 1)
gm_orthog_kernel(TV* basis, size_t ld, size_t n, int k, GmresDev* gm, double* part, double* T, int nsc, int js) {
  cg::grid_group grid = cg::this_grid();
  // ended by a step before the one that block G finishes here (the same answer
  // on every block, whenever it starts)
  const int ended = *(volatile int*)&gm->done;
  if (ended != 0 && ended < k - 1) return;
  extern __shared__ __align__(16) double orth_sm[];
  const int G = gridDim.x - 1;
  if (blockIdx.x == G) {
    if (k > 1) finish_step(gm, k - 1, part, G, T, orth_sm);
    grid.sync();
    return;
  }
  orth_step<TV, V>(grid, basis, ld, n, k, gm->kspace, gm, part, T, nsc, js, orth_sm);
}

// back-substitution (SparseGMRES_NS.f90:341-346): one block, thread l holds
// e(l); the columns of H are loaded eight at a time ahead of the steps that
// use them.  y_j comes out times the scale of slot j.  A cycle that ran all its
// steps first finishes the last one (part, T, G: of gm_orthog_kernel).
constexpr int BACKSUB_THREADS = 416;
static_assert(BACKSUB_THREADS >= OVS_MAX_KSPACE, "one thread per unknown");
__global__ void __launch_bounds__(BACKSUB_THREADS) gm_backsub_kernel(GmresDev* gm, double* part, double* T, int G) {
  __shared__ double ys;
  extern __shared__ __align__(16) double bs_sm[];
  if (!gm->done) {
    const int k = gm->kspace;
    finish_step(gm, k, part, G, T, bs_sm);
    __threadfence();
    __syncthreads();
  }
  const int iks = *(volatile int*)&gm->iks, ld = gm->kspace + 1, t = threadIdx.x;
  double e = t < iks ? __ldcg(gm->e + t) : 0.0;
  for (int j1 = iks; j1 > 0; j1 -= 8) {
    double h[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j1 - 1 - u;
      h[u] = j >= 0 && t <= j ? __ldcg(gm->H + (size_t)j * ld + t) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j1 - 1 - u;
      if (j < 0) break;
      if (t == j) ys = e / h[u];
      __syncthreads();
      const double y = ys;
      if (t == j) gm->y[j] = y * __ldcg(gm->sc + j);
      else if (t < j) e = e - y * h[u];
      __syncthreads();
    }
  }
}

// sol += sum_j y_j v_j (SparseGMRES_NS.f90:349-352), eight vectors' loads in
// flight per value; sol is by fields, the basis by nodes
template <typename TV>
__global__ void __launch_bounds__(256)
gm_update_kernel(double* __restrict__ sol, const TV* __restrict__ basis, size_t n, size_t ld, int nf,
                 const GmresDev* __restrict__ gm) {
  __shared__ double y[OVS_MAX_KSPACE];
  const int iks = gm->iks;
  for (int j = threadIdx.x; j < iks; j += blockDim.x) y[j] = gm->y[j];
  __syncthreads();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t node = i / (unsigned)nf, o = (i - node * nf) * (n / (unsigned)nf) + node;
    double s = sol[o];
    int j = 0;
    for (; j + 8 <= iks; j += 8) {
      TV x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __ldcs(basis + (size_t)(j + u) * ld + i);
#pragma unroll
      for (int u = 0; u < 8; ++u) s = s + y[j + u] * (double)x[u];
    }
    for (; j < iks; ++j) s = s + y[j] * (double)basis[(size_t)j * ld + i];
    sol[o] = s;
  }
}

// elementwise helpers
template <typename TS, typename TD>
__global__ void convert_kernel(const TS* __restrict__ a, TD* __restrict__ b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b[i] = (TD)a[i];
}

// --------------------------------------------------------- host drivers
template <typename T> const T* as(const void* p) { return reinterpret_cast<const T*>(p); }

int ensure_basis(ovs_ctx* c, int prec, size_t bytes) {
  if (c->basis_bytes[prec] >= bytes) return OVS_OK;
  if (c->basis[prec]) cudaFree(c->basis[prec]);
  c->basis[prec] = nullptr;
  c->basis_bytes[prec] = 0;
  if (cudaMalloc(&c->basis[prec], bytes) != cudaSuccess) {
    cudaGetLastError();
    return OVS_ERR_NOMEM;
  }
  c->basis_bytes[prec] = bytes;
  return OVS_OK;
}

// Launch plan of the Arnoldi iterations of a cycle.  Default: the
// preconditioned SpMV as an ordinary launch, then gm_orthog_kernel (one
// 512-thread block per SM at most, cooperative).  fused = 1 (environment
// OVS_ARNOLDI_FUSED=1, or when the blocks cannot be made co-resident):
// gm_arnoldi_kernel alone.
struct ArnoldiPlan {
  bool fused = false;
  int grid = 0;
  int v = 1;           // values per lane (1, 4 or 8)
  int nsc = 0;         // sub-chunks of 32 V values
  double* T = nullptr;
};

template <typename TM, typename TV, bool ACC64>
using ArnoldiKern = void (*)(int, const int*, const int*, const TM*, const TM*, TV*, size_t, size_t, int,
                             GmresDev*, double*);

template <typename TM, typename TV, bool ACC64>
ArnoldiKern<TM, TV, ACC64> fused_kernel(int sys) {
  if (sys == OVS_SYS_NS) return gm_arnoldi_kernel<TM, TV, OVS_SYS_NS, ACC64>;
  if (sys == OVS_SYS_NSVOF) return gm_arnoldi_kernel<TM, TV, OVS_SYS_NSVOF, ACC64>;
  return gm_arnoldi_kernel<TM, TV, OVS_SYS_TEM, ACC64>;
}

template <typename TV>
auto orthog_kernel(int v) {
  using Kern = void (*)(TV*, size_t, size_t, int, GmresDev*, double*, double*, int, int);
  if constexpr (sizeof(TV) == 4)
    if (v == 8) return (Kern)gm_orthog_kernel<TV, 8>;
  return v == 4 ? (Kern)gm_orthog_kernel<TV, 4> : (Kern)gm_orthog_kernel<TV, 1>;
}

// Shares into which the groups of vectors of step k are split over the warps of
// the grid (a share's warps take a group through all their sub-chunks).  FP64: as
// many as leave every warp one sub-chunk at most; more shares than that even out
// the warps' rounds but read w and v_k once more each, which long FP64 vectors pay
// for (296K values 37 against 33 us).  FP32: the fewest rounds of eight loads for
// the warp that has the most, a sum over the lanes counted as two rounds (Gram-
// Schmidt at k = 25, with two sub-chunks at a time in phase B: 78K values 22.5 ->
// 18.8 us, 176K 29.5 -> 27.6, 345K 36 -> 32).
template <typename TV>
int orth_split(const ArnoldiPlan& pl, int k) {
  const int groups = (k + JG - 1) / JG, W = pl.grid * ORTH_WARPS;
  if (sizeof(TV) == 8) return std::min(groups, std::max(1, W / std::max(1, pl.nsc)));
  int best = 1;
  long cost = 0;
  for (int js = 1; js <= groups && js <= W; ++js) {
    const long wj = W / js, c = ((pl.nsc + wj - 1) / wj + 2) * ((groups + js - 1) / js);
    if (js == 1 || c < cost) { best = js; cost = c; }
  }
  return best;
}

template <typename TM, typename TV, bool ACC64>
int plan_arnoldi(ovs_ctx* c, int sys, size_t n, int kspace, bool want_fused, ArnoldiPlan* pl) {
  int st;
  // the partial sums (fused variant: two per block; gm_orthog_kernel: 2 k per
  // block and two rows of dots), then T, kspace x kspace; kept by the context,
  // grown when needed
  const size_t parts = std::max((size_t)2 * OVS_COOP_MAX_BLOCKS, (size_t)2 * (kspace + 1) * (c->num_sms + 1));
  const size_t need = sizeof(double) * (parts + (size_t)kspace * kspace);
  if (c->coop_bytes < need) {
    if (c->coop_part) cudaFree(c->coop_part);
    c->coop_part = nullptr;
    c->coop_bytes = 0;
    if ((st = ovs_ensure((void**)&c->coop_part, need))) return st;
    c->coop_bytes = need;
  }
  pl->T = c->coop_part + parts;
  pl->fused = want_fused;
  if (!want_fused) {
    // V = 4 once it gives every warp of the chip a sub-chunk; FP32 V = 8 (32-byte
    // loads, as V = 4 in FP64) once it gives every warp four: Gram-Schmidt at k = 25
    // 0.132 against 0.139 ms at 3.2M values, 0.180 against 0.192 at 4.6M, but 0.110
    // against 0.104 at 2.1M
    const size_t chip = (size_t)32 * ORTH_WARPS * c->num_sms;
    pl->v = sizeof(TV) == 4 && n >= 32 * chip ? 8 : (n >= 4 * chip ? 4 : 1);
    const size_t per = 32 * pl->v, nsc = (n + per - 1) / per;
    auto kern = orthog_kernel<TV>(pl->v);
    const size_t bytes = orth_smem(kspace);
    int per_sm = 0;
    // the limit belongs to the kernel, whatever the context: always the largest
    // space's (121,616 bytes), so that no call lowers it under another thread's cycle
    OVS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)orth_smem(OVS_MAX_KSPACE)));
    OVS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, ORTH_THREADS, bytes));
    if (per_sm >= 1 && c->num_sms >= 2 && nsc < ((size_t)1 << 31)) {
      pl->nsc = (int)nsc;
      // one SM is left for the block that finishes the step before
      pl->grid = c->num_sms - 1;
      const int shares = sizeof(TV) == 8 ? orth_split<TV>(*pl, kspace) : (kspace + JG - 1) / JG;
      pl->grid = (int)std::min((long)pl->grid, ((long)nsc * shares + ORTH_WARPS - 1) / ORTH_WARPS);
      return OVS_OK;
    }
    pl->fused = true;
  }
  int per_sm = 0;
  OVS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_kernel<TM, TV, ACC64>(sys), 256, 0));
  if (per_sm < 1) return OVS_ERR_CUDA;
  pl->grid = per_sm * c->num_sms;
  if (pl->grid > OVS_COOP_MAX_BLOCKS) pl->grid = OVS_COOP_MAX_BLOCKS;
  return OVS_OK;
}

// Arnoldi iteration k (1-based) on basis V (leading dimension ld, n values)
template <typename TM, typename TV, bool ACC64>
int launch_arnoldi(ovs_ctx* c, int sys, const ArnoldiPlan& pl, const TM* vals, const TM* pre, TV* V, size_t ld,
                   size_t n, int k) {
  GmresDev* gm = c->gm;
  double* part = c->coop_part;
  if (pl.fused) {
    int Nn = c->N, kk = k;
    const int* rp = c->rowptr;
    const int* ci = c->colidx;
    size_t ldv = ld, nn = n;
    void* args[] = {&Nn, &rp, &ci, (void*)&vals, (void*)&pre, &V, &ldv, &nn, &kk, &gm, &part};
    OVS_CUDA_TRY(cudaLaunchCooperativeKernel((void*)fused_kernel<TM, TV, ACC64>(sys), pl.grid, 256, args, 0,
                                             c->stream));
    ++c->launches;
    return OVS_OK;
  }
  int st = launch_spmv<TM, TV, TV, 1, ACC64, true>(c, sys, vals, V + ld * (size_t)(k - 1), V + ld * (size_t)k, pre,
                                               nullptr, &gm->done);
  if (st) return st;
  int kk = k, nsc = pl.nsc, js = orth_split<TV>(pl, k);
  size_t ldv = ld, nn = n;
  double* T = pl.T;
  void* args[] = {&V, &ldv, &nn, &kk, &gm, &part, &T, &nsc, &js};
  OVS_CUDA_TRY(cudaLaunchCooperativeKernel((void*)orthog_kernel<TV>(pl.v), pl.grid + 1, ORTH_THREADS, args,
                                           orth_smem(k), c->stream));
  ++c->launches;
  return OVS_OK;
}

// One GMRES cycle on system `sys` with matrix/preconditioner precision TM
// and basis precision TV.  rhs and sol are FP64 device vectors (nf*N).
// rhs_pre: rhs is P^-1 times the right-hand side already (the cycle then
// solves P^-1 A x = rhs)
// feed: sol is still on its way from the host (SolFeed)
template <typename TM, typename TV, bool ACC64 = true>
int gmres_cycle(ovs_ctx* c, int sys, const double* rhs, double* sol, double tol, int kspace,
                int kmin, ovs_gmres_info* info, bool rhs_pre = false, SolFeed* feed = nullptr) {
  const int N = c->N, nf = ovs_sys_nf(sys);
  const size_t n = (size_t)N * nf;
  const int prec = sizeof(TM) == 8 ? OVS_FP64 : OVS_FP32;
  SysStore& S = c->sys[sys][prec];
  if (!S.vals || !S.binv) return OVS_ERR_STATE;
  if (kspace < 1 || kspace > OVS_MAX_KSPACE) return OVS_ERR_ARG;
  const int bprec = sizeof(TV) == 8 ? OVS_FP64 : OVS_FP32;
  const size_t ld = basis_ld(n);
  int st;
  if ((st = ensure_basis(c, bprec, sizeof(TV) * ld * (size_t)(kspace + 1)))) return st;
  if ((st = ovs_ensure((void**)&c->wvec, sizeof(double) * basis_ld(5 * (size_t)N)))) return st;
  TV* V = reinterpret_cast<TV*>(c->basis[bprec]);
  // v_1 = P^-1 rhs / ||P^-1 rhs|| through the FP64 work vector; later
  // vectors are orthogonalized in place in their basis slot
  double* wd = c->wvec;
  GmresDev* gm = c->gm;
  cudaStream_t s = c->stream;
  const TM* vals = as<TM>(S.vals);
  const TM* pre = as<TM>(S.binv);
  // set kspace/kmin and clear the Hessenberg matrix
  int km[2] = {kspace, kmin};
  OVS_CUDA_TRY(cudaMemcpyAsync(&gm->kspace, km, sizeof(km), cudaMemcpyHostToDevice, s));
  OVS_CUDA_TRY(cudaMemsetAsync(gm->H, 0, sizeof(double) * (size_t)(kspace + 1) * kspace, s));
  OVS_CUDA_TRY(cudaMemsetAsync(gm->e, 0, sizeof(double) * (size_t)(kspace + 1), s));
  gm_start_kernel<TM, double><<<OVS_RED_BLOCKS, OVS_RED_THREADS, 0, s>>>(N, nf, sys, rhs, pre, wd, tol, gm,
                                                                         rhs_pre ? 1 : 0);
  gm_normalize_kernel<TV><<<OVS_RED_BLOCKS, OVS_RED_THREADS, 0, s>>>(wd, V, n, gm);
  c->launches += 2;
  OVS_CUDA_TRY(cudaGetLastError());
  // one Arnoldi iteration per step (see ArnoldiPlan)
  ArnoldiPlan pl;
  if ((st = plan_arnoldi<TM, TV, ACC64>(c, sys, n, kspace, c->arnoldi_fused, &pl))) return st;
  // the host reads the done word of a batch while the next one runs; what is
  // queued after the end of the cycle returns at once
  const int batch = N > 200000 ? 4 : 8;
  c->h_pinned[0] = c->h_pinned[1] = 0;
  for (int k = 1, q = 0; k <= kspace; ++q) {
    const int kend = (k + batch - 1 < kspace) ? k + batch - 1 : kspace;
    for (; k <= kend; ++k)
      if ((st = launch_arnoldi<TM, TV, ACC64>(c, sys, pl, vals, pre, V, ld, n, k))) return st;
    // a piece takes the host less time than the device has work queued (27 ms for
    // all five columns of 2.1M nodes, 7 ms for four steps)
    if (feed && (st = ovs_feed(c, feed, feed->n * feed->ncol / 5 + 1))) return st;
    if (k > kspace) break;
    OVS_CUDA_TRY(cudaMemcpyAsync(c->h_pinned + (q & 1), &gm->done, sizeof(int), cudaMemcpyDeviceToHost, s));
    OVS_CUDA_TRY(cudaEventRecord(c->ev_poll[q & 1], s));
    if (q > 0) {
      OVS_CUDA_TRY(cudaEventSynchronize(c->ev_poll[(q - 1) & 1]));
      if (c->h_pinned[(q - 1) & 1]) break;
    }
  }
  if (feed) {
    if ((st = ovs_feed(c, feed, 0))) return st;
    OVS_CUDA_TRY(cudaEventRecord(c->ev_sol, c->sol_stream));
    OVS_CUDA_TRY(cudaStreamWaitEvent(s, c->ev_sol, 0));
  }
  gm_backsub_kernel<<<1, BACKSUB_THREADS, sizeof(double) * 12 * kspace, s>>>(gm, c->coop_part, pl.T, pl.grid);
  ++c->launches;
  gm_update_kernel<TV><<<ovs_grid(n, 256, 8 * c->num_sms), 256, 0, s>>>(sol, V, n, ld, nf, gm);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  if (info) {
    GmresDev h;
    OVS_CUDA_TRY(cudaMemcpyAsync(&h, gm, offsetof(GmresDev, H), cudaMemcpyDeviceToHost, s));
    OVS_CUDA_TRY(cudaStreamSynchronize(s));
    info->iterations = h.iks;
    info->converged = h.converged;
    info->breakdown = h.breakdown;
    info->res0 = h.unorm0;
    info->ercheck = h.ercheck;
  }
  return OVS_OK;
}

int dot64(ovs_ctx* c, const double* a, const double* b, size_t n, double* out) {
  dot_kernel<double, double><<<OVS_RED_BLOCKS, OVS_RED_THREADS, 0, c->stream>>>(a, b, n, c->gm, 0);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  OVS_CUDA_TRY(cudaMemcpyAsync(c->h_pinned_d, c->gm->scal, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  OVS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  *out = c->h_pinned_d[0];
  return OVS_OK;
}

}  // namespace

template <typename TV>
__global__ void fill_kernel(TV* __restrict__ p, size_t n, double v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    p[i] = (TV)(v * (1.0 + 1e-3 * (double)(i % 97)));
}

// Time one Arnoldi iteration (k = 25 of a 50-vector cycle) or one
// preconditioned SpMV on the resident system.
template <typename TM, bool ACC64>
int profile_krylov_t(ovs_ctx* c, int what, int sys, int reps, double* ms) {
  const int prec = sizeof(TM) == 8 ? OVS_FP64 : OVS_FP32;
  SysStore& S = c->sys[sys][prec];
  if (!S.vals) return OVS_ERR_STATE;
  int st;
  if ((st = ovs_precond_setup(c, sys, prec))) return st;
  const size_t n = (size_t)c->N * ovs_sys_nf(sys);
  const size_t ld = basis_ld(n);
  const int kspace = 50, k = 25;
  if ((st = ensure_basis(c, prec, sizeof(TM) * ld * (kspace + 1)))) return st;
  TM* V = reinterpret_cast<TM*>(c->basis[prec]);
  fill_kernel<TM><<<1184, 256, 0, c->stream>>>(V, ld * (kspace + 1), 1.0);
  ++c->launches;
  GmresDev* gm = c->gm;
  int km[2] = {kspace, 1};
  OVS_CUDA_TRY(cudaMemcpyAsync(&gm->kspace, km, sizeof(km), cudaMemcpyHostToDevice, c->stream));
  OVS_CUDA_TRY(cudaMemsetAsync(&gm->done, 0, sizeof(int), c->stream));
  // no exit test passes, and the slots hold what they hold
  const double eps = -1.0;
  const std::vector<double> ones(OVS_MAX_KSPACE + 1, 1.0);
  OVS_CUDA_TRY(cudaMemcpyAsync(&gm->epsnrm, &eps, sizeof(double), cudaMemcpyHostToDevice, c->stream));
  OVS_CUDA_TRY(cudaMemcpyAsync(gm->sc, ones.data(), sizeof(gm->sc), cudaMemcpyHostToDevice, c->stream));
  const TM* vals = as<TM>(S.vals);
  const TM* pre = as<TM>(S.binv);
  ArnoldiPlan pl;
  if ((st = plan_arnoldi<TM, TM, ACC64>(c, sys, n, kspace, what == OVS_PROF_ARNOLDI_FUSED, &pl))) return st;
  OVS_CUDA_TRY(cudaMemsetAsync(pl.T, 0, sizeof(double) * kspace * kspace, c->stream));
  fill_kernel<double><<<1, 256, 0, c->stream>>>(c->coop_part, 2 * ((size_t)pl.grid + kspace), 1.0);   // a norm before
  ++c->launches;
  auto run = [&]() -> int {
    if (what == OVS_PROF_SPMV) {
      st = launch_spmv<TM, TM, TM, 1, ACC64, true>(c, sys, vals, V, V + ld, pre, nullptr, nullptr);
      return st;
    }
    return launch_arnoldi<TM, TM, ACC64>(c, sys, pl, vals, pre, V, ld, n, k);
  };
  if ((st = run())) return st;
  OVS_CUDA_TRY(cudaEventRecord(c->ev0, c->stream));
  for (int r = 0; r < reps; ++r)
    if ((st = run())) return st;
  OVS_CUDA_TRY(cudaEventRecord(c->ev1, c->stream));
  OVS_CUDA_TRY(cudaEventSynchronize(c->ev1));
  float t = 0.f;
  OVS_CUDA_TRY(cudaEventElapsedTime(&t, c->ev0, c->ev1));
  *ms = (double)t / reps;
  return OVS_OK;
}

int ovs_profile_krylov(ovs_ctx* c, int what, int sys, int prec, int reps, double* ms) {
  if (prec == OVS_FP64) return profile_krylov_t<double, true>(c, what, sys, reps, ms);
  return profile_krylov_t<float, false>(c, what, sys, reps, ms);
}

// calculate_residual: the sums of squares of the four residual fields (rhs:
// nfs N flow values - u, p and, for nfs = 5, phi - and N temperature values;
// either may be null), all in one launch with the fixed order of every
// reduction here (one launch and one read-back: a copy, a dot and a wait per
// field were 8 launches and 4 waits).
template <typename T>
__global__ void __launch_bounds__(OVS_RED_THREADS)
resnorm_kernel(const T* __restrict__ flow, int nfs, const T* __restrict__ tem, size_t N, GmresDev* gm) {
  __shared__ double sh[32];
  __shared__ int is_last;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  const size_t t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  auto add = [&](const T* p, size_t n, double& acc) {
    for (size_t i = t0; i < n; i += stride) acc += (double)p[i] * (double)p[i];
  };
  if (flow) {
    add(flow, 3 * N, s[0]);
    add(flow + 3 * N, N, s[1]);
    if (nfs == 5) add(flow + 4 * N, N, s[2]);
  }
  if (tem) add(tem, N, s[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double p = block_sum(s[k], sh);
    if (threadIdx.x == 0) gm->partials[(size_t)k * OVS_RED_BLOCKS + blockIdx.x] = p;
  }
  if (threadIdx.x == 0) {
    __threadfence();
    is_last = atomicAdd(&gm->counter, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
      v += __ldcg(gm->partials + (size_t)k * OVS_RED_BLOCKS + b);
    const double t = block_sum(v, sh);
    if (threadIdx.x == 0) gm->scal[k] = t;
  }
  if (threadIdx.x == 0) gm->counter = 0;
}

int ovs_resnorm_impl(ovs_ctx* c, int prec, double r[4]) {
  // momentum/continuity/VOF from the NS+VOF system if assembled, else NS
  const int fs = c->sys[OVS_SYS_NSVOF][prec].rhs ? OVS_SYS_NSVOF : OVS_SYS_NS;
  const void *flow = c->sys[fs][prec].rhs, *tem = c->sys[OVS_SYS_TEM][prec].rhs;
  const int nfs = ovs_sys_nf(fs);
  const int grid = ovs_grid((size_t)c->N * 3, OVS_RED_THREADS, OVS_RED_BLOCKS);
  if (prec == OVS_FP64)
    resnorm_kernel<double><<<grid, OVS_RED_THREADS, 0, c->stream>>>(as<double>(flow), nfs, as<double>(tem),
                                                                    (size_t)c->N, c->gm);
  else
    resnorm_kernel<float><<<grid, OVS_RED_THREADS, 0, c->stream>>>(as<float>(flow), nfs, as<float>(tem),
                                                                   (size_t)c->N, c->gm);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  OVS_CUDA_TRY(cudaMemcpyAsync(c->h_pinned_d, c->gm->scal, sizeof(double) * 4, cudaMemcpyDeviceToHost, c->stream));
  OVS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  memcpy(r, c->h_pinned_d, sizeof(double) * 4);
  return OVS_OK;
}

int ovs_precond_setup(ovs_ctx* c, int sys, int prec) {
  SysStore& S = c->sys[sys][prec];
  if (!S.vals) return OVS_ERR_STATE;
  const size_t ts = prec == OVS_FP64 ? 8 : 4;
  const size_t w = sys == OVS_SYS_TEM ? 1 : 11;
  int st;
  if ((st = ovs_ensure(&S.binv, ts * w * (size_t)c->N))) return st;
  if (prec == OVS_FP64)
    {
      precond_setup_kernel<double><<<ovs_grid(c->N, 256, 1 << 30), 256, 0, c->stream>>>(
          c->N, sys, c->diag, as<double>(S.vals), reinterpret_cast<double*>(S.binv));
      ++c->launches;
    }
  else
    {
      precond_setup_kernel<float><<<ovs_grid(c->N, 256, 1 << 30), 256, 0, c->stream>>>(
          c->N, sys, c->diag, as<float>(S.vals), reinterpret_cast<float*>(S.binv));
      ++c->launches;
    }
  OVS_CUDA_TRY(cudaGetLastError());
  return OVS_OK;
}

// y = P^-1 x with the block-diagonal preconditioner in `pre` (the layout of
// precond_setup_kernel: 3x3 velocity inverses, then 1/M and 1/LS per node;
// one value per node for the temperature system)
template <typename TM>
__global__ void precond_apply_kernel(int N, int sys, const TM* __restrict__ pre, const double* __restrict__ x,
                                     double* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const size_t n = N;
  if (sys == OVS_SYS_TEM) { y[i] = (double)pre[i] * x[i]; return; }
  const TM* B = pre + (size_t)i * 9;
  const double x0 = x[i], x1 = x[n + i], x2 = x[2 * n + i];
  for (int g = 0; g < 3; ++g)
    y[g * n + i] = (double)B[3 * g] * x0 + (double)B[3 * g + 1] * x1 + (double)B[3 * g + 2] * x2;
  y[3 * n + i] = x[3 * n + i] * (double)pre[9 * n + i];
  if (sys == OVS_SYS_NSVOF) y[4 * n + i] = x[4 * n + i] * (double)pre[10 * n + i];
}

int ovs_precond_apply_impl(ovs_ctx* c, int sys, int prec, const double* dx, double* dy) {
  SysStore& S = c->sys[sys][prec];
  if (!S.binv) return OVS_ERR_STATE;
  if (prec == OVS_FP64)
    precond_apply_kernel<double><<<ovs_grid(c->N, 256, 1 << 30), 256, 0, c->stream>>>(c->N, sys, as<double>(S.binv), dx, dy);
  else
    precond_apply_kernel<float><<<ovs_grid(c->N, 256, 1 << 30), 256, 0, c->stream>>>(c->N, sys, as<float>(S.binv), dx, dy);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  return OVS_OK;
}

// y = P^-1 A x (dx, dy FP64 device vectors), preconditioned product
int ovs_spmv_pre_impl(ovs_ctx* c, int sys, int prec, const double* dx, double* dy) {
  SysStore& S = c->sys[sys][prec];
  if (!S.vals || !S.binv) return OVS_ERR_STATE;
  if (prec == OVS_FP64)
    return launch_spmv<double, double, double, 1>(c, sys, as<double>(S.vals), dx, dy, as<double>(S.binv), nullptr, nullptr);
  return launch_spmv<float, double, double, 1>(c, sys, as<float>(S.vals), dx, dy, as<float>(S.binv), nullptr, nullptr);
}

// the same products on a list of rows (device int array, local indices)
int ovs_spmv_rows_impl(ovs_ctx* c, int sys, int prec, bool precond, const double* dx, double* dy, const int* rows,
                       int nrows) {
  SysStore& S = c->sys[sys][prec];
  if (!S.vals || (precond && !S.binv)) return OVS_ERR_STATE;
  if (prec == OVS_FP64) {
    if (precond) return launch_spmv_rows<double, 1>(c, sys, as<double>(S.vals), dx, dy, as<double>(S.binv), rows, nrows);
    return launch_spmv_rows<double, 0>(c, sys, as<double>(S.vals), dx, dy, nullptr, rows, nrows);
  }
  if (precond) return launch_spmv_rows<float, 1>(c, sys, as<float>(S.vals), dx, dy, as<float>(S.binv), rows, nrows);
  return launch_spmv_rows<float, 0>(c, sys, as<float>(S.vals), dx, dy, nullptr, rows, nrows);
}

// y = A x (dx, dy FP64 device vectors), plain product
int ovs_spmv_impl(ovs_ctx* c, int sys, int prec, const double* dx, double* dy) {
  SysStore& S = c->sys[sys][prec];
  if (!S.vals) return OVS_ERR_STATE;
  if (prec == OVS_FP64) return launch_spmv<double, double, double, 0>(c, sys, as<double>(S.vals), dx, dy, nullptr, nullptr, nullptr);
  return launch_spmv<float, double, double, 0>(c, sys, as<float>(S.vals), dx, dy, nullptr, nullptr, nullptr);
}

// Reference-semantics single cycle in FP64 (SparseGMRES_up / _ns_conv / _tem)
int ovs_feed(ovs_ctx* c, SolFeed* f, size_t count) {
  const size_t total = f->n * f->ncol;
  const size_t end = count == 0 || count >= total - f->at ? total : f->at + count;
  while (f->at < end) {
    const size_t col = f->at / f->n, off = f->at - col * f->n;
    const size_t m = std::min(end - f->at, f->n - off);
    OVS_CUDA_TRY(cudaMemcpyAsync(f->dst + f->at, f->cols[col] + off, sizeof(double) * m, cudaMemcpyHostToDevice,
                                 c->sol_stream));
    if (f->out) {
      constexpr size_t PAGE = 4096 / sizeof(double);
      volatile double* o = f->out[col] + off;
      for (size_t i = 0; i < m; i += PAGE) o[i] = 0.0;
    }
    f->at += m;
  }
  return OVS_OK;
}

int ovs_gmres_ref_impl(ovs_ctx* c, int sys, double tol, int kspace, int kmin, double* dsol,
                       ovs_gmres_info* info, SolFeed* feed) {
  SysStore& S = c->sys[sys][OVS_FP64];
  if (!S.vals || !S.rhs) return OVS_ERR_STATE;
  int st;
  if ((st = ovs_precond_setup(c, sys, OVS_FP64))) return st;
  const double* rhs = reinterpret_cast<const double*>(S.rhs);
  if (sys == OVS_SYS_TEM) {
    // SparseGMRES_tem.f90:63-71: sol = 0 and return when ||rhs|| == 0
    double rr;
    if ((st = dot64(c, rhs, rhs, (size_t)c->N, &rr))) return st;
    if (rr == 0.0) {
      OVS_CUDA_TRY(cudaMemsetAsync(dsol, 0, sizeof(double) * c->N, c->stream));
      OVS_CUDA_TRY(cudaStreamSynchronize(c->stream));
      if (info) { memset(info, 0, sizeof(*info)); info->converged = 1; }
      return OVS_OK;
    }
  }
  st = gmres_cycle<double, double>(c, sys, rhs, dsol, tol, kspace, kmin, info, false, feed);
  if (st) return st;
  OVS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return OVS_OK;
}

// The FP32 matrix of `sys` := the FP32 rounding of its FP64 matrix (queued
// on the context stream).
int ovs_round_impl(ovs_ctx* c, int sys) {
  SysStore& S = c->sys[sys][OVS_FP64];
  if (!S.vals) return OVS_ERR_STATE;
  SysStore& S32 = c->sys[sys][OVS_FP32];
  const size_t nv = (size_t)c->nnz * ovs_sys_nv(sys);
  int st;
  if ((st = ovs_ensure(&S32.vals, sizeof(float) * nv))) return st;
  convert_kernel<double, float><<<ovs_grid(nv, 256, 16 * c->num_sms), 256, 0, c->stream>>>(
      as<double>(S.vals), reinterpret_cast<float*>(S32.vals), nv);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  S32.have_mat = true;
  return OVS_OK;
}

// y = y + a x and y = a x over n values (y FP64)
template <typename TX>
__global__ void axpy64_kernel(double* __restrict__ y, const TX* __restrict__ x, double a, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] += a * (double)x[i];
}
__global__ void scale64_kernel(double* __restrict__ y, const double* __restrict__ x, double a, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = a * x[i];
}

// OVS_MIXED with a flexible Krylov outer (FGMRES(m), Saad 1993): the outer
// iteration runs in FP64 on the FP64 system, and each of its directions is
// preconditioned by one FP32 GMRES cycle on the FP32 rounding of the matrix
// (z_j ~ A^-1 v_j), so the corrections of successive inner cycles are
// combined by a least-squares fit instead of added one after another.  The
// outer basis V (m + 1 vectors) and the preconditioned directions Z (m) are
// FP64; the outer Gram-Schmidt is modified Gram-Schmidt with FP64 dots.
// After m directions, or when the outer residual estimate reaches rtol, x
// is updated and the true residual b - A x recomputed with the FP64 matrix.
// x, r, b: FP64 device vectors (r = b - A x on entry); cycles counts inner
// cycles (max_cycles bounds them), iters inner iterations.
static int solve_flexible(ovs_ctx* c, int sys, double rtol, int kspace, int max_cycles, int m, double* x,
                          double* r, const double* b, double bnorm, int& cycles, int& iters, double& rel) {
  const size_t n = (size_t)c->N * ovs_sys_nf(sys);
  cudaStream_t s = c->stream;
  SysStore& S = c->sys[sys][OVS_FP64];
  const int gr = ovs_grid(n, 256, 8 * c->num_sms);
  // V (m + 1 FP64 vectors) and Z (m FP32 vectors: a direction rounded to
  // FP32 before its product is taken is as good a direction, and A z_j is
  // formed from the rounded z_j), kept by the context between solves
  const size_t need = sizeof(double) * n * ((size_t)m + 1) + sizeof(float) * n * (size_t)m;
  if (c->fg_bytes < need) {
    if (c->fg_buf) cudaFree(c->fg_buf);
    c->fg_buf = nullptr;
    c->fg_bytes = 0;
    if (cudaMalloc(&c->fg_buf, need) != cudaSuccess) {
      cudaGetLastError();
      c->fg_buf = nullptr;
      return OVS_ERR_NOMEM;
    }
    c->fg_bytes = need;
  }
  double* V = reinterpret_cast<double*>(c->fg_buf);
  float* Z = reinterpret_cast<float*>(V + n * ((size_t)m + 1));
  double* zw = r;   // the inner cycle's FP64 correction, in the residual's storage until the update
  std::vector<double> H((size_t)(m + 1) * m), g(m + 1), cs(m), sn(m), y(m);
  int st = OVS_OK;
  if ((st = ovs_precond_setup(c, sys, OVS_FP64))) return st;
  while (rel > rtol && cycles < max_cycles) {
    // the outer iteration minimizes the preconditioned residual P^-1 (b - A x)
    // (the block-Jacobi scaling balances the fields, whose raw residuals
    // differ by orders of magnitude); v_1 = P^-1 r / |P^-1 r|
    if ((st = ovs_precond_apply_impl(c, sys, OVS_FP64, r, V))) break;
    double vv;
    if ((st = dot64(c, V, V, n, &vv))) break;
    const double beta = sqrt(vv);
    if (!(beta > 0.0)) break;
    scale64_kernel<<<gr, 256, 0, s>>>(V, V, 1.0 / beta, n);
    ++c->launches;
    const double target = 0.5 * beta * rtol / rel;   // the reduction the true residual still needs
    std::fill(H.begin(), H.end(), 0.0);
    std::fill(g.begin(), g.end(), 0.0);
    g[0] = beta;
    int j = 0;
    bool stop = false;
    for (; j < m && !stop && cycles < max_cycles; ++j) {
      double* vj = V + n * (size_t)j;
      float* zj = Z + n * (size_t)j;
      double* w = V + n * (size_t)(j + 1);
      OVS_CUDA_TRY(cudaMemsetAsync(zw, 0, sizeof(double) * n, s));
      double tin = target / fabs(g[j]);
      if (tin < 1e-6) tin = 1e-6;
      if (tin > 0.5) tin = 0.5;
      ovs_gmres_info gi;
      if ((st = gmres_cycle<float, float, false>(c, sys, vj, zw, tin, kspace, 1, &gi, true))) break;
      iters += gi.iterations;
      ++cycles;
      convert_kernel<double, float><<<gr, 256, 0, s>>>(zw, zj, n);
      ++c->launches;
      if ((st = launch_spmv<double, float, double, 1>(c, sys, as<double>(S.vals), zj, w, as<double>(S.binv),
                                                        nullptr, nullptr)))
        break;
      for (int i = 0; i <= j; ++i) {
        double h;
        if ((st = dot64(c, w, V + n * (size_t)i, n, &h))) break;
        H[(size_t)j * (m + 1) + i] = h;
        axpy64_kernel<<<gr, 256, 0, s>>>(w, V + n * (size_t)i, -h, n);
        ++c->launches;
      }
      if (st) break;
      double ww;
      if ((st = dot64(c, w, w, n, &ww))) break;
      const double hn = sqrt(ww);
      H[(size_t)j * (m + 1) + j + 1] = hn;
      if (hn > 0.0) {
        scale64_kernel<<<gr, 256, 0, s>>>(w, w, 1.0 / hn, n);
        ++c->launches;
      }
      // Givens rotations of column j
      double* hc = &H[(size_t)j * (m + 1)];
      for (int i = 0; i < j; ++i) {
        const double t = cs[i] * hc[i] + sn[i] * hc[i + 1];
        hc[i + 1] = -sn[i] * hc[i] + cs[i] * hc[i + 1];
        hc[i] = t;
      }
      const double den = sqrt(hc[j] * hc[j] + hc[j + 1] * hc[j + 1]);
      if (den == 0.0) { stop = true; break; }   // a zero column: the directions so far span the solution
      cs[j] = hc[j] / den;
      sn[j] = hc[j + 1] / den;
      hc[j] = den;
      hc[j + 1] = 0.0;
      g[j + 1] = -sn[j] * g[j];
      g[j] = cs[j] * g[j];
      if (!(hn > 0.0) || fabs(g[j + 1]) <= target) stop = true;
    }
    if (st) break;
    // x += Z y with H y = g (upper triangular, j x j)
    for (int i = j - 1; i >= 0; --i) {
      double t = g[i];
      for (int k = i + 1; k < j; ++k) t -= H[(size_t)k * (m + 1) + i] * y[k];
      y[i] = H[(size_t)i * (m + 1) + i] != 0.0 ? t / H[(size_t)i * (m + 1) + i] : 0.0;
    }
    for (int i = 0; i < j; ++i) {
      axpy64_kernel<<<gr, 256, 0, s>>>(x, Z + n * (size_t)i, y[i], n);
      ++c->launches;
    }
    // (zw, the residual's storage, is rewritten with the true residual next)
    // the true residual with the FP64 matrix
    if ((st = launch_spmv<double, double, double, 2>(c, sys, as<double>(S.vals), x, r, nullptr, b, nullptr))) break;
    double rr;
    if ((st = dot64(c, r, r, n, &rr))) break;
    rel = sqrt(rr) / bnorm;
    if (!(rel == rel) || j == 0) break;
  }
  OVS_CUDA_TRY(cudaGetLastError());
  return st;
}

// Restarted / iteratively refined solve to a true FP64 relative residual.
// `outer` is the system whose residual b - A x is driven to rtol (matrix and
// right-hand side of that precision, FP64 arithmetic), `inner` the matrix
// precision of the GMRES cycles that compute the corrections:
//   OVS_FP64  outer FP64, inner FP64 (restarted GMRES);
//   OVS_MIXED outer FP64, inner FP32 = the rounding of the FP64 matrix;
//   OVS_FP32  outer FP32, inner FP32 (the FP32-assembled system).
int ovs_solve_impl(ovs_ctx* c, int sys, int mode, double rtol, int kspace, int max_cycles,
                   ovs_solve_info* info) {
  const int outer = mode == OVS_FP32 ? OVS_FP32 : OVS_FP64;
  const int prec = mode == OVS_FP64 ? OVS_FP64 : OVS_FP32;   // inner
  SysStore& S = c->sys[sys][outer];
  if (!S.vals || !S.rhs) return OVS_ERR_STATE;
  const int N = c->N, nf = ovs_sys_nf(sys);
  const size_t n = (size_t)N * nf;
  int st;
  cudaStream_t s = c->stream;
  if ((st = ovs_ensure((void**)&c->sol[sys], sizeof(double) * 5 * (size_t)N))) return st;
  if ((st = ovs_ensure((void**)&c->work64, sizeof(double) * 10 * (size_t)N))) return st;
  double* x = c->sol[sys];
  double* b = c->work64;
  double* r = c->work64 + 5 * (size_t)N;
  OVS_CUDA_TRY(cudaEventRecord(c->ev0, s));
  // the inner operator of OVS_MIXED: FP32 rounding of the FP64 matrix values
  if (mode == OVS_MIXED && (st = ovs_round_impl(c, sys))) return st;
  if ((st = ovs_precond_setup(c, sys, prec))) return st;
  if (outer == OVS_FP64) {
    OVS_CUDA_TRY(cudaMemcpyAsync(b, S.rhs, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  } else {
    convert_kernel<float, double><<<ovs_grid(n, 256, 4096), 256, 0, s>>>(as<float>(S.rhs), b, n);
    ++c->launches;
  }
  OVS_CUDA_TRY(cudaMemsetAsync(x, 0, sizeof(double) * n, s));
  OVS_CUDA_TRY(cudaMemcpyAsync(r, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  double bb;
  if ((st = dot64(c, b, b, n, &bb))) return st;
  const double bnorm = sqrt(bb);
  double rel = bnorm > 0.0 ? 1.0 : 0.0;
  int cycles = 0, iters = 0;
  const double floor_tol = prec == OVS_FP32 ? 1e-6 : 1e-14;
  if (mode == OVS_MIXED && c->mixed_outer > 0 && rel > rtol) {
    if ((st = solve_flexible(c, sys, rtol, kspace, max_cycles, c->mixed_outer, x, r, b, bnorm, cycles, iters, rel)))
      return st;
  }
  while (rel > rtol && cycles < max_cycles) {
    double tin = rtol / rel;
    if (tin < floor_tol) tin = floor_tol;
    if (tin > 0.5) tin = 0.5;
    ovs_gmres_info gi;
    if (prec == OVS_FP64) st = gmres_cycle<double, double, true>(c, sys, r, x, tin, kspace, 1, &gi);
    else st = gmres_cycle<float, float, false>(c, sys, r, x, tin, kspace, 1, &gi);
    if (st) return st;
    iters += gi.iterations;
    ++cycles;
    // r = b - A x in FP64 arithmetic, with the outer system's matrix
    if (outer == OVS_FP64) st = launch_spmv<double, double, double, 2>(c, sys, as<double>(S.vals), x, r, nullptr, b, nullptr);
    else st = launch_spmv<float, double, double, 2>(c, sys, as<float>(S.vals), x, r, nullptr, b, nullptr);
    if (st) return st;
    double rr;
    if ((st = dot64(c, r, r, n, &rr))) return st;
    rel = sqrt(rr) / bnorm;
    if (!(rel == rel)) break;
    if (gi.iterations == 0) break;
  }
  OVS_CUDA_TRY(cudaEventRecord(c->ev1, s));
  OVS_CUDA_TRY(cudaEventSynchronize(c->ev1));
  float ms = 0.f;
  OVS_CUDA_TRY(cudaEventElapsedTime(&ms, c->ev0, c->ev1));
  if (info) {
    info->cycles = cycles;
    info->iterations = iters;
    info->converged = rel <= rtol;
    info->rel_residual = rel;
    info->seconds = ms * 1e-3;
  }
  return OVS_OK;
}

// ------------------------------------------------------ transposed solve
// Slot of (j, i) for every slot (i, j): the pattern of a finite-element
// matrix is symmetric, so row j holds column i; a missing entry flags an
// error instead.
__global__ void transpose_map_kernel(int N, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                                     int* __restrict__ tmap, int* __restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
    const int j = colidx[k];
    int lo = rowptr[j], hi = rowptr[j + 1];
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (colidx[mid] > i) hi = mid; else lo = mid;
    }
    if (colidx[lo] != i) { atomicOr(err, 1); tmap[k] = k; }
    else tmap[k] = lo;
  }
}

__global__ void gather_vals_kernel(const double* __restrict__ v, const int* __restrict__ tmap,
                                   double* __restrict__ vt, size_t nnz) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nnz; k += (size_t)gridDim.x * blockDim.x)
    vt[k] = v[tmap[k]];
}

// A^T x = rhs for the scalar temperature system: the transposed values
// stand in for the system's values during one reference-semantics cycle;
// the diagonal, and so the Jacobi preconditioner, is the same.
int ovs_gmres_transposed_impl(ovs_ctx* c, int sys, const double* drhs, double tol, int kspace, int kmin,
                              double* dsol, ovs_gmres_info* info) {
  if (sys != OVS_SYS_TEM) return OVS_ERR_ARG;
  SysStore& S = c->sys[sys][OVS_FP64];
  if (!S.vals) return OVS_ERR_STATE;
  int st;
  cudaStream_t s = c->stream;
  const size_t nnz = c->nnz;
  if (!c->tmap) {
    if ((st = ovs_ensure((void**)&c->tmap, sizeof(int) * (nnz > 0 ? nnz : 1)))) return st;
    OVS_CUDA_TRY(cudaMemsetAsync(c->flags, 0, sizeof(int) * 4, s));
    transpose_map_kernel<<<ovs_grid(c->N, 128, 1 << 30), 128, 0, s>>>(c->N, c->rowptr, c->colidx, c->tmap,
                                                                      c->flags + 2);
    ++c->launches;
    int herr = 0;
    OVS_CUDA_TRY(cudaMemcpyAsync(&herr, c->flags + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    OVS_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr) { cudaFree(c->tmap); c->tmap = nullptr; return OVS_ERR_PATTERN; }
  }
  if ((st = ovs_ensure(&c->vals_t, sizeof(double) * (nnz > 0 ? nnz : 1)))) return st;
  gather_vals_kernel<<<4 * c->num_sms, 256, 0, s>>>(reinterpret_cast<const double*>(S.vals), c->tmap,
                                                    reinterpret_cast<double*>(c->vals_t), nnz);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  if ((st = ovs_precond_setup(c, sys, OVS_FP64))) return st;
  double rr;
  if ((st = dot64(c, drhs, drhs, (size_t)c->N, &rr))) return st;
  if (rr == 0.0) {   // SparseGMRES_tem.f90:63-71
    OVS_CUDA_TRY(cudaMemsetAsync(dsol, 0, sizeof(double) * c->N, s));
    OVS_CUDA_TRY(cudaStreamSynchronize(s));
    if (info) { memset(info, 0, sizeof(*info)); info->converged = 1; }
    return OVS_OK;
  }
  void* saved = S.vals;
  S.vals = c->vals_t;
  st = gmres_cycle<double, double>(c, sys, drhs, dsol, tol, kspace, kmin, info);
  S.vals = saved;
  if (st) return st;
  OVS_CUDA_TRY(cudaStreamSynchronize(s));
  return OVS_OK;
}
