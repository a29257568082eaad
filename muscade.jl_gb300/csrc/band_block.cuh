// Banded LU with partial pivoting for bands of up to 256, one thread-block
// cluster per component (3D frames of a few storeys: hundreds to thousands of
// dofs, bands of 50 to 250).
//
// What bounds it: n kl (kl+ku) FP64 multiply-adds on one component, of which a
// single SM does two a clock (a 6 x 5 x 4 frame, 900 dofs of band 143, is 9 ms of
// one SM's FP64 pipe), and the chain of n pivot steps.  So the columns go by
// panels of 16: the first block of the cluster factorises the panel in shared
// memory (a thread per row), the cluster's blocks then share out the trailing
// columns, a warp per column with its rows in registers, and one cluster barrier
// stands on either side.  Multipliers, interchanges and updates are those of
// LAPACK gbtf2, each entry updated in the order of the pivots, so the factors are
// bitwise those of the row-band kernels (band_rows.cuh).  Measured on that frame:
// 1.93 ms a factorisation, most of it the panels' pivot steps (two block barriers,
// the reciprocal, up to 15 multiply-adds for a warp's rows each); 64 ms with one
// block working on the band in global memory.
//
// Storage: LAPACK's, A(i, j) at base[kv + i − j + ld j], ld = 2kl + ku + 1.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "band_rows.cuh"

namespace mgpu {

constexpr int kBlkNB = 16;        // columns of a panel
constexpr int kBlkMaxBand = 256;  // widest kl or ku
constexpr int kBlkRows = kBlkNB + kBlkMaxBand;
constexpr int kBlkThreads = 288;  // one thread per row of a panel
constexpr int kBlkWarps = kBlkThreads / 32;
constexpr int kBlkSlots = kBlkThreads / 32;  // rows of a trailing column per lane
static_assert(kBlkRows <= kBlkThreads, "a thread per row");

__global__ void band_gather(int64_t nnz, const int64_t* __restrict__ bmap, const double* __restrict__ nzval,
                            double* __restrict__ AB) {
  const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < nnz) AB[bmap[k]] = nzval[k];
}

// grid: cl blocks per component, launched as clusters of cl
__global__ void __launch_bounds__(kBlkThreads) band_lu(const int64_t* cbase, const int32_t* cn, const int32_t* ckl,
                                                       const int32_t* cku, const int32_t* cdof0, double* AB,
                                                       int32_t* ipiv, double* rdg, int* info, int cl) {
  __shared__ double S[kBlkRows * kBlkNB];  // the panel: row r, column c at r + kBlkRows c
  __shared__ unsigned whi[kBlkWarps], wlo[kBlkWarps], wix[kBlkWarps];
  __shared__ double s_rp[2], prow[2][kBlkNB], crow[kBlkNB];  // 1/pivot, the pivot's row, the row that it replaces
  __shared__ int sjp[kBlkNB];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int cc = blockIdx.x / cl, rank = blockIdx.x % cl;
  const int n = cn[cc], kl = ckl[cc], ku = cku[cc], kv = kl + ku, ld = 2 * kl + ku + 1;
  double* A = AB + cbase[cc];
  int32_t* piv = ipiv + cdof0[cc];
  double* rdiag = rdg + cdof0[cc];  // reciprocal pivots for the backward substitution
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto sync = [&] {
    if (cl > 1)
      cluster.sync();
    else
      __syncthreads();
  };
  int ju = 0;  // last column an interchange or the band has reached
  for (int k0 = 0; k0 < n; k0 += kBlkNB) {
    const int nb = min(kBlkNB, n - k0), rows = min(nb + kl, n - k0);
    if (rank == 0) {
      // the panel, row `tid` in registers
      double a[kBlkNB];
#pragma unroll
      for (int c = 0; c < kBlkNB; ++c) {
        const int q = kv + tid - c;
        a[c] = (c < nb && tid < rows && q >= 0 && q < ld) ? A[q + int64_t(ld) * (k0 + c)] : 0.0;
      }
#pragma unroll
      for (int c = 0; c < kBlkNB; ++c) {
        if (c >= nb) break;
        const int km = min(kl, n - 1 - (k0 + c)), par = c & 1;
        // pivot: the first row of the largest |a|; a NaN only where there is nothing else
        unsigned hi = 0u, lo = 0u;
        const bool in = tid >= c && tid <= c + km;
        if (in) {
          const unsigned long long v = static_cast<unsigned long long>(__double_as_longlong(a[c])) & 0x7fffffffffffffffull;
          if (v <= 0x7ff0000000000000ull) {
            hi = static_cast<unsigned>(v >> 32) + 2u;
            lo = static_cast<unsigned>(v);
          } else {
            hi = 1u;
          }
        }
        const unsigned mh = __reduce_max_sync(RB_FULL, hi);
        const unsigned ml = __reduce_max_sync(RB_FULL, hi == mh ? lo : 0u);
        const unsigned mi = __reduce_min_sync(RB_FULL, in && hi == mh && lo == ml ? unsigned(tid) : 0xffffffffu);
        if (lane == 0) {
          whi[warp] = mh;
          wlo[warp] = ml;
          wix[warp] = mi;
        }
        __syncthreads();
        const unsigned h2 = lane < kBlkWarps ? whi[lane] : 0u, l2 = lane < kBlkWarps ? wlo[lane] : 0u,
                       i2 = lane < kBlkWarps ? wix[lane] : 0xffffffffu;
        const unsigned fh = __reduce_max_sync(RB_FULL, h2);
        const unsigned fl = __reduce_max_sync(RB_FULL, h2 == fh ? l2 : 0u);
        const int pr = int(__reduce_min_sync(RB_FULL, h2 == fh && l2 == fl ? i2 : 0xffffffffu));
        if (tid == pr) {
          const double p = a[c], rp = p != 0.0 ? __drcp_rn(p) : 0.0;
          s_rp[par] = rp;
#pragma unroll
          for (int j = c + 1; j < kBlkNB; ++j) prow[par][j] = a[j];
          prow[par][c] = p;
          sjp[c] = pr - c;
          piv[k0 + c] = k0 + pr;
          rdiag[k0 + c] = p != 0.0 ? rp : 1.0 / p;
          if (p == 0.0 && *info == 0) atomicCAS(info, 0, cc + 1);
        }
        if (pr != c && tid == c)
#pragma unroll
          for (int j = c; j < kBlkNB; ++j) crow[j] = a[j];
        __syncthreads();
        if (pr != c) {  // interchange within the panel; the multipliers to the left stay
          if (tid == pr)
#pragma unroll
            for (int j = c; j < kBlkNB; ++j) a[j] = crow[j];
          if (tid == c)
#pragma unroll
            for (int j = c; j < kBlkNB; ++j) a[j] = prow[par][j];
        }
        if (tid > c && tid <= c + km) {
          const double l = a[c] * s_rp[par];
          a[c] = l;
#pragma unroll
          for (int j = c + 1; j < kBlkNB; ++j) a[j] = fma(-l, prow[par][j], a[j]);
        }
      }
#pragma unroll
      for (int c = 0; c < kBlkNB; ++c) {
        const int q = kv + tid - c;
        if (tid < kBlkRows) S[tid + kBlkRows * c] = a[c];
        if (c < nb && tid < rows && q >= 0 && q < ld) A[q + int64_t(ld) * (k0 + c)] = a[c];
      }
    }
    sync();
    if (rank != 0) {
      double l[kBlkNB];  // all in flight at once
#pragma unroll
      for (int c = 0; c < kBlkNB; ++c) {
        const int q = kv + tid - c;
        l[c] = (c < nb && tid < rows && q >= 0 && q < ld) ? A[q + int64_t(ld) * (k0 + c)] : 0.0;
      }
#pragma unroll
      for (int c = 0; c < kBlkNB; ++c)
        if (tid < kBlkRows) S[tid + kBlkRows * c] = l[c];
      if (tid < nb) sjp[tid] = piv[k0 + tid] - (k0 + tid);
      __syncthreads();
    }
    for (int c = 0; c < nb; ++c) ju = max(ju, min(k0 + c + ku + sjp[c], n - 1));
    // trailing columns: rows k0 .. k0 + rows − 1 of column j, row r on lane r mod 32
    for (int j = k0 + nb + rank * kBlkWarps + warp; j <= ju; j += cl * kBlkWarps) {
      double* a = A + kv + k0 - j + int64_t(ld) * j;  // row r at a[r]
      const int r0 = j - k0 - kv;                     // first row within the band
      double v[kBlkSlots];
#pragma unroll
      for (int s = 0; s < kBlkSlots; ++s) {
        const int r = lane + 32 * s;
        v[s] = (r < rows && r >= r0) ? a[r] : 0.0;
      }
      for (int p = 0; p < nb; ++p) {
        const int jp = sjp[p];
        if (jp) {  // rows p and p + jp
          const int r = p + jp, sl = r >> 5;
          double x = 0.0;
#pragma unroll
          for (int s = 0; s < kBlkSlots; ++s)
            if (s == sl) x = v[s];
          const double vp = __shfl_sync(RB_FULL, v[0], p), vr = __shfl_sync(RB_FULL, x, r & 31);
          if (lane == p) v[0] = vr;
#pragma unroll
          for (int s = 0; s < kBlkSlots; ++s)
            if (s == sl && lane == (r & 31)) v[s] = vp;
        }
        const double u = __shfl_sync(RB_FULL, v[0], p);
        const double* L = S + kBlkRows * p;  // zero beyond row p + kl
        if (lane > p) v[0] = fma(-L[lane], u, v[0]);
#pragma unroll
        for (int s = 1; s < kBlkSlots; ++s) {
          if (32 * s >= rows) break;
          if (lane + 32 * s < kBlkRows) v[s] = fma(-L[lane + 32 * s], u, v[s]);
        }
      }
#pragma unroll
      for (int s = 0; s < kBlkSlots; ++s) {
        const int r = lane + 32 * s;
        if (r < rows && r >= r0) a[r] = v[s];
      }
    }
    sync();
  }
}

// Solve with the factors, one block per component: permute, L with interchanges, U.
// Bound by the chain of 2n steps, so everything on it is on chip: the vector's
// window in registers (a thread per row; two backward), the factor's columns by
// chunks of 16 in shared memory, the next chunk on its way (cp.async).  One warp
// takes a chunk's triangle, the other rows follow behind a single barrier; a chunk
// with interchanges goes step by step.  (A step in global memory with two block
// barriers: 1.54 ms for 900 dofs; step by step as here: 0.68 ms.)
constexpr int kBlkBack = kBlkNB + 2 * kBlkMaxBand;  // rows a backward chunk touches
static_assert(kBlkBack <= 2 * kBlkThreads, "two rows per thread");
inline size_t band_solve_smem(int maxkl, int maxkv) {
  return 2 * size_t(kBlkNB) * (kBlkNB + (maxkv > maxkl ? maxkv : maxkl)) * sizeof(double);
}

__global__ void __launch_bounds__(kBlkThreads) band_solve(const int64_t* cbase, const int32_t* cn, const int32_t* ckl,
                                                          const int32_t* cku, const int32_t* cdof0,
                                                          const int32_t* perm, const double* AB, const int32_t* ipiv,
                                                          const double* rdg, const double* Ll, double* rhs,
                                                          double* dx) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double wb[2 * kBlkThreads], sb[2], sx[2], sbv[kBlkNB], srd[2][kBlkNB];
  __shared__ int spv[kBlkNB];
  const int cc = blockIdx.x;
  const int n = cn[cc], kl = ckl[cc], kv = kl + cku[cc], ld = kv + kl + 1;
  const double* A = AB + cbase[cc];
  const int32_t *piv = ipiv + cdof0[cc], *pm = perm + cdof0[cc];
  const double* rd = rdg + cdof0[cc];
  double* b = rhs + cdof0[cc];
  const int tid = threadIdx.x;
  // ---- forward: L y = P b; thread r holds row k0 + r
  const int lf = kBlkNB + kl;  // rows of a chunk
  auto lchunk = [&](int k0, int buf) {
    double* d = sm + size_t(buf) * kBlkNB * lf;
    for (int c = 0; c < kBlkNB && k0 + c < n; ++c)
      if (tid > c && tid <= c + kl && k0 + tid < n) rb_cp_async(d + tid + lf * c, A + kv + tid - c + int64_t(ld) * (k0 + c), 8);
  };
  lchunk(0, 0);
  rb_cp_commit();
  double y = tid < min(lf, n) ? Ll[pm[tid]] : 0.0;
  for (int k0 = 0, buf = 0; k0 < n; k0 += kBlkNB, buf ^= 1) {
    const int nb = min(kBlkNB, n - k0);
    if (k0 + kBlkNB < n) lchunk(k0 + kBlkNB, buf ^ 1);
    rb_cp_commit();
    if (tid < nb) spv[tid] = piv[k0 + tid] - (k0 + tid);
    // the rows that enter the window with the next chunk
    const int kn = k0 + kBlkNB + tid;
    const bool enter = tid >= kl && tid < lf && kn < n;
    const double fresh = enter ? Ll[pm[kn]] : 0.0;
    rb_cp_wait<1>();
    __syncthreads();
    const double* L = sm + size_t(buf) * kBlkNB * lf;
    const bool swaps = __syncthreads_or(tid < nb && spv[tid] != 0);
    if (!swaps) {  // the chunk's triangle by the first warp, then every other row on its own
      if (tid < 32) {
        double l[kBlkNB];
#pragma unroll
        for (int p = 0; p < kBlkNB; ++p)
          l[p] = (p < nb && tid > p && tid <= p + kl && k0 + tid < n) ? L[tid + lf * p] : 0.0;
#pragma unroll
        for (int p = 0; p < kBlkNB; ++p) {
          if (p >= nb) break;
          y = fma(-l[p], __shfl_sync(RB_FULL, y, p), y);
        }
        if (tid < nb) sbv[tid] = y;
      }
      __syncthreads();
      if (tid >= 32)
#pragma unroll
        for (int p = 0; p < kBlkNB; ++p)
          if (p < nb && tid <= p + kl && k0 + tid < n) y = fma(-L[tid + lf * p], sbv[p], y);
    } else {
      for (int p = 0; p < nb; ++p) {
        const int jp = spv[p];
        if (jp) {
          if (tid == p) sx[0] = y;
          if (tid == p + jp) sx[1] = y;
          __syncthreads();
          if (tid == p) y = sx[1];
          if (tid == p + jp) y = sx[0];
        }
        if (tid == p) sb[p & 1] = y;
        __syncthreads();
        if (tid > p && tid <= p + kl && k0 + tid < n) y = fma(-L[tid + lf * p], sb[p & 1], y);
      }
    }
    wb[tid] = y;
    if (tid < nb) b[k0 + tid] = y;
    __syncthreads();
    y = enter ? fresh : (tid + kBlkNB < lf ? wb[tid + kBlkNB] : 0.0);
  }
  rb_cp_wait<0>();
  __syncthreads();
  // ---- backward: U x = y; thread t holds rows w − t and w − t − kBlkThreads, w the
  // last row of the chunk
  const int lb = kBlkNB + kv;
  auto uchunk = [&](int w, int buf) {
    double* d = sm + size_t(buf) * kBlkNB * lb;
    for (int c = 0; c < kBlkNB && w - c >= 0; ++c)
      for (int i = tid; i <= c + kv && i <= w; i += kBlkThreads)
        if (i > c) rb_cp_async(d + i + lb * c, A + kv - (i - c) + int64_t(ld) * (w - c), 8);
  };
  uchunk(n - 1, 0);
  rb_cp_commit();
  const int i2 = tid + kBlkThreads;
  double z0 = (tid < lb && tid <= n - 1) ? b[n - 1 - tid] : 0.0, z1 = (i2 < lb && i2 <= n - 1) ? b[n - 1 - i2] : 0.0;
  for (int w = n - 1, buf = 0; w >= 0; w -= kBlkNB, buf ^= 1) {
    const int nb = min(kBlkNB, w + 1);
    if (w - kBlkNB >= 0) uchunk(w - kBlkNB, buf ^ 1);
    rb_cp_commit();
    if (tid < nb) srd[buf][tid] = rd[w - tid];
    const int wn = w - kBlkNB;  // the next chunk's last row; rows wn − kv and on enter with it
    const bool e0 = tid >= kv && tid < lb && wn - tid >= 0, e1 = i2 >= kv && i2 < lb && wn - i2 >= 0;
    const double f0 = e0 ? b[wn - tid] : 0.0, f1 = e1 ? b[wn - i2] : 0.0;
    rb_cp_wait<1>();
    __syncthreads();
    const double* U = sm + size_t(buf) * kBlkNB * lb;
    if (tid < 32) {
      double u[kBlkNB];
      const double rdl = tid < nb ? srd[buf][tid] : 0.0;
#pragma unroll
      for (int p = 0; p < kBlkNB; ++p) u[p] = (p < nb && tid > p && tid <= p + kv && tid <= w) ? U[tid + lb * p] : 0.0;
#pragma unroll
      for (int p = 0; p < kBlkNB; ++p) {
        if (p >= nb) break;
        const double x = __shfl_sync(RB_FULL, z0 * rdl, p);
        z0 = tid == p ? x : fma(-u[p], x, z0);
      }
      if (tid < nb) sbv[tid] = z0;
    }
    __syncthreads();
    if (tid >= 32) {
#pragma unroll
      for (int p = 0; p < kBlkNB; ++p)
        if (p < nb && tid <= p + kv && tid <= w) z0 = fma(-U[tid + lb * p], sbv[p], z0);
    }
#pragma unroll
    for (int p = 0; p < kBlkNB; ++p)
      if (p < nb && i2 <= p + kv && i2 <= w) z1 = fma(-U[i2 + lb * p], sbv[p], z1);
    wb[tid] = z0;
    wb[i2] = z1;
    if (tid < nb) dx[pm[w - tid]] = z0;
    __syncthreads();
    z0 = e0 ? f0 : (tid + kBlkNB < lb ? wb[tid + kBlkNB] : 0.0);
    z1 = e1 ? f1 : (i2 + kBlkNB < lb ? wb[i2 + kBlkNB] : 0.0);
  }
  rb_cp_wait<0>();
}

}  // namespace mgpu
