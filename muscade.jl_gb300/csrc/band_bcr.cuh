// Block cyclic reduction of the separators' Schur complement (band_torn.cuh).
//
// Per component the Schur complement is block tridiagonal with N = P-1 blocks
// of s x s:  L_k x_{k-1} + D_k x_k + U_k x_{k+1} = r_k  (L_0 = U_{N-1} = 0).
// Level l (stride h = 2^l) eliminates the active blocks k with (k/h) odd:
//     W_L(k) = D_k^-1 L_k,  W_U(k) = D_k^-1 U_k   (LU of D_k, partial pivoting)
// and the kept blocks e (k/h even) take
//     D_e' = D_e - U_e W_L(e+h) - L_e W_U(e-h),
//     U_e' = -U_e W_U(e+h),   L_e' = -L_e W_L(e-h)
// until block 0 alone remains.  A solve reduces the right-hand side the same
// way (z_k = D_k^-1 r_k, r_e -= U_e z_{e+h} + L_e z_{e-h}), solves block 0 and
// substitutes back level by level (x_k = z_k - W_L(k) x_{k-h} - W_U(k) x_{k+h}).
// The factorisation runs one launch per level over all blocks of all
// components (one warp per block, dense s x s work), so the separators cost
// log2(N) levels instead of a sequential band factorisation of N s rows.  A
// solve either does the same, level by level, or (components of few
// interiors) runs inside the fused per-component solve of band_torn.cuh, one
// block barrier per level.
//
// Storage (per separator k, global index; component offset sep0, local index
// k - sep0; SS = 16 x 16 doubles per block whatever s):
//   DLU[lvl][k] D, L, U of level lvl     FA[k]: LU factors of D at elimination (bcr_factor), PV[k]: the row at each pivoted place
//   WL[k], WU[k]: D^-1 L and D^-1 U      rhs / z / x: vectors of N s entries per component
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "band_rows.cuh"

namespace mgpu {

constexpr int BCR_S = 16;                 // largest block
constexpr int BCR_SS = BCR_S * BCR_S;     // doubles per stored block

struct BcrSep {
  int32_t comp;     // component
  int32_t kloc;     // local block index 0..N-1
  int32_t N;        // blocks of its component
  int32_t s;        // block size
  int32_t sep0;     // global index of block 0 of its component
  int32_t nlev;     // levels of its component: ceil(log2 N)
};

// role of block kloc at level l: 0 inactive, 1 eliminated, 2 kept
__device__ __forceinline__ int bcr_role(int kloc, int N, int l) {
  const int h = 1 << l;
  if (kloc % h != 0 || kloc >= N) return 0;
  return ((kloc / h) & 1) ? 1 : 2;
}

// 1/pivot in the factors' type
__device__ __forceinline__ double bcr_rcp(double p) { return __drcp_rn(p); }
__device__ __forceinline__ float bcr_rcp(float p) { return __frcp_rn(p); }

// The dense work of one block, one warp, a matrix row per lane in registers:
// what bounds it is the chain of s pivots and, in FP64, the instructions issued
// (64 cycles each), so every step is one multiply-add per remaining column for all
// rows at once and nothing goes through memory.  One chain of 490 separators, a level
// (FP64): bcr_eliminate 58 -> 25 us (L and U sides on a warp each; blocks of 13 and
// then 11), bcr_update 21 -> 6, bcr_fwd_elim 12.6 -> 3.2, against blocks in shared
// memory, row by row, with divisions on the chain.
//
// LU with partial pivoting of d (ties to the first row), x <- d^-1 x for s columns.
// Rows stay on their lanes: *pos is the place of the lane's row in the pivoted
// order.  On return the row holds L left of the diagonal, 1/pivot on it and
// U(i, j)/U(j, j) right of it.  Returns whether a pivot was zero.
template <typename T, bool RHS>
__device__ __forceinline__ bool bcr_factor(T d[BCR_S], T x[BCR_S], int s, int lane, int* pos_out) {
  int pos = lane < s ? lane : (1 << 30);
  T rpo = T(0);
  bool singular = false;
#pragma unroll
  for (int j = 0; j < BCR_S; ++j) {
    if (j >= s) break;
    int pl;
    const int jp = rb_argmax(d[j], pos >= j && pos < s, pos, &pl);
    const T p = __shfl_sync(RB_FULL, d[j], pl);
    if (lane == pl)
      pos = j;
    else if (pos == j)
      pos = jp;
    const bool zero = p == T(0);
    singular = singular || zero;
    const T rp = zero ? T(0) : bcr_rcp(p);
    if (lane == pl) rpo = rp;
    T l = T(0);
    if (pos > j && pos < s && !zero) l = d[j] = d[j] * rp;
#pragma unroll
    for (int c = j + 1; c < BCR_S; ++c) {
      if (c >= s) break;
      d[c] = fma(-l, __shfl_sync(RB_FULL, d[c], pl), d[c]);
    }
    if constexpr (RHS)
#pragma unroll
      for (int c = 0; c < BCR_S; ++c) {
        if (c >= s) break;
        x[c] = fma(-l, __shfl_sync(RB_FULL, x[c], pl), x[c]);
      }
  }
#pragma unroll
  for (int j = BCR_S - 1; j >= 0; --j) {
    if (j >= s) continue;
    const int pl = __ffs(__ballot_sync(RB_FULL, pos == j)) - 1;
    const T rp = __shfl_sync(RB_FULL, rpo, pl);
    T e = T(0);
    if (pos < j) e = d[j] = d[j] * rp;
    if (pos == j) d[j] = rpo;
    if constexpr (RHS)
#pragma unroll
      for (int c = 0; c < BCR_S; ++c) {
        if (c >= s) break;
        x[c] = fma(-e, __shfl_sync(RB_FULL, x[c], pl), x[c]);
      }
  }
  if constexpr (RHS)
#pragma unroll
    for (int c = 0; c < BCR_S; ++c) x[c] *= rpo;
  *pos_out = pos;
  return singular;
}
template <typename T>
__device__ __forceinline__ void bcr_row_load(T v[BCR_S], const T* M, int s, int row) {
#pragma unroll
  for (int c = 0; c < BCR_S; ++c) v[c] = (row < s && c < s) ? M[row * BCR_S + c] : T(0);
}
template <typename T>
__device__ __forceinline__ void bcr_row_store(const T v[BCR_S], T* M, int s, int row) {
  if (row < s)
#pragma unroll
    for (int c = 0; c < BCR_S; ++c)
      if (c < s) M[row * BCR_S + c] = v[c];
}

// level l, eliminated blocks: factor D_k, W_L = D^-1 L (first warp), W_U = D^-1 U (second)
template <typename T>
__global__ void __launch_bounds__(64) bcr_eliminate(int nsep, const BcrSep* __restrict__ bs, int l,
                                                    const T* __restrict__ DLU, T* __restrict__ FA,
                                                    int* __restrict__ PV, T* __restrict__ WL, T* __restrict__ WU,
                                                    const int* __restrict__ only, int* __restrict__ info) {
  const int k = blockIdx.x, lane = threadIdx.x & 31, side = threadIdx.x >> 5;
  if (k >= nsep) return;
  const BcrSep B = bs[k];
  if (only && only[B.comp] == 0) return;
  const int role = l < B.nlev ? bcr_role(B.kloc, B.N, l) : 0;
  if (role != 1) return;
  const int s = B.s, h = 1 << l;
  const T* D = DLU + (int64_t(l) * nsep * 3 + 3 * int64_t(k)) * BCR_SS;
  T* W = (side ? WU : WL) + int64_t(k) * BCR_SS;
  T d[BCR_S], x[BCR_S];
  if (side && B.kloc + h >= B.N) {  // no block above
#pragma unroll
    for (int c = 0; c < BCR_S; ++c) x[c] = T(0);
    bcr_row_store(x, W, s, lane);
    return;
  }
  bcr_row_load(d, D, s, lane);
  bcr_row_load(x, D + (1 + side) * BCR_SS, s, lane);
  int pos;
  const bool sing = bcr_factor<T, true>(d, x, s, lane, &pos);
  bcr_row_store(x, W, s, pos);
  if (side) return;
  bcr_row_store(d, FA + int64_t(k) * BCR_SS, s, pos);
  if (lane < s) PV[int64_t(k) * BCR_S + pos] = lane;
  if (lane == 0 && sing && info) atomicCAS(info, 0, B.comp + 1);
}

// level l, kept blocks: D' = D - U W_L(k+h) - L W_U(k-h), U' = -U W_U(k+h), L' = -L W_L(k-h)
// into level l + 1.  The six blocks in shared memory, a thread per two entries.
template <typename T>
__global__ void __launch_bounds__(128) bcr_update(int nsep, const BcrSep* __restrict__ bs, int l, T* __restrict__ DLU,
                                                  const T* __restrict__ WL, const T* __restrict__ WU,
                                                  const int* __restrict__ only) {
  __shared__ T sU[BCR_SS], sL[BCR_SS], uL[BCR_SS], uU[BCR_SS], dL[BCR_SS], dU[BCR_SS];
  const int k = blockIdx.x, tid = threadIdx.x;
  if (k >= nsep) return;
  const BcrSep B = bs[k];
  if (only && only[B.comp] == 0) return;
  const int role = l < B.nlev ? bcr_role(B.kloc, B.N, l) : 0;
  if (role != 2) return;
  const int s = B.s, h = 1 << l;
  const T* cur = DLU + (int64_t(l) * nsep * 3 + 3 * int64_t(k)) * BCR_SS;
  T* nxt = DLU + (int64_t(l + 1) * nsep * 3 + 3 * int64_t(k)) * BCR_SS;
  const bool up = B.kloc + h < B.N, dn = B.kloc >= h;
  const int64_t kup = int64_t(k + h) * BCR_SS, kdn = int64_t(k - h) * BCR_SS;
#pragma unroll
  for (int q = 0; q < BCR_SS / 128; ++q) {
    const int e = tid + 128 * q;
    const bool in = e / BCR_S < s && e % BCR_S < s;
    sL[e] = in && dn ? cur[BCR_SS + e] : T(0);
    sU[e] = in && up ? cur[2 * BCR_SS + e] : T(0);
    uL[e] = in && up ? WL[kup + e] : T(0);
    uU[e] = in && up ? WU[kup + e] : T(0);
    dL[e] = in && dn ? WL[kdn + e] : T(0);
    dU[e] = in && dn ? WU[kdn + e] : T(0);
  }
  __syncthreads();
  for (int t = tid; t < s * s; t += 128) {
    const int i = t / s, j = t % s, e = i * BCR_S + j;
    T a = T(0), b = T(0), u = T(0), v = T(0);
    for (int q = 0; q < s; ++q) {
      const T x = sU[i * BCR_S + q], y = sL[i * BCR_S + q];
      a = fma(x, uL[q * BCR_S + j], a);
      b = fma(y, dU[q * BCR_S + j], b);
      u = fma(x, uU[q * BCR_S + j], u);
      v = fma(y, dL[q * BCR_S + j], v);
    }
    nxt[e] = (cur[e] - a) - b;
    nxt[BCR_SS + e] = -v;
    nxt[2 * BCR_SS + e] = -u;
  }
}

// the last block (kloc = 0) of every component: LU of its final D
template <typename T>
__global__ void __launch_bounds__(32) bcr_root(int nsep, const BcrSep* __restrict__ bs, const T* __restrict__ DLU,
                                               T* __restrict__ FA, int* __restrict__ PV, const int* __restrict__ only,
                                               int* __restrict__ info) {
  const int k = blockIdx.x, lane = threadIdx.x;
  if (k >= nsep) return;
  const BcrSep B = bs[k];
  if (B.kloc != 0 || (only && only[B.comp] == 0)) return;
  T d[BCR_S], x[BCR_S];
  bcr_row_load(d, DLU + (int64_t(B.nlev) * nsep * 3 + 3 * int64_t(k)) * BCR_SS, B.s, lane);
  int pos;
  const bool sing = bcr_factor<T, false>(d, x, B.s, lane, &pos);
  bcr_row_store(d, FA + int64_t(k) * BCR_SS, B.s, pos);
  if (lane < B.s) PV[int64_t(k) * BCR_S + pos] = lane;
  if (lane == 0 && sing && info) atomicCAS(info, 0, B.comp + 1);
}

// ---- solve: r (FP64, per separator s entries at row0[k]) -> x, stored in FP64
// and computed in the factors' type (with FP32 factors the solve is a
// refinement correction).  One warp per block; the per-block steps are device
// functions shared by the level-by-level kernels below and by the fused
// per-component solve (band_torn.cuh).

// z_k = D_k^-1 r_k with the factors FA[k] (an eliminated block at its level, or the
// root): row `lane` of the factors and entry `lane` of the vector in registers, the
// substitutions by shuffles
template <typename T>
__device__ void bcr_diag_solve_warp(const BcrSep& B, int k, const T* __restrict__ FA, const int* __restrict__ PV,
                                    const int64_t* __restrict__ row0, const double* r, double* z, int lane) {
  const int s = B.s;
  const int64_t o = row0[k];
  T f[BCR_S];
  bcr_row_load(f, FA + int64_t(k) * BCR_SS, s, lane);
  T v = lane < s ? T(r[o + PV[int64_t(k) * BCR_S + lane]]) : T(0);
  T rp = T(0);
#pragma unroll
  for (int j = 0; j < BCR_S; ++j) {  // unit lower
    if (j >= s) break;
    const T y = __shfl_sync(RB_FULL, v, j);
    if (lane > j) v = fma(-f[j], y, v);
    if (lane == j) rp = f[j];
  }
#pragma unroll
  for (int j = BCR_S - 1; j >= 0; --j) {  // upper, rows over their pivots at the end
    if (j >= s) continue;
    const T y = __shfl_sync(RB_FULL, v, j);
    if (lane < j) v = fma(-f[j], y, v);
  }
  if (lane < s) z[o + lane] = double(v * rp);
  __syncwarp();
}

// v − M1 w1 − M2 w2 for row `lane` of two blocks and the entries `lane` of two vectors
template <typename T>
__device__ __forceinline__ T bcr_row_sub(T v, const T m1[BCR_S], T w1, const T m2[BCR_S], T w2, int s) {
  T a = T(0);
#pragma unroll
  for (int q = 0; q < BCR_S; ++q) {
    if (q >= s) break;
    v = fma(-m1[q], __shfl_sync(RB_FULL, w1, q), v);
    a = fma(-m2[q], __shfl_sync(RB_FULL, w2, q), a);
  }
  return v + a;
}

// kept block e at level l: r_e -= U_e z_{e+h} + L_e z_{e-h}
template <typename T>
__device__ void bcr_keep_warp(const BcrSep& B, int k, int l, int nsep, const T* __restrict__ DLU,
                              const int64_t* __restrict__ row0, double* r, const double* z, int lane) {
  const int s = B.s, h = 1 << l;
  const T* cur = DLU + (int64_t(l) * nsep * 3 + 3 * int64_t(k)) * BCR_SS;
  const bool up = B.kloc + h < B.N, dn = B.kloc >= h;
  T u[BCR_S], d[BCR_S];
  bcr_row_load(u, cur + 2 * BCR_SS, up ? s : 0, lane);
  bcr_row_load(d, cur + BCR_SS, dn ? s : 0, lane);
  const T wu = up && lane < s ? T(z[row0[k + h] + lane]) : T(0), wd = dn && lane < s ? T(z[row0[k - h] + lane]) : T(0);
  const int64_t o = row0[k];
  const T v = bcr_row_sub(lane < s ? T(r[o + lane]) : T(0), u, wu, d, wd, s);
  if (lane < s) r[o + lane] = double(v);
  __syncwarp();
}

// eliminated block k at level l: x_k = z_k - W_L(k) x_{k-h} - W_U(k) x_{k+h}  (z holds z_k and the kept x)
template <typename T>
__device__ void bcr_back_warp(const BcrSep& B, int k, int l, const T* __restrict__ WL, const T* __restrict__ WU,
                              const int64_t* __restrict__ row0, double* z, int lane) {
  const int s = B.s, h = 1 << l;
  const bool up = B.kloc + h < B.N;
  const int64_t o = row0[k];
  T wl[BCR_S], wu[BCR_S];
  bcr_row_load(wl, WL + int64_t(k) * BCR_SS, s, lane);
  bcr_row_load(wu, WU + int64_t(k) * BCR_SS, up ? s : 0, lane);
  const T xl = lane < s ? T(z[row0[k - h] + lane]) : T(0), xu = up && lane < s ? T(z[row0[k + h] + lane]) : T(0);
  const T v = bcr_row_sub(lane < s ? T(z[o + lane]) : T(0), wl, xl, wu, xu, s);
  if (lane < s) z[o + lane] = double(v);
  __syncwarp();
}

// level-by-level kernels: one warp per separator of every component
// forward, level l: eliminated z_k = D_k^-1 r_k
template <typename T>
__global__ void __launch_bounds__(32) bcr_fwd_elim(int nsep, const BcrSep* __restrict__ bs, int l,
                                                   const T* __restrict__ FA, const int* __restrict__ PV,
                                                   const int64_t* __restrict__ row0, const double* __restrict__ r,
                                                   double* __restrict__ z, const int* __restrict__ only) {
  const int k = blockIdx.x;
  if (k >= nsep) return;
  const BcrSep B = bs[k];
  if (only && only[B.comp] == 0) return;
  if (!(l < B.nlev && bcr_role(B.kloc, B.N, l) == 1)) return;
  bcr_diag_solve_warp(B, k, FA, PV, row0, r, z, threadIdx.x);
}

// forward, level l: kept r_e -= U_e z_{e+h} + L_e z_{e-h}
template <typename T>
__global__ void __launch_bounds__(32) bcr_fwd_keep(int nsep, const BcrSep* __restrict__ bs, int l,
                                                   const T* __restrict__ DLU, const int64_t* __restrict__ row0,
                                                   double* __restrict__ r, const double* __restrict__ z,
                                                   const int* __restrict__ only) {
  const int k = blockIdx.x;
  if (k >= nsep) return;
  const BcrSep B = bs[k];
  if (only && only[B.comp] == 0) return;
  if (!(l < B.nlev && bcr_role(B.kloc, B.N, l) == 2)) return;
  bcr_keep_warp(B, k, l, nsep, DLU, row0, r, z, threadIdx.x);
}

// root: x_0 = D_0^-1 r_0 (into z, which then holds x for every block as the back-substitution proceeds)
template <typename T>
__global__ void __launch_bounds__(32) bcr_root_solve(int nsep, const BcrSep* __restrict__ bs,
                                                     const T* __restrict__ FA, const int* __restrict__ PV,
                                                     const int64_t* __restrict__ row0, const double* __restrict__ r,
                                                     double* __restrict__ z, const int* __restrict__ only) {
  const int k = blockIdx.x;
  if (k >= nsep) return;
  const BcrSep B = bs[k];
  if (B.kloc != 0 || (only && only[B.comp] == 0)) return;
  bcr_diag_solve_warp(B, k, FA, PV, row0, r, z, threadIdx.x);
}

// backward, level l
template <typename T>
__global__ void __launch_bounds__(32) bcr_back(int nsep, const BcrSep* __restrict__ bs, int l,
                                               const T* __restrict__ WL, const T* __restrict__ WU,
                                               const int64_t* __restrict__ row0, double* __restrict__ z,
                                               const int* __restrict__ only) {
  const int k = blockIdx.x;
  if (k >= nsep) return;
  const BcrSep B = bs[k];
  if (only && only[B.comp] == 0) return;
  if (!(l < B.nlev && bcr_role(B.kloc, B.N, l) == 1)) return;
  bcr_back_warp(B, k, l, WL, WU, row0, z, threadIdx.x);
}

}  // namespace mgpu
