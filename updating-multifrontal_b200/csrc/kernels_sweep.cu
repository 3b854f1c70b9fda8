// Forward / backward sweeps of one front per CTA (src/DE/mf2d.cpp:976-1054),
// for the levels of many small fronts, and of pivoted LU fronts (nonsymmetric
// problems, FP64; factors from kernels_lu.cu).
//
// A front's 32-column blocks are solved in order.  Bound: the chain of blocks
// (one 32 x 32 triangular solve each), and HBM once enough CTAs overlap their
// chains.  So the chain is kept short and everything else is off it:
//   * warp 0 keeps the block's right-hand sides in registers, a row per lane
//     (a column per lane in the transposed solves), scaled by the reciprocal
//     diagonal beforehand: a step of the substitution is one shuffle and one
//     multiply-add, with no division, barrier or shared-memory round trip;
//   * warp 0 also applies the block solved just before (its 32 x 32 block of
//     L is in shared memory), so the other warps' work is a step behind and
//     one barrier per block orders everything;
//   * meanwhile the other warps apply the last solved block to the rows
//     below (forward), or form the products of the next block's columns with
//     the rows already solved (backward), and bring the next two 32 x 32
//     blocks to shared memory with cp.async.
// Measured against a substitution through shared memory (a division and two
// warp barriers per column) followed by the updates: 2D 1023^2 leaves (4096
// fronts of 285 x 225), 4 right-hand sides, forward 989 -> 389 us, backward
// 1310 -> 457 us (3 TB/s); a 2D 63^2 solve of 10 launches 250 -> 116 us.
#include <algorithm>
#include <atomic>
#include <cstdint>

#include "device.cuh"

namespace mfgpu {

extern std::atomic<long long> g_launches;

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kMaxHelpers = 8;               // warps beside warp 0
constexpr int kSweepThreads = 32 * (1 + kMaxHelpers);

// Shared memory of a sweep: the diagonal block and the block beside it of the
// current and the next step (column t of the block is [t][*]), the solved
// block and the helpers' products of both.
template <class T, int NR>
struct SweepSm {
  T D[2][kPanel][kPanel + 1];
  T S[2][kPanel][kPanel + 1];
  T v[2][kPanel][NR];
  T p[2][kPanel][NR];
};

// Block (rows rs .., columns cs ..) of A, 32 x 32, entries outside rend / cend
// zero, to B (column-major), by the helpers (thread u of nu).
template <class T>
__device__ __forceinline__ void fetch_block(T (*B)[kPanel + 1], const T* __restrict__ A, int64_t ld,
                                            int rs, int cs, int rend, int cend, int u, int nu) {
  for (int idx = u; idx < kPanel * kPanel; idx += nu) {
    const int r = idx & 31, c = idx >> 5;
    const bool take = rs + r < rend && cs + c < cend;
    cp_elem(&B[c][r], take ? A + (rs + r) + (int64_t)(cs + c) * ld : A, take);
  }
}

// w <- L^{-1} w (lower, row per lane: entry (lane, j) is D[j][lane]).  UNIT:
// the stored diagonal is not L's.  rows beyond kb hold zero.
template <class T, int NR, bool UNIT>
__device__ __forceinline__ void lower_solve(const T (*D)[kPanel + 1], int kb, int lane, T (&w)[NR]) {
  const T rd = UNIT || lane >= kb ? T(1) : T(1) / D[lane][lane];
  if (!UNIT)
#pragma unroll
    for (int c = 0; c < NR; c++) w[c] *= rd;
#pragma unroll 8
  for (int j = 0; j < kPanel - 1; j++) {
    const T l = lane > j && lane < kb ? (UNIT ? D[j][lane] : D[j][lane] * rd) : T(0);
#pragma unroll
    for (int c = 0; c < NR; c++) {
      const T y = __shfl_sync(kAll, w[c], j);
      if (lane > j) w[c] = fma(-l, y, w[c]);
    }
  }
}

// w <- U^{-1} w, upper: entry (lane, j), j > lane, is D[lane][j] (TR: U = L^T,
// D holds L) or D[j][lane] (D holds U).
template <class T, int NR, bool TR>
__device__ __forceinline__ void upper_solve(const T (*D)[kPanel + 1], int kb, int lane, T (&w)[NR]) {
  const T rd = lane < kb ? T(1) / D[lane][lane] : T(1);
#pragma unroll
  for (int c = 0; c < NR; c++) w[c] *= rd;
#pragma unroll 8
  for (int j = kPanel - 1; j > 0; j--) {
    const T u = lane < j && j < kb ? (TR ? D[lane][j] : D[j][lane]) * rd : T(0);
#pragma unroll
    for (int c = 0; c < NR; c++) {
      const T x = __shfl_sync(kAll, w[c], j);
      if (lane < j) w[c] = fma(-u, x, w[c]);
    }
  }
}

// W(r, :) -= L(r, k : k + kb) v for rows r0 + u, + nu, ... below N.
template <class T, int NR>
__device__ __forceinline__ void apply_block(const T* __restrict__ A, int64_t ld, int k, int kb,
                                            const T (*v)[NR], int r0, int N, T* W, int nrhs, int u,
                                            int nu) {
  for (int r = r0 + u; r < N; r += nu) {
    T acc[NR];
#pragma unroll
    for (int c = 0; c < NR; c++) acc[c] = T(0);
    const T* Lr = A + r + (int64_t)k * ld;
    if (kb == kPanel) {
#pragma unroll
      for (int h = 0; h < kPanel; h += 16) {   // 16 loads in flight
        T l[16];
#pragma unroll
        for (int t = 0; t < 16; t++) l[t] = Lr[(int64_t)(h + t) * ld];
#pragma unroll
        for (int t = 0; t < 16; t++)
#pragma unroll
          for (int c = 0; c < NR; c++) acc[c] = fma(l[t], v[h + t][c], acc[c]);
      }
    } else {
      for (int t = 0; t < kb; t++) {
        const T l = Lr[(int64_t)t * ld];
#pragma unroll
        for (int c = 0; c < NR; c++) acc[c] = fma(l, v[t][c], acc[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < NR; c++)
      if (c < nrhs) W[r + (int64_t)c * N] -= acc[c];
  }
}

// Forward solve: W[0,n) <- L11^{-1} W[0,n), W[n,N) -= L21 W[0,n).  W is the
// front's right-hand-side block (N x nrhs, ld N) in shared or global memory.
// UNIT: L11 of a pivoted LU front.
template <class T, int NR, bool UNIT = false>
__device__ void front_forward(const FrontDev& d, const T* __restrict__ A, T* W, int nrhs,
                              SweepSm<T, NR>& sm) {
  const int N = d.N, n = d.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t ld = d.ld;
  const int u = (int)threadIdx.x - 32, nu = (int)blockDim.x - 32;
  if (n <= 0) return;
  if (warp > 0) fetch_block(sm.D[0], A, ld, 0, 0, n, n, u, nu);
  cp_commit();
  cp_wait<0>();
  __syncthreads();
  int b = 0, k = 0;
  for (; k < n; k += kPanel, b ^= 1) {
    const int kb = min(kPanel, n - k);
    if (warp == 0) {
      T w[NR];
#pragma unroll
      for (int c = 0; c < NR; c++)
        w[c] = lane < kb && c < nrhs ? W[k + lane + (int64_t)c * N] : T(0);
      if (k > 0) {   // the block before
        T a0[NR], a1[NR];
#pragma unroll
        for (int c = 0; c < NR; c++) a0[c] = a1[c] = T(0);
#pragma unroll 8
        for (int t = 0; t < kPanel; t += 2) {
          const T s0 = sm.S[b][t][lane], s1 = sm.S[b][t + 1][lane];
#pragma unroll
          for (int c = 0; c < NR; c++) {
            a0[c] = fma(s0, sm.v[b ^ 1][t][c], a0[c]);
            a1[c] = fma(s1, sm.v[b ^ 1][t + 1][c], a1[c]);
          }
        }
        if (lane < kb)
#pragma unroll
          for (int c = 0; c < NR; c++) w[c] -= a0[c] + a1[c];
      }
      lower_solve<T, NR, UNIT>(sm.D[b], kb, lane, w);
#pragma unroll
      for (int c = 0; c < NR; c++) {
        sm.v[b][lane][c] = w[c];
        if (lane < kb && c < nrhs) W[k + lane + (int64_t)c * N] = w[c];
      }
    } else {
      if (k + kPanel < n) {
        fetch_block(sm.D[b ^ 1], A, ld, k + kPanel, k + kPanel, n, n, u, nu);
        fetch_block(sm.S[b ^ 1], A, ld, k + kPanel, k, n, n, u, nu);
        cp_commit();
      }
      if (k > 0) apply_block<T, NR>(A, ld, k - kPanel, kPanel, sm.v[b ^ 1], k + kb, N, W, nrhs, u, nu);
      cp_wait<0>();
    }
    __syncthreads();
  }
  // the last block on the boundary rows
  const int kl = k - kPanel;
  apply_block<T, NR>(A, ld, kl, n - kl, sm.v[b ^ 1], n, N, W, nrhs, threadIdx.x, blockDim.x);
  __syncthreads();
}

// Sums v[0 .. V) over the warp: lane l ends with the sum of entry l / (32 / V)
// in v[0] (V a power of two up to 32), V - 1 exchanges instead of 5 V.
template <class T, int V>
__device__ __forceinline__ void warp_sum_scatter(T* v, int lane) {
  int o = 16;
#pragma unroll
  for (int h = V / 2; h >= 1; h >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; i++) {
      const T send = up ? v[i] : v[i + h];
      const T keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(kAll, send, o);
    }
    o >>= 1;
  }
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(kAll, v[0], o);
}

// p(j, :) = sum over rows r in [r0, N) of L(r, k + j) W(r, :), j < kb: CPW
// columns of a warp at a time (helper h of nh), lanes along the rows.
template <class T, int NR>
__device__ __forceinline__ void column_products(const T* __restrict__ A, int64_t ld, int k, int kb,
                                                int r0, int N, const T* W, int nrhs, T (*p)[NR],
                                                int h, int nh, int lane) {
  constexpr int CPW = NR >= 16 ? 2 : 4, V = CPW * NR, RU = NR <= 4 ? 4 : 2;
  for (int j = h * CPW; j < kPanel; j += nh * CPW) {
    T acc[V];
#pragma unroll
    for (int i = 0; i < V; i++) acc[i] = T(0);
    for (int r = r0 + lane; r < N; r += 32 * RU) {
      T l[RU][CPW];
#pragma unroll
      for (int q = 0; q < RU; q++)
#pragma unroll
        for (int i = 0; i < CPW; i++)
          l[q][i] = (r + 32 * q < N && j + i < kb) ? A[r + 32 * q + (int64_t)(k + j + i) * ld] : T(0);
#pragma unroll
      for (int q = 0; q < RU; q++)
        if (r + 32 * q < N)
#pragma unroll
          for (int c = 0; c < NR; c++) {
            const T x = c < nrhs ? W[r + 32 * q + (int64_t)c * N] : T(0);
#pragma unroll
            for (int i = 0; i < CPW; i++) acc[i * NR + c] = fma(l[q][i], x, acc[i * NR + c]);
          }
    }
    warp_sum_scatter<T, V>(acc, lane);
    const int e = lane / (32 / V);
    if (lane % (32 / V) == 0) p[j + e / NR][e % NR] = acc[0];
  }
}

// Backward solve: W[0,n) <- L11^{-T} (W[0,n) - L21^T W[n,N)).
template <class T, int NR>
__device__ void front_backward(const FrontDev& d, const T* __restrict__ A, T* W, int nrhs,
                               SweepSm<T, NR>& sm) {
  const int N = d.N, n = d.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t ld = d.ld;
  const int u = (int)threadIdx.x - 32, nu = (int)blockDim.x - 32, nh = nu / 32;
  if (n <= 0) return;
  int k = (n - 1) / kPanel * kPanel, b = 0;
  if (warp > 0) {
    fetch_block(sm.D[0], A, ld, k, k, n, n, u, nu);
    cp_commit();
    column_products<T, NR>(A, ld, k, n - k, n, N, W, nrhs, sm.p[0], warp - 1, nh, lane);
    cp_wait<0>();
  }
  __syncthreads();
  for (bool first = true; k >= 0; k -= kPanel, b ^= 1, first = false) {
    const int kb = min(kPanel, n - k);
    if (warp == 0) {
      T w[NR];
#pragma unroll
      for (int c = 0; c < NR; c++)
        w[c] = lane < kb && c < nrhs ? W[k + lane + (int64_t)c * N] - sm.p[b][lane][c] : T(0);
      if (!first) {   // the block solved before, below this one
        T a0[NR], a1[NR];
#pragma unroll
        for (int c = 0; c < NR; c++) a0[c] = a1[c] = T(0);
#pragma unroll 8
        for (int t = 0; t < kPanel; t += 2) {
          const T s0 = sm.S[b][lane][t], s1 = sm.S[b][lane][t + 1];
#pragma unroll
          for (int c = 0; c < NR; c++) {
            a0[c] = fma(s0, sm.v[b ^ 1][t][c], a0[c]);
            a1[c] = fma(s1, sm.v[b ^ 1][t + 1][c], a1[c]);
          }
        }
#pragma unroll
        for (int c = 0; c < NR; c++) w[c] -= a0[c] + a1[c];
      }
      upper_solve<T, NR, true>(sm.D[b], kb, lane, w);
#pragma unroll
      for (int c = 0; c < NR; c++) {
        sm.v[b][lane][c] = w[c];
        if (lane < kb && c < nrhs) W[k + lane + (int64_t)c * N] = w[c];
      }
    } else if (k > 0) {
      const int kn = k - kPanel;
      fetch_block(sm.D[b ^ 1], A, ld, kn, kn, n, n, u, nu);
      fetch_block(sm.S[b ^ 1], A, ld, k, kn, n, n, u, nu);
      cp_commit();
      column_products<T, NR>(A, ld, kn, kPanel, k + kb, N, W, nrhs, sm.p[b ^ 1], warp - 1, nh, lane);
      cp_wait<0>();
    }
    __syncthreads();
  }
}

template <class T, int NR>
__device__ __forceinline__ T* rhs_block(SweepSm<T, NR>& sm, T* Wg, int use_smem) {
  return use_smem ? reinterpret_cast<T*>(&sm + 1) : Wg;
}

template <class T, int NR>
__global__ void __launch_bounds__(kSweepThreads, NR <= 4 ? 3 : 2)
    k_solve_fwd(const int* __restrict__ flist, const FrontDev* __restrict__ fr,
                const T* __restrict__ F, const int* __restrict__ dofs, T* X, int64_t ldx, int nrhs,
                T* Wb, const int64_t* __restrict__ woff, int use_smem) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SweepSm<T, NR>& sm = *reinterpret_cast<SweepSm<T, NR>*>(smraw);
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  T* Wg = Wb + woff[f] * nrhs;
  T* W = rhs_block(sm, Wg, use_smem);
  const int* dl = dofs + d.dof_off;
  for (int idx = threadIdx.x; idx < d.N * nrhs; idx += blockDim.x) {
    const int i = idx % d.N, c = idx / d.N;
    W[idx] = i < d.n ? X[dl[i] + (int64_t)c * ldx] : T(0);
  }
  __syncthreads();
  front_forward<T, NR>(d, F + d.off, W, nrhs, sm);
  for (int idx = threadIdx.x; idx < d.N * nrhs; idx += blockDim.x) {
    const int i = idx % d.N, c = idx / d.N;
    if (i < d.n) X[dl[i] + (int64_t)c * ldx] = W[idx];
    else if (use_smem) Wg[idx] = W[idx];    // boundary part for the separator gather
  }
}

template <class T, int NR>
__global__ void __launch_bounds__(kSweepThreads, NR <= 4 ? 3 : 2)
    k_solve_bwd(const int* __restrict__ flist, const FrontDev* __restrict__ fr,
                const T* __restrict__ F, const int* __restrict__ dofs, T* X, int64_t ldx, int nrhs,
                T* Wb, const int64_t* __restrict__ woff, int use_smem) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SweepSm<T, NR>& sm = *reinterpret_cast<SweepSm<T, NR>*>(smraw);
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  T* W = rhs_block(sm, Wb + woff[f] * nrhs, use_smem);
  const int* dl = dofs + d.dof_off;
  for (int idx = threadIdx.x; idx < d.N * nrhs; idx += blockDim.x) {
    const int i = idx % d.N, c = idx / d.N;
    W[idx] = X[dl[i] + (int64_t)c * ldx];
  }
  __syncthreads();
  front_backward<T, NR>(d, F + d.off, W, nrhs, sm);
  for (int idx = threadIdx.x; idx < d.n * nrhs; idx += blockDim.x) {
    const int i = idx % d.n, c = idx / d.n;
    X[dl[i] + (int64_t)c * ldx] = W[i + (int64_t)c * d.N];
  }
}

template <class T, int NR>
__global__ void __launch_bounds__(kSweepThreads, 2)
    k_root_solve(int f, const FrontDev* __restrict__ fr, const T* __restrict__ F,
                 const int* __restrict__ dofs, T* X, int64_t ldx, int nrhs, T* Wb,
                 const int64_t* __restrict__ woff, int use_smem) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SweepSm<T, NR>& sm = *reinterpret_cast<SweepSm<T, NR>*>(smraw);
  const FrontDev d = fr[f];
  T* W = rhs_block(sm, Wb + woff[f] * nrhs, use_smem);
  const int* dl = dofs + d.dof_off;
  for (int idx = threadIdx.x; idx < d.N * nrhs; idx += blockDim.x) {
    const int i = idx % d.N, c = idx / d.N;
    W[idx] = X[dl[i] + (int64_t)c * ldx];
  }
  __syncthreads();
  front_forward<T, NR>(d, F + d.off, W, nrhs, sm);
  front_backward<T, NR>(d, F + d.off, W, nrhs, sm);
  for (int idx = threadIdx.x; idx < d.n * nrhs; idx += blockDim.x) {
    const int i = idx % d.n, c = idx / d.n;
    X[dl[i] + (int64_t)c * ldx] = W[i + (int64_t)c * d.N];
  }
}

// ---------------------------------------------------------------------------
// Pivoted LU fronts: P A22 = L11 U11, L21 = A12 U11^{-1}, U12 = L11^{-1} P A21.
// The reference's upward step b_sk -= XL b_rd, b_rd <- A22^{-1} b_rd and
// downward step b_rd -= XR b_sk (src/DE/mf2d.cpp:976-1054) become
//   forward:  y = L11^{-1} P b_piv (kept as the pivot part), W[n,N) = -L21 y
//   backward: x_piv = U11^{-1} (y - U12 x_bd)
// since XL = L21 L11^{-1} P and XR = U11^{-1} U12.
// ---------------------------------------------------------------------------

// q[h](i, :) = sum over columns c in [c0, N), c = c0 + h mod nh, of
// U(k + i, c) W(c, :), a row per lane (helper h of nh).
template <int NR>
__device__ __forceinline__ void row_products(const double* __restrict__ A, int64_t ld, int k, int kb,
                                             int c0, int N, const double* W, int nrhs,
                                             double (*q)[NR], int h, int nh, int lane) {
  double acc[NR];
#pragma unroll
  for (int c = 0; c < NR; c++) acc[c] = 0.0;
  if (lane < kb) {
    const double* Ur = A + k + lane;
    int c = c0 + h;
    for (; c + 7 * nh < N; c += 8 * nh) {   // eight loads in flight
      double a[8];
#pragma unroll
      for (int t = 0; t < 8; t++) a[t] = Ur[(int64_t)(c + t * nh) * ld];
#pragma unroll
      for (int t = 0; t < 8; t++)
#pragma unroll
        for (int e = 0; e < NR; e++)
          if (e < nrhs) acc[e] = fma(a[t], W[c + t * nh + (int64_t)e * N], acc[e]);
    }
    for (; c < N; c += nh) {
      const double a = Ur[(int64_t)c * ld];
#pragma unroll
      for (int e = 0; e < NR; e++)
        if (e < nrhs) acc[e] = fma(a, W[c + (int64_t)e * N], acc[e]);
    }
  }
#pragma unroll
  for (int c = 0; c < NR; c++) q[lane][c] = acc[c];
}

// Backward solve: W[0,n) <- U11^{-1} (W[0,n) - U12 W[n,N)).
template <int NR>
__device__ void front_backward_lu(const FrontDev& d, const double* __restrict__ A, double* W,
                                  int nrhs, SweepSm<double, NR>& sm,
                                  double (*q)[kMaxHelpers][kPanel][NR]) {
  const int N = d.N, n = d.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t ld = d.ld;
  const int u = (int)threadIdx.x - 32, nu = (int)blockDim.x - 32, nh = nu / 32;
  if (n <= 0) return;
  int k = (n - 1) / kPanel * kPanel, b = 0;
  if (warp > 0) {
    fetch_block(sm.D[0], A, ld, k, k, n, n, u, nu);
    cp_commit();
    row_products<NR>(A, ld, k, n - k, n, N, W, nrhs, q[0][warp - 1], warp - 1, nh, lane);
    cp_wait<0>();
  }
  __syncthreads();
  for (bool first = true; k >= 0; k -= kPanel, b ^= 1, first = false) {
    const int kb = min(kPanel, n - k);
    if (warp == 0) {
      double w[NR];
#pragma unroll
      for (int c = 0; c < NR; c++) w[c] = 0.0;
      for (int h = 0; h < nh; h++)
#pragma unroll
        for (int c = 0; c < NR; c++) w[c] += q[b][h][lane][c];
      if (!first) {
#pragma unroll 8
        for (int t = 0; t < kPanel; t++) {
          const double s = sm.S[b][t][lane];
#pragma unroll
          for (int c = 0; c < NR; c++) w[c] = fma(s, sm.v[b ^ 1][t][c], w[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < NR; c++)
        w[c] = lane < kb && c < nrhs ? W[k + lane + (int64_t)c * N] - w[c] : 0.0;
      upper_solve<double, NR, false>(sm.D[b], kb, lane, w);
#pragma unroll
      for (int c = 0; c < NR; c++) {
        sm.v[b][lane][c] = w[c];
        if (lane < kb && c < nrhs) W[k + lane + (int64_t)c * N] = w[c];
      }
    } else if (k > 0) {
      const int kn = k - kPanel;
      fetch_block(sm.D[b ^ 1], A, ld, kn, kn, n, n, u, nu);
      fetch_block(sm.S[b ^ 1], A, ld, kn, k, n, n, u, nu);
      cp_commit();
      row_products<NR>(A, ld, kn, kPanel, k + kb, N, W, nrhs, q[b ^ 1][warp - 1], warp - 1, nh, lane);
      cp_wait<0>();
    }
    __syncthreads();
  }
}

template <int NR>
__global__ void __launch_bounds__(kSweepThreads, 2)
    k_lu_solve_fwd(const int* __restrict__ flist, const FrontDev* __restrict__ fr,
                   const double* __restrict__ F, const int* __restrict__ ipiv,
                   const int* __restrict__ dofs, double* X, int64_t ldx, int nrhs, double* Wb,
                   const int64_t* __restrict__ woff, int use_smem) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SweepSm<double, NR>& sm = *reinterpret_cast<SweepSm<double, NR>*>(smraw);
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  double* Wg = Wb + woff[f] * nrhs;
  double* W = rhs_block(sm, Wg, use_smem);
  const int* dl = dofs + d.dof_off;
  const int* pv = ipiv + d.dof_off;
  for (int idx = threadIdx.x; idx < d.N * nrhs; idx += blockDim.x) {
    const int i = idx % d.N, c = idx / d.N;
    W[idx] = i < d.n ? X[dl[i] + (int64_t)c * ldx] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < 32) {   // b_piv <- P b_piv: the swaps in factorization order, a lane per vector
    const int lane = threadIdx.x;
    double* w = W + (int64_t)lane * d.N;
    int next = lane < d.n ? pv[lane] : 0;
    for (int j0 = 0; j0 < d.n; j0 += 32) {
      const int mine = next;
      next = j0 + 32 + lane < d.n ? pv[j0 + 32 + lane] : 0;
      for (int t = 0; t < min(32, d.n - j0); t++) {
        const int j = j0 + t, p = __shfl_sync(kAll, mine, t);
        if (p != j && lane < nrhs) {
          const double x = w[j];
          w[j] = w[p];
          w[p] = x;
        }
      }
    }
  }
  __syncthreads();
  front_forward<double, NR, true>(d, F + d.off, W, nrhs, sm);
  for (int idx = threadIdx.x; idx < d.N * nrhs; idx += blockDim.x) {
    const int i = idx % d.N, c = idx / d.N;
    if (i < d.n) X[dl[i] + (int64_t)c * ldx] = W[idx];
    else if (use_smem) Wg[idx] = W[idx];    // boundary part for the separator gather
  }
}

template <int NR>
__global__ void __launch_bounds__(kSweepThreads, 2)
    k_lu_solve_bwd(const int* __restrict__ flist, const FrontDev* __restrict__ fr,
                   const double* __restrict__ F, const int* __restrict__ dofs, double* X,
                   int64_t ldx, int nrhs, double* Wb, const int64_t* __restrict__ woff,
                   int use_smem) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SweepSm<double, NR>& sm = *reinterpret_cast<SweepSm<double, NR>*>(smraw);
  using Parts = double[kMaxHelpers][kPanel][NR];
  Parts* q = reinterpret_cast<Parts*>(&sm + 1);
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  double* W = use_smem ? reinterpret_cast<double*>(q + 2) : Wb + woff[f] * nrhs;
  const int* dl = dofs + d.dof_off;
  for (int idx = threadIdx.x; idx < d.N * nrhs; idx += blockDim.x) {
    const int i = idx % d.N, c = idx / d.N;
    W[idx] = X[dl[i] + (int64_t)c * ldx];
  }
  __syncthreads();
  front_backward_lu<NR>(d, F + d.off, W, nrhs, sm, q);
  for (int idx = threadIdx.x; idx < d.n * nrhs; idx += blockDim.x) {
    const int i = idx % d.n, c = idx / d.n;
    X[dl[i] + (int64_t)c * ldx] = W[i + (int64_t)c * d.N];
  }
}

// Threads per CTA: warp 0 and enough helpers for the level's largest front (a
// thread per row below a block), so that small fronts (the leaves of a batch)
// leave room for more CTAs per SM.  A Cholesky front's values are computed by
// the same operations in the same order whatever the block size.
int sweep_threads(int maxN) { return 32 * (1 + (maxN <= 64 ? 2 : maxN <= 128 ? 4 : kMaxHelpers)); }

// Dynamic shared memory: `fixed` bytes, then the front's right-hand-side block
// when the level's largest front's fits.
constexpr size_t kSweepSmemMax = 227 * 1024;
size_t sweep_smem(size_t fixed, int maxN, int nrhs, size_t elem, int& use) {
  const size_t need = fixed + (size_t)maxN * nrhs * elem;
  use = need <= kSweepSmemMax;
  return use ? need : fixed;
}

// Launch configuration of kernel K with `fixed` bytes of shared memory besides
// the right-hand sides (the attribute is set once, thread-safely).
#define MFGPU_SWEEP(K, FIXED, ELEM, GRID, MAXN, ...)                                             \
  do {                                                                                           \
    static const bool attr_ = (cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                    (int)kSweepSmemMax),                          \
                               true);                                                            \
    (void)attr_;                                                                                 \
    int use;                                                                                     \
    const size_t sm = sweep_smem(FIXED, MAXN, nrhs, ELEM, use);                                   \
    K<<<GRID, sweep_threads(MAXN), sm, st>>>(__VA_ARGS__, use);                                   \
  } while (0)

template <class T, int NR>
void sweep_fwd(const int* flist, int nf, int maxN, const FrontDev* fr, const T* F, const int* dofs,
               T* X, int64_t ldx, int nrhs, T* W, const int64_t* woff, cudaStream_t st) {
  MFGPU_SWEEP((k_solve_fwd<T, NR>), sizeof(SweepSm<T, NR>), sizeof(T), nf, maxN, flist, fr, F, dofs,
              X, ldx, nrhs, W, woff);
}
template <class T, int NR>
void sweep_bwd(const int* flist, int nf, int maxN, const FrontDev* fr, const T* F, const int* dofs,
               T* X, int64_t ldx, int nrhs, T* W, const int64_t* woff, cudaStream_t st) {
  MFGPU_SWEEP((k_solve_bwd<T, NR>), sizeof(SweepSm<T, NR>), sizeof(T), nf, maxN, flist, fr, F, dofs,
              X, ldx, nrhs, W, woff);
}
template <class T, int NR>
void sweep_root(int f, int N, const FrontDev* fr, const T* F, const int* dofs, T* X, int64_t ldx,
                int nrhs, T* W, const int64_t* woff, cudaStream_t st) {
  MFGPU_SWEEP((k_root_solve<T, NR>), sizeof(SweepSm<T, NR>), sizeof(T), 1, N, f, fr, F, dofs, X, ldx,
              nrhs, W, woff);
}
template <int NR>
void sweep_lu(bool forward, const int* flist, int nf, int maxN, const FrontDev* fr, const double* F,
              const int* ipiv, const int* dofs, double* X, int64_t ldx, int nrhs, double* W,
              const int64_t* woff, cudaStream_t st) {
  constexpr size_t fixed = sizeof(SweepSm<double, NR>);
  if (forward)
    MFGPU_SWEEP((k_lu_solve_fwd<NR>), fixed, sizeof(double), nf, maxN, flist, fr, F, ipiv, dofs, X,
                ldx, nrhs, W, woff);
  else
    MFGPU_SWEEP((k_lu_solve_bwd<NR>), fixed + 2 * sizeof(double) * kMaxHelpers * kPanel * NR,
                sizeof(double), nf, maxN, flist, fr, F, dofs, X, ldx, nrhs, W, woff);
}

}  // namespace

// The kernels are templated on a bound of the right-hand-side count.
#define MFGPU_BY_NRHS(FN, ...)              \
  do {                                      \
    if (nrhs == 1) FN(1)(__VA_ARGS__);      \
    else if (nrhs <= 4) FN(4)(__VA_ARGS__); \
    else if (nrhs <= 8) FN(8)(__VA_ARGS__); \
    else FN(16)(__VA_ARGS__);               \
  } while (0)

template <class T>
void launch_solve_fwd(const int* flist, int nf, int maxN, const FrontDev* fr, const T* F,
                      const int* dofs, T* X, int64_t ldx, int nrhs, T* W, const int64_t* woff,
                      cudaStream_t st) {
  if (nf <= 0) return;
#define MFGPU_FN(NR) sweep_fwd<T, NR>
  MFGPU_BY_NRHS(MFGPU_FN, flist, nf, maxN, fr, F, dofs, X, ldx, nrhs, W, woff, st);
#undef MFGPU_FN
  g_launches++;
}

template <class T>
void launch_solve_bwd(const int* flist, int nf, int maxN, const FrontDev* fr, const T* F,
                      const int* dofs, T* X, int64_t ldx, int nrhs, T* W, const int64_t* woff,
                      cudaStream_t st) {
  if (nf <= 0) return;
#define MFGPU_FN(NR) sweep_bwd<T, NR>
  MFGPU_BY_NRHS(MFGPU_FN, flist, nf, maxN, fr, F, dofs, X, ldx, nrhs, W, woff, st);
#undef MFGPU_FN
  g_launches++;
}

template <class T>
void launch_root_solve(int f, int N, const FrontDev* fr, const T* F, const int* dofs, T* X,
                       int64_t ldx, int nrhs, T* W, const int64_t* woff, cudaStream_t st) {
#define MFGPU_FN(NR) sweep_root<T, NR>
  MFGPU_BY_NRHS(MFGPU_FN, f, N, fr, F, dofs, X, ldx, nrhs, W, woff, st);
#undef MFGPU_FN
  g_launches++;
}

void launch_lu_solve(bool forward, const int* flist, int nf, int maxN, const FrontDev* fr,
                     const double* F, const int* ipiv, const int* dofs, double* X, int64_t ldx,
                     int nrhs, double* W, const int64_t* woff, cudaStream_t st) {
  if (nf <= 0) return;
#define MFGPU_FN(NR) sweep_lu<NR>
  MFGPU_BY_NRHS(MFGPU_FN, forward, flist, nf, maxN, fr, F, ipiv, dofs, X, ldx, nrhs, W, woff, st);
#undef MFGPU_FN
  g_launches++;
}

#define MFGPU_INSTANTIATE(T)                                                                       \
  template void launch_solve_fwd<T>(const int*, int, int, const FrontDev*, const T*, const int*,    \
                                    T*, int64_t, int, T*, const int64_t*, cudaStream_t);            \
  template void launch_solve_bwd<T>(const int*, int, int, const FrontDev*, const T*, const int*,    \
                                    T*, int64_t, int, T*, const int64_t*, cudaStream_t);            \
  template void launch_root_solve<T>(int, int, const FrontDev*, const T*, const int*, T*, int64_t,  \
                                     int, T*, const int64_t*, cudaStream_t);
MFGPU_INSTANTIATE(double)
MFGPU_INSTANTIATE(float)
#undef MFGPU_INSTANTIATE

}  // namespace mfgpu
