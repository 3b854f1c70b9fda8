// Flag-ordered forward / backward sweeps for the levels of large fronts.
//
// The one-CTA-per-front sweeps (kernels_sweep.cu) serialise a front's whole
// triangular solve on one SM, which leaves a level of a few large fronts (the
// top of a 3D tree, the root of every problem) far below HBM bandwidth.  These
// kernels spread every front of a level over all SMs with one persistent
// cooperative launch and a blocked substitution over 64-row blocks, ordered
// by ready flags instead of grid barriers:
//
//   forward  (src/DE/mf2d.cpp:976-1014, the per-box L11 solve and the
//   boundary update b_bd -= L21 y): a task per 64-row block of a front
//   accumulates L(block, j) y_j over the solved blocks j before it and, for a
//   pivot block, solves y = L_bb^{-1}(b - acc) with the block's explicit
//   inverse and raises the block's flag;
//   backward (src/DE/mf2d.cpp:1016-1054, x_piv = L11^{-T}(y - L21^T x_bd)): a
//   task per 64-column pivot block accumulates L(rows below, block)^T x over
//   the boundary rows and the solved blocks after it, then x = L_bb^{-T}(...)
//   and the flag.
// The inverses (left by the tile kernel; k_diag_inv after the other kernels and
// for loaded factors) take the sequential substitution out of every block; the
// chain of dependent blocks costs one hand-off and two 64 x 64 products per
// block, and the rest of the work (every element of L read once) overlaps it.
//
// W is the front's right-hand-side block (N x nrhs, ld N) in the same
// workspace the per-front kernels use, so the separator gathers between
// levels are unchanged; the solved pivot blocks go to the launch's scratch (Y,
// 64 rows per pivot block and nrhs columns a front), where other tasks read them.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <vector>

#include "device.cuh"

namespace cg = cooperative_groups;

namespace mfgpu {

extern std::atomic<long long> g_launches;

namespace {

constexpr int SB = 64;          // diagonal block of the substitution
constexpr int SCT = 256;        // threads per CTA
constexpr int kMaxSolveCoopFronts = 1024;

__host__ __device__ __forceinline__ int cdiv(int a, int b) { return (a + b - 1) / b; }

// Diagonal-block inverses of the flag-ordered sweeps' pivot blocks: block b of
// front f (rows and columns [64 b, 64 b + kb)) gets Dinv = L_bb^{-1} (lower,
// column-major 64 x 64, zero outside kb x kb) at Dv + dinv_off[f] + b * 8192
// and its transpose right after it.  Column t of the inverse is computed by
// thread t with forward substitution on the block staged in shared memory.
template <class T>
__global__ void __launch_bounds__(SB) k_diag_inv(const int* __restrict__ flist,
                                                 const FrontDev* __restrict__ fr,
                                                 const T* __restrict__ F, T* __restrict__ Dv,
                                                 const int64_t* __restrict__ dinv_off) {
  extern __shared__ __align__(16) unsigned char dsm[];   // Ls and Iv, 2 x 64 x 65
  T(*Ls)[SB + 1] = reinterpret_cast<T(*)[SB + 1]>(dsm);
  T(*Iv)[SB + 1] = Ls + SB;
  const int f = flist[blockIdx.y];
  const FrontDev d = fr[f];
  const int b = blockIdx.x, k = b * SB;
  if (k >= d.n || dinv_off[f] < 0) return;
  const int kb = min(SB, d.n - k), t = threadIdx.x;
  const T* A = F + d.off;
  for (int c = 0; c < kb; c++)
    if (t < kb) Ls[t][c] = t >= c ? A[(k + t) + (int64_t)(k + c) * d.ld] : T(0);
  __syncthreads();
  if (t < kb) {
    for (int i = 0; i < t; i++) Iv[i][t] = T(0);
    for (int i = t; i < kb; i++) {
      T acc = i == t ? T(1) : T(0);
      for (int q = t; q < i; q++) acc = fma(-Ls[i][q], Iv[q][t], acc);
      Iv[i][t] = acc / Ls[i][i];
    }
  }
  __syncthreads();
  T* D = Dv + dinv_off[f] + (int64_t)b * 2 * SB * SB;
  for (int c = 0; c < SB; c++) {
    const int r = t;
    D[r + c * SB] = (r < kb && c < kb) ? Iv[r][c] : T(0);                 // Dinv
    D[SB * SB + r + c * SB] = (r < kb && c < kb) ? Iv[c][r] : T(0);       // Dinv^T
  }
}

// Hand-off of the solved pivot blocks.  A launch starts with its scratch set to
// all ones: a block's flag is negative until its values are visible device-wide,
// and a value holds the all-ones NaN until it is written.  The task of the next
// link of the chain polls the values themselves, with its L in registers, which
// saves the writer's fence, the flag and a second trip through L2; every other
// task waits for the flag, the less often the farther it is from the front's
// chain, so that the hundreds of waiting CTAs do not queue at the flag's L2
// slice.  In a level of one front, where nothing but its chain bounds the sweep,
// that goes for the next kChainTail links: a task takes the block before its last
// dependency while that one is being solved, so that block must not lag either
// (3D 63^3 root in FP32, three refinements' sweeps, 3.49 -> 2.65 ms; levels of
// several fronts lose a tenth to the registers and stay with one).  A wait
// gives up after the error word's poll limit (default kFlowSpin), records error
// code 3 and lets the CTA go on, so the launch always ends.
constexpr int kChainTail = 3;
constexpr unsigned kFlowSpin = 1u << 25;

// One poll of a bounded wait has failed: true to give up.
__device__ __forceinline__ bool flow_give_up(unsigned& it, unsigned lim, DevError* err) {
  if (++it > lim) {
    if (err) atomicCAS(&err->code, 0, 3);
    return true;
  }
  return (it & 1023u) == 0 && err && *(volatile int*)&err->code == 3;   // another CTA gave up
}

// dist: blocks between this task's chain and the flag's.
__device__ __forceinline__ void flow_wait(const int* flag, DevError* err, int dist = 0) {
  const volatile int* f = flag;
  const unsigned lim = wait_limit(err, kFlowSpin);
  unsigned it = 0;
  while (*f < 0) {
    if (flow_give_up(it, lim, err)) break;
    __nanosleep(32 + 32 * min(dist, 32));
  }
  __threadfence();
}

__device__ __forceinline__ void flow_publish(int* flag) {
  __threadfence();
  atomicExch(flag, 1);
}

// The value at p once it is written.
__device__ __forceinline__ bool unwritten(float v) { return __float_as_int(v) == -1; }
__device__ __forceinline__ bool unwritten(double v) { return __double_as_longlong(v) == -1ll; }
template <class T>
__device__ __forceinline__ T flow_value(const T* p, DevError* err) {
  const volatile T* q = p;
  T v = *q;
  if (unwritten(v)) {
    const unsigned lim = wait_limit(err, kFlowSpin);
    unsigned it = 0;
    while (unwritten(v = *q))
      if (flow_give_up(it, lim, err)) return T(0);
  }
  return v;
}
// A value to hand off: never the unwritten pattern (a NaN stays a NaN).
__device__ __forceinline__ float written(float v) { return unwritten(v) ? __int_as_float(0x7fffffff) : v; }
__device__ __forceinline__ double written(double v) {
  return unwritten(v) ? __longlong_as_double(0x7fffffffffffffffll) : v;
}

template <class T>
__device__ __forceinline__ T ldcg(const T* p) {
  return __ldcg(p);
}

// Forward sweep of one level without grid barriers.  Row blocks of every
// front (pivot blocks [64 R, 64 R + 64) of [0, n), then boundary blocks of 64
// rows from n) are tasks, listed R-major across the fronts; CTAs take them
// round-robin.  Task (i, R) accumulates L(rows, block j) y_j over the pivot
// column blocks j before it as their ready flags come up, then a pivot block
// forms y_R = Dinv_R (b_R - acc), writes it to X and to the launch's scratch (Y)
// and raises its flag; a boundary block leaves -acc in W
// for the separator gather.  Everything the last dependency does not change -
// its L block, the block's row of the inverse, the right-hand side - is in
// registers before the task waits for it, so a step of the chain of dependent
// blocks costs one small load, a product and two four-lane reductions.  The
// four lanes of a row (tid & 3) split its 64 columns; a warp's loads of one
// column offset still cover whole 32-byte sectors.  A task waits only on
// tasks listed before it, and a cooperative launch keeps every CTA resident,
// so the sweep cannot stall.
template <class T, int NR, int TAIL>
__global__ void __launch_bounds__(SCT) k_solve_flow_fwd(const int* __restrict__ flist,
                                                        const FrontDev* __restrict__ fr,
                                                        const T* __restrict__ F,
                                                        const int* __restrict__ dofs, T* X,
                                                        int64_t ldx, int nrhs, T* Wb,
                                                        const int64_t* __restrict__ woff,
                                                        const T* __restrict__ Dv,
                                                        const int64_t* __restrict__ dinv_off,
                                                        const int2* __restrict__ tasks, int ntasks,
                                                        const int* __restrict__ flagoff, int* flags,
                                                        T* Yb, DevError* err) {
  constexpr int CH = 4;                       // column blocks per shared-memory round
  __shared__ T ys[CH * SB][NR + 1];           // solved blocks
  __shared__ T ws[SB][NR + 1];                // b_R - acc of the block
  const int tid = threadIdx.x, rl = tid >> 2, g = tid & 3;   // row, column quarter
  for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
    const int2 tk = tasks[t];
    const int i = tk.x, R = tk.y, f = flist[i];
    const FrontDev d = fr[f];
    const T* A = F + d.off;
    T* W = Wb + woff[f] * nrhs;
    const int ldy = cdiv(d.n, SB) * SB;
    T* Y = Yb + (int64_t)flagoff[i] * SB * nrhs;
    const int* dl = dofs + d.dof_off;
    const int* fl = flags + flagoff[i];
    const int nb = cdiv(d.n, SB);
    const bool piv = R < nb;
    const int row0 = piv ? R * SB : d.n + (R - nb) * SB;
    const int rows = min(SB, (piv ? d.n : d.N) - row0);
    const bool live = rl < rows;
    const int jmax = piv ? R : nb;
    const T* Ar = A + row0 + rl;
    T acc[NR];
#pragma unroll
    for (int c = 0; c < NR; c++) acc[c] = T(0);
    // every block but the last TAIL, CH at a time as their flags come up.  These
    // bulk loads go by (row tid & 63, column group tid >> 6): a warp reads 32
    // consecutive rows of a column (coalesced); the sums are handed to the
    // (row, quarter) lanes once, after the loop.
    const int jbulk = max(0, jmax - TAIL);
    const int rl2 = tid & (SB - 1), g2 = tid >> 6;
    const T* Ar2 = A + row0 + rl2;
    T acc2[NR];
#pragma unroll
    for (int c = 0; c < NR; c++) acc2[c] = T(0);
    for (int j0 = 0; j0 < jbulk; j0 += CH) {
      const int jc = min(CH, jbulk - j0);
      __syncthreads();                        // ys of the previous round is consumed
      if (tid == 0)
        for (int jj = 0; jj < jc; jj++) flow_wait(fl + j0 + jj, err, jmax - 1 - j0 - jj);
      __syncthreads();
      for (int idx = tid; idx < jc * SB * nrhs; idx += SCT) {
        const int r = idx % (jc * SB), c = idx / (jc * SB);
        const int col = j0 * SB + r;
        ys[r][c] = col < d.n ? ldcg(Y + col + (int64_t)c * ldy) : T(0);
      }
      __syncthreads();
      if (rl2 < rows) {
        for (int jj = 0; jj < jc; jj++) {
          const int cb = (j0 + jj) * SB + 16 * g2;
          T l[16];
#pragma unroll
          for (int q = 0; q < 16; q++) l[q] = cb + q < d.n ? Ar2[(int64_t)(cb + q) * d.ld] : T(0);
#pragma unroll
          for (int q = 0; q < 16; q++)
#pragma unroll
            for (int c = 0; c < NR; c++) acc2[c] = fma(l[q], ys[jj * SB + 16 * g2 + q][c], acc2[c]);
        }
      }
    }
    // before the last waits: those blocks' L values, this row's quarter of
    // Dinv_R (lower triangular, column-major) and the right-hand side
    T ll[TAIL][16], dv[16], w[NR];
#pragma unroll
    for (int u = 0; u < TAIL; u++)
#pragma unroll
      for (int q = 0; q < 16; q++) {
        const int c = (jbulk + u) * SB + 16 * g + q;
        ll[u][q] = (jbulk + u < jmax && live && c < d.n) ? Ar[(int64_t)c * d.ld] : T(0);
      }
    if (piv) {
      const T* D = Dv + dinv_off[f] + (int64_t)R * 2 * SB * SB;
#pragma unroll
      for (int q = 0; q < 16; q++) dv[q] = 16 * g + q <= rl ? D[rl + (16 * g + q) * SB] : T(0);
#pragma unroll
      for (int c = 0; c < NR; c++)
        w[c] = (live && g == 0 && c < nrhs) ? X[dl[row0 + rl] + (int64_t)c * ldx] : T(0);
    }
    if (jbulk > 0) {                          // hand the sums to the (row, quarter) lanes
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NR; c++) ys[g2 * SB + rl2][c] = acc2[c];
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NR; c++) acc[c] = ys[g * SB + rl][c];
    }
    if (jmax > 0) __syncthreads();            // ys of the previous round is consumed
    // the last blocks, each in its own part of ys, as their values come up
#pragma unroll
    for (int u = 0; u < TAIL; u++) {
      if (jbulk + u < jmax) {
        for (int idx = tid; idx < SB * nrhs; idx += SCT) {
          const int r = idx % SB, c = idx / SB;
          const int col = (jbulk + u) * SB + r;
          ys[u * SB + r][c] = col < d.n ? flow_value(Y + col + (int64_t)c * ldy, err) : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; q++)
#pragma unroll
          for (int c = 0; c < NR; c++) acc[c] = fma(ll[u][q], ys[u * SB + 16 * g + q][c], acc[c]);
      }
    }
    // sum the four quarters of the row
#pragma unroll
    for (int c = 0; c < NR; c++) {
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
    }
    if (!piv) {
      if (live && g == 0)
#pragma unroll
        for (int c = 0; c < NR; c++)
          if (c < nrhs) W[row0 + rl + (int64_t)c * d.N] = -acc[c];
      continue;
    }
    if (g == 0)
#pragma unroll
      for (int c = 0; c < NR; c++) ws[rl][c] = live ? w[c] - acc[c] : T(0);
    __syncthreads();
    // y_R = Dinv_R w_R: each lane its quarter, then the four-lane sum
    T y[NR];
#pragma unroll
    for (int c = 0; c < NR; c++) y[c] = T(0);
#pragma unroll
    for (int q = 0; q < 16; q++)
#pragma unroll
      for (int c = 0; c < NR; c++) y[c] = fma(dv[q], ws[16 * g + q][c], y[c]);
#pragma unroll
    for (int c = 0; c < NR; c++) {
      y[c] += __shfl_xor_sync(0xffffffffu, y[c], 1);
      y[c] += __shfl_xor_sync(0xffffffffu, y[c], 2);
    }
    if (live && g == 0)
#pragma unroll
      for (int c = 0; c < NR; c++)
        if (c < nrhs) {
          Y[row0 + rl + (int64_t)c * ldy] = written(y[c]);
          X[dl[row0 + rl] + (int64_t)c * ldx] = y[c];
        }
    __syncthreads();
    if (tid == 0) flow_publish(flags + flagoff[i] + R);
  }
}

// Backward sweep of one level without grid barriers: x_piv = L11^{-T}
// (y - L21^T x_bd).  Task (i, j), pivot column block j of front i, listed by
// distance from the front's last block: r = sum over the rows below block j of
// L(r, block j)^T x_r, the boundary rows first (x_bd is final on entry), then
// the solved pivot blocks from the last one down as their flags come up (the
// nearest block, the last dependency, with its L values, this column's
// quarter of Dinv_j^T and y_j in registers before the wait); then
// x_j = Dinv_j^T (y_j - r) to X and Y and the flag.  The four lanes of a
// column (tid & 3) split the rows.
template <class T, int NR, int TAIL>
__global__ void __launch_bounds__(SCT) k_solve_flow_bwd(const int* __restrict__ flist,
                                                        const FrontDev* __restrict__ fr,
                                                        const T* __restrict__ F,
                                                        const int* __restrict__ dofs, T* X,
                                                        int64_t ldx, int nrhs, T* Wb,
                                                        const int64_t* __restrict__ woff,
                                                        const T* __restrict__ Dv,
                                                        const int64_t* __restrict__ dinv_off,
                                                        const int2* __restrict__ tasks, int ntasks,
                                                        const int* __restrict__ flagoff, int* flags,
                                                        T* Yb, DevError* err) {
  constexpr int BR = 4;                       // boundary row blocks per shared-memory round
  // Up to four right-hand sides the rows below go warp by column: warp wp
  // takes columns 8 wp .. 8 wp + 7 of the block, its lanes 32 consecutive rows
  // per load (coalesced), and a shuffle reduction sums the lanes at the end.
  constexpr bool CW = NR <= 4;
  __shared__ T xs[BR * SB][NR + 1];
  __shared__ T vs[SB][NR + 1];
  __shared__ T red[CW ? SB : 1][NR + 1];
  const int tid = threadIdx.x, cl = tid >> 2, q = tid & 3;   // column of the block, row quarter
  const int wl = tid & 31, wp = tid >> 5;
  for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
    const int2 tk = tasks[t];
    const int i = tk.x, j = tk.y, f = flist[i];
    const FrontDev d = fr[f];
    const T* A = F + d.off;
    T* W = Wb + woff[f] * nrhs;
    const int ldy = cdiv(d.n, SB) * SB;
    T* Y = Yb + (int64_t)flagoff[i] * SB * nrhs;
    const int* dl = dofs + d.dof_off;
    const int* fl = flags + flagoff[i];
    const int nb = cdiv(d.n, SB), col0 = j * SB, kbj = min(SB, d.n - col0);
    const bool live = cl < kbj;
    const T* Lc = A + (int64_t)(col0 + cl) * d.ld;
    T acc[NR];
#pragma unroll
    for (int c = 0; c < NR; c++) acc[c] = T(0);
    T accw[CW ? 8 : 1][NR];
#pragma unroll
    for (int k = 0; k < (CW ? 8 : 1); k++)
#pragma unroll
      for (int c = 0; c < NR; c++) accw[k][c] = T(0);
    // rows [r0, r0 + nr) (nr <= 64) against xs rows [x0, x0 + nr), every
    // load in flight before the products
    auto chunk = [&](int r0, int nr, int x0) {
      if constexpr (CW) {
        T l0[8], l1[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int c = 8 * wp + k;
          const T* Lk = A + (int64_t)(col0 + c) * d.ld + r0;
          l0[k] = (c < kbj && wl < nr) ? Lk[wl] : T(0);
          l1[k] = (c < kbj && wl + 32 < nr) ? Lk[wl + 32] : T(0);
        }
#pragma unroll
        for (int k = 0; k < 8; k++)
#pragma unroll
          for (int c = 0; c < NR; c++)
            accw[k][c] = fma(l1[k], xs[x0 + wl + 32][c], fma(l0[k], xs[x0 + wl][c], accw[k][c]));
      } else {
        // lanes (cl, q) take rows 16 q .. 16 q + 15
        if (!live) return;
        T l[16];
#pragma unroll
        for (int rr = 0; rr < 16; rr++) l[rr] = 16 * q + rr < nr ? Lc[r0 + 16 * q + rr] : T(0);
#pragma unroll
        for (int rr = 0; rr < 16; rr++)
#pragma unroll
          for (int c = 0; c < NR; c++) acc[c] = fma(l[rr], xs[x0 + 16 * q + rr][c], acc[c]);
      }
    };
    for (int r0 = d.n; r0 < d.N; r0 += BR * SB) {      // boundary rows: x_bd from X
      const int nr = min(BR * SB, d.N - r0);
      __syncthreads();
      for (int idx = tid; idx < BR * SB * nrhs; idx += SCT) {
        const int r = idx % (BR * SB), c = idx / (BR * SB);
        xs[r][c] = r < nr ? X[dl[r0 + r] + (int64_t)c * ldx] : T(0);
      }
      __syncthreads();
#pragma unroll
      for (int s = 0; s < BR; s++)
        if (s * SB < nr) chunk(r0 + s * SB, min(SB, nr - s * SB), s * SB);
    }
    for (int R = nb - 1; R > j + TAIL; R--) {           // solved pivot blocks below but the nearest
      const int r0 = R * SB, nr = min(SB, d.n - r0);
      __syncthreads();
      if (tid == 0) flow_wait(fl + R, err, R - j - 1);
      __syncthreads();
      for (int idx = tid; idx < SB * nrhs; idx += SCT) {
        const int r = idx % SB, c = idx / SB;
        xs[r][c] = r < nr ? ldcg(Y + r0 + r + (int64_t)c * ldy) : T(0);
      }
      __syncthreads();
      chunk(r0, nr, 0);
    }
    if constexpr (CW) {                      // the warps' column sums to the (cl, q) lanes
#pragma unroll
      for (int k = 0; k < 8; k++)
#pragma unroll
        for (int c = 0; c < NR; c++) {
          T v = accw[k][c];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (wl == 0) red[8 * wp + k][c] = v;
        }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NR; c++) acc[c] = (q == 0 && live) ? red[cl][c] : T(0);
    }
    // before the last waits: the L values of blocks j + TAIL .. j + 1, this
    // column's quarter of Dinv_j^T (upper triangular, column-major) and y_j
    T ln[TAIL][16], dt[16], v[NR];
#pragma unroll
    for (int u = 0; u < TAIL; u++)
#pragma unroll
      for (int rr = 0; rr < 16; rr++) {
        const int r = (j + TAIL - u) * SB + 16 * q + rr;
        ln[u][rr] = (live && r < d.n) ? Lc[r] : T(0);
      }
    {
      const T* D = Dv + dinv_off[f] + (int64_t)j * 2 * SB * SB + SB * SB;
#pragma unroll
      for (int p = 0; p < 16; p++) dt[p] = 16 * q + p >= cl ? D[cl + (16 * q + p) * SB] : T(0);
#pragma unroll
      for (int c = 0; c < NR; c++)
        v[c] = (live && q == 0 && c < nrhs) ? X[dl[col0 + cl] + (int64_t)c * ldx] : T(0);
    }
    __syncthreads();                          // xs of the previous round is consumed
    // the nearest blocks, each in its own part of xs, as their values come up
#pragma unroll
    for (int u = 0; u < TAIL; u++) {
      const int rn = (j + TAIL - u) * SB;
      if (rn < d.n) {
        for (int idx = tid; idx < SB * nrhs; idx += SCT) {
          const int r = idx % SB, c = idx / SB;
          xs[u * SB + r][c] = rn + r < d.n ? flow_value(Y + rn + r + (int64_t)c * ldy, err) : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int rr = 0; rr < 16; rr++)
#pragma unroll
          for (int c = 0; c < NR; c++)
            acc[c] = fma(ln[u][rr], xs[u * SB + 16 * q + rr][c], acc[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < NR; c++) {
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
      acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
    }
    __syncthreads();                          // vs of the previous task is consumed
    if (q == 0)
#pragma unroll
      for (int c = 0; c < NR; c++) vs[cl][c] = live ? v[c] - acc[c] : T(0);
    __syncthreads();
    // x_j = Dinv_j^T v: each lane its quarter, then the four-lane sum
    T x[NR];
#pragma unroll
    for (int c = 0; c < NR; c++) x[c] = T(0);
#pragma unroll
    for (int p = 0; p < 16; p++)
#pragma unroll
      for (int c = 0; c < NR; c++) x[c] = fma(dt[p], vs[16 * q + p][c], x[c]);
#pragma unroll
    for (int c = 0; c < NR; c++) {
      x[c] += __shfl_xor_sync(0xffffffffu, x[c], 1);
      x[c] += __shfl_xor_sync(0xffffffffu, x[c], 2);
    }
    if (live && q == 0)
#pragma unroll
      for (int c = 0; c < NR; c++)
        if (c < nrhs) {
          Y[col0 + cl + (int64_t)c * ldy] = written(x[c]);
          X[dl[col0 + cl] + (int64_t)c * ldx] = x[c];
        }
    __syncthreads();
    if (tid == 0) flow_publish(flags + flagoff[i] + j);
  }
}

// ---------------------------------------------------------------------------
// The same sweeps in FP64 on the FP64 tensor cores (mma.sync m8n8k4), eight
// right-hand sides a product, up to NT = 2 products.  Warp w owns rows (columns,
// backward) 8 w .. 8 w + 7 of the task's 64; its operand fragments of L come
// straight from global memory (forward four columns of 64 bytes, backward eight
// columns of 64 bytes a load), so an element of L is loaded once for all
// right-hand sides, and a lane's state is two values per product instead of a
// sum per right-hand side: 16 right-hand sides fit the registers of two CTAs an
// SM where the scalar form spilled with one.  Bound: HBM for many blocks, the
// chain of blocks (flag, 64 x 64 product, inverse product) for one front.
// Against the scalar form: 3D 63^3, 16 right-hand sides, forward 6.05 -> 1.64
// ms, backward 7.65 -> 1.78 ms; 2D 1023^2, 4, 428 -> 192 and 420 -> 228 us; 3D 79
// x 63 x 50, one, 1287 -> 992 and 1181 -> 954 us.
// ---------------------------------------------------------------------------
constexpr int MS = 12;           // row stride of 8 right-hand sides in shared memory (no bank conflicts)

__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// c[t] += A x for 64 columns: a[s] is the lane's fragment of columns 4 s .. + 3,
// x(k, 8 t + rhs) at xs[t * SB * MS + k * MS + rhs], in four chains (a product's
// result takes 65 cycles).
template <int NT>
__device__ __forceinline__ void mma_block(double (&c)[NT][4][2], const double (&a)[16],
                                          const double* xs, int rr, int cc) {
#pragma unroll
  for (int s = 0; s < 16; s++)
#pragma unroll
    for (int t = 0; t < NT; t++)
      mma884(c[t][s & 3], a[s], xs[t * SB * MS + (4 * s + cc) * MS + rr]);
}

template <int NT>
__device__ __forceinline__ void mma_zero(double (&c)[NT][4][2]) {
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int s = 0; s < 4; s++) c[t][s][0] = c[t][s][1] = 0.0;
}
__device__ __forceinline__ double mma_sum(const double (&c)[4][2], int e) {
  return (c[0][e] + c[1][e]) + (c[2][e] + c[3][e]);
}

// x(k, rhs) of 64 rows into shared memory, zero outside [0, nr) x [0, nrhs).
template <int NT, class Get>
__device__ __forceinline__ void stage_rhs(double* xs, int nr, int nrhs, Get&& get) {
  for (int idx = threadIdx.x; idx < SB * 8 * NT; idx += SCT) {
    const int r = idx & (SB - 1), c = idx / SB;
    xs[(c >> 3) * SB * MS + r * MS + (c & 7)] = r < nr && c < nrhs ? get(r, c) : 0.0;
  }
}

template <int NT, int NEAR>
__global__ void __launch_bounds__(SCT, 2)
    k_flow_fwd64(const int* __restrict__ flist, const FrontDev* __restrict__ fr,
                 const double* __restrict__ F, const int* __restrict__ dofs, double* X, int64_t ldx,
                 int nrhs, double* Wb, const int64_t* __restrict__ woff,
                 const double* __restrict__ Dv, const int64_t* __restrict__ dinv_off,
                 const int2* __restrict__ tasks, int ntasks, const int* __restrict__ flagoff,
                 int* flags, double* Yb, DevError* err) {
  __shared__ double xs[2][SB * MS * NT];
  const int tid = threadIdx.x, lane = tid & 31, w8 = 8 * (tid >> 5), rr = lane >> 2, cc = lane & 3;
  for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
    const int2 tk = tasks[t];
    const int i = tk.x, R = tk.y, f = flist[i];
    const FrontDev d = fr[f];
    double* W = Wb + woff[f] * nrhs;
    const int ldy = cdiv(d.n, SB) * SB;
    double* Y = Yb + (int64_t)flagoff[i] * SB * nrhs;
    const int* dl = dofs + d.dof_off;
    const int* fl = flags + flagoff[i];
    const int nb = cdiv(d.n, SB);
    const bool piv = R < nb;
    const int row0 = piv ? R * SB : d.n + (R - nb) * SB;
    const int rows = min(SB, (piv ? d.n : d.N) - row0);
    const int jmax = piv ? R : nb;
    const bool live = w8 + rr < rows;
    // this lane's row, first column cc (dead rows read the block's first row)
    const double* Ar = F + d.off + row0 + (live ? w8 + rr : 0) + (int64_t)min(cc, d.N - 1) * d.ld;
    double acc[NT][4][2];
    mma_zero(acc);
    auto load = [&](double (&a)[16], int j) {   // L(row, block j)
      const int c0 = j * SB + cc;
#pragma unroll
      for (int s = 0; s < 16; s++)
        a[s] = Ar[c0 + 4 * s < d.n ? (int64_t)(j * SB + 4 * s) * d.ld : 0];
      if (j * SB + SB > d.n)
#pragma unroll
        for (int s = 0; s < 16; s++)
          if (c0 + 4 * s >= d.n) a[s] = 0.0;
    };
    auto solved = [&](int j) {
      return [&, j](int r, int c) {
        return j * SB + r < d.n ? ldcg(Y + j * SB + r + (int64_t)c * ldy) : 0.0;
      };
    };
    auto value = [&](int j) {
      return [&, j](int r, int c) {
        return j * SB + r < d.n ? flow_value(Y + j * SB + r + (int64_t)c * ldy, err) : 0.0;
      };
    };
    double a[16], an[16];
    if (jmax > 0) load(a, 0);
    for (int j = 0; j < jmax - 1; j++) {
      if (NEAR > 1 && jmax - 1 - j < NEAR) {
        load(an, j + 1);                        // the next block in flight
        stage_rhs<NT>(xs[j & 1], SB, nrhs, value(j));
      } else {
        if (tid == 0) flow_wait(fl + j, err, jmax - 1 - j);
        __syncthreads();
        stage_rhs<NT>(xs[j & 1], SB, nrhs, solved(j));
        load(an, j + 1);
      }
      __syncthreads();
      mma_block<NT>(acc, a, xs[j & 1], rr, cc);
#pragma unroll
      for (int s = 0; s < 16; s++) a[s] = an[s];
    }
    // before the last wait: the inverse (in `an`) and the right-hand side
    double b[NT][2];
    if (piv) {
      const double* D = Dv + dinv_off[f] + (int64_t)R * 2 * SB * SB + w8 + rr + cc * SB;
#pragma unroll
      for (int s = 0; s < 16; s++) an[s] = D[4 * s * SB];
#pragma unroll
      for (int q = 0; q < NT; q++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int c = 8 * q + 2 * cc + e;
          b[q][e] = live && c < nrhs ? X[dl[row0 + w8 + rr] + (int64_t)c * ldx] : 0.0;
        }
    }
    if (jmax > 0) {
      const int j = jmax - 1;
      __syncthreads();                          // xs of the round before the last is consumed
      stage_rhs<NT>(xs[j & 1], SB, nrhs, value(j));
      __syncthreads();
      mma_block<NT>(acc, a, xs[j & 1], rr, cc);
    }
    if (!piv) {
#pragma unroll
      for (int q = 0; q < NT; q++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int c = 8 * q + 2 * cc + e;
          if (live && c < nrhs)
            W[row0 + w8 + rr + (int64_t)c * d.N] = -mma_sum(acc[q], e);
        }
      __syncthreads();                          // xs is free for the next task
      continue;
    }
    // y_R = Dinv_R (b_R - acc)
    double* ws = xs[jmax & 1];
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
      for (int e = 0; e < 2; e++)
        ws[q * SB * MS + (w8 + rr) * MS + 2 * cc + e] =
            live ? b[q][e] - mma_sum(acc[q], e) : 0.0;
    __syncthreads();
    mma_zero(acc);
    mma_block<NT>(acc, an, ws, rr, cc);
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = 8 * q + 2 * cc + e;
        const double y = mma_sum(acc[q], e);
        if (live && c < nrhs) {
          Y[row0 + w8 + rr + (int64_t)c * ldy] = written(y);
          X[dl[row0 + w8 + rr] + (int64_t)c * ldx] = y;
        }
      }
    __syncthreads();
    if (tid == 0) flow_publish(flags + flagoff[i] + R);
  }
}

// Backward: row blocks of 64 from row 0, so that a fragment takes two rows a
// load (rows 8 s + 2 cc and + 1 of columns rr; the products take them as two
// steps of four rows 8 s + {0, 2, 4, 6} and {1, 3, 5, 7}).  Blocks from the last
// one up: boundary rows from X, pivot rows from Y as their flags come up; the
// block holding the last pivots may hold both.
template <int NT, int NEAR>
__global__ void __launch_bounds__(SCT, 2)
    k_flow_bwd64(const int* __restrict__ flist, const FrontDev* __restrict__ fr,
                 const double* __restrict__ F, const int* __restrict__ dofs, double* X, int64_t ldx,
                 int nrhs, double* Wb, const int64_t* __restrict__ woff,
                 const double* __restrict__ Dv, const int64_t* __restrict__ dinv_off,
                 const int2* __restrict__ tasks, int ntasks, const int* __restrict__ flagoff,
                 int* flags, double* Yb, DevError* err) {
  __shared__ double xs[2][SB * MS * NT];
  const int tid = threadIdx.x, lane = tid & 31, w8 = 8 * (tid >> 5), rr = lane >> 2, cc = lane & 3;
  for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
    const int2 tk = tasks[t];
    const int i = tk.x, j = tk.y, f = flist[i];
    const FrontDev d = fr[f];
    const int ldy = cdiv(d.n, SB) * SB;
    double* Y = Yb + (int64_t)flagoff[i] * SB * nrhs;
    const int* dl = dofs + d.dof_off;
    const int* fl = flags + flagoff[i];
    const int nb = cdiv(d.n, SB), nbr = cdiv(d.N, SB), col0 = j * SB, kbj = min(SB, d.n - col0);
    const bool live = w8 + rr < kbj;
    const double* Lc = F + d.off + (int64_t)(col0 + (live ? w8 + rr : 0)) * d.ld + 2 * cc;
    double acc[NT][4][2];
    mma_zero(acc);
    // rows of block R this task takes: below its pivots, inside the front
    auto load = [&](double (&a)[16], int R) {
      const int r0 = R * SB, lo = R == j ? d.n : r0;
      if (lo == r0 && r0 + SB <= d.N) {
#pragma unroll
        for (int s = 0; s < 8; s++) {
          const double2 v = *reinterpret_cast<const double2*>(Lc + r0 + 8 * s);
          a[2 * s] = v.x;
          a[2 * s + 1] = v.y;
        }
      } else {
#pragma unroll
        for (int s = 0; s < 8; s++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int r = r0 + 8 * s + 2 * cc + e;
            a[2 * s + e] = r >= lo && r < d.N ? Lc[r0 + 8 * s + e] : 0.0;
          }
      }
    };
    auto stage = [&](double* x, int R, bool near) {   // x(row, rhs) in the fragments' row order
      const int r0 = R * SB, lo = R == j ? d.n : r0;
      for (int idx = tid; idx < SB * 8 * NT; idx += SCT) {
        const int r = idx & (SB - 1), c = idx / SB, g = r0 + r;
        double v = 0.0;
        if (g >= lo && g < d.N && c < nrhs)
          v = g >= d.n ? X[dl[g] + (int64_t)c * ldx]
              : near   ? flow_value(Y + g + (int64_t)c * ldy, err)
                       : ldcg(Y + g + (int64_t)c * ldy);
        const int k = (r & ~7) + 4 * (r & 1) + ((r & 7) >> 1);
        x[(c >> 3) * SB * MS + k * MS + (c & 7)] = v;
      }
    };
    // last block this task reads last: the one after it, or its own boundary rows
    const int Rlast = (d.n & (SB - 1)) && j == nb - 1 && d.N > d.n ? j : j + 1;
    double a[16], an[16];
    if (Rlast < nbr) load(a, nbr - 1);
    for (int R = nbr - 1; R > Rlast; R--) {
      if (NEAR > 1 && R - j <= NEAR) {
        load(an, R - 1);                        // the next block in flight
        stage(xs[R & 1], R, true);
      } else {
        if (R < nb) {
          if (tid == 0) flow_wait(fl + R, err, R - j - 1);
          __syncthreads();
        }
        stage(xs[R & 1], R, false);
        load(an, R - 1);
      }
      __syncthreads();
      mma_block<NT>(acc, a, xs[R & 1], rr, cc);
#pragma unroll
      for (int s = 0; s < 16; s++) a[s] = an[s];
    }
    // before the last wait: the inverse's transpose (in `an`) and y_j
    const double* D = Dv + dinv_off[f] + (int64_t)j * 2 * SB * SB + SB * SB + w8 + rr + cc * SB;
#pragma unroll
    for (int s = 0; s < 16; s++) an[s] = D[4 * s * SB];
    double b[NT][2];
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = 8 * q + 2 * cc + e;
        b[q][e] = live && c < nrhs ? X[dl[col0 + w8 + rr] + (int64_t)c * ldx] : 0.0;
      }
    if (Rlast < nbr) {
      stage(xs[Rlast & 1], Rlast, true);
      __syncthreads();
      mma_block<NT>(acc, a, xs[Rlast & 1], rr, cc);
    }
    // x_j = Dinv_j^T (y_j - acc)
    double* ws = xs[(Rlast + 1) & 1];
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
      for (int e = 0; e < 2; e++)
        ws[q * SB * MS + (w8 + rr) * MS + 2 * cc + e] =
            live ? b[q][e] - mma_sum(acc[q], e) : 0.0;
    __syncthreads();
    mma_zero(acc);
    mma_block<NT>(acc, an, ws, rr, cc);
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = 8 * q + 2 * cc + e;
        const double x = mma_sum(acc[q], e);
        if (live && c < nrhs) {
          Y[col0 + w8 + rr + (int64_t)c * ldy] = written(x);
          X[dl[col0 + w8 + rr] + (int64_t)c * ldx] = x;
        }
      }
    __syncthreads();
    if (tid == 0) flow_publish(flags + flagoff[i] + j);
  }
}

// Persistent grid: every CTA the SMs hold at once (a cooperative launch checks
// that they are all resident, which the flag waits rely on).  As many CTAs as
// fit, so that the row blocks of a long chain (a root front has hundreds) each
// get their own CTA from the start and accumulate the solved blocks as they
// come, instead of queueing behind other tasks of the same CTA.
int flowGrid(const void* kern) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, SCT, 0);
  return sms * std::max(1, per);
}

size_t flag_bytes(int nflags) { return ((size_t)std::max(1, nflags) * sizeof(int) + 15) & ~(size_t)15; }

// Kernels of a direction and bound of the right-hand-side count: the scalar
// form in FP32, the tensor-core form in FP64.
template <class T, int NR, int TAIL>
struct FlowKernels {
  static const void* fwd() { return (const void*)k_solve_flow_fwd<T, NR, TAIL>; }
  static const void* bwd() { return (const void*)k_solve_flow_bwd<T, NR, TAIL>; }
};
template <int NR, int TAIL>
struct FlowKernels<double, NR, TAIL> {
  static const void* fwd() { return (const void*)k_flow_fwd64<NR / 8, TAIL>; }
  static const void* bwd() { return (const void*)k_flow_bwd64<NR / 8, TAIL>; }
};

template <class T, int NR, int TAIL>
cudaError_t launchFlowSolve(bool fwd, const int* flist, const FrontDev* fr, const T* F,
                            const int* dofs, T* X, int64_t ldx, int nrhs, T* W,
                            const int64_t* woff, const T* Dv, const int64_t* dinv_off,
                            const int2* tasks, int ntasks, const int* flagoff, int* flags,
                            int nflags, DevError* err, cudaStream_t st) {
  // flags and, from a 16-byte boundary behind them, the solved blocks
  const size_t fb = flag_bytes(nflags);
  T* Y = reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(flags) + fb);
  cudaError_t me = cudaMemsetAsync(flags, 0xff, fb + (size_t)nflags * SB * nrhs * sizeof(T), st);
  if (me != cudaSuccess) return me;
  using K = FlowKernels<T, NR, TAIL>;
  static const int gf = flowGrid(K::fwd());   // thread-safe one-time set-up
  static const int gb = flowGrid(K::bwd());
  const int grid = std::max(1, std::min(fwd ? gf : gb, ntasks));
  void* args[] = {(void*)&flist, (void*)&fr,    (void*)&F,      (void*)&dofs,    (void*)&X,
                  (void*)&ldx,   (void*)&nrhs,  (void*)&W,      (void*)&woff,    (void*)&Dv,
                  (void*)&dinv_off, (void*)&tasks, (void*)&ntasks, (void*)&flagoff, (void*)&flags,
                  (void*)&Y,     (void*)&err};
  g_launches++;
  return cudaLaunchCooperativeKernel(fwd ? K::fwd() : K::bwd(), dim3(grid), dim3(SCT), args, 0, st);
}

}  // namespace

int solve_coop_max_fronts() { return kMaxSolveCoopFronts; }

size_t flow_scratch_bytes(int nflags, int elem_bytes) {
  return flag_bytes(nflags) + (size_t)nflags * SB * 16 * elem_bytes;
}

void flow_tasks(const std::vector<int>& n, const std::vector<int>& N, std::vector<int>& fwd,
                std::vector<int>& bwd, std::vector<int>& flagoff) {
  const int nf = (int)n.size();
  std::vector<int> nb(nf), rb(nf);
  int maxrb = 0, maxnb = 0;
  flagoff.assign(nf + 1, 0);
  for (int i = 0; i < nf; i++) {
    nb[i] = cdiv(n[i], SB);
    rb[i] = nb[i] + cdiv(N[i] - n[i], SB);
    maxrb = std::max(maxrb, rb[i]);
    maxnb = std::max(maxnb, nb[i]);
    flagoff[i + 1] = flagoff[i] + nb[i];
  }
  fwd.clear();
  bwd.clear();
  for (int R = 0; R < maxrb; R++)
    for (int i = 0; i < nf; i++)
      if (R < rb[i]) fwd.insert(fwd.end(), {i, R});
  for (int t = 0; t < maxnb; t++)
    for (int i = 0; i < nf; i++)
      if (t < nb[i]) bwd.insert(bwd.end(), {i, nb[i] - 1 - t});
}

template <class T>
cudaError_t launch_solve_flow(bool forward, const int* flist, const FrontDev* fr, const T* F,
                              const int* dofs, T* X, int64_t ldx, int nrhs, T* W,
                              const int64_t* woff, const T* Dv, const int64_t* dinv_off,
                              const int* tasks, int ntasks, const int* flagoff, int* flags,
                              int nflags, bool chain, DevError* err, cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  if (nrhs > 16) return cudaErrorInvalidValue;
  const int2* tk = reinterpret_cast<const int2*>(tasks);
#define MFGPU_FLOW(NRV, TAIL)                                                                     \
  return launchFlowSolve<T, NRV, TAIL>(forward, flist, fr, F, dofs, X, ldx, nrhs, W, woff, Dv,      \
                                       dinv_off, tk, ntasks, flagoff, flags, nflags, err, st)
  if constexpr (sizeof(T) == sizeof(float)) {
    if (nrhs == 1 && chain) MFGPU_FLOW(1, kChainTail);
    if (nrhs == 1) MFGPU_FLOW(1, 1);
    if (nrhs <= 4 && chain) MFGPU_FLOW(4, kChainTail);
    if (nrhs <= 4) MFGPU_FLOW(4, 1);
    if (nrhs <= 8) MFGPU_FLOW(8, 1);
    MFGPU_FLOW(16, 1);
  } else {
    if (nrhs <= 8 && chain) MFGPU_FLOW(8, kChainTail);
    if (nrhs <= 8) MFGPU_FLOW(8, 1);
    if (chain) MFGPU_FLOW(16, kChainTail);
    MFGPU_FLOW(16, 1);
  }
#undef MFGPU_FLOW
}

template <class T>
void launch_diag_inv(const int* flist, int nf, int maxn, const FrontDev* fr, const T* F, T* Dv,
                     const int64_t* dinv_off, cudaStream_t st) {
  if (nf <= 0 || maxn <= 0) return;
  const int sm = 2 * SB * (SB + 1) * (int)sizeof(T);
  static const bool attr = (cudaFuncSetAttribute(k_diag_inv<T>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, sm),
                            true);
  (void)attr;
  k_diag_inv<T><<<dim3(cdiv(maxn, SB), nf), SB, sm, st>>>(flist, fr, F, Dv, dinv_off);
  g_launches++;
}

template cudaError_t launch_solve_flow<double>(bool, const int*, const FrontDev*, const double*,
                                               const int*, double*, int64_t, int, double*,
                                               const int64_t*, const double*, const int64_t*,
                                               const int*, int, const int*, int*, int, bool,
                                               DevError*, cudaStream_t);
template cudaError_t launch_solve_flow<float>(bool, const int*, const FrontDev*, const float*,
                                              const int*, float*, int64_t, int, float*,
                                              const int64_t*, const float*, const int64_t*,
                                              const int*, int, const int*, int*, int, bool,
                                              DevError*, cudaStream_t);
template void launch_diag_inv<double>(const int*, int, int, const FrontDev*, const double*, double*,
                                      const int64_t*, cudaStream_t);
template void launch_diag_inv<float>(const int*, int, int, const FrontDev*, const float*, float*,
                                     const int64_t*, cudaStream_t);

}  // namespace mfgpu
