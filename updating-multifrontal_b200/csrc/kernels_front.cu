// Front kernels for both precisions (T = double for the FP64 path, T = float
// for the mixed-precision factorization): front / separator assembly from
// task tables, partial Cholesky of every front of a level fused per front (or in
// one cooperative launch, FP32 sub-panels only), the separator gather of the
// sweeps and the apply of LU fronts.  FP64 tiles use the FP64 tensor cores
// (mma.sync m8n8k4); FP32 tiles use CUDA-core FMAs with the same fragment layout.
//
// Fronts are column-major with leading dimension ld; only the lower triangle
// is read or written.  After the partial factorization of a front with n
// pivots and m boundary rows:
//   rows/cols [0,n) x [0,n)  hold L11 (A22 = L11 L11^T),
//   rows [n,N) x cols [0,n)  hold L21 (= A12 L11^{-T}),
//   rows/cols [n,N)^2        hold the update matrix: Schur complement
//                            S = -L21 L21^T on the separator diagonal blocks,
//                            A11 + S elsewhere (the reference's A11post).
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <vector>

#include "device.cuh"

namespace cg = cooperative_groups;

namespace mfgpu {

std::atomic<long long> g_launches{0};

namespace {

// Assembly, one warp per 32 x 32 tile of a task, kTaskWarps tiles per CTA.
// Bound: HBM writes (every element of the fronts) for the leaf levels, the
// chain of dependent loads (tile -> task -> DOFs -> CSR rows) for small levels.
// So a tile names its task and place (no search), the rows of a tile are spread
// over the lanes, block moves keep kTaskUnroll columns in flight, and launches
// without transposed copies take no shared memory (twice the warps an SM).
// Sparse tiles: a lane holds its row's CSR entries (eight at a time) in
// registers and matches them against the tile's columns, broadcast one by one,
// so each column is written as it is found.  Against a serial search through
// tile prefixes, a pass over all rows with every lane reading the same entries,
// and four launches a level: 2D 1023^2 leaves 2.20 -> 0.78 ms, a 2D 127^2 step's
// assemblies 549 -> 184 us.
constexpr int kTaskWarps = 4;
constexpr int kTaskUnroll = 8;

template <class T, bool STAGED>
__global__ void __launch_bounds__(32 * kTaskWarps) k_tasks(const Task* __restrict__ tasks,
                                                           const int2* __restrict__ tiles,
                                                           int64_t ntiles, T* __restrict__ F,
                                                           T* __restrict__ SA,
                                                           const int* __restrict__ rp,
                                                           const int* __restrict__ ci,
                                                           const double* __restrict__ va,
                                                           const int* __restrict__ dofs,
                                                           const double* __restrict__ scale) {
  __shared__ T sm[STAGED ? kTaskWarps : 1][STAGED ? kTaskTile : 1][kTaskTile + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t tile = ((int64_t)blockIdx.x + (int64_t)blockIdx.y * gridDim.x) * kTaskWarps + w;
  if (tile >= ntiles) return;
  const int2 at = tiles[tile];
  const int t = at.x;
  const Task Tk = tasks[t];
  const int i0 = (at.y & 0xffff) * kTaskTile, j0 = (int)((unsigned)at.y >> 16) * kTaskTile;
  T* dst = (Tk.dst_arena == AR_FRONT ? F : SA) + Tk.dst_off;
  const T* src = (Tk.src_arena == AR_FRONT ? F : SA) + Tk.src_off;
  const int rows = min(kTaskTile, Tk.rows - i0), cols = min(kTaskTile, Tk.cols - j0);
  T(*tb)[kTaskTile + 1] = sm[STAGED ? w : 0];
  const int i = i0 + lane;   // this lane's row of the tile in the column-major writes
  // first column this lane does not write (its row's diagonal in lower tiles)
  const int jend = lane >= rows ? 0 : Tk.lower ? min(cols, i - j0 + 1) : cols;
  T* d = dst + i + (int64_t)j0 * Tk.dst_ld;
  if (STAGED && Tk.kind == TK_COPY && Tk.trans) {
    // dst(i, j) = src[j + i*ld]: read src rows with lanes along j, write dst
    // columns with lanes along i, through the warp's shared-memory tile
    const T* sr = src + j0 + lane + (int64_t)i0 * Tk.src_ld;
    for (int ii = 0; ii < rows; ii += kTaskUnroll) {
      T v[kTaskUnroll];
#pragma unroll
      for (int q = 0; q < kTaskUnroll; q++)
        v[q] = lane < cols && ii + q < rows ? sr[(int64_t)(ii + q) * Tk.src_ld] : T(0);
#pragma unroll
      for (int q = 0; q < kTaskUnroll; q++) tb[ii + q][lane] = v[q];
    }
    __syncwarp();
#pragma unroll 4
    for (int jj = 0; jj < jend; jj++) d[(int64_t)jj * Tk.dst_ld] = tb[lane][jj];
    return;
  }
  if (Tk.kind == TK_SPARSE) {
    // A(r, c) for the tile (Sparse::operator(), src/LinAlg/sparse.cpp:80-92).
    // Values of this task's matrix: src_off is the element offset of its CSR
    // values (0 but for the serving loop's batches of several matrices).
    va += Tk.src_off;
    const int cj = lane < cols ? dofs[Tk.col_dof + j0 + lane] : -1;
    const int rl = lane < rows ? dofs[Tk.row_dof + i] : 0;
    const double sc = (scale && lane < cols) ? scale[cj] : 1.0;
    const double sr = (scale && lane < rows) ? scale[rl] : 1.0;
    const int p0 = lane < rows ? rp[rl] : 0, p1 = lane < rows ? rp[rl + 1] : 0;
    const bool lng = STAGED && __any_sync(0xffffffffu, p1 - p0 > 8);   // rows of wider stencils
    if (lng)
      for (int jj = 0; jj < cols; jj++) tb[lane][jj] = T(0);
    for (int pb = p0;; pb += 8) {
      int c[8];
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) c[q] = pb + q < p1 ? ci[pb + q] : -2;
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = pb + q < p1 ? va[pb + q] : 0.0;
      for (int jj = 0; jj < cols; jj++) {
        const int cc = __shfl_sync(0xffffffffu, cj, jj);
        const double scj = __shfl_sync(0xffffffffu, sc, jj);
        double x = 0.0;
        bool hit = false;
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (c[q] == cc) {
            x = v[q];
            hit = true;
          }
        if (scale) x = x * sr * scj;   // symmetric diagonal scaling
        if (lng) {
          if (hit) tb[lane][jj] = (T)x;
        } else if (jj < jend) {
          d[(int64_t)jj * Tk.dst_ld] = (T)x;
        }
      }
      if (!lng || !__any_sync(0xffffffffu, pb + 8 < p1)) break;
    }
    if (lng)
      for (int jj = 0; jj < jend; jj++) d[(int64_t)jj * Tk.dst_ld] = tb[lane][jj];
    return;
  }
  if (Tk.kind == TK_ZERO) {
#pragma unroll 8
    for (int jj = 0; jj < jend; jj++) d[(int64_t)jj * Tk.dst_ld] = T(0);
    return;
  }
  const T* s0 = src + i + (int64_t)j0 * Tk.src_ld;
  if (Tk.kind == TK_COPY) {
    for (int jj = 0; jj < jend; jj += kTaskUnroll) {
      T v[kTaskUnroll];
#pragma unroll
      for (int q = 0; q < kTaskUnroll; q++)
        if (jj + q < jend) v[q] = s0[(int64_t)(jj + q) * Tk.src_ld];
#pragma unroll
      for (int q = 0; q < kTaskUnroll; q++)
        if (jj + q < jend) d[(int64_t)(jj + q) * Tk.dst_ld] = v[q];
    }
    return;
  }
  // TK_ADD, listed in pairs (the second has no tiles of its own):
  // dst = (dst + box 0's block) + box 1's block, the reference's order
  const Task T1 = tasks[t + 1];
  const T* s1 = (T1.src_arena == AR_FRONT ? F : SA) + T1.src_off + i + (int64_t)j0 * T1.src_ld;
  for (int jj = 0; jj < jend; jj += kTaskUnroll) {
    T v[kTaskUnroll], a[kTaskUnroll], c[kTaskUnroll];
#pragma unroll
    for (int q = 0; q < kTaskUnroll; q++)
      if (jj + q < jend) {
        v[q] = d[(int64_t)(jj + q) * Tk.dst_ld];
        a[q] = s0[(int64_t)(jj + q) * Tk.src_ld];
        c[q] = s1[(int64_t)(jj + q) * T1.src_ld];
      }
#pragma unroll
    for (int q = 0; q < kTaskUnroll; q++)
      if (jj + q < jend) d[(int64_t)(jj + q) * Tk.dst_ld] = (v[q] + a[q]) + c[q];
  }
}

// ---------------------------------------------------------------------------
// Partial Cholesky building blocks.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void report(DevError* err, int code, int front, int col) {
  if (atomicCAS(&err->code, 0, code) == 0) {
    err->front = front;
    err->col = col;
  }
}

constexpr unsigned kFull = 0xffffffffu;

// Cholesky of a kb x kb (kb <= 32) SPD block held one row per lane (row[t] is
// element (lane, t), lower triangle).  Each pivot is scaled by 1/sqrt(d) from
// rsqrt(d), so the column scaling is a multiply; lane j keeps 1/L(j,j) in
// `inv`.  Returns the first failing column or -1.
__device__ __forceinline__ int warp_potrf32(double (&row)[kPanel], int lane, int kb, double& inv) {
  int bad = -1;
  inv = 1.0;
#pragma unroll
  for (int j = 0; j < kPanel; j++) {
    if (j < kb) {
      double djj = __shfl_sync(kFull, row[j], j);
      if (!(djj > 0.0)) {               // non-positive or NaN pivot: not SPD
        if (bad < 0) bad = j;
        djj = 1.0;
      }
      const double r = rsqrt(djj);
      if (lane == j) {
        row[j] = djj * r;
        inv = r;
      } else if (lane > j) {
        row[j] = row[j] * r;
      }
#pragma unroll
      for (int l = j + 1; l < kPanel; l++) {
        const double llj = __shfl_sync(kFull, row[j], l);
        if (lane >= l && l < kb) row[l] -= row[j] * llj;
      }
    }
  }
  return bad;
}

// Load the kb x kb diagonal block at (k, k) of A into one row per lane, factor
// it, write it back to A and to Ds / Dinv (shared).  Called by one full warp.
__device__ __forceinline__ void warp_factor_diag(double* A, int64_t ld, int k, int kb,
                                                 double (*Ds)[kPanel + 1], double* Dinv,
                                                 DevError* err, int f) {
  const int lane = threadIdx.x & 31;
  double row[kPanel];
#pragma unroll
  for (int t = 0; t < kPanel; t++)
    row[t] = (lane < kb && t < kb && t <= lane) ? A[(k + lane) + (int64_t)(k + t) * ld] : 0.0;
  double inv;
  const int bad = warp_potrf32(row, lane, kb, inv);
  if (bad >= 0 && lane == 0) report(err, 1, f, k + bad);
#pragma unroll
  for (int t = 0; t < kPanel; t++) {
    if (lane < kb && t < kb && t <= lane) A[(k + lane) + (int64_t)(k + t) * ld] = row[t];
    Ds[lane][t] = row[t];
  }
  Dinv[lane] = inv;
}

// Left-looking Cholesky of the kb x kb diagonal block at (k, k) of A by one
// warp, followed by the explicit inverse of the factor.  Lane i keeps row i in
// registers; column j is finished with a dot product against row j (published
// in Ls) and a reciprocal square root, so the dependent chain per column is
// short.  On exit A and Ls hold L, Li holds L^{-1} (lower, stride kLi) and
// Dinv the reciprocals of the diagonal.  Called by one full warp.
constexpr int kLi = 36;
__device__ __forceinline__ double rsq(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsq(float x) { return rsqrtf(x); }

template <class T>
__device__ void warp_factor_inv(T* A, int64_t ld, int k, int kb, T (*Ls)[kPanel + 1],
                                T* Li, T* Dinv, DevError* err, int f) {
  const int lane = threadIdx.x & 31;
  T row[kPanel];
#pragma unroll
  for (int t = 0; t < kPanel; t++)
    row[t] = (lane < kb && t < kb && t <= lane) ? A[(k + lane) + (int64_t)(k + t) * ld] : T(0);
  int bad = -1;
#pragma unroll
  for (int j = 0; j < kPanel; j++) {
    if (j < kb) {
      T s0 = row[j], s1 = T(0), s2 = T(0), s3 = T(0);
#pragma unroll
      for (int t = 0; t < j; t++) {
        const T l = Ls[j][t];
        if ((t & 3) == 0) s0 -= row[t] * l;
        else if ((t & 3) == 1) s1 -= row[t] * l;
        else if ((t & 3) == 2) s2 -= row[t] * l;
        else s3 -= row[t] * l;
      }
      const T sv = (s0 + s1) + (s2 + s3);
      T piv = __shfl_sync(kFull, sv, j);
      if (!(piv > T(0))) {                // non-positive or NaN pivot: not SPD
        if (bad < 0) bad = j;
        piv = T(1);
      }
      const T r = rsq(piv);
      row[j] = lane == j ? piv * r : (lane > j ? sv * r : T(0));
      if (lane >= j && lane < kb) Ls[lane][j] = row[j];
      if (lane == j) Dinv[j] = r;
      __syncwarp();
    }
  }
  if (bad >= 0 && lane == 0) report(err, 1, f, k + bad);
#pragma unroll
  for (int t = 0; t < kPanel; t++)
    if (lane < kb && t < kb && t <= lane) A[(k + lane) + (int64_t)(k + t) * ld] = row[t];
  // inverse: lane c computes column c, x_i = -(sum_{c<=t<i} L(i,t) x_t) / L(i,i)
  T x[kPanel];
#pragma unroll
  for (int i = 0; i < kPanel; i++) {
    T v = T(0);
    if (i < kb) {
      T s0 = T(0), s1 = T(0), s2 = T(0), s3 = T(0);
#pragma unroll
      for (int t = 0; t < i; t++) {
        const T l = Ls[i][t];
        const T xt = t >= lane ? x[t] : T(0);
        if ((t & 3) == 0) s0 += l * xt;
        else if ((t & 3) == 1) s1 += l * xt;
        else if ((t & 3) == 2) s2 += l * xt;
        else s3 += l * xt;
      }
      const T di = Dinv[i];
      v = i == lane ? di : (i > lane ? -((s0 + s1) + (s2 + s3)) * di : T(0));
    }
    x[i] = v;
    Li[i * kLi + lane] = v;
  }
  __syncwarp();
}

// One FP64 tensor-core MMA: D(8x8) += A(8x4) B(4x8).  Fragments: a = A(lane/4,
// lane%4), b = B(lane%4, lane/4), c/d = C(lane/4, 2*(lane%4) + {0,1}).
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

constexpr int kPS = 36;   // shared-memory row stride (doubles) of a staged panel

// acc(32x32) += X[I0:I0+32, 0:kk] * Y[J0:J0+32, 0:kk]^T for row-major operands
// in shared memory (strides sx, sy; rows padded with zeros to the tile edge).
// Lane (rr = lane/4, cc = lane%4) owns rows I0 + 8a + rr and columns
// J0 + 8b + 2cc + q of the tile: the FP64 tensor-core (m8n8k4) accumulator
// layout, which the FP32 version reproduces with CUDA-core FMAs.
__device__ __forceinline__ void warp_gemm_nt_acc(const double* X, int sx, int I0, const double* Y,
                                                 int sy, int J0, int kk, int lane,
                                                 double (&acc)[4][4][2]) {
  const int rr = lane >> 2, cc = lane & 3;
  for (int k = 0; k < kk; k += 4) {
    double fa[4], fb[4];
#pragma unroll
    for (int a = 0; a < 4; a++) fa[a] = X[(I0 + 8 * a + rr) * sx + k + cc];
#pragma unroll
    for (int b = 0; b < 4; b++) fb[b] = Y[(J0 + 8 * b + rr) * sy + k + cc];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) dmma(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
  }
}

__device__ __forceinline__ void warp_gemm_nt_acc(const float* X, int sx, int I0, const float* Y,
                                                 int sy, int J0, int kk, int lane,
                                                 float (&acc)[4][4][2]) {
  const int rr = lane >> 2, cc = lane & 3;
  for (int k = 0; k < kk; k++) {
    float fa[4], fb[4][2];
#pragma unroll
    for (int a = 0; a < 4; a++) fa[a] = X[(I0 + 8 * a + rr) * sx + k];
#pragma unroll
    for (int b = 0; b < 4; b++) {
      fb[b][0] = Y[(J0 + 8 * b + 2 * cc) * sy + k];
      fb[b][1] = Y[(J0 + 8 * b + 2 * cc + 1) * sy + k];
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) {
        acc[a][b][0] = fmaf(fa[a], fb[b][0], acc[a][b][0]);
        acc[a][b][1] = fmaf(fa[a], fb[b][1], acc[a][b][1]);
      }
  }
}

template <class T>
__device__ __forceinline__ void acc_zero(T (&acc)[4][4][2]) {
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) acc[a][b][0] = acc[a][b][1] = T(0);
}

template <class T>
__device__ __forceinline__ void warp_gemm_nt(const T* X, int sx, int I0, const T* Y, int sy, int J0,
                                             int kk, int lane, T (&acc)[4][4][2]) {
  acc_zero(acc);
  warp_gemm_nt_acc(X, sx, I0, Y, sy, J0, kk, lane, acc);
}

template <class T>
__device__ __forceinline__ void warp_syrk_tile(const T* P, int I0, int J0, int kk, int lane,
                                               T (&acc)[4][4][2]) {
  warp_gemm_nt(P, kPS, I0, P, kPS, J0, kk, lane, acc);
}

// Panel triangular solve of the 32-row block R0 of P in place with the explicit
// inverse: P(R0 block) <- P(R0 block) Li^T; rows < M are also written to A at
// (r0 + row, k + col), cols < kb.
template <class T>
__device__ __forceinline__ void warp_trsm_block(T* P, int R0, const T* Li, int kb, T* A, int64_t ld,
                                                int r0, int k, int M, int lane) {
  T acc[4][4][2];
  warp_gemm_nt(P, kPS, R0, Li, kLi, 0, (kb + 3) & ~3, lane, acc);
  __syncwarp();
  const int rr = lane >> 2, cc = lane & 3;
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int row = R0 + 8 * a + rr, col = 8 * b + 2 * cc + q;
        P[row * kPS + col] = acc[a][b][q];
        if (row < M && col < kb) A[(r0 + row) + (int64_t)(k + col) * ld] = acc[a][b][q];
      }
}

// C(r0 + i, r0 + j) -= acc for the tile at (I0, J0); lower triangle and i, j < M.
template <class T>
__device__ __forceinline__ void warp_tile_sub(T* A, int64_t ld, int r0, int M, int I0, int J0,
                                              int lane, const T (&acc)[4][4][2]) {
  const int rr = lane >> 2, cc = lane & 3;
  // all loads first, then all stores, so the accesses overlap
  T cur[4][4][2];
#pragma unroll
  for (int b = 0; b < 4; b++)
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int j = J0 + 8 * b + 2 * cc + q;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int i = I0 + 8 * a + rr;
        cur[a][b][q] = (i < M && j < M && i >= j) ? A[(r0 + i) + (int64_t)(r0 + j) * ld] : T(0);
      }
    }
#pragma unroll
  for (int b = 0; b < 4; b++)
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int j = J0 + 8 * b + 2 * cc + q;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int i = I0 + 8 * a + rr;
        if (i < M && j < M && i >= j) A[(r0 + i) + (int64_t)(r0 + j) * ld] = cur[a][b][q] - acc[a][b][q];
      }
    }
}

__device__ __forceinline__ void tri_index(int t, int& I, int& J) {
  I = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while (I * (I + 1) / 2 > t) I--;
  while ((I + 1) * (I + 2) / 2 <= t) I++;
  J = t - I * (I + 1) / 2;
}

// Triangular solve of one row against the factored diagonal block:
// x(0:kb) <- x L^{-T}, with the reciprocals of the diagonal in Dinv.
__device__ __forceinline__ void row_trsm(double (&x)[kPanel], const double (*L)[kPanel + 1],
                                         const double* Dinv, int kb) {
#pragma unroll
  for (int j = 0; j < kPanel; j++) {
    if (j < kb) {
      double s = x[j];
#pragma unroll
      for (int t = 0; t < j; t++) s -= x[t] * L[j][t];
      x[j] = s * Dinv[j];
    }
  }
}

// ---------------------------------------------------------------------------
// Fused partial factorization, one CTA per front (small_front_fits).
// The panel of each step is staged in shared memory for the tensor-core update.
// ---------------------------------------------------------------------------
template <class T, int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_front_small(const int* __restrict__ flist,
                                                     const FrontDev* __restrict__ fr,
                                                     T* __restrict__ F, DevError* err) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* Psm = reinterpret_cast<T*>(smraw);
  __shared__ T Ls[kPanel][kPanel + 1];
  __shared__ T Li[kPanel * kLi];
  __shared__ T Dinv[kPanel];
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  T* A = F + d.off;
  const int64_t ld = d.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (warp == 0) warp_factor_inv(A, ld, 0, min(kPanel, d.n), Ls, Li, Dinv, err, f);
  for (int k = 0; k < d.n; k += kPanel) {
    const int kb = min(kPanel, d.n - k);
    const int r0 = k + kb;
    const int M = d.N - r0;
    const int Mp = (M + 31) & ~31;
    // stage the panel rows below the diagonal block (zero padded)
    for (int idx = tid; idx < Mp * kPanel; idx += blockDim.x) {
      const int rr = idx % Mp, t = idx / Mp;
      Psm[rr * kPS + t] = (rr < M && t < kb) ? A[(r0 + rr) + (int64_t)(k + t) * ld] : T(0);
    }
    __syncthreads();
    for (int R0 = warp * 32; R0 < Mp; R0 += NT) warp_trsm_block(Psm, R0, Li, kb, A, ld, r0, k, M, lane);
    __syncthreads();
    const int TT = Mp >> 5;
    const int ntile = TT * (TT + 1) / 2;
    const int kk = (kb + 3) & ~3;
    if (warp == 0) {
      // lookahead: tile (0, 0) holds the next diagonal block; update it, then
      // factor it while the other warps finish the trailing update
      if (ntile > 0) {
        T acc[4][4][2];
        warp_syrk_tile(Psm, 0, 0, kk, lane, acc);
        warp_tile_sub(A, ld, r0, M, 0, 0, lane, acc);
      }
      __syncwarp();
      if (r0 < d.n) warp_factor_inv(A, ld, r0, min(kPanel, d.n - r0), Ls, Li, Dinv, err, f);
    } else {
      for (int t = warp; t < ntile; t += NT / 32 - 1) {   // the other warps take tiles 1, 2, ...
        int I, J;
        tri_index(t, I, J);
        T acc[4][4][2];
        warp_syrk_tile(Psm, I * 32, J * 32, kk, lane, acc);
        warp_tile_sub(A, ld, r0, M, I * 32, J * 32, lane, acc);
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Stepped path for large fronts: one launch per kernel per panel step, all
// fronts of the level in each launch.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(32) k_potrf(const int* __restrict__ flist,
                                              const FrontDev* __restrict__ fr,
                                              double* __restrict__ F, int k, DevError* err) {
  __shared__ double Ds[kPanel][kPanel + 1];
  __shared__ double Dinv[kPanel];
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  if (k >= d.n) return;
  warp_factor_diag(F + d.off, d.ld, k, min(kPanel, d.n - k), Ds, Dinv, err, f);
}

// Rows below the diagonal block: X = A(r, k:k+kb) L_kk^{-T}.
__global__ void __launch_bounds__(128) k_trsm(const int* __restrict__ flist,
                                              const FrontDev* __restrict__ fr,
                                              double* __restrict__ F, int k) {
  const int f = flist[blockIdx.y];
  const FrontDev d = fr[f];
  if (k >= d.n) return;
  const int kb = min(kPanel, d.n - k);
  __shared__ double L[kPanel][kPanel + 1];
  __shared__ double Linv[kPanel];
  double* A = F + d.off;
  for (int idx = threadIdx.x; idx < kb * kb; idx += blockDim.x) {
    int i = idx % kb, j = idx / kb;
    if (i >= j) L[i][j] = A[(k + i) + (int64_t)(k + j) * d.ld];
  }
  __syncthreads();
  if (threadIdx.x < kb) Linv[threadIdx.x] = 1.0 / L[threadIdx.x][threadIdx.x];
  __syncthreads();
  const int r = k + kb + blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= d.N) return;
  double x[kPanel];
#pragma unroll
  for (int t = 0; t < kPanel; t++) x[t] = t < kb ? A[r + (int64_t)(k + t) * d.ld] : 0.0;
  row_trsm(x, L, Linv, kb);
#pragma unroll
  for (int t = 0; t < kPanel; t++)
    if (t < kb) A[r + (int64_t)(k + t) * d.ld] = x[t];
}

// Trailing update C(r, c) -= sum_t X(r, t) X(c, t), r >= c, over [k+kb, N)^2,
// 64 x 64 tiles per CTA (four warps of 32 x 32) on the FP64 tensor cores.
constexpr int UT = 64;
__global__ void __launch_bounds__(128) k_syrk(const int* __restrict__ flist,
                                              const FrontDev* __restrict__ fr,
                                              double* __restrict__ F, int k) {
  const int f = flist[blockIdx.y];
  const FrontDev d = fr[f];
  if (k >= d.n) return;
  const int kb = min(kPanel, d.n - k);
  const int r0 = k + kb;
  const int M = d.N - r0;
  if (M <= 0) return;
  const int T = (M + UT - 1) / UT;
  if ((int)blockIdx.x >= T * (T + 1) / 2) return;
  int I, J;
  tri_index(blockIdx.x, I, J);
  __shared__ double Xa[UT * kPS];
  __shared__ double Xb[UT * kPS];
  double* A = F + d.off;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int idx = tid; idx < UT * kPanel; idx += blockDim.x) {
    const int i = idx % UT, t = idx / UT;
    const int ra = r0 + I * UT + i, rb = r0 + J * UT + i;
    const bool ok = t < kb;
    Xa[i * kPS + t] = (ok && ra < d.N) ? A[ra + (int64_t)(k + t) * d.ld] : 0.0;
    Xb[i * kPS + t] = (ok && rb < d.N) ? A[rb + (int64_t)(k + t) * d.ld] : 0.0;
  }
  __syncthreads();
  const int wi = warp >> 1, wj = warp & 1;
  if (I == J && wi < wj) return;             // strictly upper quarter of a diagonal tile
  double acc[4][4][2];
  const int kk = (kb + 3) & ~3;
  {  // tile rows from Xa, tile columns from Xb
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
    const int rr = lane >> 2, cc = lane & 3;
    for (int t = 0; t < kk; t += 4) {
      double fa[4], fb[4];
#pragma unroll
      for (int a = 0; a < 4; a++) fa[a] = Xa[(wi * 32 + 8 * a + rr) * kPS + t + cc];
#pragma unroll
      for (int b = 0; b < 4; b++) fb[b] = Xb[(wj * 32 + 8 * b + rr) * kPS + t + cc];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) dmma(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
    }
  }
  warp_tile_sub(A, d.ld, r0, M, I * UT + wi * 32, J * UT + wj * 32, lane, acc);
}

// ---------------------------------------------------------------------------
// The tensor-core levels' sub-panels under MFGPU_SUBPANEL=0: one cooperative
// persistent launch.  Two-level
// blocking: outer panels of `outer` columns (kOuter = 512 unless the caller
// asks for narrower ones); inside each, 32-column steps
//   A  triangular solve of the rows below the diagonal block (every work item
//      factors the 32 x 32 diagonal block itself, from the not yet overwritten
//      values, so no extra phase is needed),
//   B  the diagonal block is written back and the outer panel's remaining
//      columns are updated with the 32 new columns,
// and after the outer panel
//   C  the trailing matrix is updated with the whole outer panel.
// Phases are separated by grid-wide barriers; work items (row blocks, 64 x 64
// tiles) of all fronts of the level are spread over all CTAs.
// ---------------------------------------------------------------------------
constexpr int kOuter = 512;
constexpr int kCT = 128;           // threads per CTA of the cooperative kernel
constexpr int kMaxCoopFronts = 8192;

// C(tile) -= X(rows) X(cols)^T over columns [k0, k1) of the front, 64 x 64 tile
// at rows [ri, ri+64), cols [ci, ci+64); rows < N, cols < cmax, row >= col.
template <class T>
__device__ void coop_tile_update(T* A, int64_t ld, int N, int cmax, int ri, int ci, int k0, int k1,
                                 T* Xa, T* Xb) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wi = warp >> 1, wj = warp & 1;
  T acc[4][4][2];
  acc_zero(acc);
  const bool diag = (ri == ci);
  const bool live = !(diag && wi < wj);
  for (int kc = k0; kc < k1; kc += kPanel) {
    const int kb = min(kPanel, k1 - kc);
    __syncthreads();
    for (int idx = tid; idx < 64 * kPanel; idx += kCT) {
      const int i = idx % 64, t = idx / 64;
      const bool ok = t < kb;
      const int ra = ri + i, rb = ci + i;
      Xa[i * kPS + t] = (ok && ra < N) ? A[ra + (int64_t)(kc + t) * ld] : T(0);
      Xb[i * kPS + t] = (ok && rb < N) ? A[rb + (int64_t)(kc + t) * ld] : T(0);
    }
    __syncthreads();
    if (live) warp_gemm_nt_acc(Xa, kPS, wi * 32, Xb, kPS, wj * 32, (kb + 3) & ~3, lane, acc);
  }
  if (!live) return;
  const int rr = lane >> 2, cc = lane & 3;
  // all loads first, then all stores, so the accesses overlap
  T cur[4][4][2];
#pragma unroll
  for (int b = 0; b < 4; b++)
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int c = ci + wj * 32 + 8 * b + 2 * cc + q;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int r = ri + wi * 32 + 8 * a + rr;
        cur[a][b][q] = (r < N && c < cmax && r >= c) ? A[r + (int64_t)c * ld] : T(0);
      }
    }
#pragma unroll
  for (int b = 0; b < 4; b++)
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int c = ci + wj * 32 + 8 * b + 2 * cc + q;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int r = ri + wi * 32 + 8 * a + rr;
        if (r < N && c < cmax && r >= c) A[r + (int64_t)c * ld] = cur[a][b][q] - acc[a][b][q];
      }
    }
}

// Factored diagonal blocks are handed from the CTA that completes their update
// to every work item of the next step through a per-front slot in global
// memory holding the inverse of the factor (32 rows of stride kLi).
constexpr int kDiagSlot = kPanel * kLi;

// Warp 0 of the calling CTA factors the diagonal block at (k, k), writes it
// back into the front and publishes it in `slot`.  Every thread must call.
template <class T>
__device__ void coop_factor_publish(T* A, int64_t ld, int k, int kb, T* slot,
                                    T (*Ls)[kPanel + 1], T* Li, T* Dinv,
                                    DevError* err, int f) {
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    warp_factor_inv(A, ld, k, kb, Ls, Li, Dinv, err, f);
    for (int i = 0; i < kPanel; i++) slot[i * kLi + lane] = Li[i * kLi + lane];
  }
}

__device__ __forceinline__ int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Per-phase work-item prefixes come from the host (coop_phase_prefix): for
// phase p, pref[p * (nf + 1) + i] is the first item of front i.  Each CTA
// copies the phase's prefix into shared memory and binary-searches it.
//
// One launch covers the outer panels [K0, K1) (K0 a multiple of outer);
// phase0 is the index of the first phase of outer panel K0 in phase_pref.  With
// trailing == 0 the last outer panel's phase C is left to the caller (the
// tensor-core trailing update of the mixed path), and the next launch factors
// and publishes its first diagonal block itself.
template <class T>
__global__ void __launch_bounds__(kCT) k_level_coop(const int* __restrict__ flist, int nf,
                                                    const FrontDev* __restrict__ fr,
                                                    T* __restrict__ F, DevError* err, int maxn,
                                                    T* __restrict__ slots,
                                                    const int* __restrict__ phase_pref, int K0,
                                                    int K1, int phase0, int trailing, int outer,
                                                    unsigned* gbar) {
  unsigned gtarget = 0;
  __shared__ T Ls[kPanel][kPanel + 1];
  __shared__ T Li[kPanel * kLi];
  __shared__ T Dinv[kPanel];
  extern __shared__ __align__(16) unsigned char smraw[];
  T* Xa = reinterpret_cast<T*>(smraw);      // phase B / C tile operands
  T* Xb = Xa + 64 * kPS;
  T* Rows = Xa;                             // phase A: kCT = 128 staged rows
  int* pre = reinterpret_cast<int*>(Xa + 2 * 64 * kPS);
  const int tid = threadIdx.x;
  int phase = phase0;
  auto load_phase = [&]() {
    __syncthreads();
    const int* p = phase_pref + (int64_t)(phase++) * (nf + 1);
    for (int i = tid; i <= nf; i += kCT) pre[i] = p[i];
    __syncthreads();
  };
  auto find = [&](int item) {   // largest i with pre[i] <= item
    int lo = 0, hi = nf - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pre[mid] <= item) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  };
  // the first diagonal block of every front
  for (int i = blockIdx.x; i < nf; i += gridDim.x) {
    const int f = flist[i];
    const FrontDev d = fr[f];
    if (d.n > K0)
      coop_factor_publish(F + d.off, d.ld, K0, min(kPanel, d.n - K0), slots + (int64_t)i * kDiagSlot,
                          Ls, Li, Dinv, err, f);
  }
  grid_barrier(gbar, gtarget, err);
  for (int K = K0; K < K1 && K < maxn; K += outer) {
    for (int k = K; k < K + outer && k < maxn; k += kPanel) {
      // ---- phase A: rows below the (already factored) diagonal block ----
      load_phase();
      for (int item = blockIdx.x; item < pre[nf]; item += gridDim.x) {
        const int i = find(item);
        const FrontDev d = fr[flist[i]];
        T* A = F + d.off;
        const int kb = min(kPanel, d.n - k);
        const T* slot = slots + (int64_t)i * kDiagSlot;
        const int rbase = k + kb + (item - pre[i]) * kCT;
        const int Mi = min(kCT, d.N - rbase);
        __syncthreads();
        for (int idx = tid; idx < kPanel * kLi; idx += kCT) Li[idx] = slot[idx];
        for (int idx = tid; idx < kCT * kPanel; idx += kCT) {
          const int rr = idx % kCT, t = idx / kCT;
          Rows[rr * kPS + t] = (rr < Mi && t < kb) ? A[(rbase + rr) + (int64_t)(k + t) * d.ld] : T(0);
        }
        __syncthreads();
        warp_trsm_block(Rows, (tid >> 5) * 32, (const T*)Li, kb, A, d.ld, rbase, k, Mi, tid & 31);
      }
      grid_barrier(gbar, gtarget, err);
      // ---- phase B: update the outer panel's remaining columns; the CTA that
      // updates the next diagonal block factors and publishes it ----
      load_phase();
      for (int item = blockIdx.x; item < pre[nf]; item += gridDim.x) {
        const int i = find(item);
        const int f = flist[i];
        const FrontDev d = fr[f];
        T* A = F + d.off;
        const int kb = min(kPanel, d.n - k);
        int local = item - pre[i];
        const int c0 = k + kb, cmax = min(K + outer, d.n);
        const int TI = ceil_div(d.N - c0, 64);
        int J = 0;
        while (local >= TI - J) {
          local -= TI - J;
          J++;
        }
        const int I = J + local;
        coop_tile_update(A, d.ld, d.N, cmax, c0 + I * 64, c0 + J * 64, k, k + kb, Xa, Xb);
        if (I == 0 && J == 0)
          coop_factor_publish(A, d.ld, c0, min(kPanel, d.n - c0), slots + (int64_t)i * kDiagSlot, Ls,
                              Li, Dinv, err, f);
      }
      grid_barrier(gbar, gtarget, err);
    }
    // ---- phase C: trailing update with the outer panel ----
    if (!trailing && K + outer >= K1) break;
    load_phase();
    for (int item = blockIdx.x; item < pre[nf]; item += gridDim.x) {
      const int i = find(item);
      const int f = flist[i];
      const FrontDev d = fr[f];
      const int k1 = min(K + outer, d.n);
      int I, J;
      tri_index(item - pre[i], I, J);
      coop_tile_update(F + d.off, d.ld, d.N, d.N, k1 + I * 64, k1 + J * 64, K, k1, Xa, Xb);
      if (I == 0 && J == 0 && k1 < d.n)
        coop_factor_publish(F + d.off, d.ld, k1, min(kPanel, d.n - k1), slots + (int64_t)i * kDiagSlot,
                            Ls, Li, Dinv, err, f);
    }
    grid_barrier(gbar, gtarget, err);
  }
}

// Trailing update of the panel-by-panel factorization (kernels_panel.cu):
// C(k1:N, k1:N) -= P P^T, P = L(k1:N, Ks:k1), k1 = min(Ks + w, n), lower
// 64 x 64 tiles of every front over a persistent grid.
template <class T>
__global__ void __launch_bounds__(kCT) k_trail_syrk(const int* __restrict__ flist, int nf,
                                                    const FrontDev* __restrict__ fr,
                                                    T* __restrict__ F, int Ks, int w) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* Xa = reinterpret_cast<T*>(smraw);
  T* Xb = Xa + 64 * kPS;
  __shared__ int pre[kMaxPanelFronts + 1];
  const int tid = threadIdx.x;
  for (int i = tid; i < nf; i += kCT) {
    const FrontDev d = fr[flist[i]];
    const int k1 = min(Ks + w, d.n), t = (d.N - k1 + 63) / 64;
    pre[i + 1] = Ks < d.n && d.N > k1 ? t * (t + 1) / 2 : 0;
  }
  __syncthreads();
  if (tid == 0) {
    pre[0] = 0;
    for (int i = 0; i < nf; i++) pre[i + 1] += pre[i];
  }
  __syncthreads();
  const int total = pre[nf];
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    int lo = 0, hi = nf - 1;   // largest i with pre[i] <= item
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pre[mid] <= item) lo = mid;
      else hi = mid - 1;
    }
    const FrontDev d = fr[flist[lo]];
    const int k1 = min(Ks + w, d.n);
    int I, J;
    tri_index(item - pre[lo], I, J);
    coop_tile_update(F + d.off, d.ld, d.N, d.N, k1 + I * 64, k1 + J * 64, Ks, k1, Xa, Xb);
  }
}

// ---------------------------------------------------------------------------
// Separator gather of the sweeps, and the apply of pivoted LU fronts.  W is a
// front's workspace (N x nrhs, ld N) inside a shared buffer.
// ---------------------------------------------------------------------------
constexpr int ST = 256;

// X(sep) = (X(sep) + W_box0(sep rows)) + W_box1(sep rows), the reference's
// per-box accumulation order (mf2d.cpp:992-1011, 1036-1047).
template <class T>
__global__ void __launch_bounds__(ST) k_sep_gather(const int* __restrict__ slist,
                                                   const SepDev* __restrict__ sp,
                                                   const int* __restrict__ dofs, T* X,
                                                   int64_t ldx, int nrhs,
                                                   const T* __restrict__ Wb,
                                                   const int64_t* __restrict__ woff,
                                                   const FrontDev* __restrict__ fr) {
  const SepDev s = sp[slist[blockIdx.x]];
  const int* dl = dofs + s.dof_off;
  const int N0 = fr[s.box0].N, N1 = fr[s.box1].N;
  const T* W0 = Wb + woff[s.box0] * nrhs;
  const T* W1 = Wb + woff[s.box1] * nrhs;
  for (int idx = threadIdx.x; idx < s.s * nrhs; idx += blockDim.x) {
    const int i = idx % s.s, c = idx / s.s;
    T* x = X + dl[i] + (int64_t)c * ldx;
    *x = (*x + W0[s.pos0 + i + (int64_t)c * N0]) + W1[s.pos1 + i + (int64_t)c * N1];
  }
}

// Apply, downward part, of a pivoted LU front: W[n,N) = L21 t (t read from T by DOF).
__global__ void __launch_bounds__(ST) k_lu_apply_down(const int* __restrict__ flist,
                                                   const FrontDev* __restrict__ fr,
                                                   const double* __restrict__ F,
                                                   const int* __restrict__ dofs, int64_t ldx,
                                                   int nrhs, double* Wb,
                                                   const int64_t* __restrict__ woff,
                                                   const double* __restrict__ Tb) {
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  double* W = Wb + woff[f] * nrhs;
  const int* dl = dofs + d.dof_off;
  const double* A = F + d.off;
  double* Tt = W + (int64_t)d.N * nrhs;
  for (int idx = threadIdx.x; idx < d.n * nrhs; idx += blockDim.x) {
    const int i = idx % d.n, c = idx / d.n;
    Tt[i + (int64_t)c * d.n] = Tb[dl[i] + (int64_t)c * ldx];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < d.m * nrhs; idx += blockDim.x) {
    const int r = d.n + idx % d.m, c = idx / d.m;
    const double* t = Tt + (int64_t)c * d.n;
    double s = double(0);
    for (int j = 0; j < d.n; j++) s += A[r + (int64_t)j * d.ld] * t[j];
    W[r + (int64_t)c * d.N] = s;
  }
}

// Apply, upward part, of a pivoted LU front: u = U11 b_piv + U12 b_bd,
// b_piv <- P^T L11 u (= A22 t with t = b_piv + XR b_bd), T(piv) = u; the
// downward part W[n,N) = L21 u (= XL A22 t) is k_lu_apply_down's.
__global__ void __launch_bounds__(ST) k_lu_apply_up(const int* __restrict__ flist,
                                                    const FrontDev* __restrict__ fr,
                                                    const double* __restrict__ F,
                                                    const int* __restrict__ ipiv,
                                                    const int* __restrict__ dofs, double* X,
                                                    int64_t ldx, int nrhs, double* Wb,
                                                    const int64_t* __restrict__ woff, double* Tb) {
  const int f = flist[blockIdx.x];
  const FrontDev d = fr[f];
  double* W = Wb + woff[f] * nrhs;
  const int* dl = dofs + d.dof_off;
  const int* pv = ipiv + d.dof_off;
  const double* A = F + d.off;
  const int N = d.N, n = d.n, ld = d.ld;
  for (int idx = threadIdx.x; idx < N * nrhs; idx += blockDim.x) {
    const int i = idx % N, c = idx / N;
    W[idx] = X[dl[i] + (int64_t)c * ldx];
  }
  __syncthreads();
  double* u = W + (int64_t)N * nrhs;   // second half of the front's workspace (n x nrhs, ld n)
  // u(j) = sum_{c >= j} U(j, c) W(c): columns in order, rows across threads
  for (int idx = threadIdx.x; idx < n * nrhs; idx += blockDim.x) {
    const int j = idx % n, c = idx / n;
    const double* w = W + (int64_t)c * N;
    double s = 0.0;
    // from the warp's first row, so that a warp's loads of a column coalesce
    for (int col = j & ~31; col < N; col++)
      if (col >= j) s += A[j + (int64_t)col * ld] * w[col];
    u[j + (int64_t)c * n] = s;
  }
  __syncthreads();
  // v(r) = u(r) + sum_{j < r} L(r, j) u(j)
  for (int idx = threadIdx.x; idx < n * nrhs; idx += blockDim.x) {
    const int r = idx % n, c = idx / n;
    const double* uc = u + (int64_t)c * n;
    double s = uc[r];
    for (int j = 0; j < r; j++) s += A[r + (int64_t)j * ld] * uc[j];
    W[r + (int64_t)c * N] = s;
  }
  __syncthreads();
  if (threadIdx.x < nrhs) {   // P^T: the swaps undone in reverse order
    double* w = W + (int64_t)threadIdx.x * N;
    for (int j = n - 1; j >= 0; j--) {
      const int p = pv[j];
      if (p != j) {
        const double t = w[j];
        w[j] = w[p];
        w[p] = t;
      }
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < n * nrhs; idx += blockDim.x) {
    const int i = idx % n, c = idx / n;
    X[dl[i] + (int64_t)c * ldx] = W[i + (int64_t)c * N];
    Tb[dl[i] + (int64_t)c * ldx] = u[i + (int64_t)c * n];
  }
}

}  // namespace

template <class T>
void launch_tasks(const Task* tasks, const int2* tiles, int64_t ntiles, bool staged, T* fronts,
                  T* seps, const int* rp, const int* ci, const double* va, const int* dofs,
                  const double* scale, cudaStream_t st) {
  if (ntiles <= 0) return;
  const int64_t blocks = (ntiles + kTaskWarps - 1) / kTaskWarps;
  const int64_t gx = blocks < 65535 * 32 ? blocks : 65535 * 32;
  const int64_t gy = (blocks + gx - 1) / gx;
  const dim3 grid((unsigned)gx, (unsigned)gy);
  if (staged)
    k_tasks<T, true><<<grid, 32 * kTaskWarps, 0, st>>>(tasks, tiles, ntiles, fronts, seps, rp, ci,
                                                       va, dofs, scale);
  else
    k_tasks<T, false><<<grid, 32 * kTaskWarps, 0, st>>>(tasks, tiles, ntiles, fronts, seps, rp, ci,
                                                        va, dofs, scale);
  g_launches++;
}

void launch_potrf(const int* flist, int nf, const FrontDev* fr, double* F, int k, DevError* err,
                  cudaStream_t st) {
  if (nf <= 0) return;
  k_potrf<<<nf, 32, 0, st>>>(flist, fr, F, k, err);
  g_launches++;
}
void launch_trsm(const int* flist, int nf, const FrontDev* fr, double* F, int k, int max_rows,
                 cudaStream_t st) {
  const int rows = max_rows - k - 1;
  if (nf <= 0 || rows <= 0) return;
  k_trsm<<<dim3((rows + 127) / 128, nf), 128, 0, st>>>(flist, fr, F, k);
  g_launches++;
}
void launch_syrk(const int* flist, int nf, const FrontDev* fr, double* F, int k, int max_rows,
                 cudaStream_t st) {
  const int rows = max_rows - k - 1;
  if (nf <= 0 || rows <= 0) return;
  const int T = (rows + UT - 1) / UT;
  k_syrk<<<dim3(T * (T + 1) / 2, nf), 128, 0, st>>>(flist, fr, F, k);
  g_launches++;
}

long long launches_total() { return g_launches.load(); }

bool small_front_fits(int maxN, int elem_bytes) {
  // the staged panel (maxN x kPS) plus static shared memory must fit in 227 KB
  return (size_t)((maxN + 31) & ~31) * kPS * elem_bytes <= 200 * 1024;
}

size_t coop_slot_elems() { return (size_t)kMaxCoopFronts * kDiagSlot; }

// Work items per phase of k_level_coop for fronts (n_i, N_i), in the kernel's
// phase order: for each outer panel K, for each 32-column step k, phases A and
// B; then phase C.  Returns the per-phase prefixes (nf + 1 ints each).
std::vector<int> coop_phase_prefix(const std::vector<int>& n, const std::vector<int>& N, int maxn,
                                   int outer) {
  if (outer <= 0) outer = kOuter;
  const int nf = (int)n.size();
  std::vector<int> out;
  auto cdiv = [](int a, int b) { return (a + b - 1) / b; };
  auto push = [&](auto count) {
    int acc = 0;
    out.push_back(0);
    for (int i = 0; i < nf; i++) {
      acc += count(i);
      out.push_back(acc);
    }
  };
  for (int K = 0; K < maxn; K += outer) {
    for (int k = K; k < K + outer && k < maxn; k += kPanel) {
      push([&](int i) { return k < n[i] ? cdiv(N[i] - k - std::min(kPanel, n[i] - k), kCT) : 0; });
      push([&](int i) {
        if (k >= n[i]) return 0;
        const int kb = std::min(kPanel, n[i] - k), c0 = k + kb, cmax = std::min(K + outer, n[i]);
        if (cmax <= c0) return 0;
        const int TI = cdiv(N[i] - c0, 64), TJ = cdiv(cmax - c0, 64);
        int c = 0;
        for (int J = 0; J < TJ; J++) c += TI - J;
        return c;
      });
    }
    push([&](int i) {
      const int k1 = std::min(K + outer, n[i]);
      if (K >= n[i] || N[i] <= k1) return 0;
      const int T = cdiv(N[i] - k1, 64);
      return T * (T + 1) / 2;
    });
  }
  return out;
}

int coop_outer() { return kOuter; }

int coop_phases(int K, int maxn, int outer) {
  if (outer <= 0) outer = kOuter;
  return 2 * ((std::min(outer, maxn - K) + kPanel - 1) / kPanel) + 1;
}

template <class T>
cudaError_t launch_level_coop(const int* flist, int nf, int maxn, const FrontDev* fr, T* F,
                              DevError* err, T* slots, const int* phase_pref, unsigned* gbar,
                              cudaStream_t st, int K0, int K1, int phase0, int trailing,
                              int max_items, int outer) {
  if (nf <= 0) return cudaSuccess;
  if (outer <= 0) outer = kOuter;
  if (nf > kMaxCoopFronts || outer % kPanel || K0 % outer) return cudaErrorInvalidValue;
  cudaError_t me = cudaMemsetAsync(gbar, 0, sizeof(unsigned), st);
  if (me != cudaSuccess) return me;
  if (K1 < 0) K1 = maxn;
  const size_t sm = 2 * 64 * kPS * sizeof(T) + (size_t)(kMaxCoopFronts + 1) * sizeof(int);
  // co-resident CTAs of this instantiation (thread-safe one-time set-up: the
  // serving loop launches from several host threads)
  static const int grid = [sm]() {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(k_level_coop<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_level_coop<T>, kCT, sm);
    return sms * (per > 0 ? per : 1);
  }();
  void* args[] = {(void*)&flist, (void*)&nf,    (void*)&fr,         (void*)&F,
                  (void*)&err,   (void*)&maxn,  (void*)&slots,      (void*)&phase_pref,
                  (void*)&K0,    (void*)&K1,    (void*)&phase0,     (void*)&trailing,
                  (void*)&outer, (void*)&gbar};
  // levels with little parallel work: one CTA per work item, at least an
  // eighth of the full grid (a grid barrier costs more the more CTAs arrive)
  int g = grid;
  if (max_items > 0) g = std::min(grid, std::max(max_items, std::max(1, grid / 8)));
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_level_coop<T>, dim3(g), dim3(kCT),
                                              args, sm, st);
  g_launches++;
  return e;
}

// 128 threads a front when no front has more than four 32-row blocks (four CTAs
// an SM overlap their diagonal blocks' chains: the leaves of 24 2D problems, 1.45
// -> 0.96 ms), 256 otherwise.
template <class T, int NT>
void front_small(const int* flist, int nf, size_t sm, const FrontDev* fr, T* F, DevError* err,
                 cudaStream_t st) {
  // the largest dynamic size any launch asks for, set once (launches from
  // several host threads must not race on the attribute)
  static const bool attr = (cudaFuncSetAttribute(k_front_small<T, NT>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 200 * 1024),
                            true);
  (void)attr;
  k_front_small<T, NT><<<nf, NT, sm, st>>>(flist, fr, F, err);
}

template <class T>
void launch_front_small(const int* flist, int nf, int maxN, const FrontDev* fr, T* F, DevError* err,
                        cudaStream_t st) {
  if (nf <= 0) return;
  const size_t sm = (size_t)((maxN + 31) & ~31) * kPS * sizeof(T);
  if (maxN <= 128) front_small<T, 128>(flist, nf, sm, fr, F, err, st);
  else front_small<T, 256>(flist, nf, sm, fr, F, err, st);
  g_launches++;
}

template <class T>
void launch_sep_gather(const int* slist, int ns, const SepDev* sp, const int* dofs, T* X,
                       int64_t ldx, int nrhs, const T* W, const int64_t* woff, const FrontDev* fr,
                       cudaStream_t st) {
  if (ns <= 0) return;
  k_sep_gather<T><<<ns, ST, 0, st>>>(slist, sp, dofs, X, ldx, nrhs, W, woff, fr);
  g_launches++;
}

void launch_lu_apply_up(const int* flist, int nf, const FrontDev* fr, const double* F,
                        const int* ipiv, const int* dofs, double* X, int64_t ldx, int nrhs,
                        double* W, const int64_t* woff, double* Tb, cudaStream_t st) {
  if (nf <= 0) return;
  k_lu_apply_up<<<nf, ST, 0, st>>>(flist, fr, F, ipiv, dofs, X, ldx, nrhs, W, woff, Tb);
  g_launches++;
}

void launch_lu_apply_down(const int* flist, int nf, const FrontDev* fr, const double* F,
                          const int* dofs, int64_t ldx, int nrhs, double* W, const int64_t* woff,
                          const double* Tb, cudaStream_t st) {
  if (nf <= 0) return;
  k_lu_apply_down<<<nf, ST, 0, st>>>(flist, fr, F, dofs, ldx, nrhs, W, woff, Tb);
  g_launches++;
}

template <class T>
cudaError_t launch_trail_syrk(const int* flist, int nf, const FrontDev* fr, T* F, int Ks, int w,
                              cudaStream_t st) {
  if (nf <= 0) return cudaSuccess;
  if (nf > kMaxPanelFronts || w <= 0) return cudaErrorInvalidValue;
  const size_t sm = 2 * 64 * kPS * sizeof(T);
  static const int grid = [sm]() {   // thread-safe one-time set-up: every resident CTA
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(k_trail_syrk<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_trail_syrk<T>, kCT, sm);
    return sms * std::max(1, per);
  }();
  k_trail_syrk<T><<<grid, kCT, sm, st>>>(flist, nf, fr, F, Ks, w);
  g_launches++;
  return cudaGetLastError();
}

#define MFGPU_INSTANTIATE(T)                                                                      \
  template void launch_tasks<T>(const Task*, const int2*, int64_t, bool, T*, T*, const int*,       \
                                const int*, const double*, const int*, const double*, cudaStream_t); \
  template void launch_front_small<T>(const int*, int, int, const FrontDev*, T*, DevError*,        \
                                      cudaStream_t);                                                \
  template void launch_sep_gather<T>(const int*, int, const SepDev*, const int*, T*, int64_t, int, \
                                     const T*, const int64_t*, const FrontDev*, cudaStream_t);      \
  template cudaError_t launch_trail_syrk<T>(const int*, int, const FrontDev*, T*, int, int,       \
                                            cudaStream_t);

MFGPU_INSTANTIATE(double)
MFGPU_INSTANTIATE(float)
#undef MFGPU_INSTANTIATE
template cudaError_t launch_level_coop<float>(const int*, int, int, const FrontDev*, float*,
                                              DevError*, float*, const int*, unsigned*, cudaStream_t,
                                              int, int, int, int, int, int);

}  // namespace mfgpu
