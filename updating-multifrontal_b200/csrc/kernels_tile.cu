// Partial Cholesky of the fronts of a level as a dataflow of 64 x 64 tiles
// (the reference's per-box LU and Schur complement, src/DE/mf2d.cpp:558-576,
// in the symmetric form), both precisions, over all SMs.
//
// Left-looking: a task owns one tile and keeps it in registers while it
// applies every block column to its left, so a tile of the front is read once
// and written once, and no phase of a level waits for another.
//   pivot tile (J, J)   A_JJ - sum_k L_Jk L_Jk^T, then its Cholesky factor and
//                       the inverse of the factor (diag_factor below);
//   pivot tile (I, J)   A_IJ - sum_k L_Ik L_Jk^T, then times L_JJ^{-T};
//   Schur tile (I, J)   A_IJ - sum_k L_Ik L_Jk^T over all pivot columns.
// A launch may also cover one panel of block columns (kbeg: its first column):
// the same pivot tiles, with the sums over the panel's columns only, for levels
// whose trailing matrix takes each panel from another kernel (the tensor-core
// levels of the mixed path).
// Tiles are cut from row and column 0 of the front, so the block column that
// holds the last pivots may hold boundary columns too: its tiles are listed
// twice, once for the columns left of n, once for the Schur part.
//
// done[I] counts the finished block columns of block row I (they finish in
// order, each needs the one before), so one word per block row orders
// everything: a task polls the words of its two block rows (bounded), and the
// inverse of L_JJ is there once done[J] > J.  Tasks are listed column by
// column, each after the ones it waits for, and CTAs take them from a counter
// in that order, so the smallest unfinished task always runs.
//
// The inverse of L_JJ stays in the unused upper triangle of the diagonal
// block (transposed, without its diagonal), and goes to the sweeps' block
// inverses where the level has them.
//
// Measured against a cooperative kernel with a grid barrier after each 32
// columns' panel and update phases (about 50 us per 64 columns, a trailing
// update that reads and writes every tile once per 512 columns), FP64: the root
// of a 2D 1023^2 tree (2045 x 2045) 1.94 -> 1.04 ms, 127^2 (253 x 253) 256 ->
// 110 us, the four levels of a 3D 79 x 63 x 50 tree 78.7 -> 43 ms (27 TFLOP/s at
// the root, 11886 x 11886).
//
// Bound: the FP64 units (64 multiply-adds a cycle and SM; mma.sync m8n8k4
// moves the operands of 256 per warp instruction) or FP32 units for many or
// large fronts; the chain of diagonal tiles for a few small ones.  64 x 64
// tiles in four warps leave three CTAs on an SM, one computing while another
// waits for a block column.
#include <algorithm>
#include <atomic>
#include <cstdint>

#include "device.cuh"

namespace mfgpu {

extern std::atomic<long long> g_launches;

namespace {

constexpr int B = kTileBlock;         // tile edge
constexpr int KS = 32;                // columns per shared-memory stage
constexpr int TS = B + 4;             // stage stride: fragment loads without bank conflicts
constexpr int DS = 2 * B + 4;         // stride of the diagonal tile's work array (128 rows)
constexpr int TT = 128;               // threads per CTA
constexpr unsigned kTileSpin = 1u << 25;

// Shared memory: two stages of two operands; afterwards a tile and a block
// inverse (64 x TS each), or the diagonal tile's work array (64 x DS).
template <class T>
constexpr size_t tile_smem() {
  return (size_t)4 * KS * TS * sizeof(T);
}
static_assert(B * DS <= 4 * KS * TS, "the diagonal tile's work array fits the stages");

__device__ __forceinline__ double rsq(double x) { return rsqrt(x); }
// One Newton step on rsqrtf (up to two units off): L's diagonal, its reciprocal
// and the inverse then agree to rounding.
__device__ __forceinline__ float rsq(float x) {
  const float r = rsqrtf(x);
  return fmaf(0.5f * r, fmaf(-x * r, r, 1.0f), r);
}

// 16 bytes global -> shared through L2 only (L written by other SMs in this
// launch), the last (16 - bytes) zero.
__device__ __forceinline__ void cp16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}

// The accumulator of a 64 x 64 tile and its products, spread over the CTA.
// gemm: acc(r, c) += sum_{t < kk} X[t * sx + r] Y(c, t) with Y(c, t) at
// Y[t * sy + c] (YT false) or Y[c * sy + t] (YT true).
template <class T>
struct Acc;

// FP64: four warps of 32 x 32, m8n8k4 fragments.
template <>
struct Acc<double> {
  double v[4][4][2];
  int wi, wj, rr, cc;
  __device__ __forceinline__ Acc() {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    wi = (w >> 1) * 32;
    wj = (w & 1) * 32;
    rr = lane >> 2;
    cc = lane & 3;
  }
  template <class F>
  __device__ __forceinline__ void each(F&& f) {
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
      for (int q = 0; q < 2; q++)
#pragma unroll
        for (int a = 0; a < 4; a++) f(wi + 8 * a + rr, wj + 8 * b + 2 * cc + q, v[a][b][q]);
  }
  __device__ __forceinline__ void zero() {
    each([](int, int, double& x) { x = 0.0; });
  }
  __device__ __forceinline__ void add(const Acc& o) {
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) {
        v[a][b][0] += o.v[a][b][0];
        v[a][b][1] += o.v[a][b][1];
      }
  }
  // Whether the thread's values lie wholly outside rows [rlo, rhi) x columns
  // [clo, chi) of the tile, or above its diagonal (`diag`).
  __device__ __forceinline__ bool outside(int rlo, int rhi, int clo, int chi, bool diag) const {
    return wi >= rhi || wi + 32 <= rlo || wj >= chi || wj + 32 <= clo || (diag && wi < wj);
  }
  // Columns of a product with a lower triangular Y^T: the warp's need none beyond wj + 32.
  __device__ __forceinline__ int reach() const { return wj + 32; }
  template <bool YT>
  __device__ __forceinline__ void gemm(int kk, const double* X, int sx, const double* Y, int sy) {
#pragma unroll 4
    for (int k = 0; k < kk; k += 4) {
      double fa[4], fb[4];
#pragma unroll
      for (int a = 0; a < 4; a++) fa[a] = X[(k + cc) * sx + wi + 8 * a + rr];
#pragma unroll
      for (int b = 0; b < 4; b++)
        fb[b] = YT ? Y[(wj + 8 * b + rr) * sy + k + cc] : Y[(k + cc) * sy + wj + 8 * b + rr];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
          asm volatile(
              "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
              : "+d"(v[a][b][0]), "+d"(v[a][b][1])
              : "d"(fa[a]), "d"(fb[b]));
    }
  }
};

// FP32: 8 x 4 values per thread, rows 4 ty .. + 3 and 32 more, columns tx + 16 j,
// as pairs of rows: one instruction does both multiply-adds of a pair
// (fma.rn.f32x2, each rounded as fmaf), which leaves the issue slots to the
// operands' loads (64 fronts of 1981 x 631: 3.10 ms with scalar ones, 2.78 so).
template <>
struct Acc<float> {
  unsigned long long v[4][4];   // [row pair][column]
  int tx, ty;
  __device__ __forceinline__ Acc() {
    tx = threadIdx.x & 15;
    ty = threadIdx.x >> 4;
  }
  template <class F>
  __device__ __forceinline__ void each(F&& f) {
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v[i][j]));
        const int r = (i >> 1) * 32 + 4 * ty + 2 * (i & 1), c = tx + 16 * j;
        f(r, c, lo);
        f(r + 1, c, hi);
        asm("mov.b64 %0, {%1, %2};" : "=l"(v[i][j]) : "f"(lo), "f"(hi));
      }
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) v[i][j] = 0ull;
  }
  __device__ __forceinline__ void add(const Acc& o) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++)
        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v[i][j]) : "l"(o.v[i][j]));
  }
  __device__ __forceinline__ bool outside(int, int, int, int, bool) const { return false; }
  __device__ __forceinline__ int reach() const { return B; }
  template <bool YT>
  __device__ __forceinline__ void gemm(int kk, const float* X, int sx, const float* Y, int sy) {
#pragma unroll 2
    for (int k = 0; k < kk; k += 4) {
      float y[4][4];   // [column][k]
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (YT) {
          const float4 q = *reinterpret_cast<const float4*>(Y + (tx + 16 * j) * sy + k);
          y[j][0] = q.x; y[j][1] = q.y; y[j][2] = q.z; y[j][3] = q.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; e++) y[j][e] = Y[(k + e) * sy + tx + 16 * j];
        }
      }
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(X + (k + e) * sx + 4 * ty);
        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(X + (k + e) * sx + 32 + 4 * ty);
        const unsigned long long x[4] = {p.x, p.y, q.x, q.y};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          unsigned long long yy;
          asm("mov.b64 %0, {%1, %1};" : "=l"(yy) : "f"(y[j][e]));
#pragma unroll
          for (int i = 0; i < 4; i++)
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[i][j]) : "l"(x[i]), "l"(yy));
        }
      }
    }
  }
};

// Four consecutive values from 16-byte aligned shared memory.
__device__ __forceinline__ void ld4s(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ld4s(const double* p, double (&v)[4]) {
  const double2 a = *reinterpret_cast<const double2*>(p);
  const double2 b = *reinterpret_cast<const double2*>(p + 2);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// Cholesky factor of the 64 x 64 block in w (column c at w[c * DS], rows 0 ..
// 63, lower triangle, zeros above) over its first kb columns, and beside it
// the same column operations on the 64 rows of an identity (rows 64 .. 127),
// which become L^{-T}; rows kb .. 63 become rows of L below the block.  A row
// per thread, 32 of its columns at a time in registers; four columns a step:
// every thread factors the 4 x 4 pivot block for itself (no hand-off between
// the four dependent reciprocal roots), finishes its own four entries, and
// after one exchange of the rows' new entries updates its later columns, the
// next step's first.  The right half takes the left one as a product.
// Returns the first non-positive pivot or -1.
template <class T>
__device__ int diag_factor(T* w, int kb, T (*q4)[B][4], T (*d4)[4][4]) {
  const int tid = threadIdx.x;
  int bad = -1;
#pragma unroll 1
  for (int h = 0; h < 2; h++) {
    const int c0 = 32 * h;
    if (c0 >= kb) break;
    T row[32];
#pragma unroll
    for (int c = 0; c < 32; c++) row[c] = w[(c0 + c) * DS + tid];
    if (tid >= c0 && tid < c0 + 4)
#pragma unroll
      for (int j = 0; j < 4; j++) d4[0][tid - c0][j] = row[j];
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 8; p++) {
      const int cp = c0 + 4 * p;   // first column of the step
      if (cp < kb) {
        T l[4][4], r[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j <= i; j++) l[i][j] = d4[p & 1][i][j];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          T dj = l[j][j];
#pragma unroll
          for (int t = 0; t < j; t++) dj -= l[j][t] * l[j][t];
          if (cp + j >= kb) dj = T(1);
          if (!(dj > T(0))) {        // non-positive or NaN pivot: not SPD
            if (bad < 0) bad = cp + j;
            dj = T(1);
          }
          r[j] = rsq(dj);
#pragma unroll
          for (int i = j + 1; i < 4; i++) {
            T s = l[i][j];
#pragma unroll
            for (int t = 0; t < j; t++) s -= l[i][t] * l[j][t];
            l[i][j] = s * r[j];
          }
        }
        // this row's entries (zero right of a pivot row's diagonal)
        T x[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          T s = row[4 * p + j];
#pragma unroll
          for (int t = 0; t < j; t++) s -= x[t] * l[j][t];
          x[j] = (cp + j < kb && !(tid < B && tid < cp + j)) ? s * r[j] : T(0);
          row[4 * p + j] = x[j];
        }
        if (tid < B)
#pragma unroll
          for (int j = 0; j < 4; j++) q4[p & 1][tid][j] = x[j];
        __syncthreads();
        // the rows' entries of the later columns, the next step's first
#pragma unroll
        for (int c = 4 * p + 4; c < 32; c++) {
          const T* y = q4[p & 1][c0 + c];
          row[c] -= fma(x[3], y[3], fma(x[2], y[2], fma(x[1], y[1], x[0] * y[0])));
          if (c == 4 * p + 7 && tid >= cp + 4 && tid < cp + 8)
#pragma unroll
            for (int j = 0; j < 4; j++) d4[(p + 1) & 1][tid - cp - 4][j] = row[4 * p + 4 + j];
        }
        __syncthreads();
      }
    }
#pragma unroll
    for (int c = 0; c < 32; c++) w[(c0 + c) * DS + tid] = c0 + c < kb ? row[c] : T(0);
    __syncthreads();
    if (h == 0 && kb > 32) {
      // columns 32 .. 63: - X(:, 0:32) L(32:64, 0:32)^T for the rows that have
      // some, 32 .. 63 of the block and the first 32 of the identity, 4 x 4 a thread
      const int rg = 32 + (tid & 15) * 4, cg = 32 + (tid >> 4) * 4;
      T a[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) a[i][j] = T(0);
#pragma unroll 8
      for (int t = 0; t < 32; t++) {
        T xr[4], yc[4];
        ld4s(w + t * DS + rg, xr);
        ld4s(w + t * DS + cg, yc);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) a[i][j] = fma(xr[i], yc[j], a[i][j]);
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (rg + i >= cg + j) w[(cg + j) * DS + rg + i] -= a[i][j];   // (entries above stay zero)
      __syncthreads();
    }
  }
  return bad;
}

template <class T>
__global__ void __launch_bounds__(TT, 3)
    k_front_tiles(const int* __restrict__ flist, const FrontDev* __restrict__ fr, T* __restrict__ F,
                  const int2* __restrict__ tasks, int ntasks, const int* __restrict__ rowoff,
                  int* done, int* counter, T* __restrict__ Dv,
                  const int64_t* __restrict__ dinv_off, DevError* err, int kbeg) {
  extern __shared__ __align__(16) unsigned char tile_raw[];
  T* sm = reinterpret_cast<T*>(tile_raw);
  __shared__ __align__(16) T q4[2][B][4];
  __shared__ __align__(16) T d4[2][4][4];
  __shared__ int s_task, s_ready;
  constexpr int V = 16 / (int)sizeof(T);   // values per 16-byte copy
  const int tid = threadIdx.x;
  while (true) {
    __syncthreads();                       // the previous task's shared memory is free
    if (tid == 0) s_task = atomicAdd(counter, 1);
    __syncthreads();
    if (s_task >= ntasks) return;
    const int2 tk = tasks[s_task];
    const int slot = tk.x, I = tk.y & 0x7fff, J = (tk.y >> 15) & 0x7fff, schur = tk.y >> 30;
    const int f = flist[slot];
    const FrontDev d = fr[f];
    T* A = F + d.off;
    const int64_t ld = d.ld;
    const int n = d.n, N = d.N, r0 = I * B, c0 = J * B;
    int* dI = done + rowoff[slot] + I;
    int* dJ = done + rowoff[slot] + J;
    // wait until block rows I and J have more than k finished block columns;
    // returns how many both have
    auto wait = [&](int k) {
      if (tid == 0) {
        volatile int* a = dI;
        volatile int* b = dJ;
        volatile int* code = err ? &err->code : nullptr;
        const unsigned lim = wait_limit(err, kTileSpin);
        unsigned it = 0;
        int v = min(*a, *b);
        while (v <= k) {
          if (++it > lim) {
            if (err) atomicCAS(&err->code, 0, 3);
            break;
          }
          if ((it & 1023u) == 0 && code && *code == 3) break;   // another CTA gave up
          __nanosleep(20);
          v = min(*a, *b);
        }
        __threadfence();
        s_ready = max(v, k + 1);
      }
      __syncthreads();
      return s_ready;
    };
    auto publish = [&](int cols) {
      __threadfence();
      __syncthreads();
      if (tid == 0) atomicExch(dI, cols);
    };
    // the tile, negated: the products are added to it, each `chunk` columns'
    // summed from zero first (the sums' rounding errors then grow with the
    // chunk and the number of chunks, not with their product)
    const int chunk = n <= 1024 ? KS : n <= 4096 ? 2 * KS : 8 * KS;
    const int clo = schur ? n : 0, chi = schur ? N : n, rlo = schur ? n : 0;
    Acc<T> tot, acc;
    const T* C = A + r0 + (int64_t)c0 * ld;
    const bool dead = acc.outside(rlo - r0, N - r0, clo - c0, chi - c0, I == J);
    // (loads from a clamped address and a select: 32 loads in flight, no branches)
    tot.each([&](int r, int c, T& v) {
      const int gr = r0 + r, gc = c0 + c;
      const bool in = gr >= rlo && gr < N && gc >= clo && gc < chi && gr >= gc;
      v = *(in ? C + r + (int64_t)c * ld : A);
    });
    tot.each([&](int r, int c, T& v) {
      const int gr = r0 + r, gc = c0 + c;
      const bool in = gr >= rlo && gr < N && gc >= clo && gc < chi && gr >= gc;
      v = in ? -v : T(0);
    });
    acc.zero();
    // stages of KS columns of block rows I and J
    const int kend = schur ? n : c0, ns = (kend - kbeg + KS - 1) / KS;
    auto block_of = [&](int s) { return (kbeg + s * KS) / B; };   // block column of stage s
    auto issue = [&](int s, int buf) {
      const int k0 = kbeg + s * KS;
      T* X = sm + buf * 2 * KS * TS;
#pragma unroll
      for (int o = 0; o < 2; o++) {
        if (o == 1 && I == J) break;
        const int rb = o == 0 ? r0 : c0;
        T* Y = X + o * KS * TS;
        for (int idx = tid; idx < KS * (B / V); idx += TT) {
          const int rv = (idx % (B / V)) * V, c = idx / (B / V);
          const int take = k0 + c < n ? max(0, min(V, N - rb - rv)) : 0;
          cp16(Y + c * TS + rv, take ? A + (rb + rv) + (int64_t)(k0 + c) * ld : A,
               take * (int)sizeof(T));
        }
      }
      cp_commit();
    };
    int ready = 0;
    if (ns > 0) {
      ready = wait(block_of(0));
      issue(0, 0);
    }
    for (int s = 0; s < ns; s++) {
      const bool more = s + 1 < ns, pre = more && block_of(s + 1) < ready;
      if (pre) {
        issue(s + 1, (s + 1) & 1);
        cp_wait<1>();
      } else {
        cp_wait<0>();
      }
      __syncthreads();
      const T* X = sm + (s & 1) * 2 * KS * TS;
      if (!dead) acc.template gemm<false>(KS, X, TS, I == J ? X : X + KS * TS, TS);
      if (!more || (s + 1) * KS % chunk == 0) {
        tot.add(acc);
        acc.zero();
      }
      __syncthreads();
      if (more && !pre) {   // the next block column is not there yet: computed first, wait now
        ready = wait(block_of(s + 1));
        issue(s + 1, (s + 1) & 1);
      }
    }
    if (schur) {
      tot.each([&](int r, int c, T& v) {
        const int gr = r0 + r, gc = c0 + c;
        if (gr >= n && gr < N && gc >= n && gc < N && gr >= gc) A[gr + (int64_t)gc * ld] = -v;
      });
      continue;
    }
    const int kb = min(B, n - c0);
    if (I == J) {
      // factor, inverse
      tot.each([&](int r, int c, T& v) { sm[c * DS + r] = r >= c ? -v : T(0); });
      for (int idx = tid; idx < B * B; idx += TT) {
        const int r = idx & (B - 1), c = idx / B;
        sm[c * DS + B + r] = r == c ? T(1) : T(0);
      }
      __syncthreads();
      const int bad = diag_factor<T>(sm, kb, q4, d4);
      if (tid == 0 && bad >= 0 && atomicCAS(&err->code, 0, 1) == 0) {
        err->front = f;
        err->col = c0 + bad;
      }
      // L below the diagonal; above it the inverse: column c, row i < c, holds Linv(c, i)
      {
        const int r = tid & (B - 1);
        T* P = A + (r0 + r) + (int64_t)c0 * ld;
#pragma unroll 8
        for (int c = tid >> 6; c < kb; c += 2)
          if (r0 + r < N && (r >= c || r < kb))
            P[(int64_t)c * ld] = r >= c ? sm[c * DS + r] : sm[c * DS + B + r];
      }
      publish(J + 1);
      if (dinv_off[f] >= 0) {
        T* D = Dv + dinv_off[f] + (int64_t)J * 2 * B * B;
        for (int idx = tid; idx < B * B; idx += TT) {
          const int r = idx & (B - 1), c = idx / B;
          const bool in = r < kb && c < kb;
          D[B * B + idx] = in ? sm[c * DS + B + r] : T(0);   // Linv^T(r, c) = Linv(c, r)
          D[idx] = in ? sm[r * DS + B + c] : T(0);           // Linv(r, c)
        }
      }
      continue;
    }
    // times L_JJ^{-T}
    tot.each([&](int r, int c, T& v) { sm[c * TS + r] = -v; });
    if (ready <= J) {   // the inverse of this column
      if (tid == 0) {
        volatile int* b = dJ;
        volatile int* code = err ? &err->code : nullptr;
        const unsigned lim = wait_limit(err, kTileSpin);
        unsigned it = 0;
        while (*b <= J) {
          if (++it > lim) {
            if (err) atomicCAS(&err->code, 0, 3);
            break;
          }
          if ((it & 1023u) == 0 && code && *code == 3) break;
          __nanosleep(20);
        }
        __threadfence();
      }
      __syncthreads();
    }
    T* Li = sm + B * TS;                     // Li[c * TS + t] = Linv(c, t), t <= c
    {
      const int t = tid & (B - 1), ch = tid >> 6;
      const T* U = A + (c0 + t) + (int64_t)c0 * ld;   // column c, row t
      const T dg = t < kb ? __ldcg(U + (int64_t)t * ld) : T(1);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        T v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) {
          const int c = 32 * h + 2 * q + ch;
          v[q] = __ldcg(t < c && c < kb ? U + (int64_t)c * ld : A);
        }
#pragma unroll
        for (int q = 0; q < 16; q++) {
          const int c = 32 * h + 2 * q + ch;
          if (t != c) Li[c * TS + t] = t < c && c < kb ? v[q] : T(0);
        }
      }
      if (ch == 0) Li[t * TS + t] = t < kb ? T(1) / dg : T(0);
    }
    __syncthreads();
    if (!dead) acc.template gemm<true>(min(acc.reach(), (kb + 3) & ~3), sm, TS, Li, TS);
    acc.each([&](int r, int c, T& v) {
      const int gr = r0 + r;
      if (gr < N && c < kb) A[gr + (int64_t)(c0 + c) * ld] = v;
    });
    publish(J + 1);
  }
}

}  // namespace

// Fronts in groups of about one task per CTA, each group going through its
// phases (diagonal tile, then the tiles below it, of every block column; the
// Schur tiles last) one step behind the group before it.  So the tiles of a
// column are listed a group's work after the diagonal tile that they wait for,
// and the fronts in flight at a time stay in L2 (4096 fronts of 285 x 225:
// 5.0 ms with the diagonal tiles of 48 MB of fronts first, 4.5 ms so).
void tile_tasks(const std::vector<int>& n, const std::vector<int>& N, std::vector<int>& tasks,
                std::vector<int>& rowoff) {
  constexpr int kGroupTasks = 444;
  const int nf = (int)n.size();
  auto cdiv = [](int a, int b) { return (a + b - 1) / b; };
  int row = 0;
  for (int i = 0; i < nf; i++) {
    rowoff.push_back(row);
    row += cdiv(N[i], B);
  }
  rowoff.push_back(row);
  auto add = [&](int i, int I, int J, int schur) {
    tasks.push_back(i);
    tasks.push_back(I | (J << 15) | (schur << 30));
  };
  std::vector<int> first;   // first front of each group
  std::vector<int> phases;  // of each group
  for (int i = 0, t = kGroupTasks; i < nf; i++) {
    if (t >= kGroupTasks) {
      first.push_back(i);
      phases.push_back(0);
      t = 0;
    }
    const int nb = cdiv(N[i], B), np = cdiv(n[i], B);
    t += nb * (nb + 1) / 2;
    phases.back() = std::max(phases.back(), 2 * np + 1);
  }
  first.push_back(nf);
  const int ng = (int)phases.size();
  // group g is at phase step - g; lo: the first group with phases left
  for (int lo = 0, step = 0; lo < ng; step++) {
    for (int g = lo; g < ng && g <= step; g++) {
      const int ph = step - g, s = ph / 2;
      if (ph >= phases[g]) continue;
      for (int i = first[g]; i < first[g + 1]; i++) {
        const int nb = cdiv(N[i], B), np = cdiv(n[i], B);
        if (s < np) {
          if (ph % 2 == 0) add(i, s, s, 0);
          else
            for (int I = s + 1; I < nb; I++) add(i, I, s, 0);
        } else if (ph == 2 * np) {
          for (int J = n[i] / B; J < nb && N[i] > n[i]; J++)
            for (int I = J; I < nb; I++) add(i, I, J, 1);
        }
      }
    }
    while (lo < ng && step - lo + 1 >= phases[lo]) lo++;
  }
}

// The pivot tiles of the block columns [K, K + w), diagonal tiles first.
void tile_panel_tasks(const std::vector<int>& n, const std::vector<int>& N, int K, int w,
                      std::vector<int>& tasks) {
  for (int J = K / B; J < (K + w) / B; J++) {
    for (size_t i = 0; i < n.size(); i++)
      if (J * B < n[i]) tasks.insert(tasks.end(), {(int)i, J | (J << 15)});
    for (size_t i = 0; i < n.size(); i++)
      for (int I = J + 1; J * B < n[i] && I * B < N[i]; I++)
        tasks.insert(tasks.end(), {(int)i, I | (J << 15)});
  }
}

template <class T>
cudaError_t launch_front_tiles(const int* flist, const FrontDev* fr, T* F, const int* tasks,
                               int ntasks, const int* rowoff, int nrows, int* done, T* Dv,
                               const int64_t* dinv_off, DevError* err, cudaStream_t st, int kbeg) {
  if (ntasks <= 0) return cudaSuccess;
  if (kbeg % B) return cudaErrorInvalidValue;
  // done words and, behind them, the task counter; the words of a level
  // factored by panels carry on from the panel before
  cudaError_t e = kbeg == 0 ? cudaMemsetAsync(done, 0, sizeof(int) * (size_t)(nrows + 1), st)
                            : cudaMemsetAsync(done + nrows, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  static const int grid = []() {   // thread-safe one-time set-up: every resident CTA
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(k_front_tiles<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)tile_smem<T>());
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_front_tiles<T>, TT, tile_smem<T>());
    return sms * std::max(1, per);
  }();
  k_front_tiles<T><<<std::min(grid, ntasks), TT, tile_smem<T>(), st>>>(
      flist, fr, F, reinterpret_cast<const int2*>(tasks), ntasks, rowoff, done, done + nrows, Dv,
      dinv_off, err, kbeg);
  g_launches++;
  return cudaGetLastError();
}

template cudaError_t launch_front_tiles<double>(const int*, const FrontDev*, double*, const int*, int,
                                                const int*, int, int*, double*, const int64_t*,
                                                DevError*, cudaStream_t, int);
template cudaError_t launch_front_tiles<float>(const int*, const FrontDev*, float*, const int*, int,
                                               const int*, int, int*, float*, const int64_t*,
                                               DevError*, cudaStream_t, int);

}  // namespace mfgpu
