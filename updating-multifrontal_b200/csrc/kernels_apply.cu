// Application of the factored operator, b = A x with A = L L^T over the tree
// (the reference's Apply, src/DE/mf2d.cpp:904-974), for Cholesky fronts.
//
// A front contributes t = [L11; L21]^T [x_piv; x_bd], b_piv = L11 t and
// L21 t for its separators.  Every front reads only the input vector, so the
// fronts of all levels go through two launches together:
//   k_apply_t   items of 64 columns of a front: t = L(:, cols)^T x;
//   k_apply_l   items of 64 rows of a front: L(rows, :) t, pivot rows to b,
//               boundary rows to the front's workspace for the separator
//               gathers, which follow level by level.
// Bound: HBM, each element of L read once per launch.  Items of a fixed width
// spread a large front over all SMs.  Against one CTA per front and level
// (where the root of a 2D 511^2 tree took 2.5 of 5.85 ms on one SM), 4 vectors:
// 2D 511^2 5.78 -> 0.44 ms, 3D 34 x 24 x 47 with 9 vectors 61.5 -> 0.72 ms.
#include <atomic>
#include <cstdint>

#include "device.cuh"

namespace mfgpu {

extern std::atomic<long long> g_launches;

namespace {

constexpr int AB = 64;     // columns (k_apply_t) or rows (k_apply_l) of an item
constexpr int ACT = 256;   // threads per CTA
constexpr int ARC = 128;   // rows of x staged per round in k_apply_t
constexpr int ACC = 128;   // columns of t staged per round in k_apply_l

// Sums v[0 .. V) over the warp; afterwards lane l holds in v[0] the sum of
// entry l / (32 / V) (V a power of two, at most 32): each step halves the
// entries a lane still carries, so V values cost V - 1 exchanges instead of
// 5 V.
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
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    o >>= 1;
  }
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

// t = L(:, cols)^T x.  A warp takes CPW columns at a time, its lanes 32
// consecutive rows per load; x is gathered through the DOF list into shared
// memory, ARC rows a round.  CPW falls with the right-hand sides to keep the
// CPW * NR sums in registers.
template <class T, int NR, int CPW>
__global__ void __launch_bounds__(ACT) k_apply_t(const int2* __restrict__ items,
                                                 const FrontDev* __restrict__ fr,
                                                 const T* __restrict__ F,
                                                 const int* __restrict__ dofs,
                                                 const T* __restrict__ X, int64_t ldx, int nrhs,
                                                 T* __restrict__ Wb,
                                                 const int64_t* __restrict__ woff) {
  __shared__ T xs[NR][ARC];
  constexpr int V = CPW * NR < 32 ? CPW * NR : 32;
  const int2 it = items[blockIdx.x];
  const FrontDev d = fr[it.x];
  const T* A = F + d.off;
  const int* dl = dofs + d.dof_off;
  T* t = Wb + woff[it.x] * nrhs + (int64_t)d.N * nrhs;   // n x nrhs, ld n
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int jend = min(it.y + AB, d.n);
  for (int jb = it.y; jb < jend; jb += 8 * CPW) {
    const int j0 = jb + warp * CPW;
    T acc[CPW * NR];
#pragma unroll
    for (int i = 0; i < CPW * NR; i++) acc[i] = T(0);
    for (int r0 = jb; r0 < d.N; r0 += ARC) {
      __syncthreads();
      for (int idx = tid; idx < ARC * NR; idx += ACT) {
        const int r = idx % ARC, c = idx / ARC;
        xs[c][r] = (c < nrhs && r0 + r < d.N) ? X[dl[r0 + r] + (int64_t)c * ldx] : T(0);
      }
      __syncthreads();
      if (j0 >= jend) continue;
#pragma unroll
      for (int q = 0; q < ARC / 32; q++) {
        const int r = r0 + 32 * q + lane;
        T l[CPW];
#pragma unroll
        for (int k = 0; k < CPW; k++)
          l[k] = (r < d.N && j0 + k < jend && r >= j0 + k) ? A[r + (int64_t)(j0 + k) * d.ld] : T(0);
        const bool below = r0 + 32 * q >= jb + 8 * CPW;   // no row of the 32 above its column
#pragma unroll
        for (int c = 0; c < NR; c++) {
          const T x = xs[c][32 * q + lane];
#pragma unroll
          for (int k = 0; k < CPW; k++)   // (an infinite x above the diagonal stays out)
            if (below || r >= j0 + k) acc[k * NR + c] = fma(l[k], x, acc[k * NR + c]);
        }
      }
    }
#pragma unroll
    for (int g = 0; g < CPW * NR; g += V) {
      warp_sum_scatter<T, V>(acc + g, lane);
      const int e = g + lane / (32 / V), k = e / NR, c = e % NR;
      if (lane % (32 / V) == 0 && j0 + k < jend && c < nrhs)
        t[j0 + k + (int64_t)c * d.n] = acc[g];
    }
  }
}

// L(rows, :) t for 64 rows: thread (row tid & 63, column group tid >> 6), a
// warp reading 32 consecutive rows of a column; the four groups' sums are added
// in shared memory.
template <class T, int NR>
__global__ void __launch_bounds__(ACT) k_apply_l(const int2* __restrict__ items,
                                                 const FrontDev* __restrict__ fr,
                                                 const T* __restrict__ F,
                                                 const int* __restrict__ dofs, T* __restrict__ X,
                                                 int64_t ldx, int nrhs, T* __restrict__ Wb,
                                                 const int64_t* __restrict__ woff) {
  __shared__ T sm[ACC * NR > 4 * AB * NR ? ACC * NR : 4 * AB * NR];
  const int2 it = items[blockIdx.x];
  const FrontDev d = fr[it.x];
  T* W = Wb + woff[it.x] * nrhs;
  const T* t = W + (int64_t)d.N * nrhs;
  const int* dl = dofs + d.dof_off;
  const int tid = threadIdx.x, rl = tid & (AB - 1), g = tid >> 6;
  const int row = it.y + rl;
  const bool live = row < d.N;
  const int cend = min(d.n, it.y + AB);            // columns the item's last row reaches
  const int rend = live ? min(d.n, row + 1) : 0;   // columns of this row
  const T* Ar = F + d.off + row;
  T acc[NR];
#pragma unroll
  for (int c = 0; c < NR; c++) acc[c] = T(0);
  for (int c0 = 0; c0 < cend; c0 += ACC) {
    __syncthreads();
    for (int idx = tid; idx < ACC * NR; idx += ACT) {
      const int k = idx % ACC, c = idx / ACC;
      sm[k * NR + c] = (c < nrhs && c0 + k < d.n) ? t[c0 + k + (int64_t)c * d.n] : T(0);
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < ACC / 4; h += 16) {
      const int cb = c0 + g * (ACC / 4) + h;
      T l[16];
#pragma unroll
      for (int q = 0; q < 16; q++) l[q] = cb + q < rend ? Ar[(int64_t)(cb + q) * d.ld] : T(0);
      const bool left = cb + 16 <= it.y;   // no column right of a row's diagonal entry
#pragma unroll
      for (int q = 0; q < 16; q++)
#pragma unroll
        for (int c = 0; c < NR; c++)
          if (left || cb + q < rend) acc[c] = fma(l[q], sm[(cb - c0 + q) * NR + c], acc[c]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < NR; c++) sm[(g * NR + c) * AB + rl] = acc[c];
  __syncthreads();
  for (int idx = tid; idx < AB * nrhs; idx += ACT) {
    const int r = idx % AB, c = idx / AB, rw = it.y + r;
    if (rw >= d.N) continue;
    T s = T(0);
#pragma unroll
    for (int q = 0; q < 4; q++) s += sm[(q * NR + c) * AB + r];
    if (rw < d.n) X[dl[rw] + (int64_t)c * ldx] = s;
    else W[rw + (int64_t)c * d.N] = s;
  }
}

}  // namespace

void apply_items(const std::vector<int>& n, const std::vector<int>& N, std::vector<int>& cols,
                 std::vector<int>& rows) {
  cols.clear();
  rows.clear();
  for (size_t f = 0; f < n.size(); f++) {
    for (int j = 0; j < n[f]; j += AB) cols.insert(cols.end(), {(int)f, j});
    for (int r = 0; r < N[f]; r += AB) rows.insert(rows.end(), {(int)f, r});
  }
}

template <class T>
void launch_apply(const int* cols, int ncols, const int* rows, int nrows, const FrontDev* fr,
                  const T* F, const int* dofs, T* X, int64_t ldx, int nrhs, T* W,
                  const int64_t* woff, cudaStream_t st) {
  const int2* ci = reinterpret_cast<const int2*>(cols);
  const int2* ri = reinterpret_cast<const int2*>(rows);
#define MFGPU_APPLY(NR, CPW)                                                                  \
  do {                                                                                        \
    if (ncols > 0)                                                                            \
      k_apply_t<T, NR, CPW><<<ncols, ACT, 0, st>>>(ci, fr, F, dofs, X, ldx, nrhs, W, woff);    \
    if (nrows > 0) k_apply_l<T, NR><<<nrows, ACT, 0, st>>>(ri, fr, F, dofs, X, ldx, nrhs, W, woff); \
  } while (0)
  if (nrhs == 1) MFGPU_APPLY(1, 8);
  else if (nrhs <= 4) MFGPU_APPLY(4, 8);
  else if (nrhs <= 8) MFGPU_APPLY(8, 4);
  else MFGPU_APPLY(16, 2);
#undef MFGPU_APPLY
  g_launches += 2;
}

template void launch_apply<double>(const int*, int, const int*, int, const FrontDev*, const double*,
                                   const int*, double*, int64_t, int, double*, const int64_t*,
                                   cudaStream_t);
template void launch_apply<float>(const int*, int, const int*, int, const FrontDev*, const float*,
                                  const int*, float*, int64_t, int, float*, const int64_t*,
                                  cudaStream_t);

}  // namespace mfgpu
