// dense_solve.cu — the global solve of small scenes as one product with the
// explicit inverse of the global-step matrix (SimulationSpeed::solve,
// src/physics/SimulationSpeed.cpp:171-187, for scenes where the supernodal
// sweeps of sweep_kernels.cu are a chain of short launches).
//
// The matrix is block diagonal over the connected components, whose columns
// are contiguous in the pivot order; row r of the inverse holds the n_c
// entries of its component, rows padded to 16 bytes.
#include <cuda_runtime.h>

#include <algorithm>

#include "device.cuh"
#include "kernels.hpp"

namespace pdfb {

// 16 bytes of the inverse, and the dot products with as many entries of b
constexpr int kVec = 2;
__device__ __forceinline__ double2 ld16(const double* p) { return __ldcg(reinterpret_cast<const double2*>(p)); }
__device__ __forceinline__ void dot16(double2 w, const double* b, double& s0, double& s1) {
  const double2 v = *reinterpret_cast<const double2*>(b);
  s0 += w.x * v.x;
  s1 += w.y * v.y;
}

// x = inv(A) b, with the write-back of v and q^k (as the sweeps').  One warp a
// row, 16 bytes a lane and load, b of the whole scene in shared memory (each
// component from a 16-byte boundary, zero between them, as the rows' padding is).
// Bound by the launch and a few memory latencies for cloths of some hundred
// vertices (30 x 30: 6.5 MB that stay in L2), by L2 bandwidth at the limit of
// kDenseBytes.  The solve alone, events around it, sweeps in brackets: 30 x 30
// 12 us (33), 53 x 53 25 us (45).
//
// FP64 solves only.  An inverse kept in FP32 rounds each of its entries, and
// nothing of that averages out over the rows as the sweeps' roundings do: v of
// small cloths on a sphere was two to four times as far from the FP64 solve's as
// with the FP32 sweeps (43 x 43: 2.5e-8 relative against 7e-9).
constexpr int kDenseUnroll = 4;
__global__ void __launch_bounds__(512, 2)
    k_dense_solve(const DenseRow* __restrict__ rows, const double* __restrict__ A, const double* __restrict__ b, int n, int np,
                  const int* __restrict__ perm, WriteBack wb, DTrace trace) {
  trace_stamp(trace, DTrace::kSolve);
  extern __shared__ __align__(16) double sb[];
  const int lane = threadIdx.x & 31;
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  // what the row needs besides b, in flight while b is staged
  DenseRow R{};
  double qv = 0.;
  int64_t d = 0;
  if (r < n) {
    R = rows[r];
    if (lane < 3) {
      d = 3 * (int64_t)perm[r] + lane;
      qv = wb.q[d];
    }
  }
  if (np == n) {  // one component, nothing between the planes
    for (int k = threadIdx.x; k < 3 * n; k += blockDim.x) sb[k] = __ldcg(b + k);
  } else {
    for (int k = threadIdx.x; k < 3 * np; k += blockDim.x) sb[k] = 0.;
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
      const int at = k + rows[k].shift;
      for (int c = 0; c < 3; ++c) sb[at + c * np] = __ldcg(b + k + (int64_t)c * n);
    }
  }
  __syncthreads();
  if (r >= n) return;
  const int ld = (R.n + kVec - 1) / kVec * kVec;
  const double* a = A + R.off;
  const double* bx = sb + R.c0 + R.shift;
  double s[3][2] = {};
  int j = kVec * lane;
  for (; j + 32 * kVec * (kDenseUnroll - 1) < ld; j += 32 * kVec * kDenseUnroll) {
    double2 w[kDenseUnroll];
#pragma unroll
    for (int u = 0; u < kDenseUnroll; ++u) w[u] = ld16(a + j + 32 * kVec * u);
#pragma unroll
    for (int u = 0; u < kDenseUnroll; ++u)
#pragma unroll
      for (int c = 0; c < 3; ++c) dot16(w[u], bx + j + 32 * kVec * u + c * np, s[c][0], s[c][1]);
  }
  for (; j < ld; j += 32 * kVec) {
    const double2 w = ld16(a + j);
#pragma unroll
    for (int c = 0; c < 3; ++c) dot16(w, bx + j + c * np, s[c][0], s[c][1]);
  }
  double x[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    x[c] = s[c][0] + s[c][1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x[c] += __shfl_xor_sync(0xffffffffu, x[c], o);
  }
  if (lane < 3) {
    const double val = lane == 0 ? x[0] : lane == 1 ? x[1] : x[2];
    wb.v[d] = val;
    wb.qk[d] = qv + wb.dt * val;
  }
}

bool launch_dense_solve(cudaStream_t st, const DenseRow* rows, const double* A, const double* b, int n, int np,
                        const int* perm, WriteBack wb, DTrace trace) {
  const size_t smem = 3 * (size_t)np * sizeof(double);
  if (cudaFuncSetAttribute(k_dense_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, kDenseSmem) != cudaSuccess)
    return false;
  // the CTAs of all rows resident at once, on as many SMs as there are
  const int warps = std::max(4, std::min(16, (n + 147) / 148));
  k_dense_solve<<<(n + warps - 1) / warps, 32 * warps, smem, st>>>(rows, A, b, n, np, perm, wb, trace);
  return true;
}

// Building the inverse: the right-hand sides e_k, e_k+1, e_k+2 of every
// component at once (k = *column), and their solutions v (vertex order) as rows
// k .. k+2 of the components' inverses (they are symmetric).
__global__ void k_dense_unit(const DenseRow* __restrict__ rows, double* __restrict__ b, int n, const int* column) {
  const int k = *column;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int c = 0; c < 3; ++c) b[i + (int64_t)c * n] = i - rows[i].c0 == k + c ? 1. : 0.;
}
__global__ void k_dense_rows(const DenseRow* __restrict__ rows, const double* __restrict__ v, int n,
                             const int* __restrict__ perm, double* __restrict__ A, const int* column) {
  const int k = *column;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int c0 = rows[i].c0;
    for (int c = 0; c < 3; ++c)
      if (k + c < rows[i].n) A[rows[c0 + k + c].off + i - c0] = v[3 * (int64_t)perm[i] + c];
  }
}
__global__ void k_dense_next(int* column, int step) { *column += step; }

void launch_dense_unit(cudaStream_t st, const DenseRow* rows, double* b, int n, const int* column) {
  k_dense_unit<<<std::min(148, (n + 255) / 256), 256, 0, st>>>(rows, b, n, column);
}
void launch_dense_rows(cudaStream_t st, const DenseRow* rows, const double* v, int n, const int* perm, double* A,
                       int* column, int step) {
  k_dense_rows<<<std::min(148, (n + 255) / 256), 256, 0, st>>>(rows, v, n, perm, A, column);
  k_dense_next<<<1, 1, 0, st>>>(column, step);
}

}  // namespace pdfb
