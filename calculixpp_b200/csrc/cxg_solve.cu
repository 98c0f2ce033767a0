// The device solve of the reduced system.
//
// Jacobi-preconditioned conjugate gradients on the CSR K_ff with a warp-per-row
// SpMV and two-stage reductions; the reference's solve_sparse (SciPP spsolve / IC0-CG,
// src/compute/cpu_backend.cpp:24-72) is the CPU counterpart.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "cxg_internal.cuh"

namespace cxg {
namespace {

// y = A x (CSR, one warp per row), optionally also r = b - A x.
__global__ void spmv_kernel(int32_t nrows, const int64_t* rp, const int32_t* ci, const double* v, const double* x,
                            double* y) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < nrows; r += nw) {
    double s = 0.0;
    for (int64_t k = rp[r] + lane; k < rp[r + 1]; k += 32) s += v[k] * x[ci[k]];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) y[r] = s;
  }
}

__global__ void diag_inv_kernel(int32_t nrows, const int64_t* rp, const int32_t* ci, const double* v, double* dinv) {
  for (int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; r < nrows;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double d = 0.0;
    int64_t lo = rp[r], hi = rp[r + 1];
    while (lo < hi) {  // columns are sorted
      const int64_t mid = (lo + hi) >> 1;
      if (ci[mid] < r)
        lo = mid + 1;
      else
        hi = mid;
    }
    if (lo < rp[r + 1] && ci[lo] == r) d = v[lo];
    dinv[r] = d != 0.0 ? 1.0 / d : 1.0;
  }
}

// partial dot products: out[block] = sum a*b over the block's stride
__global__ void dot_kernel(int32_t n, const double* a, const double* b, double* partial) {
  __shared__ double sh[32];
  double s = 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    s += a[i] * b[i];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
  }
}

__global__ void finish_dot_kernel(const double* partial, int nparts, double* out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < nparts; i += 32) s += partial[i];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if (threadIdx.x == 0) *out = s;
}

// CG vector updates driven by device scalars (no host round trip per update)
__global__ void cg_update_xr(int32_t n, const double* rz, const double* pAp, double* x, double* r, const double* p,
                             const double* Ap) {
  const double alpha = *pAp != 0.0 ? *rz / *pAp : 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    x[i] += alpha * p[i];
    r[i] -= alpha * Ap[i];
  }
}

__global__ void cg_precond(int32_t n, const double* dinv, const double* r, double* z) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    z[i] = dinv[i] * r[i];
}

__global__ void cg_update_p(int32_t n, const double* rz_new, const double* rz_old, const double* z, double* p) {
  const double beta = *rz_old != 0.0 ? *rz_new / *rz_old : 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    p[i] = z[i] + beta * p[i];
}

__global__ void residual_kernel(int32_t n, const double* b, const double* Ax, double* r) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    r[i] = b[i] - Ax[i];
}

unsigned g1(int64_t n) { return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 2048))); }

}  // namespace

cudaError_t launch_spmv(int32_t nrows, const int64_t* rp, const int32_t* ci, const double* v, const double* x, double* y,
                        cudaStream_t s) {
  const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((nrows + 7) / 8, 148 * 32)));
  spmv_kernel<<<grid, 256, 0, s>>>(nrows, rp, ci, v, x, y);
  return cudaGetLastError();
}

// Jacobi-PCG. work: 5*n + 2048 + 8 doubles. Host reads the residual every 20
// iterations; returns iterations and the final relative residual.
cudaError_t cg_solve(int32_t n, const int64_t* rp, const int32_t* ci, const double* v, const double* b, double* x,
                     double rtol, int max_iter, double* work, int* iters_out, double* rel_out, cudaStream_t s) {
  double* dinv = work + 4 * static_cast<int64_t>(n);
  diag_inv_kernel<<<g1(n), 256, 0, s>>>(n, rp, ci, v, dinv);
  const Preconditioner jacobi = [&](const double* r, double* z) {
    cg_precond<<<g1(n), 256, 0, s>>>(n, dinv, r, z);
    return cudaGetLastError();
  };
  return pcg_solve(n, rp, ci, v, b, x, rtol, max_iter, work, iters_out, rel_out, s, jacobi);
}

// Preconditioned CG with z = M^-1 r from `precond`. work: 5*n + 2048 + 8 doubles (the
// fifth n-vector is left to the preconditioner's owner).
cudaError_t pcg_solve(int32_t n, const int64_t* rp, const int32_t* ci, const double* v, const double* b, double* x,
                      double rtol, int max_iter, double* work, int* iters_out, double* rel_out, cudaStream_t s,
                      const Preconditioner& precond) {
  double* r = work;
  double* z = r + n;
  double* p = z + n;
  double* Ap = p + n;
  double* partial = Ap + 2 * static_cast<int64_t>(n);
  double* sc = partial + 2048;  // rz, rz_new, pAp, bb, rr
  const unsigned gd = g1(n);
  cudaError_t e;
  if ((e = launch_spmv(n, rp, ci, v, x, Ap, s)) != cudaSuccess) return e;
  residual_kernel<<<gd, 256, 0, s>>>(n, b, Ap, r);
  if ((e = precond(r, z)) != cudaSuccess) return e;
  cudaMemcpyAsync(p, z, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
  auto dot = [&](const double* a, const double* c, double* out) {
    dot_kernel<<<gd, 256, 0, s>>>(n, a, c, partial);
    finish_dot_kernel<<<1, 32, 0, s>>>(partial, static_cast<int>(gd), out);
  };
  dot(b, b, sc + 3);
  dot(r, z, sc + 0);
  double hb = 0.0;
  cudaMemcpyAsync(&hb, sc + 3, sizeof(double), cudaMemcpyDeviceToHost, s);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
  const double bnorm = std::sqrt(hb) > 0.0 ? std::sqrt(hb) : 1.0;
  int it = 0;
  double rel = 1.0;
  for (; it < max_iter; ++it) {
    if ((e = launch_spmv(n, rp, ci, v, p, Ap, s)) != cudaSuccess) return e;
    dot(p, Ap, sc + 2);
    cg_update_xr<<<gd, 256, 0, s>>>(n, sc + 0, sc + 2, x, r, p, Ap);
    if ((e = precond(r, z)) != cudaSuccess) return e;
    dot(r, z, sc + 1);
    cg_update_p<<<gd, 256, 0, s>>>(n, sc + 1, sc + 0, z, p);
    cudaMemcpyAsync(sc + 0, sc + 1, sizeof(double), cudaMemcpyDeviceToDevice, s);
    if ((it + 1) % 20 == 0 || it + 1 == max_iter) {
      dot(r, r, sc + 4);
      double hr = 0.0;
      cudaMemcpyAsync(&hr, sc + 4, sizeof(double), cudaMemcpyDeviceToHost, s);
      if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
      rel = std::sqrt(hr) / bnorm;
      if (rel <= rtol) {
        ++it;
        break;
      }
    }
  }
  if (iters_out) *iters_out = it;
  if (rel_out) *rel_out = rel;
  return cudaGetLastError();
}

}  // namespace cxg
