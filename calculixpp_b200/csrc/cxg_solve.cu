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

constexpr int kSpmvThreads = 512, kVecThreads = 256;
// Blocks of the kernels that leave one partial sum each: the product 4 of 512 threads per
// SM of a B200, the vector updates 3 of 256.
constexpr int kSpmvBlocks = 592, kVecBlocks = 444;

// Sums of u and v over the block, on every thread.
__device__ __forceinline__ double2 block_sum(double u, double v) {
  __shared__ double2 sh[33];
  for (int off = 16; off > 0; off >>= 1) {
    u += __shfl_down_sync(0xffffffffu, u, off);
    v += __shfl_down_sync(0xffffffffu, v, off);
  }
  __syncthreads();  // a second sum in the same kernel reuses sh
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_double2(u, v);
  __syncthreads();
  if (threadIdx.x < 32) {
    double2 t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : make_double2(0.0, 0.0);
    for (int off = 16; off > 0; off >>= 1) {
      t.x += __shfl_down_sync(0xffffffffu, t.x, off);
      t.y += __shfl_down_sync(0xffffffffu, t.y, off);
    }
    if (threadIdx.x == 0) sh[32] = t;
  }
  __syncthreads();
  return sh[32];
}

// Sums of the partial sums p[np] and q[nq], the same on every block.
__device__ __forceinline__ double2 sum_parts(const double* p, int np, const double* q, int nq) {
  double u = 0.0, v = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) u += p[i];
  for (int i = threadIdx.x; i < nq; i += blockDim.x) v += q[i];
  return block_sum(u, v);
}

// Sum over the lane's entries of a row of len entries, W loads of each kind in flight: a loop
// that the compiler unrolls takes the last of them one by one, and most rows are shorter than
// one round of it.
template <int W>
__device__ __forceinline__ double row_sum(const double* v, const int32_t* cols, int len, const double* x, int lane) {
  double s = 0.0;
  for (int c0 = lane; c0 < len; c0 += 32 * W) {
    double xc[W], a[W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const int c = c0 + 32 * i;
      xc[i] = a[i] = 0.0;
      if (c < len) {
        xc[i] = __ldg(x + __ldg(cols + c));
        a[i] = __ldg(v + c);
      }
    }
#pragma unroll
    for (int i = 0; i < W; ++i) s = fma(a[i], xc[i], s);
  }
  return s;
}

// y = A x, and with parts the block's share of x . y. NODES: a plan's own pattern, whose
// nodes' rows share one column structure: a warp per node reads each column index and
// each entry of x once for up to three rows, which are three independent streams of
// values (us, one warp a row / one load in flight / two: C3D8 48^3 92 / 70 / 55, C3D20 22^3
// 55 / 68 / 47, C3D10 18^3 42 / 48 / 33). Otherwise a warp per row: rows of up to 96 entries in
// one round of three loads, longer ones eight at a time (the reference pattern's rows, C3D8 48^3
// 94 us one at a time, 77 so; C3D20 40^3 314 and 304). back: from the last row to the first;
// products one after the other that change direction find in L2 what the last one read
// last (a matrix a little larger than L2 is otherwise evicted just before its next use).
template <bool NODES>
__global__ void __launch_bounds__(kSpmvThreads, 4) spmv_kernel(int32_t nrows, const int64_t* rp, const int32_t* ci,
                                                            const double* v, const NodeRec* node, int64_t n_nodes,
                                                            const double* x, double* y, double* parts, bool back) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  double dot = 0.0;
  if constexpr (NODES) {
    for (int64_t w = w0; w < n_nodes; w += nw) {
      const int64_t a = back ? n_nodes - 1 - w : w;
      const uint32_t lm = node[a].len_mask;
      const int L = lm & 0xfffffff, nf = __popc(lm >> 28);
      if (nf == 0) continue;
      const int64_t base = node[a].base;
      const double *v0 = v + base, *v1 = nf > 1 ? v0 + L : v0, *v2 = nf > 2 ? v1 + L : v1;
      const int32_t* cols = ci + base;
      double s0 = 0.0, s1 = 0.0, s2 = 0.0;
      constexpr int W = 2;  // (as in row_sum; 32 registers, 64 warps a SM: three spill and lose)
      for (int c0 = lane; c0 < L; c0 += 32 * W) {
        double xc[W], a0[W], a1[W], a2[W];
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const int c = c0 + 32 * i;
          xc[i] = a0[i] = a1[i] = a2[i] = 0.0;
          if (c < L) {
            xc[i] = __ldg(x + __ldg(cols + c));
            a0[i] = __ldg(v0 + c);
            a1[i] = __ldg(v1 + c);
            a2[i] = __ldg(v2 + c);
          }
        }
#pragma unroll
        for (int i = 0; i < W; ++i) {
          s0 = fma(a0[i], xc[i], s0);
          s1 = fma(a1[i], xc[i], s1);
          s2 = fma(a2[i], xc[i], s2);
        }
      }
      for (int off = 16; off > 0; off >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, off);
        s1 += __shfl_xor_sync(0xffffffffu, s1, off);
        s2 += __shfl_xor_sync(0xffffffffu, s2, off);
      }
      if (lane < nf) {
        const int64_t row = node[a].eq0 + lane;
        const double t = lane == 0 ? s0 : lane == 1 ? s1 : s2;
        y[row] = t;
        if (parts) dot = fma(x[row], t, dot);
      }
    }
  } else {
    for (int64_t w = w0; w < nrows; w += nw) {
      const int64_t r = back ? nrows - 1 - w : w;
      const int64_t begin = rp[r];
      const int len = static_cast<int>(rp[r + 1] - begin);
      double s = len <= 96 ? row_sum<3>(v + begin, ci + begin, len, x, lane) : row_sum<8>(v + begin, ci + begin, len, x, lane);
      for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
      if (lane == 0) {
        y[r] = s;
        if (parts) dot = fma(x[r], s, dot);
      }
    }
  }
  if (parts) {
    const double t = block_sum(dot, 0.0).x;
    if (threadIdx.x == 0) parts[blockIdx.x] = t;
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

// The Jacobi-preconditioned loop, three kernels an iteration: the product with the share
// of p . A p of every block, the update of x and r with the shares of r . M^-1 r and r . r,
// and the update of p. Scalars are summed from the shares by every block of the next
// kernel, in the same order, so nothing waits for a kernel of one block; z = M^-1 r is
// formed where it is used. (Nine kernels an iteration, dot products in two stages each,
// took 87 us on a system of 203,400 rows; this way 56 us.)
__global__ void __launch_bounds__(kVecThreads) cg_start(int32_t n, const double* b, const double* Ax, const double* dinv,
                                                        double* r, double* p, double* rz, double* bb) {
  double s = 0.0, q = 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double t = b[i] - Ax[i], z = dinv[i] * t;
    r[i] = t;
    p[i] = z;
    s += t * z;
    q += b[i] * b[i];
  }
  const double2 t = block_sum(s, q);
  if (threadIdx.x == 0) {
    rz[blockIdx.x] = t.x;
    bb[blockIdx.x] = t.y;
  }
}

__global__ void __launch_bounds__(kVecThreads) cg_step(int32_t n, int np, int nv, const double* pAp, const double* rz,
                                                       const double* dinv, const double* p, const double* Ap, double* x,
                                                       double* r, double* rz_new, double* rr) {
  // the first element's loads go out before the scalars are known
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  double xi = 0.0, ri = 0.0, pi = 0.0, ai = 0.0, di = 0.0;
  auto load = [&]() {
    if (i < n) {
      xi = x[i];
      ri = r[i];
      pi = p[i];
      ai = Ap[i];
      di = dinv[i];
    }
  };
  load();
  const double2 dg = sum_parts(pAp, np, rz, nv);
  const double alpha = dg.x != 0.0 ? dg.y / dg.x : 0.0;
  double s = 0.0, q = 0.0;
  for (; i < n; i += stride, load()) {
    x[i] = xi + alpha * pi;
    const double t = ri - alpha * ai;
    r[i] = t;
    s += t * (di * t);
    q += t * t;
  }
  const double2 t = block_sum(s, q);
  if (threadIdx.x == 0) {
    rz_new[blockIdx.x] = t.x;
    rr[blockIdx.x] = t.y;
  }
}

__global__ void __launch_bounds__(kVecThreads) cg_direction(int32_t n, int nv, const double* rz_new, const double* rz_old,
                                                            const double* dinv, const double* r, double* p) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  double z = i < n ? dinv[i] * r[i] : 0.0, pi = i < n ? p[i] : 0.0;
  const double2 gh = sum_parts(rz_old, nv, rz_new, nv);
  const double beta = gh.x != 0.0 ? gh.y / gh.x : 0.0;
  for (; i < n;) {
    p[i] = z + beta * pi;
    i += stride;
    if (i < n) {
      z = dinv[i] * r[i];
      pi = p[i];
    }
  }
}

__global__ void sum_kernel(const double* parts, int n, double* out) {
  const double s = sum_parts(parts, n, nullptr, 0).x;
  if (threadIdx.x == 0) *out = s;
}

unsigned spmv_grid(int64_t units) {
  return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((units + kSpmvThreads / 32 - 1) / (kSpmvThreads / 32), kSpmvBlocks)));
}
unsigned vec_grid(int32_t n) {
  return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((static_cast<int64_t>(n) + kVecThreads - 1) / kVecThreads, kVecBlocks)));
}

cudaError_t product(int32_t n, const int64_t* rp, const int32_t* ci, const double* v, const NodeRec* node, int64_t n_nodes,
                    const double* x, double* y, double* parts, bool back, cudaStream_t s) {
  if (node)
    spmv_kernel<true><<<spmv_grid(n_nodes), kSpmvThreads, 0, s>>>(n, rp, ci, v, node, n_nodes, x, y, parts, back);
  else
    spmv_kernel<false><<<spmv_grid(n), kSpmvThreads, 0, s>>>(n, rp, ci, v, node, n_nodes, x, y, parts, back);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_spmv(int32_t nrows, const int64_t* rp, const int32_t* ci, const double* v, const double* x, double* y,
                        cudaStream_t s, const NodeRec* node, int64_t n_nodes) {
  return product(nrows, rp, ci, v, node, n_nodes, x, y, nullptr, false, s);
}

// Jacobi-PCG. work: 5*n + 2048 + 8 doubles. Host reads the residual every 20
// iterations; returns iterations and the final relative residual.
cudaError_t cg_solve(int32_t n, const int64_t* rp, const int32_t* ci, const double* v, const double* b, double* x,
                     double rtol, int max_iter, double* work, int* iters_out, double* rel_out, cudaStream_t s,
                     const NodeRec* node, int64_t n_nodes) {
  double* r = work;
  double* p = r + n;
  double* Ap = p + n;
  double* dinv = Ap + n;
  double* parts = work + 5 * static_cast<int64_t>(n);  // p . Ap, r . z (two in turn), r . r
  double* pAp = parts;
  double *rz[2] = {pAp + kSpmvBlocks, pAp + kSpmvBlocks + kVecBlocks}, *rr = rz[1] + kVecBlocks, *scalar = rr + kVecBlocks;
  static_assert(kSpmvBlocks + 3 * kVecBlocks + 1 <= 2056, "partial sums exceed the work area");
  const unsigned gv = vec_grid(n);
  const int np = static_cast<int>(spmv_grid(node ? n_nodes : n)), nv = static_cast<int>(gv);
  cudaError_t e;
  auto read = [&](const double* from, double* to) {
    sum_kernel<<<1, kVecThreads, 0, s>>>(from, nv, scalar);
    cudaMemcpyAsync(to, scalar, sizeof(double), cudaMemcpyDeviceToHost, s);
    return cudaStreamSynchronize(s);
  };
  diag_inv_kernel<<<g1(n), 256, 0, s>>>(n, rp, ci, v, dinv);
  if ((e = product(n, rp, ci, v, node, n_nodes, x, Ap, nullptr, false, s)) != cudaSuccess) return e;
  cg_start<<<gv, kVecThreads, 0, s>>>(n, b, Ap, dinv, r, p, rz[0], rr);
  double hb = 0.0;
  if ((e = read(rr, &hb)) != cudaSuccess) return e;
  const double bnorm = std::sqrt(hb) > 0.0 ? std::sqrt(hb) : 1.0;
  int it = 0;
  double rel = 1.0;
  for (; it < max_iter; ++it) {
    double *old = rz[it & 1], *now = rz[(it + 1) & 1];
    if ((e = product(n, rp, ci, v, node, n_nodes, p, Ap, pAp, (it & 1) == 0, s)) != cudaSuccess) return e;
    cg_step<<<gv, kVecThreads, 0, s>>>(n, np, nv, pAp, old, dinv, p, Ap, x, r, now, rr);
    if ((it + 1) % 20 == 0 || it + 1 == max_iter) {
      double hr = 0.0;
      if ((e = read(rr, &hr)) != cudaSuccess) return e;
      rel = std::sqrt(hr) / bnorm;
      if (rel <= rtol) {
        ++it;
        break;
      }
    }
    cg_direction<<<gv, kVecThreads, 0, s>>>(n, nv, now, old, dinv, r, p);
  }
  if (iters_out) *iters_out = it;
  if (rel_out) *rel_out = rel;
  return cudaGetLastError();
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
  if ((e = product(n, rp, ci, v, nullptr, 0, x, Ap, nullptr, false, s)) != cudaSuccess) return e;
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
    if ((e = product(n, rp, ci, v, nullptr, 0, p, Ap, nullptr, (it & 1) == 0, s)) != cudaSuccess) return e;
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
