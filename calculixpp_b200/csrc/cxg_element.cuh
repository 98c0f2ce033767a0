// Device helpers shared by the element passes (cxg_v2.cu: FP32 blocks, cxg_fp64.cu: FP64
// blocks): element-buffer slots, bulk stores, the FP64 J2 return, hourglass base vectors.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "cxg_internal.cuh"

namespace cxg {

namespace {

constexpr int kT1 = 128;  // element-pass threads per block
constexpr int kW1 = kT1 / 32;
constexpr double kSqrt3_2v2 = 1.224744871391589;

// Slot of element e in the element buffer, a ring of `ring` elements (the whole mesh when
// the assembly runs as one window; ring_base 0): e mod ring. Every element a window's
// passes touch lies in [ring_base, ring_base + 2 ring), so one conditional subtraction
// gives the slot, with no division in the inner loops.
__device__ __forceinline__ int64_t ring_slot(int64_t e, const V2Args& V) {
  const int64_t d = e - V.ring_base;
  return d < V.ring ? d : d - V.ring;
}

// Bulk copy of `bytes` (a multiple of 16) from 16-byte aligned shared memory to 16-byte
// aligned global memory, by one lane after every lane's writes are fenced and joined.
__device__ __forceinline__ void bulk_store(void* dst, const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(static_cast<unsigned>(__cvta_generic_to_shared(src))), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// The lane's earlier bulk copies have read their shared memory.
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// FP64 products and sums that the compiler must not contract its own way: the Gauss-point
// phase is inlined into several kernels (FP32 and FP64 blocks, batches), whose strains,
// stresses and histories are the same bit for bit.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }

// Inverse and determinant of the Jacobian J[i][j] = dx_i / dxi_j; returns the determinant.
__device__ __forceinline__ double invert(const double (&J)[3][3], double (&it)[3][3]) {
  const double c00 = fma(J[1][1], J[2][2], -mul(J[1][2], J[2][1]));
  const double c01 = fma(J[1][2], J[2][0], -mul(J[1][0], J[2][2]));
  const double c02 = fma(J[1][0], J[2][1], -mul(J[1][1], J[2][0]));
  const double det = fma(J[0][0], c00, fma(J[0][1], c01, mul(J[0][2], c02)));
  const double inv = 1.0 / det;
  it[0][0] = mul(c00, inv);
  it[0][1] = mul(c01, inv);
  it[0][2] = mul(c02, inv);
  it[1][0] = mul(fma(J[0][2], J[2][1], -mul(J[0][1], J[2][2])), inv);
  it[1][1] = mul(fma(J[0][0], J[2][2], -mul(J[0][2], J[2][0])), inv);
  it[1][2] = mul(fma(J[0][1], J[2][0], -mul(J[0][0], J[2][1])), inv);
  it[2][0] = mul(fma(J[0][1], J[1][2], -mul(J[0][2], J[1][1])), inv);
  it[2][1] = mul(fma(J[0][2], J[1][0], -mul(J[0][0], J[1][2])), inv);
  it[2][2] = mul(fma(J[0][0], J[1][1], -mul(J[0][1], J[1][0])), inv);
  return det;
}

// row x of sigma (Voigt xx yy zz xy xz yz) times g, added to f
__device__ __forceinline__ void add_force(double (&f)[3], const double* S, double gx, double gy, double gz) {
  f[0] = fma(S[0], gx, fma(S[3], gy, fma(S[4], gz, f[0])));
  f[1] = fma(S[3], gx, fma(S[1], gy, fma(S[5], gz, f[1])));
  f[2] = fma(S[4], gx, fma(S[5], gy, fma(S[2], gz, f[2])));
}

__device__ __forceinline__ void hardening2(const J2Mat& M, double ep, double& sy, double& h) {
  const int n = M.n;
  if (n == 1 || ep <= M.ep[0]) {
    sy = M.sy[0];
    h = 0.0;
    return;
  }
  if (ep >= M.ep[n - 1]) {
    sy = M.sy[n - 1];
    h = 0.0;
    return;
  }
  for (int i = 0; i + 1 < n; ++i) {
    if (ep >= M.ep[i] && ep <= M.ep[i + 1]) {
      h = (M.sy[i + 1] - M.sy[i]) / (M.ep[i + 1] - M.ep[i]);
      sy = fma(h, ep - M.ep[i], M.sy[i]);
      return;
    }
  }
  sy = M.sy[n - 1];
  h = 0.0;
}

// J2 radial return + consistent tangent (restating src/fem/plasticity.cpp:90-236), FP64.
// Returns true on the plastic branch; lam_t/mu_t/c_t: tangent parameters, nv: direction.
__device__ __forceinline__ bool j2_point(const J2Mat& M, double lam, double mu_el, double mu, const double* eps,
                                         const double* cs, double* ts, double* sig, double& lam_t, double& mu_t,
                                         double& c_t, double* nv, double& mu_hg) {
  const double lam2mu = lam + 2.0 * mu_el;
  double el[6];
  for (int i = 0; i < 6; ++i) el[i] = eps[i] - cs[i];
  double st[6];
  st[0] = fma(lam2mu, el[0], fma(lam, el[1], mul(lam, el[2])));
  st[1] = fma(lam, el[0], fma(lam2mu, el[1], mul(lam, el[2])));
  st[2] = fma(lam, el[0], fma(lam, el[1], mul(lam2mu, el[2])));
  st[3] = mul(mu_el, el[3]);
  st[4] = mul(mu_el, el[4]);
  st[5] = mul(mu_el, el[5]);
  const double p = (st[0] + st[1] + st[2]) / 3.0;
  const double s_tr[6] = {st[0] - p, st[1] - p, st[2] - p, st[3], st[4], st[5]};
  double xi[6];
  for (int i = 0; i < 6; ++i) xi[i] = s_tr[i] - cs[7 + i];
  const double xi_norm = sqrt(fma(2.0, fma(xi[3], xi[3], fma(xi[4], xi[4], mul(xi[5], xi[5]))),
                                  fma(xi[0], xi[0], fma(xi[1], xi[1], mul(xi[2], xi[2])))));
  const double q_tr = mul(kSqrt3_2v2, xi_norm);
  double sy0 = 0.0, h0 = 0.0;
  if (M.plastic) hardening2(M, cs[6], sy0, h0);
  if (!M.plastic || q_tr - sy0 <= 0.0 || xi_norm == 0.0) {
    for (int i = 0; i < 6; ++i) sig[i] = st[i];
    for (int i = 0; i < kStateDoubles; ++i) ts[i] = cs[i];
    lam_t = lam;
    mu_t = mu_el;
    c_t = 0.0;
    mu_hg = mu_el;
    return false;
  }
  const double ep0 = cs[6], mu3 = mul(3.0, mu);
  double dgamma = 0.0;
  for (int it = 0; it < 50; ++it) {
    double sy, h_iso;
    hardening2(M, ep0 + dgamma, sy, h_iso);
    const double g = fma(-M.h_kin, dgamma, fma(-mu3, dgamma, q_tr)) - sy;
    const double dg = -(mu3 + M.h_kin + h_iso);
    const double step = -g / dg;
    dgamma += step;
    if (dgamma < 0.0) dgamma = 0.0;
    if (fabs(step) <= mul(1e-14, 1.0 + fabs(dgamma))) break;
  }
  for (int i = 0; i < 6; ++i) nv[i] = xi[i] / xi_norm;
  const double dev_scale = mul(mul(2.0 * mu, dgamma), kSqrt3_2v2);
  const double alpha_scale = mul(mul(mul(2.0 / 3.0, M.h_kin), dgamma), kSqrt3_2v2);
  const double dep_scale = mul(dgamma, kSqrt3_2v2);
  for (int i = 0; i < 6; ++i) {
    sig[i] = fma(-dev_scale, nv[i], s_tr[i]) + (i < 3 ? p : 0.0);
    ts[i] = fma(i < 3 ? dep_scale : 2.0 * dep_scale, nv[i], cs[i]);
    ts[7 + i] = fma(alpha_scale, nv[i], cs[7 + i]);
  }
  ts[6] = ep0 + dgamma;
  double sy, h_iso;
  hardening2(M, ep0 + dgamma, sy, h_iso);
  const double theta = 1.0 - dev_scale / xi_norm;
  const double denom = 1.0 + (h_iso + M.h_kin) / mu3;
  const double theta_bar = 1.0 / denom - (1.0 - theta);
  lam_t = fma(mul(2.0 / 3.0, 1.0 - theta), mu, lam);
  mu_t = fma(-(1.0 - theta), mu, mu_el);
  c_t = mul(2.0 * mu, theta_bar);
  mu_hg = fma(-mul(c_t, nv[3]), nv[3], mu_t);
  return true;
}

__constant__ double c_hg2[4][8] = {
    {1, 1, -1, -1, -1, -1, 1, 1},
    {1, -1, -1, 1, -1, 1, 1, -1},
    {1, -1, 1, -1, 1, -1, 1, -1},
    {-1, 1, -1, 1, 1, -1, 1, -1},
};

// Persistent grid: blocks_per_sm (0 = as many as are resident) blocks on every SM,
// capped by the work available.
int64_t persistent_grid(int64_t need, int resident, int sms, int blocks_per_sm) {
  const int per_sm = blocks_per_sm > 0 ? std::min(blocks_per_sm, std::max(resident, 1)) : std::max(resident, 1);
  return std::max<int64_t>(1, std::min<int64_t>(need, static_cast<int64_t>(per_sm) * sms));
}

// Launches an element pass on a persistent grid (see launch_kernel).
cudaError_t launch_persistent(const void* kern, size_t smem, int64_t need, int blocks_per_sm, cudaStream_t s, void** args) {
  int per_sm = 0, sms = 0;
  const cudaError_t e = kernel_shape(kern, kT1, smem, &per_sm, &sms);
  return e != cudaSuccess ? e : launch_kernel(kern, persistent_grid(need, per_sm, sms, blocks_per_sm), kT1, smem, s, args);
}

// Slot k of a pass is one group (one element type, the concatenated models of that type)
// and owns blocks [blk0_k, blk0_{k+1}) of the grid. A block reads its slot's arguments
// in place from the kernel's parameter space (a copy in shared memory measured slower:
// the bodies' shared-memory stores made every argument a reload) and runs the group's
// element-pass or row-gather body with its index among the slot's blocks in place of
// blockIdx. The bodies are the ones the
// per-group kernels inline, so every value is the same bit for bit; the kernel holds
// the largest register count of its bodies, which is what a group pays for sharing
// the launch.
struct BatchSlot {
  ElemArgs a;
  V2Args v;
  int64_t blk0;
  int32_t type, tile;
};
struct BatchPass {
  BatchSlot s[kMaxBatchSlots];
  int32_t n;
};
static_assert(sizeof(BatchPass) <= 4096, "batch pass arguments exceed the kernel parameter space");

// Slot of this block (block-uniform), the block's index among the slot's and their count.
__device__ __forceinline__ int slot_blocks(const BatchPass& P, unsigned& bid, unsigned& nblk) {
  int k = 0;
  while (k + 1 < P.n && static_cast<int64_t>(blockIdx.x) >= P.s[k + 1].blk0) ++k;
  const int64_t end = k + 1 < P.n ? P.s[k + 1].blk0 : static_cast<int64_t>(gridDim.x);
  bid = blockIdx.x - static_cast<unsigned>(P.s[k].blk0);
  nblk = static_cast<unsigned>(end - P.s[k].blk0);
  return k;
}

}  // namespace

// Per-family figures a batch launch needs: shared memory per block, elements per warp.
struct P1Shape {
  size_t smem = 0;
  int epw = 1;
};
// FP64 element pass (cxg_fp64.cu): one launch, and the batch kernel with its figures.
cudaError_t launch_p1_fp64(int t, int mode, const ElemArgs& a, const V2Args& v, const LaunchCfg& c, cudaStream_t s);
const void* p1_fp64_batch(int mode);
// After an element pass: nothing to do unless some element names a node twice.
cudaError_t launch_named_twice(int precision, const ElemArgs& a, const V2Args& v, cudaStream_t s);
P1Shape p1_fp64_shape(int t, int mode);

}  // namespace cxg
