// Fields from a displacement: recovery (recover_gauss_stress / recover_fields,
// src/fem/stress.cpp:147-271; linear elasticity), the thermal-strain load vector
// (thermal_strain_load_vector, src/fem/loads.cpp:515-560; element_thermal_load,
// element.cpp:636-665), and the compliance adjoint.
//
// Thermal strain, when the plan has it: te_k = T_k - t_ref at the element's nodes with an
// applied temperature (0 elsewhere), eps_th = alpha sum_k N_k te_k on the normal
// components at every Gauss point; the stress is D (eps - eps_th) and the element force
// sum_q detJ w sigma_q g_a is then K_e u_e - f_th_e. In thermal-load mode the element pass
// forms D eps_th instead (no displacement), and the node pass sums f_th.
//
// Adjoint. For K(theta) u = f with a load independent of the design and zero prescribed
// values, the compliance c = f^T u has dc/dtheta = -u^T (dK/dtheta) u, and u^T K_e u =
// sum_q s_q sigma_q : eps_q (s = w det J). Per Gauss point, with H = sum_k u_k (x) g_k, eps
// = sym(H), sigma = lam tr(eps) I + 2 mu eps, W = sigma : eps:
//   d/dE_e : u^T K_e u is linear in E (lam, mu proportional to E), so
//            dc/dE_e = -(1/E_e) sum_q s_q W_q;
//   d/dx_m : dg_k/dx_m = -g_m g_k^T (from J^-1 derivative), d(det J)/dx_m = det J g_m,
//            so d(s W)/dx_m = s (W I - 2 H^T sigma) g_m and dc/dx_m = -sum of that.
// The reference obtains the coordinate part by central differences of the assembled
// reduced operator (src/numerics/sensitivity.cpp:77-108); this is its closed form.
//
// Element pass: a warp takes as many elements as fill its lanes with (element, Gauss
// point) tasks: gradients, strain, and the 3x3 matrix T whose products with the gradients
// are the nodal values (s sigma, or minus s (W I - 2 H^T sigma)). Then lanes take (element,
// component) means over the points, which the hex and wedge families give every element
// node (extrapolation.hpp:34-41; C3D10 nodes get the corner extrapolation and midside
// averages of extrapolation.hpp:43-54), and (element, node) sums over the points.
// Node pass: one thread per node and component adds up the incident elements in element
// order (the order of the reference's element loop).
//
// One element per warp, its points on a quarter of the lanes, natural derivatives read
// from constant memory at a different address per lane, and for the adjoint a butterfly
// and an atomic per nodal value took 590 us for C3D20R 49x41x37 and 1300 us for the 96 x
// 96 x 48 C3D8 adjoint; with every lane on a task and plain sums 124 and 224 us, and the node
// passes 88 and 33.
#include <cuda_runtime.h>

#include <algorithm>

#include "cxg_element.cuh"

namespace cxg {

namespace {

enum FieldKind : int { RECOVER = 0, THERMAL_LOAD = 1, ADJOINT = 2 };

// Value sets of 12 (strain, stress) per element that the node pass reads: one per node
// for C3D10 (its corner extrapolation differs per node), one (the mean) otherwise.
template <int ET>
constexpr int rec_sets() {
  return ET == C3D10 ? nodes_of(ET) : 1;
}

template <int ET, int KIND>
struct FieldSmem {
  static constexpr int n = nodes_of(ET), nq = gauss_of(ET);
  static constexpr int EPB = 32 / nq;  // elements per warp
  // gradients [component][point][node], rows of odd length: the tasks' stores (a lane per
  // point) and the sums' loads (a lane per node) both spread over the banks
  static constexpr int ROW = n | 1, P = nq * ROW;
  static constexpr int ES = EPB == 1 ? 3 * P : (3 * P + 15) / 16 * 16 + 8;
  static constexpr int TS = KIND == ADJOINT ? 9 : 6;
  double g[EPB * ES];
  double T[EPB * nq * TS + 1];                     // Voigt s sigma, or the adjoint's 3x3
  double es[KIND == RECOVER ? EPB * nq * 12 : 1];  // strain, stress of the points
  double w[KIND == ADJOINT ? EPB * nq : 1];        // s W
  double x[EPB][3 * n];
  double u[KIND == THERMAL_LOAD ? 1 : EPB][3 * n];
  double te[KIND == ADJOINT ? 1 : EPB][n];
};

template <int ET, int KIND>
constexpr size_t field_smem_bytes() {
  constexpr int n = nodes_of(ET), nq = gauss_of(ET);
  return (sizeof(double) * (n * 3 * nq + nq + n * nq) + 15) / 16 * 16 +
         kW1 * ((sizeof(FieldSmem<ET, KIND>) + 15) / 16 * 16);
}

template <int ET, int KIND>
__global__ void __launch_bounds__(kT1) field_elem_kernel(ElemArgs A, double* gp_stress, double* emean, double* felem,
                                                         double* dc_dE) {
  using WS = FieldSmem<ET, KIND>;
  constexpr int n = WS::n, nq = WS::nq, EPB = WS::EPB, ROW = WS::ROW, P = WS::P, ES = WS::ES, TS = WS::TS;
  extern __shared__ __align__(16) unsigned char smem[];
  double* sdN = reinterpret_cast<double*>(smem);  // [n][3][nq]
  double* sw = sdN + n * 3 * nq;
  double* sN = sw + nq;  // [n][nq]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WS& W = *reinterpret_cast<WS*>(smem + (sizeof(double) * (n * 3 * nq + nq + n * nq) + 15) / 16 * 16 +
                                 warp * ((sizeof(WS) + 15) / 16 * 16));
  for (int i = threadIdx.x; i < n * 3 * nq; i += blockDim.x) sdN[i] = c_dN[dn_offset(ET) + i];
  for (int i = threadIdx.x; i < nq; i += blockDim.x) sw[i] = c_w[ET][i];
  for (int i = threadIdx.x; i < n * nq; i += blockDim.x) sN[i] = c_N[nn_offset(ET) + i];
  __syncthreads();
  const int64_t gwarp = static_cast<int64_t>(blockIdx.x) * kW1 + warp;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * kW1;
  for (int64_t e0 = gwarp * EPB; e0 < A.n_elems; e0 += nwarps * EPB) {
    for (int t = lane; t < EPB * n; t += 32) {
      const int ei = t / n, k = t % n;
      const int64_t e = e0 + ei;
      if (e >= A.n_elems) break;
      const int64_t node = A.conn[e0 * n + t];
      for (int d = 0; d < 3; ++d) {
        W.x[ei][3 * k + d] = A.coords[3 * node + d];
        if (KIND != THERMAL_LOAD) W.u[ei][3 * k + d] = A.u[3 * node + d];
      }
      if (KIND != ADJOINT)
        W.te[ei][k] = A.th_temp && A.th_alpha[e] != 0.0 && (!A.th_applied || A.th_applied[node])
                          ? A.th_temp[node] - A.th_tref[e]
                          : 0.0;
    }
    __syncwarp();
    for (int t = lane; t < EPB * nq; t += 32) {
      const int ei = t / nq, q = t % nq;
      const int64_t e = e0 + ei;
      if (e >= A.n_elems) continue;
      double J[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
      for (int k = 0; k < n; ++k) {
        const double d0 = sdN[(3 * k) * nq + q], d1 = sdN[(3 * k + 1) * nq + q], d2 = sdN[(3 * k + 2) * nq + q];
        for (int i = 0; i < 3; ++i) {
          const double xk = W.x[ei][3 * k + i];
          J[i][0] = fma(xk, d0, J[i][0]);
          J[i][1] = fma(xk, d1, J[i][1]);
          J[i][2] = fma(xk, d2, J[i][2]);
        }
      }
      double it[3][3];
      const double det = invert(J, it);
      if (!(det > 0.0)) {
        atomicCAS(&A.status->code, 0, 4);
        atomicMin(&A.status->bad_elem, static_cast<unsigned long long>(e));
      }
      double H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
      double* gq = W.g + ei * ES + q * ROW;
      for (int k = 0; k < n; ++k) {
        const double d0 = sdN[(3 * k) * nq + q], d1 = sdN[(3 * k + 1) * nq + q], d2 = sdN[(3 * k + 2) * nq + q];
        double gk[3];
        for (int i = 0; i < 3; ++i) {
          gk[i] = fma(it[i][0], d0, fma(it[i][1], d1, mul(it[i][2], d2)));
          gq[i * P + k] = gk[i];
        }
        if (KIND != THERMAL_LOAD)
          for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) H[i][j] = fma(W.u[ei][3 * k + i], gk[j], H[i][j]);
      }
      const double E = A.young[e], nu = A.poisson[e];
      const double um2 = E / (1.0 + nu);
      const double lam = nu * um2 / (1.0 - 2.0 * nu), mu = um2 / 2.0;
      const double s = det * sw[q];
      double* T = W.T + (ei * nq + q) * TS;
      if constexpr (KIND == ADJOINT) {
        double eps[3][3], sig[3][3];
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) eps[i][j] = 0.5 * (H[i][j] + H[j][i]);
        const double tr = eps[0][0] + eps[1][1] + eps[2][2];
        double wq = 0.0;
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) {
            sig[i][j] = 2.0 * mu * eps[i][j] + (i == j ? lam * tr : 0.0);
            wq += sig[i][j] * eps[i][j];
          }
        W.w[ei * nq + q] = s * wq;
        for (int a = 0; a < 3; ++a)
          for (int b = 0; b < 3; ++b) {
            double hs = 0.0;  // (H^T sigma)_{ab}
            for (int i = 0; i < 3; ++i) hs += H[i][a] * sig[i][b];
            T[3 * a + b] = -s * ((a == b ? wq : 0.0) - 2.0 * hs);
          }
      } else {
        double eth = 0.0;  // alpha sum_k N_k te_k
        if (A.th_temp && A.th_alpha[e] != 0.0) {
          double dT = 0.0;
          for (int k = 0; k < n; ++k) dT += sN[k * nq + q] * W.te[ei][k];
          eth = A.th_alpha[e] * dT;
        }
        const double st[6] = {H[0][0], H[1][1], H[2][2], H[0][1] + H[1][0], H[0][2] + H[2][0], H[1][2] + H[2][1]};
        // elastic strain: eps - eps_th, or eps_th itself in thermal-load mode (D eps_th)
        constexpr bool THL = KIND == THERMAL_LOAD;
        const double e0n = THL ? eth : st[0] - eth, e1n = THL ? eth : st[1] - eth, e2n = THL ? eth : st[2] - eth;
        const double tr = e0n + e1n + e2n;
        const double sg[6] = {lam * tr + 2.0 * mu * e0n, lam * tr + 2.0 * mu * e1n, lam * tr + 2.0 * mu * e2n,
                              THL ? 0.0 : mu * st[3],    THL ? 0.0 : mu * st[4],    THL ? 0.0 : mu * st[5]};
        for (int c = 0; c < 6; ++c) T[c] = s * sg[c];
        if constexpr (KIND == RECOVER) {
          double* es = W.es + (ei * nq + q) * 12;
          for (int c = 0; c < 6; ++c) {
            es[c] = st[c];
            es[6 + c] = sg[c];
          }
          if (gp_stress)
            for (int c = 0; c < 6; ++c) gp_stress[(e * nq + q) * 6 + c] = sg[c];
        }
      }
    }
    __syncwarp();
    if constexpr (KIND == ADJOINT) {
      if (dc_dE)
        for (int ei = lane; ei < EPB && e0 + ei < A.n_elems; ei += 32) {
          double tot = 0.0;
          for (int q = 0; q < nq; ++q) tot += W.w[ei * nq + q];
          dc_dE[e0 + ei] = -tot / A.young[e0 + ei];
        }
    }
    if constexpr (KIND == RECOVER) {
      if (emean) {
        if constexpr (ET == C3D10) {
          // corners: the a4 extrapolation matrix of CalculiX extrapolate.f; midsides: the
          // mean of their edge's corners (extrapolation.hpp:18-55)
          constexpr double kA4diag = 1.927050983124842, kA4off = -0.309016994374947;
          constexpr int kMid[6][2] = {{0, 1}, {1, 2}, {2, 0}, {0, 3}, {1, 3}, {2, 3}};
          for (int t = lane; t < EPB * n * 12; t += 32) {
            const int ei = t / (n * 12), i = t / 12 % n, c = t % 12;
            if (e0 + ei >= A.n_elems) break;
            auto corner = [&](int cn) {
              double v = 0.0;
              for (int l = 0; l < 4; ++l) v += (cn == l ? kA4diag : kA4off) * W.es[(ei * nq + l) * 12 + c];
              return v;
            };
            emean[e0 * (n * 12) + t] = i < 4 ? corner(i) : 0.5 * (corner(kMid[i - 4][0]) + corner(kMid[i - 4][1]));
          }
        } else {
          for (int t = lane; t < EPB * 12; t += 32) {
            const int ei = t / 12, c = t % 12;
            if (e0 + ei >= A.n_elems) break;
            double m = 0.0;
            for (int q = 0; q < nq; ++q) m += W.es[(ei * nq + q) * 12 + c];
            emean[e0 * 12 + t] = m * (1.0 / nq);
          }
        }
      }
    }
    if (felem)
      for (int t = lane; t < EPB * n; t += 32) {
        const int ei = t / n, a = t % n;
        if (e0 + ei >= A.n_elems) break;
        const double* ga = W.g + ei * ES + a;
        double f[3] = {0.0, 0.0, 0.0};
        for (int q = 0; q < nq; ++q) {
          const double* T = W.T + (ei * nq + q) * TS;
          const double gx = ga[q * ROW], gy = ga[P + q * ROW], gz = ga[2 * P + q * ROW];
          if constexpr (KIND == ADJOINT) {
            for (int d = 0; d < 3; ++d) f[d] += T[3 * d] * gx + T[3 * d + 1] * gy + T[3 * d + 2] * gz;
          } else {
            add_force(f, T, gx, gy, gz);
          }
        }
        for (int d = 0; d < 3; ++d) felem[(e0 * n + t) * 3 + d] = f[d];
      }
    __syncwarp();
  }
}

// Values per node that the node pass forms: 0..5 strain, 6..11 stress, 12..14 force.
template <int ET>
__global__ void __launch_bounds__(256) field_node_kernel(ElemArgs A, const int64_t* inc_ptr, const int32_t* inc_code,
                                                         const double* emean, const double* felem, const double* f_ext,
                                                         double* strain, double* stress, double* reaction, int first) {
  constexpr int n = nodes_of(ET);
  const int per = 15 - first;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < per * A.n_nodes;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t a = t / per;
    const int c = first + static_cast<int>(t % per);
    double* out = c < 6 ? strain : c < 12 ? stress : reaction;
    if (!out) continue;
    const int64_t i0 = inc_ptr[a], i1 = inc_ptr[a + 1];
    double v = 0.0;
    if (c < 12) {
#pragma unroll 4
      for (int64_t i = i0; i < i1; ++i) {
        const int code = __ldg(inc_code + i);
        v += emean[static_cast<int64_t>(rec_sets<ET>() == 1 ? code / n : code) * 12 + c];
      }
      out[6 * a + c % 6] = i1 > i0 ? v / static_cast<double>(i1 - i0) : 0.0;
    } else {
      const int d = c - 12;
#pragma unroll 4
      for (int64_t i = i0; i < i1; ++i) v += felem[3 * static_cast<int64_t>(__ldg(inc_code + i)) + d];
      out[3 * a + d] = v - (f_ext ? f_ext[3 * a + d] : 0.0);
    }
  }
}

template <int ET, int KIND>
cudaError_t launch_elem(const ElemArgs& a, double* gp_stress, double* emean, double* felem, double* dc_dE,
                        cudaStream_t s) {
  if (a.n_elems == 0) return cudaSuccess;
  auto kern = field_elem_kernel<ET, KIND>;
  constexpr size_t smem = field_smem_bytes<ET, KIND>();
  static_assert(smem <= 227 * 1024, "field pass shared memory");
  int per_sm = 0, sms = 0;
  const cudaError_t err = kernel_shape(reinterpret_cast<const void*>(kern), kT1, smem, &per_sm, &sms);
  if (err != cudaSuccess) return err;
  constexpr int per_block = kW1 * FieldSmem<ET, KIND>::EPB;
  const int64_t grid = persistent_grid((a.n_elems + per_block - 1) / per_block, per_sm, sms, 0);
  kern<<<static_cast<unsigned>(grid), kT1, smem, s>>>(a, gp_stress, emean, felem, dc_dE);
  return cudaGetLastError();
}

template <int ET>
cudaError_t launch_nodes(const ElemArgs& a, const int64_t* inc_ptr, const int32_t* inc_code, const double* emean,
                         const double* felem, const double* f_ext, double* strain, double* stress, double* reaction,
                         cudaStream_t s) {
  const int first = emean && (strain || stress) ? 0 : 12;
  const int64_t count = (15 - first) * a.n_nodes;
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((count + 255) / 256, 148 * 8));
  field_node_kernel<ET><<<static_cast<unsigned>(grid), 256, 0, s>>>(a, inc_ptr, inc_code, emean, felem, f_ext, strain,
                                                                   stress, reaction, first);
  return cudaGetLastError();
}

template <int ET>
cudaError_t launch_recover_t(const ElemArgs& a, const int64_t* inc_ptr, const int32_t* inc_code, double* gp_stress,
                             double* emean, double* felem, const double* f_ext, double* strain, double* stress,
                             double* reaction, bool thermal_load, cudaStream_t s) {
  const cudaError_t err = thermal_load ? launch_elem<ET, THERMAL_LOAD>(a, nullptr, nullptr, felem, nullptr, s)
                                       : launch_elem<ET, RECOVER>(a, gp_stress, emean, felem, nullptr, s);
  if (err != cudaSuccess || !felem || !inc_ptr) return err;
  return launch_nodes<ET>(a, inc_ptr, inc_code, emean, felem, f_ext, strain, stress, reaction, s);
}

template <int ET>
cudaError_t launch_adjoint_t(const ElemArgs& a, const int64_t* inc_ptr, const int32_t* inc_code, double* felem,
                             double* dc_dE, double* dc_dX, cudaStream_t s) {
  const cudaError_t err = launch_elem<ET, ADJOINT>(a, nullptr, nullptr, dc_dX ? felem : nullptr, dc_dE, s);
  if (err != cudaSuccess || !dc_dX) return err;
  return launch_nodes<ET>(a, inc_ptr, inc_code, nullptr, felem, nullptr, nullptr, nullptr, dc_dX, s);
}

}  // namespace

cudaError_t launch_recover(int t, const ElemArgs& a, const int64_t* inc_ptr, const int32_t* inc_code,
                           double* gp_stress, double* emean, double* felem, const double* f_ext, double* strain,
                           double* stress, double* reaction, bool thermal_load, cudaStream_t s) {
  switch (t) {
#define CXG_REC(T)                                                                                             \
  case T:                                                                                                      \
    return launch_recover_t<T>(a, inc_ptr, inc_code, gp_stress, emean, felem, f_ext, strain, stress, reaction, \
                               thermal_load, s);
    CXG_REC(C3D4)
    CXG_REC(C3D10)
    CXG_REC(C3D8)
    CXG_REC(C3D8R)
    CXG_REC(C3D20)
    CXG_REC(C3D20R)
    CXG_REC(C3D6)
    CXG_REC(C3D15)
#undef CXG_REC
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_adjoint(int t, const ElemArgs& a, const int64_t* inc_ptr, const int32_t* inc_code, double* felem,
                           double* dc_dE, double* dc_dX, cudaStream_t s) {
  switch (t) {
#define CXG_ADJ(T) \
  case T:          \
    return launch_adjoint_t<T>(a, inc_ptr, inc_code, felem, dc_dE, dc_dX, s);
    CXG_ADJ(C3D4)
    CXG_ADJ(C3D10)
    CXG_ADJ(C3D8)
    CXG_ADJ(C3D20)
    CXG_ADJ(C3D20R)
    CXG_ADJ(C3D6)
    CXG_ADJ(C3D15)
#undef CXG_ADJ
    default: return cudaErrorNotSupported;
  }
}

}  // namespace cxg
