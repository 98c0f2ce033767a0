// The element pass in mixed precision, and the dispatch of both passes of an assembly:
// P1 integrates the elements, P2 (the row gather, cxg_gather.cu) writes every CSR value
// once, with no atomics. P1 in FP64 is in cxg_fp64.cu.
//
// Each warp integrates EPW elements at once. Lanes first handle (element, Gauss point)
// tasks: Jacobian, its inverse and the physical gradients in FP64 (plus the J2 return in
// material-point mode, whose trial history is written here, once per Gauss point). Then
// every lane owns a tile of node pairs of one element and accumulates their 3x3 blocks of
// K_e in FP32 registers over the Gauss points from float4 gradient loads; elastic points
// use the Gram form K_ab = lam G + mu (G^T + tr(G) I) with G = sum_q s_q g_a g_b^T,
// plastic elements the full tangent sum_q s [lam* g_a g_b^T + mu* (g_b g_a^T +
// (g_a.g_b) I) - c m_a m_b^T] (m = N g, N the return direction, formed in the tile loop
// from the gradients and the stored N of the Gauss point). The upper blocks (a <= b) go to
// a per-element buffer; the internal force goes beside them in FP64.
//
// What bounds it: the shared-memory pipe (78 % busy on C3D20), since every tile reads the
// Gauss points' gradients again. Staging the finished blocks and sending them as one bulk
// copy per element took C3D20 64^3 from 1583 to 1525 us, and lets the gather read blocks
// without padding. The rounding sequence of a block is the same for every tile shape.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>

#include "cxg_element.cuh"

namespace cxg {

namespace {

struct TileList {
  int count;
  unsigned char r[64];
  unsigned char c[64];
};

// Node-pair tiles of TR rows x TC columns covering the upper triangle (a <= b).
constexpr TileList make_tiles(int n, int TR, int TC) {
  TileList t{};
  const int npad = (n + 3) / 4 * 4;
  for (int r = 0; r < npad / TR; ++r)
    for (int c = 0; c < npad / TC; ++c) {
      bool any = false;
      for (int i = 0; i < TR; ++i)
        for (int j = 0; j < TC; ++j) {
          const int a = TR * r + i, b = TC * c + j;
          if (a < n && b < n && a <= b) any = true;
        }
      if (any) {
        t.r[t.count] = static_cast<unsigned char>(r);
        t.c[t.count] = static_cast<unsigned char>(c);
        ++t.count;
      }
    }
  return t;
}

// Tile shapes of the element pass (TILE codes): 0 = 2x4 (default), 1 = 2x2, 2 = 4x4.
constexpr int tile_rows(int tile) { return tile == 2 ? 4 : 2; }
constexpr int tile_cols(int tile) { return tile == 1 ? 2 : 4; }

template <int ET, int TILE = 0>
struct Geo {
  static constexpr int n = nodes_of(ET);
  static constexpr int nq = gauss_of(ET);
  static constexpr int npad = (n + 3) / 4 * 4;
  static constexpr int NB = n * (n + 1) / 2;
  static constexpr int TR = tile_rows(TILE), TC = tile_cols(TILE);
  static constexpr TileList tiles = make_tiles(n, TR, TC);
  static constexpr int NT = tiles.count;
  static constexpr int EPW = NT >= 32 ? 1 : 32 / NT;
};

// Band around the yield surface, as a fraction of the current yield stress, inside which
// the mixed-precision path decides and returns in FP64.
constexpr float kYieldBandFp32 = 1e-3f;

// J2 return of the mixed-precision path: the same steps as j2_point
// (src/fem/plasticity.cpp:90-236) with the trial stress, the local Newton on the plastic
// multiplier, the stress and history update and the consistent-tangent parameters in
// FP32. The consistency scalar f = q_tr - sigma_y(ep0) decides the branch in FP32 only
// when |f| exceeds kYieldBandFp32 * sigma_y, clear of the FP32 rounding of q_tr; points
// inside the band, and points whose FP32 Newton does not settle, take the FP64 return:
// the function then returns kJ2Fp64 and writes nothing, and the caller runs j2_point (one
// call site, so the FP64 return is inlined once). Else it returns 1 for a plastic step and
// 0 for an elastic one. The hardening table is read in FP64 (it is indexed by the FP64
// history).
constexpr int kJ2Fp64 = 2;
__device__ __forceinline__ int j2_point_mixed(const J2Mat& M, double lam, double mu_el, double mu, const double* eps,
                               const double* cs, double* ts, double* sig, double& lam_t, double& mu_t,
                               double& c_t, double* nv, double& mu_hg) {
  const float l = static_cast<float>(lam), me = static_cast<float>(mu_el), m = static_cast<float>(mu);
  const float hk = static_cast<float>(M.h_kin);
  float el[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) el[i] = static_cast<float>(eps[i] - cs[i]);
  const float l2m = l + 2.0f * me;
  float st[6];
  st[0] = l2m * el[0] + l * el[1] + l * el[2];
  st[1] = l * el[0] + l2m * el[1] + l * el[2];
  st[2] = l * el[0] + l * el[1] + l2m * el[2];
  st[3] = me * el[3];
  st[4] = me * el[4];
  st[5] = me * el[5];
  const float p = (st[0] + st[1] + st[2]) / 3.0f;
  const float s_tr[6] = {st[0] - p, st[1] - p, st[2] - p, st[3], st[4], st[5]};
  float xi[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) xi[i] = s_tr[i] - static_cast<float>(cs[7 + i]);
  const float xi_norm = sqrtf(xi[0] * xi[0] + xi[1] * xi[1] + xi[2] * xi[2] +
                              2.0f * (xi[3] * xi[3] + xi[4] * xi[4] + xi[5] * xi[5]));
  const float sq32 = static_cast<float>(kSqrt3_2v2);
  const float q_tr = sq32 * xi_norm;
  double sy0 = 0.0, h0 = 0.0;
  if (M.plastic) hardening2(M, cs[6], sy0, h0);
  const float f = q_tr - static_cast<float>(sy0);
  if (M.plastic && fabsf(f) <= kYieldBandFp32 * static_cast<float>(sy0)) return kJ2Fp64;
  if (!M.plastic || f <= 0.0f || xi_norm == 0.0f) {
#pragma unroll
    for (int i = 0; i < 6; ++i) sig[i] = st[i];
#pragma unroll
    for (int i = 0; i < kStateDoubles; ++i) ts[i] = cs[i];
    lam_t = lam;
    mu_t = mu_el;
    c_t = 0.0;
    mu_hg = mu_el;
    return 0;
  }
  const double ep0 = cs[6];
  float dgamma = 0.0f;
  bool settled = false;
  for (int it = 0; it < 50; ++it) {
    double sy, h_iso;
    hardening2(M, ep0 + dgamma, sy, h_iso);
    const float g = q_tr - 3.0f * m * dgamma - hk * dgamma - static_cast<float>(sy);
    const float dg = -(3.0f * m + hk + static_cast<float>(h_iso));
    const float step = -g / dg;
    dgamma += step;
    if (dgamma < 0.0f) dgamma = 0.0f;
    if (fabsf(step) <= 4e-7f * dgamma) {
      settled = true;
      break;
    }
  }
  if (!settled) return kJ2Fp64;
  float n32[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) n32[i] = xi[i] / xi_norm;
  const float dev_scale = 2.0f * m * dgamma * sq32;
  const float alpha_scale = (2.0f / 3.0f) * hk * dgamma * sq32;
  const float dep_scale = dgamma * sq32;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    nv[i] = n32[i];
    sig[i] = (s_tr[i] - dev_scale * n32[i]) + (i < 3 ? p : 0.0f);
    ts[i] = cs[i] + static_cast<double>(dep_scale * n32[i] * (i < 3 ? 1.0f : 2.0f));
    ts[7 + i] = cs[7 + i] + static_cast<double>(alpha_scale * n32[i]);
  }
  ts[6] = ep0 + static_cast<double>(dgamma);
  double sy, h_iso;
  hardening2(M, ep0 + dgamma, sy, h_iso);
  const float theta = 1.0f - dev_scale / xi_norm;
  const float denom = 1.0f + (static_cast<float>(h_iso) + hk) / (3.0f * m);
  const float theta_bar = 1.0f / denom - (1.0f - theta);
  const float lt = l + (2.0f / 3.0f) * (1.0f - theta) * m;
  const float mt = me - (1.0f - theta) * m;
  const float ct = 2.0f * m * theta_bar;
  lam_t = lt;
  mu_t = mt;
  c_t = ct;
  mu_hg = mt - ct * n32[3] * n32[3];
  return 1;
}

// Shared-memory layout of per-(element, Gauss point) node vectors: node k lives in
// slot(k) = k/2 for even k and npad/2 + k/2 for odd k, so the row nodes 2r + i of the
// lanes' tiles occupy consecutive slots, float4 each: one warp-wide vector load touches
// distinct banks. The plane block of each (element, Gauss point) is followed by 16 bytes of
// padding: the blocks then start 16 (mod 128) bytes apart, so the lanes of the Gauss-point
// phase, one block each, store their vectors into 8 distinct 16-byte bank groups.
__host__ __device__ constexpr int node_slot(int k, int npad) { return (k & 1) ? npad / 2 + (k >> 1) : (k >> 1); }

template <typename R, int NPAD>
struct VecIdx {
  static_assert(sizeof(R) == 4, "FP32 pass");
  // elements of one plane block (b = element*nq + q), padding included
  static constexpr int kBlock = NPAD * 4 + 4;
  // flat index of component c of the vector in `slot` of plane block b
  __device__ __forceinline__ static int at(int b, int slot, int c) { return b * kBlock + slot * 4 + c; }
};

// one vector store (x, y, z, 0) of a node vector
template <typename R, int NPAD>
__device__ __forceinline__ void st3(R* base, int b, int slot, double x, double y, double z) {
  *reinterpret_cast<float4*>(base + VecIdx<R, NPAD>::at(b, slot, 0)) =
      make_float4(static_cast<float>(x), static_cast<float>(y), static_cast<float>(z), 0.f);
}

template <typename R, int NPAD>
__device__ __forceinline__ void ld3(const R* base, int b, int slot, R& x, R& y, R& z) {
  const float4 v = *reinterpret_cast<const float4*>(base + VecIdx<R, NPAD>::at(b, slot, 0));
  x = v.x;
  y = v.y;
  z = v.z;
}

template <int ET, int MODE, typename R, int TILE>
struct P1Smem {
  using G = Geo<ET, TILE>;
  static constexpr int n = G::n, nq = G::nq, npad = G::npad, EPW = G::EPW;
  static constexpr bool T = MODE == MODE_TANGENT;
  // Staged blocks: the finished blocks of a warp's elements are put together in shared
  // memory, unpadded, and leave as one bulk copy per element. With one tile per lane
  // (ALIAS) they take the place of the gradient vectors, which are dead by then.
  static constexpr int kElem = blocks_padded(n) * 9;  // values of one element
  static constexpr bool ALIAS = EPW * G::NT <= 32;
  static constexpr int kGrad = EPW * nq * VecIdx<R, npad>::kBlock;
  static constexpr int kVec = ALIAS && EPW * kElem > kGrad ? EPW * kElem : kGrad;
  static constexpr int HG = ET == C3D8R ? EPW : 1;  // hourglass data (C3D8R only)
  alignas(16) R g[kVec];                          // node vectors, see VecIdx
  alignas(16) R stg[ALIAS ? 4 : EPW * kElem];
  R nvq[T ? EPW * nq * 8 : 4];  // return direction N (Voigt, 6 used) per plastic Gauss point
  R s[EPW][nq];
  R dp[T ? EPW : 1][T ? nq : 1][4];
  double x[EPW][3 * n];
  double u[T ? EPW : 1][T ? 3 * n : 1];
  double sig[T ? EPW : 1][T ? nq : 1][6];
  double lam[EPW], mu[EPW], mu_j2[EPW];
  double gam[HG][32];
  double kappa[HG];
  double gc[HG][3 * n];
  double vol[HG];
  double mu_hg[HG];
  int plastic[EPW];
  int id[EPW][n];  // mesh nodes
};

template <int ET, int MODE, typename R, int TILE>
constexpr size_t p1_smem_bytes() {
  using WS = P1Smem<ET, MODE, R, TILE>;
  constexpr int n = nodes_of(ET), nq = gauss_of(ET);
  return (sizeof(double) * (n * 3 * nq + nq) + 15) / 16 * 16 + kW1 * ((sizeof(WS) + 15) / 16 * 16);
}

// Resident blocks per SM the element pass asks the register allocator for: as many as
// its shared memory allows, at most 3 (<= 170 registers per thread) for the tiles whose
// accumulators fit that budget without spilling (2x2 and 2x4), else 2 (no limit below the
// 255-register ceiling). The material-point pass takes 4 (<= 128 registers): it spills 28
// bytes per thread there and still ran 10 % faster on the C3D8 J2 block.
template <int ET, int MODE, typename R, int TILE>
constexpr int p1_min_blocks() {
  constexpr size_t per_sm = 227 * 1024;
  constexpr int by_smem = static_cast<int>(per_sm / (p1_smem_bytes<ET, MODE, R, TILE>() + 1024));
  constexpr int cap = MODE == MODE_TANGENT ? 4 : TILE <= 1 ? 3 : 2;
  return by_smem < 1 ? 1 : (by_smem > cap ? cap : by_smem);
}

// J2F32 (mixed-precision material-point pass only): the J2 return in FP32
// (j2_point_mixed) instead of FP64.
// bid / nblk: this block's index among the nblk blocks that share the element range.
template <int ET, int MODE, typename R, int TILE, bool J2F32>
__device__ __forceinline__ void p1_body(const ElemArgs& A, const V2Args& V, unsigned bid, unsigned nblk) {
  using G = Geo<ET, TILE>;
  constexpr int n = G::n, nq = G::nq, npad = G::npad, EPW = G::EPW, NT = G::NT, NB = G::NB;
  constexpr int TR = G::TR, TC = G::TC;
  constexpr bool TAN = MODE == MODE_TANGENT;
  using WS = P1Smem<ET, MODE, R, TILE>;
  extern __shared__ __align__(16) unsigned char smem[];
  double* sdN = reinterpret_cast<double*>(smem);  // [n][3][nq]
  double* sw = sdN + n * 3 * nq;
  constexpr size_t cta_bytes = (sizeof(double) * (n * 3 * nq + nq) + 15) / 16 * 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WS& W = *reinterpret_cast<WS*>(smem + cta_bytes + warp * ((sizeof(WS) + 15) / 16 * 16));
  __shared__ unsigned char s_tr[64], s_tc[64];
  for (int i = threadIdx.x; i < n * 3 * nq; i += blockDim.x) sdN[i] = c_dN[dn_offset(ET) + i];
  for (int i = threadIdx.x; i < nq; i += blockDim.x) sw[i] = c_w[ET][i];
  if (threadIdx.x == 0) {
    constexpr TileList tl = make_tiles(n, TR, TC);
    for (int i = 0; i < NT; ++i) {
      s_tr[i] = tl.r[i];
      s_tc[i] = tl.c[i];
    }
  }
  // zero the padded gradient slots once; they are never written afterwards
  for (int t = lane; t < WS::kVec; t += 32) {
    W.g[t] = R(0);
  }
  __syncthreads();

  const int64_t gwarp = static_cast<int64_t>(bid) * kW1 + warp;
  const int64_t nwarps = static_cast<int64_t>(nblk) * kW1;
  const int64_t e_end = V.e_end;  // elements [V.e_begin, V.e_end) of this window
  // The connectivity of a warp's next elements is loaded while it integrates the current
  // ones, so the coordinate gather of the next iteration waits for one round of loads.
  constexpr int PA = (EPW * n + 31) / 32;
  int conn_next[PA];
  auto load_conn = [&](int64_t e0x) {
#pragma unroll
    for (int p = 0; p < PA; ++p) {
      const int t = lane + 32 * p;
      const int64_t e = e0x + t / n;
      conn_next[p] = t < EPW * n && e < e_end ? A.conn[e * n + t % n] : -1;
    }
  };
  wait_for_kernel_before();
  // Only in a launch of one batch per warp: blocks of the gather that settle beside a longer
  // element pass would run in the little L1 its shared memory leaves (C3D20 64^3 mixed 3530
  // -> 3706 us an assembly).
  if (e_end - V.e_begin <= nwarps * EPW) let_next_kernel_start();
  load_conn(V.e_begin + gwarp * EPW);
  for (int64_t e0 = V.e_begin + gwarp * EPW; e0 < e_end; e0 += nwarps * EPW) {
    // ---- phase A ---------------------------------------------------------------
#pragma unroll
    for (int p = 0; p < PA; ++p) {
      const int t = lane + 32 * p;
      const int node = conn_next[p];
      if (node >= 0) {
        const int ei = t / n, k = t % n;
        W.id[ei][k] = node;
        for (int d = 0; d < 3; ++d) {
          W.x[ei][3 * k + d] = A.coords[3 * static_cast<int64_t>(node) + d];
          if (TAN) W.u[ei][3 * k + d] = A.u[3 * static_cast<int64_t>(node) + d];
        }
      }
    }
    load_conn(e0 + nwarps * EPW);
    if (lane == 0) bulk_wait_read();  // the staged blocks of the last elements have left
    if (lane < EPW) {
      const int64_t e = e0 + lane;
      const double E = e < e_end ? A.young[e] : 1.0, nu = e < e_end ? A.poisson[e] : 0.0;
      const double um2 = E / (1.0 + nu);
      W.lam[lane] = nu * um2 / (1.0 - 2.0 * nu);
      W.mu[lane] = um2 / 2.0;
      W.mu_j2[lane] = E / (2.0 * (1.0 + nu));
      W.plastic[lane] = 0;
    }
    __syncwarp();
    // ---- phase B: (element, Gauss point) tasks ----------------------------------------
    for (int t = lane; t < EPW * nq; t += 32) {
      const int ei = t / nq, q = t % nq;
      const int64_t e = e0 + ei;
      if (e >= e_end) continue;
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
      const double sq = mul(det, sw[q]);
      W.s[ei][q] = static_cast<R>(sq);
      if constexpr (ET == C3D8R) W.vol[ei] = sq;
      double H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
      for (int k = 0; k < n; ++k) {
        const double d0 = sdN[(3 * k) * nq + q], d1 = sdN[(3 * k + 1) * nq + q], d2 = sdN[(3 * k + 2) * nq + q];
        double gk[3];
        for (int i = 0; i < 3; ++i) {
          gk[i] = fma(it[i][0], d0, fma(it[i][1], d1, mul(it[i][2], d2)));
          if constexpr (ET == C3D8R) W.gc[ei][i * n + k] = gk[i];
        }
        st3<R, npad>(W.g, ei * nq + q, node_slot(k, npad), gk[0], gk[1], gk[2]);
        if (TAN)
          for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) H[i][j] = fma(W.u[ei][3 * k + i], gk[j], H[i][j]);
      }
      if (TAN) {
        const double eps[6] = {H[0][0], H[1][1], H[2][2], H[0][1] + H[1][0], H[0][2] + H[2][0], H[1][2] + H[2][1]};
        const int mat = A.elem_mat ? A.elem_mat[e] : 0;
        const int64_t gidx = e * nq + q;
        double cs[kStateDoubles], ts[kStateDoubles], sig[6], nv[6] = {0, 0, 0, 0, 0, 0};
        // plastic strain and equivalent plastic strain always; the back stress only when
        // some material moves it (state_comps 13), else it is zero
        const bool back = A.state_comps > 7;
#pragma unroll
        for (int c = 0; c < 7; ++c) cs[c] = A.state_c[c * A.n_gauss + gidx];
        if (back) {
#pragma unroll
          for (int c = 7; c < kStateDoubles; ++c) cs[c] = A.state_c[c * A.n_gauss + gidx];
        } else {
#pragma unroll
          for (int c = 7; c < kStateDoubles; ++c) cs[c] = 0.0;
        }
        double lt, mt, ct, mhg;
        // FP64 return, or with J2F32 the FP32 return (with the FP64 band near yield)
        const int r = !J2F32 ? kJ2Fp64
                             : j2_point_mixed(A.mats[mat], W.lam[ei], W.mu[ei], W.mu_j2[ei], eps, cs, ts, sig, lt, mt, ct,
                                              nv, mhg);
        const bool pl = r == kJ2Fp64
                            ? j2_point(A.mats[mat], W.lam[ei], W.mu[ei], W.mu_j2[ei], eps, cs, ts, sig, lt, mt, ct, nv, mhg)
                            : r != 0;
#pragma unroll
        for (int c = 0; c < 7; ++c) A.state_t[c * A.n_gauss + gidx] = ts[c];
        if (back) {
#pragma unroll
          for (int c = 7; c < kStateDoubles; ++c) A.state_t[c * A.n_gauss + gidx] = ts[c];
        }
        for (int c = 0; c < 6; ++c) W.sig[ei][q][c] = mul(sq, sig[c]);
        W.dp[ei][q][0] = static_cast<R>(sq * lt);
        W.dp[ei][q][1] = static_cast<R>(sq * mt);
        W.dp[ei][q][2] = static_cast<R>(sq * ct);
        if (pl) {
          W.plastic[ei] = 1;
#pragma unroll
          for (int c = 0; c < 6; ++c) W.nvq[(ei * nq + q) * 8 + c] = static_cast<R>(nv[c]);
        }
        if constexpr (ET == C3D8R) {
          if (q == nq - 1) W.mu_hg[ei] = mhg;
        }
      }
    }
    __syncwarp();
    // ---- C3D8R hourglass vectors (src/fem/element.cpp:545-579) ------------------------
    if constexpr (ET == C3D8R) {
      for (int t = lane; t < EPW * 4; t += 32) {
        const int ei = t / 4, al = t % 4;
        double gx[3] = {0, 0, 0};
        for (int j = 0; j < 8; ++j)
          for (int d = 0; d < 3; ++d) gx[d] = fma(c_hg2[al][j], W.x[ei][3 * j + d], gx[d]);
        for (int j = 0; j < 8; ++j) {
          double corr = 0.0;
          for (int d = 0; d < 3; ++d) corr = fma(gx[d], W.gc[ei][d * n + j], corr);
          W.gam[ei][al * 8 + j] = c_hg2[al][j] - corr;
        }
      }
      if (lane < EPW) {
        double b2 = 0.0;
        for (int t = 0; t < 3 * n; ++t) b2 = fma(W.gc[lane][t], W.gc[lane][t], b2);
        W.kappa[lane] = 0.05 * (TAN ? W.mu_hg[lane] : W.mu_j2[lane]) * W.vol[lane] * b2;
      }
      __syncwarp();
    }
    // ---- internal force per element (material-point mode) --------------------
    if (TAN) {
      for (int t = lane; t < EPW * n; t += 32) {
        const int ei = t / n, a = t % n;
        const int64_t e = e0 + ei;
        if (e >= e_end) continue;
        double f[3] = {0, 0, 0};
        for (int q = 0; q < nq; ++q) {
          const double* S = W.sig[ei][q];
          R rx, ry, rz;
          ld3<R, npad>(W.g, ei * nq + q, node_slot(a, npad), rx, ry, rz);
          const double gx = rx, gy = ry, gz = rz;
          add_force(f, S, gx, gy, gz);
        }
        if constexpr (ET == C3D8R) {
          for (int al = 0; al < 4; ++al) {
            double gu[3] = {0, 0, 0};
            for (int j = 0; j < 8; ++j)
              for (int d = 0; d < 3; ++d) gu[d] = fma(W.gam[ei][al * 8 + j], W.u[ei][3 * j + d], gu[d]);
            const double ka = mul(W.kappa[ei], W.gam[ei][al * 8 + a]);
            for (int d = 0; d < 3; ++d) f[d] = fma(ka, gu[d], f[d]);
          }
        }
        for (int d = 0; d < 3; ++d) V.fdata[ring_slot(e, V) * (3 * n) + 3 * a + d] = f[d];
      }
    }
    // ---- phase C: TR x TC node-pair tiles ---------------------------------------------
    // Blocks are staged in shared memory and leave as bulk copies: a lane that writes its
    // own blocks to the element's buffer touches about one cache line per lane and store
    // instruction, and the gather would read the padding that aligns such stores.
    R* stg = WS::ALIAS ? W.g : W.stg;
    R acc[TR][TC][9];
    auto stage_tile = [&](int task) {
      const int ei = task / NT, ti = task % NT, a0 = TR * s_tr[ti], b0 = TC * s_tc[ti];
#pragma unroll
      for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          const int a = a0 + i, b = b0 + j;
          if (a < n && b < n && a <= b) {
            R h = R(0);
            if constexpr (ET == C3D8R) {
              double hd = 0.0;
              for (int al = 0; al < 4; ++al) hd = fma(W.gam[ei][al * 8 + a], W.gam[ei][al * 8 + b], hd);
              h = static_cast<R>(hd * W.kappa[ei]);
            }
            // FP32 diagonal blocks are not used: the gather forms them (GATHER_DIAG)
            const bool drop = a == b;
            R* d = stg + ei * WS::kElem + blk_index(n, a, b) * 9;
            // in mesh order of the two nodes: transposed when b precedes a
            const int na = W.id[ei][a], nb = W.id[ei][b], sx = na > nb ? 1 : 3, sy = 4 - sx;
#pragma unroll
            for (int x = 0; x < 3; ++x)
#pragma unroll
              for (int y = 0; y < 3; ++y)
                d[x * sx + y * sy] = drop ? R(0) : acc[i][j][3 * x + y] + (x == y ? h : R(0));
          }
        }
    };
    for (int task = lane; task < EPW * NT; task += 32) {
      const int ei = task / NT, ti = task % NT;
      const int64_t e = e0 + ei;
      if (e < e_end) {
        const int a0 = TR * s_tr[ti], b0 = TC * s_tc[ti];
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
          for (int j = 0; j < TC; ++j)
#pragma unroll
            for (int k = 0; k < 9; ++k) acc[i][j][k] = R(0);
        const bool pl = TAN && W.plastic[ei];
        if (!pl) {
#pragma unroll 3
          for (int q = 0; q < nq; ++q) {
            const R s = W.s[ei][q];
            R ga[TR][3], gb[TC][3];
#pragma unroll
            for (int i = 0; i < TR; ++i) {
              ld3<R, npad>(W.g, ei * nq + q, node_slot(a0 + i, npad), ga[i][0], ga[i][1], ga[i][2]);
              ga[i][0] *= s;
              ga[i][1] *= s;
              ga[i][2] *= s;
            }
#pragma unroll
            for (int j = 0; j < TC; ++j)
              ld3<R, npad>(W.g, ei * nq + q, node_slot(b0 + j, npad), gb[j][0], gb[j][1], gb[j][2]);
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
              for (int j = 0; j < TC; ++j)
#pragma unroll
                for (int x = 0; x < 3; ++x)
#pragma unroll
                  for (int y = 0; y < 3; ++y) acc[i][j][3 * x + y] += ga[i][x] * gb[j][y];
          }
          const R lam = static_cast<R>(W.lam[ei]), mu = static_cast<R>(W.mu[ei]);
#pragma unroll
          for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) {
              R Gm[9];
#pragma unroll
              for (int k = 0; k < 9; ++k) Gm[k] = acc[i][j][k];
              const R tr = Gm[0] + Gm[4] + Gm[8];
#pragma unroll
              for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y)
                  acc[i][j][3 * x + y] = lam * Gm[3 * x + y] + mu * Gm[3 * y + x] + (x == y ? mu * tr : R(0));
            }
        } else if (TAN) {
          for (int q = 0; q < nq; ++q) {
            const R sl = W.dp[ei][q][0], sm = W.dp[ei][q][1], sc = W.dp[ei][q][2];
            R ga[TR][3], gb[TC][3];
#pragma unroll
            for (int i = 0; i < TR; ++i)
              ld3<R, npad>(W.g, ei * nq + q, node_slot(a0 + i, npad), ga[i][0], ga[i][1], ga[i][2]);
#pragma unroll
            for (int j = 0; j < TC; ++j)
              ld3<R, npad>(W.g, ei * nq + q, node_slot(b0 + j, npad), gb[j][0], gb[j][1], gb[j][2]);
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
              for (int j = 0; j < TC; ++j) {
                const R dot = sm * (ga[i][0] * gb[j][0] + ga[i][1] * gb[j][1] + ga[i][2] * gb[j][2]);
#pragma unroll
                for (int x = 0; x < 3; ++x)
#pragma unroll
                  for (int y = 0; y < 3; ++y)
                    acc[i][j][3 * x + y] += (sl * ga[i][x]) * gb[j][y] + (sm * gb[j][x]) * ga[i][y] + (x == y ? dot : R(0));
              }
            if (sc != R(0)) {
              // m = N g for the tile's nodes, from the stored return direction
              const R* N = W.nvq + (ei * nq + q) * 8;
              const R n0 = N[0], n1 = N[1], n2 = N[2], n3 = N[3], n4 = N[4], n5 = N[5];
              R ma[TR][3], mb[TC][3];
#pragma unroll
              for (int i = 0; i < TR; ++i) {
                ma[i][0] = n0 * ga[i][0] + n3 * ga[i][1] + n4 * ga[i][2];
                ma[i][1] = n3 * ga[i][0] + n1 * ga[i][1] + n5 * ga[i][2];
                ma[i][2] = n4 * ga[i][0] + n5 * ga[i][1] + n2 * ga[i][2];
              }
#pragma unroll
              for (int j = 0; j < TC; ++j) {
                mb[j][0] = n0 * gb[j][0] + n3 * gb[j][1] + n4 * gb[j][2];
                mb[j][1] = n3 * gb[j][0] + n1 * gb[j][1] + n5 * gb[j][2];
                mb[j][2] = n4 * gb[j][0] + n5 * gb[j][1] + n2 * gb[j][2];
              }
#pragma unroll
              for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j)
#pragma unroll
                  for (int x = 0; x < 3; ++x)
#pragma unroll
                    for (int y = 0; y < 3; ++y) acc[i][j][3 * x + y] -= (sc * ma[i][x]) * mb[j][y];
            }
          }
        }
        if constexpr (!WS::ALIAS) stage_tile(task);
      }
    }
    if constexpr (WS::ALIAS) {
      __syncwarp();  // every lane is done reading the gradient vectors
      if (lane < EPW * NT && e0 + lane / NT < e_end) stage_tile(lane);
    }
    if constexpr (WS::kElem * sizeof(R) % 16 != 0) {
      __syncwarp();
      for (int ei = 0; ei < EPW && e0 + ei < e_end; ++ei) {
        float2* out = reinterpret_cast<float2*>(reinterpret_cast<R*>(V.edata) + ring_slot(e0 + ei, V) * WS::kElem);
        const float2* sb = reinterpret_cast<const float2*>(stg + ei * WS::kElem);
        for (int t = lane; t < WS::kElem / 2; t += 32) out[t] = sb[t];
      }
    } else {
      fence_async_shared();
      __syncwarp();
    }
    if (WS::kElem * sizeof(R) % 16 == 0 && lane == 0) {
      for (int ei = 0; ei < EPW && e0 + ei < e_end; ++ei)
        bulk_store(reinterpret_cast<R*>(V.edata) + ring_slot(e0 + ei, V) * WS::kElem, stg + ei * WS::kElem,
                   WS::kElem * sizeof(R));
      bulk_commit();
    }
    __syncwarp();
  }
  if (lane == 0) bulk_wait();
}

template <int ET, int MODE, typename R, int TILE, bool J2F32>
__global__ void __launch_bounds__(kT1, (p1_min_blocks<ET, MODE, R, TILE>())) p1_kernel(ElemArgs A, V2Args V) {
  p1_body<ET, MODE, R, TILE, J2F32>(A, V, blockIdx.x, gridDim.x);
}

template <int ET, int MODE, typename R, int TILE>
cudaError_t launch_p1_tile(const ElemArgs& a, const V2Args& v, const LaunchCfg& cfg, cudaStream_t s) {
  constexpr size_t smem = p1_smem_bytes<ET, MODE, R, TILE>();
  static_assert(smem <= 227 * 1024, "element pass shared memory");
  auto kern = p1_kernel<ET, MODE, R, TILE, false>;
  if constexpr (MODE == MODE_TANGENT && sizeof(R) == 4) {
    if (cfg.j2_fp32) kern = p1_kernel<ET, MODE, R, TILE, true>;
  }
  const int64_t count = v.e_end - v.e_begin;
  if (count <= 0) return cudaSuccess;
  constexpr int per_block = kW1 * Geo<ET, TILE>::EPW;
  ElemArgs A = a;
  V2Args V = v;
  void* args[] = {&A, &V};
  const cudaError_t e = launch_persistent(reinterpret_cast<const void*>(kern), smem, (count + per_block - 1) / per_block,
                                          cfg.p1_blocks_per_sm, s, args);
  return e == cudaSuccess ? launch_named_twice(1, a, v, s) : e;
}

// Tile shapes of the FP32 pass: 2x4, 2x2 and 4x4 in linear mode. The material-point pass
// has 2x2 tiles whatever was asked (its tiles carry three accumulator terms: 2x4 measured
// 1.6 times slower), and so has the FP64 pass its own (cxg_fp64.cu).
template <int ET, int MODE>
cudaError_t launch_p1_t(const ElemArgs& a, const V2Args& v, const LaunchCfg& cfg, cudaStream_t s) {
  if (MODE == MODE_TANGENT || cfg.tile == 1) return launch_p1_tile<ET, MODE, float, 1>(a, v, cfg, s);
  if constexpr (MODE == MODE_LINEAR) {
    if (cfg.tile == 2) return launch_p1_tile<ET, MODE, float, 2>(a, v, cfg, s);
    if (cfg.tile == 0) return launch_p1_tile<ET, MODE, float, 0>(a, v, cfg, s);
  }
  return cudaErrorInvalidValue;
}

template <int ET>
cudaError_t launch_v2_pair(int mode, int precision, const ElemArgs& a, const V2Args& v, const LaunchCfg& c,
                           cudaStream_t s);

// Every window's element pass and row gather in order on one stream: the row gather of
// window w reads element blocks that stay in the ring (and in L2) until the element
// pass of window w+1 overwrites the slots of elements no later node needs.
template <int ET>
cudaError_t launch_v2_type(int mode, int precision, const ElemArgs& a, const V2Args& v, const LaunchCfg& c,
                           cudaStream_t s) {
  if (v.n_win <= 1) return launch_v2_pair<ET>(mode, precision, a, v, c, s);
  V2Args w = v;
  for (int32_t k = 0; k < v.n_win; ++k) {
    w.e_begin = v.win_e[k];
    w.e_end = v.win_e[k + 1];
    // both passes of window k touch elements in [e_end - ring, e_end) only
    const int64_t lo = std::max<int64_t>(0, w.e_end - v.ring);
    w.ring_base = lo / v.ring * v.ring;
    w.n_begin = v.win_n[k];
    w.n_end = v.win_n[k + 1];
    const cudaError_t err = launch_v2_pair<ET>(mode, precision, a, w, c, s);
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

template <int ET>
cudaError_t launch_v2_pair(int mode, int precision, const ElemArgs& a, const V2Args& v, const LaunchCfg& c,
                           cudaStream_t s) {
  cudaError_t err = cudaSuccess;
  if (mode == MODE_LINEAR) {
    if (c.passes & 1)
      err = precision ? launch_p1_t<ET, MODE_LINEAR>(a, v, c, s) : launch_p1_fp64(ET, MODE_LINEAR, a, v, c, s);
    if (err != cudaSuccess || !(c.passes & 2)) return err;
    return launch_gather(precision ? GATHER_DIAG : GATHER_FULL, false, a, v, c, s);
  }
  if (c.passes & 1)
    err = precision ? launch_p1_t<ET, MODE_TANGENT>(a, v, c, s) : launch_p1_fp64(ET, MODE_TANGENT, a, v, c, s);
  if (err != cudaSuccess || !(c.passes & 2)) return err;
  return launch_gather(precision ? GATHER_DIAG : GATHER_FULL, true, a, v, c, s);
}

}  // namespace

void share_blocks(const double* weight, const int64_t* need, int n, int64_t total, int64_t* grid) {
  double sum = 0.0;
  for (int k = 0; k < n; ++k) sum += weight[k] > 0.0 ? weight[k] : 0.0;
  for (int k = 0; k < n; ++k) {
    const double f = sum > 0.0 ? std::max(weight[k], 0.0) / sum : 1.0 / n;
    const int64_t g = static_cast<int64_t>(std::llround(f * static_cast<double>(total)));
    grid[k] = std::max<int64_t>(1, std::min<int64_t>(need[k], g));
  }
}

size_t v2_bytes_per_element(int t, int precision, bool tangent) {
  return v2_edata_bytes(t, 1, precision) + (tangent ? sizeof(double) * 3 * nodes_of(t) : 0);
}

size_t v2_edata_bytes(int t, int64_t n_elems, int precision) {
  return static_cast<size_t>(n_elems) * blocks_padded(nodes_of(t)) * 9 * (precision ? sizeof(float) : sizeof(double));
}

cudaError_t launch_v2(int t, int mode, int precision, const ElemArgs& a, const V2Args& v, cudaStream_t s,
                      const LaunchCfg& c) {
  switch (t) {
    case C3D4: return launch_v2_type<C3D4>(mode, precision, a, v, c, s);
    case C3D10: return launch_v2_type<C3D10>(mode, precision, a, v, c, s);
    case C3D8: return launch_v2_type<C3D8>(mode, precision, a, v, c, s);
    case C3D8R: return launch_v2_type<C3D8R>(mode, precision, a, v, c, s);
    case C3D20: return launch_v2_type<C3D20>(mode, precision, a, v, c, s);
    case C3D20R: return launch_v2_type<C3D20R>(mode, precision, a, v, c, s);
    case C3D6: return launch_v2_type<C3D6>(mode, precision, a, v, c, s);
    case C3D15: return launch_v2_type<C3D15>(mode, precision, a, v, c, s);
    default: return cudaErrorInvalidValue;
  }
}

// ---- one launch per pass for a batch of element-type groups ---------------------------
// The batch kernels carry the tiles whose accumulators fit 168 registers, so that 3
// blocks of 4 warps stay resident per SM whatever families share the launch: 2x2
// everywhere and 2x4 in the mixed-precision linear pass.
bool batch_tile_ok(int mode, int precision, int tile) {
  return tile == 1 || (tile == 0 && mode == MODE_LINEAR && precision);
}

template <int ET, int MODE, typename R, bool J2F32>
__device__ __forceinline__ void p1_slot_tile(int tile, const ElemArgs& A, const V2Args& V, unsigned bid, unsigned nblk) {
  if constexpr (MODE == MODE_LINEAR && sizeof(R) == 4) {
    if (tile == 0) {
      p1_body<ET, MODE, R, 0, J2F32>(A, V, bid, nblk);
      return;
    }
  }
  p1_body<ET, MODE, R, 1, J2F32>(A, V, bid, nblk);
}

template <int MODE, typename R, bool J2F32>
__global__ void __launch_bounds__(kT1, 3) p1_batch_kernel(const __grid_constant__ BatchPass P) {
  // the slot's arguments are read in place from the (read-only) parameter space
  unsigned bid, nblk;
  const int k = slot_blocks(P, bid, nblk);
  const BatchSlot& S = P.s[k];
  switch (S.type) {
    case C3D4: p1_slot_tile<C3D4, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    case C3D10: p1_slot_tile<C3D10, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    case C3D8: p1_slot_tile<C3D8, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    case C3D8R: p1_slot_tile<C3D8R, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    case C3D20: p1_slot_tile<C3D20, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    case C3D20R: p1_slot_tile<C3D20R, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    case C3D6: p1_slot_tile<C3D6, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    case C3D15: p1_slot_tile<C3D15, MODE, R, J2F32>(S.tile, S.a, S.v, bid, nblk); break;
    default: break;
  }
}

template <int ET, int MODE, typename R, int TILE>
P1Shape p1_shape_of() {
  return {p1_smem_bytes<ET, MODE, R, TILE>(), Geo<ET, TILE>::EPW};
}
template <int ET, int MODE, typename R>
P1Shape p1_shape_tile(int tile) {
  if constexpr (MODE == MODE_LINEAR && sizeof(R) == 4) {
    if (tile == 0) return p1_shape_of<ET, MODE, R, 0>();
  }
  return p1_shape_of<ET, MODE, R, 1>();
}
template <int MODE, typename R>
P1Shape p1_shape(int t, int tile) {
  switch (t) {
    case C3D4: return p1_shape_tile<C3D4, MODE, R>(tile);
    case C3D10: return p1_shape_tile<C3D10, MODE, R>(tile);
    case C3D8: return p1_shape_tile<C3D8, MODE, R>(tile);
    case C3D8R: return p1_shape_tile<C3D8R, MODE, R>(tile);
    case C3D20: return p1_shape_tile<C3D20, MODE, R>(tile);
    case C3D20R: return p1_shape_tile<C3D20R, MODE, R>(tile);
    case C3D6: return p1_shape_tile<C3D6, MODE, R>(tile);
    default: return p1_shape_tile<C3D15, MODE, R>(tile);
  }
}
// Element pass of the whole batch: the kernel and the per-family figures of the mode and
// precision (FP64 blocks: cxg_fp64.cu).
cudaError_t launch_p1_batch(int mode, int precision, bool j2f32, const BatchSlotIn* in, int n, cudaStream_t s) {
  const void* kern = !precision             ? p1_fp64_batch(mode)
                     : mode == MODE_LINEAR ? reinterpret_cast<const void*>(p1_batch_kernel<MODE_LINEAR, float, false>)
                     : j2f32               ? reinterpret_cast<const void*>(p1_batch_kernel<MODE_TANGENT, float, true>)
                                           : reinterpret_cast<const void*>(p1_batch_kernel<MODE_TANGENT, float, false>);
  BatchPass P{};
  size_t smem = 0;
  int64_t need[kMaxBatchSlots], grid[kMaxBatchSlots];
  double w[kMaxBatchSlots];
  for (int k = 0; k < n; ++k) {
    const P1Shape sh = !precision            ? p1_fp64_shape(in[k].type, mode)
                       : mode == MODE_LINEAR ? p1_shape<MODE_LINEAR, float>(in[k].type, in[k].cfg.tile)
                                             : p1_shape<MODE_TANGENT, float>(in[k].type, in[k].cfg.tile);
    smem = std::max(smem, sh.smem);
    const int64_t count = in[k].v.e_end - in[k].v.e_begin;
    need[k] = std::max<int64_t>(1, (count + kW1 * sh.epw - 1) / (kW1 * sh.epw));
    w[k] = in[k].p1_weight;
  }
  if (smem > 227 * 1024) return cudaErrorInvalidConfiguration;
  int per_sm = 0, sms = 0;
  const cudaError_t err = kernel_shape(kern, kT1, smem, &per_sm, &sms);
  if (err != cudaSuccess) return err;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  share_blocks(w, need, n, static_cast<int64_t>(per_sm) * sms, grid);
  int64_t blk = 0;
  for (int k = 0; k < n; ++k) {
    P.s[k].a = in[k].a;
    P.s[k].v = in[k].v;
    P.s[k].blk0 = blk;
    P.s[k].type = in[k].type;
    P.s[k].tile = in[k].cfg.tile;
    blk += grid[k];
  }
  P.n = n;
  void* args[] = {&P};
  cudaError_t e = launch_kernel(kern, blk, kT1, smem, s, args);
  for (int k = 0; k < n && e == cudaSuccess; ++k) e = launch_named_twice(precision, in[k].a, in[k].v, s);
  return e;
}

cudaError_t launch_v2_batch(int mode, int precision, const BatchSlotIn* in, int n, int passes, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (n > kMaxBatchSlots) return cudaErrorInvalidValue;
  const bool j2f32 = mode == MODE_TANGENT && precision && in[0].cfg.j2_fp32;
  for (int k = 0; k < n; ++k) {
    if (in[k].type < kFirstType || in[k].type > kLastType || in[k].v.n_win > 1 || in[k].v.node_order)
      return cudaErrorInvalidValue;
    if ((mode == MODE_TANGENT && precision && (in[k].cfg.j2_fp32 != 0) != j2f32) ||
        !batch_tile_ok(mode, precision, in[k].cfg.tile))
      return cudaErrorInvalidValue;
  }
  cudaError_t err = cudaSuccess;
  if (passes & 1) {
    err = launch_p1_batch(mode, precision, j2f32, in, n, s);
    if (err != cudaSuccess) return err;
  }
  if (passes & 2) return launch_gather_batch(precision ? GATHER_DIAG : GATHER_FULL, mode == MODE_TANGENT, in, n, s);
  return err;
}

}  // namespace cxg
