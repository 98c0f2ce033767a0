// P1 in FP64: the element pass on the FP64 tensor cores.
//
// Every 3x3 block of K_e is built from sums over the Gauss points of outer products of
// node gradients, G_ab = sum_q s_q g_a g_b^T: for 8 nodes a, 8 nodes b and one component
// each (x of a, y of b) that is one 8x8 matrix product with the Gauss points as inner
// dimension, mma.m8n8k4 in FP64. A lane's operand is one gradient component of one (node,
// Gauss point), the same registers serving as rows and as columns, and of the nine (x, y)
// products a lane holds the same two node pairs, so it has their whole 3x3 blocks and
// finishes them alone: K_ab = lam G + mu (G^T + tr(G) I). An element with plastic points
// adds up two such sets, with the points' own lam and mu, and the products of m = N g:
// K = sum s lam* g g^T - s c m m^T, + the mu* set as above; a lane forms m from the
// operands it already holds.
//
// Against tiles of node pairs with FP64 FMAs, which read each gradient vector from shared
// memory once per tile (the L1 pipe was the bound at 80 %), an operand here is one 8-byte
// read per lane for up to 27 products, and the accumulators take 36 registers (72 plastic)
// whatever the family.
//
// What bounds it: latency of the phases a warp goes through in turn, with the matrix unit
// 46 % and the shared-memory pipe 56 % busy on C3D20 (8 or 12 warps per SM ran alike).
// C3D8 J2 128^3 4605 us with tiles of FMAs, 3087 so; C3D20 41x37x33
// linear 510 -> 529 us, for a gather that takes 408 us instead of 574 from the blocks' order.
//
// Lanes first take (element, Gauss point) tasks: Jacobian, inverse, gradients, and in
// material-point mode the strain and the J2 return, as in the FP32 pass.
#include <cuda_runtime.h>

#include "cxg_element.cuh"

namespace cxg {

namespace {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// The transposed 8x8 result: v holds entries (row, 2 col), (row, 2 col + 1) of it on lane
// (row, col), and then those of its transpose. 2x2 parts first, then the parts themselves.
__device__ __forceinline__ void transposed(const double (&v)[2], double (&t)[2], int row, int col) {
  const bool odd = row & 1;
  const double got = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], 4);
  const int src = (2 * col + (row & 1)) * 4 + (row >> 1);
  t[0] = __shfl_sync(0xffffffffu, odd ? got : v[0], src);
  t[1] = __shfl_sync(0xffffffffu, odd ? v[1] : got, src);
}

template <int ET>
struct DGeo {
  static constexpr int n = nodes_of(ET), nq = gauss_of(ET);
  static constexpr int NTL = (n + 7) / 8;                // tiles of 8 nodes
  static constexpr int KS = (nq + 3) / 4, NQP = 4 * KS;  // steps of 4 Gauss points
  // Gradients as [component][node][Gauss point], QS values per node. With 8 points a node
  // the halves of nodes 2, 3 (mod 4) change places (turn), so that the 4 nodes x 4 points
  // of a half warp's operand lie in different banks.
  static constexpr int QS = NQP;
  __host__ __device__ static constexpr int turn(int k) { return NQP == 8 ? (k & 2) << 1 : 0; }
  static constexpr int ROWS = n < 8 ? 8 : n;
  static constexpr int P = ROWS * QS;                    // one component
  // (a last tile of fewer than 8 nodes reads past its component: results it drops)
  static constexpr int kRaw = 3 * P + (NTL * 8 - ROWS) * QS;
  // Elements per warp and batch: 32 lanes of (element, Gauss point) tasks where shared
  // memory allows; they start 8 (mod 16) values apart for the tasks' stores.
  static constexpr int EPB = n > 8 ? (nq == 27 ? 1 : nq == 4 ? 4 : 2) : (nq == 8 ? 4 : 8);
  static constexpr int ES = EPB == 1 ? kRaw : (kRaw + 15) / 16 * 16 + 8;
  static constexpr int kElem = blocks_padded(n) * 9;
  // Staged blocks: one element, leaving as one bulk copy, or one tile pair. C3D4, with four
  // nodes and one point, would fill a sixteenth of a product: its lanes take a block each
  // (PAIRS), and a batch's elements are staged together.
  static constexpr bool BULK = NTL == 1, PAIRS = n == 4 && nq == 1;
  static constexpr int kStage = PAIRS ? EPB * kElem : BULK ? kElem : 578;
  // (rows of 8 blocks, one value further from row 2 and two from row 6 on: a half warp's
  // stores then lie in different banks; C3D20 536 -> 529 us)
  static __host__ __device__ constexpr int stage_row(int r) { return r * 72 + (r + 2) / 4; }
};

template <int ET, bool TAN>
struct DSmem {
  using G = DGeo<ET>;
  static constexpr int n = G::n, nq = G::nq, EPB = G::EPB, NQP = G::NQP;
  static constexpr int T = TAN ? EPB : 1, HG = ET == C3D8R ? EPB : 1;
  alignas(16) double stg[G::kStage];
  double g[EPB * G::ES];
  double s[EPB][NQP];            // det J w (zero in the padding)
  double dp[T][3][TAN ? NQP : 1];  // s lam*, s mu*, s c of the points
  double N[T][6][TAN ? NQP : 1];   // return direction (zero at elastic points)
  double x[EPB][3 * n];
  double u[T][TAN ? 3 * n : 1];
  double sig[T][TAN ? nq : 1][6];
  double lam[EPB], mu[EPB], mu_j2[EPB];
  double gam[HG][32];
  double kappa[HG];
  double gc[HG][3 * n];
  double vol[HG];
  double mu_hg[HG];
  int plastic[EPB];
  int id[EPB][n];
};

template <int ET, bool TAN>
constexpr size_t p1d_smem_bytes() {
  constexpr int n = nodes_of(ET), nq = gauss_of(ET);
  return (sizeof(double) * (n * 3 * nq + nq) + 15) / 16 * 16 + kW1 * ((sizeof(DSmem<ET, TAN>) + 15) / 16 * 16);
}

// Resident blocks per SM asked of the register allocator: what shared memory allows, at
// most 4 (128 registers), in material-point mode 3 (168: two accumulator sets and the J2
// return).
template <int ET, bool TAN>
constexpr int p1d_min_blocks() {
  constexpr int by_smem = static_cast<int>(227 * 1024 / (p1d_smem_bytes<ET, TAN>() + 1024));
  constexpr int cap = TAN ? 3 : 4;
  return by_smem < 1 ? 1 : by_smem < cap ? by_smem : cap;
}

template <int ET, bool TAN>
__device__ __forceinline__ void p1d_body(const ElemArgs& A, const V2Args& V, unsigned bid, unsigned nblk) {
  using G = DGeo<ET>;
  using WS = DSmem<ET, TAN>;
  constexpr int n = G::n, nq = G::nq, EPB = G::EPB, QS = G::QS, P = G::P, ES = G::ES, KS = G::KS;
  extern __shared__ __align__(16) unsigned char smem[];
  double* sdN = reinterpret_cast<double*>(smem);  // [n][3][nq]
  double* sw = sdN + n * 3 * nq;
  constexpr size_t cta_bytes = (sizeof(double) * (n * 3 * nq + nq) + 15) / 16 * 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WS& W = *reinterpret_cast<WS*>(smem + cta_bytes + warp * ((sizeof(WS) + 15) / 16 * 16));
  for (int i = threadIdx.x; i < n * 3 * nq; i += blockDim.x) sdN[i] = c_dN[dn_offset(ET) + i];
  for (int i = threadIdx.x; i < nq; i += blockDim.x) sw[i] = c_w[ET][i];
  // the padding of the Gauss points stays zero
  for (int t = lane; t < EPB * ES; t += 32) W.g[t] = 0.0;
  for (int t = lane; t < EPB * G::NQP; t += 32) W.s[t / G::NQP][t % G::NQP] = 0.0;
  if (TAN)
    for (int t = lane; t < EPB * G::NQP; t += 32) {
      for (int c = 0; c < 3; ++c) W.dp[t / G::NQP][c][t % G::NQP] = 0.0;
      for (int c = 0; c < 6; ++c) W.N[t / G::NQP][c][t % G::NQP] = 0.0;
    }
  __syncthreads();

  const int64_t gwarp = static_cast<int64_t>(bid) * kW1 + warp;
  const int64_t nwarps = static_cast<int64_t>(nblk) * kW1;
  const int64_t e_end = V.e_end;
  constexpr int PA = (EPB * n + 31) / 32;
  int conn_next[PA];
  auto load_conn = [&](int64_t e0x) {
#pragma unroll
    for (int p = 0; p < PA; ++p) {
      const int t = lane + 32 * p;
      const int64_t e = e0x + t / n;
      conn_next[p] = t < EPB * n && e < e_end ? A.conn[e * n + t % n] : -1;
    }
  };
  wait_for_kernel_before();
  // Only in a launch of one batch per warp: blocks of the gather that settle beside a longer
  // element pass would run in the little L1 its shared memory leaves (C3D20 64^3 mixed 3530
  // -> 3706 us an assembly).
  if (e_end - V.e_begin <= nwarps * EPB) let_next_kernel_start();
  load_conn(V.e_begin + gwarp * EPB);
  for (int64_t e0 = V.e_begin + gwarp * EPB; e0 < e_end; e0 += nwarps * EPB) {
    // ---- coordinates and displacements of the batch's nodes
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
    load_conn(e0 + nwarps * EPB);
    if (lane < EPB) {
      const int64_t e = e0 + lane;
      const double E = e < e_end ? A.young[e] : 1.0, nu = e < e_end ? A.poisson[e] : 0.0;
      const double um2 = E / (1.0 + nu);
      W.lam[lane] = nu * um2 / (1.0 - 2.0 * nu);
      W.mu[lane] = um2 / 2.0;
      W.mu_j2[lane] = E / (2.0 * (1.0 + nu));
      W.plastic[lane] = 0;
    }
    __syncwarp();
    // ---- (element, Gauss point) tasks
    for (int t = lane; t < EPB * nq; t += 32) {
      const int ei = t / nq, q = t % nq;
      const int64_t e = e0 + ei;
      if (e >= e_end) continue;
      double J[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll(n <= 10 ? n : 5)
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
      W.s[ei][q] = sq;
      if constexpr (ET == C3D8R) W.vol[ei] = sq;
      double H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
      double* gq = W.g + ei * ES;
#pragma unroll(n <= 10 ? n : 5)
      for (int k = 0; k < n; ++k) {
        const double d0 = sdN[(3 * k) * nq + q], d1 = sdN[(3 * k + 1) * nq + q], d2 = sdN[(3 * k + 2) * nq + q];
        double gk[3];
        for (int i = 0; i < 3; ++i) {
          gk[i] = fma(it[i][0], d0, fma(it[i][1], d1, mul(it[i][2], d2)));
          if constexpr (ET == C3D8R) W.gc[ei][i * n + k] = gk[i];
          gq[i * P + k * QS + (q ^ G::turn(k))] = gk[i];
        }
        if (TAN)
          for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) H[i][j] = fma(W.u[ei][3 * k + i], gk[j], H[i][j]);
      }
      if constexpr (TAN) {
        const double eps[6] = {H[0][0], H[1][1], H[2][2], H[0][1] + H[1][0], H[0][2] + H[2][0], H[1][2] + H[2][1]};
        const int mat = A.elem_mat ? A.elem_mat[e] : 0;
        const int64_t gidx = e * nq + q;
        double cs[kStateDoubles], ts[kStateDoubles], sig[6], nv[6] = {0, 0, 0, 0, 0, 0};
        const bool back = A.state_comps > 7;  // else the back stress is zero
#pragma unroll
        for (int c = 0; c < kStateDoubles; ++c) cs[c] = c < 7 || back ? A.state_c[c * A.n_gauss + gidx] : 0.0;
        double lt, mt, ct, mhg;
        const bool pl = j2_point(A.mats[mat], W.lam[ei], W.mu[ei], W.mu_j2[ei], eps, cs, ts, sig, lt, mt, ct, nv, mhg);
#pragma unroll
        for (int c = 0; c < kStateDoubles; ++c)
          if (c < 7 || back) A.state_t[c * A.n_gauss + gidx] = ts[c];
        for (int c = 0; c < 6; ++c) W.sig[ei][q][c] = mul(sq, sig[c]);
        W.dp[ei][0][q] = sq * lt;
        W.dp[ei][1][q] = sq * mt;
        W.dp[ei][2][q] = sq * ct;
#pragma unroll
        for (int c = 0; c < 6; ++c) W.N[ei][c][q] = nv[c];
        if (pl) W.plastic[ei] = 1;
        if constexpr (ET == C3D8R) W.mu_hg[ei] = mhg;
      }
    }
    __syncwarp();
    // ---- C3D8R hourglass vectors (src/fem/element.cpp:545-579)
    if constexpr (ET == C3D8R) {
      for (int t = lane; t < EPB * 4; t += 32) {
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
      if (lane < EPB) {
        double b2 = 0.0;
        for (int t = 0; t < 3 * n; ++t) b2 = fma(W.gc[lane][t], W.gc[lane][t], b2);
        W.kappa[lane] = 0.05 * (TAN ? W.mu_hg[lane] : W.mu_j2[lane]) * W.vol[lane] * b2;
      }
      __syncwarp();
    }
    // ---- internal force per element
    if constexpr (TAN) {
      for (int t = lane; t < EPB * n; t += 32) {
        const int ei = t / n, a = t % n;
        const int64_t e = e0 + ei;
        if (e >= e_end) continue;
        double f[3] = {0, 0, 0};
        const double* ga = W.g + ei * ES + a * QS;
        for (int q = 0; q < nq; ++q) {
          const double* S = W.sig[ei][q];
          const int qt = q ^ G::turn(a);
          const double gx = ga[qt], gy = ga[P + qt], gz = ga[2 * P + qt];
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
    if constexpr (G::PAIRS) {
      // ---- blocks, one node pair a lane (196,608 C3D4, J2: element pass 182 us by products, 101 so)
      bulk_wait_read();  // the last batch's copies have left
      __syncwarp();
      for (int t = lane; t < EPB * (n * (n + 1) / 2); t += 32) {
        const int ei = t / (n * (n + 1) / 2), blk = t - ei * (n * (n + 1) / 2);
        if (e0 + ei >= e_end) break;
        int a = 0;
        while (blk >= blk_index(n, a + 1, a + 1)) ++a;
        const int b = blk - blk_index(n, a, a) + a;
        double ga[3], gb[3], k[3][3];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          ga[x] = W.g[ei * ES + x * P + a * QS];
          gb[x] = W.g[ei * ES + x * P + b * QS];
        }
        const double sl = TAN ? W.dp[ei][0][0] : W.s[ei][0] * W.lam[ei], sm = TAN ? W.dp[ei][1][0] : W.s[ei][0] * W.mu[ei];
        const double tr = sm * (ga[0] * gb[0] + ga[1] * gb[1] + ga[2] * gb[2]);
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
          for (int y = 0; y < 3; ++y)
            k[x][y] = fma(sl, mul(ga[x], gb[y]), mul(sm, mul(ga[y], gb[x]))) + (x == y ? tr : 0.0);
        if (TAN && W.plastic[ei]) {
          const double sc = W.dp[ei][2][0];
          auto turned = [&](const double (&v)[3], double (&m)[3]) {  // m = N g
            const auto& N = W.N[ei];
            m[0] = fma(N[0][0], v[0], fma(N[3][0], v[1], mul(N[4][0], v[2])));
            m[1] = fma(N[3][0], v[0], fma(N[1][0], v[1], mul(N[5][0], v[2])));
            m[2] = fma(N[4][0], v[0], fma(N[5][0], v[1], mul(N[2][0], v[2])));
          };
          double ma[3], mb[3];
          turned(ga, ma);
          turned(gb, mb);
#pragma unroll
          for (int x = 0; x < 3; ++x)
#pragma unroll
            for (int y = 0; y < 3; ++y) k[x][y] = fma(-sc, mul(ma[x], mb[y]), k[x][y]);
        }
        const int sx = W.id[ei][a] > W.id[ei][b] ? 1 : 3, sy = 4 - sx;
        double* d = W.stg + ei * G::kElem + blk * 9;
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
          for (int y = 0; y < 3; ++y) d[x * sx + y * sy] = k[x][y];
      }
      fence_async_shared();
      __syncwarp();
      if (lane < EPB && e0 + lane < e_end) {
        bulk_store(reinterpret_cast<double*>(V.edata) + ring_slot(e0 + lane, V) * G::kElem, W.stg + lane * G::kElem,
                   G::kElem * sizeof(double));
        bulk_commit();
      }
      continue;
    }
    // ---- blocks, one element after the other, one pair of node tiles at a time
    const int row = lane >> 2, col = lane & 3, turn = G::turn(row);
#pragma unroll 1
    for (int ei = 0; ei < EPB && e0 + ei < e_end; ++ei) {
      const bool pl = TAN && W.plastic[ei];
      double* out = reinterpret_cast<double*>(V.edata) + ring_slot(e0 + ei, V) * G::kElem;
#pragma unroll 1
      for (int ta = 0; ta < G::NTL; ++ta)
#pragma unroll 1
        for (int tb = ta; tb < G::NTL; ++tb) {
          const double* gA = W.g + ei * ES + (8 * ta + row) * QS + col;
          const double* gB = W.g + ei * ES + (8 * tb + row) * QS + col;
          double L[3][3][2] = {};  // block entries (x, y) of pairs (a, b), (a, b + 1)
          // A tile with itself: entry (y, x) of (a, b) is entry (x, y) of (b, a), so three of
          // the nine products are transposes of others, 9 shuffles of doubles for 3 KS (an
          // element with plastic points: 18 for 9 KS) products. C3D8 J2 128^3: 3258 -> 3087
          // us; elastic elements of several tiles lost (C3D20 FP64 529 -> 539) and form all.
          const bool self = G::NTL == 1, selfp = G::NTL == 1 || ta == tb;
          auto mirror = [&](double (&m)[3][3][2]) {
#pragma unroll
            for (int x = 0; x < 3; ++x)
#pragma unroll
              for (int y = x + 1; y < 3; ++y) transposed(m[x][y], m[y][x], row, col);
          };
          if (!pl) {
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
              const double s = W.s[ei][4 * ks + col];
              double a[3], b[3];
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                a[x] = s * gA[x * P + ((4 * ks) ^ turn)];
                b[x] = gB[x * P + ((4 * ks) ^ turn)];
              }
#pragma unroll
              for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y)
                  if (y >= x || !self) dmma(L[x][y], a[x], b[y]);
            }
            if (self) mirror(L);
            const double lam = W.lam[ei], mu = W.mu[ei];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const double tr = mu * (L[0][0][h] + L[1][1][h] + L[2][2][h]);
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                L[x][x][h] = fma(lam + mu, L[x][x][h], tr);
#pragma unroll
                for (int y = x + 1; y < 3; ++y) {
                  const double p = L[x][y][h], q = L[y][x][h];
                  L[x][y][h] = fma(lam, p, mu * q);
                  L[y][x][h] = fma(lam, q, mu * p);
                }
              }
            }
          } else if constexpr (TAN) {
            double M[3][3][2] = {};
#pragma unroll(KS == 2 ? 2 : 1)
            for (int ks = 0; ks < KS; ++ks) {
              const int q = 4 * ks + col;
              const double sl = W.dp[ei][0][q], sm = W.dp[ei][1][q], sc = W.dp[ei][2][q];
              const double n0 = W.N[ei][0][q], n1 = W.N[ei][1][q], n2 = W.N[ei][2][q], n3 = W.N[ei][3][q],
                           n4 = W.N[ei][4][q], n5 = W.N[ei][5][q];
              double a[3], b[3];
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                a[x] = gA[x * P + ((4 * ks) ^ turn)];
                b[x] = gB[x * P + ((4 * ks) ^ turn)];
              }
#pragma unroll
              for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y)
                  if (y >= x || !selfp) {
                    dmma(L[x][y], sl * a[x], b[y]);
                    dmma(M[x][y], sm * a[x], b[y]);
                  }
              // m = N g
              auto turned = [&](const double (&v)[3], double (&m)[3]) {
                m[0] = fma(n0, v[0], fma(n3, v[1], mul(n4, v[2])));
                m[1] = fma(n3, v[0], fma(n1, v[1], mul(n5, v[2])));
                m[2] = fma(n4, v[0], fma(n5, v[1], mul(n2, v[2])));
              };
              double ma[3], mb[3];
              turned(a, ma);
              turned(b, mb);
#pragma unroll
              for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y)
                  if (y >= x || !selfp) dmma(L[x][y], -sc * ma[x], mb[y]);
            }
            if (selfp) {
              mirror(L);
              mirror(M);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const double tr = M[0][0][h] + M[1][1][h] + M[2][2][h];
#pragma unroll
              for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y) L[x][y][h] += M[y][x][h] + (x == y ? tr : 0.0);
            }
          }
          // ---- stage the blocks, transposed where b precedes a in the mesh
          const int a = 8 * ta + row;
          if (G::BULK && lane == 0) bulk_wait_read();  // the last element's copy has left
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int b = 8 * tb + 2 * col + h;
            if (a < n && b < n && a <= b) {
              if constexpr (ET == C3D8R) {
                double hd = 0.0;
                for (int al = 0; al < 4; ++al) hd = fma(W.gam[ei][al * 8 + a], W.gam[ei][al * 8 + b], hd);
                for (int x = 0; x < 3; ++x) L[x][x][h] = fma(hd, W.kappa[ei], L[x][x][h]);
              }
              const int sx = W.id[ei][a] > W.id[ei][b] ? 1 : 3, sy = 4 - sx;
              double* d = W.stg + (G::BULK ? blk_index(n, a, b) * 9 : G::stage_row(row) + (2 * col + h) * 9);
#pragma unroll
              for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y) d[x * sx + y * sy] = L[x][y][h];
            }
          }
          if constexpr (G::BULK) {
            fence_async_shared();
            __syncwarp();
            if (lane == 0) {
              bulk_store(out, W.stg, G::kElem * sizeof(double));
              bulk_commit();
            }
          } else {
            __syncwarp();
            // rows of up to 8 blocks, contiguous in the element's buffer
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const int ar = 8 * ta + r;
              if (ar >= n) break;
              double* o = out + (blk_index(n, ar, ar) + 8 * tb - ar) * 9;
#pragma unroll
              for (int t = lane; t < 72; t += 32) {
                const int b = 8 * tb + t / 9;
                if (b < n && b >= ar) o[t] = W.stg[G::stage_row(r) + t];
              }
            }
          }
        }
    }
    __syncwarp();
  }
  if (G::PAIRS || (G::BULK && lane == 0)) bulk_wait();
}

template <int ET, bool TAN>
__global__ void __launch_bounds__(kT1, (p1d_min_blocks<ET, TAN>())) p1_fp64_kernel(ElemArgs A, V2Args V) {
  p1d_body<ET, TAN>(A, V, blockIdx.x, gridDim.x);
}

template <int ET, bool TAN>
cudaError_t launch_t(const ElemArgs& a, const V2Args& v, const LaunchCfg& cfg, cudaStream_t s) {
  constexpr size_t smem = p1d_smem_bytes<ET, TAN>();
  static_assert(smem <= 227 * 1024, "element pass shared memory");
  const int64_t count = v.e_end - v.e_begin;
  if (count <= 0) return cudaSuccess;
  constexpr int per_block = kW1 * DGeo<ET>::EPB;
  ElemArgs A = a;
  V2Args V = v;
  void* args[] = {&A, &V};
  return launch_persistent(reinterpret_cast<const void*>(p1_fp64_kernel<ET, TAN>), smem, (count + per_block - 1) / per_block,
                           cfg.p1_blocks_per_sm, s, args);
}

// Elements that name a mesh node at two places a < b: the gather adds block (a, b) for the
// pair and again for (b, a), K_ab + K_ab^T in all, so it is given the symmetric part; zeros in
// FP32, where the gather forms all of a node's own block. A pass of its own, for the meshes that
// have such elements: a comparison where the blocks are staged cost every mesh 1 to 7 % of the
// element pass (C3D20 41x37x33 FP64 529 -> 543 us, C3D4 87 -> 93, C3D8 J2 mixed 292 -> 297).
template <typename R>
__global__ void __launch_bounds__(256) named_twice_kernel(ElemArgs A, V2Args V) {
  for (int64_t e = V.e_begin + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < V.e_end;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    R* blocks = reinterpret_cast<R*>(V.edata) + ring_slot(e, V) * (V.nbp * 9);
    const int32_t* id = A.conn + e * V.npe;
    for (int a = 0; a < V.npe; ++a)
      for (int b = a + 1; b < V.npe; ++b) {
        if (id[a] != id[b]) continue;
        R* k = blocks + blk_index(V.npe, a, b) * 9;
        for (int x = 0; x < 3; ++x)
          for (int y = x; y < 3; ++y)
            k[3 * x + y] = k[3 * y + x] = sizeof(R) == 4 ? R(0) : R(0.5) * (k[3 * x + y] + k[3 * y + x]);
      }
  }
}

template <bool TAN>
__global__ void __launch_bounds__(kT1, 2) p1_fp64_batch_kernel(const __grid_constant__ BatchPass P) {
  unsigned bid, nblk;
  const int k = slot_blocks(P, bid, nblk);
  const BatchSlot& S = P.s[k];
  switch (S.type) {
    case C3D4: p1d_body<C3D4, TAN>(S.a, S.v, bid, nblk); break;
    case C3D10: p1d_body<C3D10, TAN>(S.a, S.v, bid, nblk); break;
    case C3D8: p1d_body<C3D8, TAN>(S.a, S.v, bid, nblk); break;
    case C3D8R: p1d_body<C3D8R, TAN>(S.a, S.v, bid, nblk); break;
    case C3D20: p1d_body<C3D20, TAN>(S.a, S.v, bid, nblk); break;
    case C3D20R: p1d_body<C3D20R, TAN>(S.a, S.v, bid, nblk); break;
    case C3D6: p1d_body<C3D6, TAN>(S.a, S.v, bid, nblk); break;
    case C3D15: p1d_body<C3D15, TAN>(S.a, S.v, bid, nblk); break;
    default: break;
  }
}

// ---- scalar operators ------------------------------------------------------------------
// Mass, geometric stiffness and conduction give every node pair one value (times I): m_ab
// = sum_q rho detJ w N_a N_b (element_mass, src/fem/element.cpp:786-812), its row sums on
// the diagonal for the lumped mass (element.cpp:814-831), k_ab = sum_q detJ w g_a .
// sigma_q . g_b (element_geometric_stiffness + accumulate_kgeo, element.cpp:482-508,
// 833-854), k_ab = sum_q k detJ w g_a . g_b (element_conduction, element.cpp:745-765).
// The same tasks and operands as above, one accumulator per tile pair: the three
// components are three more products. A lane's two values go straight to the element's
// packed row (8 bytes a pair; the 3x3 blocks this replaced were nine values, eight of them
// zeros or copies, written and read back: C3D15 conduction of 85,050 elements 399 + 720 us
// for pass and gather).
enum ScalarKind : int { MASS = 1, LUMPED = 2, GEOMETRIC = 3, CONDUCTION = 4 };

template <int ET, int KIND>
struct SSmem {
  using G = DGeo<ET>;
  static constexpr bool GRAD = KIND >= GEOMETRIC, GEO = KIND == GEOMETRIC;
  double g[GRAD ? G::EPB * G::ES : 1];
  double s[G::EPB][G::NQP];                        // detJ w, times rho or k
  double sig[GEO ? G::EPB : 1][6][GEO ? G::NQP : 1];  // stress of the points
  double x[G::EPB][3 * G::n];
};

// Per block: natural derivatives and weights, and for the masses the shape functions, one
// row of NQP values per node (rows and points padded with zeros).
template <int ET, int KIND>
constexpr int scalar_table() {
  using G = DGeo<ET>;
  return (G::n * 3 + 1) * G::nq + (KIND <= LUMPED ? G::NTL * 8 * G::NQP : 0);
}
template <int ET, int KIND>
constexpr size_t scalar_smem_bytes() {
  return (sizeof(double) * scalar_table<ET, KIND>() + 15) / 16 * 16 + kW1 * ((sizeof(SSmem<ET, KIND>) + 15) / 16 * 16);
}

template <int ET, int KIND>
__global__ void __launch_bounds__(kT1, 4) scalar_kernel(ElemArgs A, V2Args V, const double* density,
                                                        const double* gp_stress) {
  using G = DGeo<ET>;
  using WS = SSmem<ET, KIND>;
  constexpr int n = G::n, nq = G::nq, EPB = G::EPB, QS = G::QS, P = G::P, ES = G::ES, KS = G::KS, NQP = G::NQP;
  constexpr int NB = n * (n + 1) / 2;
  constexpr bool GRAD = WS::GRAD, GEO = WS::GEO;
  extern __shared__ __align__(16) unsigned char smem[];
  double* sdN = reinterpret_cast<double*>(smem);  // [n][3][nq]
  double* sw = sdN + n * 3 * nq;
  double* sN = sw + nq;  // [node][NQP]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WS& W = *reinterpret_cast<WS*>(smem + (sizeof(double) * scalar_table<ET, KIND>() + 15) / 16 * 16 +
                                 warp * ((sizeof(WS) + 15) / 16 * 16));
  for (int i = threadIdx.x; i < n * 3 * nq; i += blockDim.x) sdN[i] = c_dN[dn_offset(ET) + i];
  for (int i = threadIdx.x; i < nq; i += blockDim.x) sw[i] = c_w[ET][i];
  if constexpr (!GRAD)
    for (int i = threadIdx.x; i < G::NTL * 8 * NQP; i += blockDim.x) {
      const int k = i / NQP, q = i % NQP;
      sN[i] = k < n && q < nq ? c_N[nn_offset(ET) + k * nq + q] : 0.0;
    }
  if (GRAD)
    for (int t = lane; t < EPB * ES; t += 32) W.g[t] = 0.0;
  for (int t = lane; t < EPB * NQP; t += 32) W.s[t / NQP][t % NQP] = 0.0;
  if (GEO)
    for (int t = lane; t < EPB * 6 * NQP; t += 32) W.sig[t / (6 * NQP)][t / NQP % 6][t % NQP] = 0.0;
  __syncthreads();
  wait_for_kernel_before();
  const int64_t gwarp = static_cast<int64_t>(blockIdx.x) * kW1 + warp;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * kW1;
  if (A.n_elems <= nwarps * EPB) let_next_kernel_start();  // (see the element pass)
  for (int64_t e0 = gwarp * EPB; e0 < A.n_elems; e0 += nwarps * EPB) {
    for (int t = lane; t < EPB * n; t += 32) {
      if (e0 + t / n >= A.n_elems) break;
      const int64_t node = A.conn[e0 * n + t];
      for (int d = 0; d < 3; ++d) W.x[t / n][3 * (t % n) + d] = A.coords[3 * node + d];
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
      W.s[ei][q] = GEO ? det * sw[q] : density[e] * det * sw[q];
      if constexpr (GRAD) {
        double* gq = W.g + ei * ES;
        for (int k = 0; k < n; ++k) {
          const double d0 = sdN[(3 * k) * nq + q], d1 = sdN[(3 * k + 1) * nq + q], d2 = sdN[(3 * k + 2) * nq + q];
          for (int i = 0; i < 3; ++i)
            gq[i * P + k * QS + (q ^ G::turn(k))] = fma(it[i][0], d0, fma(it[i][1], d1, mul(it[i][2], d2)));
        }
      }
      if constexpr (GEO)
        for (int c = 0; c < 6; ++c) W.sig[ei][c][q] = gp_stress ? gp_stress[(e * nq + q) * 6 + c] : 0.0;
    }
    __syncwarp();
    const int row = lane >> 2, col = lane & 3, turn = G::turn(row);
#pragma unroll 1
    for (int ei = 0; ei < EPB && e0 + ei < A.n_elems; ++ei) {
      double* out = reinterpret_cast<double*>(V.edata) + (e0 + ei) * blocks_padded(n);
      if constexpr (KIND == LUMPED) {
        // row sums sum_b sum_q s N_a N_b on the diagonal, zeros elsewhere
        for (int t = lane; t < NB; t += 32) out[t] = 0.0;
        __syncwarp();
        for (int a = lane; a < n; a += 32) {
          double m = 0.0;
          for (int b = 0; b < n; ++b) {
            double v = 0.0;
            for (int q = 0; q < nq; ++q) v += W.s[ei][q] * sN[a * NQP + q] * sN[b * NQP + q];
            m += v;
          }
          out[blk_index(n, a, a)] = m;
        }
        continue;
      }
#pragma unroll 1
      for (int ta = 0; ta < G::NTL; ++ta)
#pragma unroll 1
        for (int tb = ta; tb < G::NTL; ++tb) {
          double acc[3][2] = {};  // one sum per component, so that the products overlap
          const double* gA = (GRAD ? W.g + ei * ES : sN) + (8 * ta + row) * QS + col;
          const double* gB = (GRAD ? W.g + ei * ES : sN) + (8 * tb + row) * QS + col;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            const double s = W.s[ei][4 * ks + col];
            if constexpr (!GRAD) {
              dmma(acc[ks % 3], s * gA[4 * ks], gB[4 * ks]);
            } else {
              double a[3];
#pragma unroll
              for (int x = 0; x < 3; ++x) a[x] = s * gA[x * P + ((4 * ks) ^ turn)];
              if constexpr (GEO) {
                const int q = 4 * ks + col;
                const double s0 = W.sig[ei][0][q], s1 = W.sig[ei][1][q], s2 = W.sig[ei][2][q], s3 = W.sig[ei][3][q],
                             s4 = W.sig[ei][4][q], s5 = W.sig[ei][5][q], a0 = a[0], a1 = a[1], a2 = a[2];
                a[0] = s0 * a0 + s3 * a1 + s4 * a2;
                a[1] = s3 * a0 + s1 * a1 + s5 * a2;
                a[2] = s4 * a0 + s5 * a1 + s2 * a2;
              }
#pragma unroll
              for (int x = 0; x < 3; ++x) dmma(acc[x], a[x], gB[x * P + ((4 * ks) ^ turn)]);
            }
          }
          const int a = 8 * ta + row;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int b = 8 * tb + 2 * col + h;
            if (a < n && b < n && a <= b) out[blk_index(n, a, b)] = (acc[0][h] + acc[1][h]) + acc[2][h];
          }
        }
    }
    __syncwarp();
  }
}

template <int ET, int KIND>
cudaError_t launch_scalar_t(const ElemArgs& a, const V2Args& v, const double* density, const double* gp_stress,
                            cudaStream_t s) {
  if (a.n_elems == 0) return cudaSuccess;
  constexpr size_t smem = scalar_smem_bytes<ET, KIND>();
  constexpr int per_block = kW1 * DGeo<ET>::EPB;
  ElemArgs A = a;
  V2Args V = v;
  void* args[] = {&A, &V, &density, &gp_stress};
  return launch_persistent(reinterpret_cast<const void*>(scalar_kernel<ET, KIND>), smem,
                           (a.n_elems + per_block - 1) / per_block, 0, s, args);
}

template <int ET>
cudaError_t launch_scalar_type(int kind, const ElemArgs& a, const V2Args& v, const double* density,
                               const double* gp_stress, cudaStream_t s) {
  switch (kind) {
    case MASS: return launch_scalar_t<ET, MASS>(a, v, density, gp_stress, s);
    case LUMPED: return launch_scalar_t<ET, LUMPED>(a, v, density, gp_stress, s);
    case GEOMETRIC: return launch_scalar_t<ET, GEOMETRIC>(a, v, density, gp_stress, s);
    case CONDUCTION: return launch_scalar_t<ET, CONDUCTION>(a, v, density, gp_stress, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_scalar_pass(int t, int kind, const ElemArgs& a, const V2Args& v, const double* density,
                               const double* gp_stress, cudaStream_t s) {
  switch (t) {
    case C3D4: return launch_scalar_type<C3D4>(kind, a, v, density, gp_stress, s);
    case C3D10: return launch_scalar_type<C3D10>(kind, a, v, density, gp_stress, s);
    case C3D8: return launch_scalar_type<C3D8>(kind, a, v, density, gp_stress, s);
    case C3D8R: return launch_scalar_type<C3D8R>(kind, a, v, density, gp_stress, s);
    case C3D20: return launch_scalar_type<C3D20>(kind, a, v, density, gp_stress, s);
    case C3D20R: return launch_scalar_type<C3D20R>(kind, a, v, density, gp_stress, s);
    case C3D6: return launch_scalar_type<C3D6>(kind, a, v, density, gp_stress, s);
    case C3D15: return launch_scalar_type<C3D15>(kind, a, v, density, gp_stress, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_named_twice(int precision, const ElemArgs& a, const V2Args& v, cudaStream_t s) {
  const int64_t count = v.e_end - v.e_begin;
  if (!v.named_twice || count <= 0) return cudaSuccess;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((count + 255) / 256, 148 * 8));
  if (precision)
    named_twice_kernel<float><<<grid, 256, 0, s>>>(a, v);
  else
    named_twice_kernel<double><<<grid, 256, 0, s>>>(a, v);
  return cudaGetLastError();
}

cudaError_t launch_p1_fp64(int t, int mode, const ElemArgs& a, const V2Args& v, const LaunchCfg& c, cudaStream_t s) {
  const bool tan = mode == MODE_TANGENT;
  cudaError_t e = cudaErrorInvalidValue;
  switch (t) {
#define CXG_P1(T) \
  case T:                                                                     \
    e = tan ? launch_t<T, true>(a, v, c, s) : launch_t<T, false>(a, v, c, s); \
    break;
    CXG_P1(C3D4)
    CXG_P1(C3D10)
    CXG_P1(C3D8)
    CXG_P1(C3D8R)
    CXG_P1(C3D20)
    CXG_P1(C3D20R)
    CXG_P1(C3D6)
    CXG_P1(C3D15)
#undef CXG_P1
    default: break;
  }
  return e == cudaSuccess ? launch_named_twice(0, a, v, s) : e;
}

const void* p1_fp64_batch(int mode) {
  return mode == MODE_TANGENT ? reinterpret_cast<const void*>(p1_fp64_batch_kernel<true>)
                              : reinterpret_cast<const void*>(p1_fp64_batch_kernel<false>);
}

P1Shape p1_fp64_shape(int t, int mode) {
  const bool tan = mode == MODE_TANGENT;
  switch (t) {
#define CXG_SH(T) \
  case T:         \
    return {tan ? p1d_smem_bytes<T, true>() : p1d_smem_bytes<T, false>(), DGeo<T>::EPB};
    CXG_SH(C3D4)
    CXG_SH(C3D10)
    CXG_SH(C3D8)
    CXG_SH(C3D8R)
    CXG_SH(C3D20)
    CXG_SH(C3D20R)
    CXG_SH(C3D6)
#undef CXG_SH
    default: return {tan ? p1d_smem_bytes<C3D15, true>() : p1d_smem_bytes<C3D15, false>(), DGeo<C3D15>::EPB};
  }
}

}  // namespace cxg
