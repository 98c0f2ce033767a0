// CSR pattern of the reduced free/free system, built on the device.
//
// The reference accumulates (row, col) keys into an unordered_map element by element
// (src/fem/assembly.cpp:76-100) and flushes unordered COO triplets (211-221). Here the
// pattern is built once per mesh and DOF map, in canonical sorted CSR form, node by node:
//   1. the node -> element incidence comes from one stable sort of the connectivity;
//   2. one warp per node gathers the nodes of its incident elements (its candidates, in
//      element order), and orders them by (node, position) in shared memory (lists of more
//      than 2048 by a block each beforehand): equal nodes are then one neighbour of the node
//      and its contributions in element order;
//   3. a first sweep counts: neighbours, the row length (all rows of a node share one
//      column structure, the free components of its neighbours, ascending), the cuts of
//      the contribution list; scans over the nodes give every node its place in the CSR
//      arrays and in the record lists. This relies on the reference's free numbering being
//      ascending in g = 3*node + comp (constraint_transform.cpp:78-82), which is validated;
//   4. a second sweep orders the candidates again and writes row_ptr, col_idx, the
//      records that the row gather reads (NodeRec, PairRec) and, for the nodes with a
//      neighbour that is not fully free (their rows are compressed), the neighbours and
//      their columns (BndRec).
// A global sort of all element node pairs would carry 24 bytes of scratch per pair through
// six passes, and its allocations alone took longer than both sweeps together.
// The pattern is topological: an entry whose every element contribution is exactly
// zero is kept (the reference skips exact-zero contributions, assembly.cpp:90).
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>

#include "cxg_internal.cuh"

namespace cxg {
namespace {

struct BuildFlags {
  int bad_conn, bad_numbering, too_many, named_twice;
  unsigned long long bad_elem;
};

__global__ void check_conn_kernel(const int32_t* conn, int64_t total, int64_t n_nodes, int npe, int32_t* codes,
                                  BuildFlags* f) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t v = conn[i];
    codes[i] = static_cast<int32_t>(i);
    if (v < 0 || v >= n_nodes) {
      atomicExch(&f->bad_conn, 1);
      atomicMin(&f->bad_elem, static_cast<unsigned long long>(i / npe));
    }
  }
}

// Free-component mask and first equation of every node, and the free count scanned below.
__global__ void node_info_kernel(const int32_t* dof_eq, int64_t n_nodes, uint8_t* mask, int32_t* eq0, int32_t* free) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n_nodes;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int m = 0;
    int32_t first = -1;
    for (int d = 0; d < 3; ++d) {
      const int32_t eq = dof_eq[3 * a + d];
      if (eq >= 0) {
        m |= 1 << d;
        if (first < 0) first = eq;
      }
    }
    mask[a] = static_cast<uint8_t>(m);
    eq0[a] = first;
    free[a] = __popc(m);
  }
}

__global__ void check_numbering_kernel(const int32_t* dof_eq, const int32_t* scan, const uint8_t* mask, int64_t n_nodes,
                                       int32_t n_free, BuildFlags* f) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n_nodes;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int32_t next = scan[a];
    for (int d = 0; d < 3; ++d) {
      const int32_t eq = dof_eq[3 * a + d];
      if (eq < -1 || (eq >= 0 && eq != next)) atomicExch(&f->bad_numbering, 1);
      next += eq >= 0;
    }
    if (a == n_nodes - 1 && next != n_free) atomicExch(&f->bad_numbering, 1);
  }
}

__global__ void inc_ptr_kernel(const int32_t* sorted_nodes, int64_t m, int64_t n_nodes, int64_t* ptr) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a <= n_nodes;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t lo = 0, hi = m;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (sorted_nodes[mid] < a)
        lo = mid + 1;
      else
        hi = mid;
    }
    ptr[a] = lo;
  }
}

__global__ void max_inc_kernel(const int64_t* inc_ptr, int64_t n_nodes, int* out) {
  int m = 0;
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n_nodes;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x)
    m = max(m, static_cast<int>(inc_ptr[a + 1] - inc_ptr[a]));
  m = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(m));
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(out, m);
}

constexpr int kWarps = 4;

// What both sweeps read of the mesh. Candidate c of a node is local node c % npe of its
// c / npe-th incident element.
struct Sweep {
  const int32_t* conn;
  const int64_t* inc_ptr;
  const int32_t* inc_code;
  int npe, nbp;
};

// A candidate: its node and its position, ordered by (node, position).
struct __align__(8) Cand {
  int32_t c, node;
  __device__ bool operator<(const Cand& o) const { return node < o.node || (node == o.node && c < o.c); }
};

// The candidates of node a in order; returns their number. A bitonic sort in the warp's list,
// filled up to a power of two: counting for each candidate the smaller ones takes cnt^2 / 32
// steps a lane, and C3D10 corner nodes have 240 (49,266 C3D10, both sweeps: 560 -> 413 us).
__device__ int order_candidates(const Sweep& S, int64_t a, Cand* k) {
  const int lane = threadIdx.x & 31;
  const int64_t i0 = S.inc_ptr[a];
  const int n = S.npe, cnt = static_cast<int>(S.inc_ptr[a + 1] - i0) * n;
  int m = 2;
  while (m < cnt) m *= 2;
  for (int c = lane; c < m; c += 32)
    k[c] = Cand{c, c < cnt ? S.conn[static_cast<int64_t>(S.inc_code[i0 + c / n] / n) * n + c % n] : 0x7fffffff};
  __syncwarp();
  for (int len = 2; len <= m; len *= 2)
    for (int d = len / 2; d > 0; d /= 2) {
      for (int t = lane; t < m / 2; t += 32) {
        const int lo = 2 * t - (t & (d - 1)), hi = lo + d;
        const Cand x = k[lo], y = k[hi];
        if ((y < x) == ((lo & len) == 0)) {
          k[lo] = y;
          k[hi] = x;
        }
      }
      __syncwarp();
    }
  return cnt;
}

// Nodes with more candidates than a warp's list in shared memory holds (kList): a block each
// orders them, in shared memory up to kBlockList of them, and both sweeps read the result.
// (In the sweeps themselves, one warp and every node's list in global memory, a fan of 360
// wedges took 3.0 ms for a plan, 1.0 so; with a sort of all pairs 2.2.)
constexpr int kList = 2048, kBlockList = 16384, kHubThreads = 1024;
struct Hub {
  int64_t at;  // its list's place
  int32_t node;
};
struct HubTotals {
  unsigned long long count, cands;
};

__device__ __forceinline__ int64_t power_of_two(int64_t n) {
  int64_t m = 2;
  while (m < n) m *= 2;
  return m;
}

// hubs null: their number and their lists' total length.
__global__ void hubs_kernel(Sweep S, int64_t n_nodes, HubTotals* t, Hub* hubs) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n_nodes;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t cnt = (S.inc_ptr[a + 1] - S.inc_ptr[a]) * S.npe;
    if (cnt <= kList) continue;
    const unsigned long long i = atomicAdd(&t->count, 1ull), at = atomicAdd(&t->cands, static_cast<unsigned long long>(power_of_two(cnt)));
    if (hubs) hubs[i] = Hub{static_cast<int64_t>(at), static_cast<int32_t>(a)};
  }
}

__global__ void __launch_bounds__(kHubThreads) sort_hubs_kernel(Sweep S, const Hub* hubs, int64_t n_hubs, Cand* lists) {
  extern __shared__ Cand sh[];
  for (int64_t h = blockIdx.x; h < n_hubs; h += gridDim.x) {
    const int64_t a = hubs[h].node, i0 = S.inc_ptr[a], cnt = (S.inc_ptr[a + 1] - i0) * S.npe, m = power_of_two(cnt);
    Cand* out = lists + hubs[h].at;
    Cand* k = m <= kBlockList ? sh : out;
    for (int64_t c = threadIdx.x; c < m; c += kHubThreads)
      k[c] = Cand{static_cast<int32_t>(c),
                  c < cnt ? S.conn[static_cast<int64_t>(S.inc_code[i0 + c / S.npe] / S.npe) * S.npe + c % S.npe] : 0x7fffffff};
    __syncthreads();
    for (int64_t len = 2; len <= m; len *= 2)
      for (int64_t d = len / 2; d > 0; d /= 2) {
        for (int64_t t = threadIdx.x; t < m / 2; t += kHubThreads) {
          const int64_t lo = 2 * t - (t & (d - 1)), hi = lo + d;
          const Cand x = k[lo], y = k[hi];
          if ((y < x) == ((lo & len) == 0)) {
            k[lo] = y;
            k[hi] = x;
          }
        }
        __syncthreads();
      }
    if (k != out)
      for (int64_t c = threadIdx.x; c < cnt; c += kHubThreads) out[c] = k[c];
    __syncthreads();
  }
}

// The nodes of a sweep: those with lists of at most kList candidates, ordered in the warp's
// part of shared memory, or the hubs, whose lists are ordered (HUBS).
template <bool HUBS>
struct Nodes {
  int64_t n;         // nodes, or hubs
  const Hub* hubs;
  Cand* lists;
};

// Neighbours before and contribution runs: calls at(r, p, first) for every candidate rank
// r on its lane, p its neighbour's position and first whether it opens that neighbour.
template <class F>
__device__ void each_candidate(const Cand* k, int cnt, F at) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int r0 = 0; r0 < cnt; r0 += 32) {
    const int r = r0 + lane;
    const bool first = r < cnt && (r == 0 || k[r].node != k[r - 1].node);
    const unsigned w = __ballot_sync(0xffffffffu, first);
    const int p = before + __popc(w & ((2u << lane) - 1)) - 1;
    at(r, p, first);
    before += __popc(w);
  }
}

// Node a and its ordered candidates k for number a of the sweep; returns how many, or less than
// none for a hub, which has a sweep of its own.
__device__ __forceinline__ int candidates(const Sweep& S, const Nodes<false>&, int64_t& a, Cand*& k) {
  if ((S.inc_ptr[a + 1] - S.inc_ptr[a]) * S.npe > kList) return -1;
  return order_candidates(S, a, k);
}
__device__ __forceinline__ int candidates(const Sweep& S, const Nodes<true>& N, int64_t& a, Cand*& k) {
  const Hub h = N.hubs[a];
  a = h.node;
  k = N.lists + h.at;
  return static_cast<int>(S.inc_ptr[a + 1] - S.inc_ptr[a]) * S.npe;
}

// First sweep: counts, row length, cuts.
template <bool HUBS>
__global__ void __launch_bounds__(kWarps * 32) count_kernel(Sweep S, Nodes<HUBS> N, const uint8_t* mask, int cap,
                                                            NodeRec* node, int64_t* node_nnz, int64_t* bnd_len,
                                                            int64_t* n_rec, BuildFlags* f) {
  extern __shared__ Cand sh[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t gw = static_cast<int64_t>(blockIdx.x) * kWarps + warp, nw = static_cast<int64_t>(gridDim.x) * kWarps;
  for (int64_t w = gw; w < N.n; w += nw) {
    Cand* k = sh + warp * cap;
    int64_t a = w;
    const int cnt = candidates(S, N, a, k);
    if (cnt < 0) continue;
    int len = 0, K = 0, self = 0, own = 0;
    // the neighbour starts nearest to one and two thirds of the contributions
    int cut[2] = {cnt, cnt}, pos[2] = {0, 0}, err[2] = {3 * cnt + 1, 3 * cnt + 1};
    each_candidate(k, cnt, [&](int r, int p, bool first) {
      if (r >= cnt) return;
      own += k[r].node == a;
      if (first) {
        len += __popc(mask[k[r].node]);
        if (k[r].node == a) self = p;
        for (int g = 0; g < 2; ++g) {
          const int d = abs(3 * r - (g + 1) * cnt);
          if (d < err[g]) {
            err[g] = d;
            cut[g] = r;
            pos[g] = p;
          }
        }
      }
      K = max(K, p + 1);
    });
    len = __reduce_add_sync(0xffffffffu, static_cast<unsigned>(len));
    K = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(K));
    self = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(self));
    own = __reduce_add_sync(0xffffffffu, static_cast<unsigned>(own));
    for (int g = 0; g < 2; ++g) {
      // (the end of the list is a cut too, for nodes with one or two neighbours)
      const unsigned e = __reduce_min_sync(0xffffffffu, static_cast<unsigned>(err[g]));
      const unsigned win = __ballot_sync(0xffffffffu, static_cast<unsigned>(err[g]) == e && cut[g] < cnt);
      const int src = win ? __ffs(win) - 1 : 0;
      const bool end = static_cast<unsigned>(3 * cnt - (g + 1) * cnt) < e || !win;
      const int c = __shfl_sync(0xffffffffu, cut[g], src), q = __shfl_sync(0xffffffffu, pos[g], src);
      cut[g] = end ? cnt : c;
      pos[g] = end ? K : q;
    }
    if (lane == 0) {
      const int longest = max(cut[0], max(cut[1] - cut[0], cnt - cut[1]));
      NodeRec r{};
      r.len_mask = static_cast<uint32_t>(len);
      r.rounds = static_cast<uint32_t>((longest + kPairRec - 1) / kPairRec);
      r.npair = static_cast<uint16_t>(K);
      r.diag = static_cast<uint16_t>(self);
      r.pair1 = static_cast<uint16_t>(pos[0]);
      r.pair2 = static_cast<uint16_t>(pos[1]);
      r.pad[0] = static_cast<uint32_t>(cut[0]);
      r.pad[1] = static_cast<uint32_t>(cut[1]);
      if (K > 65535) atomicExch(&f->too_many, 1);  // list positions are uint16
      if (own * S.npe != cnt) atomicExch(&f->named_twice, 1);  // not once per incident element
      node[a] = r;
      node_nnz[a] = static_cast<int64_t>(__popc(mask[a])) * len;
      bnd_len[a] = len == 3 * K ? 0 : K;
      n_rec[a] = 3 * static_cast<int64_t>(r.rounds);
    }
    __syncwarp();
  }
}

// Second sweep: the CSR rows, the records and the lists of the compressed-row nodes.
template <bool HUBS>
__global__ void __launch_bounds__(kWarps * 32) write_kernel(Sweep S, Nodes<HUBS> N, const uint8_t* mask,
                                                            const int32_t* eq0, const double* prescribed,
                                                            const int64_t* node_base, const int64_t* bnd_ptr,
                                                            const int64_t* rec_ptr, int cap, NodeRec* node,
                                                            int64_t* row_ptr, int32_t* col_idx, PairRec* pairs,
                                                            BndRec* bnd) {
  extern __shared__ Cand sh[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t gw = static_cast<int64_t>(blockIdx.x) * kWarps + warp, nw = static_cast<int64_t>(gridDim.x) * kWarps;
  for (int64_t w = gw; w < N.n; w += nw) {
    Cand* k = sh + warp * cap;
    int64_t a = w;
    const int cnt = candidates(S, N, a, k);
    if (cnt < 0) continue;
    NodeRec nd = node[a];
    const int cut1 = static_cast<int>(nd.pad[0]), cut2 = static_cast<int>(nd.pad[1]);
    const int L = static_cast<int>(nd.len_mask), ma = mask[a], nfa = __popc(ma), K = nd.npair;
    nd.base = node_base[a];
    nd.list0 = static_cast<uint32_t>(rec_ptr[a]);
    nd.bnd0 = static_cast<uint32_t>(bnd_ptr[a]);
    nd.eq0 = eq0[a];
    nd.len_mask = static_cast<uint32_t>(L) | static_cast<uint32_t>(ma) << 28;
    nd.pad[0] = nd.pad[1] = 0;
    __syncwarp();
    if (lane == 0) node[a] = nd;
    if (lane < nfa) row_ptr[nd.eq0 + lane] = nd.base + static_cast<int64_t>(lane) * L;
    // columns: the free components of the neighbours in order
    int run = 0, own = -1;  // free components of the neighbours before this chunk; rank of the own pair
    each_candidate(k, cnt, [&](int r, int p, bool first) {
      const int b = first ? k[r].node : 0;
      const int mb = first ? mask[b] : 0, pc = __popc(mb);
      int incl = pc;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
      }
      const int col = run + incl - pc;
      run += __shfl_sync(0xffffffffu, incl, 31);
      if (!first) return;
      if (b == a) own = r;
      const int32_t e = eq0[b];
      for (int i = 0; i < nfa; ++i)
        for (int j = 0; j < pc; ++j) col_idx[nd.base + static_cast<int64_t>(i) * L + col + j] = e + j;
      if (L != 3 * K) {
        bool moves = false;
        for (int d = 0; d < 3; ++d) moves = moves || (!((mb >> d) & 1) && prescribed[3 * static_cast<int64_t>(b) + d] != 0.0);
        bnd[nd.bnd0 + p] = BndRec{static_cast<uint32_t>(col) | static_cast<uint32_t>(mb) << 28 | (moves ? 0x80000000u : 0u), b};
      }
    });
    own = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(own + 1)) - 1;
    // records: run g holds ranks [lo, hi), record r of it 11 of them
    const int from[4] = {0, cut1, cut2, cnt};
    int turn = -1;  // round in which the pair before the own one ends (not at a run's start)
    for (int g = 0; g < 3; ++g)
      if (own > from[g] && own < from[g + 1]) turn = (own - 1 - from[g]) / kPairRec;
    const int64_t i0 = S.inc_ptr[a];
    const int n = S.npe;
    auto block = [&](int r) {
      const int c = k[r].c, code = S.inc_code[i0 + c / n], la = code % n, lb = c % n;
      return static_cast<uint32_t>((code / n) * S.nbp + (la <= lb ? blk_index(n, la, lb) : blk_index(n, lb, la)));
    };
    for (int i = lane; i < 3 * static_cast<int>(nd.rounds); i += 32) {
      const int g = i % 3, lo = g == 0 ? 0 : g == 1 ? cut1 : cut2, hi = g == 0 ? cut1 : g == 1 ? cut2 : cnt;
      PairRec rec;
      rec.flags = i / 3 == turn ? 0x80000000u : 0u;
      for (int j = 0; j < kPairRec; ++j) {
        const int r = lo + i / 3 * kPairRec + j;
        if (r < hi) {
          rec.block[j] = block(r);
          if (r + 1 == cnt || k[r].node != k[r + 1].node) rec.flags |= 1u << j;
          if (r + 1 == own && r + 1 < hi) rec.flags |= 0x10000u << j;
        } else {
          rec.block[j] = block(hi > lo ? hi - 1 : 0);
        }
      }
      pairs[nd.list0 + i] = rec;
    }
    __syncwarp();
  }
}

unsigned grid_for(int64_t n, int threads = 256) {
  return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 65536)));
}

// Parts of one device block, each 256-byte aligned.
struct Parts {
  size_t bytes = 0;
  template <typename T>
  size_t add(size_t count) {
    const size_t at = bytes;
    bytes += (std::max<size_t>(count, 1) * sizeof(T) + 255) / 256 * 256;
    return at;
  }
};
template <typename T>
T* part(void* base, size_t at) {
  return reinterpret_cast<T*>(static_cast<char*>(base) + at);
}

}  // namespace

#define CXG_TRY(expr)                                  \
  do {                                                 \
    cudaError_t _e = (expr);                           \
    if (_e != cudaSuccess) {                           \
      *msg = cudaGetErrorString(_e);                   \
      rc = _e == cudaErrorMemoryAllocation ? 3 : 2;    \
      goto done;                                       \
    }                                                  \
  } while (0)

int build_pattern(int elem_type, int64_t n_nodes, int64_t n_elems, const int32_t* d_conn,
                  const int32_t* d_dof_eq, const double* d_prescribed, int32_t n_free, PatternOut* out, const char** msg,
                  cudaStream_t s) {
  const int npe = nodes_of(elem_type);
  const int64_t P = n_elems * npe * npe, m = n_elems * npe;
  int rc = 0;
  if (P >= (static_cast<int64_t>(1) << 31)) {
    *msg = "mesh too large for one plan (n_elems * nodes^2 >= 2^31); split it into partitions";
    return 5;
  }
  if (n_nodes >= (static_cast<int64_t>(1) << 31)) {
    *msg = "node count exceeds int32 indexing";
    return 5;
  }
  const int in = static_cast<int>(n_nodes), im = static_cast<int>(m);
  int node_bits = 1;
  while (node_bits < 31 && (n_nodes >> node_bits) != 0) ++node_bits;

  // What stays with the plan and has a known size, and the build's scratch: one block each.
  void* scratch = nullptr;
  void* hub_mem = nullptr;
  Parts keep, tmp;
  const size_t k_mask = keep.add<uint8_t>(n_nodes), k_node = keep.add<NodeRec>(n_nodes),
               k_row = keep.add<int64_t>(static_cast<size_t>(n_free) + 1), k_inc = keep.add<int64_t>(n_nodes + 1),
               k_code = keep.add<int32_t>(m);
  size_t sort_bytes = 0, scan32 = 0, scan64 = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, static_cast<const int32_t*>(nullptr),
                                  static_cast<int32_t*>(nullptr), static_cast<const int32_t*>(nullptr),
                                  static_cast<int32_t*>(nullptr), im, 0, node_bits, s);
  cub::DeviceScan::ExclusiveSum(nullptr, scan32, static_cast<int32_t*>(nullptr), static_cast<int32_t*>(nullptr), in, s);
  cub::DeviceScan::ExclusiveSum(nullptr, scan64, static_cast<int64_t*>(nullptr), static_cast<int64_t*>(nullptr), in, s);
  const size_t cub_bytes = std::max(sort_bytes, std::max(scan32, scan64));
  const size_t t_flags = tmp.add<BuildFlags>(1), t_max = tmp.add<int>(1), t_hubs = tmp.add<HubTotals>(2), t_cub = tmp.add<char>(cub_bytes),
               t_eq0 = tmp.add<int32_t>(n_nodes), t_free = tmp.add<int32_t>(n_nodes), t_scan = tmp.add<int32_t>(n_nodes),
               t_sorted = tmp.add<int32_t>(m), t_codes = tmp.add<int32_t>(m);
  size_t t_len[3], t_off[3];  // node_nnz, bnd_len, n_rec and their scans
  for (int i = 0; i < 3; ++i) {
    t_len[i] = tmp.add<int64_t>(n_nodes);
    t_off[i] = tmp.add<int64_t>(n_nodes);
  }
  BuildFlags hf{};
  int max_inc = 0, cap = 0;
  int64_t last[3] = {0, 0, 0}, len[3] = {0, 0, 0};
  Sweep S{};
  Nodes<false> nodes{n_nodes, nullptr, nullptr};
  Nodes<true> hubs{0, nullptr, nullptr};
  unsigned sweep_grid = 0, hub_grid = 0;
  size_t sweep_smem = 0;
  {
    CXG_TRY(device_alloc(&out->mem[0], keep.bytes));
    out->device_bytes += static_cast<int64_t>(keep.bytes);
    CXG_TRY(device_alloc(&scratch, tmp.bytes));
    out->node_mask = part<uint8_t>(out->mem[0], k_mask);
    out->node = part<NodeRec>(out->mem[0], k_node);
    out->row_ptr = part<int64_t>(out->mem[0], k_row);
    out->inc_ptr = part<int64_t>(out->mem[0], k_inc);
    out->inc_code = part<int32_t>(out->mem[0], k_code);
    BuildFlags* f = part<BuildFlags>(scratch, t_flags);
    int* d_max = part<int>(scratch, t_max);
    hf.bad_elem = ~0ull;
    CXG_TRY(cudaMemcpyAsync(f, &hf, sizeof hf, cudaMemcpyHostToDevice, s));
    CXG_TRY(cudaMemsetAsync(d_max, 0, sizeof(int), s));
    int32_t* eq0 = part<int32_t>(scratch, t_eq0);
    int32_t* codes = part<int32_t>(scratch, t_codes);
    int32_t* sorted = part<int32_t>(scratch, t_sorted);
    check_conn_kernel<<<grid_for(m), 256, 0, s>>>(d_conn, m, n_nodes, npe, codes, f);
    node_info_kernel<<<grid_for(n_nodes), 256, 0, s>>>(d_dof_eq, n_nodes, out->node_mask, eq0,
                                                       part<int32_t>(scratch, t_free));
    CXG_TRY(cudaGetLastError());
    size_t cb = cub_bytes;
    CXG_TRY(cub::DeviceScan::ExclusiveSum(part<char>(scratch, t_cub), cb, part<int32_t>(scratch, t_free),
                                          part<int32_t>(scratch, t_scan), in, s));
    check_numbering_kernel<<<grid_for(n_nodes), 256, 0, s>>>(d_dof_eq, part<int32_t>(scratch, t_scan), out->node_mask,
                                                             n_nodes, n_free, f);
    // node -> element incidence: stable sort of (node, e*n + local) by node. Nodes outside
    // the mesh (an error, reported below) sort by their low bits and are not followed.
    CXG_TRY(cub::DeviceRadixSort::SortPairs(part<char>(scratch, t_cub), cb, d_conn, sorted, codes, out->inc_code, im, 0,
                                            node_bits, s));
    CXG_TRY(cudaMemcpyAsync(&hf, f, sizeof hf, cudaMemcpyDeviceToHost, s));
    inc_ptr_kernel<<<grid_for(n_nodes + 1), 256, 0, s>>>(sorted, m, n_nodes, out->inc_ptr);
    max_inc_kernel<<<grid_for(n_nodes), 256, 0, s>>>(out->inc_ptr, n_nodes, d_max);
    CXG_TRY(cudaGetLastError());
    CXG_TRY(cudaMemcpyAsync(&max_inc, d_max, sizeof(int), cudaMemcpyDeviceToHost, s));
    CXG_TRY(cudaStreamSynchronize(s));
    if (hf.bad_conn) {
      static thread_local char buf[160];
      snprintf(buf, sizeof buf, "element references unknown node (element index %llu)", hf.bad_elem);
      *msg = buf;
      rc = 6;
      goto done;
    }
    if (hf.bad_numbering) {
      *msg = "dof_eq must number the free DOFs 0..n_free-1 in increasing global DOF order "
             "(SPC-only constraint transform)";
      rc = 5;
      goto done;
    }
    S = Sweep{d_conn, out->inc_ptr, out->inc_code, npe, blocks_padded(npe)};
    for (cap = 2; cap < max_inc * npe && cap < kList;) cap *= 2;
    sweep_smem = sizeof(Cand) * kWarps * static_cast<size_t>(cap);
    sweep_grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n_nodes + kWarps - 1) / kWarps, 65536)));
    CXG_TRY(allow_smem(reinterpret_cast<const void*>(count_kernel<false>), sweep_smem));
    CXG_TRY(allow_smem(reinterpret_cast<const void*>(write_kernel<false>), sweep_smem));
    if (static_cast<int64_t>(max_inc) * npe > kList) {
      HubTotals* totals = part<HubTotals>(scratch, t_hubs);  // counted, then taken up again while the lists are placed
      HubTotals h{};
      CXG_TRY(cudaMemsetAsync(totals, 0, 2 * sizeof(HubTotals), s));
      hubs_kernel<<<grid_for(n_nodes), 256, 0, s>>>(S, n_nodes, totals, nullptr);
      CXG_TRY(cudaMemcpyAsync(&h, totals, sizeof h, cudaMemcpyDeviceToHost, s));
      CXG_TRY(cudaStreamSynchronize(s));
      Parts hp;
      const size_t h_hub = hp.add<Hub>(h.count), h_list = hp.add<Cand>(h.cands);
      CXG_TRY(device_alloc(&hub_mem, hp.bytes));
      hubs = Nodes<true>{static_cast<int64_t>(h.count), part<Hub>(hub_mem, h_hub), part<Cand>(hub_mem, h_list)};
      hub_grid = static_cast<unsigned>(std::min<int64_t>((hubs.n + kWarps - 1) / kWarps, 65536));
      hubs_kernel<<<grid_for(n_nodes), 256, 0, s>>>(S, n_nodes, totals + 1, part<Hub>(hub_mem, h_hub));
      CXG_TRY(cudaGetLastError());
      CXG_TRY(allow_smem(reinterpret_cast<const void*>(sort_hubs_kernel), sizeof(Cand) * kBlockList));
      sort_hubs_kernel<<<static_cast<unsigned>(std::min<int64_t>(hubs.n, 65536)), kHubThreads, sizeof(Cand) * kBlockList, s>>>(
          S, hubs.hubs, hubs.n, hubs.lists);
      CXG_TRY(cudaGetLastError());
    }
    int64_t *lens[3], *offs[3];
    for (int i = 0; i < 3; ++i) {
      lens[i] = part<int64_t>(scratch, t_len[i]);
      offs[i] = part<int64_t>(scratch, t_off[i]);
    }
    count_kernel<false><<<sweep_grid, kWarps * 32, sweep_smem, s>>>(S, nodes, out->node_mask, cap, out->node, lens[0],
                                                                    lens[1], lens[2], f);
    if (hub_grid)
      count_kernel<true><<<hub_grid, kWarps * 32, 0, s>>>(S, hubs, out->node_mask, 0, out->node, lens[0], lens[1],
                                                          lens[2], f);
    CXG_TRY(cudaGetLastError());
    for (int i = 0; i < 3; ++i) {
      cb = cub_bytes;
      CXG_TRY(cub::DeviceScan::ExclusiveSum(part<char>(scratch, t_cub), cb, lens[i], offs[i], in, s));
      if (n_nodes > 0) {
        CXG_TRY(cudaMemcpyAsync(&last[i], offs[i] + n_nodes - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        CXG_TRY(cudaMemcpyAsync(&len[i], lens[i] + n_nodes - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
      }
    }
    CXG_TRY(cudaMemcpyAsync(&hf, f, sizeof hf, cudaMemcpyDeviceToHost, s));
    CXG_TRY(cudaStreamSynchronize(s));
    if (hf.too_many) {
      *msg = "a node has more than 65535 neighbours; not supported";
      rc = 5;
      goto done;
    }
    out->named_twice = hf.named_twice != 0;
    out->nnz = last[0] + len[0];
    // (one more: the gather reads the record after a list's last)
    const size_t nbnd = static_cast<size_t>(last[1] + len[1]) + 1;
    Parts rest;
    const size_t r_col = rest.add<int32_t>(static_cast<size_t>(out->nnz)),
                 r_pairs = rest.add<PairRec>(static_cast<size_t>(last[2] + len[2])), r_bnd = rest.add<BndRec>(nbnd);
    CXG_TRY(device_alloc(&out->mem[1], rest.bytes));
    out->device_bytes += static_cast<int64_t>(rest.bytes);
    out->col_idx = part<int32_t>(out->mem[1], r_col);
    out->pairs = part<PairRec>(out->mem[1], r_pairs);
    out->bnd = part<BndRec>(out->mem[1], r_bnd);
    CXG_TRY(cudaMemcpyAsync(out->row_ptr + n_free, &out->nnz, sizeof(int64_t), cudaMemcpyHostToDevice, s));
    write_kernel<false><<<sweep_grid, kWarps * 32, sweep_smem, s>>>(S, nodes, out->node_mask, eq0, d_prescribed, offs[0],
                                                                    offs[1], offs[2], cap, out->node, out->row_ptr,
                                                                    out->col_idx, out->pairs, out->bnd);
    if (hub_grid)
      write_kernel<true><<<hub_grid, kWarps * 32, 0, s>>>(S, hubs, out->node_mask, eq0, d_prescribed, offs[0], offs[1],
                                                          offs[2], 0, out->node, out->row_ptr, out->col_idx, out->pairs,
                                                          out->bnd);
    CXG_TRY(cudaGetLastError());
    CXG_TRY(cudaStreamSynchronize(s));
  }

done:
  cudaStreamSynchronize(s);  // (an error may have left work on the scratch)
  device_free(hub_mem);
  device_free(scratch);
  return rc;
}

}  // namespace cxg
