// P2, the row gather: every CSR value written exactly once, no atomics, no shared memory (an
// accumulating assembly adds each value once, as a reduction in L2).
//
// One warp per node a. The plan lists the element blocks that contribute to a's node pairs
// (a, b), pair by pair and in element order, in records of 11 (NodeRec, PairRec). Three
// groups of nine lanes each walk a third of that list; a lane carries one entry of the 3x3
// block. A contribution is one coalesced 72-byte (FP32: 36-byte) read and one add in a
// register, and where a pair ends the group writes its block, three runs of three values
// that the next pairs of the same rows continue. The three runs are padded to the same
// number of records, so a round is straight-line code: 11 block reads in flight per lane,
// the next record fetched meanwhile.
//
// What bounds it: the L1's wavefronts (66 to 69 % of its rate) and issue slots. The element
// blocks come in from HBM once and the values go out once; in between the L1 serves every
// block twice (rows of a and of b), one contribution to a read of nine lanes. Against the
// rows summed in shared memory: C3D8 J2 128^3 3852 -> 2798 us, forces included, C3D20 64^3
// mixed 3141 -> 1899.
//
// Mixed precision (DIAG) forms the diagonal block as minus the FP64 sum of the row's
// other entries (per group, then the three groups in order; the element pass stores the
// blocks (a, a) as zeros), so rigid translations stay in the null space to FP64 accuracy.
// Interior nodes (every neighbour fully free) write full-width rows; at the others each
// pair's record (BndRec) gives its compressed column, and prescribed columns go to the rhs
// (-K_fc u_c, src/fem/assembly.cpp:95-96).
#include <cuda_runtime.h>

#include <algorithm>

#include "cxg_internal.cuh"

namespace cxg {

namespace {

constexpr unsigned kAll = 0xffffffffu;
// Warps per block unless the caller asks for others, one node each: blocks are handed out
// as they finish, so nodes of one and of eight incident elements, full and compressed rows
// even out (a grid of resident blocks striding over the nodes: C3D20 64^3 mixed 2885 us,
// this way 2218; blocks of 8 warps 2330).
constexpr int kWarps = 4;
// Grids that are resident at once on a B200, 24 warps a SM whatever the block, let the next
// kernel on the stream start early.
__device__ __forceinline__ bool one_wave() { return gridDim.x * (blockDim.x >> 5) <= 148 * 24; }
// (Registers: 64 a thread where the blocks are FP32, bound by the launch bounds: C3D20 64^3
// 2190 us without, 2007 with; 68 where they are FP64, 64 spill there.)

__device__ __forceinline__ NodeRec load_node(const NodeRec* p) {
  union {
    int4 q[3];
    NodeRec r;
  } u;
#pragma unroll
  for (int i = 0; i < 3; ++i) u.q[i] = __ldg(reinterpret_cast<const int4*>(p) + i);
  return u.r;
}

// The same, not merged with an earlier load.
__device__ __forceinline__ NodeRec fresh_node(const NodeRec* p) {
  union {
    int4 q[3];
    NodeRec r;
  } u;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(u.q[i].x), "=r"(u.q[i].y), "=r"(u.q[i].z), "=r"(u.q[i].w)
                 : "l"(reinterpret_cast<const int4*>(p) + i));
  return u.r;
}

__device__ __forceinline__ PairRec load_pairs(const PairRec* p) {
  union {
    int4 q[3];
    PairRec r;
  } u;
#pragma unroll
  for (int i = 0; i < 3; ++i) u.q[i] = __ldg(reinterpret_cast<const int4*>(p) + i);
  return u.r;
}

__device__ __forceinline__ BndRec load_bnd(const BndRec* p) {
  const int2 q = __ldg(reinterpret_cast<const int2*>(p));
  return {static_cast<uint32_t>(q.x), q.y};
}

// Index of a stored block in the element buffer. With windows the buffer is a ring of
// `ring` elements; every element of a window lies in [ring_base, ring_base + 2 ring), so
// one conditional subtraction gives the slot. (A plan has fewer than 2^31 blocks.)
template <bool WIN>
__device__ __forceinline__ int64_t block_slot(uint32_t block, uint32_t ring_blocks, uint32_t base_blocks) {
  if constexpr (WIN) {
    const uint32_t d = block - base_blocks;
    return d < ring_blocks ? d : d - ring_blocks;
  }
  return block;
}

// Where a pair ends: write the entry, start the next pair three columns on. Predicated
// rather than branched: some group ends a pair at most steps. ADD: onto what is there, as a
// reduction in L2 (each entry has one lane, so the sum is the same as read, added and
// written, and nothing waits for the read: 110,592 C3D8 FP64 405 -> 252 us an assembly).
template <bool SUM, bool ADD>
__device__ __forceinline__ void end_pair(unsigned last, double*& o, double& v, double& sum) {
#define CXG_SUMMED(WRITE)                                                                                  \
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %3, 0;\n@p " WRITE " [%0], %1;\n@p add.f64 %2, %2, %1;\n" \
               "@p mov.f64 %1, 0d0000000000000000;\n@p add.s64 %0, %0, 24;\n}"                             \
               : "+l"(o), "+d"(v), "+d"(sum)                                                               \
               : "r"(last)                                                                                 \
               : "memory")
#define CXG_WRITTEN(WRITE)                                                      \
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p " WRITE " [%0], %1;\n" \
               "@p mov.f64 %1, 0d0000000000000000;\n@p add.s64 %0, %0, 24;\n}"  \
               : "+l"(o), "+d"(v)                                               \
               : "r"(last)                                                      \
               : "memory")
  if constexpr (SUM && ADD) CXG_SUMMED("red.global.add.f64");
  if constexpr (SUM && !ADD) CXG_SUMMED("st.global.f64");
  if constexpr (!SUM && ADD) CXG_WRITTEN("red.global.add.f64");
  if constexpr (!SUM && !ADD) CXG_WRITTEN("st.global.f64");
#undef CXG_SUMMED
#undef CXG_WRITTEN
}

// One entry outside such a run.
template <bool ADD>
__device__ __forceinline__ void write_entry(double* o, double v) {
  if constexpr (ADD)
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(o), "d"(v) : "memory");
  else
    *o = v;
}

// The place of a lane in a node's gather: lanes 27 .. 31 follow the third group without writing.
struct Lane {
  int lane, q, ki, kj;
  __device__ __forceinline__ Lane() {
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));  // (made again rather than kept)
    q = min(lane / 9, 2);
    const int k = lane < 27 ? lane - 9 * q : 0;
    ki = k / 3;
    kj = k - 3 * ki;
  }
};

// step(x, ends, turns) for every round of the lane's run: its contributions, and where pairs
// end among them. rec: the run's first record.
template <typename R, bool SCALAR, bool WIN, class F>
__device__ __forceinline__ void each_round(const ElemArgs& A, const V2Args& V, const NodeRec& nd, const Lane& l,
                                           PairRec rec, F step) {
  constexpr int UN = kPairRec;
  const R* ed = reinterpret_cast<const R*>(V.edata) + (SCALAR ? 0 : 3 * l.ki + l.kj);
  const bool mine = !SCALAR || l.ki == l.kj;  // the other entries of a multiple of I are zero
  const uint32_t ring_blocks = static_cast<uint32_t>(V.ring * V.nbp), base_blocks = static_cast<uint32_t>(V.ring_base * V.nbp);
  const PairRec* list = A.pairs + nd.list0 + l.q;
  for (uint32_t r = 0; r < nd.rounds; ++r) {
    R x[UN];
#pragma unroll
    for (int i = 0; i < UN; ++i) {
      x[i] = R(0);
      if (mine) x[i] = ed[(SCALAR ? 1 : 9) * block_slot<WIN>(rec.block[i], ring_blocks, base_blocks)];
    }
    const bool turns = rec.flags >> 31;
    const unsigned ends = l.lane < 27 ? rec.flags : 0u;
    list += 3;
    if (r + 1 < nd.rounds) rec = load_pairs(list);
    step(x, ends, turns);
  }
}

// The diagonal block's entry of lanes 0 .. 8 (DIAG) from the lanes' sums of entry (ki, kj) of
// the blocks from the own pair on and of entry (kj, ki) of those before it.
__device__ __forceinline__ double diagonal(const Lane& l, double own, double before) {
  const double t = own + __shfl_sync(kAll, before, min(9 * (l.lane / 9) + 3 * l.kj + l.ki, 31));
  const double t1 = __shfl_sync(kAll, t, (l.lane + 9) & 31), t2 = __shfl_sync(kAll, t, (l.lane + 18) & 31);
  return -((t + t1) + t2);
}

// Row r of the rhs on lane 3 r: the load (or what is there, ADD) and v.
template <bool ADD>
__device__ __forceinline__ void write_rhs(const ElemArgs& A, const V2Args& V, const NodeRec& nd, int64_t a, int lane,
                                          double v) {
  const int ma = nd.len_mask >> 28, r = lane / 3;
  if ((lane == 0 || lane == 3 || lane == 6) && ((ma >> r) & 1)) {
    const int64_t eq = nd.eq0 + __popc(ma & ((1 << r) - 1));
    const double prev = ADD ? A.rhs[eq] : (V.f_ext ? V.f_ext[3 * a + r] : 0.0);
    A.rhs[eq] = prev + v;
  }
}

// A node with a neighbour that is not fully free. The node's record is read again where it is
// needed (fresh_node) instead of kept through the walk, which has 64 registers a thread with
// FP32 blocks (kept, the walk of the full rows spilled too: C3D8 64^3 293 -> 327 us).
template <typename R, int KIND, bool WIN, bool ADD>
__device__ __forceinline__ void gather_compressed(const ElemArgs& A, const V2Args& V, int64_t a) {
  constexpr bool DIAG = KIND == GATHER_DIAG;
  constexpr int UN = kPairRec;
  // Where the lane's entry of a pair goes: entry (ki, kj) of the block from the own pair on,
  // entry (kj, ki) before it; the row's start and the pair's column and free components
  // (BndRec): the lane's column is free, or its prescribed value is not zero, or nothing is to
  // do, as on every lane whose row is not free.
  double* row = nullptr;
  uint32_t free = 0, moves = 0, below = 0;
  auto side = [&](const NodeRec& nd, const Lane& l, bool early) {
    const int i = early ? l.kj : l.ki, j = early ? l.ki : l.kj, ma = nd.len_mask >> 28;
    const bool on = (ma >> i) & 1;
    free = on ? 1u << (28 + j) : 0u;
    moves = on ? 0x80000000u : 0u;
    below = ((1u << j) - 1) << 28;
    row = A.vals + nd.base + static_cast<int64_t>(__popc(ma & ((1 << i) - 1))) * (nd.len_mask & 0xfffffff);
  };
  // what prescribed columns move to the rhs: of row ki, and (rt) of row kj before the own pair
  double rd = 0.0, rt = 0.0;
  auto put = [&](BndRec b, double v) {
    if (b.at & free) {
      write_entry<ADD>(row + (b.at & 0xfffffff) + __popc(b.at & below), v);
    } else if (b.at & moves) {
      // (a value of zero moves nothing, not even from an infinite entry, src/fem/assembly.cpp:95)
      const double u = A.prescribed[3 * static_cast<int64_t>(b.node) + __popc(below)];
      if (u != 0.0) rd -= v * u;
    }
  };
  double own = 0.0, before = 0.0, v = 0.0;
  {
    const Lane l;
    const NodeRec nd = load_node(A.node + a);
    const int p = l.q == 0 ? 0 : l.q == 1 ? nd.pair1 : nd.pair2;
    side(nd, l, p < nd.diag);
    const BndRec* list = A.bnd + nd.bnd0 + p;
    BndRec b = load_bnd(list);
    each_round<R, KIND == GATHER_SCALAR, WIN>(
        A, V, nd, l, load_pairs(A.pairs + nd.list0 + l.q), [&](const R(&x)[UN], unsigned ends, bool) {
          // the next pair's column is on its way while the pair is summed
#pragma unroll
          for (int i = 0; i < UN; ++i) {
            v += static_cast<double>(x[i]);
            if (ends & (1u << i)) {
              put(b, v);
              if (DIAG) own += v;
              v = 0.0;
              b = load_bnd(++list);
              if (ends & (0x10000u << i)) {
                side(fresh_node(A.node + a), Lane(), false);
                rt = rd;
                rd = 0.0;
                before = own;
                own = 0.0;
              }
            }
          }
        });
  }
  const Lane l;
  const NodeRec nd = fresh_node(A.node + a);
  // a run that ends before the own pair holds earlier pairs only
  if ((l.q == 0 ? nd.pair1 : l.q == 1 ? nd.pair2 : nd.npair) <= nd.diag) {
    rt = rd;
    rd = 0.0;
    before = own;
    own = 0.0;
  }
  if constexpr (DIAG) {
    __syncwarp();  // orders the block below after the loop's write of the same place
    const double d = diagonal(l, own, before);
    if (l.lane < 9) {
      side(nd, l, false);
      put(load_bnd(A.bnd + nd.bnd0 + nd.diag), d);
    }
  }
  if (A.rhs) {
    rd += __shfl_down_sync(kAll, rd, 9) + __shfl_down_sync(kAll, rd, 18);
    rt += __shfl_down_sync(kAll, rt, 9) + __shfl_down_sync(kAll, rt, 18);
    rd += __shfl_down_sync(kAll, rd, 1) + __shfl_down_sync(kAll, rd, 2);  // lane 3 i: row i
    rt += __shfl_down_sync(kAll, rt, 3) + __shfl_down_sync(kAll, rt, 6);  // lane i: row i
    write_rhs<ADD>(A, V, nd, a, l.lane, rd + __shfl_sync(kAll, rt, l.lane / 3));
  }
}

// ADD: onto vals and rhs (V.accumulate).
template <typename R, int KIND, bool WIN, bool ADD>
__device__ __forceinline__ void gather_node(const ElemArgs& A, const V2Args& V, unsigned bid) {
  constexpr bool DIAG = KIND == GATHER_DIAG;
  constexpr int UN = kPairRec;
  const int64_t n_begin = WIN ? V.n_begin : 0, n_end = WIN ? V.n_end : A.n_nodes;
  const int64_t idx = n_begin + static_cast<int64_t>(bid) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (idx >= n_end) return;
  const Lane l;
  const int64_t a = WIN ? static_cast<int64_t>(V.node_order[idx]) : n_end - 1 - idx;
  const NodeRec nd = load_node(A.node + a);
  const int K = nd.npair, L = nd.len_mask & 0xfffffff, ma = nd.len_mask >> 28, self = nd.diag;
  PairRec rec{};
  if (ma && nd.rounds) rec = load_pairs(A.pairs + nd.list0 + l.q);
  // (the records are the plan's own; blocks and outputs are other kernels' too, and are
  // read with plain loads, since the element pass may still be writing when this starts)
  wait_for_kernel_before();
  if (one_wave()) let_next_kernel_start();
  if (!ma) return;
  if (L != 3 * K) {
    gather_compressed<R, KIND, WIN, ADD>(A, V, a);
    return;
  }
  double* const rows = A.vals + nd.base;
  const int p = l.q == 0 ? 0 : l.q == 1 ? nd.pair1 : nd.pair2;
  // before the own pair a lane writes entry (kj, ki), from there on (ki, kj)
  double* o = rows + 3 * p + (p < self ? l.kj * L + l.ki : l.ki * L + l.kj);
  const int64_t turn = static_cast<int64_t>(l.ki - l.kj) * (L - 1);
  // the off-diagonal blocks' sums (DIAG), see diagonal
  double own = 0.0, before = 0.0, v = 0.0;
  each_round<R, KIND == GATHER_SCALAR, WIN>(A, V, nd, l, rec, [&](const R(&x)[UN], unsigned ends, bool turns) {
    if (!turns) {
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        v += static_cast<double>(x[i]);
        end_pair<DIAG, ADD>(ends & (1u << i), o, v, own);
      }
    } else {
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        v += static_cast<double>(x[i]);
        end_pair<DIAG, ADD>(ends & (1u << i), o, v, own);
        if (ends & (0x10000u << i)) {
          o += turn;
          if (DIAG) before = own;
          own = DIAG ? 0.0 : own;
        }
      }
    }
  });
  if constexpr (DIAG) {
    // a run that ends before the own pair holds earlier pairs only
    if ((l.q == 0 ? nd.pair1 : l.q == 1 ? nd.pair2 : K) <= self) {
      before = own;
      own = 0.0;
    }
    __syncwarp();  // orders the block below after the loop's write of the same place
    const double d = diagonal(l, own, before);
    if (l.lane < 9 && K > 0) write_entry<ADD>(rows + l.ki * L + 3 * self + l.kj, d);
  }
  if (A.rhs) write_rhs<ADD>(A, V, nd, a, l.lane, 0.0);  // (full rows have no prescribed column)
}

// One temperature per node: a lane walks one of the three runs of a node, ten nodes to a
// warp, one value per contribution and per pair.
__device__ __forceinline__ void gather_one_dof(const ElemArgs& A, const V2Args& V) {
  constexpr int UN = kPairRec;
  const int lane = threadIdx.x & 31, j = lane / 3, q = lane - 3 * j;
  const double* ed = reinterpret_cast<const double*>(V.edata);
  const int64_t a = 10 * (static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) + j;
  const bool on = lane < 30 && a < A.n_nodes;
  NodeRec nd{};
  if (on) nd = load_node(A.node + a);
  const bool free = (nd.len_mask >> 28) & 1, full = (nd.len_mask & 0xfffffff) == nd.npair;
  wait_for_kernel_before();
  if (one_wave()) let_next_kernel_start();
  double rr = 0.0;
  if (free) {
    int p = q == 0 ? 0 : q == 1 ? nd.pair1 : nd.pair2;
    const PairRec* list = A.pairs + nd.list0 + q;
    double* o = A.vals + nd.base;
    double v = 0.0;
    const BndRec* list_b = A.bnd + nd.bnd0 + p;
    BndRec b{};
    if (!full) b = load_bnd(list_b);
    for (uint32_t r = 0; r < nd.rounds; ++r, list += 3) {
      const PairRec rec = load_pairs(list);
      double x[UN];
#pragma unroll
      for (int i = 0; i < UN; ++i) x[i] = ed[rec.block[i]];
#pragma unroll
      for (int i = 0; i < UN; ++i) {
        v += x[i];
        if (rec.flags & (1u << i)) {
          if (full) {
            o[p] = v;
          } else {
            if ((b.at >> 28) & 1) {
              o[b.at & 0xfffffff] = v;
            } else if (b.at >> 31) {
              const double u = A.prescribed[3 * static_cast<int64_t>(b.node)];
              if (u != 0.0) rr -= v * u;
            }
            b = load_bnd(++list_b);
          }
          v = 0.0;
          ++p;
        }
      }
    }
  }
  const double r1 = __shfl_down_sync(kAll, rr, 1), r2 = __shfl_down_sync(kAll, rr, 2);
  if (A.rhs && free && q == 0) A.rhs[nd.eq0] = (V.f_ext ? V.f_ext[a] : 0.0) + ((rr + r1) + r2);
}

// Internal force of every node (material-point assembly): one thread per component, the
// element forces in element order. In blocks of their own among the gather's: beside a node's
// walk the three dependent loads of this sum cost every node their latency, and a kernel of its
// own costs a launch for every group of a batch (nine small models, FP64: 348 -> 299 us). Spread
// over the grid, they run while other blocks of the SM walk (C3D8 J2 128^3: 98 us as a kernel).
template <bool WIN>
__device__ __forceinline__ void node_forces(const ElemArgs& A, const V2Args& V, unsigned bid) {
  const int64_t first = 3 * (WIN ? V.n_begin : 0), last = 3 * (WIN ? V.n_end : A.n_nodes);
  const int64_t t = first + static_cast<int64_t>(bid) * blockDim.x + threadIdx.x;
  wait_for_kernel_before();
  if (one_wave()) let_next_kernel_start();
  if (t >= last) return;
  const int64_t a = WIN ? static_cast<int64_t>(V.node_order[t / 3]) : t / 3;
  const int d = static_cast<int>(t % 3);
  const int64_t i1 = V.inc_ptr[a + 1];
  double f = 0.0;
#pragma unroll 4
  for (int64_t i = V.inc_ptr[a]; i < i1; ++i) {
    int64_t s = __ldg(V.inc_code + i);
    if constexpr (WIN) {
      s -= V.ring_base * V.npe;
      if (s >= V.ring * V.npe) s -= V.ring * V.npe;
    }
    f += V.fdata[3 * s + d];
  }
  A.f_int[3 * a + d] = f;
}

// Blocks of `threads` for n nodes: the gather's, and those of the forces, one after every
// `force_every` of them (the rest of the gather's at the end).
int64_t gather_grid(V2Args& v, bool forces, int64_t n, int block_nodes, int threads) {
  const int64_t walk = (n + block_nodes - 1) / block_nodes;
  v.force_blocks = forces ? static_cast<uint32_t>((3 * n + threads - 1) / threads) : 0;
  v.force_every = v.force_blocks ? static_cast<uint32_t>(std::max<int64_t>(1, walk / v.force_blocks)) : 0;
  return walk + v.force_blocks;
}

// Whether block bid sums forces; bid becomes its number among its own kind.
__device__ __forceinline__ bool force_block(const V2Args& V, unsigned& bid) {
  const unsigned g = bid / (V.force_every + 1), r = bid - g * (V.force_every + 1);
  const bool forces = g < V.force_blocks && r == V.force_every;
  bid = forces ? g : bid - min(g, V.force_blocks);
  return forces;
}

// What a gather does beside the walk: OVER writes vals and rhs, ADD adds onto them
// (V.accumulate), FORCES writes them and sums the internal forces.
enum GatherMode : int { OVER = 0, ADD = 1, FORCES = 2 };

template <typename R, int KIND, bool WIN, int MODE>
__device__ __forceinline__ void gather_block(const ElemArgs& A, const V2Args& V, unsigned bid) {
  if constexpr (MODE == FORCES) {
    if (force_block(V, bid)) {
      node_forces<WIN>(A, V, bid);
      return;
    }
  }
  if constexpr (KIND == GATHER_ONE_DOF)
    gather_one_dof(A, V);
  else
    gather_node<R, KIND, WIN, MODE == ADD>(A, V, bid);
}

template <typename R, int KIND, bool WIN, int MODE>
__global__ void __launch_bounds__(256, KIND == GATHER_DIAG ? 4 : 3)
    gather_kernel(const __grid_constant__ ElemArgs A, const __grid_constant__ V2Args V) {
  gather_block<R, KIND, WIN, MODE>(A, V, blockIdx.x);
}

template <typename R, int KIND>
cudaError_t launch_t(bool forces, const ElemArgs& a, const V2Args& v, const LaunchCfg& cfg, cudaStream_t s) {
  auto kern = gather_kernel<R, KIND, false, OVER>;
  if constexpr (KIND == GATHER_FULL || KIND == GATHER_DIAG) {
    if (forces)
      kern = v.node_order ? gather_kernel<R, KIND, true, FORCES> : gather_kernel<R, KIND, false, FORCES>;
    else if (v.accumulate)
      kern = v.node_order ? gather_kernel<R, KIND, true, ADD> : gather_kernel<R, KIND, false, ADD>;
    else if (v.node_order)
      kern = gather_kernel<R, KIND, true, OVER>;
  }
  const int warps = cfg.p2_warps > 0 ? std::min(cfg.p2_warps, 8) : kWarps;
  const int64_t count = v.n_end - v.n_begin;
  if (count <= 0) return cudaSuccess;
  ElemArgs A = a;
  V2Args V = v;
  const int64_t grid = gather_grid(V, forces, count, warps * (KIND == GATHER_ONE_DOF ? 10 : 1), warps * 32);
  void* args[] = {&A, &V};
  return launch_kernel(reinterpret_cast<const void*>(kern), grid, warps * 32, 0, s, args);
}

}  // namespace

cudaError_t launch_gather(int kind, bool tangent, const ElemArgs& a, const V2Args& v, const LaunchCfg& cfg,
                          cudaStream_t s) {
  const bool forces = tangent && a.f_int;
  switch (kind) {
    case GATHER_FULL: return launch_t<double, GATHER_FULL>(forces, a, v, cfg, s);
    case GATHER_DIAG: return launch_t<float, GATHER_DIAG>(forces, a, v, cfg, s);
    case GATHER_SCALAR: return launch_t<double, GATHER_SCALAR>(false, a, v, cfg, s);
    case GATHER_ONE_DOF: return launch_t<double, GATHER_ONE_DOF>(false, a, v, cfg, s);
    default: return cudaErrorInvalidValue;
  }
}

// ---- one gather for a batch of element-type groups ------------------------------------
namespace {

struct GatherSlot {
  ElemArgs a;
  V2Args v;
  int64_t blk0;
};
struct GatherPass {
  GatherSlot s[kMaxBatchSlots];
  int32_t n;
};
static_assert(sizeof(GatherPass) <= 4096, "batch pass arguments exceed the kernel parameter space");

// Slot k owns blocks [blk0_k, blk0_{k+1}) of the grid; the arguments are read in place
// from the parameter space.
template <typename R, int KIND, int MODE>
__global__ void __launch_bounds__(256, KIND == GATHER_DIAG ? 4 : 3)
    gather_batch_kernel(const __grid_constant__ GatherPass P) {
  int k = 0;
  while (k + 1 < P.n && static_cast<int64_t>(blockIdx.x) >= P.s[k + 1].blk0) ++k;
  const GatherSlot& S = P.s[k];
  gather_block<R, KIND, false, MODE>(S.a, S.v, blockIdx.x - static_cast<unsigned>(S.blk0));
}

template <typename R, int KIND>
cudaError_t launch_batch_t(bool tangent, const BatchSlotIn* in, int n, cudaStream_t s) {
  const bool forces = tangent && in[0].a.f_int;
  auto kern = forces ? gather_batch_kernel<R, KIND, FORCES> : gather_batch_kernel<R, KIND, OVER>;
  GatherPass P{};
  int warps = 0;  // one block shape for every slot: the smallest that was asked for
  for (int k = 0; k < n; ++k)
    if (in[k].cfg.p2_warps > 0) warps = warps ? std::min(warps, in[k].cfg.p2_warps) : in[k].cfg.p2_warps;
  warps = warps ? std::min(warps, 8) : kWarps;
  int64_t blk = 0;
  for (int k = 0; k < n; ++k) {
    P.s[k].a = in[k].a;
    P.s[k].v = in[k].v;
    P.s[k].blk0 = blk;
    blk += gather_grid(P.s[k].v, forces, in[k].v.n_end - in[k].v.n_begin, warps, warps * 32);
  }
  if (blk <= 0) return cudaSuccess;
  P.n = n;
  void* args[] = {&P};
  return launch_kernel(reinterpret_cast<const void*>(kern), blk, warps * 32, 0, s, args);
}

}  // namespace

cudaError_t launch_gather_batch(int kind, bool tangent, const BatchSlotIn* in, int n, cudaStream_t s) {
  if (kind == GATHER_DIAG) return launch_batch_t<float, GATHER_DIAG>(tangent, in, n, s);
  if (kind == GATHER_FULL) return launch_batch_t<double, GATHER_FULL>(tangent, in, n, s);
  return cudaErrorInvalidValue;
}

}  // namespace cxg
