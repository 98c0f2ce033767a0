// Internal declarations shared by the kernels (cxg_kernels.cu, cxg_pattern.cu) and
// the C-ABI layer (cxg_api.cu).
#pragma once

#include <cuda_runtime.h>

#include <functional>

#include <cstdint>

#include "cxg_elements.hpp"

namespace cxg {

constexpr int kStateDoubles = 13;  // plastic strain[6], eq. plastic strain, back stress[6]
constexpr int kMaxTable = 64;      // *PLASTIC table points per material

// Device record of one material (J2PlasticMaterial, src/fem/plasticity.cpp:42-65, with
// the kinematic-hardening table adjustment of its constructor already applied).
struct J2Mat {
  int32_t plastic;  // 0: linear elastic
  int32_t n;        // table length
  double h_kin;
  double ep[kMaxTable];
  double sy[kMaxTable];
};

// In-kernel error reporting: first error code and the smallest offending element.
struct DevStatus {
  int32_t code;
  int32_t pad;
  unsigned long long bad_elem;
};

enum KernelMode : int { MODE_LINEAR = 0, MODE_TANGENT = 1 };

// Constant tables (defined in cxg_kernels.cu, filled by ensure_tables): natural
// derivatives dN[k][d][q] (Gauss point fastest) and weights of every family.
constexpr int dn_size(int t) { return nodes_of(t) * 3 * gauss_of(t); }
constexpr int dn_offset(int t) {
  int off = 0;
  for (int u = kFirstType; u < t; ++u) off += dn_size(u);
  return off;
}
constexpr int kDnTotal = dn_offset(C3D15) + dn_size(C3D15);
extern __constant__ double c_dN[kDnTotal];
// Shape-function values N[k][q] (Gauss point fastest) of every family.
constexpr int nn_size(int t) { return nodes_of(t) * gauss_of(t); }
constexpr int nn_offset(int t) {
  int off = 0;
  for (int u = kFirstType; u < t; ++u) off += nn_size(u);
  return off;
}
constexpr int kNTotal = nn_offset(C3D15) + nn_size(C3D15);
extern __constant__ double c_N[kNTotal];
extern __constant__ double c_w[8][kMaxGauss];

// What the row gather needs of one node, fetched with three 16-byte loads. Its pairs
// (neighbours, itself included, ascending) are cut into three runs of near-equal numbers
// of contributions, starting at pairs 0, pair1 and pair2; run q's contributions are the
// entries of the records list0 + 3 r + q, r < rounds (PairRec). Blocks of pairs with a
// smaller node are read as stored and written transposed (see blk_index).
struct __align__(16) NodeRec {
  int64_t base;      // CSR offset of the node's first free row
  uint32_t len_mask; // length of each of the node's rows | free components << 28
  int32_t eq0;       // first free equation (or -1)
  uint32_t list0;
  uint32_t rounds;
  uint32_t bnd0;     // first of the node's BndRecs
  uint16_t npair;
  uint16_t diag;     // the node's own position among its pairs
  uint16_t pair1, pair2;
  uint32_t pad[3];   // (the pattern builder's cuts while it works)
};
static_assert(sizeof(NodeRec) == 48, "NodeRec is three 16-byte loads");

// Up to 11 contributions of element blocks to consecutive pairs of a node, in pair order
// and element order within a pair: block[i] is e * blocks_padded(n) + blk_index(n, min,
// max) of the pair's local nodes; bit i of flags: the last contribution of its pair; bit
// 16 + i: and the next pair is the node with itself (bit 31: some run of this round has
// that). Unused entries, after the last flagged one, repeat a block of the node.
constexpr int kPairRec = 11;
struct __align__(16) PairRec {
  uint32_t flags;
  uint32_t block[kPairRec];
};
static_assert(sizeof(PairRec) == 48, "PairRec is three 16-byte loads");

// A pair of a node whose rows are compressed (some neighbour is not fully free).
struct __align__(8) BndRec {
  uint32_t at;   // first column | free components << 28 | (some prescribed value is not zero) << 31
  int32_t node;  // the neighbour
};

// 3x3 blocks of an element in the element buffer: one per local node pair (a, b), a <= b,
// 9 consecutive values at 9 * blk_index. The stored block is that of the two nodes in
// ascending mesh order (K_ba where node b precedes node a), so all elements that share a
// pair store it the same way round; a node with itself, where an element names a node twice,
// as the symmetric part (zeros in FP32), since (a, b) and (b, a) are the same pair then. An element's block count is padded so that every
// element starts 16-byte aligned in both precisions, which bulk copies need (8-byte
// aligned in FP32 for the families of 4 and 6 nodes, which copy with plain stores).
__host__ __device__ constexpr int blk_index(int n, int a, int b) { return a * n - a * (a - 1) / 2 + (b - a); }
__host__ __device__ constexpr int blocks_padded(int n) {
  const int nb = n * (n + 1) / 2;
  return n < 8 ? (nb + 1) / 2 * 2 : (nb + 3) / 4 * 4;
}

// Everything an element-integration launch reads or writes. Pointers are device
// pointers; optional ones may be null.
struct ElemArgs {
  int64_t n_elems;
  int64_t n_nodes;
  // geometry: either a mesh (coords + conn) or per-element coordinates (dense mode)
  const double* coords;     // [3N]
  const int32_t* conn;      // [E*n]
  const double* elem_coords;  // [E*n*3] (dense element-level mode)
  const double* young;      // [E]
  const double* poisson;    // [E]
  const int32_t* elem_mat;  // [E] or null -> material 0
  const J2Mat* mats;        // [n_mats]
  // DOF map / CSR addressing (row gather), see PatternOut
  const NodeRec* node;        // [N]
  const double* prescribed;   // [3N]
  const PairRec* pairs;
  const BndRec* bnd;
  // state (tangent mode), SoA [13][G]
  const double* state_c;
  double* state_t;
  int64_t n_gauss;
  // history components the element pass reads and writes: 13, or 7 (plastic strain and
  // equivalent plastic strain) when the back stress is zero in both buffers and no
  // material moves it (every kinematic modulus is 0); components 7..12 are then zero
  // and left untouched
  int state_comps;
  // thermal strain (null th_temp: none): applied temperature per node, whether it is
  // applied (null: every node), expansion coefficient and reference temperature per
  // element (alpha 0: no expansion)
  const double* th_temp;      // [N]
  const uint8_t* th_applied;  // [N]
  const double* th_alpha;     // [E]
  const double* th_tref;      // [E]
  // displacement (tangent mode)
  const double* u;           // [3N] (mesh) or [E*n*3] (dense)
  // outputs
  double* vals;   // [nnz]
  double* rhs;    // [n_free]
  double* f_int;  // [3N]
  double* Ke;     // dense [E*(3n)^2]
  double* fe;     // dense [E*3n]
  DevStatus* status;
};

// Extra arguments of the two-pass assembly (cxg_v2.cu).
struct V2Args {
  void* edata;              // per-element upper 3x3 blocks, FP32 (mixed) or FP64
  double* fdata;            // per-element internal force [E*3n] (material-point mode)
  const int64_t* inc_ptr;   // node -> incident elements
  const int32_t* inc_code;
  const double* f_ext;      // [3N] load vector for the rhs, or null
  int npe, nbp;             // nodes and (padded) blocks per element
  int named_twice;          // some element names a node at two places
  int accumulate;           // add into vals / rhs instead of overwriting
  // The window of one element-pass + row-gather pair: the element pass integrates
  // elements [e_begin, e_end), the row gather the nodes node_order[n_begin..n_end)
  // (node_order null: nodes n_begin..n_end in mesh order). The element buffers hold
  // `ring` elements; element e lives in slot e mod ring.
  int64_t e_begin, e_end, ring, ring_base;
  const int32_t* node_order;
  int64_t n_begin, n_end;
  // Window schedule read by the launcher (host arrays): n_win windows with element
  // offsets win_e[0..n_win] and node-list offsets win_n[0..n_win]; n_win <= 1 runs the
  // whole mesh as one window.
  int32_t n_win;
  const int64_t* win_e;
  const int64_t* win_n;
  uint32_t force_blocks, force_every;  // set by the gather's launcher
};
// Launch shape of the two passes. tile: node-pair tile of the mixed-precision linear element
// pass (0 = 2x4, 1 = 2x2, 2 = 4x4; the others have one shape); p1_blocks_per_sm: persistent
// grid per SM of the element pass (0 = as many as are resident); p2_warps: warps per
// row-gather block, at most 8 (0 = 4); passes: bit 0 the element pass, bit 1 the row gather.
struct LaunchCfg {
  int tile = 0;
  int p1_blocks_per_sm = 0;
  int p2_warps = 0;
  int passes = 3;
  // mixed-precision material-point pass: the J2 return in FP32 (j2_point_mixed) instead
  // of FP64
  int j2_fp32 = 0;
};
// One element pass and one row gather for a whole batch of element-type groups: slot k
// is group k's arguments (one window, mesh node order), its element type and launch
// shape; the weights share the element pass's persistent grid between the slots.
constexpr int kMaxBatchSlots = 8;
struct BatchSlotIn {
  ElemArgs a;
  V2Args v;
  int32_t type = 0;
  LaunchCfg cfg;
  double p1_weight = 1.0;
};
// Blocks of a persistent grid of `total` blocks shared out in proportion to the slots'
// weights, at least one and at most `need` per slot.
void share_blocks(const double* weight, const int64_t* need, int n, int64_t total, int64_t* grid);
// Row gather (cxg_gather.cu). GATHER_FULL: FP64 blocks, every entry summed; GATHER_DIAG:
// FP32 blocks, the diagonal block from the row's other entries; GATHER_SCALAR: one FP64
// value per pair, standing for its multiple of I; GATHER_ONE_DOF: the same on a
// temperature plan, whose nodes have component 0 only (f_ext is then one value per node).
enum GatherKind : int { GATHER_FULL = 0, GATHER_DIAG = 1, GATHER_SCALAR = 2, GATHER_ONE_DOF = 3 };
cudaError_t launch_gather(int kind, bool tangent, const ElemArgs& a, const V2Args& v, const LaunchCfg& cfg,
                          cudaStream_t s);
cudaError_t launch_gather_batch(int kind, bool tangent, const BatchSlotIn* slots, int n_slots, cudaStream_t s);
cudaError_t launch_v2_batch(int mode, int precision, const BatchSlotIn* slots, int n_slots, int passes,
                            cudaStream_t s);
// Tiles the batch kernels take (2x2; 2x4 in the mixed-precision linear pass).
bool batch_tile_ok(int mode, int precision, int tile);
size_t v2_edata_bytes(int elem_type, int64_t n_elems, int precision);
// Bytes of element buffer per element (blocks, plus the internal force in tangent mode).
size_t v2_bytes_per_element(int elem_type, int precision, bool tangent);
// Element pass of the scalar-block operators (every 3x3 block is a scalar times I):
// kind 1 consistent mass rho N_a N_b, 2 lumped mass (row sums on the diagonal), 3
// geometric stiffness g_a . sigma . g_b, 4 conduction k g_a . g_b. Writes one FP64 value
// per element pair, at e * blocks_padded(n) + blk_index. density[E] is rho (kinds 1, 2) or k (kind 4), gp_stress[6 G]
// (kind 3).
cudaError_t launch_scalar_pass(int elem_type, int kind, const ElemArgs& a, const V2Args& v, const double* density,
                               const double* gp_stress, cudaStream_t s);
cudaError_t launch_v2(int elem_type, int mode, int precision, const ElemArgs& a, const V2Args& v, cudaStream_t s,
                      const LaunchCfg& cfg = LaunchCfg{});

// The reference's own pattern (cxg_refpattern.cu): launch_refmask writes, per element and
// in the FP64 element-buffer layout, 1.0 where the reference's K_e (its operation order)
// is nonzero and 0.0 where it is exactly zero; compact_pattern keeps the CSR entries whose
// gathered count is positive (row_ptr_c, col_idx_c, and src = their topological index);
// gather_values copies a topological assembly onto the kept entries.
cudaError_t launch_refmask(int elem_type, const ElemArgs& a, double* out, cudaStream_t s);
cudaError_t compact_pattern(const int64_t* row_ptr, const int32_t* col_idx, int32_t n_rows, int64_t nnz,
                            const double* counts, int64_t** row_ptr_c, int32_t** col_idx_c, int64_t** src,
                            int64_t* nnz_c, cudaStream_t s);
cudaError_t gather_values(const int64_t* src, const double* topo, int64_t nnz_c, double* out, cudaStream_t s);

// Multi-point constraints (cxg_mpc.cu): the reduced CSR of K_ff = T^T K_x T and, per
// reduced entry, the list of (extended entry, weight) pairs it sums (tgt_ptr / src / w);
// per free equation, the list of (extended row, weight) pairs of T^T (rhs_ptr / rhs_src /
// rhs_w).
struct MpcLists {
  int64_t nnz = 0;
  int64_t* row_ptr = nullptr;
  int32_t* col_idx = nullptr;
  int64_t* tgt_ptr = nullptr;
  int64_t* src = nullptr;
  double* w = nullptr;
  int64_t* rhs_ptr = nullptr;
  int64_t* rhs_src = nullptr;
  double* rhs_w = nullptr;
};
// ext_map[x]: free equation of extended equation x, or -1 - s for slave s whose terms are
// [term_ptr[s], term_ptr[s+1]) of term_eq / term_coeff.
cudaError_t build_mpc_reduce(const int64_t* x_row_ptr, const int32_t* x_col, int64_t n_x, int64_t nnz_x,
                             const int32_t* ext_map, const int64_t* term_ptr, const int32_t* term_eq,
                             const double* term_coeff, int32_t n_free, MpcLists* out, cudaStream_t s);
cudaError_t mpc_reduce_values(const MpcLists& m, const double* vals_x, double* vals, cudaStream_t s);
// rhs = T^T (rhs_x - kc), kc = K_x c (null when every constant is zero); tmp_x[n_x] scratch.
cudaError_t mpc_reduce_rhs(const MpcLists& m, const double* rhs_x, const double* kc, int64_t n_x, double* tmp_x,
                           int32_t n_free, double* rhs, cudaStream_t s);

// Launchers (cxg_kernels.cu). `precision` 0 = FP64, 1 = mixed.
cudaError_t launch_element_kernel(int elem_type, int mode, bool dense, int precision,
                                  const ElemArgs& a, cudaStream_t s);
cudaError_t launch_rhs_init(const int32_t* dof_eq, const double* f_ext, int64_t ndof,
                            double* rhs, cudaStream_t s);
cudaError_t launch_state_transpose(const double* src, double* dst, int64_t G, bool to_soa,
                                   cudaStream_t s);
// Field recovery (cxg_recover.cu): a.u is the full displacement. gp_stress[6G] may be
// null; emean[12E] and felem[3nE] are scratch for the node pass (both null: Gauss-point
// stress only); strain/stress[6N], reaction[3N] outputs.
cudaError_t launch_recover(int elem_type, const ElemArgs& a, const int64_t* inc_ptr, const int32_t* inc_code,
                           double* gp_stress, double* emean, double* felem, const double* f_ext, double* strain,
                           double* stress, double* reaction, bool thermal_load, cudaStream_t s);
// *FILM faces of a temperature plan (cxg_film.cu), device arrays built once per film set:
// films grouped by element (felem[g] owns flist[fptr[g] .. fptr[g+1]), in film order),
// and per face node the (film, face-local index) entries film * 8 + i it receives
// (fnode[g] owns fnlist[fnptr[g] .. fnptr[g+1]), in film order); load[8 * n_films] holds
// h T_sink int N_i dA between the two passes.
struct FilmArgs {
  int64_t n_films = 0, n_felem = 0, n_fnode = 0;
  const int64_t* felem = nullptr;
  const int32_t* fptr = nullptr;
  const int32_t* flist = nullptr;
  const int32_t* face = nullptr;
  const double* h = nullptr;
  const double* sink = nullptr;
  const int64_t* fnode = nullptr;
  const int32_t* fnptr = nullptr;
  const int32_t* fnlist = nullptr;
  double* load = nullptr;
};
cudaError_t launch_films(int elem_type, const ElemArgs& a, const FilmArgs& f, double* edata, double* f_ext,
                         cudaStream_t s);
// Compliance adjoint (cxg_recover.cu); felem[3nE]: scratch for dc_dX (null without it).
cudaError_t launch_adjoint(int elem_type, const ElemArgs& a, const int64_t* inc_ptr, const int32_t* inc_code,
                           double* felem, double* dc_dE, double* dc_dX, cudaStream_t s);
// y = A x on CSR; node (null: any CSR matrix) for a matrix on a plan's own pattern.
cudaError_t launch_spmv(int32_t nrows, const int64_t* rp, const int32_t* ci, const double* v, const double* x,
                        double* y, cudaStream_t s, const NodeRec* node = nullptr, int64_t n_nodes = 0);
// Jacobi-preconditioned CG on CSR; work holds 5*n + 2056 doubles; node as above.
cudaError_t cg_solve(int32_t n, const int64_t* rp, const int32_t* ci, const double* v, const double* b, double* x,
                     double rtol, int max_iter, double* work, int* iters_out, double* rel_out, cudaStream_t s,
                     const NodeRec* node = nullptr, int64_t n_nodes = 0);
// CG with z = M^-1 r given by `precond` (launched on the loop's stream);
// work holds 5*n + 2056 doubles, the fifth n-vector unused by the loop.
using Preconditioner = std::function<cudaError_t(const double* r, double* z)>;
cudaError_t pcg_solve(int32_t n, const int64_t* rp, const int32_t* ci, const double* v, const double* b, double* x,
                      double rtol, int max_iter, double* work, int* iters_out, double* rel_out, cudaStream_t s,
                      const Preconditioner& precond);
// Element tables (constant memory) are uploaded once per device.
cudaError_t ensure_tables();

// Resident blocks per SM of a kernel and the SM count of the current device, asked of the
// runtime once per thread, kernel and shape (cxg_launch.cu); sets the kernel's shared memory.
cudaError_t kernel_shape(const void* kern, int threads, size_t smem, int* per_sm, int* sms);
// Lets kern be launched with that much dynamic shared memory on the current device.
cudaError_t allow_smem(const void* kern, size_t smem);
// Launches kern. Unless s is being captured, it may start while the kernel before it on s
// drains (programmatic stream serialisation): kernels launched this way wait_for_kernel_before()
// ahead of anything an earlier kernel may have written, or may still read.
cudaError_t launch_kernel(const void* kern, int64_t grid, int threads, size_t smem, cudaStream_t s, void** args);
#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_kernel_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// Device memory of plans (cxg_pool.cu): from a pool of the current device that keeps up to
// 512 MB of what is freed. device_free expects that no work on the block is pending.
// device_free_all waits for all work of `device` (as cudaFree would, once), whichever device
// is current, frees its blocks and returns what is above the 512 MB to the device.
// device_malloc and device_malloc_async are cudaMalloc and cudaMallocAsync. Each tries again with
// the pool emptied where the device has no memory left.
cudaError_t device_alloc(void** out, size_t bytes);
cudaError_t device_malloc(void** out, size_t bytes);
cudaError_t device_malloc_async(void** out, size_t bytes, cudaStream_t s);
void device_free(void* ptr);
template <typename T>
cudaError_t device_malloc(T** out, size_t bytes) {
  return device_malloc(reinterpret_cast<void**>(out), bytes);
}
template <typename T>
cudaError_t device_malloc_async(T** out, size_t bytes, cudaStream_t s) {
  return device_malloc_async(reinterpret_cast<void**>(out), bytes, s);
}
void device_free_all(int device, void* const* blocks, int n);
// Whether a kernel on `device` can take the caller's doubles at ptr where they are: managed, or
// in that device's own memory, and aligned. Anything else cudaMemcpy takes is copied first.
bool kernel_reads(int device, const void* ptr);

// Pattern construction (cxg_pattern.cu).
struct PatternOut {
  void* mem[2] = {nullptr, nullptr};  // the device blocks that hold all of these
  int64_t nnz = 0;
  bool named_twice = false;     // some element names a node at two places
  int64_t* row_ptr = nullptr;   // [n_free+1]
  int32_t* col_idx = nullptr;   // [nnz]
  NodeRec* node = nullptr;      // [N]
  uint8_t* node_mask = nullptr; // [N]
  PairRec* pairs = nullptr;     // contributions of the element blocks, see NodeRec
  BndRec* bnd = nullptr;        // of every pair of the nodes with a neighbour that is not fully free
  // node -> incident elements, ascending element order: codes e*n + local node index
  int64_t* inc_ptr = nullptr;   // [N+1]
  int32_t* inc_code = nullptr;  // [E*n]
  int64_t device_bytes = 0;
};
// Returns a cxg_status code; on error *msg is set.
int build_pattern(int elem_type, int64_t n_nodes, int64_t n_elems, const int32_t* d_conn,
                  const int32_t* d_dof_eq, const double* d_prescribed, int32_t n_free, PatternOut* out, const char** msg,
                  cudaStream_t s);

}  // namespace cxg
