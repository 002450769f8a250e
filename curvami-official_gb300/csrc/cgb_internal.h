// cgb_internal.h — host-side internals shared by the CUDA translation units of the
// GB300 Gauss-point library (context, shape sets, assembler, device buffers).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/curvami_gb300.h"

namespace cgb {

// A failure inside the library: carries the C-ABI status code and the message that
// cgb_last_error() returns (the reference's exception text where one exists).
struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

inline void cuda_check(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw Error(CGB_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
#define CGB_CUDA(call) ::cgb::cuda_check((call), #call)

// The device has no room for an allocation, and reclaim() found none.
struct OutOfMemory : Error {
  explicit OutOfMemory(size_t bytes)
      : Error(CGB_ERR_CUDA, "device allocation of " + std::to_string(bytes) + " bytes failed: out of memory") {}
};

// Gives back what an allocation that found no room may take: the idle blocks of every context's pool, and the
// scratch of the calling thread's context unless a build is using it.
void reclaim();

// Device memory of one context's shape sets. A set is several arrays of up to a gigabyte, and mapping
// and unmapping that with cudaMalloc and cudaFree cost 1.2 ms of a 6 ms build and its destruction.
// Freed blocks stay with the pool, up to kKeep bytes, for the next set. Blocks are taken and given
// back on a stream of the pool's own: a taker waits for it (nothing else runs there), and a set's blocks
// are given back only after wait(). The context destroys the pool.
struct ShapePool {
  static constexpr uint64_t kKeep = 4ULL << 30;
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;
  mutable char* token = nullptr;   // what wait() frees
  // Every context's pool (trim_all: their idle blocks go back to the device).
  inline static std::mutex all_mutex;
  inline static std::vector<cudaMemPool_t> all;
  static void trim_all() {
    std::lock_guard<std::mutex> lock(all_mutex);
    for (cudaMemPool_t p : all) cudaMemPoolTrimTo(p, 0);
  }
  void create(int device) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    CGB_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = kKeep;
    CGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    CGB_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    CGB_CUDA(cudaMalloc(&token, 1));
    std::lock_guard<std::mutex> lock(all_mutex);
    all.push_back(pool);
  }
  // Waits for the device's work as cudaFree of a set's arrays would. Not cudaDeviceSynchronize: that
  // is an error while another thread captures a stream, and breaks the capture. 3 us when idle.
  void wait() const {
    if (!token && cudaMalloc(&token, 1) != cudaSuccess) {
      cudaGetLastError();
      cudaDeviceSynchronize();
      return;
    }
    cudaFree(token);
    if (cudaMalloc(&token, 1) != cudaSuccess) {
      cudaGetLastError();
      token = nullptr;
    }
  }
  void destroy() {
    if (token) cudaFree(token);
    token = nullptr;
    {
      std::lock_guard<std::mutex> lock(all_mutex);
      all.erase(std::remove(all.begin(), all.end(), pool), all.end());
    }
    if (stream) { cudaStreamSynchronize(stream); cudaStreamDestroy(stream); }
    if (pool) cudaMemPoolDestroy(pool);
    stream = nullptr;
    pool = nullptr;
  }
};

// Owning device buffer, freed on destruction or reset: cudaMalloc'd, or of a pool.
template <class T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  const ShapePool* from = nullptr;
  DevBuf() = default;
  explicit DevBuf(size_t count) { alloc(count); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n), from(o.from) { o.p = nullptr; o.n = 0; }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) { reset(); p = o.p; n = o.n; from = o.from; o.p = nullptr; o.n = 0; }
    return *this;
  }
  ~DevBuf() { reset(); }
  void alloc(size_t count) {
    reset();
    if (count == 0) count = 1;  // keep a valid pointer for empty sets
    cudaError_t e = take(count * sizeof(T));
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      reclaim();
      e = take(count * sizeof(T));
    }
    if (e != cudaSuccess) p = nullptr;
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      throw OutOfMemory(count * sizeof(T));
    }
    CGB_CUDA(e);
    n = count;
  }
  cudaError_t take(size_t bytes) {
    if (!from) return cudaMalloc(&p, bytes);
    const cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, from->pool, from->stream);
    return e == cudaSuccess ? cudaStreamSynchronize(from->stream) : e;
  }
  void ensure(size_t count) { if (n < count || !p) alloc(count); }
  void reset() {
    if (p) {
      if (from) cudaFreeAsync(p, from->stream);
      else cudaFree(p);
    }
    p = nullptr;
    n = 0;
  }
  size_t bytes() const { return n * sizeof(T); }
};

template <class T>
void upload(DevBuf<T>& d, const T* h, size_t count, cudaStream_t s) {
  d.alloc(count);
  if (count) CGB_CUDA(cudaMemcpyAsync(d.p, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
}

struct Crease {
  std::vector<double> xy;
  int extend_start = 0, extend_end = 0, is_closed = 0;
};

// Kinematics::NaturalCurvature (plate/Kinematics.h:21-45) as the kernels take it: the band's
// kappa_bar_XX(X) = amp * exp(-((X - x0) / width)^2), amp = sign * theta0 / (sqrt(pi) width).
struct NatCurv {
  int active = 0;
  double x0 = 0.0, width = 1.0, amp = 0.0;
};

// One cell of the FP32 tangent: its first entry and item, how many it has, and its node union's
// size (32767: direct).
struct TileCell {
  int64_t q0, i0;
  int32_t n_ent, n_items, U, pad;
};

// Scratch of the shape stage, kept by the context between builds and rebuilds (a set holds only its
// results): each such call runs on the context's stream and waits for it before it returns, and a
// context is used by one thread at a time. Grows to the largest call's need: moments and polynomials of
// a chunk of points (1.1 GB for the quadratic basis, 1.9 GB for the cubic), and arrays over all points, of
// which those above kKeep bytes are not kept. Given back with the context, by cgb_trim, and when an
// allocation of the context finds no room (reclaim). Not the pool's blocks: with them 1,000,000 mixed
// points took 6.92 ms, not 6.84, and the first build 9.3 ms, not 8.5.
struct ShapeScratch {
  static constexpr size_t kKeep = 256u << 20;
  bool busy = false;   // a build is using it
  void drop_large() {
    if (gind.bytes() > kKeep) gind.reset();
    if (gp_mask.bytes() > kKeep) gp_mask.reset();
    if (point_rec.bytes() > kKeep) point_rec.reset();
  }
  // Node cell grid and neighbour search.
  DevBuf<int64_t> cell_start, totals, bsum;
  DevBuf<unsigned long long> cell_cursor;
  DevBuf<int32_t> cell_count, node_key, node_list, cell_nodes, gp_count, bmax;
  DevBuf<float2> cell32;
  DevBuf<float> r2c32;
  DevBuf<uint32_t> gp_mask;
  // Creases and RKPM.
  DevBuf<double> cxy;        // crease vertices, all creases
  DevBuf<float2> cxyf;       // the same relative to each crease's first, in float
  DevBuf<int8_t> side;       // n_creases * n_nodes
  DevBuf<double> gind;       // n_creases * 6 * n_gp
  DevBuf<int8_t> bad, tip;   // n_gp
  DevBuf<int32_t> order;     // n_gp, the moment kernels' order
  DevBuf<int> guard;         // 4: flagged points
  DevBuf<double> fac;        // n_nodes, FP64 with per-node radius
  DevBuf<double> mom, coef;  // moment sums and polynomials of a chunk of points
  DevBuf<float4> node_pair;  // 2 * n_nodes, mixed precision
  DevBuf<float> point_rec;   // point records, mixed precision
};

}  // namespace cgb

// Opaque handles of the C ABI.
struct cgb_context {
  // Shape sets and assemblers keep their context alive: cgb_destroy only drops the
  // caller's reference, the context is freed when the last handle that uses it is.
  int refs = 1;
  bool closed = false;
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string last_error;
  // Nodes (Meshless::nodes X_ref), interleaved x y.
  int n_nodes = 0;
  std::vector<double> h_node_xy;
  cgb::DevBuf<double> node_xy;
  uint64_t node_gen = 0;  // bumped whenever cgb_set_nodes changes the coordinates
  cgb::NatCurv natcurv;   // natural curvature of every constitutive evaluation (inactive by default)
  // Device-side error word written by kernels (bounds checks, capacity).
  cgb::DevBuf<int> dev_err;
  int* h_err = nullptr;  // pinned mirror
  static inline thread_local cgb_context* active = nullptr;   // of the calling thread's entry (cgb::Active)
  double node_min[2] = {0.0, 0.0}, node_max[2] = {0.0, 0.0};  // bounds of the nodes
  cgb::ShapeScratch scratch;
  cgb::ShapePool shape_pool;
  cgb::DevBuf<double> ws_x, ws_out;  // device copies of cgb_point_state's x and rows
  // Tracing: event pairs per phase, summed when read.
  bool profile = false;
  struct Mark { int phase; cudaEvent_t start, stop; int launches; cudaStream_t stream; };
  std::vector<Mark> marks;
  std::vector<cudaEvent_t> event_pool;
  double prof_ms[CGB_N_PHASES] = {0};
  int64_t prof_launches[CGB_N_PHASES] = {0};
};

namespace cgb {
// The context of the C entry that the thread is in.
struct Active {
  cgb_context* before = cgb_context::active;
  explicit Active(cgb_context* ctx) { cgb_context::active = ctx; }
  ~Active() { cgb_context::active = before; }
};
}  // namespace cgb

struct cgb_shape {
  explicit cgb_shape(const cgb::ShapePool* from_pool) : pool(from_pool) {
    gp_xy.from = s.from = psi.from = dpsi.from = ddpsi.from = rho_node.from = pool;
    nbr_ptr.from = pool;
    nbr_idx.from = pool;
  }
  // Also of a set whose making failed half way: kernels may still write its arrays.
  ~cgb_shape() {
    if (nbr_ptr.p || gp_xy.p || rho_node.p) pool->wait();
  }
  const cgb::ShapePool* pool;
  cgb_context* ctx = nullptr;
  int n_gp = 0;
  int64_t nnz = 0;
  int max_n = 0;  // largest neighbour count of the set
  cgb::DevBuf<double> gp_xy;      // 2 per point
  bool has_xy = false;            // gp_xy holds the points' reference coordinates
  cgb::DevBuf<int64_t> nbr_ptr;   // n_gp + 1
  cgb::DevBuf<int32_t> nbr_idx;   // nnz
  cgb::DevBuf<double> s;          // nnz (normalised distance), may be empty
  cgb::DevBuf<double> psi;        // nnz
  cgb::DevBuf<double> dpsi;       // 2 * nnz (x, y)
  cgb::DevBuf<double> ddpsi;      // 3 * nnz (xx, yy, xy)
  // What a rebuild with other creases needs (sets made by cgb_shape_build only): the
  // shape parameters and the node coordinates the neighbour lists were found on.
  bool rebuildable = false;
  double rho = 0.0;
  int order = 0, kernel = 0;
  int precision = 0;              // CGB_SHAPE_FP64 / CGB_SHAPE_MIXED
  bool has_rho_node = false;
  cgb::DevBuf<double> rho_node;   // n_nodes (per-node radius) when has_rho_node
  uint64_t node_gen = 0;
  uint64_t version = 0;           // bumped by every rebuild (derived copies go stale)
};

// Per-fold data kept by the assembler (plate/PlateData.h: Fold; Constraints.h:341).
struct cgb_fold_dev {
  int n_gp = 0;
  double Kt = 0.0, theta0 = 0.0;
  const cgb_shape* left = nullptr;
  const cgb_shape* right = nullptr;
  cgb::DevBuf<double> weight, tangent, theta0_gp;
  cgb::DevBuf<int8_t> active;
  bool has_theta0_gp = false, has_active = false;
  // Merged node list of left U right per crease point (sorted unique nodes),
  // and for every left/right entry its position in that list.
  cgb::DevBuf<int64_t> u_ptr;       // n_gp + 1
  cgb::DevBuf<int32_t> u_node;      // merged nodes
  cgb::DevBuf<int32_t> l_pos, r_pos;
  cgb::DevBuf<int64_t> pair_ptr;    // n_gp + 1, pairs P <= Q over the merged list
  cgb::DevBuf<int32_t> pair_slot;   // block slot of each pair in the union pattern
  cgb::DevBuf<int32_t> pair_hslot;  // the same among the blocks that any hinge pair touches
  int max_u = 0;
  int64_t n_u = 0;      // merged-node entries over all crease points (u_ptr[n_gp])
  int64_t n_pairs = 0;
};

// Most Gauss-point chunks one assembly is split into (residual / tangent overlap).
constexpr int kMaxChunks = 16;

struct cgb_assembler {
  cgb_context* ctx = nullptr;
  const cgb_shape* faces = nullptr;
  int n_nodes = 0;
  int64_t n_blocks = 0;  // 3x3 blocks of the union pattern; nnz = 9 * n_blocks
  cgb::DevBuf<double> weight;       // face Gauss-point weights
  // Union pattern (face blocks U hinge blocks), block-column CSC:
  cgb::DevBuf<int64_t> col_ptr;     // n_nodes + 1 (block offsets)
  cgb::DevBuf<int32_t> col_nodes;   // n_blocks (block rows, ascending per column)
  cgb::DevBuf<int32_t> outer;       // 3 n_nodes + 1 (scalar CSC, the reference's K layout)
  // Face Gauss point -> block slot of each local pair (i <= j) in loop order.
  cgb::DevBuf<int64_t> map_ptr;     // n_gp + 1
  cgb::DevBuf<int32_t> map_slot;    // total pairs
  int64_t n_pairs = 0;
  std::vector<cgb_fold_dev> folds;
  double A[9] = {0}, B[9] = {0}, D[9] = {0};
  bool have_material = false;
  // Accumulators.
  cgb::DevBuf<double> kacc64;       // 9 * n_blocks
  cgb::DevBuf<float> kacc32;        // cells' tangent: 12 * n_blocks (padded for 16-byte vector atomics), then the
                                    // hinge's blocks in FP64 (9 * n_hinge_blocks)
  // The blocks that hinge pairs touch, ascending by slot: the first of each column, and each one's
  // block row within its column.
  int64_t n_hinge_blocks = 0;
  cgb::DevBuf<int64_t> hinge_col;   // n_nodes + 1
  cgb::DevBuf<int32_t> hinge_pos;
  cgb::DevBuf<double> F;            // 3 n_nodes (device scratch for host-buffer calls)
  cgb::DevBuf<double> K;            // 9 n_blocks (device scratch for host-buffer calls)
  cgb::DevBuf<double> x;            // 3 n_nodes
  cgb::DevBuf<float> dpsi32, ddpsi32; // FP32 copies of the face shape derivatives (mixed mode)
  uint64_t faces_version = 0;       // faces->version the copies (FP32, sliced-ELL) were made from
  // Tables of the FP32 tangent (tile_prepare): per face entry the index of its node in its
  // cell's sorted node union (a cell: 16 consecutive Gauss points), per cell the union's size,
  // and the cell's items, each a node J and four nodes I <= J that share a point with it: the mask of
  // J's points | tile << 16 | J << 24, and the four block slots (-1: none). Cells with too many pairs
  // or nodes are "direct" (the per-entry tangent); tc_rest: the others that the tensor-core
  // tangent does not take (union above 42 nodes).
  bool tile_ready = false;
  cgb::DevBuf<uint8_t> nbr_u;
  cgb::DevBuf<int16_t> cell_U;
  cgb::DevBuf<int64_t> item_ptr;      // n_cells + 1
  cgb::DevBuf<cgb::TileCell> cells;   // the same per cell, with its entries, in one record
  cgb::DevBuf<uint32_t> item_code;
  cgb::DevBuf<int32_t> item_slot;     // 4 per item
  cgb::DevBuf<int32_t> direct, tc_rest;
  std::vector<int32_t> direct_h, tc_rest_h;
  int64_t n_items = 0;
  int64_t n_entries = 0;              // blocks over all cells (slots that are not -1)
  int cell_max_e = 0, cell_max_u = 0, cell_max_i = 0;  // most entries, nodes, items of a cell that is not direct
  int64_t tc_n_groups = 0;            // cells on the tensor path
  int64_t tc_point_cols = 0;          // sum over them of points x MMA columns (N)
  int tc_last_per_sm = 0;             // CTAs per SM of the last tensor-core tangent launch
  cgb_tuning tuning{};                // launch shape (0 = library default)
  cgb::DevBuf<int> work_ctr;          // per-chunk work counters of the residual kernel
  uint32_t test_stage_extra_tx = 0;   // failure-detection test only: bytes the staging never gets
  int n_graphs = 0;                   // live cgb_graph objects on this assembler
  // Second stream of the chunked face launch (tangent of chunk c beside residual of c+1).
  cudaStream_t side = nullptr;
  cudaEvent_t ev_start = nullptr, ev_done = nullptr, ev_chunk[kMaxChunks] = {nullptr};
  cgb::DevBuf<float> state32;         // per-point state between the residual and tangent kernels
  cgb::DevBuf<double> state64;
  cgb::DevBuf<int32_t> ent_point;     // the point of every face entry (per-entry tangent)
  cgb::DevBuf<int64_t> sell_ptr;      // sliced-ELL copy for the FP64 phase (groups of 32 points)
  cgb::DevBuf<int32_t> sidx;
  cgb::DevBuf<double> sdpsi, sddpsi;
  // Deterministic scatter: contributions ("units") and per-block / per-node ordered lists.
  // K units are either every pair (FP64, or with direct cells) or, for the FP32 tangent, the
  // slots of the cells' items (one fixed-order sum per cell and block); hinge pairs follow.
  bool det_ready = false;             // F lists
  bool det_pairs_ready = false;       // K lists over pairs
  bool det_entries_ready = false;     // K lists over the items' slots
  cgb::DevBuf<int64_t> blk_list_ptr;  // n_blocks + 1 (pair units)
  cgb::DevBuf<int64_t> blk_list;      // pair unit ids, ascending
  cgb::DevBuf<int64_t> blk_face_end, ent_face_end;  // per block, the first hinge pair in its list
  cgb::DevBuf<int64_t> ent_list_ptr;  // n_blocks + 1 (entry units)
  cgb::DevBuf<int64_t> ent_list;      // entry unit ids, ascending
  cgb::DevBuf<int64_t> node_list_ptr; // n_nodes + 1
  cgb::DevBuf<int64_t> node_list;     // F contribution ids, ascending
  cgb::DevBuf<double> contrib64;      // 9 per contribution
  cgb::DevBuf<float> contrib32;
  cgb::DevBuf<double> hinge_contrib;  // the hinge pairs' in mixed mode
  cgb::DevBuf<double> fcontrib;       // 3 per F contribution
  int64_t n_fcontrib = 0;
  int64_t hinge_f_base = 0;
  // Energies.
  cgb::DevBuf<double> energy;       // 3
  // Pinned staging for the host-buffer entry point.
  double* h_stage = nullptr;
  size_t h_stage_bytes = 0;
};

namespace cgb {
void ctx_retain(cgb_context* ctx);
void ctx_release(cgb_context* ctx);
// Tracing helpers (capi.cu): no-ops unless profiling is enabled on the context.
void prof_begin(cgb_context* ctx, int phase, cudaStream_t stream = nullptr);
void prof_end(cgb_context* ctx, int phase, int launches, cudaStream_t stream = nullptr);
// shape.cu
void shape_build(cgb_context* ctx, const double* gp_xy, int n_gp, const cgb_shape_params& prm,
                 const std::vector<Crease>& creases, cgb_shape* out);
// Phi and its derivatives of an existing set recomputed in place with other creases
// (same points, radius and so neighbour lists).
void shape_rebuild(cgb_shape* sh, const std::vector<Crease>& creases);
// The normalised distances s of a set built in mixed precision (which skips them), computed
// on demand with the FRNN's rounded operations; a no-op when the set has them.
void shape_distances(cgb_shape* sh);
// pattern.cu
void pattern_build(cgb_assembler* a);
void deterministic_prepare(cgb_assembler* a);
void shape_concat(cgb_context* ctx, const cgb_shape* const* sets, const int32_t* node_offset, int n_sets,
                  cgb_shape* out);
// Per-block lists of K units: pairs (units [0, n_pairs) then hinge pairs) or the slots of the
// cells' items (units [0, 4 n_items) then hinge pairs; needs tile_prepare and no direct cell).
void deterministic_pair_lists(cgb_assembler* a);
void deterministic_entry_lists(cgb_assembler* a);
// The tables of the FP32 tangent, made once per assembler.
constexpr int kTcMaxUnion = 42;
constexpr int kTileMaxU = 128;
constexpr int kTileMaxList = 110;  // lists above this take the per-entry tangent throughout
void tile_prepare(cgb_assembler* a);
// assemble.cu
void assemble_device(cgb_assembler* a, const double* d_x, double* d_K, double* d_F, int flags);
// Re-derive the assembler's copies of the face shape derivatives after a rebuild of the
// face set (no-op when they are current); enqueued on the context stream.
void refresh_face_copies(cgb_assembler* a);
void energies_device(cgb_assembler* a, const double* d_x, double* out3);
// Kinematic state rows (CGB_POINT_STATE_COLS per point) of a shape set at device x.
void point_state_device(cgb_context* ctx, const cgb_shape* S, const double* d_x, const double* A, const double* B,
                        const double* D, double* d_out);
// The shape set's point coordinates when the context's natural curvature is active (the
// kernels evaluate kappa_bar at each point's X), else null; refuses a set without them.
const double* natcurv_points(const cgb_context* ctx, const cgb_shape* S, const char* what);
// err: the context's device error word (bit 8: an index of the caller's arrays was out of
// range and the access was skipped).
void face_mixed_on_arrays(const cgb_face_problem& pr, const double* d_x, double* d_K, double* d_F,
                          float* kacc, int* err, cudaStream_t st);
}  // namespace cgb
