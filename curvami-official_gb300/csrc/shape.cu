// shape.cu — stage A on sm_103a: neighbour gather (GlobalFRNN) and RKPM shape
// functions with crease visibility (GlobalRKPM), FP64 or with the per-neighbour part in FP32 pairs.
//
// Reference: core/include/curvami/FRNN.h:23-78, core/include/curvami/Enrichment.h:23-92,
// core/include/curvami/GlobalRKPM.h:15-397.
//
// Design: the node cell grid, made on the device, is a dense array over the reference's flattened cell key
// (y * cols + x, so keys that wrap across a row resolve to the same cells as the
// reference's hash map). One thread per Gauss point gathers its neighbours in the
// reference's order (dx outer, dy inner, node index ascending in a cell) with an FP64
// distance test written without FMA contraction, so the neighbour sets and their order
// are bit-exact. The RKPM runs as three kernels (four in pairs) over chunks of points, each
// with the parallelism its part has: moments, one or a few threads per point, which leave the
// weights' jets of every neighbour in the output arrays (in pairs a kernel of one thread
// per neighbour makes them first); the solve, a thread per point; the values, a thread per
// neighbour, from the jets and the point's polynomials. GB300's FP64 rate is 1/62 of the FP32 rate, so
// the FP64 pipe bounds the first form throughout and the solve alone in the second. Per-node
// crease sides are hoisted into a per-node array.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <string>
#include <type_traits>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "cgb_pair.cuh"

namespace cgb {
namespace {

constexpr int kThreads = 128;

inline unsigned blocks_for(int64_t n, int t = kThreads) { return static_cast<unsigned>((n + t - 1) / t); }

// The node cell grid (FRNN.h:33-44): the nodes of every cell in ascending order, with their float
// coordinates beside them.
struct GridDev {
  double minx, miny, cell;
  int cols;
  long long ncells;
  const int64_t* cell_start;  // ncells + 1
  const int32_t* cell_nodes;
};

// FP32 pre-test of the FRNN distance test. Coordinates relative to the grid's lower corner
// are rounded to float (cell32, per node in cell order; the point's in the kernel), the squared
// distance is formed in float, and `margin` bounds its difference from the exact squared distance
// (coordinate rounding, float arithmetic, the float radius; computed on the host from the
// extent of the nodes and points). A candidate beyond r^2 + margin is outside and one
// below r^2 - margin inside whatever FP64 gives; only those within the margin take the
// exact FP64 test, so every decision is the FP64 one.
struct FrnnPre {
  const float2* cell32;   // per node in cell order, (x - minx, y - miny) in float
  const float* r2c32;     // per node in cell order r^2 in float, or nullptr for the single radius
  float r2f;              // the single radius squared, in float
  float margin;
};

// Cell key of every node, and the nodes per cell.
__global__ void cell_count_kernel(int n_nodes, const double* __restrict__ node_xy, GridDev G, int32_t* __restrict__ key,
                                  int32_t* __restrict__ count) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_nodes) return;
  const int cx = static_cast<int>(floor(__ddiv_rn(__dsub_rn(node_xy[2 * j], G.minx), G.cell)));
  const int cy = static_cast<int>(floor(__ddiv_rn(__dsub_rn(node_xy[2 * j + 1], G.miny), G.cell)));
  const long long at = static_cast<long long>(cy) * G.cols + cx;
  const int k = at >= 0 && at < G.ncells ? static_cast<int>(at) : 0;   // (a coordinate that is not a number)
  key[j] = k;
  atomicAdd(&count[k], 1);
}

// The nodes into their cells, in any order (cursor: a copy of cell_start).
__global__ void cell_fill_kernel(int n_nodes, const int32_t* __restrict__ key, unsigned long long* __restrict__ cursor,
                                 int32_t* __restrict__ list) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n_nodes) list[atomicAdd(&cursor[key[j]], 1ULL)] = j;
}

// Ascending node index per cell: every node's rank among its cell's, and its float coordinates
// and radius at that place.
__global__ void cell_sort_kernel(int n_nodes, const double* __restrict__ node_xy, const double* __restrict__ rho_node,
                                 GridDev G, const int32_t* __restrict__ key, const int32_t* __restrict__ list,
                                 int32_t* __restrict__ sorted, float2* __restrict__ cell32, float* __restrict__ r2c32) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_nodes) return;
  const int64_t k0 = G.cell_start[key[j]], k1 = G.cell_start[key[j] + 1];
  int64_t at = k0;
  for (int64_t k = k0; k < k1; ++k) at += list[k] < j;
  sorted[at] = j;
  cell32[at] = make_float2(__double2float_rn(__dsub_rn(node_xy[2 * j], G.minx)),
                           __double2float_rn(__dsub_rn(node_xy[2 * j + 1], G.miny)));
  if (rho_node) r2c32[at] = __double2float_rn(__dmul_rn(rho_node[j], rho_node[j]));
}

// Thread per Gauss point. The counting pass (out_idx == nullptr) leaves the decisions of the first
// kMaskWords * 32 candidates as bits, [word][point]; the filling pass reads them back and tests only
// candidates beyond. Candidates of a cell are consecutive, so the counting pass makes one 8-byte
// load per candidate. 1,000,000 scattered points: both passes 2.1 ms when each tested every
// candidate through its node index.
constexpr int kMaskWords = 8;

__global__ void frnn_kernel(int n_gp, const double* __restrict__ gp_xy,
                            const double* __restrict__ node_xy, const double* __restrict__ rho_node,
                            double rho2, GridDev G, FrnnPre pre, const int64_t* __restrict__ ptr,
                            int32_t* __restrict__ count, uint32_t* __restrict__ mask, int32_t* __restrict__ out_idx) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_gp) return;
  const double gx = gp_xy[2 * g], gy = gp_xy[2 * g + 1];
  const float gxf = __double2float_rn(gx - G.minx), gyf = __double2float_rn(gy - G.miny);
  const int qx = static_cast<int>(floor(__ddiv_rn(__dsub_rn(gx, G.minx), G.cell)));
  const int qy = static_cast<int>(floor(__ddiv_rn(__dsub_rn(gy, G.miny), G.cell)));
  auto test = [&](int64_t k) {
    const float2 nf = pre.cell32[k];
    const float fdx = nf.x - gxf, fdy = nf.y - gyf;
    const float d2f = fdx * fdx + fdy * fdy;
    const float r2f = pre.r2c32 ? pre.r2c32[k] : pre.r2f;
    if (d2f > r2f + pre.margin) return false;      // outside, whatever FP64 gives
    if (d2f < r2f - pre.margin) return true;       // inside, whatever FP64 gives
    const int j = G.cell_nodes[k];
    const double ddx = __dsub_rn(node_xy[2 * j], gx);
    const double ddy = __dsub_rn(node_xy[2 * j + 1], gy);
    const double dist2 = __dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy));
    return dist2 <= (rho_node ? __dmul_rn(rho_node[j], rho_node[j]) : rho2);
  };
  const bool fill = out_idx != nullptr;
  int64_t pos = fill ? ptr[g] : 0;
  int cnt = 0, o = 0;           // neighbours; candidates so far
  uint32_t word = fill ? mask[g] : 0u;
  for (int dx = -1; dx <= 1; ++dx) {
    for (int dy = -1; dy <= 1; ++dy) {
      const long long key = static_cast<long long>(qy + dy) * G.cols + (qx + dx);
      if (key < 0 || key >= G.ncells) continue;
      int64_t k = G.cell_start[key];
      const int64_t k1 = G.cell_start[key + 1];
      if (!fill) {
        for (; k < k1; ++k, ++o) {
          const bool in = test(k);
          cnt += in;
          if (o < 32 * kMaskWords) {
            word |= static_cast<uint32_t>(in) << (o & 31);
            if ((o & 31) == 31) { mask[static_cast<int64_t>(o >> 5) * n_gp + g] = word; word = 0u; }
          }
        }
      } else {
        while (k < k1 && o < 32 * kMaskWords) {   // the set bits of this cell's candidates, word by word
          const int bit = o & 31, len = static_cast<int>(min(static_cast<int64_t>(32 - bit), k1 - k));
          uint32_t b = word >> bit;
          if (len < 32) b &= (1u << len) - 1u;
          for (; b; b &= b - 1u) out_idx[pos++] = G.cell_nodes[k + __ffs(b) - 1];
          k += len;
          o += len;
          if ((o & 31) == 0 && o < 32 * kMaskWords) word = mask[static_cast<int64_t>(o >> 5) * n_gp + g];
        }
        for (; k < k1; ++k)
          if (test(k)) out_idx[pos++] = G.cell_nodes[k];
      }
    }
  }
  if (!fill) {
    count[g] = cnt;
    if (o < 32 * kMaskWords) mask[static_cast<int64_t>(o >> 5) * n_gp + g] = word;   // the last, part-filled word
  }
}

// The point of entry e of the points [g0, g1): the warp finds it for its first entry, 32 probes at a
// time (four dependent loads for 262,144 points, where a bisection takes 18), and the lanes step
// forward from there. Every lane of the warp calls it.
__device__ __forceinline__ int point_of(const int64_t* __restrict__ ptr, int g0, int g1, int64_t e, int64_t e_end) {
  const int lane = threadIdx.x & 31;
  const int64_t ef = __shfl_sync(0xffffffffu, e < e_end ? e : e_end - 1, 0);
  int lo = g0, n = g1 - g0;            // the point is one of [lo, lo + n): ptr[lo] <= ef < ptr[lo + n]
  while (n > 1) {
    const int step = (n - 1) / 32 + 1;
    const int at = lo + lane * step;
    const bool below = lane * step < n && __ldg(ptr + at) <= ef;
    const int last = 31 - __clz(__ballot_sync(0xffffffffu, below));   // lane 0 is always below
    lo += last * step;
    n = min(step, n - last * step);
  }
  int g = lo;
  if (e < e_end)
    while (__ldg(ptr + g + 1) <= e) ++g;
  return g;
}

// Normalised distances s of the neighbour lists, with explicitly rounded operations (bitwise the
// FRNN's own). One entry per thread: the square root and the division, about 30 FP64 operations, on
// full warps; inside the FRNN's candidate loop a third of the lanes had work (300,000 points:
// 1.15 ms of its 1.79 ms). Sets built in mixed precision, whose RKPM does not read s, get it when a
// caller downloads it.
__global__ void distance_kernel(int n_gp, const double* __restrict__ gp_xy, const double* __restrict__ node_xy,
                                const double* __restrict__ rho_node, double rho, const int64_t* __restrict__ ptr,
                                const int32_t* __restrict__ idx, int64_t nnz, double* __restrict__ out_s) {
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int g = point_of(ptr, 0, n_gp, e, nnz);
  if (e >= nnz) return;
  const int j = idx[e];
  const double ddx = __dsub_rn(node_xy[2 * j], gp_xy[2 * g]);
  const double ddy = __dsub_rn(node_xy[2 * j + 1], gp_xy[2 * g + 1]);
  const double dist2 = __dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy));
  out_s[e] = __ddiv_rn(__dsqrt_rn(dist2), rho_node ? rho_node[j] : rho);
}

// The reference's guards over the points: out = {singular points, first of them, collapsed
// pivots, first of them}, preset to {0, n, 0, n}.
__global__ void guard_kernel(int n, const int8_t* __restrict__ bad, int* __restrict__ out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = g < n ? bad[g] : 0;
  if (b != 1 && b != 2) return;
  atomicAdd(out + 2 * (b - 1), 1);
  atomicMin(out + 2 * (b - 1) + 1, g);
}

// Neighbour counts -> CSR offsets on the device: ptr[g + 1] = sum of cnt[0..g], plus the
// total and the largest count for the host (two numbers instead of the whole array).
constexpr int kScanThreads = 1024;

__global__ void scan_local_kernel(int64_t n, const int32_t* __restrict__ cnt, int64_t* __restrict__ ptr,
                                  int64_t* __restrict__ block_sum, int32_t* __restrict__ block_max) {
  __shared__ int64_t sv[kScanThreads];
  __shared__ int32_t mv[kScanThreads];
  const int t = threadIdx.x;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kScanThreads + t;
  const int32_t c = i < n ? cnt[i] : 0;
  sv[t] = c;
  mv[t] = c;
  __syncthreads();
  for (int off = 1; off < kScanThreads; off <<= 1) {   // Hillis-Steele inclusive scan
    const int64_t a = t >= off ? sv[t - off] : 0;
    const int32_t m = t >= off ? mv[t - off] : 0;
    __syncthreads();
    sv[t] += a;
    mv[t] = max(mv[t], m);
    __syncthreads();
  }
  if (i < n) ptr[i + 1] = sv[t];
  if (t == kScanThreads - 1) {
    block_sum[blockIdx.x] = sv[t];
    block_max[blockIdx.x] = mv[t];
  }
}

// One warp: block totals -> exclusive block offsets (in place); totals[0] = sum, [1] = max.
__global__ void scan_blocks_kernel(int nb, int64_t* __restrict__ block_sum, const int32_t* __restrict__ block_max,
                                   int64_t* __restrict__ totals) {
  const int lane = threadIdx.x;
  int64_t run = 0;
  int32_t mx = 0;
  for (int b0 = 0; b0 < nb; b0 += 32) {
    const int b = b0 + lane;
    const int64_t v = b < nb ? block_sum[b] : 0;
    mx = max(mx, b < nb ? block_max[b] : 0);
    int64_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (b < nb) block_sum[b] = run + incl - v;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) { totals[0] = run; totals[1] = mx; }
}

__global__ void scan_add_kernel(int64_t n, int64_t* __restrict__ ptr, const int64_t* __restrict__ block_off) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kScanThreads + threadIdx.x;
  if (i < n) ptr[i + 1] += block_off[blockIdx.x];
  if (i == 0) ptr[0] = 0;
}

// ptr[i + 1] = cnt[0] + .. + cnt[i] (n > 0); tot: the sum and the largest count, on the device.
void scan_counts(cgb_context* ctx, int64_t n, const int32_t* cnt, int64_t* ptr, int64_t* tot) {
  cudaStream_t st = ctx->stream;
  const int nb = static_cast<int>((n + kScanThreads - 1) / kScanThreads);
  ShapeScratch& w = ctx->scratch;
  w.bsum.ensure(nb);
  w.bmax.ensure(nb);
  scan_local_kernel<<<nb, kScanThreads, 0, st>>>(n, cnt, ptr, w.bsum.p, w.bmax.p);
  scan_blocks_kernel<<<1, 32, 0, st>>>(nb, w.bsum.p, w.bmax.p, tot);
  scan_add_kernel<<<nb, kScanThreads, 0, st>>>(n, ptr, w.bsum.p);
  CGB_CUDA(cudaGetLastError());
}

// Per-node crease side sn = (f >= 0 ? +1 : -1) (GlobalRKPM.h:92-93).
template <int L>
__global__ void node_side_kernel(int n_nodes, const double* __restrict__ node_xy, DevCrease cr,
                                 int8_t* __restrict__ side) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, j = min(t / L, n_nodes - 1);
  const DevIndicator I = eval_indicator<L>(node_xy[2 * j], node_xy[2 * j + 1], cr);
  if (t / L < n_nodes && t % L == 0) side[j] = (I.f >= 0.0) ? 1 : -1;
}

// Crease c's indicator at every Gauss point, written in place into the [g][crease][6]
// layout the RKPM kernel reads (n_creases values per point).
template <int L>
__global__ void gp_indicator_kernel(int n_gp, const double* __restrict__ gp_xy, DevCrease cr, int c, int n_creases,
                                    double* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, g = min(t / L, n_gp - 1);
  const DevIndicator I = eval_indicator<L>(gp_xy[2 * g], gp_xy[2 * g + 1], cr);
  if (t / L >= n_gp || t % L != 0) return;
  double* o = out + 6 * (static_cast<int64_t>(g) * n_creases + c);
  o[0] = I.f; o[1] = I.gx; o[2] = I.gy; o[3] = I.hxx; o[4] = I.hyy; o[5] = I.hxy;
}

// Lanes per point of the indicator kernels: a warp's FP64 part takes as long for one point as for 32,
// so more lanes only while every warp has an SM quarter of its own.
template <class F>
void indicator_lanes(int n, int sms, F&& launch) {
  const int64_t lanes = 32LL * 4 * sms;
  if (n * 32LL <= lanes) launch(std::integral_constant<int, 32>{});
  else if (n * 4LL <= lanes) launch(std::integral_constant<int, 4>{});
  else launch(std::integral_constant<int, 1>{});
}

__device__ __forceinline__ void inv3(const double m[3][3], double r[3][3]) {
  const double c00 = m[1][1] * m[2][2] - m[1][2] * m[2][1];
  const double c10 = m[1][2] * m[2][0] - m[1][0] * m[2][2];
  const double c20 = m[1][0] * m[2][1] - m[1][1] * m[2][0];
  const double det = m[0][0] * c00 + m[0][1] * c10 + m[0][2] * c20;
  const double id = 1.0 / det;
  r[0][0] = c00 * id; r[1][0] = c10 * id; r[2][0] = c20 * id;
  r[0][1] = (m[0][2] * m[2][1] - m[0][1] * m[2][2]) * id;
  r[1][1] = (m[0][0] * m[2][2] - m[0][2] * m[2][0]) * id;
  r[2][1] = (m[0][1] * m[2][0] - m[0][0] * m[2][1]) * id;
  r[0][2] = (m[0][1] * m[1][2] - m[0][2] * m[1][1]) * id;
  r[1][2] = (m[0][2] * m[1][0] - m[0][0] * m[1][2]) * id;
  r[2][2] = (m[0][0] * m[1][1] - m[0][1] * m[1][0]) * id;
}

__device__ __forceinline__ void mm3(const double a[3][3], const double b[3][3], double c[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) c[r][k] = a[r][0] * b[0][k] + a[r][1] * b[1][k] + a[r][2] * b[2][k];
}

// Raw moments xi^a eta^b, a + b <= 2 ORDER, degree-major with b ascending; basis
// function i of Basis<ORDER> is the monomial xi^bx(i) eta^by(i).
template <int ORDER>
struct RawIdx {
  static constexpr int D = 2 * ORDER;
  static constexpr int NR = (D + 1) * (D + 2) / 2;
  __host__ __device__ static constexpr int r(int a, int b) { return (a + b) * (a + b + 1) / 2 + b; }
  __host__ __device__ static constexpr int deg(int i) {
    int d = 0;
    while ((d + 1) * (d + 2) / 2 <= i) ++d;
    return d;
  }
  __host__ __device__ static constexpr int by(int i) { return i - deg(i) * (deg(i) + 1) / 2; }
  __host__ __device__ static constexpr int bx(int i) { return deg(i) - by(i); }
};

// The polynomials of one point, scaled by their powers of rho: C, C_x, C_y, C_xx, C_yy, C_xy of
// GlobalRKPM.h:363-396, coefficients of the monomials of xi, eta.
template <int ORDER>
struct RowJets {
  static constexpr int NP = (ORDER + 1) * (ORDER + 2) / 2;
  double c0[NP], c0x[NP], c0y[NP], c0xx[NP], c0yy[NP], c0xy[NP];
};

// The per-point part of GlobalRKPM::solve (GlobalRKPM.h:161-396) from the raw-moment sums of the six
// weight jets (FP64): M, the reference's guards, and the polynomials that multiply the jets. Returns
// the guard code (0 fine, 1 singular, 2 pivot collapse).
//
// Every entry of M = sum_I w_I p_I p_I^T is a raw moment, and so is every entry of the S^g =
// sum_I (D^g w_I) p_I p_I^T. With p_x = D p (a constant matrix) M_x = S^x + D M + M D^T. The
// reference's C = b . p, b = M^-1 e0, has the derivative C_x = (b_x + D^T b) . p; written for
// c = b_x + D^T b the terms D M and M D^T of M_x b_x = -M^-1 M_x b become constants:
//   M b = e0,   M c_x = -S^x b - D_x e0,
//   M c_xx = -S^xx b - 2 S^x c_x + D_x D_x e0,   M c_xy = -S^xy b - S^x c_y - S^y c_x + D_x D_y e0
// (y alike), with D_x e0 the unit vector of xi, D_x D_x e0 twice that of xi^2, D_x D_y e0 that of
// xi eta. So neither the jets of M (135 of 1,050 FP64 operations for the quadratic basis) nor the
// derivatives of the basis on the coefficients (40) are formed. 262,144 points,
// quadratic: 485 -> 373 us, with the coefficients left as pairs 560 -> 385 us. Against extended
// precision the coefficients' errors are the same (quadratic) or a quarter smaller (cubic).
// at(g, a, b): S^g_ab = sum_I (D^g w_I) xi^a eta^b for g = 0 (w), 1 (x), 2 (y), 3 (xx), 4 (yy), 5 (xy).
template <int ORDER, class Sums>
__device__ __forceinline__ int point_solve(const Sums& at, RowJets<ORDER>& R) {
  constexpr int NP = (ORDER + 1) * (ORDER + 2) / 2;
  using RI = RawIdx<ORDER>;
  auto entry = [&](int g, int i, int j) { return at(g, RI::bx(i) + RI::bx(j), RI::by(i) + RI::by(j)); };

  // The reference inverts M by blocks (GlobalRKPM.h:197-345): the leading 3x3 block with
  // a residual guard, then one bordering step per further basis function with a Schur-pivot
  // guard, carrying the five derivative jets of the whole inverse along. Here M is factored once
  // (LDL^T, no pivoting: M is symmetric positive semi-definite). The guards are evaluated as the
  // reference does: the 3x3 residual test on the leading block, and the pivot test on the Schur
  // complements, which are the LDL^T pivots d_k for k >= 3.
  int bad = 0;
  {
    double m3[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) m3[r][c] = entry(0, r, c);
    double inv[3][3], chk[3][3];
    inv3(m3, inv);
    mm3(m3, inv, chk);
    // |chk - I| <= 1e-8 on the bits: a comparison of doubles issues on the FP64 pipe. NaN passes,
    // as it does through fmax.
    const long long mag = 0x7fffffffffffffffll, inf = 0x7ff0000000000000ll;
    const long long lim = __double_as_longlong(1e-8);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const long long res = __double_as_longlong(chk[r][c] - (r == c ? 1.0 : 0.0)) & mag;
        if (!isfinite(inv[r][c]) || (res > lim && res <= inf)) bad = 1;
      }
  }
  // LDL^T of M: L unit lower, iD the reciprocal pivots.
  double Lf[NP][NP], Dg[NP], iD[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const double mjj = entry(0, j, j);
    double d = mjj, LD[NP];
#pragma unroll
    for (int q = 0; q < j; ++q) {
      LD[q] = Lf[j][q] * Dg[q];
      d -= Lf[j][q] * LD[q];
    }
    Dg[j] = d;
    iD[j] = 1.0 / d;
    if (j >= 3 && !(fabs(d) > 1e-12 * fmax(fabs(mjj), 1.0)) && bad == 0) bad = 2;
#pragma unroll
    for (int i = j + 1; i < NP; ++i) {
      double v = entry(0, i, j);
#pragma unroll
      for (int q = 0; q < j; ++q) v -= Lf[i][q] * LD[q];
      Lf[i][j] = v * iD[j];
    }
  }
  // x <- M^-1 x in place.
  auto solve = [&](double* x) {
#pragma unroll
    for (int i = 1; i < NP; ++i)
#pragma unroll
      for (int q = 0; q < i; ++q) x[i] -= Lf[i][q] * x[q];
#pragma unroll
    for (int i = 0; i < NP; ++i) x[i] *= iD[i];
#pragma unroll
    for (int i = NP - 2; i >= 0; --i)
#pragma unroll
      for (int q = i + 1; q < NP; ++q) x[i] -= Lf[q][i] * x[q];
  };
  // y -= S^g x.
  auto symv = [&](int g, const double* x, double* y) {
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
      for (int q = 0; q < NP; ++q) y[i] -= entry(g, i, q) * x[q];
  };
  // y <- the value v at the monomial xi^a eta^b.
  auto unit = [&](double* y, int a, int b, double v) {
#pragma unroll
    for (int i = 0; i < NP; ++i) y[i] = a + b <= ORDER && i == RI::r(a, b) ? v : 0.0;
  };
  auto twice = [&](const double* x, double* y) {
#pragma unroll
    for (int i = 0; i < NP; ++i) y[i] = x[i] + x[i];
  };
  double t[NP];
  unit(R.c0, 0, 0, 1.0); solve(R.c0);
  unit(R.c0x, 1, 0, -1.0); symv(1, R.c0, R.c0x); solve(R.c0x);
  unit(R.c0y, 0, 1, -1.0); symv(2, R.c0, R.c0y); solve(R.c0y);
  unit(R.c0xx, 2, 0, 2.0); symv(3, R.c0, R.c0xx); twice(R.c0x, t); symv(1, t, R.c0xx); solve(R.c0xx);
  unit(R.c0yy, 0, 2, 2.0); symv(4, R.c0, R.c0yy); twice(R.c0y, t); symv(2, t, R.c0yy); solve(R.c0yy);
  unit(R.c0xy, 1, 1, 1.0); symv(5, R.c0, R.c0xy); symv(1, R.c0y, R.c0xy); symv(2, R.c0x, R.c0xy); solve(R.c0xy);
  return bad;
}

struct RkpmArgs {
  int n_gp, n_nodes, kernel, n_creases;
  double rho;
  const float4* node_pair;   // mixed kernel: 2 per node (node_pair_kernel)
  fp2 irho, irho2;           // mixed kernel: 1 / rho and 1 / rho^2 as pairs
  const double* gp_xy;
  const double* node_xy;
  const double* rho_node;
  const int64_t* ptr;
  const int32_t* idx;
  const double* s;
  const double* gind;        // 6 * n_creases per Gauss point
  const int8_t* node_side;   // n_creases * n_nodes
  double* psi;
  double* dpsi;
  double* ddpsi;
  int8_t* bad;
  double ir;           // FP64 kernels: 1 / rho
  const double* fac;   // rho / rho_I per node, or null (single radius)
  int8_t* tip;         // point in the cap of a crease end (its indicators vary there)
  int32_t* order;      // the points in the order the moment kernels take them (point_order_kernel)
  double* mom;         // moment sums, [sum][point of the chunk]
  double* coef;        // shape polynomials, 6 NP per point of the chunk
  int g0, g1;          // the launch's points
};

// ---- FP64 RKPM -------------------------------------------------------------------------
//
// With xi, eta the scaled differences, the six weight jets of a neighbour are w, A xi, A eta, B xi^2,
// B eta^2 and C xi eta with three radial factors (GlobalRKPM.h:59-84 with its d2x, d2y;
// f = rho / rho_I):
//   A = f^2 w'/s,   B = f^4 (w'' + w'/s) / s^2,   C = f^4 (w'' - w'/s) / s^2.
// Where no crease end caps the point, a crease only scales them (by 0 or 1), and the raw sums of the
// jets are sums of w, A, B and C against monomials:
//   S_ab = W(a, b),  S^x_ab = A(a+1, b),  S^y_ab = A(a, b+1),  S^xx_ab = B(a+2, b),
//   S^yy_ab = B(a, b+2),  S^xy_ab = C(a+1, b+1):
// 15 + 20 + 24 + 15 sums for the quadratic basis where the six jets take 90, and one division per
// neighbour. In the cap of a crease end the visibility factors vary with the point
// (GlobalRKPM.h:87-112) and mix the jets: those points sum the six jets as they come.
// GB300's FP64 pipe (2 FMA per cycle and SM) bounds all of it, so
//  - rkpm_moment_kernel takes the sums over a point's neighbours (about 130 FP64 operations each, 150
//    in a cap) and leaves the pair's w, A, B, C (or its six jets) in the output arrays;
//  - rkpm_solve_kernel, one point per thread, factors M (point_solve) and leaves the six polynomials
//    in xi, eta that multiply the jets, derivatives of the basis and powers of rho folded in;
//  - rkpm_value_kernel, one pair per thread, evaluates them (about 60 operations) over the pair's
//    jets: reading them back is a tenth of computing them again.
// Measured on 300,000 points (28 neighbours, quadratic): RKPM 10.7 ms as one kernel of 90 sums and
// both passes, about 650 operations per neighbour; 3.9 ms so (moments 2.5, solve 0.45, values 1.0).
// 32,400 points with 113 neighbours, cubic, half of them in a cap: 12.8 -> 3.3 ms.
template <int ORDER>
struct MomIdx {
  static constexpr int D = 2 * ORDER;
  static constexpr int tri(int d) { return (d + 1) * (d + 2) / 2; }   // monomials of degree <= d
  static constexpr int NW = tri(D), NA = tri(D + 1) - 1, NB = tri(D + 2) - 4, NC = NW;
  static constexpr int N = NW + NA + NB + NC;
  __host__ __device__ static constexpr int r(int a, int b) { return (a + b) * (a + b + 1) / 2 + b; }
  // Positions in [W | A | B | C]; A starts at degree 1, B at degree 2 without xi eta.
  __host__ __device__ static constexpr int w(int a, int b) { return r(a, b); }
  __host__ __device__ static constexpr int ax(int a, int b) { return NW + r(a, b) - 1; }
  __host__ __device__ static constexpr int bx(int a, int b) {
    return NW + NA + (r(a, b) == 3 ? 0 : r(a, b) == 5 ? 1 : r(a, b) - 4);
  }
  __host__ __device__ static constexpr int cx(int a, int b) { return NW + NA + NB + r(a - 1, b - 1); }
};

// The order in which the moment kernels take the points: within windows of kSortPoints, those outside
// the caps first, then by falling neighbour counts. The lanes of a warp wait for the one with the most
// neighbours, and a warp with points of both kinds is walked twice.
// RKPM of 300,000 scattered points of 28 neighbours 4.15 -> 3.94 ms, 32,400 cubic Gauss points of 113,
// half of them in a cap, 3.47 -> 3.31 ms, 1,000,000 mixed points 5.88 -> 5.79 ms.
constexpr int kSortPoints = 1024;
__global__ void __launch_bounds__(kSortPoints) point_order_kernel(RkpmArgs a) {
  constexpr int kBins = 512;
  __shared__ int s_bin[kBins];
  const int t = threadIdx.x, w0 = blockIdx.x * kSortPoints, g = w0 + t;
  if (t < kBins) s_bin[t] = 0;
  __syncthreads();
  int bin = 0, rank = 0;
  if (g < a.n_gp) {
    const double* I = a.gind + static_cast<int64_t>(g) * 6 * a.n_creases;
    bool tip = false;
    for (int c = 0; c < a.n_creases; ++c)
      for (int q = 1; q < 6; ++q) tip = tip || I[6 * c + q] != 0.0;
    a.tip[g] = tip;
    const int64_t n = a.ptr[g + 1] - a.ptr[g];
    bin = (tip ? kBins / 2 : 0) + kBins / 2 - 1 - static_cast<int>(min(n, static_cast<int64_t>(kBins / 2 - 1)));
    rank = atomicAdd(&s_bin[bin], 1);
  }
  __syncthreads();
  if (t < 32) {   // exclusive sums of the bins, 16 per lane
    int v[kBins / 32], sum = 0;
#pragma unroll
    for (int k = 0; k < kBins / 32; ++k) { v[k] = sum; sum += s_bin[t * (kBins / 32) + k]; }
    int before = sum;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int up = __shfl_up_sync(0xffffffffu, before, o);
      if (t >= o) before += up;
    }
#pragma unroll
    for (int k = 0; k < kBins / 32; ++k) s_bin[t * (kBins / 32) + k] = before - sum + v[k];
  }
  __syncthreads();
  if (g < a.n_gp) a.order[w0 + s_bin[bin] + rank] = g;
}

__global__ void node_fac_kernel(int n_nodes, const double* __restrict__ rho_node, double rho, double* __restrict__ fac) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n_nodes) fac[j] = rho / rho_node[j];
}

// Radial factors of a neighbour at normalised distance s: w, A, B, C without f.
__device__ __forceinline__ void radial(int kernel, double s, double& w, double& A, double& B, double& C) {
  double ds, dd;   // w'/s, w''
  const double is2 = s == 0.0 ? 0.0 : 1.0 / (s * s);
  if (kernel == 0) {  // quartic spline, GlobalRKPM.h:15-17
    w = fma(s * s, fma(s, fma(-3.0, s, 8.0), -6.0), 1.0);
    ds = fma(s, fma(-12.0, s, 24.0), -12.0);
    dd = fma(s, fma(-36.0, s, 48.0), -12.0);
  } else if (s <= 0.5) {  // cubic B-spline (extension)
    w = fma(s * s, fma(4.0, s, -4.0), 2.0 / 3.0);
    ds = fma(12.0, s, -8.0);
    dd = fma(24.0, s, -8.0);
  } else {
    const double r = 1.0 - s;
    w = 4.0 / 3.0 * (r * r * r);
    ds = -4.0 * (r * r) * (s * is2);
    dd = 8.0 * r;
  }
  if (s >= 1.0) { w = 0.0; ds = 0.0; dd = 0.0; }
  if (s < 1e-14) ds = 0.0;
  A = ds;
  B = (dd + ds) * is2;
  C = (dd - ds) * is2;
}

// The sums of one point's neighbours (L lanes share them). PART 0: all; the cubic basis's 132 (168 in
// a cap) do not fit the registers, so PART 1 takes W and A (the jets w, x, y) and PART 2 B and C (xx,
// yy, xy). TIP: the points in the cap of a crease end; the others otherwise.
template <int ORDER, int PART, int L, bool TIP>
__device__ __forceinline__ void moment_sums(const RkpmArgs& a) {
  using MI = MomIdx<ORDER>;
  using RI = RawIdx<ORDER>;
  constexpr bool P1 = PART != 2, P2 = PART != 1;
  constexpr int J0 = P1 ? 0 : 3, J1 = P2 ? 6 : 3;   // the jets of a cap's sums
  constexpr int LO = TIP ? J0 * RI::NR : P1 ? 0 : MI::NW + MI::NA;
  constexpr int HI = TIP ? J1 * RI::NR : P2 ? MI::N : MI::NW + MI::NA;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int slot = t / L, sub = t % L;
  const bool here = slot < a.g1 - a.g0;
  const int gc = a.order[here ? a.g0 + slot : a.g1 - 1];
  const int nc = a.n_creases;
  const double* gind = a.gind + static_cast<int64_t>(gc) * 6 * nc;
  const bool mine = here && (a.tip[gc] != 0) == TIP;
  if (!__any_sync(0xffffffffu, mine)) return;
  const int64_t p0 = a.ptr[gc];
  const int n = mine ? static_cast<int>(a.ptr[gc + 1] - p0) : 0;
  const double gx = a.gp_xy[2 * gc], gy = a.gp_xy[2 * gc + 1];
  double S[HI - LO];
#pragma unroll
  for (int k = 0; k < HI - LO; ++k) S[k] = 0.0;
  for (int q = sub; q < n; q += L) {
    const int64_t e = p0 + q;
    const int j = a.idx[e];
    const double xi = (gx - a.node_xy[2 * j]) * a.ir, eta = (gy - a.node_xy[2 * j + 1]) * a.ir;
    double w, A, B, C;
    radial(a.kernel, a.s[e], w, A, B, C);
    if (a.fac) {
      const double f = a.fac[j], f2 = f * f, f4 = f2 * f2;
      A *= f2; B *= f4; C *= f4;
    }
    C *= xi * eta;   // the xy jet, and C(a+1, b+1) = sum (C xi eta) xi^a eta^b
    double J[6];
    if constexpr (TIP) {
      J[0] = w; J[1] = A * xi; J[2] = A * eta;
      J[3] = B * (xi * xi); J[4] = B * (eta * eta); J[5] = C;
      for (int c = 0; c < nc; ++c) {   // GlobalRKPM.h:87-112
        const double* I = gind + 6 * c;
        const double sn = a.node_side[static_cast<int64_t>(c) * a.n_nodes + j] > 0 ? 0.5 : -0.5;
        const double sr = sn * a.rho, srr = sr * a.rho;
        const double V = fma(sn, I[0], 0.5), Vx = sr * I[1], Vy = sr * I[2];
        const double o0 = J[0], o1 = J[1], o2 = J[2];
        J[0] = o0 * V;
        J[1] = fma(o1, V, o0 * Vx);
        J[2] = fma(o2, V, o0 * Vy);
        J[3] = fma(J[3], V, fma(2.0 * o1, Vx, o0 * (srr * I[3])));
        J[4] = fma(J[4], V, fma(2.0 * o2, Vy, o0 * (srr * I[4])));
        J[5] = fma(J[5], V, fma(o1, Vy, fma(o2, Vx, o0 * (srr * I[5]))));
      }
      if (P1) { a.psi[e] = J[0]; a.dpsi[2 * e] = J[1]; a.dpsi[2 * e + 1] = J[2]; }
      if (P2) { a.ddpsi[3 * e] = J[3]; a.ddpsi[3 * e + 1] = J[4]; a.ddpsi[3 * e + 2] = J[5]; }
    } else {
      double vis = 1.0;
      for (int c = 0; c < nc; ++c) {
        const double f = gind[6 * c];
        vis *= 0.5 * (1.0 + (a.node_side[static_cast<int64_t>(c) * a.n_nodes + j] > 0 ? f : -f));
      }
      if (vis != 1.0) { w *= vis; A *= vis; B *= vis; C *= vis; }
      if (P1) { a.psi[e] = w; a.dpsi[2 * e] = A; }
      if (P2) { a.ddpsi[3 * e] = B; a.ddpsi[3 * e + 2] = C; }
    }
    // Monomials degree by degree, each from one of the degree before.
    double m[MI::D + 3];
    m[0] = 1.0;
#pragma unroll
    for (int d = 0; d <= MI::D + (TIP ? 0 : P2 ? 2 : 1); ++d) {
      if (d > 0) {
        m[d] = m[d - 1] * eta;
#pragma unroll
        for (int b = d - 1; b >= 0; --b) m[b] *= xi;
      }
#pragma unroll
      for (int b = 0; b <= d; ++b) {
        auto add = [&](int k, double v) { S[k - LO] = fma(v, m[b], S[k - LO]); };
        if constexpr (TIP) {
#pragma unroll
          for (int k = J0; k < J1; ++k) add(k * RI::NR + RI::r(d - b, b), J[k]);
        } else {
          if (P1 && d <= MI::D) add(MI::w(d - b, b), w);
          if (P1 && d >= 1 && d <= MI::D + 1) add(MI::ax(d - b, b), A);
          if (P2 && d >= 2 && !(d == 2 && b == 1)) add(MI::bx(d - b, b), B);
          if (P2 && d <= MI::D) add(MI::cx(d - b + 1, b + 1), C);
        }
      }
    }
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < HI - LO; ++k) S[k] += __shfl_xor_sync(0xffffffffu, S[k], o);
  if (mine && sub == 0) {
    const int64_t np = a.g1 - a.g0;
#pragma unroll
    for (int k = 0; k < HI - LO; ++k) a.mom[(LO + k) * np + slot] = S[k];
  }
}

// blockIdx.y: the part (cubic basis), then the kind of points (only launched with creases).
template <int ORDER, int L>
__global__ void __launch_bounds__(64) rkpm_moment_kernel(RkpmArgs a) {
  if constexpr (ORDER < 3) {
    if (blockIdx.y == 0) moment_sums<ORDER, 0, L, false>(a);
    else moment_sums<ORDER, 0, L, true>(a);
  } else {
    switch (blockIdx.y) {
      case 0: moment_sums<ORDER, 1, L, false>(a); break;
      case 1: moment_sums<ORDER, 2, L, false>(a); break;
      case 2: moment_sums<ORDER, 1, L, true>(a); break;
      default: moment_sums<ORDER, 2, L, true>(a); break;
    }
  }
}

template <int ORDER, bool PAIR>
__global__ void __launch_bounds__(64) rkpm_solve_kernel(RkpmArgs a) {
  constexpr int NP = (ORDER + 1) * (ORDER + 2) / 2;
  using MI = MomIdx<ORDER>;
  using RI = RawIdx<ORDER>;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.g1 - a.g0) return;
  const int g = a.order[a.g0 + t], at = g - a.g0;
  const bool tip = a.tip[g];
  const int64_t np = a.g1 - a.g0;
  const double* mom = a.mom + t;
  RowJets<ORDER> R;
  a.bad[g] = static_cast<int8_t>(point_solve<ORDER>([&](int q, int aa, int bb) {
    const int k = q == 0 ? MI::w(aa, bb) : q == 1 ? MI::ax(aa + 1, bb) : q == 2 ? MI::ax(aa, bb + 1)
                : q == 3 ? MI::bx(aa + 2, bb) : q == 4 ? MI::bx(aa, bb + 2) : MI::cx(aa + 1, bb + 1);
    return mom[(tip ? q * RI::NR + RI::r(aa, bb) : k) * np];
  }, R));
  auto put = [&](int i, double v) {   // PAIR: as FP32 pairs, in the same 8 bytes
    if constexpr (PAIR) {
      const fp2 p = fp2_from_double(v);
      reinterpret_cast<float2*>(a.coef)[static_cast<int64_t>(at) * 6 * NP + i] = make_float2(p.hi, p.lo);
    } else {
      a.coef[static_cast<int64_t>(at) * 6 * NP + i] = v;
    }
  };
  const double r1 = a.ir, r2 = a.ir * a.ir;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    put(i, R.c0[i]);
    put(NP + i, r1 * R.c0x[i]);
    put(2 * NP + i, r1 * R.c0y[i]);
    put(3 * NP + i, r2 * R.c0xx[i]);
    put(4 * NP + i, r2 * R.c0yy[i]);
    put(5 * NP + i, r2 * R.c0xy[i]);
  }
}

constexpr int kValueThreads = 256;

template <int ORDER>
__global__ void __launch_bounds__(kValueThreads) rkpm_value_kernel(RkpmArgs a) {
  constexpr int NP = (ORDER + 1) * (ORDER + 2) / 2;
  using RI = RawIdx<ORDER>;
  const int64_t e0 = a.ptr[a.g0], e1 = a.ptr[a.g1];
  const int64_t e = e0 + static_cast<int64_t>(blockIdx.x) * kValueThreads + threadIdx.x;
  if (e0 + static_cast<int64_t>(blockIdx.x) * kValueThreads + (threadIdx.x & ~31) >= e1) return;   // the whole warp
  const int g = point_of(a.ptr, a.g0, a.g1, e, e1);
  if (e >= e1) return;
  const int j = a.idx[e];
  const double x = (a.gp_xy[2 * g] - a.node_xy[2 * j]) * a.ir, y = (a.gp_xy[2 * g + 1] - a.node_xy[2 * j + 1]) * a.ir;
  const double w = a.psi[e], r2 = a.ir * a.ir;
  double Jx = a.dpsi[2 * e], Jy = a.dpsi[2 * e + 1], Jxx = a.ddpsi[3 * e], Jyy = a.ddpsi[3 * e + 1], Jxy = a.ddpsi[3 * e + 2];
  if (!a.tip[g]) { Jy = Jx * y; Jx *= x; Jyy = Jxx * (y * y); Jxx *= x * x; }
  const double* c = a.coef + static_cast<int64_t>(g - a.g0) * 6 * NP;
  double m[NP];
  m[0] = 1.0;
#pragma unroll
  for (int i = 1; i < NP; ++i) m[i] = RI::by(i) == 0 ? m[RI::r(RI::bx(i) - 1, 0)] * x : m[RI::r(RI::bx(i), RI::by(i) - 1)] * y;
  double v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    v[k] = __ldg(c + k * NP);
#pragma unroll
    for (int i = 1; i < NP; ++i) v[k] = fma(__ldg(c + k * NP + i), m[i], v[k]);
  }
  const double C2 = v[0] * r2;
  Jx *= a.ir; Jy *= a.ir;
  a.psi[e] = v[0] * w;
  a.dpsi[2 * e] = fma(v[1], w, v[0] * Jx);
  a.dpsi[2 * e + 1] = fma(v[2], w, v[0] * Jy);
  a.ddpsi[3 * e] = fma(v[3], w, fma(2.0 * v[1], Jx, C2 * Jxx));
  a.ddpsi[3 * e + 1] = fma(v[4], w, fma(2.0 * v[2], Jy, C2 * Jyy));
  a.ddpsi[3 * e + 2] = fma(v[5], w, fma(v[1], Jy, fma(v[2], Jx, C2 * Jxy)));
}

// ---- mixed precision: the per-neighbour work in FP32 pairs ----------------------------
//
// The FP64 kernels spend about 200 FP64 operations per neighbour, and GB300 issues FP64 at 1/62 of
// the FP32 rate. The mixed kernels do that per-neighbour arithmetic in FP32 pairs (cgb_pair.cuh,
// about 48 significant bits) on the FP32 pipe, conversions to and from doubles on the bits; only
// point_solve, 1/n of the work, is FP64, as in the FP64 path. 1,000,000 points of 28 neighbours,
// quadratic: RKPM 5.8 ms (jets 0.8, moments 2.3, solve 1.5, values 1.2); 7.1 ms with the FP64
// pipe's conversions, the jets of M in the solve and a bisection in each warp of the pair
// kernels.
//
// Coordinates: node and point coordinates are split into three floats each (72 bits, so
// the split of a double is exact) and differenced in pairs, so xi = (x - x_I) / rho is
// accurate to the pair precision relative to xi itself, not to the coordinates' size.

__device__ __forceinline__ void split3(double v, float& a, float& b, float& c) {
  a = __double2float_rn(v);
  const double r = v - static_cast<double>(a);
  b = __double2float_rn(r);
  c = __double2float_rn(r - static_cast<double>(b));
}

// Per node: {x0, x1, x2, y0}, {y1, y2, fac.hi, fac.lo} with x = x0 + x1 + x2 and
// fac = rho / rho_I (1 for the single radius).
__global__ void node_pair_kernel(int n_nodes, const double* __restrict__ node_xy,
                                 const double* __restrict__ rho_node, double rho, float4* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_nodes) return;
  float x0, x1, x2, y0, y1, y2;
  split3(node_xy[2 * j], x0, x1, x2);
  split3(node_xy[2 * j + 1], y0, y1, y2);
  const fp2 fac = rho_node ? fp2_from_double(rho / rho_node[j]) : fp2{1.0f, 0.0f};
  out[2 * j] = make_float4(x0, x1, x2, y0);
  out[2 * j + 1] = make_float4(y1, y2, fac.hi, fac.lo);
}

// (a0 + a1 + a2) - (b0 + b1 + b2) as a pair.
__device__ __forceinline__ fp2 diff3(float a0, float a1, float a2, float b0, float b1, float b2) {
  const fp2 h = fp2_two_sum(a0, -b0);
  const fp2 m = fp2_two_sum(a1, -b1);
  return fp2_add_exact(h, m) + __fsub_rn(a2, b2);
}

constexpr float kTwoThirdsHi = static_cast<float>(2.0 / 3.0);
constexpr float kTwoThirdsLo = static_cast<float>(2.0 / 3.0 - static_cast<double>(kTwoThirdsHi));
constexpr float kFourThirdsHi = static_cast<float>(4.0 / 3.0);
constexpr float kFourThirdsLo = static_cast<float>(4.0 / 3.0 - static_cast<double>(kFourThirdsHi));

// radial() in pairs, same branches and cut-offs; z2 = s^2 of the scaled differences. The window takes
// s^2 from s: near s = 1 its terms cancel, and so do the errors of s in them when s^2 has the same.
__device__ __forceinline__ void radial_pair(int kernel, fp2 z2, fp2& w, fp2& A, fp2& B, fp2& C) {
  const fp2 z{0.0f, 0.0f};
  const fp2 s = fp2_sqrt(z2);
  if (fp2_ge(s, 1.0f)) { w = z; A = z; B = z; C = z; return; }
  const bool at_node = fp2_is_zero(s);
  const fp2 is2 = at_node ? z : fp2_recip(z2);
  fp2 ds, dd;
  if (kernel == 0) {  // 1 - 6 s^2 + 8 s^3 - 3 s^4
    w = 1.0f + fp2_sqr(s) * (-6.0f + s * (8.0f - 3.0f * s));
    ds = -12.0f + s * (24.0f - 12.0f * s);
    dd = -12.0f + s * (48.0f - 36.0f * s);
  } else if (fp2_le(s, 0.5f)) {  // 2/3 - 4 s^2 + 4 s^3
    w = fp2{kTwoThirdsHi, kTwoThirdsLo} + fp2_sqr(s) * (-4.0f + 4.0f * s);
    ds = -8.0f + 12.0f * s;
    dd = -8.0f + 24.0f * s;
  } else {  // 4/3 (1 - s)^3
    const fp2 r = 1.0f - s;
    const fp2 r2 = fp2_sqr(r);
    w = fp2{kFourThirdsHi, kFourThirdsLo} * (r2 * r);
    ds = -4.0f * (r2 * (s * is2));
    dd = 8.0f * r;
  }
  if (s.hi < 1e-14f) ds = z;
  A = ds;
  B = (dd + ds) * is2;
  C = (dd - ds) * is2;
}

// Point records of the mixed kernels: the coordinates split in three floats each (two float4), then
// per crease the six indicators scaled for the visibility product, as pairs: 0.5 I_f, 0.5 I_gx rho,
// 0.5 I_gy rho, 0.5 I_hxx rho^2, 0.5 I_hyy rho^2, 0.5 I_hxy rho^2. They are made once per point: the
// splits and roundings of doubles issue on the FP64 pipe.
__host__ __device__ constexpr int pair_record_floats(int n_creases) { return 8 + 12 * n_creases; }

__global__ void point_pair_kernel(RkpmArgs a, float* __restrict__ rec) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= a.n_gp) return;
  float x0, x1, x2, y0, y1, y2;
  split3(a.gp_xy[2 * g], x0, x1, x2);
  split3(a.gp_xy[2 * g + 1], y0, y1, y2);
  float* o = rec + static_cast<int64_t>(g) * pair_record_floats(a.n_creases);
  reinterpret_cast<float4*>(o)[0] = make_float4(x0, x1, x2, y0);
  reinterpret_cast<float4*>(o)[1] = make_float4(y1, y2, 0.0f, 0.0f);
  for (int c = 0; c < a.n_creases; ++c) {
    const double* I = a.gind + (static_cast<int64_t>(g) * a.n_creases + c) * 6;
    const double r1 = 0.5 * a.rho, r2 = r1 * a.rho;
    for (int q = 0; q < 6; ++q) {
      const fp2 v = fp2_from_double((q == 0 ? 0.5 : q < 3 ? r1 : r2) * I[q]);
      o[8 + 12 * c + 2 * q] = v.hi;
      o[9 + 12 * c + 2 * q] = v.lo;
    }
  }
}

// Scaled differences of a pair from the split coordinates: accurate relative to themselves.
__device__ __forceinline__ void pair_xi(const RkpmArgs& a, float4 p0, float4 p1, float4 n0, float4 n1, fp2& xi, fp2& eta) {
  xi = diff3(p0.x, p0.y, p0.z, n0.x, n0.y, n0.z) * a.irho;
  eta = diff3(p0.w, p1.x, p1.y, n0.w, n1.x, n1.y) * a.irho;
}

__device__ __forceinline__ float2 as_float2(fp2 v) { return make_float2(v.hi, v.lo); }
__device__ __forceinline__ fp2 as_fp2(float2 v) { return fp2{v.x, v.y}; }

// The jets of every pair of the chunk, one pair per thread, left in the output arrays as FP32 pairs:
// w, A, -, B, -, C xi eta, or in a cap the six jets.
__global__ void __launch_bounds__(kValueThreads) rkpm_pair_jet_kernel(RkpmArgs a, const float* __restrict__ rec) {
  const int64_t e0 = a.ptr[a.g0], e1 = a.ptr[a.g1];
  const int64_t e = e0 + static_cast<int64_t>(blockIdx.x) * kValueThreads + threadIdx.x;
  if (e0 + static_cast<int64_t>(blockIdx.x) * kValueThreads + (threadIdx.x & ~31) >= e1) return;   // the whole warp
  const int g = point_of(a.ptr, a.g0, a.g1, e, e1);
  if (e >= e1) return;
  const int nc = a.n_creases;
  const float* R = rec + static_cast<int64_t>(g) * pair_record_floats(nc);
  const int j = a.idx[e];
  const float4 n0 = __ldg(a.node_pair + 2 * j), n1 = __ldg(a.node_pair + 2 * j + 1);
  fp2 xi, eta;
  pair_xi(a, *reinterpret_cast<const float4*>(R), *reinterpret_cast<const float4*>(R + 4), n0, n1, xi, eta);
  fp2 z2;
  const fp2 fac{n1.z, n1.w};
  const bool scaled = a.rho_node != nullptr;
  if (scaled) {
    const fp2 zx = xi * fac, zy = eta * fac;
    z2 = fp2_sqr(zx) + fp2_sqr(zy);
  } else {
    z2 = fp2_sqr(xi) + fp2_sqr(eta);
  }
  fp2 w, A, B, C;
  radial_pair(a.kernel, z2, w, A, B, C);
  if (scaled) {
    const fp2 f2 = fp2_sqr(fac), f4 = fp2_sqr(f2);
    A = A * f2; B = B * f4; C = C * f4;
  }
  C = C * (xi * eta);
  float2* o0 = reinterpret_cast<float2*>(a.psi) + e;
  float2* o1 = reinterpret_cast<float2*>(a.dpsi) + 2 * e;
  float2* o2 = reinterpret_cast<float2*>(a.ddpsi) + 3 * e;
  if (a.tip[g]) {
    fp2 J[6] = {w, A * xi, A * eta, B * fp2_sqr(xi), B * fp2_sqr(eta), C};
    for (int c = 0; c < nc; ++c) {   // GlobalRKPM.h:87-112
      const fp2* G = reinterpret_cast<const fp2*>(R + 8 + 12 * c);
      const float sn = a.node_side[static_cast<int64_t>(c) * a.n_nodes + j] > 0 ? 1.0f : -1.0f;
      const fp2 V = G[0] * sn + 0.5f, Vx = G[1] * sn, Vy = G[2] * sn;
      const fp2 o0j = J[0], o1j = J[1], o2j = J[2];
      J[0] = o0j * V;
      J[1] = o1j * V + o0j * Vx;
      J[2] = o2j * V + o0j * Vy;
      J[3] = J[3] * V + 2.0f * (o1j * Vx) + o0j * (G[3] * sn);
      J[4] = J[4] * V + 2.0f * (o2j * Vy) + o0j * (G[4] * sn);
      J[5] = J[5] * V + o1j * Vy + o2j * Vx + o0j * (G[5] * sn);
    }
    o0[0] = as_float2(J[0]); o1[0] = as_float2(J[1]); o1[1] = as_float2(J[2]);
    o2[0] = as_float2(J[3]); o2[1] = as_float2(J[4]); o2[2] = as_float2(J[5]);
  } else {
    float vis = 1.0f;   // exact: the indicator is 1, -1 or (on the crease) 0
    for (int c = 0; c < nc; ++c) {
      const float h = R[8 + 12 * c];
      vis *= 0.5f + (a.node_side[static_cast<int64_t>(c) * a.n_nodes + j] > 0 ? h : -h);
    }
    o0[0] = as_float2(w * vis); o1[0] = as_float2(A * vis);
    o2[0] = as_float2(B * vis); o2[2] = as_float2(C * vis);
  }
}

// The sums of moment_sums from the pairs' jets, accumulated in pairs (Dot2) and rounded to FP64, in
// three parts: W and C, A, B; in a cap two of the six jets each. All sums of a point in one thread (74
// pairs, 206 registers in two parts) left two warps per scheduler to hide the long chains of pair
// arithmetic; forming the monomials three times costs a tenth more instructions.
template <int ORDER, int PART, int L, bool TIP>
__device__ __forceinline__ void pair_moment_sums(const RkpmArgs& a, const float* __restrict__ rec) {
  using MI = MomIdx<ORDER>;
  using RI = RawIdx<ORDER>;
  constexpr int N0 = TIP ? RI::NR : PART == 0 ? MI::NW : PART == 1 ? MI::NA : MI::NB;   // sums of the first factor
  constexpr int N1 = TIP ? RI::NR : PART == 0 ? MI::NC : 0;
  constexpr int AT0 = TIP ? 2 * PART * RI::NR : PART == 0 ? 0 : PART == 1 ? MI::NW : MI::NW + MI::NA;
  constexpr int AT1 = TIP ? (2 * PART + 1) * RI::NR : MI::NW + MI::NA + MI::NB;
  constexpr int DEG = MI::D + (TIP ? 0 : PART);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int slot = t / L, sub = t % L;
  const bool here = slot < a.g1 - a.g0;
  const int gc = a.order[here ? a.g0 + slot : a.g1 - 1];
  const bool mine = here && (a.tip[gc] != 0) == TIP;
  if (!__any_sync(0xffffffffu, mine)) return;
  const int64_t p0 = a.ptr[gc];
  const int n = mine ? static_cast<int>(a.ptr[gc + 1] - p0) : 0;
  const float* R = rec + static_cast<int64_t>(gc) * pair_record_floats(a.n_creases);
  const float4 r0 = *reinterpret_cast<const float4*>(R), r1 = *reinterpret_cast<const float4*>(R + 4);
  // The array of a pair's jet k: psi, dpsi (2), ddpsi (3); w, A, B and C xi eta are jets 0, 1, 3, 5.
  auto jet = [&](int k, int64_t e) {
    const double* p = k == 0 ? a.psi + e : k < 3 ? a.dpsi + 2 * e + (k - 1) : a.ddpsi + 3 * e + (k - 3);
    return as_fp2(*reinterpret_cast<const float2*>(p));
  };
  constexpr int K0 = TIP ? 2 * PART : PART == 0 ? 0 : PART == 1 ? 1 : 3;
  constexpr int K1 = TIP ? 2 * PART + 1 : 5;
  fp2 S0[N0], S1[N1 > 0 ? N1 : 1];
#pragma unroll
  for (int k = 0; k < N0; ++k) S0[k] = fp2{0.0f, 0.0f};
#pragma unroll
  for (int k = 0; k < N1; ++k) S1[k] = fp2{0.0f, 0.0f};
  for (int q = sub; q < n; q += L) {
    const int64_t e = p0 + q;
    const int j = a.idx[e];
    fp2 xi, eta;
    pair_xi(a, r0, r1, __ldg(a.node_pair + 2 * j), __ldg(a.node_pair + 2 * j + 1), xi, eta);
    const fp2 J0 = jet(K0, e), J1 = N1 > 0 ? jet(K1, e) : fp2{0.0f, 0.0f};
    fp2 m[DEG + 1];
    m[0] = fp2{1.0f, 0.0f};
#pragma unroll
    for (int d = 0; d <= DEG; ++d) {
      if (d == 1) { m[1] = eta; m[0] = xi; }
      if (d > 1) {
        m[d] = m[d - 1] * eta;
#pragma unroll
        for (int b = d - 1; b >= 0; --b) m[b] = m[b] * xi;
      }
#pragma unroll
      for (int b = 0; b <= d; ++b) {
        const int x = d - b;
        if (TIP || PART == 0) {
          fp2_fma_acc(S0[RI::r(x, b)], J0, m[b]);
          if (N1 > 0) fp2_fma_acc(S1[RI::r(x, b)], J1, m[b]);
        } else if (PART == 1) {
          if (d >= 1) fp2_fma_acc(S0[MI::ax(x, b) - AT0], J0, m[b]);
        } else if (d >= 2 && !(d == 2 && b == 1)) {
          fp2_fma_acc(S0[MI::bx(x, b) - AT0], J0, m[b]);
        }
      }
    }
  }
  const int64_t np = a.g1 - a.g0;
  auto put = [&](int at, const auto& S) {
    constexpr int N = sizeof(S) / sizeof(S[0]);
    double v[N];
    fp2_to_double(S, v);
#pragma unroll
    for (int k = 0; k < N; ++k) {
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      if (mine && sub == 0) a.mom[(at + k) * np + slot] = v[k];
    }
  };
  put(AT0, S0);
  if constexpr (N1 > 0) put(AT1, S1);
}

// blockIdx.y: the part, then the kind of points (only launched with creases).
template <int ORDER, int L>
__global__ void __launch_bounds__(64, ORDER < 3 ? 8 : 4) rkpm_pair_moment_kernel(RkpmArgs a, const float* __restrict__ rec) {
  switch (blockIdx.y) {
    case 0: pair_moment_sums<ORDER, 0, L, false>(a, rec); break;
    case 1: pair_moment_sums<ORDER, 1, L, false>(a, rec); break;
    case 2: pair_moment_sums<ORDER, 2, L, false>(a, rec); break;
    case 3: pair_moment_sums<ORDER, 0, L, true>(a, rec); break;
    case 4: pair_moment_sums<ORDER, 1, L, true>(a, rec); break;
    default: pair_moment_sums<ORDER, 2, L, true>(a, rec); break;
  }
}

// rkpm_value_kernel in pairs; the polynomials come as pairs too.
template <int ORDER>
__global__ void __launch_bounds__(kValueThreads) rkpm_pair_value_kernel(RkpmArgs a, const float* __restrict__ rec) {
  constexpr int NP = (ORDER + 1) * (ORDER + 2) / 2;
  using RI = RawIdx<ORDER>;
  const int64_t e0 = a.ptr[a.g0], e1 = a.ptr[a.g1];
  const int64_t e = e0 + static_cast<int64_t>(blockIdx.x) * kValueThreads + threadIdx.x;
  if (e0 + static_cast<int64_t>(blockIdx.x) * kValueThreads + (threadIdx.x & ~31) >= e1) return;   // the whole warp
  const int g = point_of(a.ptr, a.g0, a.g1, e, e1);
  if (e >= e1) return;
  const float* R = rec + static_cast<int64_t>(g) * pair_record_floats(a.n_creases);
  const int j = a.idx[e];
  fp2 x, y;
  pair_xi(a, *reinterpret_cast<const float4*>(R), *reinterpret_cast<const float4*>(R + 4),
          __ldg(a.node_pair + 2 * j), __ldg(a.node_pair + 2 * j + 1), x, y);
  const float2* i1 = reinterpret_cast<const float2*>(a.dpsi) + 2 * e;
  const float2* i2 = reinterpret_cast<const float2*>(a.ddpsi) + 3 * e;
  const fp2 w = as_fp2(reinterpret_cast<const float2*>(a.psi)[e]);
  fp2 Jx = as_fp2(i1[0]), Jxx = as_fp2(i2[0]), Jy, Jyy;
  const fp2 Jxy = as_fp2(i2[2]);
  if (a.tip[g]) {
    Jy = as_fp2(i1[1]);
    Jyy = as_fp2(i2[1]);
  } else {
    Jy = Jx * y; Jx = Jx * x;
    Jyy = Jxx * fp2_sqr(y); Jxx = Jxx * fp2_sqr(x);
  }
  Jx = Jx * a.irho;
  Jy = Jy * a.irho;
  fp2 m[NP];
#pragma unroll
  for (int i = 1; i < NP; ++i) {
    if (i == 1) m[i] = x;
    else if (i == 2) m[i] = y;
    else m[i] = RI::by(i) == 0 ? m[RI::r(RI::bx(i) - 1, 0)] * x : m[RI::r(RI::bx(i), RI::by(i) - 1)] * y;
  }
  const float2* c = reinterpret_cast<const float2*>(a.coef) + static_cast<int64_t>(g - a.g0) * 6 * NP;
  fp2 v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    v[k] = as_fp2(__ldg(c + k * NP));
#pragma unroll
    for (int i = 1; i < NP; ++i) fp2_fma_acc(v[k], as_fp2(__ldg(c + k * NP + i)), m[i]);
    v[k] = fp2_norm(v[k]);
  }
  const fp2 C2 = v[0] * a.irho2, vx2 = v[1] * 2.0f, vy2 = v[2] * 2.0f;
  fp2 r[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) r[k] = v[k] * w;
  fp2_fma_acc(r[1], v[0], Jx);
  fp2_fma_acc(r[2], v[0], Jy);
  fp2_fma_acc(r[3], vx2, Jx); fp2_fma_acc(r[3], C2, Jxx);
  fp2_fma_acc(r[4], vy2, Jy); fp2_fma_acc(r[4], C2, Jyy);
  fp2_fma_acc(r[5], v[1], Jy); fp2_fma_acc(r[5], v[2], Jx); fp2_fma_acc(r[5], C2, Jxy);
  double out[6];
  fp2_to_double(r, out);
  a.psi[e] = out[0];
  a.dpsi[2 * e] = out[1]; a.dpsi[2 * e + 1] = out[2];
  a.ddpsi[3 * e] = out[3]; a.ddpsi[3 * e + 1] = out[4]; a.ddpsi[3 * e + 2] = out[5];
}

// The RKPM of a set: moments, solve, values over chunks of points that bound the scratch (the
// sums and polynomials of 1,048,576 points: 1.1 GB for the quadratic basis, 1.9 GB for the cubic).
// A chunk's kernels each end in a part-filled wave: with 262,144 points to a chunk 1,000,000 mixed
// points take 7.18 ms, not 6.87, and 300,000 FP64 points 4.94, not 4.85.
// Lanes per point of the moment kernel: more while its warps do not fill the SM quarters twice
// (adding a lane pair's sums costs as many operations as half a neighbour's).
// Returns the kernels launched.
template <int ORDER, bool PAIR>
int rkpm(cgb_context* ctx, cgb_shape* out, RkpmArgs ra, const float* rec) {
  constexpr int kChunk = 1 << 20, kLeastChunk = 1 << 15, NP = (ORDER + 1) * (ORDER + 2) / 2;
  constexpr int kSums = std::max(MomIdx<ORDER>::N, 6 * RawIdx<ORDER>::NR);
  constexpr int kParts = PAIR ? 3 : ORDER == 3 ? 2 : 1;
  cudaStream_t st = ctx->stream;
  const int n_gp = out->n_gp;
  int chunk = kChunk;
  int launches = 1;
  ctx->scratch.tip.ensure(n_gp);
  ctx->scratch.order.ensure(n_gp);
  ra.tip = ctx->scratch.tip.p;
  ra.order = ctx->scratch.order.p;
  point_order_kernel<<<blocks_for(n_gp, kSortPoints), kSortPoints, 0, st>>>(ra);
  for (;;) {   // half the points at a time where the scratch finds no room
    const size_t most = std::min(n_gp, chunk);
    try {
      ctx->scratch.mom.ensure(most * kSums);
      ctx->scratch.coef.ensure(most * 6 * NP);
      break;
    } catch (const OutOfMemory&) {
      if (most <= kLeastChunk) throw;
      while (chunk >= static_cast<int>(most)) chunk /= 2;
      ctx->scratch.mom.reset();
      ctx->scratch.coef.reset();
    }
  }
  ra.mom = ctx->scratch.mom.p;
  ra.coef = ctx->scratch.coef.p;
  int sms = 0;
  CGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  for (int g0 = 0; g0 < n_gp; g0 += chunk) {
    ra.g0 = g0;
    ra.g1 = std::min(n_gp, g0 + chunk);
    const int np = ra.g1 - g0;
    const int64_t pairs = std::min(out->nnz, static_cast<int64_t>(np) * out->max_n);
    const unsigned vb = blocks_for(std::max<int64_t>(pairs, 1), kValueThreads);
    if constexpr (PAIR) rkpm_pair_jet_kernel<<<vb, kValueThreads, 0, st>>>(ra, rec);
    const int64_t full = 2LL * 4 * 32 * sms;   // lanes of two warps per SM quarter
    auto moments = [&](auto lanes) {
      constexpr int L = decltype(lanes)::value;
      const dim3 grid(blocks_for(static_cast<int64_t>(np) * L, 64), kParts * (ra.n_creases > 0 ? 2 : 1));
      if constexpr (PAIR) rkpm_pair_moment_kernel<ORDER, L><<<grid, 64, 0, st>>>(ra, rec);
      else rkpm_moment_kernel<ORDER, L><<<grid, 64, 0, st>>>(ra);
    };
    if (np * 8LL <= full) moments(std::integral_constant<int, 8>{});
    else if (np * 2LL <= full) moments(std::integral_constant<int, 2>{});
    else moments(std::integral_constant<int, 1>{});
    rkpm_solve_kernel<ORDER, PAIR><<<blocks_for(np, 64), 64, 0, st>>>(ra);
    if constexpr (PAIR) rkpm_pair_value_kernel<ORDER><<<vb, kValueThreads, 0, st>>>(ra, rec);
    else rkpm_value_kernel<ORDER><<<vb, kValueThreads, 0, st>>>(ra);
    launches += PAIR ? 4 : 3;
  }
  CGB_CUDA(cudaGetLastError());
  return launches;
}

}  // namespace

void shape_values(cgb_context* ctx, cgb_shape* out, const std::vector<Crease>& creases);

namespace {
// A build's or rebuild's hold on the context's scratch, until its kernels have ended (however the call ends).
struct ScratchUse {
  cgb_context* ctx;
  explicit ScratchUse(cgb_context* c) : ctx(c) { ctx->scratch.busy = true; }
  ~ScratchUse() {
    cudaStreamSynchronize(ctx->stream);
    ctx->scratch.busy = false;
    ctx->scratch.drop_large();
  }
};
}  // namespace

void shape_build(cgb_context* ctx, const double* gp_xy, int n_gp, const cgb_shape_params& prm,
                 const std::vector<Crease>& creases, cgb_shape* out) {
  cudaStream_t st = ctx->stream;
  const int n_nodes = ctx->n_nodes;
  if (n_nodes <= 0) throw Error(CGB_ERR_INVALID, "cgb_shape_build: nodes not set (cgb_set_nodes)");
  if (n_gp < 0) throw Error(CGB_ERR_INVALID, "cgb_shape_build: n_gp < 0");
  if (prm.order < 1 || prm.order > 3)
    throw Error(CGB_ERR_INVALID, "cgb_shape_build: order must be 1, 2 or 3");
  if (!(prm.rho > 0.0)) throw Error(CGB_ERR_INVALID, "cgb_shape_build: rho must be > 0");
  out->ctx = ctx;
  out->n_gp = n_gp;
  out->rho = prm.rho;
  out->order = prm.order;
  out->kernel = prm.kernel;
  if (prm.precision != CGB_SHAPE_FP64 && prm.precision != CGB_SHAPE_MIXED)
    throw Error(CGB_ERR_INVALID, "cgb_shape_build: precision must be CGB_SHAPE_FP64 or CGB_SHAPE_MIXED");
  out->precision = prm.precision;
  out->node_gen = ctx->node_gen;

  // ---- node cell grid (FRNN.h:33-44) ----
  const ScratchUse use(ctx);
  ShapeScratch& w = ctx->scratch;
  double cell = prm.rho;
  if (prm.rho_node) {
    cell = 0.0;
    for (int i = 0; i < n_nodes; ++i) {
      if (!(prm.rho_node[i] > 0.0)) throw Error(CGB_ERR_INVALID, "cgb_shape_build: rho_node must be > 0");
      cell = std::max(cell, prm.rho_node[i]);
    }
  }
  const double minx = ctx->node_min[0], miny = ctx->node_min[1], maxx = ctx->node_max[0], maxy = ctx->node_max[1];
  const double cells_x = std::ceil((maxx - minx) / cell), cells_y = std::floor((maxy - miny) / cell);
  // The grid ends with the largest key; a bound on it decides except beside the limit itself.
  constexpr double kMostCells = static_cast<double>(1LL << 28);
  bool fits = cells_x < kMostCells && cells_y < kMostCells && cells_y * (cells_x + 1.0) + 1.0 <= kMostCells;
  const int cols = fits ? static_cast<int>(cells_x) + 1 : 1;
  long long ncells = fits ? (static_cast<long long>(cells_y) + 1) * cols : 0;
  if (ncells > (1LL << 28)) {
    ncells = 0;
    for (int i = 0; i < n_nodes; ++i) {
      const double* q = ctx->h_node_xy.data() + 2 * static_cast<size_t>(i);
      ncells = std::max(ncells, static_cast<long long>(std::floor((q[1] - miny) / cell)) * cols +
                                    static_cast<long long>(std::floor((q[0] - minx) / cell)) + 1);
    }
    fits = ncells <= (1LL << 28);
  }
  if (!fits)
    throw Error(CGB_ERR_CAPACITY, "cgb_shape_build: the node cell grid exceeds 2^28 cells (rho too small for the node extent)");
  out->has_rho_node = prm.rho_node != nullptr;
  if (prm.rho_node) upload(out->rho_node, prm.rho_node, n_nodes, st);
  const double* d_rn = prm.rho_node ? out->rho_node.p : nullptr;
  w.cell_start.ensure(static_cast<size_t>(ncells) + 1);
  w.cell_cursor.ensure(static_cast<size_t>(ncells) + 1);
  w.cell_count.ensure(static_cast<size_t>(ncells));
  w.node_key.ensure(n_nodes);
  w.node_list.ensure(n_nodes);
  w.cell_nodes.ensure(n_nodes);
  w.cell32.ensure(n_nodes);
  w.totals.ensure(4);
  if (d_rn) w.r2c32.ensure(n_nodes);
  const GridDev G{minx, miny, cell, cols, ncells, w.cell_start.p, w.cell_nodes.p};
  prof_begin(ctx, CGB_PHASE_FRNN);
  CGB_CUDA(cudaMemsetAsync(w.cell_count.p, 0, static_cast<size_t>(ncells) * sizeof(int32_t), st));
  cell_count_kernel<<<blocks_for(n_nodes), kThreads, 0, st>>>(n_nodes, ctx->node_xy.p, G, w.node_key.p, w.cell_count.p);
  scan_counts(ctx, ncells, w.cell_count.p, w.cell_start.p, w.totals.p + 2);
  CGB_CUDA(cudaMemcpyAsync(w.cell_cursor.p, w.cell_start.p, static_cast<size_t>(ncells) * sizeof(int64_t),
                           cudaMemcpyDeviceToDevice, st));
  cell_fill_kernel<<<blocks_for(n_nodes), kThreads, 0, st>>>(n_nodes, w.node_key.p, w.cell_cursor.p, w.node_list.p);
  cell_sort_kernel<<<blocks_for(n_nodes), kThreads, 0, st>>>(n_nodes, ctx->node_xy.p, d_rn, G, w.node_key.p,
                                                               w.node_list.p, w.cell_nodes.p, w.cell32.p,
                                                               d_rn ? w.r2c32.p : nullptr);
  CGB_CUDA(cudaGetLastError());
  prof_end(ctx, CGB_PHASE_FRNN, 6);

  upload(out->gp_xy, gp_xy, 2 * static_cast<size_t>(n_gp), st);
  out->has_xy = true;
  const double rho2 = prm.rho * prm.rho;
  // The FP32 pre-test (FrnnPre): float coordinates relative to (minx, miny) and the margin.
  // e = 2^-23 X (X the largest relative coordinate) bounds the rounding of one coordinate
  // with room to spare; c = cell = the largest radius. A candidate at distance d >= 2c (the
  // wrapped cell keys can bring far nodes) is outside under both tests: its float distance
  // is off by a relative 2^-22 at most, far above r^2 + margin. Every other candidate has
  // |dx|, |dy| < 2c and d^2 < 8 c^2; its float differences are off by eps <= 2e + 2^-24 2c
  // each, so the float d^2 is off by <= 2 (|dx| + |dy|) eps + 2 eps^2 <= 16 c e + 8 e^2 +
  // 2^-20 c^2 (+ lower order), its arithmetic by <= 2 ulp(8 c^2) = 2^-20 c^2 and the float
  // radius by <= 2^-24 c^2: below 16 c e + 8 e^2 + 64 2^-24 c^2.
  // X may be taken over the node box widened by two cells: a point farther out is more than
  // 2c from every node, truly outside, and its float distance (off by a relative 2^-23) stays
  // above 4 c^2 (1 - 2^-22)^2 > r^2 + margin, so it is classified outside too.
  const double ext = std::max(maxx - minx, maxy - miny) + 2.0 * cell;
  const double e = std::ldexp(ext, -23), fu = std::ldexp(1.0, -24);
  const double margin = 16.0 * cell * e + 8.0 * e * e + 64.0 * fu * cell * cell;
  const FrnnPre pre{w.cell32.p, d_rn ? w.r2c32.p : nullptr, static_cast<float>(rho2), static_cast<float>(margin)};
  out->nbr_ptr.alloc(static_cast<size_t>(n_gp) + 1);
  int64_t totals[2] = {0, 0};
  if (n_gp > 0) {
    w.gp_count.ensure(n_gp);
    w.gp_mask.ensure(static_cast<size_t>(n_gp) * kMaskWords);
    prof_begin(ctx, CGB_PHASE_FRNN);
    frnn_kernel<<<blocks_for(n_gp), kThreads, 0, st>>>(n_gp, out->gp_xy.p, ctx->node_xy.p, d_rn, rho2, G, pre,
                                                        nullptr, w.gp_count.p, w.gp_mask.p, nullptr);
    // CSR offsets on the device; only the total and the largest count come back.
    scan_counts(ctx, n_gp, w.gp_count.p, out->nbr_ptr.p, w.totals.p);
    prof_end(ctx, CGB_PHASE_FRNN, 4);
    CGB_CUDA(cudaMemcpyAsync(totals, w.totals.p, sizeof(totals), cudaMemcpyDeviceToHost, st));
    CGB_CUDA(cudaStreamSynchronize(st));
  } else {
    CGB_CUDA(cudaMemsetAsync(out->nbr_ptr.p, 0, sizeof(int64_t), st));
  }
  const int64_t nnz = totals[0];
  auto drop_grid = [&] {   // a sparse grid of many cells is not kept
    if (ncells <= (1LL << 24)) return;
    CGB_CUDA(cudaStreamSynchronize(st));
    w.cell_start.reset();
    w.cell_cursor.reset();
    w.cell_count.reset();
  };
  if (nnz >= (1LL << 31)) throw Error(CGB_ERR_CAPACITY, "cgb_shape_build: more than 2^31 neighbour entries");
  out->nnz = nnz;
  out->max_n = static_cast<int>(totals[1]);
  out->nbr_idx.alloc(nnz);
  // The mixed RKPM recomputes distances in FP32 pairs and does not read s, so a mixed set
  // leaves s out; cgb_shape_download computes it on demand (shape_distances), bitwise equal.
  const bool want_s = prm.precision != CGB_SHAPE_MIXED;
  if (want_s) out->s.alloc(nnz); else out->s.reset();
  prof_begin(ctx, CGB_PHASE_FRNN);
  if (n_gp > 0)
    frnn_kernel<<<blocks_for(n_gp), kThreads, 0, st>>>(n_gp, out->gp_xy.p, ctx->node_xy.p, d_rn, rho2, G, pre,
                                                        out->nbr_ptr.p, nullptr, w.gp_mask.p, out->nbr_idx.p);
  if (want_s && nnz > 0)
    distance_kernel<<<blocks_for(nnz, 256), 256, 0, st>>>(n_gp, out->gp_xy.p, ctx->node_xy.p, d_rn, prm.rho,
                                                          out->nbr_ptr.p, out->nbr_idx.p, nnz, out->s.p);
  prof_end(ctx, CGB_PHASE_FRNN, (n_gp > 0 ? 1 : 0) + (want_s && nnz > 0 ? 1 : 0));
  CGB_CUDA(cudaGetLastError());

  drop_grid();
  out->rebuildable = true;
  shape_values(ctx, out, creases);
}

// Crease indicators, RKPM and the reference's guards for the points and neighbour lists
// already in `out` (SetupHelper::recomputeShapeFunctions after the FRNN). The value
// arrays keep their allocation when they have one, so device pointers handed out
// earlier (assemblers, captured graphs) stay valid across rebuilds.
void shape_values(cgb_context* ctx, cgb_shape* out, const std::vector<Crease>& creases) {
  cudaStream_t st = ctx->stream;
  const int n_nodes = ctx->n_nodes;
  const int n_gp = out->n_gp;
  const int64_t nnz = out->nnz;
  const int nc = static_cast<int>(creases.size());
  std::vector<double> all_xy;
  std::vector<size_t> off(nc + 1, 0);
  for (int c = 0; c < nc; ++c) {
    all_xy.insert(all_xy.end(), creases[c].xy.begin(), creases[c].xy.end());
    off[c + 1] = all_xy.size();
  }
  ctx->scratch.cxy.ensure(std::max<size_t>(all_xy.size(), 1));
  ctx->scratch.cxyf.ensure(std::max<size_t>(all_xy.size() / 2, 1));
  std::vector<float2> all_f(all_xy.size() / 2);
  std::vector<float> extent(nc, 0.0f);
  for (int c = 0; c < nc; ++c)
    for (size_t v = off[c]; v < off[c + 1]; v += 2) {
      const float2 f = make_float2(static_cast<float>(all_xy[v] - all_xy[off[c]]),
                                   static_cast<float>(all_xy[v + 1] - all_xy[off[c] + 1]));
      all_f[v / 2] = f;
      extent[c] = std::max(extent[c], std::max(std::fabs(f.x), std::fabs(f.y)));
    }
  ctx->scratch.side.ensure(static_cast<size_t>(std::max(nc, 1)) * n_nodes);
  ctx->scratch.gind.ensure(static_cast<size_t>(std::max(nc, 1)) * 6 * std::max(n_gp, 1));
  ctx->scratch.bad.ensure(std::max(n_gp, 1));
  if (!all_xy.empty())
    CGB_CUDA(cudaMemcpyAsync(ctx->scratch.cxy.p, all_xy.data(), all_xy.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  if (!all_f.empty())
    CGB_CUDA(cudaMemcpyAsync(ctx->scratch.cxyf.p, all_f.data(), all_f.size() * sizeof(float2), cudaMemcpyHostToDevice, st));
  int8_t* side = ctx->scratch.side.p;
  double* gind = ctx->scratch.gind.p;
  std::vector<DevCrease> dcr(nc);
  int sms = 0;
  CGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  prof_begin(ctx, CGB_PHASE_CREASE);
  for (int c = 0; c < nc; ++c) {
    dcr[c] = DevCrease{ctx->scratch.cxy.p + off[c], static_cast<int>(creases[c].xy.size() / 2), creases[c].extend_start,
                       creases[c].extend_end, creases[c].is_closed, ctx->scratch.cxyf.p + off[c] / 2, extent[c]};
    indicator_lanes(n_nodes, sms, [&](auto lanes) {
      constexpr int L = decltype(lanes)::value;
      node_side_kernel<L><<<blocks_for(static_cast<int64_t>(n_nodes) * L, 32), 32, 0, st>>>(
          n_nodes, ctx->node_xy.p, dcr[c], side + static_cast<int64_t>(c) * n_nodes);
    });
  }
  // Gauss-point indicators laid out [g][c][6].
  if (nc > 0 && n_gp > 0)
    for (int c = 0; c < nc; ++c)
      indicator_lanes(n_gp, sms, [&](auto lanes) {
        constexpr int L = decltype(lanes)::value;
        gp_indicator_kernel<L><<<blocks_for(static_cast<int64_t>(n_gp) * L, 64), 64, 0, st>>>(n_gp, out->gp_xy.p, dcr[c],
                                                                                             c, nc, gind);
      });
  prof_end(ctx, CGB_PHASE_CREASE, nc * (1 + (n_gp > 0 ? 1 : 0)));
  CGB_CUDA(cudaGetLastError());

  // ---- RKPM ----
  if (out->psi.n < static_cast<size_t>(std::max<int64_t>(nnz, 1))) out->psi.alloc(nnz);
  if (out->dpsi.n < static_cast<size_t>(std::max<int64_t>(2 * nnz, 1))) out->dpsi.alloc(2 * nnz);
  if (out->ddpsi.n < static_cast<size_t>(std::max<int64_t>(3 * nnz, 1))) out->ddpsi.alloc(3 * nnz);
  int8_t* bad = ctx->scratch.bad.p;
  const double* d_rn = out->has_rho_node ? out->rho_node.p : nullptr;
  const bool mixed = out->precision == CGB_SHAPE_MIXED;
  auto pair_of = [](double v) {
    const float hi = static_cast<float>(v);
    return fp2{hi, static_cast<float>(v - static_cast<double>(hi))};
  };
  RkpmArgs ra{n_gp, n_nodes, out->kernel, nc, out->rho, nullptr, pair_of(1.0 / out->rho),
              pair_of(1.0 / (out->rho * out->rho)), out->gp_xy.p, ctx->node_xy.p, d_rn, out->nbr_ptr.p,
              out->nbr_idx.p, out->s.p, gind, side, out->psi.p, out->dpsi.p, out->ddpsi.p, bad,
              0.0, nullptr, nullptr, nullptr, nullptr, nullptr, 0, n_gp};
  prof_begin(ctx, CGB_PHASE_RKPM);
  if (mixed && n_nodes > 0) {
    ctx->scratch.node_pair.ensure(2 * static_cast<size_t>(n_nodes));
    node_pair_kernel<<<blocks_for(n_nodes), kThreads, 0, st>>>(n_nodes, ctx->node_xy.p, d_rn, out->rho,
                                                                 ctx->scratch.node_pair.p);
    ra.node_pair = ctx->scratch.node_pair.p;
  }
  int nl = mixed && n_nodes > 0 ? 1 : 0;
  if (n_gp > 0) {
    nl += mixed || d_rn ? 1 : 0;
    ra.ir = 1.0 / out->rho;
    const float* rec = nullptr;
    if (mixed) {
      ctx->scratch.point_rec.ensure(static_cast<size_t>(n_gp) * pair_record_floats(nc));
      point_pair_kernel<<<blocks_for(n_gp), kThreads, 0, st>>>(ra, ctx->scratch.point_rec.p);
      rec = ctx->scratch.point_rec.p;
    } else if (d_rn) {
      ctx->scratch.fac.ensure(n_nodes);
      node_fac_kernel<<<blocks_for(n_nodes), kThreads, 0, st>>>(n_nodes, d_rn, out->rho, ctx->scratch.fac.p);
      ra.fac = ctx->scratch.fac.p;
    }
    switch (out->order) {
      case 1: nl += mixed ? rkpm<1, true>(ctx, out, ra, rec) : rkpm<1, false>(ctx, out, ra, rec); break;
      case 2: nl += mixed ? rkpm<2, true>(ctx, out, ra, rec) : rkpm<2, false>(ctx, out, ra, rec); break;
      default: nl += mixed ? rkpm<3, true>(ctx, out, ra, rec) : rkpm<3, false>(ctx, out, ra, rec); break;
    }
  }
  prof_end(ctx, CGB_PHASE_RKPM, nl);
  CGB_CUDA(cudaGetLastError());
  // The reference's guards (GlobalRKPM.h:241-257 after the 3x3 block, 347-359 after
  // the bordering): singular first, then pivot collapse.
  int found[4] = {0, n_gp, 0, n_gp};
  ctx->scratch.guard.ensure(4);
  CGB_CUDA(cudaMemcpyAsync(ctx->scratch.guard.p, found, sizeof(found), cudaMemcpyHostToDevice, st));
  if (n_gp > 0) guard_kernel<<<blocks_for(n_gp, 256), 256, 0, st>>>(n_gp, bad, ctx->scratch.guard.p);
  CGB_CUDA(cudaGetLastError());
  CGB_CUDA(cudaMemcpyAsync(found, ctx->scratch.guard.p, sizeof(found), cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  const int n1 = found[0], f1 = found[1], n2 = found[2], f2 = found[3];
  auto count_of = [&](size_t g) {
    int64_t pr[2];
    CGB_CUDA(cudaMemcpy(pr, out->nbr_ptr.p + g, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost));
    return pr[1] - pr[0];
  };
  if (n1) {
    throw Error(CGB_ERR_SINGULAR,
                "RKPM: singular moment matrix at " + std::to_string(n1) + " of " + std::to_string(n_gp) +
                    " Gauss points (first is index " + std::to_string(f1) + " with " +
                    std::to_string(count_of(f1)) +
                    " neighbours). The support is rank-deficient for the requested "
                    "basis order - typically too few visible nodes, which happens "
                    "where a crease cuts most of a support away. Increase the support "
                    "radius, refine the mesh there, or lower the order.");
  }
  if (n2) {
    throw Error(CGB_ERR_PIVOT,
                "RKPM: moment-matrix pivot collapsed during block inversion at " + std::to_string(n2) +
                    " of " + std::to_string(n_gp) + " Gauss points (first is index " + std::to_string(f2) +
                    " with " + std::to_string(count_of(f2)) +
                    " neighbours). Same cause and remedies as a singular moment matrix.");
  }
}

void shape_distances(cgb_shape* sh) {
  cgb_context* ctx = sh->ctx;
  // Only sets built here in mixed precision lack s; wrapped or concatenated sets without
  // distances keep returning none, as before.
  if (sh->nnz == 0 || sh->s.n >= static_cast<size_t>(sh->nnz) || !sh->rebuildable) return;
  if (ctx->node_gen != sh->node_gen)
    throw Error(CGB_ERR_INVALID, "cgb_shape_download: s is computed on demand for mixed-precision sets and the "
                                 "nodes changed since the set was built (cgb_set_nodes)");
  sh->s.alloc(sh->nnz);
  distance_kernel<<<blocks_for(sh->nnz, 256), 256, 0, ctx->stream>>>(
      sh->n_gp, sh->gp_xy.p, ctx->node_xy.p, sh->has_rho_node ? sh->rho_node.p : nullptr, sh->rho, sh->nbr_ptr.p,
      sh->nbr_idx.p, sh->nnz, sh->s.p);
  CGB_CUDA(cudaGetLastError());
}

void shape_rebuild(cgb_shape* sh, const std::vector<Crease>& creases) {
  cgb_context* ctx = sh->ctx;
  if (!sh->rebuildable)
    throw Error(CGB_ERR_INVALID, "cgb_shape_rebuild: the set was not made by cgb_shape_build (wrapped or concatenated)");
  if (ctx->node_gen != sh->node_gen)
    throw Error(CGB_ERR_INVALID, "cgb_shape_rebuild: the nodes changed since the set was built (cgb_set_nodes)");
  // The new values stand even when a guard fires, as the reference's arrays do.
  ++sh->version;
  const ScratchUse use(ctx);
  shape_values(ctx, sh, creases);
}

}  // namespace cgb
