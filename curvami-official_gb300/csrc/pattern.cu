// pattern.cu — symbolic phase on sm_103a: the block-upper sparsity pattern of K, the
// Gauss-point -> block-slot map, and the ordered contribution lists of the
// deterministic scatter.
//
// Reference: NonLinearAssembler::initSparsityPattern (plate/Assembly.h:59-153) and the
// pattern growth of K += K_fold (plate/Meshless.h:113-127, Constraints.h:420-433).
//
// Column j of the block pattern is the sorted set of nodes i <= j that share a
// neighbour list with j. "Neighbour lists" are the face Gauss points' lists plus, for
// the hinge, each crease point's merged left/right node list (the hinge couples every
// node pair of that merged list). One warp builds one column: it walks the lists that
// contain j (node -> list inverse index), inserts every i <= j into a shared-memory hash
// set, then sorts the set by ranks. The result is the same sorted unique set the
// reference builds with sort + unique, so the pattern is bit-exact.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <string>

#include "cgb_device.cuh"
#include "cgb_internal.h"

namespace cgb {
namespace {

constexpr int kWarps = 2;
constexpr int kCap = 2048;        // hash slots per warp (8 KB)
constexpr int kMaxColumn = 1536;  // largest column the hash set accepts (75 % load)

enum : int { kErrCapacity = CGB_ERR_CAPACITY, kErrMapping = CGB_ERR_MAPPING };

// A set of lists in CSR form (face Gauss points, then crease points).
struct Lists {
  int n;
  const int64_t* ptr;
  const int32_t* idx;
};

__global__ void count_per_node(int64_t n, const int32_t* __restrict__ idx, int32_t* __restrict__ cnt) {
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e < n) atomicAdd(&cnt[idx[e]], 1);
}

// inv[cursor[node]++] = list id (+ base), one thread per list.
__global__ void fill_inverse(Lists L, int base, int64_t* __restrict__ cursor, int32_t* __restrict__ inv) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= L.n) return;
  for (int64_t e = L.ptr[g]; e < L.ptr[g + 1]; ++e) {
    const int64_t at = atomicAdd(reinterpret_cast<unsigned long long*>(&cursor[L.idx[e]]), 1ULL);
    inv[at] = base + g;
  }
}

__device__ __forceinline__ unsigned hash32(unsigned x) {
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}

// Column sets. Phase 0 counts, phase 1 writes the sorted column into col_nodes.
__global__ void __launch_bounds__(32 * kWarps) column_kernel(int n_nodes, Lists A, Lists B,
                                                              const int64_t* __restrict__ inv_ptr,
                                                              const int32_t* __restrict__ inv,
                                                              int phase, int32_t* __restrict__ col_len,
                                                              const int64_t* __restrict__ col_ptr,
                                                              int32_t* __restrict__ col_nodes, int* err) {
  __shared__ int table[kWarps][kCap];
  __shared__ int keys[kWarps][kMaxColumn];
  __shared__ int count[kWarps];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* T = table[w];
  for (int j = blockIdx.x * kWarps + w; j < n_nodes; j += gridDim.x * kWarps) {
    for (int s = lane; s < kCap; s += 32) T[s] = -1;
    if (lane == 0) count[w] = 0;
    __syncwarp();
    bool overflow = false;
    for (int64_t q = inv_ptr[j]; q < inv_ptr[j + 1]; ++q) {
      const int lid = inv[q];
      const Lists& L = lid < A.n ? A : B;
      const int li = lid < A.n ? lid : lid - A.n;
      const int64_t e0 = L.ptr[li], e1 = L.ptr[li + 1];
      for (int64_t e = e0 + lane; e < e1; e += 32) {
        const int i = L.idx[e];
        if (i > j) continue;
        unsigned h = hash32(static_cast<unsigned>(i)) & (kCap - 1);
        for (int probe = 0; probe < kCap; ++probe) {
          const int prev = atomicCAS(&T[h], -1, i);
          if (prev == -1) {
            const int at = atomicAdd(&count[w], 1);
            if (at < kMaxColumn) keys[w][at] = i; else overflow = true;
            break;
          }
          if (prev == i) break;
          h = (h + 1) & (kCap - 1);
        }
      }
    }
    __syncwarp();
    const int m = count[w];
    if (__any_sync(0xffffffffu, overflow) || m > kMaxColumn) {
      if (lane == 0) dev_fail(err, kErrCapacity);
      continue;
    }
    if (phase == 0) {
      if (lane == 0) col_len[j] = m;
    } else {
      const int64_t base = col_ptr[j];
      for (int a = lane; a < m; a += 32) {
        const int v = keys[w][a];
        int rank = 0;
        for (int b = 0; b < m; ++b) rank += (keys[w][b] < v);
        col_nodes[base + rank] = v;
      }
    }
    __syncwarp();
  }
}

// Face Gauss point -> block slot of each local pair (i <= j), in the reference's loop
// order (plate/Assembly.h:128-143). One warp per Gauss point.
__global__ void slot_map_kernel(int n_gp, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                const int64_t* __restrict__ map_ptr, const int64_t* __restrict__ col_ptr,
                                const int32_t* __restrict__ col_nodes, int32_t* __restrict__ slot, int* err) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t g = warp; g < n_gp; g += nwarps) {
    const int64_t p0 = ptr[g];
    const int n = static_cast<int>(ptr[g + 1] - p0);
    const int64_t np = static_cast<int64_t>(n) * (n + 1) / 2;
    const int64_t m0 = map_ptr[g];
    // pair p -> (i, j): walk rows of length n - i.
    int i = 0, off = lane;
    while (i < n && off >= n - i) { off -= n - i; ++i; }
    for (int64_t p = lane; p < np; p += 32) {
      const int j = i + off;
      const int ni = idx[p0 + i], nj = idx[p0 + j];
      const int lo = ni < nj ? ni : nj, hi = ni < nj ? nj : ni;
      int64_t a = col_ptr[hi], b = col_ptr[hi + 1];
      while (a < b) {
        const int64_t mid = (a + b) >> 1;
        if (col_nodes[mid] < lo) a = mid + 1; else b = mid;
      }
      int32_t s = -1;
      if (a < col_ptr[hi + 1] && col_nodes[a] == lo) s = static_cast<int32_t>(a);
      else dev_fail(err, kErrMapping);
      slot[m0 + p] = s;
      off += 32;
      while (i < n && off >= n - i) { off -= n - i; ++i; }
    }
  }
}

// CSR fill of the deterministic lists: one thread per contribution id (a negative key: no unit).
__global__ void count_slots(int64_t n, const int32_t* __restrict__ key, int64_t* __restrict__ cnt) {
  const int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (q < n && key[q] >= 0) atomicAdd(reinterpret_cast<unsigned long long*>(&cnt[key[q]]), 1ULL);
}
__global__ void fill_slots(int64_t n, int64_t base, const int32_t* __restrict__ key, int64_t* __restrict__ cursor,
                           int64_t* __restrict__ list) {
  const int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (q < n && key[q] >= 0) {
    const int64_t at = atomicAdd(reinterpret_cast<unsigned long long*>(&cursor[key[q]]), 1ULL);
    list[at] = base + q;
  }
}
// Sort each list ascending (insertion sort: lists are short and this runs once).
__global__ void sort_lists(int64_t n, const int64_t* __restrict__ lptr, int64_t* __restrict__ list) {
  const int64_t b = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (b >= n) return;
  const int64_t s = lptr[b], e = lptr[b + 1];
  for (int64_t k = s + 1; k < e; ++k) {
    const int64_t v = list[k];
    int64_t m = k - 1;
    while (m >= s && list[m] > v) { list[m + 1] = list[m]; --m; }
    list[m + 1] = v;
  }
}

// The first unit of each (sorted) list that is n_face or more.
__global__ void face_ends(int64_t n, const int64_t* __restrict__ lptr, const int64_t* __restrict__ list, int64_t n_face,
                          int64_t* __restrict__ end) {
  const int64_t b = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (b >= n) return;
  int64_t lo = lptr[b], hi = lptr[b + 1];
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (list[mid] < n_face) lo = mid + 1; else hi = mid;
  }
  end[b] = lo;
}

// ---- tables of the FP32 tangent ---------------------------------------------------------
// A cell is kMergeGroup consecutive face Gauss points (one quadrature cell with a 4x4 rule). Its
// node union, ascending, numbers the cell's nodes u; a block (I, J), I <= J, of the cell is then in
// its stored orientation (row: the lower node). The tangent's work item is a node J and a tile of
// four consecutive nodes I <= J, with the mask of J's points (the derivatives of a node that a point does
// not have are zeros; a tile that shares no point with J is no item): one CTA per cell finds the union, every entry's index in it, and the items, their
// block slots (-1 where no point has both nodes) and their order: most points first, so the lanes
// of a warp have loops of about one length, then by J, so that they share J's records.
// A cell with more than kMergePairs pairs, a list above 64 or with a node twice, or a union above
// kTileMaxU is left to the per-entry tangent ("direct").
constexpr int kMergeGroup = 16;
constexpr int kMergePairs = 16384;
constexpr int kCellEntries = 64 * kMergeGroup;
constexpr int kCellItems = kTileMaxU * (kTileMaxU / 4 + 1) / 2 + kTileMaxU;  // above sum_J (J / 4 + 1)
constexpr int kCellThreads = 128;

__global__ void __launch_bounds__(kCellThreads) tile_cells_kernel(
    int n_gp, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx, const int64_t* __restrict__ map_ptr,
    const int64_t* __restrict__ col_ptr, const int32_t* __restrict__ col_nodes, int phase, uint8_t* __restrict__ nbr_u,
    int16_t* __restrict__ cell_U, int32_t* __restrict__ n_items, const int64_t* __restrict__ item_ptr,
    uint32_t* __restrict__ item_code, int32_t* __restrict__ item_slot, unsigned long long* __restrict__ n_entries) {
  __shared__ int ids[kCellEntries];
  __shared__ unsigned mask[kTileMaxU];
  __shared__ uint8_t weight[kCellItems];   // points of every item (0: no shared point), J-major
  __shared__ uint16_t order[kCellItems];
  __shared__ int s_n, s_bad;
  const int G = blockIdx.x, t = threadIdx.x;
  const int g0 = G * kMergeGroup, g1 = min(n_gp, g0 + kMergeGroup);
  const int64_t q0 = ptr[g0], q1 = ptr[g1];
  const int items = static_cast<int>(q1 - q0);
  if (t == 0) s_bad = 0;
  __syncthreads();
  if (t < g1 - g0 && ptr[g0 + t + 1] - ptr[g0 + t] > 64) s_bad = 1;
  if (t == 0 && map_ptr[g1] - map_ptr[g0] > kMergePairs) s_bad = 1;
  __syncthreads();
  int U = 0;
  if (!s_bad) {
    int n2 = 1;
    while (n2 < items) n2 <<= 1;
    for (int i = t; i < n2; i += kCellThreads) ids[i] = i < items ? idx[q0 + i] : 0x7fffffff;
    __syncthreads();
    for (int k = 2; k <= n2; k <<= 1) {
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = t; i < n2; i += kCellThreads) {
          const int u = i ^ j;
          if (u > i) {
            const bool up = (i & k) == 0;
            const int x = ids[i], y = ids[u];
            if ((x > y) == up) { ids[i] = y; ids[u] = x; }
          }
        }
        __syncthreads();
      }
    }
    if (t == 0) {  // unique, in place
      int m = 0;
      for (int i = 0; i < items; ++i)
        if (m == 0 || ids[i] != ids[m - 1]) ids[m++] = ids[i];
      s_n = m;
    }
    __syncthreads();
    U = s_n;
  }
  if (s_bad || U > kTileMaxU) {
    if (phase == 0) {
      if (t == 0) { n_items[G] = -1; cell_U[G] = 32767; }
      for (int64_t e = q0 + t; e < q1; e += kCellThreads) nbr_u[e] = 255;
    }
    return;
  }
  for (int u = t; u < U; u += kCellThreads) mask[u] = 0;
  __syncthreads();
  for (int k = 0; k < g1 - g0; ++k)
    for (int64_t e = ptr[g0 + k] + t; e < ptr[g0 + k + 1]; e += kCellThreads) {
      const int node = idx[e];
      int lo = 0, hi = U;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ids[mid] < node) lo = mid + 1; else hi = mid;
      }
      if (phase == 0) nbr_u[e] = static_cast<uint8_t>(lo);
      if (atomicOr(&mask[lo], 1u << k) & (1u << k)) s_bad = 1;   // a node twice in one list
    }
  __syncthreads();
  if (s_bad) {
    if (phase == 0) {
      if (t == 0) { n_items[G] = -1; cell_U[G] = 32767; }
      for (int64_t e = q0 + t; e < q1; e += kCellThreads) nbr_u[e] = 255;
    }
    return;
  }
  auto tile_mask = [&](int J, int tile) {
    unsigned m = 0;
    for (int I = 4 * tile; I < 4 * tile + 4 && I <= J; ++I) m |= mask[I];
    return (m & mask[J]) ? mask[J] : 0u;
  };
  for (int J = t; J < U; J += kCellThreads) {
    const int h = J >> 2, first = 2 * h * (h + 1) + (J & 3) * (h + 1);   // sum of (j / 4 + 1), j < J
    for (int tile = 0; tile <= h; ++tile) weight[first + tile] = static_cast<uint8_t>(__popc(tile_mask(J, tile)));
  }
  __syncthreads();
  const int hU = U >> 2, total = 2 * hU * (hU + 1) + (U & 3) * (hU + 1);
  if (t == 0) {  // stable counting sort, most points first; at most a few thousand items
    int at[kMergeGroup + 1], n = 0;
    for (int c = 0; c <= kMergeGroup; ++c) at[c] = 0;
    for (int i = 0; i < total; ++i) ++at[weight[i]];
    for (int c = kMergeGroup; c >= 1; --c) { const int v = at[c]; at[c] = n; n += v; }
    for (int i = 0; i < total; ++i)
      if (weight[i]) order[at[weight[i]]++] = static_cast<uint16_t>(i);
    s_n = n;
  }
  __syncthreads();
  const int n = s_n;
  if (phase == 0) {
    if (t == 0) { n_items[G] = n; cell_U[G] = static_cast<int16_t>(U); }
    return;
  }
  const int64_t base = item_ptr[G];
  int found = 0;
  for (int i = t; i < n; i += kCellThreads) {
    const int c = order[i];
    int J = 0;   // the last J whose first item is at or below c
    for (int step = 64; step > 0; step >>= 1) {
      const int K = J + step, h = K >> 2;
      if (K < U && 2 * h * (h + 1) + (K & 3) * (h + 1) <= c) J = K;
    }
    const int h = J >> 2, tile = c - (2 * h * (h + 1) + (J & 3) * (h + 1));
    item_code[base + i] = tile_mask(J, tile) | (static_cast<unsigned>(tile) << 16) | (static_cast<unsigned>(J) << 24);
    const int64_t c0 = col_ptr[ids[J]], c1 = col_ptr[ids[J] + 1];
    for (int q = 0; q < 4; ++q) {
      const int I = 4 * tile + q;
      int32_t slot = -1;
      if (I <= J && (mask[I] & mask[J])) {
        int64_t lo = c0, hi = c1;
        while (lo < hi) {
          const int64_t mid = (lo + hi) >> 1;
          if (col_nodes[mid] < ids[I]) lo = mid + 1; else hi = mid;
        }
        slot = static_cast<int32_t>(lo);
        ++found;
      }
      item_slot[4 * (base + i) + q] = slot;
    }
  }
  if (found) atomicAdd(n_entries, static_cast<unsigned long long>(found));
}

inline unsigned nb(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

int read_err(cgb_context* ctx) {
  int e = 0;
  CGB_CUDA(cudaMemcpyAsync(&e, ctx->dev_err.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  CGB_CUDA(cudaStreamSynchronize(ctx->stream));
  return e;
}

}  // namespace

void pattern_build(cgb_assembler* a) {
  cgb_context* ctx = a->ctx;
  cudaStream_t st = ctx->stream;
  const cgb_shape* F = a->faces;
  const int n_nodes = a->n_nodes;
  CGB_CUDA(cudaMemsetAsync(ctx->dev_err.p, 0, sizeof(int), st));

  // ---- hinge lists: merged sorted node lists of every crease point (host) ----
  std::vector<int64_t> hptr(1, 0);
  std::vector<int32_t> hidx;
  for (auto& f : a->folds) {
    std::vector<int64_t> lp(f.n_gp + 1), rp(f.n_gp + 1);
    CGB_CUDA(cudaMemcpyAsync(lp.data(), f.left->nbr_ptr.p, lp.size() * 8, cudaMemcpyDeviceToHost, st));
    CGB_CUDA(cudaMemcpyAsync(rp.data(), f.right->nbr_ptr.p, rp.size() * 8, cudaMemcpyDeviceToHost, st));
    CGB_CUDA(cudaStreamSynchronize(st));
    std::vector<int32_t> li(std::max<int64_t>(lp.back(), 1)), ri(std::max<int64_t>(rp.back(), 1));
    if (lp.back()) CGB_CUDA(cudaMemcpyAsync(li.data(), f.left->nbr_idx.p, lp.back() * 4, cudaMemcpyDeviceToHost, st));
    if (rp.back()) CGB_CUDA(cudaMemcpyAsync(ri.data(), f.right->nbr_idx.p, rp.back() * 4, cudaMemcpyDeviceToHost, st));
    CGB_CUDA(cudaStreamSynchronize(st));
    std::vector<int64_t> uptr(f.n_gp + 1, 0);
    std::vector<int32_t> unode, lpos(std::max<int64_t>(lp.back(), 1)), rpos(std::max<int64_t>(rp.back(), 1));
    std::vector<int32_t> tmp;
    f.max_u = 0;
    for (int g = 0; g < f.n_gp; ++g) {
      tmp.clear();
      for (int64_t e = lp[g]; e < lp[g + 1]; ++e) tmp.push_back(li[e]);
      for (int64_t e = rp[g]; e < rp[g + 1]; ++e) tmp.push_back(ri[e]);
      std::sort(tmp.begin(), tmp.end());
      tmp.erase(std::unique(tmp.begin(), tmp.end()), tmp.end());
      for (int64_t e = lp[g]; e < lp[g + 1]; ++e)
        lpos[e] = static_cast<int32_t>(std::lower_bound(tmp.begin(), tmp.end(), li[e]) - tmp.begin());
      for (int64_t e = rp[g]; e < rp[g + 1]; ++e)
        rpos[e] = static_cast<int32_t>(std::lower_bound(tmp.begin(), tmp.end(), ri[e]) - tmp.begin());
      unode.insert(unode.end(), tmp.begin(), tmp.end());
      uptr[g + 1] = uptr[g] + static_cast<int64_t>(tmp.size());
      f.max_u = std::max<int>(f.max_u, static_cast<int>(tmp.size()));
      hidx.insert(hidx.end(), tmp.begin(), tmp.end());
      hptr.push_back(hptr.back() + static_cast<int64_t>(tmp.size()));
    }
    f.n_u = uptr[f.n_gp];
    upload(f.u_ptr, uptr.data(), uptr.size(), st);
    upload(f.u_node, unode.data(), unode.size(), st);
    upload(f.l_pos, lpos.data(), lpos.size(), st);
    upload(f.r_pos, rpos.data(), rpos.size(), st);
    CGB_CUDA(cudaStreamSynchronize(st));
  }
  const int n_hl = static_cast<int>(hptr.size() - 1);
  DevBuf<int64_t> d_hptr;
  DevBuf<int32_t> d_hidx;
  upload(d_hptr, hptr.data(), hptr.size(), st);
  upload(d_hidx, hidx.data(), hidx.size(), st);

  // ---- node -> list inverse index ----
  DevBuf<int32_t> cnt(n_nodes);
  CGB_CUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes(), st));
  if (F->nnz) count_per_node<<<nb(F->nnz, 256), 256, 0, st>>>(F->nnz, F->nbr_idx.p, cnt.p);
  if (!hidx.empty()) count_per_node<<<nb(hidx.size(), 256), 256, 0, st>>>(hidx.size(), d_hidx.p, cnt.p);
  CGB_CUDA(cudaGetLastError());
  std::vector<int32_t> hc(n_nodes);
  CGB_CUDA(cudaMemcpyAsync(hc.data(), cnt.p, cnt.bytes(), cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  std::vector<int64_t> inv_ptr(n_nodes + 1, 0);
  for (int j = 0; j < n_nodes; ++j) inv_ptr[j + 1] = inv_ptr[j] + hc[j];
  DevBuf<int64_t> d_inv_ptr, cursor;
  upload(d_inv_ptr, inv_ptr.data(), inv_ptr.size(), st);
  upload(cursor, inv_ptr.data(), n_nodes, st);
  DevBuf<int32_t> inv(inv_ptr.back());
  Lists LA{F->n_gp, F->nbr_ptr.p, F->nbr_idx.p};
  Lists LB{n_hl, d_hptr.p, d_hidx.p};
  if (LA.n) fill_inverse<<<nb(LA.n, 128), 128, 0, st>>>(LA, 0, cursor.p, inv.p);
  if (LB.n) fill_inverse<<<nb(LB.n, 128), 128, 0, st>>>(LB, LA.n, cursor.p, inv.p);
  CGB_CUDA(cudaGetLastError());

  // ---- columns: count, scan, fill ----
  DevBuf<int32_t> col_len(n_nodes);
  const unsigned cgrid = std::max(1u, std::min(nb(n_nodes, kWarps), 152u * 16u));
  column_kernel<<<cgrid, 32 * kWarps, 0, st>>>(n_nodes, LA, LB, d_inv_ptr.p, inv.p, 0, col_len.p, nullptr,
                                              nullptr, ctx->dev_err.p);
  CGB_CUDA(cudaGetLastError());
  if (int e = read_err(ctx))
    throw Error(e, "initSparsityPattern: a column of the node pattern has more than 1536 block rows");
  std::vector<int32_t> hl(n_nodes);
  CGB_CUDA(cudaMemcpyAsync(hl.data(), col_len.p, col_len.bytes(), cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  std::vector<int64_t> cptr(n_nodes + 1, 0);
  for (int j = 0; j < n_nodes; ++j) cptr[j + 1] = cptr[j] + hl[j];
  a->n_blocks = cptr[n_nodes];
  if (9 * a->n_blocks >= (1LL << 31))
    throw Error(CGB_ERR_CAPACITY, "initSparsityPattern: nnz(K) exceeds the int32 index range of the reference's K");
  upload(a->col_ptr, cptr.data(), cptr.size(), st);
  a->col_nodes.alloc(a->n_blocks);
  column_kernel<<<cgrid, 32 * kWarps, 0, st>>>(n_nodes, LA, LB, d_inv_ptr.p, inv.p, 1, col_len.p, a->col_ptr.p,
                                              a->col_nodes.p, ctx->dev_err.p);
  CGB_CUDA(cudaGetLastError());
  // Scalar CSC outer index (Assembly.h:103-107): column 3j+c starts at
  // 9 col_ptr[j] + 3 c len_j.
  std::vector<int32_t> outer(3 * static_cast<size_t>(n_nodes) + 1);
  for (int j = 0; j < n_nodes; ++j)
    for (int c = 0; c < 3; ++c) outer[3 * j + c] = static_cast<int32_t>(9 * cptr[j] + 3 * c * hl[j]);
  outer[3 * n_nodes] = static_cast<int32_t>(9 * cptr[n_nodes]);
  upload(a->outer, outer.data(), outer.size(), st);

  // ---- face slot map ----
  std::vector<int64_t> fptr(F->n_gp + 1);
  CGB_CUDA(cudaMemcpyAsync(fptr.data(), F->nbr_ptr.p, fptr.size() * 8, cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  std::vector<int64_t> mptr(F->n_gp + 1, 0);
  for (int g = 0; g < F->n_gp; ++g) {
    const int64_t n = fptr[g + 1] - fptr[g];
    mptr[g + 1] = mptr[g] + n * (n + 1) / 2;
  }
  a->n_pairs = mptr[F->n_gp];
  upload(a->map_ptr, mptr.data(), mptr.size(), st);
  a->map_slot.alloc(a->n_pairs);
  if (F->n_gp)
    slot_map_kernel<<<std::min<int64_t>(nb(F->n_gp, 8), 152 * 64), 256, 0, st>>>(
        F->n_gp, F->nbr_ptr.p, F->nbr_idx.p, a->map_ptr.p, a->col_ptr.p, a->col_nodes.p, a->map_slot.p,
        ctx->dev_err.p);
  CGB_CUDA(cudaGetLastError());
  if (int e = read_err(ctx)) {
    if (e == CGB_ERR_MAPPING)
      throw Error(e, "Assembly: Gauss-point neighbour missing from the sparsity pattern; "
                     "CSR mapping is inconsistent.");
    throw Error(e, "initSparsityPattern: device check failed");
  }

  // ---- hinge pair slots (host: crease points are few) ----
  if (!a->folds.empty()) {
    std::vector<int32_t> hcn(a->n_blocks);
    CGB_CUDA(cudaMemcpyAsync(hcn.data(), a->col_nodes.p, hcn.size() * 4, cudaMemcpyDeviceToHost, st));
    CGB_CUDA(cudaStreamSynchronize(st));
    int64_t hoff = 0;
    std::vector<std::vector<int32_t>> slots(a->folds.size());
    for (size_t k = 0; k < a->folds.size(); ++k) {
      auto& f = a->folds[k];
      std::vector<int64_t> pp(f.n_gp + 1, 0);
      std::vector<int32_t>& ps = slots[k];
      for (int g = 0; g < f.n_gp; ++g) {
        const int64_t u0 = hptr[hoff + g], u1 = hptr[hoff + g + 1];
        for (int64_t P = u0; P < u1; ++P)
          for (int64_t Q = P; Q < u1; ++Q) {
            const int lo = hidx[P], hi = hidx[Q];
            auto b0 = hcn.begin() + cptr[hi], b1 = hcn.begin() + cptr[hi + 1];
            auto it = std::lower_bound(b0, b1, lo);
            if (it == b1 || *it != lo)
              throw Error(CGB_ERR_MAPPING, "Assembly: hinge block missing from the sparsity pattern");
            ps.push_back(static_cast<int32_t>(it - hcn.begin()));
          }
        pp[g + 1] = static_cast<int64_t>(ps.size());
      }
      hoff += f.n_gp;
      f.n_pairs = static_cast<int64_t>(ps.size());
      upload(f.pair_ptr, pp.data(), pp.size(), st);
      upload(f.pair_slot, ps.data(), ps.size(), st);
      CGB_CUDA(cudaStreamSynchronize(st));
    }
    // The touched blocks numbered by slot (the mixed mode adds the hinge into FP64 blocks of its own).
    std::vector<int32_t> at(a->n_blocks, -1), pos;
    for (const auto& ps : slots)
      for (int32_t q : ps) at[q] = 0;
    std::vector<int64_t> hcol(n_nodes + 1, 0);
    for (int j = 0; j < n_nodes; ++j) {
      for (int64_t b = cptr[j]; b < cptr[j + 1]; ++b)
        if (at[b] == 0) {
          at[b] = static_cast<int32_t>(pos.size());
          pos.push_back(static_cast<int32_t>(b - cptr[j]));
        }
      hcol[j + 1] = static_cast<int64_t>(pos.size());
    }
    a->n_hinge_blocks = hcol[n_nodes];
    upload(a->hinge_col, hcol.data(), hcol.size(), st);
    upload(a->hinge_pos, pos.data(), pos.size(), st);
    for (size_t k = 0; k < a->folds.size(); ++k) {
      for (int32_t& q : slots[k]) q = at[q];
      upload(a->folds[k].pair_hslot, slots[k].data(), slots[k].size(), st);
    }
    CGB_CUDA(cudaStreamSynchronize(st));
  }
  CGB_CUDA(cudaStreamSynchronize(st));
}

void tile_prepare(cgb_assembler* a) {
  if (a->tile_ready) return;
  cudaStream_t st = a->ctx->stream;
  const cgb_shape* S = a->faces;
  const int n_gp = S->n_gp;
  const int ng = (n_gp + kMergeGroup - 1) / kMergeGroup;
  a->nbr_u.alloc(S->nnz + 32);   // the tangent stages it with bulk copies widened to 16 bytes
  a->cell_U.alloc(ng);
  DevBuf<int32_t> counts(ng);
  DevBuf<unsigned long long> entries(1);
  CGB_CUDA(cudaMemsetAsync(entries.p, 0, entries.bytes(), st));
  auto cells = [&](int phase) {
    if (ng > 0)
      tile_cells_kernel<<<ng, kCellThreads, 0, st>>>(n_gp, S->nbr_ptr.p, S->nbr_idx.p, a->map_ptr.p, a->col_ptr.p,
                                                     a->col_nodes.p, phase, a->nbr_u.p, a->cell_U.p, counts.p,
                                                     a->item_ptr.p, a->item_code.p, a->item_slot.p, entries.p);
    CGB_CUDA(cudaGetLastError());
  };
  cells(0);
  std::vector<int32_t> hc(std::max(ng, 1));
  std::vector<int16_t> cu(std::max(ng, 1));
  std::vector<int64_t> ptr(n_gp + 1);
  if (ng > 0) {
    CGB_CUDA(cudaMemcpyAsync(hc.data(), counts.p, ng * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CGB_CUDA(cudaMemcpyAsync(cu.data(), a->cell_U.p, ng * sizeof(int16_t), cudaMemcpyDeviceToHost, st));
    CGB_CUDA(cudaMemcpyAsync(ptr.data(), S->nbr_ptr.p, ptr.size() * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  }
  CGB_CUDA(cudaStreamSynchronize(st));
  std::vector<int64_t> ip(ng + 1, 0);
  std::vector<TileCell> cells_h(ng);
  a->direct_h.clear();
  a->tc_rest_h.clear();
  a->tc_n_groups = 0;
  a->tc_point_cols = 0;
  a->cell_max_e = a->cell_max_u = a->cell_max_i = 0;
  for (int G = 0; G < ng; ++G) {
    ip[G + 1] = ip[G] + std::max(hc[G], 0);
    cells_h[G] = TileCell{ptr[G * kMergeGroup], ip[G],
                          static_cast<int32_t>(ptr[std::min(n_gp, (G + 1) * kMergeGroup)] - ptr[G * kMergeGroup]),
                          std::max(hc[G], 0), cu[G], 0};
    if (hc[G] < 0) { a->direct_h.push_back(G); continue; }
    const int g1 = std::min(n_gp, (G + 1) * kMergeGroup);
    a->cell_max_e = std::max<int>(a->cell_max_e, static_cast<int>(ptr[g1] - ptr[G * kMergeGroup]));
    a->cell_max_u = std::max<int>(a->cell_max_u, cu[G]);
    a->cell_max_i = std::max<int>(a->cell_max_i, hc[G]);
    if (cu[G] > kTcMaxUnion) { a->tc_rest_h.push_back(G); continue; }
    ++a->tc_n_groups;
    a->tc_point_cols += static_cast<int64_t>(g1 - G * kMergeGroup) * std::max(16, (3 * cu[G] + 15) & ~15);
  }
  upload(a->direct, a->direct_h.data(), a->direct_h.size(), st);
  upload(a->tc_rest, a->tc_rest_h.data(), a->tc_rest_h.size(), st);
  upload(a->item_ptr, ip.data(), ip.size(), st);
  upload(a->cells, cells_h.data(), cells_h.size(), st);
  a->n_items = ip[ng];
  a->item_code.alloc(a->n_items + 8);  // staged with bulk copies widened to 16 bytes
  a->item_slot.alloc(4 * a->n_items);
  cells(1);
  unsigned long long n_ent = 0;
  CGB_CUDA(cudaMemcpyAsync(&n_ent, entries.p, sizeof(n_ent), cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  a->n_entries = static_cast<int64_t>(n_ent);
  a->tile_ready = true;
}

// Ordered lists for the deterministic scatter. F contribution ids: face entries
// [0, nnz_face), then hinge merged-node entries fold by fold. K unit ids: the face units
// (pairs, or four blocks per item of the cells), then hinge pairs fold by fold. Each K block and each node sums
// its units in ascending id order, i.e. Gauss point (or group of Gauss points) by Gauss
// point in the reference's loop order.
namespace {

// Per-block ascending lists of K units: n_face face units whose block slots are face_slot,
// then every fold's pairs.
void block_lists(cgb_assembler* a, int64_t n_face, const int32_t* face_slot, DevBuf<int64_t>& ptr,
                 DevBuf<int64_t>& list, DevBuf<int64_t>& face_end) {
  cudaStream_t st = a->ctx->stream;
  int64_t nq = n_face;
  for (auto& f : a->folds) nq += f.n_pairs;
  DevBuf<int64_t> cnt(a->n_blocks + 1);
  CGB_CUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes(), st));
  if (n_face) count_slots<<<nb(n_face, 256), 256, 0, st>>>(n_face, face_slot, cnt.p);
  for (auto& f : a->folds)
    if (f.n_pairs) count_slots<<<nb(f.n_pairs, 256), 256, 0, st>>>(f.n_pairs, f.pair_slot.p, cnt.p);
  std::vector<int64_t> hc(a->n_blocks);
  CGB_CUDA(cudaMemcpyAsync(hc.data(), cnt.p, hc.size() * 8, cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  std::vector<int64_t> lp(a->n_blocks + 1, 0);
  for (int64_t b = 0; b < a->n_blocks; ++b) lp[b + 1] = lp[b] + hc[b];
  upload(ptr, lp.data(), lp.size(), st);
  DevBuf<int64_t> cur;
  upload(cur, lp.data(), a->n_blocks, st);
  list.alloc(std::max<int64_t>(nq, 1));
  if (n_face) fill_slots<<<nb(n_face, 256), 256, 0, st>>>(n_face, 0, face_slot, cur.p, list.p);
  int64_t base = n_face;
  for (auto& f : a->folds) {
    if (f.n_pairs) fill_slots<<<nb(f.n_pairs, 256), 256, 0, st>>>(f.n_pairs, base, f.pair_slot.p, cur.p, list.p);
    base += f.n_pairs;
  }
  sort_lists<<<nb(a->n_blocks, 128), 128, 0, st>>>(a->n_blocks, ptr.p, list.p);
  face_end.alloc(a->n_blocks);
  face_ends<<<nb(a->n_blocks, 128), 128, 0, st>>>(a->n_blocks, ptr.p, list.p, n_face, face_end.p);
  CGB_CUDA(cudaGetLastError());
  CGB_CUDA(cudaStreamSynchronize(st));
}

}  // namespace

void deterministic_pair_lists(cgb_assembler* a) {
  if (a->det_pairs_ready) return;
  block_lists(a, a->n_pairs, a->map_slot.p, a->blk_list_ptr, a->blk_list, a->blk_face_end);
  a->det_pairs_ready = true;
}

void deterministic_entry_lists(cgb_assembler* a) {
  if (a->det_entries_ready) return;
  tile_prepare(a);
  if (!a->direct_h.empty()) throw Error(CGB_ERR_INVALID, "deterministic entry lists need every group merged");
  block_lists(a, 4 * a->n_items, a->item_slot.p, a->ent_list_ptr, a->ent_list, a->ent_face_end);
  a->det_entries_ready = true;
}

void deterministic_prepare(cgb_assembler* a) {
  if (a->det_ready) return;
  cgb_context* ctx = a->ctx;
  cudaStream_t st = ctx->stream;
  int64_t n_hf = 0;
  std::vector<int64_t> fnum;  // merged-node entries per fold
  for (auto& f : a->folds) {
    fnum.push_back(f.n_u);
    n_hf += f.n_u;
  }
  a->hinge_f_base = a->faces->nnz;
  a->n_fcontrib = a->faces->nnz + n_hf;

  // F lists (node of each contribution: face entries then hinge merged nodes).
  DevBuf<int64_t> fc(a->n_nodes + 1);
  CGB_CUDA(cudaMemsetAsync(fc.p, 0, fc.bytes(), st));
  if (a->faces->nnz) count_slots<<<nb(a->faces->nnz, 256), 256, 0, st>>>(a->faces->nnz, a->faces->nbr_idx.p, fc.p);
  for (size_t k = 0; k < a->folds.size(); ++k)
    if (fnum[k]) count_slots<<<nb(fnum[k], 256), 256, 0, st>>>(fnum[k], a->folds[k].u_node.p, fc.p);
  std::vector<int64_t> hf(a->n_nodes);
  CGB_CUDA(cudaMemcpyAsync(hf.data(), fc.p, hf.size() * 8, cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  std::vector<int64_t> np(a->n_nodes + 1, 0);
  for (int j = 0; j < a->n_nodes; ++j) np[j + 1] = np[j] + hf[j];
  upload(a->node_list_ptr, np.data(), np.size(), st);
  DevBuf<int64_t> fcur;
  upload(fcur, np.data(), a->n_nodes, st);
  a->node_list.alloc(a->n_fcontrib);
  if (a->faces->nnz)
    fill_slots<<<nb(a->faces->nnz, 256), 256, 0, st>>>(a->faces->nnz, 0, a->faces->nbr_idx.p, fcur.p, a->node_list.p);
  int64_t base = a->faces->nnz;
  for (size_t k = 0; k < a->folds.size(); ++k) {
    if (fnum[k]) fill_slots<<<nb(fnum[k], 256), 256, 0, st>>>(fnum[k], base, a->folds[k].u_node.p, fcur.p, a->node_list.p);
    base += fnum[k];
  }
  sort_lists<<<nb(a->n_nodes, 128), 128, 0, st>>>(a->n_nodes, a->node_list_ptr.p, a->node_list.p);
  CGB_CUDA(cudaGetLastError());
  CGB_CUDA(cudaStreamSynchronize(st));
  a->det_ready = true;
}

}  // namespace cgb
