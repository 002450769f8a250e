// tangent_tile.cuh — the FP32 tangent of a cell of 16 consecutive Gauss points with the cell's
// contributions to a block summed in registers. Included by assemble.cu.
//
// One CTA per cell. The block of a pair is sum_a phi_i[a] T_j[a] (tangent_entry.cuh), so over the
// cell's node union the blocks of a node J are products of T_J, one record per point that has J as
// a neighbour, with the derivatives phi of the nodes I <= J. A thread takes J and a tile of four
// consecutive I (an item of tile_prepare) and walks the points of J: it reads T_J (27
// values) and the normal once and phi of the four nodes, zero where a point does not have one of
// them, and adds 4 x 36 FMA to 36 sums in registers, then scatters its blocks with three 16-byte
// FP32 vector atomics each (a scattered block costs three L2 atomics and the chip sustains about
// 70 G blocks/s of them; summing the cell's points first divides their number by seven to ten).
//
// Why four nodes per item: one pair at a time, formed from frame, I and J records of 128 bytes,
// had bound the kernel by the shared-memory data pipe at 87-90 % with about 100 FMA a pair; here
// a pair reads about 55 bytes (less where lanes share J) and takes 36 FMA. The zeros cost about
// a fifth of the sums.
struct TileArgs {
  const TileCell* cells;
  const uint32_t* item_code;   // mask of J's points | tile << 16 | J << 24
  const int4* item_slot;
  const uint8_t* nbr_u;
  int max_e, max_u, max_i;     // most entries, nodes and items of a cell
  int* err;                    // set to kErrStage when a staging copy never completes
  uint32_t extra_tx;           // 0; the failure-detection test expects bytes that never arrive
  const int32_t* glist;        // the launch's cells glist[0 .. gcount), or every cell of [g_begin, g_end)
  int gcount;
};

constexpr int kTileThreads = 192;
constexpr int kTileState = (kState * kMG + kTileThreads - 1) / kTileThreads;   // state values per thread
constexpr int kTilePhi = 20;   // floats of a tile: five derivatives of four nodes
// A point's frame in shared memory, one row of nine float4: a1 a2 b, a^1 a^2 (9), r_k . a^1 and
// r_k . a^2 (15), C0^-1 (21: 00 01 11), N, M, pXY, bv, W; r0XX, r0YY, r0XY apart ([9][point]).
constexpr int kTileFrame = 36;

// Floats per T_J record: 27 (36 with B != 0) in whole float4 of an odd number, so that records a
// stride apart start in different bank groups.
__host__ __device__ constexpr int tile_rec_floats(bool bzero) { return bzero ? 28 : 36; }

// Dynamic shared memory: records, phi, point states, normals, the (point, node) -> entry table, the
// items' codes and the staging windows of grad / Hessian Phi, the union indices and the codes.
inline size_t tile_smem_bytes(int max_e, int max_u, int max_i, bool bzero) {
  const size_t tiles = (static_cast<size_t>(max_u) + 3) / 4, e = max_e;
  return e * tile_rec_floats(bzero) * sizeof(float) + kMG * tiles * kTilePhi * sizeof(float) +
         (kTileFrame + 9) * kMG * sizeof(float) + kMG * tiles * 4 * sizeof(uint16_t) +
         4 * static_cast<size_t>(max_i) + (21 * e + 4 * static_cast<size_t>(max_i) + 4 * 48);
}

__device__ __forceinline__ Frame<float> tile_frame(const float* p) {
  float v[kTileFrame];
#pragma unroll
  for (int q = 0; q < kTileFrame / 4; ++q) {
    const float4 x = reinterpret_cast<const float4*>(p)[q];
    v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
  }
  Frame<float> f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    f.a1[c] = v[c]; f.a2[c] = v[3 + c]; f.b[c] = v[6 + c];
    f.Ax[c] = v[9 + c]; f.Ay[c] = v[12 + c]; f.Bx[c] = v[15 + c]; f.By[c] = v[18 + c];
    f.N[c] = v[24 + c]; f.M[c] = v[27 + c];
  }
  f.C00 = v[21]; f.C01 = v[22]; f.C11 = v[23];
  f.pX = v[30]; f.pY = v[31]; f.bv = v[32]; f.W = v[33];
  return f;
}

template <bool BZERO, bool DET>
__global__ void __launch_bounds__(kTileThreads, 3) face_tangent_tile_kernel(FaceArgs a, const float* __restrict__ gstate,
                                                                            TileArgs tg) {
  constexpr int RS = tile_rec_floats(BZERO);
  extern __shared__ __align__(16) float tile_smem[];
  __shared__ __align__(8) uint64_t stage_bar;
  __shared__ int sptr[kMG + 1];        // the points' first entries within the cell
  __shared__ int s_next;               // the cell's next 32 items
  __shared__ TileCell s_cell[2];       // this cell and the next
  __shared__ int s_gi[2];              // their positions in the launch (nG: none)
  const int t = threadIdx.x, lane = t & 31;
  const int max_tiles = (tg.max_u + 3) / 4;
  float* rec = tile_smem;                                        // [entry][RS]
  float* phi = rec + static_cast<size_t>(tg.max_e) * RS;         // [point][tile][5][4]
  float* fr = phi + kMG * max_tiles * kTilePhi;                  // [point][kTileFrame]
  float* rr = fr + kMG * kTileFrame;                             // [9][point]
  uint16_t* ent = reinterpret_cast<uint16_t*>(rr + 9 * kMG);     // [point][4 max_tiles]
  uint32_t* codes = reinterpret_cast<uint32_t*>(ent + kMG * 4 * max_tiles);
  const size_t at = reinterpret_cast<unsigned char*>(codes + tg.max_i) - reinterpret_cast<unsigned char*>(tile_smem);
  unsigned char* s_d = reinterpret_cast<unsigned char*>(tile_smem) + ((at + 15) & ~static_cast<size_t>(15));
  unsigned char* s_dd = s_d + ((8 * static_cast<size_t>(tg.max_e) + 47) & ~static_cast<size_t>(15));
  unsigned char* s_u = s_dd + ((12 * static_cast<size_t>(tg.max_e) + 47) & ~static_cast<size_t>(15));
  unsigned char* s_code = s_u + ((static_cast<size_t>(tg.max_e) + 47) & ~static_cast<size_t>(15));
  const unsigned char* dpsi_b = static_cast<const unsigned char*>(a.dpsi_t);
  const unsigned char* ddpsi_b = static_cast<const unsigned char*>(a.ddpsi_t);
  const int G0 = a.g_begin / kMG;
  const int nG = tg.glist ? tg.gcount : (a.g_end + kMG - 1) / kMG - G0;
  auto cell = [&](int gi) { return tg.glist ? tg.glist[gi] : G0 + gi; };
  // Everything a cell needs from global memory is requested a cell ahead: its ranges (cells[]) in
  // shared memory, its copies into the staging windows, its states and list starts in registers.
  // Read where they are needed, they had cost 7,300 of a cell's 21,000 cycles.
  auto next_cell = [&](int gi) { return gi < nG ? tg.cells[cell(gi)] : TileCell{}; };
  auto keep_cell = [&](int slot, int gi, TileCell c) {   // the first cell from gi on that is not direct
    while (gi < nG && c.U > kTileMaxU) c = next_cell(gi += gridDim.x);
    s_cell[slot] = c;
    s_gi[slot] = gi;
  };
  // Thread 0 starts the copies of a cell's ranges; every thread later waits on the phase.
  auto stage = [&](const TileCell& c) {
    const StageWin wd = stage_window(c.q0, c.q0 + c.n_ent, 8), wdd = stage_window(c.q0, c.q0 + c.n_ent, 12),
                   wu = stage_window(c.q0, c.q0 + c.n_ent, 1), wc = stage_window(c.i0, c.i0 + c.n_items, 4);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect(&stage_bar, wd.len + wdd.len + wu.len + wc.len + tg.extra_tx);
    if (wd.len) bulk_load(s_d, dpsi_b + wd.lo, wd.len, &stage_bar);
    if (wdd.len) bulk_load(s_dd, ddpsi_b + wdd.lo, wdd.len, &stage_bar);
    if (wu.len) bulk_load(s_u, tg.nbr_u + wu.lo, wu.len, &stage_bar);
    if (wc.len) bulk_load(s_code, reinterpret_cast<const unsigned char*>(tg.item_code) + wc.lo, wc.len, &stage_bar);
    // The items' slots are read once per step, from DRAM: into L2 a cell ahead of their use.
    l2_prefetch(tg.item_slot, 16 * c.i0, 16 * (c.i0 + c.n_items));
  };
  float sv[kTileState];
  int64_t pv = 0;
  auto load_state = [&](int G) {
#pragma unroll
    for (int q = 0; q < kTileState; ++q) {
      const int i = t + q * kTileThreads, f = i / kMG, g = G * kMG + (i - f * kMG);
      sv[q] = i < kState * kMG && g < a.g_end ? gstate[static_cast<int64_t>(f) * a.n_gp + g] : 0.0f;
    }
    if (t <= kMG) pv = a.ptr[min(G * kMG + t, a.g_end)];
  };
  if (t == 0) {
    mbar_init(&stage_bar);
    keep_cell(0, blockIdx.x, next_cell(blockIdx.x));
    if (s_gi[0] < nG) stage(s_cell[0]);
  }
  __syncthreads();
  int gi = s_gi[0], buf = 0;
  if (gi < nG) load_state(cell(gi));
  uint32_t phase = 0;
  while (gi < nG) {
    const TileCell& C = s_cell[buf];
    const int tiles = (C.U + 3) >> 2, n_ent = C.n_ent, n_items = C.n_items;
    const int64_t q0 = C.q0, i0 = C.i0;
    TileCell ahead{};
    if (t == 0) ahead = next_cell(gi + gridDim.x);
#pragma unroll
    for (int q = 0; q < kTileState; ++q) {
      const int i = t + q * kTileThreads, f = i / kMG, k = i - f * kMG;
      if (i >= kState * kMG) break;
      if (f >= S_RXX && f < S_CI) rr[i - S_RXX * kMG] = sv[q];
      else if (f != S_CI + 2) fr[k * kTileFrame + (f < S_RXX ? f : f < S_CI + 2 ? f + 3 : f + 2)] = sv[q];
    }
    if (t == 0) s_next = 0;
    if (t <= kMG) sptr[t] = static_cast<int>(pv - q0);
    for (int i = t; i < kMG * tiles * (kTilePhi / 4); i += kTileThreads)
      reinterpret_cast<float4*>(phi)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // Every thread waits on the copies of this cell, then the CTA agrees on the outcome so
    // that no thread leaves while another waits at a barrier.
    const bool ok = mbar_wait(&stage_bar, phase);
    if (__syncthreads_or(!ok)) {
      if (t == 0) {
        atomicOr(tg.err, kErrStage);
        mbar_wait(&stage_bar, phase);   // let copies still in flight land before leaving
      }
      return;
    }
    phase ^= 1u;
    const float* sdp = reinterpret_cast<const float*>(s_d + ((q0 * 8) & 15));
    const float* sddp = reinterpret_cast<const float*>(s_dd + ((q0 * 12) & 15));
    const unsigned char* su = s_u + (q0 & 15);
    const uint32_t* scode = reinterpret_cast<const uint32_t*>(s_code + ((i0 * 4) & 15));
    for (int i = t; i < n_items; i += kTileThreads) codes[i] = scode[i];
    {   // the dual basis and its products, one of the points' 12 x 16 values per thread
      static_assert(12 * kMG <= kTileThreads, "one value per thread");
      const int q = t / kMG, k = t - q * kMG;
      float* f = fr + k * kTileFrame;
      const bool y = (q / 3) & 1;
      const float ca = y ? f[22] : f[21], cb = y ? f[23] : f[22];
      if (q < 6) {
        f[9 + q] = ca * f[q % 3] + cb * f[3 + q % 3];
      } else if (q < 12) {
        const float* r = rr + 3 * (q % 3) * kMG + k;
        const float r0 = r[0], r1 = r[kMG], r2 = r[2 * kMG];
        const float v = ca * (r0 * f[0] + r1 * f[1] + r2 * f[2]) + cb * (r0 * f[3] + r1 * f[4] + r2 * f[5]);
        f[9 + q] = q % 3 == 2 ? 2.0f * v : v;
      }
    }
    __syncthreads();
    for (int e = t; e < n_ent; e += kTileThreads) {
      int k = 0;   // the last point whose first entry is at or before e
#pragma unroll
      for (int step = 8; step > 0; step >>= 1)
        if (sptr[k + step] <= e) k += step;
      const Frame<float> f = tile_frame(fr + k * kTileFrame);
      const float dx = sdp[2 * e], dy = sdp[2 * e + 1];
      const float dxx = sddp[3 * e], dyy = sddp[3 * e + 1], dxy = sddp[3 * e + 2];
      const int u = su[e];
      float* ph = phi + (k * tiles + (u >> 2)) * kTilePhi + (u & 3);
      ph[0] = dx; ph[4] = dy; ph[8] = dxx; ph[12] = dyy; ph[16] = dxy;
      ent[k * 4 * tiles + u] = static_cast<uint16_t>(e);
      ColumnRecord<float, BZERO> R;
      column_record<float, BZERO>(f, a.mat, dx, dy, dxx, dyy, dxy, R);
      float4* o = reinterpret_cast<float4*>(rec + static_cast<size_t>(e) * RS);
      o[0] = make_float4(R.Tx[0], R.Tx[1], R.Tx[2], R.Tx[3]);
      o[1] = make_float4(R.Tx[4], R.Tx[5], R.Tx[6], R.Tx[7]);
      o[2] = make_float4(R.Tx[8], R.Ty[0], R.Ty[1], R.Ty[2]);
      o[3] = make_float4(R.Ty[3], R.Ty[4], R.Ty[5], R.Ty[6]);
      o[4] = make_float4(R.Ty[7], R.Ty[8], R.v[0], R.v[1]);
      o[5] = make_float4(R.v[2], R.v[3], R.v[4], R.v[5]);
      if constexpr (BZERO) {
        o[6] = make_float4(R.v[6], R.v[7], R.v[8], 0.0f);
      } else {
        o[6] = make_float4(R.v[6], R.v[7], R.v[8], R.w[0]);
        o[7] = make_float4(R.w[1], R.w[2], R.w[3], R.w[4]);
        o[8] = make_float4(R.w[5], R.w[6], R.w[7], R.w[8]);
      }
    }
    if (t == 0) keep_cell(buf ^ 1, gi + gridDim.x, ahead);
    __syncthreads();
    // The staging windows are free: start the next cell's copies and state loads, which land
    // while this cell's items are summed.
    buf ^= 1;
    gi = s_gi[buf];   // written by thread 0 before the barrier
    if (gi < nG) {
      if (t == 0) stage(s_cell[buf]);
      load_state(cell(gi));
    }
    // A warp takes the next 32 items at a time: they come with 16 points first and a few last,
    // so the warps finish together.
    for (;;) {
      int it = 0;
      if (lane == 0) it = atomicAdd(&s_next, 32);
      it = __shfl_sync(0xffffffffu, it, 0);
      if (it >= n_items) break;
      it += lane;
      if (it >= n_items) continue;
      const uint32_t code = codes[it];
      const int4 slot = tg.item_slot[i0 + it];
      const int J = code >> 24, tile = (code >> 16) & 255;
      unsigned mask = code & 0xffffu;
      float acc[4][9];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < 9; ++c) acc[q][c] = 0.0f;
      while (mask) {
        const int k = __ffs(mask) - 1;
        mask &= mask - 1;
        const float4* r = reinterpret_cast<const float4*>(rec + static_cast<size_t>(ent[k * 4 * tiles + J]) * RS);
        const float4* p = reinterpret_cast<const float4*>(phi + (k * tiles + tile) * kTilePhi);
        const float* fk = fr + k * kTileFrame;
        const float2 b12 = *reinterpret_cast<const float2*>(fk + 6);
        const float b[3] = {b12.x, b12.y, fk[8]};
        float T[RS];
#pragma unroll
        for (int q = 0; q < RS / 4; ++q) {
          const float4 v = r[q];
          T[4 * q] = v.x; T[4 * q + 1] = v.y; T[4 * q + 2] = v.z; T[4 * q + 3] = v.w;
        }
        const float4 X = p[0], Y = p[1], XX = p[2], YY = p[3], XY = p[4];
        const float px[4] = {X.x, X.y, X.z, X.w}, py[4] = {Y.x, Y.y, Y.z, Y.w};
        const float pxx[4] = {XX.x, XX.y, XX.z, XX.w}, pyy[4] = {YY.x, YY.y, YY.z, YY.w}, pxy[4] = {XY.x, XY.y, XY.z, XY.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float l[3];
          if constexpr (!BZERO) {
#pragma unroll
            for (int c = 0; c < 3; ++c) l[c] = fmaf(pxy[q], T[33 + c], fmaf(pyy[q], T[30 + c], pxx[q] * T[27 + c]));
          }
#pragma unroll
          for (int rr = 0; rr < 3; ++rr) {
            const float s = fmaf(pxy[q], T[24 + rr], fmaf(pyy[q], T[21 + rr], pxx[q] * T[18 + rr]));
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              float v = fmaf(s, b[c], fmaf(py[q], T[9 + 3 * rr + c], fmaf(px[q], T[3 * rr + c], acc[q][3 * rr + c])));
              if constexpr (!BZERO) v = fmaf(b[rr], l[c], v);
              acc[q][3 * rr + c] = v;
            }
          }
        }
      }
      const int sl[4] = {slot.x, slot.y, slot.z, slot.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (sl[q] < 0) continue;
        const float* v = acc[q];
        if constexpr (DET) {
          float* d = static_cast<float*>(a.Kc) + 9 * (4 * (i0 + it) + q);
#pragma unroll
          for (int c = 0; c < 9; ++c) d[c] = v[c];
        } else {
          float4* d = static_cast<float4*>(a.Kacc) + 3 * static_cast<int64_t>(sl[q]);
          atomicAdd(d, make_float4(v[0], v[1], v[2], v[3]));
          atomicAdd(d + 1, make_float4(v[4], v[5], v[6], v[7]));
          atomicAdd(d + 2, make_float4(v[8], 0.0f, 0.0f, 0.0f));
        }
      }
    }
    __syncthreads();
  }
}
