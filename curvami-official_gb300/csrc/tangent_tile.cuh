// tangent_tile.cuh — the FP32 tangent of a cell of 16 consecutive Gauss points with the cell's
// contributions to a block summed in registers. Included by assemble.cu.
//
// One CTA per cell. The block of a pair is sum_a phi_i[a] T_j[a] (tangent_entry.cuh), so over the
// cell's node union the blocks of a node J are products of T_J, one record per point that has J as
// a neighbour, with the derivatives phi of the nodes I <= J. A thread takes J and a tile of four
// consecutive I (an item of tile_prepare) and walks the points they share: it reads T_J (27
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
  const int64_t* item_ptr;
  const uint32_t* item_code;   // points mask | tile << 16 | J << 24
  const int4* item_slot;
  const uint8_t* nbr_u;
  const int16_t* cell_U;       // 32767: direct
  int max_e, max_u;            // most entries and nodes of a cell
  int* err;                    // set to kErrStage when a staging copy never completes
  uint32_t extra_tx;           // 0; the failure-detection test expects bytes that never arrive
  const int32_t* glist;        // the launch's cells glist[0 .. gcount), or every cell of [g_begin, g_end)
  int gcount;
};

constexpr int kTileThreads = 256;
constexpr int kTilePhi = 20;   // floats of a tile: five derivatives of four nodes

// Floats per T_J record: 27 (36 with B != 0) in whole float4 of an odd number, so that records a
// stride apart start in different bank groups.
__host__ __device__ constexpr int tile_rec_floats(bool bzero) { return bzero ? 28 : 36; }

// Dynamic shared memory: records, phi, point states, normals, the (point, node) -> entry table and
// the staging windows of grad / Hessian Phi and the union indices.
inline size_t tile_smem_bytes(int max_e, int max_u, bool bzero) {
  const size_t tiles = (static_cast<size_t>(max_u) + 3) / 4, e = max_e;
  return e * tile_rec_floats(bzero) * sizeof(float) + kMG * tiles * kTilePhi * sizeof(float) +
         kState * kMG * sizeof(float) + kMG * sizeof(float4) + kMG * tiles * 4 * sizeof(uint16_t) +
         (21 * e + 3 * 48);
}

template <bool BZERO, bool DET>
__global__ void __launch_bounds__(kTileThreads, 2) face_tangent_tile_kernel(FaceArgs a, const float* __restrict__ gstate,
                                                                            TileArgs tg) {
  constexpr int RS = tile_rec_floats(BZERO);
  extern __shared__ __align__(16) float tile_smem[];
  __shared__ __align__(8) uint64_t stage_bar;
  __shared__ int64_t sptr[kMG + 1];
  const int t = threadIdx.x;
  const int max_tiles = (tg.max_u + 3) / 4;
  float* rec = tile_smem;                                        // [entry][RS]
  float* phi = rec + static_cast<size_t>(tg.max_e) * RS;         // [point][tile][5][4]
  float* st = phi + kMG * max_tiles * kTilePhi;                  // [kState][kMG]
  float4* nrm = reinterpret_cast<float4*>(st + kState * kMG);    // [point]
  uint16_t* ent = reinterpret_cast<uint16_t*>(nrm + kMG);        // [point][4 max_tiles]
  const size_t at = reinterpret_cast<unsigned char*>(ent + kMG * 4 * max_tiles) - reinterpret_cast<unsigned char*>(tile_smem);
  unsigned char* s_d = reinterpret_cast<unsigned char*>(tile_smem) + ((at + 15) & ~static_cast<size_t>(15));
  unsigned char* s_dd = s_d + ((8 * static_cast<size_t>(tg.max_e) + 47) & ~static_cast<size_t>(15));
  unsigned char* s_u = s_dd + ((12 * static_cast<size_t>(tg.max_e) + 47) & ~static_cast<size_t>(15));
  const unsigned char* dpsi_b = static_cast<const unsigned char*>(a.dpsi_t);
  const unsigned char* ddpsi_b = static_cast<const unsigned char*>(a.ddpsi_t);
  const int G0 = a.g_begin / kMG;
  const int nG = tg.glist ? tg.gcount : (a.g_end + kMG - 1) / kMG - G0;
  auto cell = [&](int gi) { return tg.glist ? tg.glist[gi] : G0 + gi; };
  auto next_from = [&](int gi) {   // the next cell of this CTA that is not direct
    while (gi < nG && tg.cell_U[cell(gi)] > kTileMaxU) gi += gridDim.x;
    return gi;
  };
  // Thread 0 starts the copies of cell G's ranges; every thread later waits on the phase.
  auto stage = [&](int G) {
    const int g0 = G * kMG, g1 = min(g0 + kMG, a.g_end);
    const int64_t q0 = a.ptr[g0], q1 = a.ptr[g1];
    const StageWin wd = stage_window(q0, q1, 8), wdd = stage_window(q0, q1, 12), wu = stage_window(q0, q1, 1);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect(&stage_bar, wd.len + wdd.len + wu.len + tg.extra_tx);
    if (wd.len) bulk_load(s_d, dpsi_b + wd.lo, wd.len, &stage_bar);
    if (wdd.len) bulk_load(s_dd, ddpsi_b + wdd.lo, wdd.len, &stage_bar);
    if (wu.len) bulk_load(s_u, tg.nbr_u + wu.lo, wu.len, &stage_bar);
    // The cell's items are read once per step, from DRAM: into L2 a cell ahead of their use.
    const int64_t i0 = tg.item_ptr[G], i1 = tg.item_ptr[G + 1];
    l2_prefetch(tg.item_code, 4 * i0, 4 * i1);
    l2_prefetch(tg.item_slot, 16 * i0, 16 * i1);
  };
  auto state_of = [&](int G, int i) {
    const int f = i / kMG, k = i - f * kMG, g = G * kMG + k;
    return g < a.g_end ? gstate[static_cast<int64_t>(f) * a.n_gp + g] : 0.0f;
  };
  static_assert(kState * kMG == 2 * kTileThreads, "two state values per thread");
  int gi = next_from(blockIdx.x);
  float s0 = 0.0f, s1 = 0.0f;
  if (gi < nG) { s0 = state_of(cell(gi), t); s1 = state_of(cell(gi), t + kTileThreads); }
  if (t == 0) {
    mbar_init(&stage_bar);
    if (gi < nG) stage(cell(gi));
  }
  __syncthreads();
  uint32_t phase = 0;
  while (gi < nG) {
    const int G = cell(gi);
    const int g0 = G * kMG;
    const int kn = min(kMG, a.g_end - g0);
    const int tiles = (tg.cell_U[G] + 3) >> 2;
    st[t] = s0;
    st[t + kTileThreads] = s1;
    if (t <= kn) sptr[t] = a.ptr[g0 + t];
    for (int i = t; i < kMG * tiles * (kTilePhi / 4); i += kTileThreads)
      reinterpret_cast<float4*>(phi)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int64_t i0 = tg.item_ptr[G];
    const int n_items = static_cast<int>(tg.item_ptr[G + 1] - i0);
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
    const int64_t q0 = sptr[0];
    const int n_ent = static_cast<int>(sptr[kn] - q0);
    const float* sdp = reinterpret_cast<const float*>(s_d + ((q0 * 8) & 15));
    const float* sddp = reinterpret_cast<const float*>(s_dd + ((q0 * 12) & 15));
    const unsigned char* su = s_u + (q0 & 15);
    if (t < kMG) nrm[t] = make_float4(st[S_B * kMG + t], st[(S_B + 1) * kMG + t], st[(S_B + 2) * kMG + t], 0.0f);
    for (int e = t; e < n_ent; e += kTileThreads) {
      int k = 0;   // the last point whose first entry is at or before e
#pragma unroll
      for (int step = 8; step > 0; step >>= 1)
        if (k + step < kn && sptr[k + step] - q0 <= e) k += step;
      const Frame<float> f = load_frame(st, kMG, k);
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
    __syncthreads();
    // The staging windows are free: start the next cell's copies and state loads, which land
    // while this cell's items are summed.
    const int gn = next_from(gi + gridDim.x);
    if (gn < nG) {
      if (t == 0) stage(cell(gn));
      s0 = state_of(cell(gn), t);
      s1 = state_of(cell(gn), t + kTileThreads);
    }
    for (int it = t; it < n_items; it += kTileThreads) {
      const uint32_t code = tg.item_code[i0 + it];
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
        const float4 b4 = nrm[k];
        const float b[3] = {b4.x, b4.y, b4.z};
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
    gi = gn;
  }
}
