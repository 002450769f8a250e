// tangent_entry.cuh — the tangent of the face Gauss points with one thread per (point,
// neighbour) entry: FP64 mode, and the FP32 tangent of supports too wide for a cell.
// Included by assemble.cu.
//
// The variations of the strains are linear in the five derivatives phi = (dx, dy, dxx, dyy,
// dxy) of a neighbour's shape function, so the block of a local pair (i, j) of one point
// (K_mat + K_geo_m + T12 + T3 of plate/Assembly.h:290-300) is
//     K_ij = sum_a phi_i[a] T_j[a],     T_j[a]: 3x3, a function of neighbour j alone.
// With gJ = a^1 dx_j + a^2 dy_j (a^1, a^2 the dual basis C0^-1 of a1, a2), Bx_k = r_k . a^1 and
// By_k = r_k . a^2 (r_k = r0XX, r0YY, 2 r0XY), and P, Q, c, n the J-side factors of assemble.cu:
//     T[x]  = a1 (x) P0 + a2 (x) P2 - pX gJ (x) b + b (x) (sum_k Bx_k Q_k + bv c0 b - Tu a^1) + n0 I
//     T[y]  = a1 (x) P2 + a2 (x) P1 - pY gJ (x) b + b (x) (sum_k By_k Q_k + bv c1 b - Tu a^2) + n1 I
//     T[xx] = M0 gJ (x) b - b (x) Q0,  T[yy] = M1 gJ (x) b - b (x) Q1,  T[xy] = 2 (M2 gJ (x) b - b (x) Q2),
// all times the Gauss weight. With B = 0, Q_k = qc_k b and the last three are v (x) b: the block
// costs 9 FMA for sum v phi, then 27 for the 3x3, 36 in all (54 with B != 0).
//
// The thread of entry j keeps T_j in registers and takes the local neighbours i = j, j + 1, ...
// (mod n) up to half the list, so each unordered pair is taken once and every lane of a warp
// has work whatever n is.
//
// Bound: the FP64 pipe (2 FMA per cycle and SM). Taking threads per entry and not a warp per
// point fills the chip on small plates and needs no shared-memory records (at 113 neighbours
// they had left one CTA of four warps per SM); 36 FMA per pair replace about 90. Measured on
// one GB300, this kernel alone: 15 x 15 nodes (1,764 points) 1,340 -> 86 us; 61 x 61 nodes with
// the cubic basis (32,400 points, 113 neighbours) 37 -> 13.2 ms; 97 x 97 nodes, 4x4 rule,
// rho = 3.5h (147,456 points) 31 -> 9.2 ms.

// Per-point quantities of the tangent. Bx, By: k = XX, YY, XY (the last doubled).
template <typename TK>
struct Frame {
  TK a1[3], a2[3], b[3], Ax[3], Ay[3], Bx[3], By[3];
  TK C00, C01, C11;
  TK N[3], M[3], pX, pY, bv, W;
};

__device__ __forceinline__ Frame<double> load_frame(const double* st, int64_t stride, int64_t g) {
  Frame<double> f;
  auto S = [&](int k) { return st[k * stride + g]; };
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    f.a1[c] = S(D_A1 + c); f.a2[c] = S(D_A2 + c); f.b[c] = S(D_B + c);
    f.Ax[c] = S(D_AX + c); f.Ay[c] = S(D_AY + c); f.Bx[c] = S(D_BX + c); f.By[c] = S(D_BY + c);
    f.N[c] = S(D_N + c); f.M[c] = S(D_M + c);
  }
  f.C00 = S(D_CI); f.C01 = S(D_CI + 1); f.C11 = S(D_CI + 2);
  f.pX = S(D_P); f.pY = S(D_P + 1); f.bv = S(D_BV); f.W = S(D_W);
  return f;
}

__device__ __forceinline__ Frame<float> load_frame(const float* st, int64_t stride, int64_t g) {
  Frame<float> f;
  auto S = [&](int k) { return st[k * stride + g]; };
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    f.a1[c] = S(S_A1 + c); f.a2[c] = S(S_A2 + c); f.b[c] = S(S_B + c);
    f.N[c] = S(S_N + c); f.M[c] = S(S_M + c);
  }
  f.C00 = S(S_CI); f.C01 = S(S_CI + 1); f.C11 = S(S_CI + 3);
  f.pX = S(S_P); f.pY = S(S_P + 1); f.bv = S(S_BV); f.W = S(S_W);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    f.Ax[c] = f.C00 * f.a1[c] + f.C01 * f.a2[c];
    f.Ay[c] = f.C01 * f.a1[c] + f.C11 * f.a2[c];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int r = k == 0 ? S_RXX : (k == 1 ? S_RYY : S_RXY);
    const float m = k == 2 ? 2.0f : 1.0f;
    const float r0 = S(r), r1 = S(r + 1), r2 = S(r + 2);
    f.Bx[k] = m * (r0 * f.Ax[0] + r1 * f.Ax[1] + r2 * f.Ax[2]);
    f.By[k] = m * (r0 * f.Ay[0] + r1 * f.Ay[1] + r2 * f.Ay[2]);
  }
  return f;
}

// T_j of one neighbour: Tx, Ty row-major 3x3; v[3 a + r] the vectors of T[xx], T[yy], T[xy] on b
// (v (x) b); w the same on the left (b (x) w), B != 0 only.
template <typename TK, bool BZERO>
struct ColumnRecord {
  TK Tx[9], Ty[9], v[9];
  TK w[BZERO ? 1 : 9];
};

template <typename TK, bool BZERO>
__device__ __forceinline__ void column_record(const Frame<TK>& f, const Material& m, TK dx, TK dy, TK dxx, TK dyy,
                                              TK dxy, ColumnRecord<TK, BZERO>& R) {
  const TK be[3] = {f.Bx[0] * dx + f.By[0] * dy - dxx, f.Bx[1] * dx + f.By[1] * dy - dyy,
                    f.Bx[2] * dx + f.By[2] * dy - TK(2) * dxy};
  const TK wx = f.W * dx, wy = f.W * dy;
  TK gW[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) gW[c] = f.Ax[c] * wx + f.Ay[c] * wy;
  const TK cW0 = f.C00 * wx + f.C01 * wy, cW1 = f.C01 * wx + f.C11 * wy;
  const TK nW0 = f.N[0] * wx + f.N[2] * wy, nW1 = f.N[2] * wx + f.N[1] * wy;
  const TK TuW = wx * f.pX + wy * f.pY - f.W * (dxx * f.M[0] + TK(2) * (dxy * f.M[2]) + dyy * f.M[1]);
  TK pa[3], pb[3], qc[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    pa[r] = m.Ai<TK>(3 * r) * wx + m.Ai<TK>(3 * r + 2) * wy;
    pb[r] = m.Ai<TK>(3 * r + 1) * wy + m.Ai<TK>(3 * r + 2) * wx;
    qc[r] = f.W * (m.Di<TK>(3 * r) * be[0] + m.Di<TK>(3 * r + 1) * be[1] + m.Di<TK>(3 * r + 2) * be[2]);
  }
  // The sums on b of the first-derivative parts: b (x) (hx b - TuW a^1 [+ a1, a2 parts]).
  const TK hx = f.Bx[0] * qc[0] + f.Bx[1] * qc[1] + f.Bx[2] * qc[2] + f.bv * cW0;
  const TK hy = f.By[0] * qc[0] + f.By[1] * qc[1] + f.By[2] * qc[2] + f.bv * cW1;
  TK lx[3], ly[3], P0[3], P1[3], P2[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    P0[c] = f.a1[c] * pa[0] + f.a2[c] * pb[0];
    P1[c] = f.a1[c] * pa[1] + f.a2[c] * pb[1];
    P2[c] = f.a1[c] * pa[2] + f.a2[c] * pb[2];
    lx[c] = f.b[c] * hx - TuW * f.Ax[c];
    ly[c] = f.b[c] * hy - TuW * f.Ay[c];
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    R.v[r] = f.M[0] * gW[r] - qc[0] * f.b[r];
    R.v[3 + r] = f.M[1] * gW[r] - qc[1] * f.b[r];
    R.v[6 + r] = TK(2) * (f.M[2] * gW[r] - qc[2] * f.b[r]);
  }
  if constexpr (!BZERO) {   // P_r += b pc_r, Q_r = a1 qa_r + a2 qb_r + b qc_r
    TK Qt[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const TK pc = f.W * (m.Bi<TK>(3 * r) * be[0] + m.Bi<TK>(3 * r + 1) * be[1] + m.Bi<TK>(3 * r + 2) * be[2]);
      const TK qa = m.Bi<TK>(3 * r) * wx + m.Bi<TK>(3 * r + 2) * wy;
      const TK qb = m.Bi<TK>(3 * r + 1) * wy + m.Bi<TK>(3 * r + 2) * wx;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        (r == 0 ? P0 : (r == 1 ? P1 : P2))[c] += f.b[c] * pc;
        Qt[r][c] = f.a1[c] * qa + f.a2[c] * qb;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      lx[c] += f.Bx[0] * Qt[0][c] + f.Bx[1] * Qt[1][c] + f.Bx[2] * Qt[2][c];
      ly[c] += f.By[0] * Qt[0][c] + f.By[1] * Qt[1][c] + f.By[2] * Qt[2][c];
      R.w[c] = -Qt[0][c];
      R.w[3 + c] = -Qt[1][c];
      R.w[6 + c] = TK(-2) * Qt[2][c];
    }
  }
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      R.Tx[3 * r + c] = f.a1[r] * P0[c] + f.a2[r] * P2[c] + f.b[r] * lx[c] - f.pX * gW[r] * f.b[c] + (r == c ? nW0 : TK(0));
      R.Ty[3 * r + c] = f.a1[r] * P2[c] + f.a2[r] * P1[c] + f.b[r] * ly[c] - f.pY * gW[r] * f.b[c] + (r == c ? nW1 : TK(0));
    }
}

__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }

// The block (row i, column j) from phi_i and T_j. Written as chains of FMA: a sum that starts
// from a zeroed K costs a DADD per value on top (20 % of the FP64 instructions of a pair).
template <typename TK, bool BZERO>
__device__ __forceinline__ void form_block(const ColumnRecord<TK, BZERO>& R, const TK* b, TK dx, TK dy, TK dxx, TK dyy,
                                           TK dxy, TK K[9]) {
  TK l[3];
  if constexpr (!BZERO) {
#pragma unroll
    for (int c = 0; c < 3; ++c) l[c] = fma_t(dxy, R.w[6 + c], fma_t(dyy, R.w[3 + c], dxx * R.w[c]));
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const TK s = fma_t(dxy, R.v[6 + r], fma_t(dyy, R.v[3 + r], dxx * R.v[r]));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      TK k = fma_t(s, b[c], fma_t(dy, R.Ty[3 * r + c], dx * R.Tx[3 * r + c]));
      if constexpr (!BZERO) k = fma_t(b[r], l[c], k);
      K[3 * r + c] = k;
    }
  }
}

constexpr int kEntryThreads = 128;

// Entries [ptr[g_begin], ptr[g_end]) of the launch, one per thread, or those of the cells
// glist[0 .. gcount) of 16 points, each with `per_cell` thread blocks; ent_point: the point of
// every entry. A warp's 32 blocks of one step are turned through shared memory, so that a
// block's nine values leave on neighbouring lanes (72 consecutive bytes: 3 sectors instead of
// the 9 of one value per lane and instruction).
// TA: the type of the block accumulator (DET: of the contributions). FP32 blocks go into FP64 sums where every
// entry of the plate comes here. A node's block is the sum of up to 1,000 of them, and added in FP32
// the sums round alike at all nodes of a regular mesh, which adds up over smooth displacements: the
// first steps of a 61 x 61 cubic sheet (rho = 6h) took 10, 14 and 16 corrector iterations, and stalled where the
// points came in ascending order; with FP64 sums 4, 5 and 5, as with an FP64 tangent. K's error
// there 8.3e-7 -> 2.3e-8 of its largest entry, a step 2.55 -> 3.44 ms. Cells too large for a tile
// add to the FP32 sums of the others.
template <typename TK, typename TA, bool DET, bool BZERO>
__global__ void __launch_bounds__(kEntryThreads) face_tangent_entry_kernel(FaceArgs a, const TK* __restrict__ gstate,
                                                                         const int32_t* __restrict__ ent_point,
                                                                         const int32_t* __restrict__ glist, int per_cell) {
  __shared__ TK s_val[kEntryThreads / 32][32 * 9];
  __shared__ int64_t s_at[kEntryThreads / 32][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int gb = a.g_begin, ge = a.g_end, blk = blockIdx.x;
  if (glist) {
    gb = kMG * glist[blockIdx.x / per_cell];
    ge = min(gb + kMG, a.g_end);
    blk = blockIdx.x % per_cell;
  }
  const int64_t e_end = a.ptr[ge];
  const int64_t ew = a.ptr[gb] + static_cast<int64_t>(blk) * kEntryThreads + 32 * w;  // the warp's first
  if (ew >= e_end) return;
  const int64_t e = ew + lane;
  const bool live = e < e_end;
  const int64_t el = live ? e : e_end - 1;
  const int g = ent_point[el];
  const int64_t p0 = a.ptr[g];
  const int n = static_cast<int>(a.ptr[g + 1] - p0);
  const int j = static_cast<int>(el - p0);
  const TK* D1 = static_cast<const TK*>(a.dpsi_t);
  const TK* D2 = static_cast<const TK*>(a.ddpsi_t);
  ColumnRecord<TK, BZERO> R;
  TK b[3];
  {
    const Frame<TK> f = load_frame(gstate, a.n_gp, g);
#pragma unroll
    for (int c = 0; c < 3; ++c) b[c] = f.b[c];
    column_record<TK, BZERO>(f, a.mat, D1[2 * el], D1[2 * el + 1], D2[3 * el], D2[3 * el + 1], D2[3 * el + 2], R);
  }
  const int nj = a.idx[el];
  const int64_t m0 = a.map_ptr[g];
  const int steps = live ? n / 2 + 1 : 0;
  const int wsteps = __reduce_max_sync(0xffffffffu, steps);
  TA* acc = static_cast<TA*>(DET ? a.Kc : a.Kacc);
  constexpr int64_t kStride = (DET || sizeof(TA) == 8) ? 9 : 12;
  TK* sv = s_val[w];
  int64_t* sa = s_at[w];
  for (int d = 0; d < wsteps; ++d) {
    // With n even the last step would meet every pair twice: the lower half takes it.
    const bool on = d < steps && !(2 * d == n && j >= d);
    int64_t at = -1;
    if (on) {
      int i = j + d;
      if (i >= n) i -= n;
      const int64_t ei = p0 + i;
      const int lo = min(i, j), hi = max(i, j);
      const int64_t q = m0 + static_cast<int64_t>(lo) * n - (static_cast<int64_t>(lo) * (lo - 1)) / 2 + (hi - lo);
      at = kStride * (DET ? q : static_cast<int64_t>(a.map_slot[q]));
      TK K[9];
      form_block<TK, BZERO>(R, b, D1[2 * ei], D1[2 * ei + 1], D2[3 * ei], D2[3 * ei + 1], D2[3 * ei + 2], K);
      const int ni = a.idx[ei];
      const bool flip = ni != nj ? ni > nj : i > j;   // the stored block's row is the lower node
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) sv[9 * lane + 3 * r + c] = flip ? K[3 * c + r] : K[3 * r + c];
    }
    sa[lane] = at;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int t = 32 * k + lane, l = t / 9;
      const int64_t to = sa[l];
      if (to >= 0) {
        if constexpr (DET) acc[to + (t - 9 * l)] = sv[t];
        else if constexpr (sizeof(TA) > sizeof(TK)) atomicAdd(acc + to + (t - 9 * l), fp2_widen(sv[t]));
        else atomicAdd(acc + to + (t - 9 * l), sv[t]);
      }
    }
    __syncwarp();
  }
}
