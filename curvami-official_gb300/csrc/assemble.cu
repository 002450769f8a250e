// assemble.cu — stage B on sm_103a: the Kirchhoff-Love residual and tangent of every
// face Gauss point, the elastic hinge, and their scatter into the block-upper CSC K.
//
// Reference: NonLinearAssembler::updateStiffness (plate/Assembly.h:158-345),
// Kinematics::compute (plate/Kinematics.h:61-120), Constitutive::evaluate
// (plate/Constitutive.h:57-70), Constraints::evaluateElasticFold / foldAngleAndGrad
// (plate/Constraints.h:54-119, 341-436), Meshless::assembleSystem* (plate/Meshless.h:102-127)
// and the energies (plate/Meshless.h:197-220, Constraints.h:310-339).
//
// A step runs as two kernels: the residual (one Gauss point per thread, FP64: kinematics,
// resultants, nodal forces, and the point's state for the tangent) and the tangent, which forms
// the n(n+1)/2 blocks of every point: per cell of 16 points with the contributions to
// a block summed first (tangent_tile.cuh, FP32), or per (point, neighbour) entry (tangent_entry.cuh:
// FP64, and FP32 supports too wide for a cell). The blocks follow from
//
//     K_IJ = a1 (x) Y1 + a2 (x) Y2 + b (x) Y3 + geo I,
// which follows from Bm_I = a1 (x) (dx, 0, dy) + a2 (x) (0, dy, dx) in strain space,
// Bb_I = beta_I (x) b, Db_J = -(a1 c_J0 + a2 c_J1) (x) b with c_J = C0^-1 grad Phi_J:
//     Y1 = dx_I P_J0 + dy_I P_J2 - Tu_I c_J0 b
//     Y2 = dy_I P_J1 + dx_I P_J2 - Tu_I c_J1 b
//     Y3 = beta_I . Q_J - Tu_J (a1 c_I0 + a2 c_I1) + bv (dPhi_I . c_J) b
//     geo = dPhi_I . N dPhi_J,
// the same terms as K_mat + K_geo_m + T12 + T3 of Assembly.h:290-300. Both kernels sort them by the
// five derivatives of Phi_I, K_IJ = sum_a phi_I[a] T_J[a] (tangent_entry.cuh: 36 FMA per block, 54 with
// B, against the reference's ~90), with the Gauss weight folded into T_J; the entry point on
// caller-owned arrays uses the form above (70 FMA).
//
// Precision modes: FP64 throughout, or "mixed" (FP64 kinematics, resultants and
// residual; the per-neighbour factors and the pair loop in FP32, accumulated into an
// FP32 block array that is widened to FP64 on output, the hinge beside it in FP64; into an FP64 one
// where the supports are too wide for cells).
// Scatter modes: atomics into a block array (BSR, one 3x3 block per pattern slot), or
// deterministic: every block value goes to a contribution array and a second kernel
// sums each block's contributions in ascending Gauss-point order.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <string>
#include <type_traits>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "cgb_pair.cuh"
#include "cgb_umma.cuh"

namespace cgb {
namespace {

constexpr int kFaceWarps = 4;
constexpr int kRecI = 9;   // dx dy beta0 beta1 beta2 Tu g0 g1 g2
constexpr int kRecJ = 23;  // P(9) Q(9) cW0 cW1 nW0 nW1 TuW
constexpr int kRec = kRecI + kRecJ;
// Device error word bit: an index of caller-owned arrays was out of range (allocation-free
// entry point); the access was skipped.
constexpr int kErrIndex = 8;

struct Material {
  double A[9], B[9], D[9];
  bool bzero;   // B == 0: its products are left out
  // FP32 copies for the FP32 tangent: a double -> float conversion issues on the FP64 pipe,
  // which the records loop would otherwise pay for 9-27 times per record.
  float Af[9], Bf[9], Df[9];
  template <class T> __device__ __forceinline__ T Ai(int i) const { if constexpr (sizeof(T) == 4) return Af[i]; else return A[i]; }
  template <class T> __device__ __forceinline__ T Bi(int i) const { if constexpr (sizeof(T) == 4) return Bf[i]; else return B[i]; }
  template <class T> __device__ __forceinline__ T Di(int i) const { if constexpr (sizeof(T) == 4) return Df[i]; else return D[i]; }
};

inline Material make_material(const double* A, const double* B, const double* D) {
  Material m;
  m.bzero = true;
  for (int i = 0; i < 9; ++i) {
    m.bzero = m.bzero && B[i] == 0.0;
    m.A[i] = A[i]; m.B[i] = B[i]; m.D[i] = D[i];
    m.Af[i] = static_cast<float>(A[i]); m.Bf[i] = static_cast<float>(B[i]); m.Df[i] = static_cast<float>(D[i]);
  }
  return m;
}

struct FaceArgs {
  int n_gp;
  int g_begin, g_end;  // the Gauss points [g_begin, g_end) of this launch (multiples of 32 apart)
  int nmax;
  const int64_t* ptr;
  const int32_t* idx;
  const double* dpsi;
  const double* ddpsi;
  const void* dpsi_t;   // grad / Hessian Phi in the tangent's precision (FP32 copies in mixed mode)
  const void* ddpsi_t;
  const double* weight;
  const double* x;
  const int64_t* map_ptr;
  const int32_t* map_slot;
  const int32_t* outer;  // scalar CSC column starts (POS_MAP only)
  // POS_MAP only (caller-owned arrays): the bounds every index is checked against, and
  // the error word that records a violation (the access is skipped).
  int64_t n_blocks;
  int n_nodes;
  int* err;
  // Phase-1 copy of the neighbour data in sliced-ELL order: Gauss point 32 W + l, entry
  // q at sell_ptr[W] + 32 q + l (null: read the CSR arrays).
  const int64_t* sell_ptr;
  const int32_t* sidx;
  const double* sdpsi;
  const double* sddpsi;
  Material mat;
  NatCurv nc;               // natural curvature (inactive by default)
  const double* gp_xy;      // the points' reference coordinates (set when nc is active)
  double* F;         // atomic F (3 n_nodes)
  double* Fc;        // deterministic F contributions (3 per entry)
  void* Kacc;        // atomic block accumulator
  void* Kc;          // deterministic contributions (9 per pair)
  double2* zero;     // the block accumulator, cleared by the launch's residual (null: not)
  int64_t n_zero;
};

// Per-point kinematics and resultants (Kinematics.h:61-120, Constitutive.h:57-70).
struct PointState {
  double a1[3], a2[3], rxx[3], ryy[3], rxy[3], b[3];
  double Ci[4];   // C0^-1 row-major
  double N[3], M[3];
  double pXY[2];
  double bv;
  double e0[3], e1[3];
  double e1el[3];  // elastic bending strain E1_el = E1 + kappa_bar (Voigt), what N and M see
};

// kappa_bar_XX of the natural-curvature band at reference X (plate/Kinematics.h:25-34).
__device__ __forceinline__ double natcurv_kappa(const NatCurv& nc, double X) {
  if (!nc.active) return 0.0;
  const double t = (X - nc.x0) / nc.width;
  return nc.amp * exp(-t * t);
}

// kbar: the natural curvature's kappa_bar_XX at the point (0 without one); it enters E1_el
// only (Kinematics.h:110-111, Constitutive.h:65).
__device__ __forceinline__ void point_state(const double s[15], const Material& m, PointState& P,
                                            double kbar = 0.0) {
  P.a1[0] = 1.0 + s[0]; P.a1[1] = s[1]; P.a1[2] = s[2];
  P.a2[0] = s[3]; P.a2[1] = 1.0 + s[4]; P.a2[2] = s[5];
#pragma unroll
  for (int c = 0; c < 3; ++c) { P.rxx[c] = s[6 + c]; P.ryy[c] = s[9 + c]; P.rxy[c] = s[12 + c]; }
  const double C00 = P.a1[0] * P.a1[0] + P.a1[1] * P.a1[1] + P.a1[2] * P.a1[2];
  const double C11 = P.a2[0] * P.a2[0] + P.a2[1] * P.a2[1] + P.a2[2] * P.a2[2];
  const double C01 = P.a1[0] * P.a2[0] + P.a1[1] * P.a2[1] + P.a1[2] * P.a2[2];
  const double det = C00 * C11 - C01 * C01;
  const double id = 1.0 / det;
  P.Ci[0] = C11 * id; P.Ci[1] = -C01 * id; P.Ci[2] = -C01 * id; P.Ci[3] = C00 * id;
  double n[3] = {P.a1[1] * P.a2[2] - P.a1[2] * P.a2[1], P.a1[2] * P.a2[0] - P.a1[0] * P.a2[2],
                 P.a1[0] * P.a2[1] - P.a1[1] * P.a2[0]};
  const double inv_area = rsqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
#pragma unroll
  for (int c = 0; c < 3; ++c) P.b[c] = n[c] * inv_area;
  P.e0[0] = 0.5 * (C00 - 1.0);
  P.e0[1] = 0.5 * (C11 - 1.0);
  P.e0[2] = 2.0 * (0.5 * C01);
  P.e1[0] = -(P.rxx[0] * P.b[0] + P.rxx[1] * P.b[1] + P.rxx[2] * P.b[2]);
  P.e1[1] = -(P.ryy[0] * P.b[0] + P.ryy[1] * P.b[1] + P.ryy[2] * P.b[2]);
  P.e1[2] = 2.0 * -(P.rxy[0] * P.b[0] + P.rxy[1] * P.b[1] + P.rxy[2] * P.b[2]);
  P.e1el[0] = P.e1[0] + kbar; P.e1el[1] = P.e1[1]; P.e1el[2] = P.e1[2];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    P.N[r] = m.A[3 * r] * P.e0[0] + m.A[3 * r + 1] * P.e0[1] + m.A[3 * r + 2] * P.e0[2];
    P.M[r] = m.D[3 * r] * P.e1el[0] + m.D[3 * r + 1] * P.e1el[1] + m.D[3 * r + 2] * P.e1el[2];
  }
  if (!m.bzero) {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      P.N[r] += m.B[3 * r] * P.e1el[0] + m.B[3 * r + 1] * P.e1el[1] + m.B[3 * r + 2] * P.e1el[2];
      P.M[r] += m.B[r] * P.e0[0] + m.B[3 + r] * P.e0[1] + m.B[6 + r] * P.e0[2];
    }
  }
  double vc[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) vc[c] = P.rxx[c] * P.M[0] + 2.0 * P.rxy[c] * P.M[2] + P.ryy[c] * P.M[1];
  P.bv = P.b[0] * vc[0] + P.b[1] * vc[1] + P.b[2] * vc[2];
  const double fa = P.a1[0] * vc[0] + P.a1[1] * vc[1] + P.a1[2] * vc[2];
  const double fb = P.a2[0] * vc[0] + P.a2[1] * vc[1] + P.a2[2] * vc[2];
  P.pXY[0] = P.Ci[0] * fa + P.Ci[1] * fb;
  P.pXY[1] = P.Ci[2] * fa + P.Ci[3] * fb;
}

// Kinematic sums of one point over its neighbours, the next neighbour's loads in flight while the
// current one is summed; each(entry, u) sees every neighbour's displacement.
template <class Each>
__device__ __forceinline__ void point_sums(int64_t e0, int64_t e1, const int32_t* __restrict__ idx,
                                           const double* __restrict__ dpsi, const double* __restrict__ ddpsi,
                                           const double* __restrict__ x, double s[15], Each&& each) {
#pragma unroll
  for (int k = 0; k < 15; ++k) s[k] = 0.0;
  struct Nb { double u0, u1, u2, dx, dy, dxx, dyy, dxy; };
  auto load = [&](int64_t e, int64_t j) {
    Nb v{};
    if (e < e1) {
      const double2 d = reinterpret_cast<const double2*>(dpsi)[e];
      v = Nb{x[3 * j], x[3 * j + 1], x[3 * j + 2], d.x, d.y, ddpsi[3 * e], ddpsi[3 * e + 1], ddpsi[3 * e + 2]};
    }
    return v;
  };
  auto node = [&](int64_t e) -> int64_t { return e < e1 ? idx[e] : 0; };
  Nb A = load(e0, node(e0));
  int64_t j = node(e0 + 1);
  for (int64_t e = e0; e < e1; ++e) {
    const Nb B = load(e + 1, j);
    j = node(e + 2);
    each(e, A.u0, A.u1, A.u2);
    s[0] += A.u0 * A.dx; s[1] += A.u1 * A.dx; s[2] += A.u2 * A.dx;
    s[3] += A.u0 * A.dy; s[4] += A.u1 * A.dy; s[5] += A.u2 * A.dy;
    s[6] += A.u0 * A.dxx; s[7] += A.u1 * A.dxx; s[8] += A.u2 * A.dxx;
    s[9] += A.u0 * A.dyy; s[10] += A.u1 * A.dyy; s[11] += A.u2 * A.dyy;
    s[12] += A.u0 * A.dxy; s[13] += A.u1 * A.dxy; s[14] += A.u2 * A.dxy;
    A = B;
  }
}

// Scatter of one block into the accumulators. v is row-major in the local (I, J)
// orientation; the stored block is (min node, max node), transposed when flipped.
template <typename TK>
__device__ __forceinline__ void scatter_atomic(void* acc, int32_t slot, bool flip, const TK v[9]);

template <>
__device__ __forceinline__ void scatter_atomic<double>(void* acc, int32_t slot, bool flip, const double v[9]) {
  double* d = static_cast<double*>(acc) + 9 * static_cast<int64_t>(slot);
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) atomicAdd(d + 3 * r + c, flip ? v[3 * c + r] : v[3 * r + c]);
}

template <>
__device__ __forceinline__ void scatter_atomic<float>(void* acc, int32_t slot, bool flip, const float v[9]) {
  // 12 floats per block: three 16-byte vector atomics.
  float4* d = reinterpret_cast<float4*>(static_cast<float*>(acc) + 12 * static_cast<int64_t>(slot));
  float t[9];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) t[3 * r + c] = flip ? v[3 * c + r] : v[3 * r + c];
  atomicAdd(d, make_float4(t[0], t[1], t[2], t[3]));
  atomicAdd(d + 1, make_float4(t[4], t[5], t[6], t[7]));
  atomicAdd(d + 2, make_float4(t[8], 0.0f, 0.0f, 0.0f));
}

template <typename TK>
__device__ __forceinline__ void store_contrib(void* cbuf, int64_t q, bool flip, const TK v[9]) {
  TK* d = static_cast<TK*>(cbuf) + 9 * q;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) d[3 * r + c] = flip ? v[3 * c + r] : v[3 * r + c];
}

// Per-point state handed from the FP64 phase to the pair phase, [field][32] in shared
// memory: a1(3) a2(3) b(3) r0XX(3) r0YY(3) r0XY(3) C0^-1(4) N(3) M(3) pXY(2) bv W.
constexpr int kState = 32;
enum : int { S_A1 = 0, S_A2 = 3, S_B = 6, S_RXX = 9, S_RYY = 12, S_RXY = 15, S_CI = 18, S_N = 22,
             S_M = 25, S_P = 28, S_BV = 30, S_W = 31 };
// The FP64 tangent's state: a1(3) a2(3) b(3), the dual basis a^1(3) a^2(3), r_k . a^1 and
// r_k . a^2 for r_k = r0XX, r0YY, 2 r0XY, C0^-1 (00 01 11), N(3) M(3) pXY(2) bv W. The dual
// basis and its products cost 30 FMA once per point here instead of once per neighbour.
constexpr int kState64 = 34;
enum : int { D_A1 = 0, D_A2 = 3, D_B = 6, D_AX = 9, D_AY = 12, D_BX = 15, D_BY = 18, D_CI = 21, D_N = 24,
             D_M = 27, D_P = 30, D_BV = 32, D_W = 33 };

// TIN: element type of the grad / Hessian Phi arrays the pair phase reads (TK, or FP64
// read and rounded in the kernel). POS_MAP: map_slot holds the reference's csrMapping
// positions and the block slot is outer[3 max(ni, nj)] / 9 + position.
// BZERO: the laminate coupling matrix B is zero (every symmetric laminate, and the
// single isotropic ply of the reference's app, whose B = Q (z1^2 - z0^2) / 2 is exactly
// 0). Then P = A Bm = a1 (x) pa + a2 (x) pb and Q = D Bb = b (x) qc, and the J-side
// record shrinks from 23 to 14 values.
// Phase 1 for one Gauss point: FP64 kinematics,
// resultants and residual (F atomics, or per-entry contributions when DET).
// CHECK (caller-owned arrays only): a neighbour id outside [0, n_nodes) is flagged in the
// error word and the neighbour is left out.
// L lanes share a point (g: this lane's point, sub: its number among them): the neighbours are
// dealt to them in turn, their sums added by shuffles, and put(state, weight) is called by lane 0 of
// them as soon as the point's state is known, before the nodal forces.
// Both neighbour loops hold the next neighbour's loads in flight (and its node's index two ahead)
// while the current one is summed: its 15 FMA take 960 cycles of a quarter's FP64 pipe, about a
// load's latency, so one or two warps per quarter keep the pipe busy.
template <bool DET, bool CHECK, int L, class Put>
__device__ __forceinline__ void phase1_point(const FaceArgs& a, int g, int sub, Put&& put) {
  const Material& m = a.mat;
  const bool here = g < a.g_end;
  if (!here) g = a.g_end - 1;   // lanes past the end keep their warp's shuffles whole and write nothing
  if (!here && L == 1) return;
  const int64_t p0 = a.ptr[g];
  const int n = static_cast<int>(a.ptr[g + 1] - p0);
  // Entry q of this lane's point: CSR p0 + q, or sliced-ELL sb + 32 q (coalesced
  // across the warp: the 32 lanes read 32 consecutive entries per q).
  const bool sell = a.sell_ptr != nullptr;
  const int64_t sb = sell ? a.sell_ptr[g >> 5] + (g & 31) : p0;
  const int64_t stride = sell ? 32 : 1;
  const int32_t* Ix = sell ? a.sidx : a.idx;
  const double* Dp = sell ? a.sdpsi : a.dpsi;
  const double* Ddp = sell ? a.sddpsi : a.ddpsi;
  struct Derivs { double x, y, xx, yy, xy; };
  auto derivs = [&](int q) {
    const int64_t e = sb + q * stride;
    const double2 d = reinterpret_cast<const double2*>(Dp)[e];
    return Derivs{d.x, d.y, Ddp[3 * e], Ddp[3 * e + 1], Ddp[3 * e + 2]};
  };
  auto node = [&](int q) -> int64_t { return q < n ? Ix[sb + q * stride] : 0; };
  auto inside = [&](int64_t j) {   // caller-owned arrays: an index out of range is flagged and skipped
    if (!CHECK || (j >= 0 && j < a.n_nodes)) return true;
    atomicOr(a.err, kErrIndex);
    return false;
  };
  double s[15];
#pragma unroll
  for (int k = 0; k < 15; ++k) s[k] = 0.0;
  {
    struct Nb { Derivs d; double u0, u1, u2; };
    auto load = [&](int q, int64_t j) {
      Nb v{};
      if (q < n && inside(j)) {
        v.d = derivs(q);
        v.u0 = a.x[3 * j]; v.u1 = a.x[3 * j + 1]; v.u2 = a.x[3 * j + 2];
      }
      return v;
    };
    int64_t j = node(sub);
    Nb A = load(sub, j);
    j = node(sub + L);
    for (int q = sub; q < n; q += L) {
      const Nb B = load(q + L, j);
      j = node(q + 2 * L);
      s[0] += A.u0 * A.d.x; s[1] += A.u1 * A.d.x; s[2] += A.u2 * A.d.x;
      s[3] += A.u0 * A.d.y; s[4] += A.u1 * A.d.y; s[5] += A.u2 * A.d.y;
      s[6] += A.u0 * A.d.xx; s[7] += A.u1 * A.d.xx; s[8] += A.u2 * A.d.xx;
      s[9] += A.u0 * A.d.yy; s[10] += A.u1 * A.d.yy; s[11] += A.u2 * A.d.yy;
      s[12] += A.u0 * A.d.xy; s[13] += A.u1 * A.d.xy; s[14] += A.u2 * A.d.xy;
      A = B;
    }
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 15; ++k) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
  PointState P;
  point_state(s, m, P, a.gp_xy ? natcurv_kappa(a.nc, a.gp_xy[2 * static_cast<int64_t>(g)]) : 0.0);
  const double W = a.weight[g];
  if (here && sub == 0) put(P, W);
  // f_I = W (Bm_I^T N + Bb_I^T M) (Assembly.h:249) = W (a1 u1 + a2 u2 + b Tu_I), since
  // beta_I . M = dPhi_I . pXY - (Phi_XX M0 + 2 Phi_XY M2 + Phi_YY M1) = Tu_I, with
  // u1 = Phi_X N0 + Phi_Y N2 and u2 = Phi_Y N1 + Phi_X N2. It is linear in the five
  // derivatives of Phi_I, so per point f_I[c] = Gx[c] Phi_X + Gy[c] Phi_Y + Hxx[c] Phi_XX +
  // Hyy[c] Phi_YY + Hxy[c] Phi_XY: five FP64 FMAs per component and neighbour (GB300's
  // FP64 pipe bounds this kernel).
  double Gx[3], Gy[3], Hxx[3], Hyy[3], Hxy[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    Gx[c] = W * (P.a1[c] * P.N[0] + P.a2[c] * P.N[2] + P.b[c] * P.pXY[0]);
    Gy[c] = W * (P.a1[c] * P.N[2] + P.a2[c] * P.N[1] + P.b[c] * P.pXY[1]);
    Hxx[c] = -W * P.b[c] * P.M[0];
    Hyy[c] = -W * P.b[c] * P.M[1];
    Hxy[c] = -2.0 * W * P.b[c] * P.M[2];
  }
  if (!here) return;
  Derivs A{};
  int64_t jA = node(sub);
  if (sub < n) A = derivs(sub);
  for (int q = sub; q < n; q += L) {
    Derivs B{};
    const int64_t jB = node(q + L);
    if (q + L < n) B = derivs(q + L);
    double f[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] = Gx[c] * A.x + Gy[c] * A.y + Hxx[c] * A.xx + Hyy[c] * A.yy + Hxy[c] * A.xy;
    if (DET) {
#pragma unroll
      for (int c = 0; c < 3; ++c) a.Fc[3 * (p0 + q) + c] = f[c];
    } else if (inside(jA)) {
#pragma unroll
      for (int c = 0; c < 3; ++c) atomicAdd(a.F + 3 * jA + c, f[c]);
    }
    A = B;
    jA = jB;
  }
}

// The state of one point for a tangent kernel, st[field * stride + idx] in its precision.
__device__ __forceinline__ void store_state(const PointState& P, double W, double* st, int64_t stride, int64_t idx) {
  auto put = [&](int f, double v) { st[f * stride + idx] = v; };
  double Ax[3], Ay[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    Ax[c] = P.Ci[0] * P.a1[c] + P.Ci[1] * P.a2[c];
    Ay[c] = P.Ci[2] * P.a1[c] + P.Ci[3] * P.a2[c];
    put(D_A1 + c, P.a1[c]); put(D_A2 + c, P.a2[c]); put(D_B + c, P.b[c]);
    put(D_AX + c, Ax[c]); put(D_AY + c, Ay[c]);
    put(D_N + c, P.N[c]); put(D_M + c, P.M[c]);
  }
  put(D_BX, P.rxx[0] * Ax[0] + P.rxx[1] * Ax[1] + P.rxx[2] * Ax[2]);
  put(D_BX + 1, P.ryy[0] * Ax[0] + P.ryy[1] * Ax[1] + P.ryy[2] * Ax[2]);
  put(D_BX + 2, 2.0 * (P.rxy[0] * Ax[0] + P.rxy[1] * Ax[1] + P.rxy[2] * Ax[2]));
  put(D_BY, P.rxx[0] * Ay[0] + P.rxx[1] * Ay[1] + P.rxx[2] * Ay[2]);
  put(D_BY + 1, P.ryy[0] * Ay[0] + P.ryy[1] * Ay[1] + P.ryy[2] * Ay[2]);
  put(D_BY + 2, 2.0 * (P.rxy[0] * Ay[0] + P.rxy[1] * Ay[1] + P.rxy[2] * Ay[2]));
  put(D_CI, P.Ci[0]); put(D_CI + 1, P.Ci[1]); put(D_CI + 2, P.Ci[3]);
  put(D_P, P.pXY[0]); put(D_P + 1, P.pXY[1]); put(D_BV, P.bv); put(D_W, W);
}
__device__ __forceinline__ void store_state(const PointState& P, double W, float* st, int64_t stride, int64_t idx) {
  auto put = [&](int f, double v) { st[f * stride + idx] = static_cast<float>(v); };
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    put(S_A1 + c, P.a1[c]); put(S_A2 + c, P.a2[c]); put(S_B + c, P.b[c]);
    put(S_RXX + c, P.rxx[c]); put(S_RYY + c, P.ryy[c]); put(S_RXY + c, P.rxy[c]);
    put(S_N + c, P.N[c]); put(S_M + c, P.M[c]);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) put(S_CI + c, P.Ci[c]);
  put(S_P, P.pXY[0]); put(S_P + 1, P.pXY[1]); put(S_BV, P.bv); put(S_W, W);
}

// Phase 2 for the Gauss points g0 .. g0 + 31 across the warp, in the tangent's precision:
// per-neighbour records in shared memory, then the pair loop and the scatter. st holds
// the 32 points' states as [field][32].
template <typename TK, bool DET, typename TIN, bool POS_MAP, bool BZERO>
__device__ __forceinline__ void phase2_group(const FaceArgs& a, int g0, int lane, const TK* st, TK* rec, int* nid) {
  const Material& m = a.mat;
  const int nmax = a.nmax;
  const TIN* dpsi_t = static_cast<const TIN*>(a.dpsi_t);
  const TIN* ddpsi_t = static_cast<const TIN*>(a.ddpsi_t);
  const int kend = min(32, a.g_end - g0);
  for (int k = 0; k < kend; ++k) {
    const int gg = g0 + k;
    const int64_t p0 = a.ptr[gg];
    const int n = static_cast<int>(a.ptr[gg + 1] - p0);
    if (n == 0) continue;  // Assembly.h:208
    if (POS_MAP && n > nmax) {  // the records are staged for nmax neighbours
      if (lane == 0) atomicOr(a.err, kErrIndex);
      continue;
    }
    TK a1t[3], a2t[3], bt[3], rxx[3], ryy[3], rxy[3], Nt[3], Mt[3], Ci[4];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      a1t[c] = st[(S_A1 + c) * 32 + k]; a2t[c] = st[(S_A2 + c) * 32 + k]; bt[c] = st[(S_B + c) * 32 + k];
      rxx[c] = st[(S_RXX + c) * 32 + k]; ryy[c] = st[(S_RYY + c) * 32 + k]; rxy[c] = st[(S_RXY + c) * 32 + k];
      Nt[c] = st[(S_N + c) * 32 + k]; Mt[c] = st[(S_M + c) * 32 + k];
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) Ci[c] = st[(S_CI + c) * 32 + k];
    const TK pX = st[S_P * 32 + k], pY = st[(S_P + 1) * 32 + k];
    const TK bv = st[S_BV * 32 + k], Wt = st[S_W * 32 + k];

    // Records of the neighbours (lane per neighbour).
    for (int i = lane; i < n; i += 32) {
      const int64_t e = p0 + i;
      const TK dx = static_cast<TK>(dpsi_t[2 * e]), dy = static_cast<TK>(dpsi_t[2 * e + 1]);
      const TK dxx = static_cast<TK>(ddpsi_t[3 * e]), dyy = static_cast<TK>(ddpsi_t[3 * e + 1]);
      const TK dxy = static_cast<TK>(ddpsi_t[3 * e + 2]);
      const TK c0 = Ci[0] * dx + Ci[1] * dy;
      const TK c1 = Ci[2] * dx + Ci[3] * dy;
      TK gI[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) gI[r] = a1t[r] * c0 + a2t[r] * c1;
      const TK b0 = -dxx + (rxx[0] * gI[0] + rxx[1] * gI[1] + rxx[2] * gI[2]);
      const TK b1 = -dyy + (ryy[0] * gI[0] + ryy[1] * gI[1] + ryy[2] * gI[2]);
      const TK b2 = TK(2) * (-dxy + (rxy[0] * gI[0] + rxy[1] * gI[1] + rxy[2] * gI[2]));
      const TK Tu = dx * pX + dy * pY - (dxx * Mt[0] + TK(2) * dxy * Mt[2] + dyy * Mt[1]);
      TK* R = rec + i;
      R[0 * nmax] = dx; R[1 * nmax] = dy;
      R[2 * nmax] = b0; R[3 * nmax] = b1; R[4 * nmax] = b2;
      R[5 * nmax] = Tu;
#pragma unroll
      for (int r = 0; r < 3; ++r) R[(6 + r) * nmax] = gI[r];
      if constexpr (BZERO) {
        // J side: pa(3) pb(3) qc(3) cW(2) nW(2) TuW, all times W.
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const TK Ar0 = m.Ai<TK>(3 * r), Ar1 = m.Ai<TK>(3 * r + 1), Ar2 = m.Ai<TK>(3 * r + 2);
          const TK Dr0 = m.Di<TK>(3 * r), Dr1 = m.Di<TK>(3 * r + 1), Dr2 = m.Di<TK>(3 * r + 2);
          R[(kRecI + r) * nmax] = (Ar0 * dx + Ar2 * dy) * Wt;
          R[(kRecI + 3 + r) * nmax] = (Ar1 * dy + Ar2 * dx) * Wt;
          R[(kRecI + 6 + r) * nmax] = (Dr0 * b0 + Dr1 * b1 + Dr2 * b2) * Wt;
        }
        R[(kRecI + 9) * nmax] = c0 * Wt;
        R[(kRecI + 10) * nmax] = c1 * Wt;
        R[(kRecI + 11) * nmax] = (Nt[0] * dx + Nt[2] * dy) * Wt;
        R[(kRecI + 12) * nmax] = (Nt[2] * dx + Nt[1] * dy) * Wt;
        R[(kRecI + 13) * nmax] = Tu * Wt;
      } else {
      // P = A Bm + B Bb, Q = B Bm + D Bb (Assembly.h:255-256), times W:
      //   P(r,c) = a1_c pa_r + a2_c pb_r + b_c pc_r.
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const TK Ar0 = m.Ai<TK>(3 * r), Ar1 = m.Ai<TK>(3 * r + 1), Ar2 = m.Ai<TK>(3 * r + 2);
        const TK Br0 = m.Bi<TK>(3 * r), Br1 = m.Bi<TK>(3 * r + 1), Br2 = m.Bi<TK>(3 * r + 2);
        const TK Dr0 = m.Di<TK>(3 * r), Dr1 = m.Di<TK>(3 * r + 1), Dr2 = m.Di<TK>(3 * r + 2);
        const TK pa = (Ar0 * dx + Ar2 * dy) * Wt;
        const TK pb = (Ar1 * dy + Ar2 * dx) * Wt;
        const TK pc = (Br0 * b0 + Br1 * b1 + Br2 * b2) * Wt;
        const TK qa = (Br0 * dx + Br2 * dy) * Wt;
        const TK qb = (Br1 * dy + Br2 * dx) * Wt;
        const TK qc = (Dr0 * b0 + Dr1 * b1 + Dr2 * b2) * Wt;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          R[(kRecI + 3 * r + c) * nmax] = a1t[c] * pa + a2t[c] * pb + bt[c] * pc;
          R[(kRecI + 9 + 3 * r + c) * nmax] = a1t[c] * qa + a2t[c] * qb + bt[c] * qc;
        }
      }
      R[(kRecI + 18) * nmax] = c0 * Wt;
      R[(kRecI + 19) * nmax] = c1 * Wt;
      R[(kRecI + 20) * nmax] = (Nt[0] * dx + Nt[2] * dy) * Wt;
      R[(kRecI + 21) * nmax] = (Nt[2] * dx + Nt[1] * dy) * Wt;
      R[(kRecI + 22) * nmax] = Tu * Wt;
      }
      nid[i] = a.idx[e];
    }
    __syncwarp();

    // Pair loop: the n(n+1)/2 blocks of this point spread over the lanes.
    const int64_t np = static_cast<int64_t>(n) * (n + 1) / 2;
    const int64_t m0 = a.map_ptr[gg];
    int i = 0, off = lane;
    while (i < n && off >= n - i) { off -= n - i; ++i; }
    for (int64_t p = lane; p < np; p += 32) {
      const int j = i + off;
      const TK* RI = rec + i;
      const TK* RJ = rec + j;
      const TK dxi = RI[0], dyi = RI[nmax], be0 = RI[2 * nmax], be1 = RI[3 * nmax], be2 = RI[4 * nmax];
      const TK Tui = RI[5 * nmax], gi0 = RI[6 * nmax], gi1 = RI[7 * nmax], gi2 = RI[8 * nmax];
      TK v[9];
      if constexpr (BZERO) {
        const TK pa0 = RJ[kRecI * nmax], pa1 = RJ[(kRecI + 1) * nmax], pa2 = RJ[(kRecI + 2) * nmax];
        const TK pb0 = RJ[(kRecI + 3) * nmax], pb1 = RJ[(kRecI + 4) * nmax], pb2 = RJ[(kRecI + 5) * nmax];
        const TK qc0 = RJ[(kRecI + 6) * nmax], qc1 = RJ[(kRecI + 7) * nmax], qc2 = RJ[(kRecI + 8) * nmax];
        const TK cj0 = RJ[(kRecI + 9) * nmax], cj1 = RJ[(kRecI + 10) * nmax];
        const TK nj0 = RJ[(kRecI + 11) * nmax], nj1 = RJ[(kRecI + 12) * nmax];
        const TK TuWj = RJ[(kRecI + 13) * nmax];
        const TK s1 = Tui * cj0, s2 = Tui * cj1;
        const TK geo = dxi * nj0 + dyi * nj1;
        const TK z11 = dxi * pa0 + dyi * pa2, z12 = dxi * pb0 + dyi * pb2;
        const TK z21 = dyi * pa1 + dxi * pa2, z22 = dyi * pb1 + dxi * pb2;
        const TK z33 = be0 * qc0 + be1 * qc1 + be2 * qc2 + bv * (dxi * cj0 + dyi * cj1);
        TK Y1[3], Y2[3], Y3[3];
        const TK gi[3] = {gi0, gi1, gi2};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Y1[c] = a1t[c] * z11 + a2t[c] * z12 - s1 * bt[c];
          Y2[c] = a1t[c] * z21 + a2t[c] * z22 - s2 * bt[c];
          Y3[c] = bt[c] * z33 - TuWj * gi[c];
        }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            v[3 * r + c] = a1t[r] * Y1[c] + a2t[r] * Y2[c] + bt[r] * Y3[c] + (r == c ? geo : TK(0));
      } else {
      const TK cj0 = RJ[(kRecI + 18) * nmax], cj1 = RJ[(kRecI + 19) * nmax];
      const TK nj0 = RJ[(kRecI + 20) * nmax], nj1 = RJ[(kRecI + 21) * nmax];
      const TK TuWj = RJ[(kRecI + 22) * nmax];
      const TK s1 = Tui * cj0, s2 = Tui * cj1;
      const TK t3 = bv * (dxi * cj0 + dyi * cj1);
      const TK geo = dxi * nj0 + dyi * nj1;
      TK Y1[3], Y2[3], Y3[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const TK P0 = RJ[(kRecI + c) * nmax], P1 = RJ[(kRecI + 3 + c) * nmax], P2 = RJ[(kRecI + 6 + c) * nmax];
        const TK Q0 = RJ[(kRecI + 9 + c) * nmax], Q1 = RJ[(kRecI + 12 + c) * nmax], Q2 = RJ[(kRecI + 15 + c) * nmax];
        const TK gic = c == 0 ? gi0 : (c == 1 ? gi1 : gi2);
        Y1[c] = dxi * P0 + dyi * P2 - s1 * bt[c];
        Y2[c] = dyi * P1 + dxi * P2 - s2 * bt[c];
        Y3[c] = be0 * Q0 + be1 * Q1 + be2 * Q2 + t3 * bt[c] - TuWj * gic;
      }
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          v[3 * r + c] = a1t[r] * Y1[c] + a2t[r] * Y2[c] + bt[r] * Y3[c] + (r == c ? geo : TK(0));
      }
      const bool flip = nid[i] > nid[j];
      if (DET) {
        store_contrib<TK>(a.Kc, m0 + p, flip, v);
      } else if (POS_MAP) {
        const int hi = flip ? nid[i] : nid[j];
        const int64_t slot = hi >= 0 && hi < a.n_nodes
                                 ? a.outer[3 * static_cast<int64_t>(hi)] / 9 + a.map_slot[m0 + p] : -1;
        if (slot >= 0 && slot < a.n_blocks) scatter_atomic<TK>(a.Kacc, static_cast<int32_t>(slot), flip, v);
        else atomicOr(a.err, kErrIndex);
      } else {
        scatter_atomic<TK>(a.Kacc, a.map_slot[m0 + p], flip, v);
      }
      off += 32;
      while (i < n && off >= n - i) { off -= n - i; ++i; }
    }
    __syncwarp();
  }
}

template <typename TK, bool DET, bool WANT_K, typename TIN = TK, bool POS_MAP = false, bool BZERO = false>
__global__ void __launch_bounds__(32 * kFaceWarps, sizeof(TK) == 4 ? 5 : 3) face_kernel(FaceArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nmax = a.nmax;
  TK* base_w = reinterpret_cast<TK*>(smem_raw) + static_cast<size_t>(w) * (kState * 32 + kRec * nmax);
  TK* st = base_w;                 // [kState][32]
  TK* rec = base_w + kState * 32;  // [kRec][nmax]
  int* nid = reinterpret_cast<int*>(reinterpret_cast<TK*>(smem_raw) +
                                    static_cast<size_t>(kFaceWarps) * (kState * 32 + kRec * nmax)) + w * nmax;
  // Each warp owns 32 consecutive Gauss points per round.
  for (int g0 = (blockIdx.x * kFaceWarps + w) * 32; g0 < a.n_gp; g0 += gridDim.x * kFaceWarps * 32) {
    // Phase 1: one Gauss point per lane, FP64. Every lane does distinct work, so no FP64
    // issue slot is spent on a redundant or masked copy (on GB300 an FP64 warp
    // instruction costs the same with 1 or 32 lanes).
    phase1_point<DET, POS_MAP, 1>(a, g0 + lane, 0, [&](const PointState& P, double W) {
      if (WANT_K) store_state(P, W, st, 32, lane);
    });
    if (!WANT_K) continue;
    __syncwarp();
    phase2_group<TK, DET, TIN, POS_MAP, BZERO>(a, g0, lane, st, rec, nid);
  }
}

// The same work as two kernels, each sized for its own occupancy: the residual kernel
// (phase 1, one Gauss point per thread, FP64 bound) writes the per-point state to
// global memory ([field][n_gp]); the tangent kernel (phase 2) stages 32 points' states
// in shared memory and runs the pair loop.
// Work is handed out a warp's points at a time from a counter (zeroed per assembly), so the
// warps of a launch finish together whatever the grid: when the tangent kernel of the
// previous chunk holds most of each SM, only one residual CTA fits beside it, and a
// fixed split into CTAs would leave a partial last wave.
// LANES per point: each SM quarter issues one FP64 warp instruction in 64 cycles, and a point
// takes about 30 per neighbour and 200 by itself, so a launch that does not fill the quarters
// is as long as one warp's work; splitting the points' neighbours over lanes shortens it
// (residual_lanes).
template <typename TK, bool DET, bool STORE, int LANES>
__global__ void __launch_bounds__(256) face_residual_kernel(FaceArgs a, TK* gstate, int* __restrict__ work) {
  constexpr int PTS = 32 / LANES;
  const int lane = threadIdx.x & 31;
  // The first residual of a step clears the block accumulator that the tangent and the hinge add
  // into after it: stores beside FP64 work, and a launch less (15 x 15 nodes: step 166.8 -> 162.6 us).
  // Cleared on the tangent's stream instead, a captured step of 600,000 points took 5.66 ms, not 4.56.
  if (STORE && !DET && a.zero)
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < a.n_zero;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
      a.zero[i] = make_double2(0.0, 0.0);
  for (;;) {
    int unit = 0;
    if (lane == 0) unit = atomicAdd(work, 1);
    unit = __shfl_sync(0xffffffffu, unit, 0);
    const int64_t g0 = a.g_begin + PTS * static_cast<int64_t>(unit);
    if (g0 >= a.g_end) break;
    const int g = static_cast<int>(g0) + lane / LANES;
    phase1_point<DET, false, LANES>(a, g, lane % LANES, [&](const PointState& P, double W) {
      if (STORE) store_state(P, W, gstate, a.n_gp, g);
    });
  }
}

// Lanes per point of a residual launch over n points: as many as still leave every warp an SM
// quarter of its own. At 28 neighbours one warp's work is 1070 FP64 instructions with one lane
// per point, 665 with two, 470 with four and 380 with eight; once two warps share a quarter the
// fewer lanes win again (the point's own part is repeated by each). One in deterministic mode: a
// point's sums then do not depend on how many points the launch has.
inline int residual_lanes(int n, int sms, bool det) {
  if (det) return 1;
  const int64_t lanes = 32LL * 4 * sms;
  return n * 8LL <= lanes ? 8 : n * 4LL <= lanes ? 4 : n * 2LL <= lanes ? 2 : 1;
}

constexpr int kMG = 16;   // points per cell of the FP32 tangent (the set-up kernel uses the same)

#include "tangent_entry.cuh"

// ---- hinge (FP64) -----------------------------------------------------------------

struct HingeArgs {
  int n_gp;
  int max_u;
  const int64_t* lptr; const int32_t* lidx; const double* ldpsi;
  const int64_t* rptr; const int32_t* ridx; const double* rdpsi;
  const double* weight; const double* tangent;
  double Kt, theta0;
  const double* theta0_gp; const int8_t* active;
  const int64_t* u_ptr; const int32_t* u_node; const int32_t* l_pos; const int32_t* r_pos;
  const int64_t* pair_ptr; const int32_t* pair_slot;
  const double* x;
  int exact;
  int want_K;
  int parts;         // warps per crease point
  double* F; double* Kacc;            // atomic mode: Kacc by pair_slot
  double* Fc; double* Kc;             // deterministic mode
  int64_t f_base, k_base;             // contribution id offsets of this fold
};

__device__ __forceinline__ void cross(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ double dot(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// Constraints::foldAngleAndGrad (plate/Constraints.h:54-119): theta = atan2(-s, c) with
// c = bL . bR, s = (bL x bR) . t. The gradient is taken backwards: w_L, w_R, w_t are the
// cofactors of dbL, dbR, dt in dtheta = -(c ds - s dc) / (c^2 + s^2); through b = n / |n| and
// n = a1 x a2 a cofactor w of db becomes m = (w - (w . b) b) / |n| and then a2 x m on a1 and
// m x a1 on a2. About 150 FP64 operations, a sixth of forming the 3x6 derivative matrices
// (one warp's latency, which is what a hinge launch of a few crease points is made of).
__device__ double fold_angle(const double* F, double tx, double ty, double* grad) {
  const double *a1L = F, *a2L = F + 3, *a1R = F + 6, *a2R = F + 9;
  double nL[3], nR[3];
  cross(a1L, a2L, nL); cross(a1R, a2R, nR);
  const double iL = rsqrt(dot(nL, nL)), iR = rsqrt(dot(nR, nR));
  double bL[3], bR[3], aT[3], t[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) { bL[c] = nL[c] * iL; bR[c] = nR[c] * iR; aT[c] = a1L[c] * tx + a2L[c] * ty; }
  const double iT = rsqrt(dot(aT, aT));
#pragma unroll
  for (int c = 0; c < 3; ++c) t[c] = aT[c] * iT;
  const double cth = dot(bL, bR);
  double bxb[3];
  cross(bL, bR, bxb);
  const double sth = dot(bxb, t);
  if (grad) {
    double bRxt[3], txbL[3];
    cross(bR, t, bRxt); cross(t, bL, txbL);
    const double denom = cth * cth + sth * sth;
    const double inv = (denom > 1e-14) ? 1.0 / denom : 0.0;
    const double ci = -cth * inv, si = sth * inv;
    double mL[3], mR[3], mT[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      mL[c] = ci * bRxt[c] + si * bR[c];
      mR[c] = ci * txbL[c] + si * bL[c];
      mT[c] = ci * bxb[c];
    }
    const double pL = dot(mL, bL), pR = dot(mR, bR), pT = dot(mT, t);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      mL[c] = (mL[c] - pL * bL[c]) * iL;
      mR[c] = (mR[c] - pR * bR[c]) * iR;
      mT[c] = (mT[c] - pT * t[c]) * iT;
    }
    cross(a2L, mL, grad); cross(mL, a1L, grad + 3);
    cross(a2R, mR, grad + 6); cross(mR, a1R, grad + 9);
#pragma unroll
    for (int c = 0; c < 3; ++c) { grad[c] += tx * mT[c]; grad[3 + c] += ty * mT[c]; }
  }
  return atan2(-sth, cth);
}

constexpr int kHingeWarps = 2;

// One warp per crease Gauss point (Constraints.h:349-435). The left and right
// entries are merged per node: with G_u = sum of the dof gradients of node u over both
// sides, the reference's triplets (all k, m with node_k <= node_m) sum to
// W Kt G_P (x) G_Q (+ W moment B_P^T H B_Q) on block (P, Q) of the merged list. a.parts warps
// share a point's pairs (each repeats the angle): a crease has few points, and with one warp
// each a merged list of 160 nodes is 400 rounds of about 200 FP64 instructions.
__global__ void __launch_bounds__(32 * kHingeWarps) hinge_kernel(HingeArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Per warp: G[3*max_u], Bsum[4*max_u], H[144] (+16 spare).
  double* base = reinterpret_cast<double*>(smem_raw) + static_cast<size_t>(w) * (7 * a.max_u + 144 + 16);
  double* G = base;
  double* Bs = base + 3 * a.max_u;
  double* H = base + 7 * a.max_u;
  const int gw = blockIdx.x * kHingeWarps + w;
  const int g = gw / a.parts, part = gw - g * a.parts;
  if (g < a.n_gp) {
    if (a.active && a.active[g] == 0) return;  // Constraints.h:350
    double sL[6] = {0, 0, 0, 0, 0, 0}, sR[6] = {0, 0, 0, 0, 0, 0};
    for (int64_t e = a.lptr[g] + lane; e < a.lptr[g + 1]; e += 32) {
      const int64_t j = a.lidx[e];
      const double dX = a.ldpsi[2 * e], dY = a.ldpsi[2 * e + 1];
      for (int c = 0; c < 3; ++c) { sL[c] += a.x[3 * j + c] * dX; sL[3 + c] += a.x[3 * j + c] * dY; }
    }
    for (int64_t e = a.rptr[g] + lane; e < a.rptr[g + 1]; e += 32) {
      const int64_t j = a.ridx[e];
      const double dX = a.rdpsi[2 * e], dY = a.rdpsi[2 * e + 1];
      for (int c = 0; c < 3; ++c) { sR[c] += a.x[3 * j + c] * dX; sR[3 + c] += a.x[3 * j + c] * dY; }
    }
    double F12[12];
    for (int k = 0; k < 6; ++k) { F12[k] = warp_sum(sL[k]); F12[6 + k] = warp_sum(sR[k]); }
    F12[0] += 1.0; F12[4] += 1.0; F12[6] += 1.0; F12[10] += 1.0;
    const double tx = a.tangent[2 * g], ty = a.tangent[2 * g + 1];
    double grad[12];
    const double theta = fold_angle(F12, tx, ty, grad);
    const double th0 = a.theta0_gp ? a.theta0_gp[g] : a.theta0;
    const double W = a.weight[g];
    const double Wm = W * (a.Kt * (theta - th0));
    const double WK = W * a.Kt;
    const bool use_hess = a.exact && a.want_K && fabs(Wm) > 0.0;
    if (use_hess) {
      // Central differences of the analytic gradient (Constraints.h:402-413), one
      // perturbed evaluation per lane (24 lanes), then symmetrised.
      double mx = 0.0;
      for (int k = 0; k < 12; ++k) mx = fmax(mx, fabs(F12[k]));
      const double hs = 1e-6 * fmax(1.0, mx);
      if (lane < 24) {
        const int k = lane >> 1;
        double Fp[12];
        for (int q = 0; q < 12; ++q) Fp[q] = F12[q];
        Fp[k] += (lane & 1) ? -hs : hs;
        double gp[12];
        fold_angle(Fp, tx, ty, gp);
        // H[r][k] = (g+ - g-)/(2h): the '+' lane stores g+, the '-' lane subtracts it.
        if ((lane & 1) == 0) for (int r = 0; r < 12; ++r) H[r * 12 + k] = gp[r];
        __syncwarp(0x00ffffffu);
        if (lane & 1) for (int r = 0; r < 12; ++r) H[r * 12 + k] = (H[r * 12 + k] - gp[r]) / (2.0 * hs);
      }
      __syncwarp();
      if (lane < 12) {
        double row[12];
        for (int c = 0; c < 12; ++c) row[c] = 0.5 * (H[lane * 12 + c] + H[c * 12 + lane]);
        __syncwarp(0x00000fffu);
        for (int c = 0; c < 12; ++c) H[lane * 12 + c] = row[c];
      }
      __syncwarp();
    }
    // Per merged node: G_u (3) and the summed (dX, dY) of each side (4).
    const int64_t u0 = a.u_ptr[g];
    const int mu = static_cast<int>(a.u_ptr[g + 1] - u0);
    for (int u = lane; u < mu; u += 32) {
      G[3 * u] = 0.0; G[3 * u + 1] = 0.0; G[3 * u + 2] = 0.0;
      Bs[4 * u] = 0.0; Bs[4 * u + 1] = 0.0; Bs[4 * u + 2] = 0.0; Bs[4 * u + 3] = 0.0;
    }
    __syncwarp();
    // Left then right: within a side every node occurs once, so no two lanes collide.
    for (int64_t e = a.lptr[g] + lane; e < a.lptr[g + 1]; e += 32) {
      const int u = a.l_pos[e];
      const double dX = a.ldpsi[2 * e], dY = a.ldpsi[2 * e + 1];
      for (int d = 0; d < 3; ++d) G[3 * u + d] += grad[d] * dX + grad[d + 3] * dY;
      Bs[4 * u] += dX; Bs[4 * u + 1] += dY;
    }
    __syncwarp();
    for (int64_t e = a.rptr[g] + lane; e < a.rptr[g + 1]; e += 32) {
      const int u = a.r_pos[e];
      const double dX = a.rdpsi[2 * e], dY = a.rdpsi[2 * e + 1];
      for (int d = 0; d < 3; ++d) G[3 * u + d] += grad[6 + d] * dX + grad[9 + d] * dY;
      Bs[4 * u + 2] += dX; Bs[4 * u + 3] += dY;
    }
    __syncwarp();
    for (int u = part == 0 ? lane : mu; u < mu; u += 32) {
      const int node = a.u_node[u0 + u];
      for (int d = 0; d < 3; ++d) {
        const double f = G[3 * u + d] * Wm;
        if (a.Fc) a.Fc[3 * (a.f_base + u0 + u) + d] = f;
        else atomicAdd(a.F + 3 * static_cast<int64_t>(node) + d, f);
      }
    }
    if (a.want_K) {
      const int64_t np = static_cast<int64_t>(mu) * (mu + 1) / 2;
      const int64_t q0 = a.pair_ptr[g];
      int P = 0, off = 32 * part + lane;
      while (P < mu && off >= mu - P) { off -= mu - P; ++P; }
      for (int64_t p = 32 * part + lane; p < np; p += 32 * a.parts) {
        const int Q = P + off;
        double v[9];
        for (int dk = 0; dk < 3; ++dk)
          for (int dm = 0; dm < 3; ++dm) {
            double val = WK * (G[3 * P + dk] * G[3 * Q + dm]);
            if (use_hess) {
              // B_P(dk) has dX_L at dk, dY_L at dk+3, dX_R at 6+dk, dY_R at 9+dk.
              const int ik[4] = {dk, dk + 3, 6 + dk, 9 + dk};
              const int im[4] = {dm, dm + 3, 6 + dm, 9 + dm};
              double hb = 0.0;
              for (int s1 = 0; s1 < 4; ++s1) {
                double row = 0.0;
                for (int s2 = 0; s2 < 4; ++s2) row += H[ik[s1] * 12 + im[s2]] * Bs[4 * Q + s2];
                hb += Bs[4 * P + s1] * row;
              }
              val += Wm * hb;
            }
            v[3 * dk + dm] = val;
          }
        if (a.Kc) store_contrib<double>(a.Kc, a.k_base + q0 + p, false, v);
        else scatter_atomic<double>(a.Kacc, a.pair_slot[q0 + p], false, v);
        off += 32 * a.parts;
        while (P < mu && off >= mu - P) { off -= mu - P; ++P; }
      }
    }
  }
}

// ---- output: blocks -> the reference's CSC -------------------------------------------
// An entry as the double that K holds.
__device__ __forceinline__ double widen(float v) { return fp2_widen(v); }
__device__ __forceinline__ double widen(double v) { return v; }

// The hinge's blocks of the mixed mode, in FP64 apart from the FP32 accumulator: those of column
// j are [ptr[j], ptr[j + 1]), each at block row pos of the column. In the FP32 accumulator they
// would round whatever is added after them at their own size: on a plate of 41 x 41 nodes a
// hinge entry is a hundred times the plate's bending entries beside the crease.
struct HingeBlocks {
  const int64_t* ptr;    // null: none
  const int32_t* pos;
  const double* acc;     // 9 per block
};

// Column node j holds len_j block rows; scalar column 3j+c starts at 9 col_ptr[j] +
// 3 c len_j and lists rows 3i+r for the block rows i ascending (Assembly.h:103-107).
template <typename TA, int STRIDE>
__global__ void blocks_to_csc(int n_nodes, const int64_t* __restrict__ col_ptr, const TA* __restrict__ acc,
                              HingeBlocks hinge, double* K) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t j = warp; j < n_nodes; j += nw) {
    const int64_t b0 = col_ptr[j];
    const int len = static_cast<int>(col_ptr[j + 1] - b0);
    double* col = K + 9 * b0;
    for (int t = lane; t < 9 * len; t += 32) {
      // t enumerates the column's output in storage order: c major, then (pos, r).
      const int c = t / (3 * len), rem = t - c * 3 * len, pos = rem / 3, r = rem - 3 * pos;
      col[t] = widen(acc[(b0 + pos) * STRIDE + 3 * r + c]);
    }
    if (!hinge.ptr) continue;
    const int64_t h0 = hinge.ptr[j];
    const int nh = 9 * static_cast<int>(hinge.ptr[j + 1] - h0);
    __syncwarp();   // the column's other lanes have stored it
    for (int t = lane; t < nh; t += 32) {
      const int q = t / 9, k = t - 9 * q, r = k / 3, c = k - 3 * r;
      col[3 * c * len + 3 * hinge.pos[h0 + q] + r] += hinge.acc[9 * h0 + t];
    }
  }
}

// The same output step with the block columns taken from the scalar CSC outer index:
// column node j starts at block outer[3j] / 9 and holds (outer[3j+1] - outer[3j]) / 3 blocks.
// A column whose blocks would fall outside [0, n_blocks) is skipped and flagged.
template <typename TA, int STRIDE>
__global__ void blocks_to_csc_outer(int n_nodes, int64_t n_blocks, const int32_t* __restrict__ outer,
                                    const TA* __restrict__ acc, double* __restrict__ K, int* err) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t j = warp; j < n_nodes; j += nw) {
    const int64_t o = outer[3 * j];
    const int64_t b0 = o / 9;
    const int len = (outer[3 * j + 1] - outer[3 * j]) / 3;
    if (o < 0 || o % 9 != 0 || len < 0 || b0 + len > n_blocks) {
      if (lane == 0) atomicOr(err, kErrIndex);
      continue;
    }
    double* col = K + o;
    for (int t = lane; t < 9 * len; t += 32) {
      const int c = t / (3 * len), rem = t - c * 3 * len, pos = rem / 3, r = rem - 3 * pos;
      col[t] = widen(acc[(b0 + pos) * STRIDE + 3 * r + c]);
    }
  }
}

// Deterministic: each block sums its contributions in ascending id order. Nine lanes take one
// block, an entry each, so a contribution is one read of 9 consecutive values and the loads of
// kReduceAhead contributions are in flight before the first is added; a block of threads takes a
// column. 430,000 FP32 blocks of 9 contributions (87 x 87 nodes) with det_reduce_F: 202 -> 108 us;
// a lane per block had nine separate loads for each contribution, 36 bytes apart between the lanes.
// 12 or 16 contributions ahead, or the next block's range fetched early: 115-120 us.
// With face_end the units from there on are the hinge's (from n_face on), in FP64 in an array of their
// own, and are summed apart.
constexpr int kReduceThreads = 128;   // 14 blocks at a time
constexpr int kReduceAhead = 8;
// TWO (FP32 pair units): the sum in two floats. A node's block is the sum of as many units as points
// share it, 1,000 for the cubic basis at rho = 6h; added in one float in the same order at every node
// of a regular mesh their rounding errors are alike, and a mixed path of 61 x 61 nodes stalled on it.
// K's error there 8.5e-7 -> 2.3e-8 of its largest entry, first steps in 4 and 5 iterations like FP64's.
// The units of cells are a tenth as many: 87 x 87 nodes 562 us a step, with two floats 588.
template <typename TC, bool TWO>
__global__ void __launch_bounds__(kReduceThreads) det_reduce_blocks(int n_nodes, const int64_t* __restrict__ col_ptr,
                                                                    const int64_t* __restrict__ lptr,
                                                                    const int64_t* __restrict__ list,
                                                                    const TC* __restrict__ contrib,
                                                                    const int64_t* __restrict__ face_end, int64_t n_face,
                                                                    const double* __restrict__ hinge,
                                                                    double* __restrict__ K) {
  constexpr int kGroups = kReduceThreads / 9;
  const int group = threadIdx.x / 9, k = threadIdx.x - 9 * group;
  const int r = k / 3, c = k - 3 * r;
  if (group >= kGroups) return;
  for (int j = blockIdx.x; j < n_nodes; j += gridDim.x) {
    const int64_t b0 = col_ptr[j];
    const int len = static_cast<int>(col_ptr[j + 1] - b0);
    double* col = K + 9 * b0;
    for (int pos = group; pos < len; pos += kGroups) {
      const int64_t end = face_end ? face_end[b0 + pos] : lptr[b0 + pos + 1];
      TC s = TC(0), lo = TC(0);
      for (int64_t q = lptr[b0 + pos]; q < end; q += kReduceAhead) {
        TC v[kReduceAhead];
#pragma unroll
        for (int i = 0; i < kReduceAhead; ++i) v[i] = q + i < end ? contrib[9 * list[q + i] + k] : TC(0);
#pragma unroll
        for (int i = 0; i < kReduceAhead; ++i)
          if (q + i < end) {
            if constexpr (TWO) {   // what the sum rounds off, in lo
              const TC t = __fadd_rn(s, v[i]), d = __fsub_rn(t, s);
              lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(s, __fsub_rn(t, d)), __fsub_rn(v[i], d)));
              s = t;
            } else {
              s += v[i];
            }
          }
      }
      double sum = widen(s);
      if (TWO) sum += widen(lo);
      if (face_end) {
        double h = 0.0;
        const int64_t last = lptr[b0 + pos + 1];
#pragma unroll 4
        for (int64_t q = end; q < last; ++q) h += hinge[9 * (list[q] - n_face) + k];
        if (end < last) sum += h;
      }
      col[3 * c * len + 3 * pos + r] = sum;
    }
  }
}

// Deterministic F: a warp per node fetches its contributions, kFetch at a time; then one warp adds
// for all ten nodes of the block, a lane per node and component, in ascending id order. An FP64
// addition occupies an SM quarter for the same time with one lane or with 32: a warp per node that also added took 128 us for 7,569 nodes of
// 270 contributions.
constexpr int kReduceNodes = 10, kFetch = 128;
__global__ void __launch_bounds__(32 * kReduceNodes) det_reduce_F(int n_nodes, const int64_t* __restrict__ lptr,
                                                                  const int64_t* __restrict__ list,
                                                                  const double* __restrict__ fc,
                                                                  double* __restrict__ F) {
  __shared__ double s_v[3 * kReduceNodes][kFetch + 1];   // + 1: the adding lanes' rows in different banks
  __shared__ int s_n[kReduceNodes];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * kReduceNodes + w;
  int64_t q = j < n_nodes ? lptr[j] : 0;
  const int64_t end = j < n_nodes ? lptr[j + 1] : 0;
  double v[kFetch / 32][3];
  auto fetch = [&]() {
#pragma unroll
    for (int i = 0; i < kFetch / 32; ++i) {
      if (q + 32 * i + lane >= end) continue;
      const double* f = fc + 3 * list[q + 32 * i + lane];
      v[i][0] = f[0]; v[i][1] = f[1]; v[i][2] = f[2];
    }
  };
  const int row = min(static_cast<int>(threadIdx.x), 3 * kReduceNodes - 1);   // of the adding lane
  double s = 0.0;
  fetch();
  while (__syncthreads_or(q < end)) {
#pragma unroll
    for (int i = 0; i < kFetch / 32; ++i)
      for (int c = 0; c < 3; ++c) s_v[3 * w + c][32 * i + lane] = v[i][c];
    if (lane == 0) s_n[w] = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(kFetch), end - q)));
    __syncthreads();
    q += kFetch;
    fetch();
    if (w == 0) {
      const int n = s_n[row / 3];
      for (int i = 0; i < n; ++i) s += s_v[row][i];
    }
  }
  const int node = blockIdx.x * kReduceNodes + row / 3;
  if (threadIdx.x < 3 * kReduceNodes && node < n_nodes) F[3 * static_cast<int64_t>(blockIdx.x) * kReduceNodes + row] = s;
}

// ---- energies -----------------------------------------------------------------------
// One point per thread: the point's own part (about 150 FP64 operations) on all lanes of a warp
// with work of their own. A warp per point had issued it, and 75 additions of the lanes' sums, for
// one point at a time: 57,600 points 560 us.
__global__ void __launch_bounds__(128) face_energy_kernel(int n_gp, const int64_t* __restrict__ ptr,
                                                          const int32_t* __restrict__ idx,
                                                          const double* __restrict__ dpsi,
                                                          const double* __restrict__ ddpsi,
                                                          const double* __restrict__ weight,
                                                          const double* __restrict__ x, Material m,
                                                          NatCurv nc, const double* __restrict__ gp_xy, double* out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  double em = 0.0, eb = 0.0;
  if (g < n_gp) {
    double s[15];
    point_sums(ptr[g], ptr[g + 1], idx, dpsi, ddpsi, x, s, [](int64_t, double, double, double) {});
    PointState P;
    point_state(s, m, P, gp_xy ? natcurv_kappa(nc, gp_xy[2 * static_cast<int64_t>(g)]) : 0.0);
    // Meshless.h:204-220, with E1_el (Meshless.h:212)
    em = 0.5 * weight[g] * (P.e0[0] * P.N[0] + P.e0[1] * P.N[1] + P.e0[2] * P.N[2]);
    eb = 0.5 * weight[g] * (P.e1el[0] * P.M[0] + P.e1el[1] * P.M[1] + P.e1el[2] * P.M[2]);
  }
  em = warp_sum(em);
  eb = warp_sum(eb);
  if ((threadIdx.x & 31) == 0) { atomicAdd(out, em); atomicAdd(out + 1, eb); }
}

// ---- kinematic state of arbitrary points (post-processing) ---------------------------
// One thread per point: the displacement sum_I Psi_I u_I and Kinematics::compute /
// Constitutive::evaluate (plate/Kinematics.h:61-120, Constitutive.h:57-70) in FP64, one row
// of kPointStateCols per point: u(3) r_X(3) r_Y(3) r_XX(3) r_YY(3) r_XY(3) b(3)
// E0 (xx yy xy, tensor) E1 (xx yy xy, tensor) N (Voigt) M (Voigt).
constexpr int kPointStateCols = 33;
__global__ void __launch_bounds__(128) point_state_kernel(int n, const int64_t* __restrict__ ptr,
                                                          const int32_t* __restrict__ idx,
                                                          const double* __restrict__ psi,
                                                          const double* __restrict__ dpsi,
                                                          const double* __restrict__ ddpsi,
                                                          const double* __restrict__ x, Material m,
                                                          NatCurv nc, const double* __restrict__ gp_xy,
                                                          double* __restrict__ out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  double s[15], u[3] = {0.0, 0.0, 0.0};
  point_sums(ptr[g], ptr[g + 1], idx, dpsi, ddpsi, x, s, [&](int64_t e, double u0, double u1, double u2) {
    const double p = psi[e];
    u[0] += p * u0; u[1] += p * u1; u[2] += p * u2;
  });
  PointState P;
  point_state(s, m, P, gp_xy ? natcurv_kappa(nc, gp_xy[2 * static_cast<int64_t>(g)]) : 0.0);
  double* o = out + static_cast<int64_t>(g) * kPointStateCols;
  for (int c = 0; c < 3; ++c) {
    o[c] = u[c];
    o[3 + c] = P.a1[c]; o[6 + c] = P.a2[c];
    o[9 + c] = P.rxx[c]; o[12 + c] = P.ryy[c]; o[15 + c] = P.rxy[c];
    o[18 + c] = P.b[c];
    o[27 + c] = P.N[c]; o[30 + c] = P.M[c];
  }
  o[21] = P.e0[0]; o[22] = P.e0[1]; o[23] = 0.5 * P.e0[2];
  o[24] = P.e1[0]; o[25] = P.e1[1]; o[26] = 0.5 * P.e1[2];
}

// One warp per crease point, the neighbours dealt to its lanes.
__global__ void __launch_bounds__(128) hinge_energy_kernel(HingeArgs a, double* out) {
  const int lane = threadIdx.x & 31;
  const int g = static_cast<int>((blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5);
  if (g >= a.n_gp || (a.active && a.active[g] == 0)) return;
  double F12[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int64_t* ptr = side ? a.rptr : a.lptr;
    const int32_t* idx = side ? a.ridx : a.lidx;
    const double* d = side ? a.rdpsi : a.ldpsi;
    for (int64_t e = ptr[g] + lane; e < ptr[g + 1]; e += 32) {
      const int64_t j = idx[e];
      const double dX = d[2 * e], dY = d[2 * e + 1];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double u = a.x[3 * j + c];
        F12[6 * side + c] += u * dX;
        F12[6 * side + 3 + c] += u * dY;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 12; ++k) F12[k] = warp_sum(F12[k]);
  F12[0] += 1.0; F12[4] += 1.0; F12[6] += 1.0; F12[10] += 1.0;
  const double theta = fold_angle(F12, a.tangent[2 * g], a.tangent[2 * g + 1], nullptr);
  const double th0 = a.theta0_gp ? a.theta0_gp[g] : a.theta0;
  const double d = theta - th0;
  if (lane == 0) atomicAdd(out, a.weight[g] * (0.5 * a.Kt * (d * d)));
}

// ---- bulk-copy (TMA) staging --------------------------------------------------------
// One elected thread copies a group's contiguous ranges of grad / Hessian Phi and ids
// into shared memory with cp.async.bulk, completing on an mbarrier the CTA waits on.
constexpr int kErrStage = 4;
constexpr long long kStageCycles = 1LL << 31;  // SM clock cycles (~1 s) before a wait gives up

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :: "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait: false if the phase did not complete within kStageCycles SM cycles.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try(bar, parity))
    if (clock64() - t0 > kStageCycles) return false;
  return true;
}

// L2 prefetch of the bytes [lo, hi) of a global array whose base is 16-byte aligned: a
// hint, so the window shrinks to the whole 16-byte units inside it (the bulk prefetch's
// rule) and nothing outside the range is touched.
__device__ __forceinline__ void l2_prefetch(const void* base, int64_t lo, int64_t hi) {
  const int64_t b = (lo + 15) & ~static_cast<int64_t>(15), e = hi & ~static_cast<int64_t>(15);
  if (e > b)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;"
                 :: "l"(static_cast<const char*>(base) + b), "r"(static_cast<uint32_t>(e - b)) : "memory");
}

// Byte window [lo, lo + len) of the element range [q0, q1) of an array with `es`-byte
// elements, widened to 16-byte boundaries (the bulk copy's alignment rule).
struct StageWin { int64_t lo; uint32_t len, skip; };
__device__ __forceinline__ StageWin stage_window(int64_t q0, int64_t q1, int es) {
  const int64_t b0 = q0 * es, b1 = q1 * es;
  StageWin w;
  w.lo = b0 & ~static_cast<int64_t>(15);
  w.len = static_cast<uint32_t>(((b1 + 15) & ~static_cast<int64_t>(15)) - w.lo);
  w.skip = static_cast<uint32_t>(b0 - w.lo);
  return w;
}

#include "tangent_tile.cuh"
#include "tangent_tc.cuh"

inline unsigned nb(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

// SM count per device ordinal, looked up once per device (grids are sized from it).
int sm_count(int device) {
  constexpr int kMaxDev = 64;
  static std::atomic<int> cached[kMaxDev];
  if (device < 0 || device >= kMaxDev) {
    int v = 0;
    CGB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device));
    return v;
  }
  int v = cached[device].load(std::memory_order_relaxed);
  if (v <= 0) {
    CGB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device));
    cached[device].store(v, std::memory_order_relaxed);
  }
  return v;
}

HingeArgs hinge_args(cgb_assembler* a, cgb_fold_dev& f, const double* d_x, int flags) {
  HingeArgs h{};
  h.n_gp = f.n_gp;
  h.max_u = std::max(f.max_u, 1);
  h.lptr = f.left->nbr_ptr.p; h.lidx = f.left->nbr_idx.p; h.ldpsi = f.left->dpsi.p;
  h.rptr = f.right->nbr_ptr.p; h.ridx = f.right->nbr_idx.p; h.rdpsi = f.right->dpsi.p;
  h.weight = f.weight.p; h.tangent = f.tangent.p;
  h.Kt = f.Kt; h.theta0 = f.theta0;
  h.theta0_gp = f.has_theta0_gp ? f.theta0_gp.p : nullptr;
  h.active = f.has_active ? f.active.p : nullptr;
  h.u_ptr = f.u_ptr.p; h.u_node = f.u_node.p; h.l_pos = f.l_pos.p; h.r_pos = f.r_pos.p;
  h.pair_ptr = f.pair_ptr.p;
  h.x = d_x;
  h.exact = (flags & CGB_HINGE_EXACT) ? 1 : 0;
  h.want_K = (flags & CGB_TANGENT) ? 1 : 0;
  (void)a;
  return h;
}

__global__ void to_float(int64_t n, const double* __restrict__ src, float* __restrict__ dst) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i < n) dst[i] = static_cast<float>(src[i]);
}

// FP32 copies of grad / Hessian Phi for the FP32 pair phase (made once per assembler).
// FP32 copies of grad / Hessian Phi, each followed by kStagePad zero elements: the
// tangent stages a group's range of these arrays with bulk copies whose ends are rounded
// out to 16 bytes, which may read up to 15 bytes past the last entry.
constexpr int kStagePad = 16;

void ensure_fp32_shapes(cgb_assembler* a) {
  if (a->dpsi32.p) return;
  const cgb_shape* S = a->faces;
  a->faces_version = S->version;
  cudaStream_t st = a->ctx->stream;
  a->dpsi32.alloc(2 * S->nnz + kStagePad);
  a->ddpsi32.alloc(3 * S->nnz + kStagePad);
  CGB_CUDA(cudaMemsetAsync(a->dpsi32.p, 0, a->dpsi32.bytes(), st));
  CGB_CUDA(cudaMemsetAsync(a->ddpsi32.p, 0, a->ddpsi32.bytes(), st));
  if (S->nnz) {
    to_float<<<nb(2 * S->nnz, 256), 256, 0, st>>>(2 * S->nnz, S->dpsi.p, a->dpsi32.p);
    to_float<<<nb(3 * S->nnz, 256), 256, 0, st>>>(3 * S->nnz, S->ddpsi.p, a->ddpsi32.p);
  }
  CGB_CUDA(cudaGetLastError());
}

// Sliced-ELL copy of the face neighbour data for phase 1: groups of 32 consecutive Gauss
// points, each group padded to its longest list; entry q of point 32 W + l at
// sell_ptr[W] + 32 q + l. Padding entries are never read (q < n of the point).
__global__ void fill_sell(int n_gp, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                          const double* __restrict__ dpsi, const double* __restrict__ ddpsi,
                          const int64_t* __restrict__ sell_ptr, int32_t* __restrict__ sidx,
                          double* __restrict__ sdpsi, double* __restrict__ sddpsi) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_gp) return;
  const int64_t base = sell_ptr[g >> 5] + (g & 31);
  for (int64_t e = ptr[g], q = 0; e < ptr[g + 1]; ++e, ++q) {
    const int64_t d = base + 32 * q;
    sidx[d] = idx[e];
    sdpsi[2 * d] = dpsi[2 * e];
    sdpsi[2 * d + 1] = dpsi[2 * e + 1];
    sddpsi[3 * d] = ddpsi[3 * e];
    sddpsi[3 * d + 1] = ddpsi[3 * e + 1];
    sddpsi[3 * d + 2] = ddpsi[3 * e + 2];
  }
}

// The point of every face entry (made once per assembler: it depends on the lists only).
__global__ void entry_points(int n_gp, const int64_t* __restrict__ ptr, int32_t* __restrict__ ent_point) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_gp) return;
  for (int64_t e = ptr[g]; e < ptr[g + 1]; ++e) ent_point[e] = g;
}

void ensure_entry_points(cgb_assembler* a) {
  if (a->ent_point.p) return;
  const cgb_shape* S = a->faces;
  a->ent_point.alloc(S->nnz);
  if (S->n_gp) entry_points<<<nb(S->n_gp, 128), 128, 0, a->ctx->stream>>>(S->n_gp, S->nbr_ptr.p, a->ent_point.p);
  CGB_CUDA(cudaGetLastError());
}

void ensure_sell(cgb_assembler* a) {
  if (a->sell_ptr.p) return;
  const cgb_shape* S = a->faces;
  a->faces_version = S->version;
  cudaStream_t st = a->ctx->stream;
  std::vector<int64_t> ptr(S->n_gp + 1);
  CGB_CUDA(cudaMemcpyAsync(ptr.data(), S->nbr_ptr.p, ptr.size() * 8, cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
  const int ngroups = (S->n_gp + 31) / 32;
  std::vector<int64_t> sp(ngroups + 1, 0);
  for (int W = 0; W < ngroups; ++W) {
    int64_t mx = 0;
    for (int g = 32 * W; g < std::min(S->n_gp, 32 * W + 32); ++g) mx = std::max(mx, ptr[g + 1] - ptr[g]);
    sp[W + 1] = sp[W] + 32 * mx;
  }
  upload(a->sell_ptr, sp.data(), sp.size(), st);
  a->sidx.alloc(sp[ngroups]);
  a->sdpsi.alloc(2 * sp[ngroups]);
  a->sddpsi.alloc(3 * sp[ngroups]);
  CGB_CUDA(cudaMemsetAsync(a->sidx.p, 0, a->sidx.bytes(), st));
  if (S->n_gp)
    fill_sell<<<nb(S->n_gp, 128), 128, 0, st>>>(S->n_gp, S->nbr_ptr.p, S->nbr_idx.p, S->dpsi.p, S->ddpsi.p,
                                                a->sell_ptr.p, a->sidx.p, a->sdpsi.p, a->sddpsi.p);
  CGB_CUDA(cudaGetLastError());
}

}  // namespace

void refresh_face_copies(cgb_assembler* a) {
  const cgb_shape* S = a->faces;
  if (a->faces_version == S->version) return;
  cudaStream_t st = a->ctx->stream;
  if (a->dpsi32.p && S->nnz) {
    to_float<<<nb(2 * S->nnz, 256), 256, 0, st>>>(2 * S->nnz, S->dpsi.p, a->dpsi32.p);
    to_float<<<nb(3 * S->nnz, 256), 256, 0, st>>>(3 * S->nnz, S->ddpsi.p, a->ddpsi32.p);
  }
  if (a->sell_ptr.p && S->n_gp)
    fill_sell<<<nb(S->n_gp, 128), 128, 0, st>>>(S->n_gp, S->nbr_ptr.p, S->nbr_idx.p, S->dpsi.p, S->ddpsi.p,
                                                a->sell_ptr.p, a->sidx.p, a->sdpsi.p, a->sddpsi.p);
  CGB_CUDA(cudaGetLastError());
  a->faces_version = S->version;
}

namespace {

// Chunks of the mixed step with the library's choice. Measured, one against four: 66,564 points
// 657 / 694 us, 118,336 points 560 / 525 us, 193,600 points 853 / 832 us, 640,000 points 2.70 / 2.24 ms.
constexpr int kChunks = 4;
constexpr int kChunkPoints = 98304;

// The second stream and the events of the chunked face launch (created once per
// assembler; the stream is non-blocking and joined back into the context stream).
void ensure_side_stream(cgb_assembler* a) {
  if (a->side) return;
  CGB_CUDA(cudaStreamCreateWithFlags(&a->side, cudaStreamNonBlocking));
  CGB_CUDA(cudaEventCreateWithFlags(&a->ev_start, cudaEventDisableTiming));
  CGB_CUDA(cudaEventCreateWithFlags(&a->ev_done, cudaEventDisableTiming));
  for (int c = 0; c < kMaxChunks; ++c) CGB_CUDA(cudaEventCreateWithFlags(&a->ev_chunk[c], cudaEventDisableTiming));
}

}  // namespace

constexpr size_t kTangentSmemMax = 220 * 1024;

void assemble_device(cgb_assembler* a, const double* d_x, double* d_K, double* d_F, int flags) {
  cgb_context* ctx = a->ctx;
  cudaStream_t st = ctx->stream;
  const cgb_shape* S = a->faces;
  const bool want_K = (flags & CGB_TANGENT) != 0;
  const bool mixed = (flags & CGB_MIXED) != 0;
  const bool det = (flags & CGB_DETERMINISTIC) != 0;
  const bool hinge = (flags & CGB_HINGE) != 0;
  if (!a->have_material) throw Error(CGB_ERR_INVALID, "assemble: material not set (cgb_set_material)");
  if (want_K && !d_K) throw Error(CGB_ERR_INVALID, "assemble: K output missing with CGB_TANGENT");
  refresh_face_copies(a);
  if (det) deterministic_prepare(a);
  bool bzero = true;
  for (double v : a->B) bzero = bzero && (v == 0.0);
  // The FP32 tangent sums each cell's contributions per block; in deterministic mode those sums
  // become the K units, unless a cell is direct. Supports too wide for a cell's lists (the
  // reference app's cubic basis at rho = 6h has over 100 neighbours) take the per-entry tangent.
  bool merged = false;
  if (mixed && want_K && S->max_n <= kTileMaxList) {
    tile_prepare(a);
    merged = (!det || a->direct_h.empty()) && a->n_items > 0;
  }
  const size_t msm = merged ? tile_smem_bytes(a->cell_max_e, a->cell_max_u, a->cell_max_i, bzero) : 0;
  // The tensor-core tangent takes the cells whose node union fits one 128-row tile (its blocks
  // are the items' slots too, so the deterministic lists are the same).
  const size_t tcsm = tc_smem_bytes(std::max(S->max_n, 1), bzero);
  const bool use_tc = merged && a->tuning.tangent_kind == CGB_TANGENT_TENSOR && tcsm <= kTangentSmemMax;
  if (det && want_K) {
    if (merged) deterministic_entry_lists(a);
    else deterministic_pair_lists(a);
  }
  const int64_t k_face_units = merged ? 4 * a->n_items : a->n_pairs;
  const bool acc32 = merged;   // the block accumulator: FP32 with the cells' tangent, else FP64

  const int64_t ndof = 3 * static_cast<int64_t>(a->n_nodes);
  // Accumulators.
  prof_begin(ctx, CGB_PHASE_ZERO);
  if (!det) CGB_CUDA(cudaMemsetAsync(d_F, 0, ndof * sizeof(double), st));
  void* zero = nullptr;   // the block accumulator: whole 16-byte words, cleared by the first residual
  size_t zero_bytes = 0;
  HingeBlocks hinge_blocks{};
  if (want_K && !det) {
    auto words = [](size_t bytes) { return (bytes + 15) / 16 * 16; };
    if (acc32) {   // the hinge's FP64 blocks follow the FP32 ones (12 floats each)
      const size_t face = static_cast<size_t>(a->n_blocks) * 12 * sizeof(float);
      const size_t both = words(face + static_cast<size_t>(a->n_hinge_blocks) * 9 * sizeof(double));
      a->kacc32.ensure(both / sizeof(float));
      zero_bytes = hinge ? both : face;
      if (hinge && a->n_hinge_blocks > 0)
        hinge_blocks = {a->hinge_col.p, a->hinge_pos.p, reinterpret_cast<double*>(a->kacc32.p + 12 * a->n_blocks)};
    } else {
      zero_bytes = words(static_cast<size_t>(a->n_blocks) * 9 * sizeof(double));
      a->kacc64.ensure(zero_bytes / sizeof(double));
    }
    zero = acc32 ? static_cast<void*>(a->kacc32.p) : static_cast<void*>(a->kacc64.p);
    if (S->n_gp == 0 && zero_bytes > 0) CGB_CUDA(cudaMemsetAsync(zero, 0, zero_bytes, st));
  }
  int64_t n_hinge = 0;
  for (auto& f : a->folds) n_hinge += f.n_pairs;
  if (det) {
    a->fcontrib.ensure(3 * std::max<int64_t>(a->n_fcontrib, 1));
    if (want_K) {
      if (mixed) a->contrib32.ensure(9 * std::max<int64_t>(k_face_units, 1));
      else a->contrib64.ensure(9 * std::max<int64_t>(k_face_units + n_hinge, 1));
      if (mixed) a->hinge_contrib.ensure(9 * std::max<int64_t>(n_hinge, 1));
    }
    // Hinge entries of inactive crease points contribute zero.
    if (a->n_fcontrib > S->nnz)
      CGB_CUDA(cudaMemsetAsync(a->fcontrib.p + 3 * S->nnz, 0, 3 * (a->n_fcontrib - S->nnz) * sizeof(double), st));
    if (want_K && n_hinge > 0)
      CGB_CUDA(cudaMemsetAsync(mixed ? a->hinge_contrib.p : a->contrib64.p + 9 * k_face_units, 0,
                               9 * n_hinge * sizeof(double), st));
  }

  prof_end(ctx, CGB_PHASE_ZERO, 0);

  // Face kernel.
  FaceArgs fa{};
  fa.n_gp = S->n_gp;
  fa.g_begin = 0;
  fa.g_end = S->n_gp;
  fa.nmax = std::max(S->max_n, 1);
  fa.ptr = S->nbr_ptr.p; fa.idx = S->nbr_idx.p; fa.dpsi = S->dpsi.p; fa.ddpsi = S->ddpsi.p;
  fa.weight = a->weight.p; fa.x = d_x;
  fa.map_ptr = a->map_ptr.p; fa.map_slot = a->map_slot.p;
  ensure_sell(a);
  fa.sell_ptr = a->sell_ptr.p; fa.sidx = a->sidx.p; fa.sdpsi = a->sdpsi.p; fa.sddpsi = a->sddpsi.p;
  fa.mat = make_material(a->A, a->B, a->D);
  fa.nc = ctx->natcurv;
  fa.gp_xy = natcurv_points(ctx, S, "assemble");
  fa.F = d_F;
  fa.Fc = a->fcontrib.p;
  fa.Kacc = acc32 ? static_cast<void*>(a->kacc32.p) : static_cast<void*>(a->kacc64.p);
  fa.Kc = mixed ? static_cast<void*>(a->contrib32.p) : static_cast<void*>(a->contrib64.p);
  if (want_K && (!merged || !a->direct_h.empty())) ensure_entry_points(a);
  if (mixed && want_K) {
    ensure_fp32_shapes(a);
    fa.dpsi_t = a->dpsi32.p;
    fa.ddpsi_t = a->ddpsi32.p;
  } else {
    fa.dpsi_t = S->dpsi.p;
    fa.ddpsi_t = S->ddpsi.p;
  }
  // The entry point's limit on the neighbours per point (about 165 in FP64, 340 in mixed mode).
  const size_t tk = mixed ? sizeof(float) : sizeof(double);
  if (want_K && kFaceWarps * ((kState * 32 + kRec * static_cast<size_t>(fa.nmax)) * tk + fa.nmax * sizeof(int)) > 200 * 1024)
    throw Error(CGB_ERR_CAPACITY, "assemble: " + std::to_string(S->max_n) + " neighbours per Gauss point exceed the shared-memory staging");
  const int sms = sm_count(ctx->device);
  // Residual kernel (phase 1) then tangent kernel (phase 2), each at its own occupancy.
  const size_t state_vals = static_cast<size_t>(mixed ? kState : kState64) * std::max(S->n_gp, 1);
  if (want_K) {
    if (mixed) a->state32.ensure(state_vals);
    else a->state64.ensure(state_vals);
  }
  float* st32 = a->state32.p;
  double* st64 = a->state64.p;
  // The residual kernel of chunk c + 1 (FP64 pipe) runs beside the tangent kernel of
  // chunk c (FP32 pipe, L2 atomics) on a second stream; chunks are multiples of 32 points.
  ensure_side_stream(a);
  // Only the FP32 tangent has another pipe to overlap with; without one, chunks are just tails.
  const int n_chunks = a->tuning.n_chunks > 0 ? a->tuning.n_chunks : (mixed && want_K && S->n_gp >= kChunkPoints ? kChunks : 1);
  const int rthreads = a->tuning.residual_threads > 0 ? a->tuning.residual_threads : 256;
  const int chunk = ((S->n_gp + n_chunks - 1) / n_chunks + 31) / 32 * 32;
  // Chunk c covers [cb(c), cb(c + 1)). The first chunk is a quarter of the others: the
  // tangent stream waits for its residual, and from then on the tangent stream is the
  // longer of the two, so a short first chunk shortens the step; the rest share the
  // remaining points evenly. All bounds are multiples of 32 points.
  const int first = n_chunks > 1 ? std::max(32, (chunk / 4 + 31) / 32 * 32) : chunk;
  const int rest = n_chunks > 1 ? ((std::max(S->n_gp - first, 0) + n_chunks - 2) / (n_chunks - 1) + 31) / 32 * 32 : 0;
  auto cb = [&](int c) {
    const int64_t b = c == 0 ? 0 : static_cast<int64_t>(first) + static_cast<int64_t>(c - 1) * rest;
    return static_cast<int>(std::min<int64_t>(b, S->n_gp));
  };
  int nface = 0;
  // Work counters of the chunks' residual launches.
  a->work_ctr.ensure(kMaxChunks);
  CGB_CUDA(cudaMemsetAsync(a->work_ctr.p, 0, kMaxChunks * sizeof(int), st));
  // Hinge: it reads x, its shape sets and the fold state and adds into F and the block
  // accumulator (mixed: its own FP64 blocks) with atomics (or into its own contribution slots in deterministic mode), none
  // of which the face kernels read, so it runs beside them: on the side stream when the residual
  // is all there is (a hinge launch is mostly the latency of one warp), else on the context
  // stream beside the last tangent chunks.
  auto launch_hinge = [&](cudaStream_t hst) {
    prof_begin(ctx, CGB_PHASE_HINGE, hst);
    int nl = 0;
    int64_t kb = mixed ? 0 : k_face_units, fb = a->hinge_f_base;
    for (auto& f : a->folds) {
      if (f.n_gp == 0) continue;
      HingeArgs h = hinge_args(a, f, d_x, flags);
      h.F = d_F;
      h.Kacc = acc32 ? const_cast<double*>(hinge_blocks.acc) : a->kacc64.p;
      h.pair_slot = acc32 ? f.pair_hslot.p : f.pair_slot.p;
      if (det) {
        h.Fc = a->fcontrib.p;
        h.Kc = mixed ? a->hinge_contrib.p : a->contrib64.p;
        h.f_base = fb; h.k_base = kb;
      }
      // Warps per point: two per SM quarter over the launch, each with at least 4 rounds of pairs.
      const int64_t rounds = static_cast<int64_t>(h.max_u) * (h.max_u + 1) / 2 / 128;
      h.parts = want_K ? static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(rounds, 8 * sms / f.n_gp))) : 1;
      const size_t hs = static_cast<size_t>(kHingeWarps) * (7 * h.max_u + 144 + 16) * sizeof(double);
      if (hs > 48 * 1024) CGB_CUDA(cudaFuncSetAttribute(hinge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(hs)));
      hinge_kernel<<<nb(static_cast<int64_t>(f.n_gp) * h.parts, kHingeWarps), 32 * kHingeWarps, hs, hst>>>(h);
      CGB_CUDA(cudaGetLastError());
      ++nl;
      kb += f.n_pairs;
      fb += f.n_u;
    }
    prof_end(ctx, CGB_PHASE_HINGE, nl, hst);
  };
  const bool hinge_first = hinge && !want_K;
  const bool use_side = want_K || hinge_first;
  if (use_side) {
    CGB_CUDA(cudaEventRecord(a->ev_start, st));
    CGB_CUDA(cudaStreamWaitEvent(a->side, a->ev_start, 0));
  }
  if (hinge_first) launch_hinge(a->side);
  for (int c = 0; c < n_chunks && S->n_gp > 0; ++c) {
    int* work = a->work_ctr.p + c;
    fa.g_begin = cb(c);
    fa.g_end = cb(c + 1);
    if (fa.g_begin >= fa.g_end) break;
    const int ncg = fa.g_end - fa.g_begin;
    fa.zero = c == 0 ? static_cast<double2*>(zero) : nullptr;
    fa.n_zero = static_cast<int64_t>(zero_bytes / sizeof(double2));
    prof_begin(ctx, CGB_PHASE_FACE);
    auto rl = [&](auto lanes, auto* stp) {
      constexpr int L = decltype(lanes)::value;
      using TK = std::remove_pointer_t<decltype(stp)>;
      auto kern = det ? (want_K ? face_residual_kernel<TK, true, true, L> : face_residual_kernel<TK, true, false, L>)
                      : (want_K ? face_residual_kernel<TK, false, true, L> : face_residual_kernel<TK, false, false, L>);
      // Beside the FP32 tangent the SMs must stay set up for its shared memory: an SM drains before
      // it changes the split between L1 and shared memory, so a residual that asks for none (and
      // gets the largest L1) and the tangent would never share one.
      if (merged) CGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
      // Few points: small blocks, so that every SM gets a share (25,600 points are only 100
      // blocks of 256 threads). Beside the previous chunk's tangent: small blocks too, and as many
      // warps per SM as leave the tangent's blocks their registers (8: 640,000 points in 4 chunks
      // take 2.22 ms, against 2.40 with 16 and 2.88 with 4).
      const bool beside = merged && c > 0;
      const int rt = L > 1 ? 32 : (a->tuning.residual_threads == 0 && (beside || ncg < 256 * 4 * sms) ? 64 : rthreads);
      const int64_t pts = rt / L;
      const unsigned most = static_cast<unsigned>(beside ? sms * std::max(1, 256 / rt) : sms * 16 * (256 / rt));
      kern<<<std::max(1u, std::min(nb(ncg, static_cast<int>(pts)), most)), rt, 0, st>>>(fa, stp, work);
    };
    auto rk = [&](auto* stp) {
      switch (residual_lanes(ncg, sms, det)) {
        case 8: rl(std::integral_constant<int, 8>{}, stp); break;
        case 4: rl(std::integral_constant<int, 4>{}, stp); break;
        case 2: rl(std::integral_constant<int, 2>{}, stp); break;
        default: rl(std::integral_constant<int, 1>{}, stp); break;
      }
    };
    if (mixed) rk(st32);
    else rk(st64);
    ++nface;
    prof_end(ctx, CGB_PHASE_FACE, 1);
    CGB_CUDA(cudaGetLastError());
    if (!want_K) continue;
    CGB_CUDA(cudaEventRecord(a->ev_chunk[c], st));
    CGB_CUDA(cudaStreamWaitEvent(a->side, a->ev_chunk[c], 0));
    prof_begin(ctx, CGB_PHASE_TANGENT, a->side);
    // One thread per entry of the chunk (at most max_n per point; the surplus CTAs leave), or of
    // the chunk's direct cells.
    auto tl = [&](auto kern, auto* stp, const int32_t* glist = nullptr, int gcount = 0) {
      const int per_cell = glist ? static_cast<int>(nb(static_cast<int64_t>(kMG) * fa.nmax, kEntryThreads)) : 0;
      const unsigned egrid = glist ? static_cast<unsigned>(gcount) * per_cell
                                   : std::max(1u, nb(std::min(S->nnz, static_cast<int64_t>(ncg) * fa.nmax), kEntryThreads));
      kern<<<egrid, kEntryThreads, 0, a->side>>>(fa, stp, a->ent_point.p, glist, per_cell);
    };
    int ntan = 1;
    if (merged) {
      TileArgs tg{a->cells.p, a->item_code.p, reinterpret_cast<const int4*>(a->item_slot.p), a->nbr_u.p,
                  a->cell_max_e, a->cell_max_u, a->cell_max_i, ctx->dev_err.p, a->test_stage_extra_tx, nullptr, 0};
      auto kern = det ? (bzero ? face_tangent_tile_kernel<true, true> : face_tangent_tile_kernel<false, true>)
                      : (bzero ? face_tangent_tile_kernel<true, false> : face_tangent_tile_kernel<false, false>);
      CGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(msm)));
      CGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
      int per_sm = 0;
      CGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kTileThreads, msm));
      const int Gb = fa.g_begin / kMG, Ge = (fa.g_end + kMG - 1) / kMG;
      const int groups = Ge - Gb;
      if (a->tuning.tangent_ctas_per_sm > 0) per_sm = std::min(per_sm, a->tuning.tangent_ctas_per_sm);
      per_sm = std::max(per_sm, 1);
      // The part of a sorted cell list that lies in this chunk.
      auto part = [&](const std::vector<int32_t>& v) {
        const auto lo = std::lower_bound(v.begin(), v.end(), Gb), hi = std::lower_bound(lo, v.end(), Ge);
        return std::make_pair(static_cast<int>(lo - v.begin()), static_cast<int>(hi - lo));
      };
      if (use_tc) {
        // Cells whose node union fits one 128-row tile: one tensor-core product each; the
        // others on the CUDA cores.
        TcArgs tca{a->nbr_u.p, a->cell_U.p, a->item_ptr.p};
        auto tk = det ? (bzero ? face_tangent_tc_kernel<true, true> : face_tangent_tc_kernel<false, true>)
                      : (bzero ? face_tangent_tc_kernel<true, false> : face_tangent_tc_kernel<false, false>);
        CGB_CUDA(cudaFuncSetAttribute(tk, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(tcsm)));
        CGB_CUDA(cudaFuncSetAttribute(tk, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        // Each CTA holds 256 of the SM's 512 tensor-memory columns: two CTAs per SM at most,
        // when the shared memory of two (dynamic + static + the 1 KB the runtime reserves per
        // CTA) fits the SM's.
        cudaFuncAttributes fat{};
        CGB_CUDA(cudaFuncGetAttributes(&fat, tk));
        int smem_sm = 0;
        CGB_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx->device));
        int tc_per_sm = 2 * (tcsm + fat.sharedSizeBytes + 1024) <= static_cast<size_t>(smem_sm) ? 2 : 1;
        if (a->tuning.tangent_ctas_per_sm > 0) tc_per_sm = std::min(tc_per_sm, a->tuning.tangent_ctas_per_sm);
        a->tc_last_per_sm = tc_per_sm;
        const unsigned tgrid2 = static_cast<unsigned>(std::max(1, std::min(groups, tc_per_sm * sms)));
        tk<<<tgrid2, kTcThreads, tcsm, a->side>>>(fa, st32, tg, tca);
        const auto [at, count] = part(a->tc_rest_h);
        if (count > 0) {
          tg.glist = a->tc_rest.p + at;
          tg.gcount = count;
          kern<<<static_cast<unsigned>(std::min(count, per_sm * sms)), kTileThreads, msm, a->side>>>(fa, st32, tg);
          ++ntan;
        }
      } else {
        kern<<<static_cast<unsigned>(std::max(1, std::min(groups, per_sm * sms))), kTileThreads, msm, a->side>>>(fa, st32, tg);
      }
      const auto [at, count] = part(a->direct_h);
      if (count > 0) {
        if (bzero) tl(face_tangent_entry_kernel<float, float, false, true>, st32, a->direct.p + at, count);
        else tl(face_tangent_entry_kernel<float, float, false, false>, st32, a->direct.p + at, count);
        ++ntan;
      }
    } else if (mixed) {
      if (det) { if (bzero) tl(face_tangent_entry_kernel<float, float, true, true>, st32); else tl(face_tangent_entry_kernel<float, float, true, false>, st32); }
      else { if (bzero) tl(face_tangent_entry_kernel<float, double, false, true>, st32); else tl(face_tangent_entry_kernel<float, double, false, false>, st32); }
    } else {
      if (det) { if (bzero) tl(face_tangent_entry_kernel<double, double, true, true>, st64); else tl(face_tangent_entry_kernel<double, double, true, false>, st64); }
      else { if (bzero) tl(face_tangent_entry_kernel<double, double, false, true>, st64); else tl(face_tangent_entry_kernel<double, double, false, false>, st64); }
    }
    ++nface;
    prof_end(ctx, CGB_PHASE_TANGENT, ntan, a->side);
    CGB_CUDA(cudaGetLastError());
  }
  (void)nface;

  if (hinge && !hinge_first) launch_hinge(st);
  if (use_side) {
    CGB_CUDA(cudaEventRecord(a->ev_done, a->side));
    CGB_CUDA(cudaStreamWaitEvent(st, a->ev_done, 0));
  }

  // Reductions / output.
  const unsigned cg = std::max(1u, std::min(nb(a->n_nodes, 4), static_cast<unsigned>(sms * 32)));
  prof_begin(ctx, CGB_PHASE_REDUCE);
  int nred = 0;
  if (det) {
    nred = want_K ? 2 : 1;
    det_reduce_F<<<nb(a->n_nodes, kReduceNodes), 32 * kReduceNodes, 0, st>>>(a->n_nodes, a->node_list_ptr.p, a->node_list.p, a->fcontrib.p, d_F);
    if (want_K) {
      const unsigned dg = static_cast<unsigned>(std::max(a->n_nodes, 1));
      const double* hc = a->hinge_contrib.p;
      const int64_t* fe = n_hinge > 0 ? (merged ? a->ent_face_end.p : a->blk_face_end.p) : nullptr;
      if (merged) det_reduce_blocks<float, false><<<dg, kReduceThreads, 0, st>>>(a->n_nodes, a->col_ptr.p, a->ent_list_ptr.p, a->ent_list.p, a->contrib32.p, fe, k_face_units, hc, d_K);
      else if (mixed) det_reduce_blocks<float, true><<<dg, kReduceThreads, 0, st>>>(a->n_nodes, a->col_ptr.p, a->blk_list_ptr.p, a->blk_list.p, a->contrib32.p, fe, k_face_units, hc, d_K);
      else det_reduce_blocks<double, false><<<dg, kReduceThreads, 0, st>>>(a->n_nodes, a->col_ptr.p, a->blk_list_ptr.p, a->blk_list.p, a->contrib64.p, nullptr, 0, nullptr, d_K);
    }
  } else if (want_K) {
    nred = 1;
    if (acc32) blocks_to_csc<float, 12><<<cg, 128, 0, st>>>(a->n_nodes, a->col_ptr.p, a->kacc32.p, hinge_blocks, d_K);
    else blocks_to_csc<double, 9><<<cg, 128, 0, st>>>(a->n_nodes, a->col_ptr.p, a->kacc64.p, hinge_blocks, d_K);
  }
  prof_end(ctx, CGB_PHASE_REDUCE, nred);
  CGB_CUDA(cudaGetLastError());
}

// Mixed-precision face assembly on caller-owned device arrays, with the FP32 block
// accumulator supplied by the caller (the allocation-free entry point, noalloc.cu).
void face_mixed_on_arrays(const cgb_face_problem& pr, const double* d_x, double* d_K, double* d_F,
                          float* kacc, int* err, cudaStream_t st) {
  FaceArgs fa{};
  fa.n_gp = pr.n_gp;
  fa.g_begin = 0;
  fa.g_end = pr.n_gp;
  fa.nmax = std::max(pr.max_neighbours, 1);
  fa.ptr = pr.nbr_ptr; fa.idx = pr.nbr_idx; fa.dpsi = pr.dpsi; fa.ddpsi = pr.ddpsi;
  fa.dpsi_t = pr.dpsi; fa.ddpsi_t = pr.ddpsi;
  fa.weight = pr.weight; fa.x = d_x;
  fa.map_ptr = pr.map_ptr; fa.map_slot = pr.csr_map; fa.outer = pr.outer;
  fa.mat = make_material(pr.A, pr.B, pr.D);
  fa.F = d_F;
  fa.Kacc = kacc;
  const int64_t n_blocks = static_cast<int64_t>(pr.nnz / 9);
  fa.n_blocks = n_blocks;
  fa.n_nodes = pr.n_nodes;
  fa.err = err;
  CGB_CUDA(cudaMemsetAsync(d_F, 0, 3 * static_cast<size_t>(pr.n_nodes) * sizeof(double), st));
  if (pr.n_gp == 0) {  // no face point: K is zero, and outer is not needed
    if (pr.nnz > 0) CGB_CUDA(cudaMemsetAsync(d_K, 0, static_cast<size_t>(pr.nnz) * sizeof(double), st));
    return;
  }
  CGB_CUDA(cudaMemsetAsync(kacc, 0, 12 * static_cast<size_t>(n_blocks) * sizeof(float), st));
  const size_t smem = static_cast<size_t>(kFaceWarps) * ((kState * 32 + kRec * fa.nmax) * sizeof(float) +
                                                        fa.nmax * sizeof(int));
  auto kern = face_kernel<float, false, true, double, true>;
  if (smem > 48 * 1024) CGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  int dev = 0;
  CGB_CUDA(cudaGetDevice(&dev));
  const int sms = sm_count(dev);
  const unsigned grid = std::max(1u, std::min(nb(pr.n_gp, 32 * kFaceWarps), static_cast<unsigned>(sms * 8)));
  kern<<<grid, 32 * kFaceWarps, smem, st>>>(fa);
  const unsigned cg = std::max(1u, std::min(nb(pr.n_nodes, 4), static_cast<unsigned>(sms * 32)));
  blocks_to_csc_outer<float, 12><<<cg, 128, 0, st>>>(pr.n_nodes, n_blocks, pr.outer, kacc, d_K, err);
  CGB_CUDA(cudaGetLastError());
}

void point_state_device(cgb_context* ctx, const cgb_shape* S, const double* d_x, const double* A, const double* B,
                        const double* D, double* d_out) {
  if (S->n_gp == 0) return;
  if (!S->psi.p || S->psi.n < static_cast<size_t>(std::max<int64_t>(S->nnz, 1)))
    throw Error(CGB_ERR_INVALID, "point state: the shape set has no Psi");
  const Material m = make_material(A, B, D);
  const double* xy = natcurv_points(ctx, S, "point state");
  point_state_kernel<<<nb(S->n_gp, 64), 64, 0, ctx->stream>>>(S->n_gp, S->nbr_ptr.p, S->nbr_idx.p, S->psi.p,
                                                                S->dpsi.p, S->ddpsi.p, d_x, m, ctx->natcurv, xy,
                                                                d_out);
  CGB_CUDA(cudaGetLastError());
}

void energies_device(cgb_assembler* a, const double* d_x, double* out3) {
  cgb_context* ctx = a->ctx;
  cudaStream_t st = ctx->stream;
  a->energy.ensure(3);
  CGB_CUDA(cudaMemsetAsync(a->energy.p, 0, 3 * sizeof(double), st));
  const Material m = make_material(a->A, a->B, a->D);
  const cgb_shape* S = a->faces;
  if (S->n_gp)
    face_energy_kernel<<<nb(S->n_gp, 64), 64, 0, st>>>(
        S->n_gp, S->nbr_ptr.p, S->nbr_idx.p, S->dpsi.p, S->ddpsi.p, a->weight.p, d_x, m, ctx->natcurv,
        natcurv_points(ctx, S, "energies"), a->energy.p);
  for (auto& f : a->folds) {
    if (!f.n_gp) continue;
    HingeArgs h = hinge_args(a, f, d_x, 0);
    hinge_energy_kernel<<<nb(f.n_gp, 4), 128, 0, st>>>(h, a->energy.p + 2);
  }
  CGB_CUDA(cudaGetLastError());
  CGB_CUDA(cudaMemcpyAsync(out3, a->energy.p, 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
  CGB_CUDA(cudaStreamSynchronize(st));
}

}  // namespace cgb
