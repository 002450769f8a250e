// cgb_device.cuh — device helpers shared by the kernels of the GB300 Gauss-point library.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace cgb {

// Device error word: the first failing check stores its code; the host reads it back.
__device__ __forceinline__ void dev_fail(int* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Device-side crease polyline: vertices packed in one array for all creases.
struct DevCrease {
  const double* xy;  // 2 * n_vertices
  int n_vertices;
  int extend_start, extend_end, is_closed;
  const float2* xyf;  // the vertices relative to the first, in float
  float extent;       // their largest coordinate
};

// Squared distance in float of a point (relative to the crease's first vertex) to segment i, its ends
// not extended.
__device__ __forceinline__ float segment_dist2f(const DevCrease& c, int i, float px, float py) {
  const float2 A = c.xyf[i], B = c.xyf[i + 1];
  const float vx = B.x - A.x, vy = B.y - A.y, wx = px - A.x, wy = py - A.y;
  const float v2 = vx * vx + vy * vy;
  const float t = v2 > 0.0f ? __saturatef(__fdividef(wx * vx + wy * vy, v2)) : 0.0f;
  const float ex = wx - t * vx, ey = wy - t * vy;
  return ex * ex + ey * ey;
}

// Enrichment::evaluateIndicator (core/include/curvami/Enrichment.h:23-92). The
// geometric decisions (closest segment with a strict '<', clamping of t, the 1e-12
// validity distance, the end caps, the side test) are evaluated with explicitly
// rounded operations, so they are taken exactly as a non-contracted FP64 CPU run
// takes them.
// Segments that cannot be the closest are left out by a float pass. With X a bound on the relative
// coordinates, rounding them (2^-24 X each) and the float arithmetic move a segment's distance by
// less than eps = 2^-18 X (the foot's error along the segment, 2^-20 X, is the largest part); a
// segment more than 4 eps beyond the closest one's float distance is therefore farther than it by
// 2 eps, far more than the FP64 comparison resolves, and the walk over the others in their order
// ends where the walk over all would. That holds for feet within the segment: on an extended end the
// rounding of the segment's direction grows with the distance along it, without bound, so extended
// segments take no part in the float pass and are always walked. The FP64 work of a point, some 45 operations a segment with a
// division, falls from all segments to a few (a point that all are equally far from keeps all).
// L lanes (an aligned group of the warp, all with the same point) share the float pass: on 152 SMs 32
// for up to 608 points, 4 for up to 4,864, else one (indicator_lanes in shape.cu). The three sets and
// the node sides of a cubic rebuild of 61 x 61 nodes: 290 -> 110 us.
struct DevIndicator {
  double f, gx, gy, hxx, hyy, hxy;
};

template <int L>
__device__ __forceinline__ DevIndicator eval_indicator(double px, double py, const DevCrease& c) {
  const int lane = threadIdx.x & 31, sub = lane % L;
  const unsigned group = L == 32 ? 0xffffffffu : ((1u << (L % 32)) - 1u) << (lane - sub);
  DevIndicator out{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const int N = c.n_vertices;
  if (N < 2) return out;
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  double d = inf;
  double Cx = 0, Cy = 0, t_best = 0, snx = 0, sny = 0;
  int idx_best = 0;
  const bool sift = N > 4;
  const int s0 = c.extend_start ? 1 : 0, s1 = N - 1 - (c.extend_end ? 1 : 0);   // the segments of the float pass
  float fx = 0.0f, fy = 0.0f, limit = 0.0f;
  if (sift) {
    fx = __double2float_rn(px - c.xy[0]);
    fy = __double2float_rn(py - c.xy[1]);
    float least = __int_as_float(0x7f800000);
#pragma unroll 4
    for (int i = s0 + sub; i < s1; i += L) least = fminf(least, segment_dist2f(c, i, fx, fy));
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) least = fminf(least, __shfl_xor_sync(group, least, o));
    const float eps = fmaxf(fmaxf(fabsf(fx), fabsf(fy)), c.extent) * (1.0f / 262144.0f);
    limit = sqrtf(least) + 4.0f * eps;
    limit *= limit;
    if (!(eps >= 0x1p-70f)) limit = __int_as_float(0x7f800000);   // squares would lose their bits: keep all
  }
  auto closer = [&](int i) {
    const double Ax = c.xy[2 * i], Ay = c.xy[2 * i + 1];
    const double Bx = c.xy[2 * i + 2], By = c.xy[2 * i + 3];
    const double vx = __dsub_rn(Bx, Ax), vy = __dsub_rn(By, Ay);
    const double v_sq = __dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy));
    if (v_sq == 0.0) return;
    const double wx = __dsub_rn(px, Ax), wy = __dsub_rn(py, Ay);
    const double t = __ddiv_rn(__dadd_rn(__dmul_rn(wx, vx), __dmul_rn(wy, vy)), v_sq);
    const double t_min = (i == 0 && c.extend_start) ? -inf : 0.0;
    const double t_max = (i == N - 2 && c.extend_end) ? inf : 1.0;
    const double tm = (t < t_max) ? t : t_max;     // std::min(t_max, t)
    const double tc = (t_min < tm) ? tm : t_min;   // std::max(t_min, .)
    const double cx = __dadd_rn(Ax, __dmul_rn(tc, vx)), cy = __dadd_rn(Ay, __dmul_rn(tc, vy));
    const double ex = __dsub_rn(px, cx), ey = __dsub_rn(py, cy);
    const double cur = __dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey));
    if (cur < __dmul_rn(d, d)) {
      d = __dsqrt_rn(cur);
      Cx = cx; Cy = cy; idx_best = i; t_best = tc;
      const double len = __dsqrt_rn(v_sq);
      snx = __ddiv_rn(-vy, len);
      sny = __ddiv_rn(vx, len);
    }
  };
  auto left_out = [&](int i) { return sift && i >= s0 && i < s1 && segment_dist2f(c, i, fx, fy) > limit; };
  // The segments that are left, in their order: kStep decisions, then the walk over those that stay.
  constexpr int kStep = L == 1 ? 8 : L;
  for (int base = 0; base < N - 1; base += kStep) {
    unsigned keep = 0u;
    if constexpr (L == 1) {
#pragma unroll
      for (int k = 0; k < kStep; ++k)
        if (base + k < N - 1 && !left_out(base + k)) keep |= 1u << k;
    } else {
      const int i = base + sub;
      keep = __ballot_sync(group, i < N - 1 && !left_out(i)) >> (lane - sub);
    }
    for (; keep; keep &= keep - 1u) closer(base + __ffs(keep) - 1);
  }
  if (!(d > 1e-12)) return out;  // invalid: f = 0, no derivatives
  const double ux = __ddiv_rn(__dsub_rn(px, Cx), d), uy = __ddiv_rn(__dsub_rn(py, Cy), d);
  const double dp = __dadd_rn(__dmul_rn(ux, snx), __dmul_rn(uy, sny));
  const bool start_cap = (idx_best == 0 && t_best == 0.0 && !c.extend_start && !c.is_closed);
  const bool end_cap = (idx_best == N - 2 && t_best == 1.0 && !c.extend_end && !c.is_closed);
  if (start_cap || end_cap) {
    out.f = dp;
    out.gx = (snx - out.f * ux) / d;
    out.gy = (sny - out.f * uy) / d;
    const double d2 = d * d;
    out.hxx = (3 * out.f * ux * ux - 2 * snx * ux - out.f) / d2;
    out.hyy = (3 * out.f * uy * uy - 2 * sny * uy - out.f) / d2;
    out.hxy = (3 * out.f * ux * uy - (snx * uy + ux * sny)) / d2;
  } else {
    out.f = (dp >= 0.0) ? 1.0 : -1.0;
  }
  return out;
}

}  // namespace cgb
