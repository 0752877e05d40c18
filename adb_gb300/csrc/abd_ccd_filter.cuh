// FP32 certificates that a trajectory has no time of impact.
//
// pt_collision_time / ee_collision_time (abd_exact.cuh) return 1 unless the coplanarity
// cubic has a root in [0, 1] at which the primitives are found to touch. Both conditions can
// be refuted in FP32 with error bounds, and a refuted candidate returns exactly 1 in the FP64
// test, so skipping that test changes nothing. What this is for: on this part a warp's FP64
// instruction takes 64 cycles whatever the lanes, an FP32 one takes one, and an exact test is
// about 900 FP64 instructions; the certificates are about 250 FP32 ones.
//
// Inputs are the positions at both ends of the step rounded to the nearest float. With m the
// largest coordinate, a difference of two positions computed in FP32 is off by at most
// E = 4.5e-7 m in norm (both roundings 2^-24 m per coordinate, the subtraction's 2^-24 times
// at most 2 m, times sqrt 3). Every bound below takes that as the uncertainty of each edge
// vector and adds the rounding of its own FP32 arithmetic, so a certificate is a proof for
// the FP64 positions; the rounding of the FP64 test itself is orders of magnitude inside the
// slack. Comparisons are written so that a NaN or an infinity certifies nothing.
//
//  1. No root: the cubic w . (u x v) in Bernstein form on [0, 1] has all four coefficients of
//     one sign, by more than their error. (A polynomial lies between its Bernstein
//     coefficients, so the FP64 polynomial has that sign at every point the root finder
//     evaluates, and it reports no root.)
//  2. Point-triangle, any root fails: through the whole step the point's projection stays
//     outside one edge of the triangle by an area above the FP64 test's 1e-8 tolerance.
//  3. Edge-edge, any root fails: through the whole step one of the two crossing tests keeps
//     both ends of one edge on the same side of the other.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "abd_exact.cuh"

namespace abd {

struct f3 {
  float x, y, z;
};
#define CFD __host__ __device__ __forceinline__
CFD f3 f3_sub(f3 a, f3 b) { return f3{a.x - b.x, a.y - b.y, a.z - b.z}; }
CFD f3 f3_add(f3 a, f3 b) { return f3{a.x + b.x, a.y + b.y, a.z + b.z}; }
CFD f3 f3_mid(f3 a, f3 b) { return f3{0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)}; }
CFD f3 f3_cross(f3 a, f3 b) { return f3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
CFD float f3_dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// norm, enlarged past the rounding of the sum and the square root
CFD float f3_len(f3 a) { return 1.000001f * sqrtf(f3_dot(a, a)) + 1e-30f; }
CFD float f3_maxabs(f3 a) { return fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)); }

// Certificate 1 for the edge vectors u, v, w at the start (0) and the end (1) of the step;
// E: error of each in norm, m: largest coordinate.
// |w . (u x v)| moves by at most E (UV + UW + VW) + E^2 (U + V + W) + E^3 with the vectors; the
// FP32 evaluation adds less than 33 roundings of UVW; the FP64 coefficients are sums of at most
// 576 m^3 in absolute value rounded some ten times, evaluated by Horner's rule on [0, 1]:
// below 1e-11 m^3.
CFD bool f_no_root(f3 u0, f3 u1, f3 v0, f3 v1, f3 w0, f3 w1, float E, float m) {
  const f3 n0 = f3_cross(u0, v0), n2 = f3_cross(u1, v1), n1 = f3_add(f3_cross(u0, v1), f3_cross(u1, v0));
  const float b0 = f3_dot(w0, n0), b1 = (f3_dot(w1, n0) + f3_dot(w0, n1)) * (1.f / 3.f),
              b2 = (f3_dot(w1, n1) + f3_dot(w0, n2)) * (1.f / 3.f), b3 = f3_dot(w1, n2);
  const float U = fmaxf(f3_len(u0), f3_len(u1)), V = fmaxf(f3_len(v0), f3_len(v1)), W = fmaxf(f3_len(w0), f3_len(w1));
  const float err = 1.01f * E * (U * V + U * W + V * W + E * (U + V + W + E)) + 2e-6f * U * V * W +
                    1.01e-11f * m * m * m + 1e-30f;
  const float lo = fminf(fminf(b0, b1), fminf(b2, b3)), hi = fmaxf(fmaxf(b0, b1), fmaxf(b2, b3));
  const bool fin = hi - lo < 1e30f;  // false for a NaN or an infinity
  return fin && (lo > err || hi < -err);
}

// A vector along the step: its value half-way and a bound on its distance from that at any
// time (half its change, plus its error E and the rounding of the mean, 2^-24 of it).
struct f3m {
  f3 c;
  float len, dev;
};
CFD f3m f3m_of(f3 a0, f3 a1, float E) {
  f3m r;
  r.c = f3_mid(a0, a1);
  r.len = f3_len(r.c);
  r.dev = 0.5f * f3_len(f3_sub(a1, a0)) + E + 6.1e-8f * r.len;
  return r;
}
// Cross product of two such vectors: value half-way and a bound on its distance from that,
// the rounding of the FP32 product included.
CFD f3m f3m_cross(const f3m& a, const f3m& b) {
  f3m r;
  r.c = f3_cross(a.c, b.c);
  r.len = f3_len(r.c);
  r.dev = 1.00001f * (a.dev * b.len + a.len * b.dev + a.dev * b.dev) + 1e-6f * a.len * b.len;
  return r;
}
// Bound on how far the product of two such vectors can be from that of their values half-way.
CFD float f3m_slack(const f3m& a, const f3m& b) {
  return 1.00001f * (a.len * b.dev + a.dev * b.len + a.dev * b.dev) + 1e-6f * a.len * b.len;
}

// Point p against the triangle t: true when pt_collision_time is certainly 1.
CFD bool f_pt_miss(f3 p0, f3 p1, const f3* t0, const f3* t1) {
  float m = fmaxf(f3_maxabs(p0), f3_maxabs(p1));
#pragma unroll
  for (int k = 0; k < 3; ++k) m = fmaxf(m, fmaxf(f3_maxabs(t0[k]), f3_maxabs(t1[k])));
  const float E = 4.5e-7f * m + 1e-30f;
  const f3 u0 = f3_sub(t0[1], t0[0]), u1 = f3_sub(t1[1], t1[0]), v0 = f3_sub(t0[2], t0[0]), v1 = f3_sub(t1[2], t1[0]);
  const f3 w0 = f3_sub(p0, t0[0]), w1 = f3_sub(p1, t1[0]);
  if (f_no_root(u0, u1, v0, v1, w0, w1, E, m)) return true;
  // twice the signed area of (edge k, projected point) is n . (e_k x r_k) / |n|; below
  // -(1e-6 + 1e-12 m^2) through the whole step, the three areas exceed the triangle's by
  // more than the tolerance of the FP64 test. The 4e-6 of the lengths keeps slivers, whose
  // FP64 normal is inaccurate, out.
  const f3m u = f3m_of(u0, u1, E), v = f3m_of(v0, v1, E), n = f3m_cross(u, v);
  const float gam = (1e-6f + 1e-12f * m * m) * (n.len + n.dev);
  bool out = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int b = (k + 1) % 3;
    const f3m e = f3m_of(f3_sub(t0[b], t0[k]), f3_sub(t1[b], t1[k]), E);
    const f3m r = f3m_of(f3_sub(p0, t0[k]), f3_sub(p1, t1[k]), E);
    const f3m c = f3m_cross(e, r);
    out |= f3_dot(n.c, c.c) + f3m_slack(n, c) + gam + 4e-6f * (u.len * v.len) * (e.len * r.len) < 0.f;
  }
  return out && n.len < 1e18f;
}

// Edge a against edge b: true when ee_collision_time is certainly 1.
CFD bool f_ee_miss(const f3* a0, const f3* a1, const f3* b0, const f3* b1) {
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    m = fmaxf(m, fmaxf(fmaxf(f3_maxabs(a0[k]), f3_maxabs(a1[k])), fmaxf(f3_maxabs(b0[k]), f3_maxabs(b1[k]))));
  const float E = 4.5e-7f * m + 1e-30f;
  const f3 u0 = f3_sub(a0[1], a0[0]), u1 = f3_sub(a1[1], a1[0]), v0 = f3_sub(b0[1], b0[0]), v1 = f3_sub(b1[1], b1[0]);
  const f3 w0 = f3_sub(b0[0], a0[0]), w1 = f3_sub(b1[0], a1[0]);
  if (f_no_root(u0, u1, v0, v1, w0, w1, E, m)) return true;
  // (u x (b_0 - a_0)) . (u x (b_1 - a_0)) > 0 through the whole step, or the same with the
  // edges exchanged
  const f3m u = f3m_of(u0, u1, E), v = f3m_of(v0, v1, E);
  const f3m q00 = f3m_of(w0, w1, E), q01 = f3m_of(f3_sub(b0[1], a0[0]), f3_sub(b1[1], a1[0]), E);
  const f3m q10 = f3m_of(f3_sub(b0[0], a0[1]), f3_sub(b1[0], a1[1]), E);
  const f3m c0 = f3m_cross(u, q00), c1 = f3m_cross(u, q01);
  const f3m d0 = f3m_cross(v, q00), d1 = f3m_cross(v, q10);
  const bool s = f3_dot(c0.c, c1.c) - f3m_slack(c0, c1) - 4e-6f * (u.len * u.len) * (q00.len * q01.len) > 0.f;
  const bool t = f3_dot(d0.c, d1.c) - f3m_slack(d0, d1) - 4e-6f * (v.len * v.len) * (q00.len * q10.len) > 0.f;
  return (s || t) && u.len < 1e9f && v.len < 1e9f && q00.len < 1e9f;
}

// The verification of a root in FP32: 1 passes, 0 fails, -1 not certain (the FP64 test then
// decides). The vectors at the root's time t are off by E (both ends'), by 2^-24 of t times
// the change of the vector (at most sqrt 3 times its largest coordinate, cheaper than its norm)
// for each rounding of t, of the change and of their product, and by 2^-24 of the vector for
// that of the sum; the slacks are those of the certificates.
CFD f3m f3m_at(f3 a0, f3 a1, float t, float E) {
  const f3 d = f3_sub(a1, a0);
  f3m r;
  r.c = f3{a0.x + t * d.x, a0.y + t * d.y, a0.z + t * d.z};
  r.len = f3_len(r.c);
  r.dev = E + 6.1e-8f * (5.2f * t * f3_maxabs(d) + r.len);
  return r;
}
CFD int f_pt_verify(f3 p0, f3 p1, const f3* t0, const f3* t1, float t) {
  float m = fmaxf(f3_maxabs(p0), f3_maxabs(p1));
#pragma unroll
  for (int k = 0; k < 3; ++k) m = fmaxf(m, fmaxf(f3_maxabs(t0[k]), f3_maxabs(t1[k])));
  const float E = 4.5e-7f * m + 1e-30f;
  const f3m u = f3m_at(f3_sub(t0[1], t0[0]), f3_sub(t1[1], t1[0]), t, E);
  const f3m v = f3m_at(f3_sub(t0[2], t0[0]), f3_sub(t1[2], t1[0]), t, E);
  const f3m n = f3m_cross(u, v);
  const float gam = (1e-6f + 1e-12f * m * m) * (n.len + n.dev);
  bool in = u.len * v.len < 1e4f, out = false;  // larger areas round by more than a part of the tolerance
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int b = (k + 1) % 3;
    const f3m e = f3m_at(f3_sub(t0[b], t0[k]), f3_sub(t1[b], t1[k]), t, E);
    const f3m r = f3m_at(f3_sub(p0, t0[k]), f3_sub(p1, t1[k]), t, E);
    const f3m c = f3m_cross(e, r);
    const float g = f3_dot(n.c, c.c), sl = f3m_slack(n, c) + 4e-6f * (u.len * v.len) * (e.len * r.len);
    in &= g - sl > 0.f;
    out |= g + sl + gam < 0.f;
  }
  if (!(n.len < 1e18f)) return -1;
  return in ? 1 : (out ? 0 : -1);
}
CFD int f_ee_verify(const f3* a0, const f3* a1, const f3* b0, const f3* b1, float t) {
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    m = fmaxf(m, fmaxf(fmaxf(f3_maxabs(a0[k]), f3_maxabs(a1[k])), fmaxf(f3_maxabs(b0[k]), f3_maxabs(b1[k]))));
  const float E = 4.5e-7f * m + 1e-30f;
  const f3m u = f3m_at(f3_sub(a0[1], a0[0]), f3_sub(a1[1], a1[0]), t, E);
  const f3m v = f3m_at(f3_sub(b0[1], b0[0]), f3_sub(b1[1], b1[0]), t, E);
  const f3m q00 = f3m_at(f3_sub(b0[0], a0[0]), f3_sub(b1[0], a1[0]), t, E);
  const f3m q01 = f3m_at(f3_sub(b0[1], a0[0]), f3_sub(b1[1], a1[0]), t, E);
  const f3m q10 = f3m_at(f3_sub(b0[0], a0[1]), f3_sub(b1[0], a1[1]), t, E);
  const f3m c0 = f3m_cross(u, q00), c1 = f3m_cross(u, q01), d0 = f3m_cross(v, q00), d1 = f3m_cross(v, q10);
  const float c = f3_dot(c0.c, c1.c), cs = f3m_slack(c0, c1) + 4e-6f * (u.len * u.len) * (q00.len * q01.len);
  const float d = f3_dot(d0.c, d1.c), ds = f3m_slack(d0, d1) + 4e-6f * (v.len * v.len) * (q00.len * q10.len);
  if (!(u.len < 1e9f && v.len < 1e9f && q00.len < 1e9f)) return -1;
  if (c - cs > 0.f || d - ds > 0.f) return 0;
  return c + cs < 0.f && d + ds < 0.f ? 1 : -1;
}

// pt_collision_time and ee_collision_time with the roots verified in FP32 where that is
// certain (about 220 and 100 FP64 instructions less a root). p / q: the four points at the
// start and at the end.
HD f3 f3_of(d3 a) { return f3{(float)a.x, (float)a.y, (float)a.z}; }
template <int KIND>
HD double toi_fast(const d3* p, const d3* q) {
  double roots[3];
  const int found = coplanar_roots(p, q, roots);
  for (int i = 0; i < found; ++i) {
    const double r = roots[i];
    f3 a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = f3_of(p[k]);
      b[k] = f3_of(q[k]);
    }
    int ok = KIND == 0 ? f_pt_verify(a[0], b[0], a + 1, b + 1, (float)r) : f_ee_verify(a, b, a + 2, b + 2, (float)r);
    if (ok < 0) {
      d3 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = lerp(q[k], p[k], r);
      ok = KIND == 0 ? verify_root_pt(x[0], x[1], x[2], x[3]) : verify_root_ee(x[0], x[1], x[2], x[3]);
    }
    if (ok) return r;
  }
  return 1.0;
}

#ifdef __CUDACC__
// Times of impact of n trajectories (24 doubles each: four points at the start, four at the
// end; KIND 0: point-triangle, 1: edge-edge) into toi, calling min_of with each time below 1.
// A warp takes 32 trajectories at a time (grid-stride), certifies them in FP32 and queues the
// others (64 slots of shared memory a warp); as soon as 32 wait it runs the FP64 test on
// them, so that test always has a full warp.
template <int KIND, typename F>
__device__ __forceinline__ void toi_stream(int n, const double* x, double* toi, int* queue, F&& min_of) {
  const int lane = threadIdx.x & 31;
  const int warps = (int)((gridDim.x * blockDim.x) >> 5), warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const unsigned below = (1u << lane) - 1u;
  int waiting = 0;
  for (int c = warp;; c += warps) {
    const bool last = (long long)c * 32 >= n;
    if (!last) {
      const int i = c * 32 + lane;
      bool keep = false;
      if (i < n) {
        const double* p = x + 24 * (size_t)i;
        f3 a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          a[k] = f3{(float)p[3 * k], (float)p[3 * k + 1], (float)p[3 * k + 2]};
          b[k] = f3{(float)p[12 + 3 * k], (float)p[13 + 3 * k], (float)p[14 + 3 * k]};
        }
        keep = !(KIND == 0 ? f_pt_miss(a[0], b[0], a + 1, b + 1) : f_ee_miss(a, b, a + 2, b + 2));
        if (!keep) toi[i] = 1.0;
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) queue[waiting + __popc(m & below)] = i;
      waiting += __popc(m);
      __syncwarp();
    }
    if (waiting >= 32 || (last && waiting > 0)) {
      const int take = waiting < 32 ? waiting : 32;
      if (lane < take) {
        const int i = queue[waiting - take + lane];
        const double* p = x + 24 * (size_t)i;
        d3 a[4], b[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          a[v] = mk(p[3 * v], p[3 * v + 1], p[3 * v + 2]);
          b[v] = mk(p[12 + 3 * v], p[13 + 3 * v], p[14 + 3 * v]);
        }
        const double t = toi_fast<KIND>(a, b);
        toi[i] = t;
        if (t < 1.0) min_of(t);
      }
      waiting -= take;
      __syncwarp();
    }
    if (last) break;
  }
}
// Blocks of a streamed batch: a warp per 32 trajectories until every SM has the `per` CTAs
// that its registers allow.
inline int toi_blocks(int n, int threads, int per) {
  const int b = (n + threads - 1) / threads;
  return b < 152 * per ? b : 152 * per;
}
#endif

}  // namespace abd
