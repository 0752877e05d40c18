// iAABB culling on the GPU (the reference's IAABB::iaabb_brute_force,
// model/iaabb.cpp:545-568, with the narrow phase of model/thread_local_culling.cpp):
//
//  1. vertex projection x = A xbar + p at q, q + alpha dq, or both (trajectory)
//  2. body boxes: inflated rest box through A (iaabb.cpp:40-72), or the union over the
//     trajectory (vtn 3)
//  3. body overlaps: every pair of one scene whose boxes overlap, as a symmetric CSR
//     (both (I,J) and (J,I)) whose upper entries are the unique overlaps, each with its
//     intersection ("cull") box (iaabb.cpp:98-202)
//  4. binning: the vertices, edges and faces of each side that touch the cull box
//     (iaabb.cpp:315-443)
//  5. narrow phase over the flattened candidate space of all overlaps:
//     (v of I) x (f of J), (v of J) x (f of I), (e of I) x (e of J); AABB test, then the
//     exact distance type and distance < dhat (vtn 1/2) or the CCD root (vtn 3)
//  6. vertex-ground pairs (y + 0.5)^2 < dhat, or the ground time of impact
//
// All stage outputs are produced by count -> scan -> ordered write, so every pair list
// comes out in the same order on every run (overlap, then candidate order). The AABB
// tests first run on float copies of the boxes rounded outward (__double2float_rd/_ru):
// a float miss implies an exact miss, so the float prefilter never changes the result
// and saves the scarce FP64 pipe (GB300: 1.2 TFLOP/s FP64 vs 70 TFLOP/s FP32).
#include <algorithm>
#include "abd_ccd_filter.cuh"
#include "abd_engine.h"
#include "abd_exact.cuh"

namespace abd {

namespace {

__device__ __forceinline__ d3 ldX(const double* X, int nv, int v) { return mk(X[v], X[nv + v], X[2 * nv + v]); }

struct fbox6 {
  float lo[3], hi[3];
};
__device__ __forceinline__ void put_fbox(float* dst, const box& b) {
  dst[0] = __double2float_rd(b.lo.x); dst[1] = __double2float_rd(b.lo.y); dst[2] = __double2float_rd(b.lo.z);
  dst[3] = __double2float_ru(b.hi.x); dst[4] = __double2float_ru(b.hi.y); dst[5] = __double2float_ru(b.hi.z);
}
// Clusters: the unions of the boxes of 32 primitives in a row, which the binning tests before the
// primitives (BinClusters; in memory order, so a cluster can hold the ends of two bodies). A
// box without an order (NaN) adds nothing: it hits no box either.
struct BinClusters {
  float *v, *e, *f;  // null: not wanted
  float* tight;      // the boxes of the bodies (k_bin_caps)
};
__device__ __forceinline__ int ford(float x) {  // order-preserving, its own inverse on the bits
  const int i = __float_as_int(x);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ void put_cluster(float* cl, int t, const float (&o)[6]) {  // whole warps
  float mine = 0.f;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int r = c < 3 ? __reduce_min_sync(0xffffffffu, ford(fminf(o[c], INFINITY)))
                        : __reduce_max_sync(0xffffffffu, ford(fmaxf(o[c], -INFINITY)));
    if (lane == c) mine = __int_as_float(r >= 0 ? r : r ^ 0x7fffffff);
  }
  if (lane < 6) cl[6 * (size_t)(t >> 5) + lane] = mine;
}

// ---------------------------------------------------------------------------------
// 1. projection: which 0 -> X0 at q0; 1 -> X and Xq at q; 2 -> X at q + alpha dq;
//    3 -> Xq at q only
// The trial state q + alpha dq of every body (alpha per scene when given), once per body
// rather than once per vertex.
__global__ void k_trial_state(Geo g, double alpha) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 12 * g.nb) return;
  const int b = i / 12;
  const double a = g.alpha_s ? g.alpha_s[g.bscene[b]] : alpha;
  g.qa[i] = XA(g.q[i], XM(g.dq[i], a));
}

// With vb the float boxes of the vertices (which 1, 2: at X; 3: of the path from Xq to X, already
// there) and, with cl, of their clusters are written too: a kernel of their own read the positions
// again (pile 26 + 16 us, now 33 us).
__global__ void __launch_bounds__(256) k_project(Geo g, int which, float* vb, float* cl) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if ((v & ~31) >= g.nv) return;
  float o[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (v < g.nv) {
    int b = g.vbody[v];
    const double* qq = (which == 0) ? g.q0 + 12 * b : ((which == 2) ? g.qa + 12 * b : g.q + 12 * b);
    d3 x = project(qq, g.rest[3 * v], g.rest[3 * v + 1], g.rest[3 * v + 2]);
    double* dst = (which == 0) ? g.X0 : ((which == 3) ? g.Xq : g.X);
    dst[v] = x.x;
    dst[g.nv + v] = x.y;
    dst[2 * g.nv + v] = x.z;
    if (which == 1) {
      g.Xq[v] = x.x;
      g.Xq[g.nv + v] = x.y;
      g.Xq[2 * g.nv + v] = x.z;
    }
    if (vb) {
      put_fbox(o, which == 3 ? box2(ldX(g.X, g.nv, v), x) : box{x, x});
#pragma unroll
      for (int c = 0; c < 6; ++c) vb[6 * (size_t)v + c] = o[c];
    }
  }
  if (cl) put_cluster(cl, v, o);
}

// 2. body boxes
__global__ void k_body_boxes(Geo g, int vtn, double alpha, double* bbox, float* fbox) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= g.nb) return;
  box r{mk(g.rest_box[6 * b], g.rest_box[6 * b + 1], g.rest_box[6 * b + 2]),
        mk(g.rest_box[6 * b + 3], g.rest_box[6 * b + 4], g.rest_box[6 * b + 5])};
  double q[12], qt[12];
  if (vtn == 2 && g.alpha_s) alpha = g.alpha_s[g.bscene[b]];
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    q[i] = g.q[12 * b + i];
    qt[i] = XA(q[i], XM(g.dq[12 * b + i], alpha));
  }
  box o;
  if (vtn == 1) o = affine_box(r, q);
  else if (vtn == 2) o = affine_box(r, qt);
  else o = merge(affine_box(r, q), affine_box(r, qt));
  bbox[6 * b] = o.lo.x; bbox[6 * b + 1] = o.lo.y; bbox[6 * b + 2] = o.lo.z;
  bbox[6 * b + 3] = o.hi.x; bbox[6 * b + 4] = o.hi.y; bbox[6 * b + 5] = o.hi.z;
  // the same box in float, rounded outward: a float miss is an exact miss
  fbox[6 * b] = __double2float_rd(o.lo.x); fbox[6 * b + 1] = __double2float_rd(o.lo.y);
  fbox[6 * b + 2] = __double2float_rd(o.lo.z); fbox[6 * b + 3] = __double2float_ru(o.hi.x);
  fbox[6 * b + 4] = __double2float_ru(o.hi.y); fbox[6 * b + 5] = __double2float_ru(o.hi.z);
}

// Float overlap of body boxes i and j (closed intervals, like intersection()).
__device__ __forceinline__ bool fbox_meet(const float* fb, int i, int j) {
  const float* a = fb + 6 * i;
  const float* b = fb + 6 * j;
  return a[0] <= b[3] && a[3] >= b[0] && a[1] <= b[4] && a[4] >= b[1] && a[2] <= b[5] && a[5] >= b[2];
}

__device__ __forceinline__ box ldbox(const double* bb, int i) {
  return box{mk(bb[6 * i], bb[6 * i + 1], bb[6 * i + 2]), mk(bb[6 * i + 3], bb[6 * i + 4], bb[6 * i + 5])};
}

// 3. overlaps: one warp per body row i, j over its scene (j != i), in increasing j; the
// FP64 intersection runs only where the outward-rounded float boxes meet.
__global__ void k_ov_count(Geo g, const double* bbox, const float* fbb, int* cnt_all, int* cnt_up) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= g.nb) return;
  int i = warp;
  if (!scene_on(g, i)) {
    if (lane == 0) cnt_all[i] = cnt_up[i] = 0;
    return;
  }
  box bi = ldbox(bbox, i);
  int ca = 0, cu = 0;
  for (int j0 = g.scene_beg[i]; j0 < g.scene_end[i]; j0 += 32) {
    int j = j0 + lane;
    bool hit = false;
    if (j < g.scene_end[i] && j != i && fbox_meet(fbb, i, j)) {
      box c;
      hit = intersection(bi, ldbox(bbox, j), c);
    }
    unsigned m = __ballot_sync(0xffffffffu, hit);
    unsigned mu = __ballot_sync(0xffffffffu, hit && j > i);
    ca += __popc(m);
    cu += __popc(mu);
  }
  if (lane == 0) {
    cnt_all[i] = ca;
    cnt_up[i] = cu;
  }
}

__global__ void k_ov_fill(Geo g, const double* bbox, const float* fbb, const int* row_ptr, const int* up_ptr, int* col,
                          int* rowid, int* upidx, int* ovI, int* ovJ, double* ovcull, float* ovcull_f) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= g.nb) return;
  int i = warp;
  if (!scene_on(g, i)) return;
  box bi = ldbox(bbox, i);
  int pa = row_ptr[i], pu = up_ptr[i];
  unsigned below = (1u << lane) - 1u;
  for (int j0 = g.scene_beg[i]; j0 < g.scene_end[i]; j0 += 32) {
    int j = j0 + lane;
    bool hit = false;
    box c;
    if (j < g.scene_end[i] && j != i && fbox_meet(fbb, i, j)) hit = intersection(bi, ldbox(bbox, j), c);
    unsigned m = __ballot_sync(0xffffffffu, hit);
    unsigned mu = __ballot_sync(0xffffffffu, hit && j > i);
    if (hit) {
      int e = pa + __popc(m & below);
      col[e] = j;
      rowid[e] = i;
      if (j > i) {
        int u = pu + __popc(mu & below);
        upidx[e] = u;
        ovI[u] = i;
        ovJ[u] = j;
        double* cb = ovcull + 6 * u;
        cb[0] = c.lo.x; cb[1] = c.lo.y; cb[2] = c.lo.z; cb[3] = c.hi.x; cb[4] = c.hi.y; cb[5] = c.hi.z;
        float* cf = ovcull_f + 6 * u;
        cf[0] = __double2float_rd(c.lo.x); cf[1] = __double2float_rd(c.lo.y); cf[2] = __double2float_rd(c.lo.z);
        cf[3] = __double2float_ru(c.hi.x); cf[4] = __double2float_ru(c.hi.y); cf[5] = __double2float_ru(c.hi.z);
      } else {
        upidx[e] = -1;
      }
    }
    pa += __popc(m);
    pu += __popc(mu);
  }
}

// lower entries (i > j): unique overlap of (j, i) by binary search in row j
__global__ void k_ov_lower(int nnz, const int* row_ptr, const int* col, const int* rowid, int* upidx) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nnz) return;
  int i = rowid[e], j = col[e];
  if (j > i) return;
  int lo = row_ptr[j], hi = row_ptr[j + 1];
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (col[mid] < i) lo = mid + 1;
    else hi = mid;
  }
  upidx[e] = (lo < row_ptr[j + 1] && col[lo] == i) ? upidx[lo] : -1;
}

// ---------------------------------------------------------------------------------
// Float prefilter boxes of every primitive (outward rounded). Vertices first, from their FP64
// positions (here at X; k_project writes those of the culls, at X or of the trajectory from
// Xq to X); edges and faces are then the float unions of their vertices' boxes: rounding down
// (up) commutes with min (max), so rd(min(a, b)) = min(rd a, rd b) and the result equals
// rounding the FP64 box, without any FP64 min/max.
__global__ void k_vert_boxes(Geo g, float* vb) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.nv) return;
  d3 p = ldX(g.X, g.nv, t);
  put_fbox(vb + 6 * t, box{p, p});
}
// Float positions (to nearest) of every vertex at q and at the target, for the FP32
// certificates of the trajectories.
__global__ void k_traj_floats(Geo g, float* ve) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.nv) return;
  const d3 p = ldX(g.Xq, g.nv, t), q = ldX(g.X, g.nv, t);
  float* o = ve + 6 * (size_t)t;
  o[0] = __double2float_rn(p.x); o[1] = __double2float_rn(p.y); o[2] = __double2float_rn(p.z);
  o[3] = __double2float_rn(q.x); o[4] = __double2float_rn(q.y); o[5] = __double2float_rn(q.z);
}
__device__ __forceinline__ void fbox_union(float* o, const float* a, const float* b) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    o[c] = fminf(o[c], fminf(a[c], b[c]));
    o[c + 3] = fmaxf(o[c + 3], fmaxf(a[c + 3], b[c + 3]));
  }
}
__global__ void k_prim_boxes(Geo g, const float* vb, float* eb, float* fb, BinClusters cl) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  float o[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  const int ne32 = (g.ne + 31) & ~31;  // the faces start a warp of their own
  if (t < ne32) {
    if (t < g.ne) {
      fbox_union(o, vb + 6 * g.ev[2 * t], vb + 6 * g.ev[2 * t + 1]);
#pragma unroll
      for (int c = 0; c < 6; ++c) eb[6 * t + c] = o[c];
    }
    if (cl.e) put_cluster(cl.e, t, o);
    return;
  }
  t -= ne32;
  if ((t & ~31) >= g.nf) return;
  if (t < g.nf) {
    const float* v2 = vb + 6 * g.fv[3 * t + 2];
    fbox_union(o, vb + 6 * g.fv[3 * t], vb + 6 * g.fv[3 * t + 1]);
    fbox_union(o, v2, v2);
#pragma unroll
    for (int c = 0; c < 6; ++c) fb[6 * t + c] = o[c];
  }
  if (cl.f) put_cluster(cl.f, t, o);
}

__device__ __forceinline__ bool f_overlap(const float* a, const float* b) {
  return a[0] <= b[3] && a[3] >= b[0] && a[1] <= b[4] && a[4] >= b[1] && a[2] <= b[5] && a[5] >= b[2];
}

// Exact primitive boxes (same construction as the reference's compute_aabb overloads).
__device__ __forceinline__ box vbox_exact(const Geo& g, int v, int traj) {
  d3 p = ldX(g.X, g.nv, v);
  return traj ? box2(p, ldX(g.Xq, g.nv, v)) : box{p, p};
}
__device__ __forceinline__ box ebox_exact(const Geo& g, int e, int traj) {
  int a = g.ev[2 * e], c = g.ev[2 * e + 1];
  d3 p0 = ldX(g.X, g.nv, a), p1 = ldX(g.X, g.nv, c);
  return traj ? box4(p0, p1, ldX(g.Xq, g.nv, a), ldX(g.Xq, g.nv, c)) : box2(p0, p1);
}
__device__ __forceinline__ box fbox_exact(const Geo& g, int f, int traj) {
  int a = g.fv[3 * f], c = g.fv[3 * f + 1], d = g.fv[3 * f + 2];
  box b = box3(ldX(g.X, g.nv, a), ldX(g.X, g.nv, c), ldX(g.X, g.nv, d));
  if (traj) b = merge(box3(ldX(g.Xq, g.nv, a), ldX(g.Xq, g.nv, c), ldX(g.Xq, g.nv, d)), b);
  return b;
}

__device__ __forceinline__ void finflate(const float* s, float ds, float* o) {
  o[0] = __fsub_rd(s[0], ds); o[1] = __fsub_rd(s[1], ds); o[2] = __fsub_rd(s[2], ds);
  o[3] = __fadd_ru(s[3], ds); o[4] = __fadd_ru(s[4], ds); o[5] = __fadd_ru(s[5], ds);
}

// Union of the vertex boxes of a body, by a warp: the clusters inside its range, the rest one by one.
__device__ __forceinline__ void tight_box(const Geo& g, int body, const float* vb, const float* cl, float (&o)[6]) {
  const int lane = threadIdx.x & 31, beg = g.v_off[body], end = g.v_off[body + 1];
  const int cb = (beg + 31) >> 5, ce = end >> 5;
  float q[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (cb < ce) {
    for (int c = cb + lane; c < ce; c += 32) fbox_union(q, cl + 6 * (size_t)c, cl + 6 * (size_t)c);
    if (beg + lane < 32 * cb) fbox_union(q, vb + 6 * (size_t)(beg + lane), vb + 6 * (size_t)(beg + lane));
    if (32 * ce + lane < end) fbox_union(q, vb + 6 * (size_t)(32 * ce + lane), vb + 6 * (size_t)(32 * ce + lane));
  } else {
    for (int k = beg + lane; k < end; k += 32) fbox_union(q, vb + 6 * (size_t)k, vb + 6 * (size_t)k);
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int r = c < 3 ? __reduce_min_sync(0xffffffffu, ford(q[c])) : __reduce_max_sync(0xffffffffu, ford(q[c]));
    o[c] = __int_as_float(r >= 0 ? r : r ^ 0x7fffffff);
  }
}

// 4. binning: one warp per (overlap, side); kinds per side: vertices, edges, faces.
// list slot k of overlap u: 0 vi, 1 ei, 2 fi, 3 vj, 4 ej, 5 fj.
// Binning passes: BIN_COUNT counts each list, BIN_WRITE writes it at offsets from a scan
// of those counts, BIN_ONCE writes it at offsets sized by the body's primitive counts and
// stores the count (one pass instead of two when that capacity fits).
enum { BIN_COUNT = 0, BIN_WRITE = 1, BIN_ONCE = 2 };

// Capacity of list slot (overlap u, side, kind): the primitive count of that body (cap null: not
// wanted), and the box of each body's vertex boxes (a warp a body).
__global__ void k_bin_caps(Geo g, int nov, const int* ovI, const int* ovJ, const float* vb, const float* cl, int* cap,
                           float* tight) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, w = t >> 5, lane = threadIdx.x & 31;
  if (w < g.nb) {
    float o[6];
    tight_box(g, w, vb, cl, o);
    if (lane == 0)
#pragma unroll
      for (int c = 0; c < 6; ++c) tight[6 * w + c] = o[c];
  }
  if (!cap || t >= 6 * nov) return;
  int u = t / 6, side = (t / 3) & 1, kind = t % 3;
  int body = side ? ovJ[u] : ovI[u];
  const int* o = kind == 0 ? g.v_off : (kind == 1 ? g.e_off : g.f_off);
  cap[t] = o[body + 1] - o[body];
}

// A body has thousands of boxes and an overlap meets a few per cent of them: the clusters are
// tested first, a lane each, and only the primitives of those that meet the cull box are read
// (bodies of up to 64 primitives of a kind: all). The boxes of both bodies of every overlap came
// from L2 before (1.8 GB on the pile's 9871 overlaps, 168 us; with the clusters 108 us).
// The cull box comes from body boxes that are loose (the affine images of the rest boxes), so the
// lists also leave out what no box of the other body can hit: entries on the A side of their
// sub-problem (vertices, and the first body's edges), inflated by ds, that miss the union of the
// other body's vertex boxes, and entries on the B side that miss that union inflated (inflating
// rounds monotonically, so this is the union of the inflated boxes); where neither body's box
// meets the other's inflated one the lists are empty. Now 54 us, and k_refine 91 -> 27 us.
__global__ void __launch_bounds__(256, 3) k_bin(Geo g, float ds, int nov, int pass, int traj, const int* ovI, const int* ovJ,
                                                const double* ovcull, const float* ovcull_f, const float* vb,
                                                const float* eb, const float* fb, BinClusters cl, const float* tights, int* cnt,
                                                const int* off, int* lst) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= 2 * nov) return;
  int u = warp >> 1, side = warp & 1;
  int body = side ? ovJ[u] : ovI[u];
  float cf[6], ci[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) cf[k] = ovcull_f[6 * u + k];
  // Float bounds inside the FP64 cull box: cull.lo <= ci[0..2], cull.hi >= ci[3..5]. The
  // float box of a primitive is (rd(lo), ru(hi)) of its FP64 box, so rd(lo) < ci_hi gives
  // lo <= nextup(rd(lo)) <= ci_hi <= cull.hi; a primitive passing that on all six sides
  // overlaps the cull box exactly and needs no FP64 test.
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ci[k] = nextafterf(cf[k], INFINITY);
    ci[k + 3] = nextafterf(cf[k + 3], -INFINITY);
  }
  unsigned below = (1u << lane) - 1u;
  float tight[6];  // of the other body
  {
    float own[6], x[6];
    const int other = side ? ovI[u] : ovJ[u];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      tight[k] = tights[6 * other + k];
      own[k] = tights[6 * body + k];
    }
    finflate(own, ds, x);
    bool meet = f_overlap(x, tight);
    finflate(tight, ds, x);
    meet = (meet || f_overlap(own, x)) && f_overlap(cf, own);
    if (!meet) {
      if (pass != BIN_WRITE && lane < 3) cnt[6 * u + 3 * side + lane] = 0;
      return;
    }
  }
#pragma unroll 1
  for (int kind = 0; kind < 3; ++kind) {
    const bool on_a = kind == 0 || (kind == 1 && side == 0);
    float tb[6];
    finflate(tight, on_a ? 0.f : ds, tb);
    const float da = on_a ? ds : 0.f;
    auto near_body = [&](const float (&q)[6]) {
      float x[6];
      finflate(q, da, x);
      return f_overlap(x, tb);
    };
    int beg, end;
    const float *fbx, *cbx;
    if (kind == 0) { beg = g.v_off[body]; end = g.v_off[body + 1]; fbx = vb; cbx = cl.v; }
    else if (kind == 1) { beg = g.e_off[body]; end = g.e_off[body + 1]; fbx = eb; cbx = cl.e; }
    else { beg = g.f_off[body]; end = g.f_off[body + 1]; fbx = fb; cbx = cl.f; }
    int slot = u * 6 + side * 3 + kind;
    int c = 0, base = pass != BIN_COUNT ? off[slot] : 0;
    const bool few = end - beg <= 64;
    const int c_end = (end + 31) >> 5;  // clusters of [beg, end): beg / 32 .. c_end - 1
    for (int c0 = beg >> 5; c0 < c_end; c0 += 32) {
      bool near = c0 + lane < c_end;
      if (near && !few) {
        const float2* src = reinterpret_cast<const float2*>(cbx + 6 * (size_t)(c0 + lane));
        const float2 a = src[0], b = src[1], d = src[2];
        const float q[6] = {a.x, a.y, b.x, b.y, d.x, d.y};
        near = f_overlap(cf, q) && near_body(q);
      }
      unsigned todo = __ballot_sync(0xffffffffu, near);
      // BIN_R clusters per step: their boxes are loaded before any is tested, so the warp
      // keeps several L2 loads in flight
      constexpr int BIN_R = 4;
      while (todo) {
        float q[BIN_R][6];
        const unsigned taken = todo;
        auto next = [&](unsigned& bits) {  // this lane's primitive of the next cluster
          const int k = bits ? 32 * (c0 + __ffs(bits) - 1) + lane : end;
          bits &= bits - 1;
          return k;
        };
#pragma unroll
        for (int r = 0; r < BIN_R; ++r) {
          const int k = next(todo);
          if (k >= beg && k < end) {
            const float2* src = reinterpret_cast<const float2*>(fbx + 6 * (size_t)k);
            float2 a = src[0], b = src[1], d = src[2];
            q[r][0] = a.x; q[r][1] = a.y; q[r][2] = b.x; q[r][3] = b.y; q[r][4] = d.x; q[r][5] = d.y;
          } else {
            q[r][0] = q[r][1] = q[r][2] = INFINITY;  // misses every box
            q[r][3] = q[r][4] = q[r][5] = -INFINITY;
          }
        }
        unsigned hits = 0, open = 0;  // bit r
#pragma unroll
        for (int r = 0; r < BIN_R; ++r) {
          const bool in = q[r][0] < ci[3] && q[r][1] < ci[4] && q[r][2] < ci[5] && q[r][3] > ci[0] &&
                          q[r][4] > ci[1] && q[r][5] > ci[2];
          const bool meets = f_overlap(cf, q[r]) && near_body(q[r]);
          hits |= (unsigned)(meets && in) << r;
          open |= (unsigned)(meets && !in) << r;
        }
        if (__any_sync(0xffffffffu, open)) {  // rare: the boxes of these end within a rounding
          unsigned bits = taken;
#pragma unroll 1
          for (int r = 0; r < BIN_R; ++r) {
            const int k = next(bits);
            if (!(open >> r & 1)) continue;
            box b = (kind == 0) ? vbox_exact(g, k, traj) : (kind == 1 ? ebox_exact(g, k, traj) : fbox_exact(g, k, traj));
            hits |= (unsigned)overlaps(box{mk(ovcull[6 * u], ovcull[6 * u + 1], ovcull[6 * u + 2]),
                                           mk(ovcull[6 * u + 3], ovcull[6 * u + 4], ovcull[6 * u + 5])}, b) << r;
          }
        }
        unsigned bits = taken;
#pragma unroll
        for (int r = 0; r < BIN_R; ++r) {
          const int k = next(bits);
          const bool hit = hits >> r & 1;
          unsigned m = __ballot_sync(0xffffffffu, hit);
          if (pass != BIN_COUNT && hit) lst[base + c + __popc(m & below)] = k - beg;
          c += __popc(m);
        }
      }
    }
    if (pass != BIN_WRITE && lane == 0) cnt[slot] = c;
  }
}

constexpr int NT = 256;     // narrow-phase threads per CTA
constexpr int TILE = 384;   // primitives of one list staged in shared memory (2 x 9 kB)
constexpr int REC_CAP = 2048;  // candidates of one overlap kept in shared memory for sorting
// Box-phase candidates per thread between two test phases (STEP), and the queue of
// float-box hits they fill (NT * STEP entries). A longer box phase runs the phase after it
// less often; a shorter one leaves shared memory for more CTAs per SM. The result does not
// depend on STEP (candidates are sorted by key before they are written, TOIs are
// min-reduced), so the autotuner picks among these variants by time: pair cull (mode 0)
// 16 / 8 / 48, CCD (mode 2) 24 / 36 / 64. No variant wins everywhere (medians of seven
// handles, us): 1024 bodies of the pile 153 / 193 / 149 and 144 / 145 / 114, 64 of them
// 31 / 29 / 28 and 22 / 17 / 17, 256 columns 195 / 156 / 230 and 78 / 68 / 112, a chain of 200
// 25 / 24 / 24 and 24 / 19 / 20. The middle ones are the defaults: the best of the small scenes,
// which are the ones that are not tuned, and within a third of the best elsewhere.
constexpr int kNarrowVariants = 3;
constexpr int kNarrowStep[2][kNarrowVariants] = {{16, 8, 48}, {24, 36, 64}};
constexpr int kNarrowDefault = 1;
// dynamic shared memory of k_narrow_scan<MODE, STEP>: boxes, queue, candidates (MODE 0)
// (MODE 0 also stages the vertex ids of the staged primitives: 2 per A entry, 3 per B)
__host__ __device__ constexpr size_t narrow_smem(int mode, int step) {
  return 2 * TILE * 6 * sizeof(float) + (size_t)NT * step * sizeof(unsigned) +
         (mode == 0 ? REC_CAP * sizeof(unsigned long long) + 5 * TILE * sizeof(int) : 0);
}

// Order-preserving key of a double for atomicMin on unsigned 64-bit.
__device__ __forceinline__ unsigned long long dkey(double x) {
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// Exact narrow-phase test of one candidate at the culled configuration (vtn 1/2):
// returns 0 (no pair) or 1 + distance type. sub 0/1: vertex v (global) of body A vs
// face f (global) of body B; sub 2: edge ea vs edge eb.
// The candidate is given by its four vertex ids: (point, triangle) for sub 0/1, (edge a,
// edge b) for sub 2.
__device__ __forceinline__ int exact_pair_v(const Geo& g, const Params& P, int sub, int v0, int v1, int v2, int v3) {
  int nv = g.nv;
  if (sub < 2) {
    d3 p = ldX(g.X, nv, v0);
    box bv = inflate(box{p, p}, P.d_sqrt);
    d3 t0 = ldX(g.X, nv, v1), t1 = ldX(g.X, nv, v2), t2 = ldX(g.X, nv, v3);
    if (!overlaps(bv, box3(t0, t1, t2))) return 0;
    int ty = pt_type(p, t0, t1, t2);
    return (pt_dist(p, t0, t1, t2, ty) < P.dhat) ? 1 + ty : 0;
  }
  d3 a0 = ldX(g.X, nv, v0), a1 = ldX(g.X, nv, v1);
  d3 b0 = ldX(g.X, nv, v2), b1 = ldX(g.X, nv, v3);
  if (!overlaps(inflate(box2(a0, a1), P.d_sqrt), box2(b0, b1))) return 0;
  int ty = ee_type(a0, a1, b0, b1);
  return (ee_dist(a0, a1, b0, b1, ty) < P.dhat) ? 1 + ty : 0;
}
// Vertex ids of candidate (pa, pb): point pa and face pb (sub 0/1), edges pa and pb (sub 2).
__device__ __forceinline__ void pair_vertex_ids(const Geo& g, int sub, int pa, int pb, int (&v)[4]) {
  if (sub < 2) {
    v[0] = pa; v[1] = g.fv[3 * pb]; v[2] = g.fv[3 * pb + 1]; v[3] = g.fv[3 * pb + 2];
  } else {
    v[0] = g.ev[2 * pa]; v[1] = g.ev[2 * pa + 1]; v[2] = g.ev[2 * pb]; v[3] = g.ev[2 * pb + 1];
  }
}
__device__ __forceinline__ int exact_pair(const Geo& g, const Params& P, int sub, int pa, int pb) {
  int v[4];
  pair_vertex_ids(g, sub, pa, pb, v);
  return exact_pair_v(g, P, sub, v[0], v[1], v[2], v[3]);
}

// ---- FP32 lower bounds of pair distances with tracked rounding errors ----
// A value v carries a bound e on |v - exact|, where "exact" is the same expression in real
// arithmetic on the FP64 positions. Inputs are the lower corners of the vertex float
// boxes (rd(x), |x - rd(x)| <= 2^-23 |x|); every operation adds its rounding (u |v| with
// u = 2^-24, slightly enlarged, plus an underflow term), and the error terms themselves
// are accumulated rounding up. The bounds are therefore rigorous; they let most float-box
// hits be rejected without the FP64 test (GB300 issues FP64 at 1/64 of the FP32 rate).
struct EF {
  float v, e;
};
__device__ __forceinline__ EF ef_in(float x) { return {x, __fadd_ru(__fmul_ru(fabsf(x), 1.2042e-7f), 1e-37f)}; }
__device__ __forceinline__ float ef_rnd(float v) { return __fadd_ru(__fmul_ru(fabsf(v), 6.0e-8f), 1e-37f); }
__device__ __forceinline__ EF ef_add(EF a, EF b) {
  const float v = __fadd_rn(a.v, b.v);
  return {v, __fadd_ru(__fadd_ru(a.e, b.e), ef_rnd(v))};
}
__device__ __forceinline__ EF ef_sub(EF a, EF b) {
  const float v = __fsub_rn(a.v, b.v);
  return {v, __fadd_ru(__fadd_ru(a.e, b.e), ef_rnd(v))};
}
__device__ __forceinline__ EF ef_mul(EF a, EF b) {
  const float v = __fmul_rn(a.v, b.v);
  float e = __fadd_ru(__fmul_ru(fabsf(a.v), b.e), __fmul_ru(fabsf(b.v), a.e));
  e = __fadd_ru(e, __fmul_ru(a.e, b.e));
  return {v, __fadd_ru(e, ef_rnd(v))};
}
struct EF3 {
  EF x[3];
};
__device__ __forceinline__ EF3 ef3_in(const float* p) { return {{ef_in(p[0]), ef_in(p[1]), ef_in(p[2])}}; }
__device__ __forceinline__ EF3 ef3_sub(const EF3& a, const EF3& b) {
  return {{ef_sub(a.x[0], b.x[0]), ef_sub(a.x[1], b.x[1]), ef_sub(a.x[2], b.x[2])}};
}
__device__ __forceinline__ EF3 ef3_cross(const EF3& a, const EF3& b) {
  return {{ef_sub(ef_mul(a.x[1], b.x[2]), ef_mul(a.x[2], b.x[1])),
           ef_sub(ef_mul(a.x[2], b.x[0]), ef_mul(a.x[0], b.x[2])),
           ef_sub(ef_mul(a.x[0], b.x[1]), ef_mul(a.x[1], b.x[0]))}};
}
__device__ __forceinline__ EF ef3_dot(const EF3& a, const EF3& b) {
  return ef_add(ef_add(ef_mul(a.x[0], b.x[0]), ef_mul(a.x[1], b.x[1])), ef_mul(a.x[2], b.x[2]));
}
// lower bound of num^2 / den for num known positive by at least lo > 0, den <= den.v + den.e
__device__ __forceinline__ float ef_ratio_lb(float lo, EF den) {
  return __fdiv_rd(__fmul_rd(lo, lo), __fadd_ru(den.v, den.e));
}
// lower bound of |x| (0 when the sign is not certain)
__device__ __forceinline__ float ef_abs_lb(EF x) { return fmaxf(__fsub_rd(fabsf(x.v), x.e), 0.f); }

// Lower bound of the squared point-triangle distance: the point-plane distance combined
// with the largest distance of the point beyond one of the triangle's edge lines in the
// plane (the two components are orthogonal).
__device__ __forceinline__ float lb2_pt_f(const float* p, const float* t0, const float* t1, const float* t2) {
  const EF3 P = ef3_in(p), T0 = ef3_in(t0), T1 = ef3_in(t1), T2 = ef3_in(t2);
  const EF3 e1 = ef3_sub(T1, T0), e2 = ef3_sub(T2, T0), e3 = ef3_sub(T2, T1), w = ef3_sub(P, T0);
  const EF3 n = ef3_cross(e1, e2);
  const EF nn = ef3_dot(n, n);
  const float sl = ef_abs_lb(ef3_dot(w, n));
  float lb = sl > 0.f ? ef_ratio_lb(sl, nn) : 0.f;
  // outward in-plane edge normals m = edge x n (edges t0->t1, t1->t2, t2->t0)
  const EF3 me[3] = {ef3_cross(e1, n), ef3_cross(e3, n), ef3_cross(ef3_sub(T0, T2), n)};
  const EF3 ve[3] = {w, ef3_sub(P, T1), ef3_sub(P, T2)};
  float side = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const EF num = ef3_dot(ve[k], me[k]);
    const float lo = __fsub_rd(num.v, num.e);
    if (lo > 0.f) side = fmaxf(side, ef_ratio_lb(lo, ef3_dot(me[k], me[k])));
  }
  return __fadd_rd(lb, side);
}

// Lower bound of the squared segment-segment distance: the line-line distance combined
// with one in-plane separation: one segment entirely on one side of the other's line, or
// beyond one of its ends along its direction.
__device__ __forceinline__ float lb2_ee_f(const float* a0, const float* a1, const float* b0, const float* b1) {
  const EF3 A0 = ef3_in(a0), A1 = ef3_in(a1), B0 = ef3_in(b0), B1 = ef3_in(b1);
  const EF3 u = ef3_sub(A1, A0), v = ef3_sub(B1, B0);
  const EF3 n = ef3_cross(u, v);
  const EF nn = ef3_dot(n, n);
  const float sl = ef_abs_lb(ef3_dot(ef3_sub(B0, A0), n));
  float lb = sl > 0.f ? ef_ratio_lb(sl, nn) : 0.f;
  float sep = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const EF3& d = k == 0 ? u : v;
    const EF3& base = k == 0 ? A0 : B0;
    const EF3 q0 = ef3_sub(k == 0 ? B0 : A0, base), q1 = ef3_sub(k == 0 ? B1 : A1, base);
    // the other segment on one side of this one's line (in-plane normal n x d)
    const EF3 m = ef3_cross(n, d);
    const EF x0 = ef3_dot(q0, m), x1 = ef3_dot(q1, m);
    float lo = 0.f;
    if (__fsub_rd(x0.v, x0.e) > 0.f && __fsub_rd(x1.v, x1.e) > 0.f)
      lo = fminf(__fsub_rd(x0.v, x0.e), __fsub_rd(x1.v, x1.e));
    else if (__fadd_ru(x0.v, x0.e) < 0.f && __fadd_ru(x1.v, x1.e) < 0.f)
      lo = fminf(-__fadd_ru(x0.v, x0.e), -__fadd_ru(x1.v, x1.e));
    if (lo > 0.f) sep = fmaxf(sep, ef_ratio_lb(lo, ef3_dot(m, m)));
    // the other segment beyond one end of this one along d
    const EF dd = ef3_dot(d, d);
    const EF y0 = ef3_dot(q0, d), y1 = ef3_dot(q1, d);
    const EF z0 = ef_sub(y0, dd), z1 = ef_sub(y1, dd);
    lo = 0.f;
    if (__fsub_rd(z0.v, z0.e) > 0.f && __fsub_rd(z1.v, z1.e) > 0.f)
      lo = fminf(__fsub_rd(z0.v, z0.e), __fsub_rd(z1.v, z1.e));
    else if (__fadd_ru(y0.v, y0.e) < 0.f && __fadd_ru(y1.v, y1.e) < 0.f)
      lo = fminf(-__fadd_ru(y0.v, y0.e), -__fadd_ru(y1.v, y1.e));
    if (lo > 0.f) sep = fmaxf(sep, ef_ratio_lb(lo, dd));
  }
  return __fadd_rd(lb, sep);
}

// Rejects a float-box hit when the float lower bound of its squared distance reaches
// dhat (1 + 1e-4) and the primitives are well shaped (no edge with squared length below
// 2e-6 dhat, no triangle or edge pair with |n|^2 below 2e-6 of the product of the squared
// edge lengths, so the FP64 distance formulas are accurate far inside the 1e-4 margin):
// such a pair is one the FP64 test rejects too, so it never reaches that test.
// The candidate is given by its four vertex ids, as for exact_pair_v.
__device__ __forceinline__ bool f_reject_v(const float* vb, int sub, int v0, int v1, int v2, int v3, float lim) {
  const float *x0 = vb + 6 * v0, *x1 = vb + 6 * v1, *x2 = vb + 6 * v2, *x3 = vb + 6 * v3;
  // well-shaped guards in plain float with twice the FP64 guards' margins
  float ea[3], eb[3];
  for (int c = 0; c < 3; ++c) {
    ea[c] = sub < 2 ? x2[c] - x1[c] : x1[c] - x0[c];
    eb[c] = sub < 2 ? x3[c] - x1[c] : x3[c] - x2[c];
  }
  const float la = ea[0] * ea[0] + ea[1] * ea[1] + ea[2] * ea[2];
  const float lb = eb[0] * eb[0] + eb[1] * eb[1] + eb[2] * eb[2];
  const float nx = ea[1] * eb[2] - ea[2] * eb[1], ny = ea[2] * eb[0] - ea[0] * eb[2], nz = ea[0] * eb[1] - ea[1] * eb[0];
  const float nn = nx * nx + ny * ny + nz * nz;
  float lmin = fminf(la, lb);
  if (sub < 2) {
    const float d0 = x3[0] - x2[0], d1 = x3[1] - x2[1], d2 = x3[2] - x2[2];
    lmin = fminf(lmin, d0 * d0 + d1 * d1 + d2 * d2);
  }
  if (!(lmin >= 2e-6f * lim) || !(nn >= 2e-6f * la * lb)) return false;
  const float l2 = sub < 2 ? lb2_pt_f(x0, x1, x2, x3) : lb2_ee_f(x0, x1, x2, x3);
  return l2 >= lim;
}

// Trajectory time of impact of one candidate (vtn 3), exact box test included.
__device__ __forceinline__ double exact_toi(const Geo& g, int sub, int pa, int pb) {
  int nv = g.nv;
  d3 p[4], q[4];  // at q and at the target
  if (sub < 2) {
    const int vid[4] = {pa, g.fv[3 * pb], g.fv[3 * pb + 1], g.fv[3 * pb + 2]};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      p[k] = ldX(g.Xq, nv, vid[k]);
      q[k] = ldX(g.X, nv, vid[k]);
    }
    if (!overlaps(box2(p[0], q[0]), merge(box3(p[1], p[2], p[3]), box3(q[1], q[2], q[3])))) return 1.0;
    return toi_fast<0>(p, q);
  }
  const int vid[4] = {g.ev[2 * pa], g.ev[2 * pa + 1], g.ev[2 * pb], g.ev[2 * pb + 1]};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    p[k] = ldX(g.Xq, nv, vid[k]);
    q[k] = ldX(g.X, nv, vid[k]);
  }
  if (!overlaps(box4(p[0], p[1], q[0], q[1]), box4(p[2], p[3], q[2], q[3]))) return 1.0;
  return toi_fast<1>(p, q);
}

// Certificate that exact_toi of the candidate is 1, from the vertices' float positions at q
// and at the target (6 floats each).
__device__ __forceinline__ f3 ldf3(const float* p) { return f3{p[0], p[1], p[2]}; }
__device__ __forceinline__ bool f_toi_miss(const Geo& g, const float* ve, int sub, int pa, int pb) {
  if (sub < 2) {
    f3 t0[3], t1[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float* p = ve + 6 * (size_t)g.fv[3 * pb + k];
      t0[k] = ldf3(p);
      t1[k] = ldf3(p + 3);
    }
    const float* p = ve + 6 * (size_t)pa;
    return f_pt_miss(ldf3(p), ldf3(p + 3), t0, t1);
  }
  f3 a0[2], a1[2], b0[2], b1[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float *p = ve + 6 * (size_t)g.ev[2 * pa + k], *q = ve + 6 * (size_t)g.ev[2 * pb + k];
    a0[k] = ldf3(p);
    a1[k] = ldf3(p + 3);
    b0[k] = ldf3(q);
    b1[k] = ldf3(q + 3);
  }
  return f_ee_miss(a0, a1, b0, b1);
}

// Candidates of the trajectory narrow phase left to the FP64 test: (point, face) or (~edge,
// edge) by their global ids.
struct ToiCand {
  const float* ve;   // float positions of the vertices at q and at the target
  int2* cand;
  unsigned* n;
  unsigned cap;
};
// Room for as many candidates as the overlaps' lists can have entries (two spheres of 3842
// primitives each: 7684), 4096 at least and 16 MB at most; a candidate past it is evaluated
// where it is found, and the list is then large enough for the next call. (16 MB for every handle
// made one of ten cubes 21.8 MB instead of 2.9.)
constexpr unsigned kToiCandMin = 1u << 12, kToiCandMax = 1u << 21;

// Candidates of the pair cull left to the FP64 test, by overlap, each overlap's sorted by
// (sub, i, j): the point-triangle ones from the front of the buffer, the edge-edge ones from its
// end, so that a warp of k_narrow_exact runs one kind. seg: an overlap's two segments (first
// entry, count; first entry -1: not staged); total: both kinds' candidates (more than cap
// together: the segments are not valid and the cull is repeated with a larger buffer).
struct StageOut {
  unsigned long long* key;
  int* ov;
  int8_t* ty;  // distance type, -1: rejected (k_narrow_exact)
  int4* seg;   // {first PT, PT count, first EE, EE count}
  int* total;
  int cap;
  __device__ __forceinline__ bool valid() const { return (long long)total[0] + total[1] <= cap; }
};

struct NarrowOut {
  int *pt, *pt_ov, *ee, *ee_ov;
  int8_t *pt_ty, *ee_ty;
};

struct SubLists {
  int A, B, nA, nB, offA, offB;
  const int *LA, *LB;
  const float *boxA, *boxB;
};

__device__ __forceinline__ SubLists sub_lists(const Geo& g, int sub, int I, int J, const int* n, const int* o,
                                              const int* lst, const float* vb, const float* eb, const float* fb) {
  SubLists L;
  int la = sub == 0 ? 0 : (sub == 1 ? 3 : 1);  // vi / vj / ei
  int lb = sub == 0 ? 5 : (sub == 1 ? 2 : 4);  // fj / fi / ej
  L.A = (sub == 1) ? J : I;
  L.B = (sub == 1) ? I : J;
  L.nA = n[la];
  L.nB = n[lb];
  L.boxA = sub < 2 ? vb : eb;
  L.boxB = sub < 2 ? fb : eb;
  L.offA = sub < 2 ? g.v_off[L.A] : g.e_off[L.A];
  L.offB = sub < 2 ? g.f_off[L.B] : g.e_off[L.B];
  L.LA = lst + o[la];
  L.LB = lst + o[lb];
  return L;
}

// Warp-wide union of float boxes (min of lo, max of hi); every lane gets it.
__device__ __forceinline__ void warp_box_union(float* b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      float v = __shfl_xor_sync(0xffffffffu, b[c], o);
      b[c] = c < 3 ? fminf(b[c], v) : fmaxf(b[c], v);
    }
}

// Keeps, in order and in place, the entries of list L[0..n) whose float box (inflated by
// ds when `infl`) hits box `q`; returns the new length. Each chunk of 32 entries is read
// before any of it is written, and writes never pass reads.
__device__ __forceinline__ int warp_compact(int* L, int n, int off, const float* boxes, bool infl, float ds,
                                            const float* q) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int kept = 0;
  for (int k0 = 0; k0 < n; k0 += 32) {
    int k = k0 + lane;
    int id = 0;
    bool keep = false;
    if (k < n) {
      id = L[k];
      float bx[6];
      const float* src = boxes + 6 * (off + id);
      if (infl) finflate(src, ds, bx);
      else
#pragma unroll
        for (int c = 0; c < 6; ++c) bx[c] = src[c];
      keep = f_overlap(bx, q);
    }
    unsigned m = __ballot_sync(0xffffffffu, keep);
    if (keep) L[kept + __popc(m & below)] = id;
    kept += __popc(m);
  }
  return kept;
}

// 4b. Shrinks the two lists of every sub-problem (one warp per overlap and sub-problem) so
// that every candidate pair whose float boxes hit survives: A keeps the entries hitting
// the union of the B boxes, then B keeps the entries hitting the union of the kept A boxes
// (A inflated by ds for the pair cull, not for trajectories). The reference's loose body
// boxes bin whole caps of both bodies; this leaves the part near the other body, and most
// sub-problems of a pile end up empty before any CTA of the narrow phase is spent on them.
template <bool INFL>
__global__ void k_refine(Geo g, float ds, int nov, const int* ovI, const int* ovJ, int* cnt, const int* off, int* lst,
                         const float* vb, const float* eb, const float* fb) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= 3 * nov) return;
  const int u = warp / 3, sub = warp - 3 * u;
  int* n = cnt + 6 * u;
  SubLists L = sub_lists(g, sub, ovI[u], ovJ[u], n, off + 6 * u, lst, vb, eb, fb);
  if (L.nA == 0 || L.nB == 0) return;
  float bb[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int k = lane; k < L.nB; k += 32) {
    const float* b = L.boxB + 6 * (L.offB + L.LB[k]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      bb[c] = fminf(bb[c], b[c]);
      bb[c + 3] = fmaxf(bb[c + 3], b[c + 3]);
    }
  }
  warp_box_union(bb);
  int* LA = const_cast<int*>(L.LA);
  int* LB = const_cast<int*>(L.LB);
  const int nA = warp_compact(LA, L.nA, L.offA, L.boxA, INFL, ds, bb);
  float ba[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int k = lane; k < nA; k += 32) {
    float a[6];
    const float* src = L.boxA + 6 * (L.offA + LA[k]);
    if (INFL) finflate(src, ds, a);
    else
#pragma unroll
      for (int c = 0; c < 6; ++c) a[c] = src[c];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ba[c] = fminf(ba[c], a[c]);
      ba[c + 3] = fmaxf(ba[c + 3], a[c + 3]);
    }
  }
  warp_box_union(ba);
  const int nB = nA ? warp_compact(LB, L.nB, L.offB, L.boxB, false, ds, ba) : 0;
  if (lane == 0) {
    const int la = sub == 0 ? 0 : (sub == 1 ? 3 : 1), lb = sub == 0 ? 5 : (sub == 1 ? 2 : 4);
    n[la] = nA;
    n[lb] = nB;
  }
}

// One entry of a list into shared memory: the float box of A entry k (inflated by sqrt(dhat),
// rounded outward, for the pair cull) or B entry k, and for the pair cull (v not null) the vertex
// ids (A: a point's id or an edge's two at v[0 ..]; B: a face's three or an edge's two).
__device__ __forceinline__ void stage_a(const Geo& g, int sub, const SubLists& L, int k, bool inflate, float ds_f,
                                        float* s, int* v) {
  const int pa = L.offA + L.LA[k];
  const float* src = L.boxA + 6 * pa;
  if (inflate) finflate(src, ds_f, s);
  else
#pragma unroll
    for (int c = 0; c < 6; ++c) s[c] = src[c];
  if (v) {
    if (sub < 2) {
      v[0] = pa;
    } else {
      v[0] = g.ev[2 * pa];
      v[1] = g.ev[2 * pa + 1];
    }
  }
}
__device__ __forceinline__ void stage_b(const Geo& g, int sub, const SubLists& L, int k, float* s, int* v) {
  const int pb = L.offB + L.LB[k];
  const float* src = L.boxB + 6 * pb;
#pragma unroll
  for (int c = 0; c < 6; ++c) s[c] = src[c];
  if (v) {
    if (sub < 2) {
      v[0] = g.fv[3 * pb];
      v[1] = g.fv[3 * pb + 1];
      v[2] = g.fv[3 * pb + 2];
    } else {
      v[0] = g.ev[2 * pb];
      v[1] = g.ev[2 * pb + 1];
    }
  }
}

__device__ __forceinline__ bool f_hit(const float* a, const float* b) {
  return a[0] <= b[3] && a[3] >= b[0] && a[1] <= b[4] && a[4] >= b[1] && a[2] <= b[5] && a[5] >= b[2];
}

// Order in which the narrow-phase CTAs take the overlaps: the heaviest sub-problem sets
// first (after refinement a pile's work sits in ~1700 of ~10000 overlaps, from 1k to 56k
// candidate pairs each), so the long ones do not start in the last wave. The outputs of
// an overlap do not depend on when it is processed.
constexpr int NBUCKET = 4;
__device__ __forceinline__ int work_bucket(const int* n) {
  long long c = (long long)n[0] * n[5] + (long long)n[3] * n[2] + (long long)n[1] * n[4];
  return c >= 16384 ? 0 : (c >= 2048 ? 1 : (c > 0 ? 2 : 3));
}
// Bucket b's overlaps at order[b * nov ...], bc[b] of them.
__global__ void k_order(int nov, const int* cnt, int* bc, int* order) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int b = u < nov ? work_bucket(cnt + 6 * u) : NBUCKET - 1;
#pragma unroll
  for (int k = 0; k < NBUCKET - 1; ++k) {  // the empty ones are not taken
    const unsigned m = __ballot_sync(0xffffffffu, b == k);
    if (!m) continue;
    int base = 0;
    if (lane == 0) base = atomicAdd(&bc[k], __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (b == k) order[k * (size_t)nov + base + __popc(m & ((1u << lane) - 1u))] = u;
  }
}
// The overlap of place i of the order, -1 past the last.
struct Order {
  const int *at, *bc;
  int nov;
  __device__ __forceinline__ int operator[](int i) const {
    for (int k = 0; k < NBUCKET - 1; ++k) {
      const int n = bc[k];
      if (i < n) return at[k * (size_t)nov + i];
      i -= n;
    }
    return -1;
  }
};

// The FP64 test of one candidate into its scene's key.
__device__ __noinline__ void toi_one(const Geo& g, int sub, int pa, int pb, unsigned long long* toi_key) {
  const double t = exact_toi(g, sub, pa, pb);
  if (t < 1.0) atomicMin(toi_key + 2 * g.bscene[g.vbody[sub < 2 ? pa : g.ev[2 * pa]]], dkey(t));
}
__global__ void __launch_bounds__(128) k_toi_list(Geo g, ToiCand tc, unsigned long long* toi_key) {
  const unsigned n = min(*tc.n, tc.cap);
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int2 c = tc.cand[t];
    if (c.x >= 0) toi_one(g, 0, c.x, c.y, toi_key);
    else toi_one(g, 2, ~c.x, c.y, toi_key);
  }
}

// 5a. Narrow phase, one CTA per overlap: pair cull (MODE 0) or trajectory (MODE 2).
// For each sub-problem (v(I) x f(J), v(J) x f(I), e(I) x e(J)) the float boxes of both
// lists are staged in shared memory, all three together while they fit. The work alternates
// between two phases so that the tests are spread evenly over the CTA:
//  - box phase: each thread keeps one A box in registers and walks its B boxes (a
//    shared-memory broadcast per step), STEP candidates per thread, and appends the
//    float-box hits to a shared queue (warp-aggregated);
//  - test phase: the whole CTA takes the queued candidates round-robin for the FP32 tests:
//    lower bounds of the distance (MODE 0, f_reject), certificates that there is no time of
//    impact (MODE 2, abd_ccd_filter.cuh).
// No FP64 runs here. The candidates left go to lists that k_narrow_exact and k_toi_list
// evaluate, a thread each: an FP64 test is a chain of some 300 (distance) or 900 (time of
// impact) instructions of 64 cycles a warp, which a CTA with a handful of candidates used to
// pay for each sub-problem and box phase. MODE 0 keeps an overlap's candidates in shared
// memory and writes them sorted, so that the accepted ones come out in order. One cull of a
// batch of columns (7291 overlaps, 11 candidates each) 893 -> 238 us, of the pile (9871, 19
// each) 583 -> 300 us, the FP64 kernel included.
template <int MODE, int STEP>
__global__ void __launch_bounds__(NT, MODE == 0 ? (STEP <= 8 ? 4 : STEP <= 16 ? 3 : 2) : (STEP <= 36 ? 4 : 2))
    k_narrow_scan(Geo g, Params P, float ds_f, const int* ovI, const int* ovJ, int* cnt, const int* off, int* lst,
                  const float* vb, const float* eb, const float* fb, unsigned long long* toi_key, StageOut so,
                  Order order, ToiCand tc) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  unsigned long long* recK = reinterpret_cast<unsigned long long*>(smem_dyn);  // REC_CAP (MODE 0)
  float* sA = reinterpret_cast<float*>(smem_dyn + (MODE == 0 ? REC_CAP * sizeof(unsigned long long) : 0));
  float* sB = sA + TILE * 6;
  unsigned int* sq = reinterpret_cast<unsigned int*>(sB + TILE * 6);
  int* sVA = MODE == 0 ? reinterpret_cast<int*>(sq + NT * STEP) : nullptr;  // 2 * TILE (MODE 0)
  int* sVB = MODE == 0 ? sVA + 2 * TILE : nullptr;                          // 3 * TILE (MODE 0)
  __shared__ int sq_n[2];
  __shared__ int rec_n, rec_np, rec_base[2];
  __shared__ SubLists sL[3];
  const int u = order[blockIdx.x];
  if (u < 0) return;  // no candidates: k_narrow_tally sees that from the lists
  const float lim_f = __double2float_ru(P.dhat * (1.0 + 1e-4));
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  if (threadIdx.x < 3) {
    SubLists L = sub_lists(g, threadIdx.x, ovI[u], ovJ[u], cnt + 6 * u, off + 6 * u, lst, vb, eb, fb);  // refined
    if (L.nA == 0 || L.nB == 0) L.nA = L.nB = 0;
    sL[threadIdx.x] = L;
  }
  if (threadIdx.x == 0) {
    rec_n = rec_np = 0;
    sq_n[0] = 0;
    sq_n[1] = 0;
  }
  __syncthreads();
  // Box phase over rows of one staged chunk: thread t has the rows i = t mod ca (ca < NT) or
  // t, t + NT, ... (ca >= NT) and the columns j = ph, ph + phases, ... with phases = NT / ca
  // threads sharing a row.
  struct Walk {
    int ca, cb, rows, phases, ph, row0, ncol, nrow, max_items, ri, cj;
  };
  auto walk_of = [&](int ca, int cb) {
    Walk w;
    w.ca = ca;
    w.cb = cb;
    w.rows = ca < NT ? ca : NT;
    w.phases = ca < NT ? NT / ca : 1;
    w.ph = ca < NT ? threadIdx.x / ca : 0;
    w.row0 = threadIdx.x % w.rows;
    w.ncol = w.ph < w.phases ? (cb - w.ph + w.phases - 1) / w.phases : 0;
    w.nrow = w.ncol > 0 ? (ca - w.row0 + w.rows - 1) / w.rows : 0;
    w.max_items = (ca < NT ? 1 : (ca + NT - 1) / NT) * ((cb + w.phases - 1) / w.phases);
    w.ri = w.cj = 0;
    return w;
  };
  // its candidates: the hits to the queue (qa, qb: the chunk's first A and B entry in it)
  auto boxes = [&](Walk& w, int items, const float* A, const float* B, float (&a)[6], int par, unsigned tag) {
#pragma unroll 1
    for (int it = 0; it < items; ++it) {
      bool hit = false;
      unsigned code = 0;
      if (w.ri < w.nrow) {
        const int i = w.row0 + w.ri * w.rows, j = w.ph + w.cj * w.phases;
        hit = i < w.ca && j < w.cb && f_hit(a, B + 6 * j);
        code = tag + (((unsigned)i << 15) | (unsigned)j);
        if (++w.cj == w.ncol) {
          w.cj = 0;
          if (++w.ri < w.nrow)
#pragma unroll
            for (int c = 0; c < 6; ++c) a[c] = A[6 * (w.row0 + w.ri * w.rows) + c];
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (m) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&sq_n[par], __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        const int pos = base + __popc(m & below);
        if (hit && pos < NT * STEP) sq[pos] = code;
      }
    }
  };
  // test of a candidate: A entry i and B entry j of the lists, staged at (si, sj)
  auto test = [&](int sub, const SubLists& L, int i, int j, int si, int sj) {
    if (MODE == 2) {
      const int pa = L.offA + L.LA[i], pb = L.offB + L.LB[j];
      if (f_toi_miss(g, tc.ve, sub, pa, pb)) return;
      const unsigned o = atomicAdd(tc.n, 1u);
      if (o < tc.cap) tc.cand[o] = make_int2(sub < 2 ? pa : ~pa, pb);
      else toi_one(g, sub, pa, pb, toi_key);
    } else {
      const int w0 = sVA[2 * si];
      const int w1 = sub < 2 ? sVB[3 * sj] : sVA[2 * si + 1];
      const int w2 = sub < 2 ? sVB[3 * sj + 1] : sVB[3 * sj];
      const int w3 = sub < 2 ? sVB[3 * sj + 2] : sVB[3 * sj + 1];
      if (f_reject_v(vb, sub, w0, w1, w2, w3, lim_f)) return;
      const int slot = atomicAdd(&rec_n, 1);
      if (slot < REC_CAP)
        recK[slot] = ((unsigned long long)sub << 60) | ((unsigned long long)i << 30) | (unsigned long long)j;
    }
  };
  const int a1 = sL[0].nA, a2 = a1 + sL[1].nA, a3 = a2 + sL[2].nA;
  const int b1 = sL[0].nB, b2 = b1 + sL[1].nB, b3 = b2 + sL[2].nB;
  // Short lists: the three sub-problems are staged together and share one box and one test
  // phase, so the CTA waits once for the lists, the boxes and the vertices instead of three
  // times. On the pile's trajectories 235 -> 151 us, on columns 207 -> 172 us (pair cull) and 132 -> 82 us.
  bool general = a3 > TILE || b3 > TILE;
  if (!general && a3 > 0) {
    for (int k = threadIdx.x; k < a3; k += NT) {
      const int sub = (k >= a1) + (k >= a2);
      stage_a(g, sub, sL[sub], k - (sub == 0 ? 0 : (sub == 1 ? a1 : a2)), MODE != 2, ds_f, sA + 6 * k,
              MODE == 0 ? sVA + 2 * k : nullptr);
    }
    for (int k = threadIdx.x; k < b3; k += NT) {
      const int sub = (k >= b1) + (k >= b2);
      stage_b(g, sub, sL[sub], k - (sub == 0 ? 0 : (sub == 1 ? b1 : b2)), sB + 6 * k,
              MODE == 0 ? sVB + 3 * k : nullptr);
    }
    __syncthreads();
#pragma unroll 1
    for (int sub = 0; sub < 3; ++sub) {
      const int ca = sL[sub].nA, cb = sL[sub].nB;
      if (ca == 0) continue;
      const int qa = sub == 0 ? 0 : (sub == 1 ? a1 : a2), qb = sub == 0 ? 0 : (sub == 1 ? b1 : b2);
      Walk w = walk_of(ca, cb);
      float a[6];
      if (w.nrow > 0)
#pragma unroll
        for (int c = 0; c < 6; ++c) a[c] = sA[6 * (qa + w.row0) + c];
      boxes(w, w.max_items, sA + 6 * qa, sB + 6 * qb, a, 0,
            ((unsigned)sub << 30) + ((unsigned)qa << 15) + (unsigned)qb);
    }
    __syncthreads();
    const int nq = sq_n[0];
    general = nq > NT * STEP;  // more hits than the queue holds
    if (!general) {
#pragma unroll 1
      for (int k = threadIdx.x; k < nq; k += NT) {
        const unsigned code = sq[k];
        const int sub = (int)(code >> 30), si = (int)(code >> 15 & 0x7fffu), sj = (int)(code & 0x7fffu);
        test(sub, sL[sub], si - (sub == 0 ? 0 : (sub == 1 ? a1 : a2)), sj - (sub == 0 ? 0 : (sub == 1 ? b1 : b2)), si,
             sj);
      }
    } else {
      __syncthreads();
      if (threadIdx.x == 0) sq_n[0] = 0;
    }
  }
  if (general) {
    int par = 0;
#pragma unroll 1
    for (int sub = 0; sub < 3; ++sub) {
      const SubLists L = sL[sub];
#pragma unroll 1
      for (int a0 = 0; a0 < L.nA; a0 += TILE) {
        const int ca = min(TILE, L.nA - a0);
#pragma unroll 1
        for (int b0 = 0; b0 < L.nB; b0 += TILE) {
          const int cb = min(TILE, L.nB - b0);
          __syncthreads();
          for (int k = threadIdx.x; k < ca; k += NT)
            stage_a(g, sub, L, a0 + k, MODE != 2, ds_f, sA + 6 * k, MODE == 0 ? sVA + 2 * k : nullptr);
          for (int k = threadIdx.x; k < cb; k += NT)
            stage_b(g, sub, L, b0 + k, sB + 6 * k, MODE == 0 ? sVB + 3 * k : nullptr);
          __syncthreads();
          Walk w = walk_of(ca, cb);
          float a[6];
          if (w.nrow > 0)
#pragma unroll
            for (int c = 0; c < 6; ++c) a[c] = sA[6 * w.row0 + c];
#pragma unroll 1
          for (int st = 0; st < w.max_items; st += STEP) {
            boxes(w, min(STEP, w.max_items - st), sA, sB, a, par, 0u);
            __syncthreads();
            const int nq = sq_n[par];
            if (threadIdx.x == 0) sq_n[par ^ 1] = 0;
#pragma unroll 1
            for (int k = threadIdx.x; k < nq; k += NT) {
              const unsigned code = sq[k];
              const int i = (int)(code >> 15), j = (int)(code & 0x7fffu);
              test(sub, L, a0 + i, b0 + j, i, j);
            }
            par ^= 1;
            __syncthreads();
          }
        }
      }
    }
  }
  if (MODE == 0) {
    // Sort the (sub, i, j) keys and stage them: up to NT by rank (keys differ; each thread
    // counts the keys below its own), more by a bitonic sort in shared memory. Overlaps with more
    // candidates than REC_CAP are marked and go through passes that recompute their tests.
    __syncthreads();
    const int nr = rec_n;
    if (nr > REC_CAP || nr == 0) {
      if (threadIdx.x == 0) so.seg[u] = make_int4(nr == 0 ? 0 : -1, 0, 0, 0);
      return;
    }
    unsigned long long key = threadIdx.x < nr ? recK[threadIdx.x] : ~0ull;
    int c = 0;
    for (int k = threadIdx.x; k < nr; k += NT) c += (int)(recK[k] >> 60) < 2;
    if (c) atomicAdd(&rec_np, c);
    if (nr <= NT) {
      int r = 0;
      if (threadIdx.x < nr)
        for (int k = 0; k < nr; ++k) r += recK[k] < key;
      __syncthreads();
      if (threadIdx.x < nr) recK[r] = key;
    } else {
      int np2 = NT;
      while (np2 < nr) np2 <<= 1;
      for (int k = nr + threadIdx.x; k < np2; k += NT) recK[k] = ~0ull;
      __syncthreads();
      for (int size = 2; size <= np2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          for (int t = threadIdx.x; t < (np2 >> 1); t += NT) {
            int lo = 2 * t - (t & (stride - 1));
            int hi = lo + stride;
            bool up = ((lo & size) == 0);
            unsigned long long a = recK[lo], b = recK[hi];
            if ((a > b) == up) {
              recK[lo] = b;
              recK[hi] = a;
            }
          }
          __syncthreads();
        }
    }
    __syncthreads();
    const int np = rec_np, ne = nr - np;
    if (threadIdx.x == 0) {
      const int bp = np ? atomicAdd(so.total, np) : 0, be = ne ? atomicAdd(so.total + 1, ne) : 0;
      const bool ok = bp <= so.cap - np && be <= so.cap - ne;
      rec_base[0] = ok ? bp : -1;
      rec_base[1] = so.cap - be - ne;
      so.seg[u] = make_int4(rec_base[0], np, rec_base[1], ne);
    }
    __syncthreads();
    if (rec_base[0] >= 0)
      for (int k = threadIdx.x; k < nr; k += NT) {
        const int p = k < np ? rec_base[0] + k : rec_base[1] + (k - np);
        so.key[p] = recK[k];
        so.ov[p] = u;
      }
  }
}

// 5a'. The FP64 test of every staged candidate, a thread each: its distance type, or -1. Bound by
// FP64 issue (189 k candidates of the pile, of which 181 k are pairs: 90 us; 185 us while warps
// held both kinds and ran both tests).
__global__ void __launch_bounds__(128) k_narrow_exact(Geo g, Params P, const int* ovI, const int* ovJ, const int* cnt,
                                                      const int* off, const int* lst, StageOut so) {
  if (!so.valid()) return;
  const int np = so.total[0], ne = so.total[1], np32 = (np + 31) & ~31;  // whole warps of one kind
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np32 + ne; k += gridDim.x * blockDim.x) {
    if (k >= np && k < np32) continue;
    const int t = k < np ? k : so.cap - ne + (k - np32);
    const unsigned long long key = so.key[t];
    const int u = so.ov[t], sub = (int)(key >> 60), i = (int)((key >> 30) & 0x3fffffffull), j = (int)(key & 0x3fffffffull);
    const SubLists L = sub_lists(g, sub, ovI[u], ovJ[u], cnt + 6 * u, off + 6 * u, lst, nullptr, nullptr, nullptr);
    so.ty[t] = (int8_t)(exact_pair(g, P, sub, L.offA + L.LA[i], L.offB + L.LB[j]) - 1);
  }
}

// Ordered count and write of an overlap whose candidates did not fit the shared-memory sort:
// the (i, j) space of each sub-problem is walked in row-major order (the order of the
// reference's nested loops), a CTA's threads at a time; f(sub, hit, i, j, type, L) is called by
// all threads for each step of the walk.
template <typename F>
__device__ __forceinline__ void narrow_walk(const Geo& g, const Params& P, float ds_f, int I, int J, const int* n,
                                            const int* o, const int* lst, const float* vb, const float* eb,
                                            const float* fb, F&& f) {
#pragma unroll 1
  for (int sub = 0; sub < 3; ++sub) {
    SubLists L = sub_lists(g, sub, I, J, n, o, lst, vb, eb, fb);
    const long long tot = (long long)L.nA * L.nB;
#pragma unroll 1
    for (long long k0 = 0; k0 < tot; k0 += blockDim.x) {
      const long long k = k0 + threadIdx.x;
      int ty = 0, i = 0, j = 0;
      if (k < tot) {
        i = (int)(k / L.nB);
        j = (int)(k - (long long)i * L.nB);
        float a[6];
        finflate(L.boxA + 6 * (L.offA + L.LA[i]), ds_f, a);
        if (f_hit(a, L.boxB + 6 * (L.offB + L.LB[j])))
          ty = exact_pair(g, P, sub, L.offA + L.LA[i], L.offB + L.LB[j]);
      }
      f(sub, ty != 0, i, j, ty - 1, L);
    }
  }
}

// 5b. Accepted pairs of every overlap: point-triangle and edge-edge.
constexpr int NW = 128;  // threads of the tally and of the ordered writes
__global__ void __launch_bounds__(NW) k_narrow_tally(Geo g, Params P, float ds_f, const int* ovI, const int* ovJ,
                                                     const int* cnt, const int* off, const int* lst, const float* vb,
                                                     const float* eb, const float* fb, StageOut so, int* npt, int* nee) {
  __shared__ int s_pt, s_ee;
  const int u = blockIdx.x;
  const int4 sg = so.seg[u];  // not written where no list pair is left
  const bool none = work_bucket(cnt + 6 * u) == NBUCKET - 1 || (sg.x >= 0 && sg.y + sg.w == 0);
  if (none || !so.valid()) {
    if (threadIdx.x == 0) {
      npt[u] = nee[u] = 0;
      if (none) so.seg[u] = make_int4(0, 0, 0, 0);
    }
    return;
  }
  if (threadIdx.x == 0) s_pt = s_ee = 0;
  __syncthreads();
  int c[2] = {0, 0};
  if (sg.x >= 0) {
    for (int k = threadIdx.x; k < sg.y; k += NW) c[0] += so.ty[sg.x + k] >= 0;
    for (int k = threadIdx.x; k < sg.w; k += NW) c[1] += so.ty[sg.z + k] >= 0;
  } else {
    narrow_walk(g, P, ds_f, ovI[u], ovJ[u], cnt + 6 * u, off + 6 * u, lst, vb, eb, fb,
                [&](int sub, bool hit, int, int, int, const SubLists&) { (sub < 2 ? c[0] : c[1]) += hit; });
  }
#pragma unroll
  for (int q = 16; q > 0; q >>= 1) {
    c[0] += __shfl_xor_sync(0xffffffffu, c[0], q);
    c[1] += __shfl_xor_sync(0xffffffffu, c[1], q);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&s_pt, c[0]);
    atomicAdd(&s_ee, c[1]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    npt[u] = s_pt;
    nee[u] = s_ee;
  }
}

// 5c. Ordered write: the accepted candidates of each overlap in the order of their keys
// (point-triangle ones first), or those of the walk.
__global__ void __launch_bounds__(NW) k_narrow_write(Geo g, Params P, float ds_f, const int* ovI, const int* ovJ,
                                                     const int* cnt, const int* off, const int* lst, const float* vb,
                                                     const float* eb, const float* fb, StageOut so, const int* npt,
                                                     const int* ov_pt_off, const int* ov_ee_off, NarrowOut out) {
  __shared__ int wcnt[2][NW / 32];
  const int u = blockIdx.x;
  const int4 sg = so.seg[u];
  const int nr = sg.y + sg.w;
  if (sg.x >= 0 && nr == 0) return;
  const int I = ovI[u], J = ovJ[u];
  const int* n = cnt + 6 * u;
  const int* o = off + 6 * u;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int pt0 = ov_pt_off[u], ee0 = ov_ee_off[u], np = npt[u];
  int done = 0, par = 0;  // accepted pairs written (both kinds)
  auto put = [&](int sub, bool hit, int i, int j, int ty, const SubLists& L) {
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) wcnt[par][w] = __popc(m);
    __syncthreads();
    int r = done + __popc(m & below), total = 0;
#pragma unroll
    for (int q = 0; q < NW / 32; ++q) {
      r += (q < w) ? wcnt[par][q] : 0;
      total += wcnt[par][q];
    }
    if (hit) {
      const int idx = sub < 2 ? pt0 + r : ee0 + (r - np);
      int* dst = sub < 2 ? out.pt : out.ee;
      dst[4 * idx] = L.A; dst[4 * idx + 1] = L.LA[i]; dst[4 * idx + 2] = L.B; dst[4 * idx + 3] = L.LB[j];
      (sub < 2 ? out.pt_ty : out.ee_ty)[idx] = (int8_t)ty;
      (sub < 2 ? out.pt_ov : out.ee_ov)[idx] = u;
    }
    done += total;
    par ^= 1;  // the counts of the step before are read while these are written
  };
  if (sg.x < 0) {
    narrow_walk(g, P, ds_f, I, J, n, o, lst, vb, eb, fb, put);
    return;
  }
  for (int k0 = 0; k0 < nr; k0 += NW) {
    const int k = k0 + threadIdx.x;
    const int p = k < sg.y ? sg.x + k : sg.z + (k - sg.y);
    const unsigned long long key = k < nr ? so.key[p] : 0;
    const int ty = k < nr ? so.ty[p] : -1;
    const int sub = (int)(key >> 60);
    const SubLists L = sub_lists(g, sub, I, J, n, o, lst, vb, eb, fb);
    put(sub, ty >= 0, (int)((key >> 30) & 0x3fffffffull), (int)(key & 0x3fffffffull), ty, L);
  }
}

// 6a. vertex-ground pairs: flags + per-CTA counts, then ordered write
__global__ void k_vg_count(Geo g, Params P, int* blk_cnt) {
  __shared__ int sh[32];
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  bool hit = false;
  if (v < g.nv && scene_on(g, g.vbody[v])) {
    double d = XA(g.X[g.nv + v], P.ground_offset);
    d = XM(d, d);
    hit = d < P.dhat;
  }
  unsigned m = __ballot_sync(0xffffffffu, hit);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = __popc(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += sh[i];
    blk_cnt[blockIdx.x] = s;
  }
}
__global__ void k_vg_write(Geo g, Params P, const int* blk_off, int* vg) {
  __shared__ int sh[32];
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  bool hit = false;
  if (v < g.nv && scene_on(g, g.vbody[v])) {
    double d = XA(g.X[g.nv + v], P.ground_offset);
    d = XM(d, d);
    hit = d < P.dhat;
  }
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned m = __ballot_sync(0xffffffffu, hit);
  if (lane == 0) sh[w] = __popc(m);
  __syncthreads();
  int pre = 0;
  for (int i = 0; i < w; ++i) pre += sh[i];
  if (hit) {
    int idx = blk_off[blockIdx.x] + pre + __popc(m & ((1u << lane) - 1u));
    int b = g.vbody[v];
    vg[2 * idx] = b;
    vg[2 * idx + 1] = v - g.v_off[b];
  }
}
// VG segment per body: first VG pair of body b (pairs are in vertex order)
__global__ void k_vg_seg(int nb, int nvg, const int* vg, int* seg) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > nb) return;
  int lo = 0, hi = nvg;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (vg[2 * mid] < b) lo = mid + 1;
    else hi = mid;
  }
  seg[b] = lo;
}

// 6b. ground time of impact (collision.cpp:83-105); toi_key points at the ground slot
// of scene 0 (slots alternate pt/ee, ground per scene).
__global__ void k_vg_toi(Geo g, Params P, unsigned long long* toi_key) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= g.nv || !scene_on(g, g.vbody[v])) return;
  double d2 = XA(g.X[g.nv + v], P.ground_offset);
  if (d2 < 0) {
    double d1 = XA(g.Xq[g.nv + v], P.ground_offset);
    double t = XD(d1, XS(d1, d2));
    if (t < 1.0) atomicMin(toi_key + 2 * g.bscene[g.vbody[v]], dkey(t));
  }
}

__global__ void k_fill_u64(unsigned long long* p, int n, unsigned long long v) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

// Smallest float >= d (host side).
// Lets the narrow-phase CTAs use more than the default 48 kB of shared memory (once per
// device; the setting is part of this process's context only).
static void narrow_smem_attr() {
  static int done_dev = -1;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (done_dev == dev) return;
#define ABD_NARROW_ATTR(M, ST) \
  CK(cudaFuncSetAttribute(k_narrow_scan<M, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)narrow_smem(M, ST)))
  ABD_NARROW_ATTR(0, 8);
  ABD_NARROW_ATTR(0, 16);
  ABD_NARROW_ATTR(0, 48);
  ABD_NARROW_ATTR(2, 24);
  ABD_NARROW_ATTR(2, 36);
  ABD_NARROW_ATTR(2, 64);
#undef ABD_NARROW_ATTR
  done_dev = dev;
}

// Arguments of one narrow-phase launch.
struct NarrowLaunch {
  Geo g;
  Params P;
  float ds_f;
  const int *ovI, *ovJ;
  int* cnt;
  const int* off;
  int* lst;
  const float *vb, *eb, *fb;
  unsigned long long* toi_key;
  StageOut so;
  Order order;
  ToiCand tc;
};

// k_narrow_scan<mode, kNarrowStep[mode][variant]> over nov overlaps
static void launch_narrow(int mode, int variant, int nov, const NarrowLaunch& a, cudaStream_t s) {
  const int tag = mode == 2 ? K_NARROW_TOI : K_NARROW_SCAN;
#define ABD_NARROW_LAUNCH(M, ST)                                                                                   \
  KLAUNCH(tag, s, k_narrow_scan<M, ST><<<nov, NT, narrow_smem(M, ST), s>>>(                                       \
                      a.g, a.P, a.ds_f, a.ovI, a.ovJ, a.cnt, a.off, a.lst, a.vb, a.eb, a.fb, a.toi_key, a.so,      \
                      a.order, a.tc))
  const int st = kNarrowStep[mode == 2 ? 1 : 0][variant];
  if (mode == 2) {
    if (st == 24) ABD_NARROW_LAUNCH(2, 24);
    else if (st == 36) ABD_NARROW_LAUNCH(2, 36);
    else ABD_NARROW_LAUNCH(2, 64);
  } else {
    if (st == 8) ABD_NARROW_LAUNCH(0, 8);
    else if (st == 16) ABD_NARROW_LAUNCH(0, 16);
    else ABD_NARROW_LAUNCH(0, 48);
  }
#undef ABD_NARROW_LAUNCH
}

// The narrow phase of `mode` (0: pair cull, 1 in the tables: CCD) with the handle's
// chosen variant. The first launch with at least kTuneMinOverlaps overlaps runs every
// variant on the same input, timed with CUDA events, keeps the fastest for the life of
// the handle and leaves the outputs of the last run (all variants give the same outputs;
// `reset`, when given, clears the pair cull's staging counters before each run).
constexpr int kTuneMinOverlaps = 64;
static void narrow_phase(int mode, int nov, const NarrowLaunch& a, CullScratch& cs, int* reset, cudaStream_t s) {
  const int m = mode == 2 ? 1 : 0;
  if (cs.narrow_variant[m] >= 0 || !cs.autotune || nov < kTuneMinOverlaps) {
    CK(cudaMemsetAsync(reset, 0, 2 * sizeof(int), s));
    launch_narrow(mode, cs.narrow_variant[m] >= 0 ? cs.narrow_variant[m] : kNarrowDefault, nov, a, s);
    return;
  }
  cudaEvent_t ev[kNarrowVariants + 1];
  for (auto& e : ev) CK(cudaEventCreate(&e));
  CK(cudaEventRecord(ev[0], s));
  for (int v = 0; v < kNarrowVariants; ++v) {
    CK(cudaMemsetAsync(reset, 0, 2 * sizeof(int), s));
    launch_narrow(mode, v, nov, a, s);
    CK(cudaEventRecord(ev[v + 1], s));
  }
  CK(cudaEventSynchronize(ev[kNarrowVariants]));
  int best = kNarrowDefault;
  for (int v = 0; v < kNarrowVariants; ++v) {
    float t = 0;
    CK(cudaEventElapsedTime(&t, ev[v], ev[v + 1]));
    cs.narrow_ms[m][v] = t;
    if (t < cs.narrow_ms[m][best]) best = v;
  }
  // the default keeps ties and near-ties (within 3%)
  if (!(cs.narrow_ms[m][best] < 0.97f * cs.narrow_ms[m][kNarrowDefault])) best = kNarrowDefault;
  cs.narrow_variant[m] = best;
  for (auto& e : ev) CK(cudaEventDestroy(e));
}


// Fills cs.order with the overlaps that have work, heaviest bucket first.
static void order_overlaps(int nov, CullScratch& cs, cudaStream_t s, int tag) {
  cs.order.ensure((NBUCKET - 1) * (size_t)nov + 1);
  cs.order_cnt.ensure(NBUCKET);
  CK(cudaMemsetAsync(cs.order_cnt.p, 0, NBUCKET * sizeof(int), s));
  KLAUNCH(tag, s, k_order<<<nblk(nov, 256), 256, 0, s>>>(nov, cs.bin_cnt.p, cs.order_cnt.p, cs.order.p));
}

float float_round_up(double d) {
  float f = (float)d;
  if ((double)f < d) f = nextafterf(f, INFINITY);
  return f;
}

double key_to_double(unsigned long long k) {
  unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  double d;
  memcpy(&d, &b, sizeof(d));
  return d;
}

// launch_project, with the vertices' float boxes (and their clusters') when vb (and cl) are given
static void project_boxes(const Geo& g, int which, double alpha, float* vb, float* cl, cudaStream_t s) {
  if (which == 2 && g.nb > 0) KLAUNCH(K_PROJECT, s, k_trial_state<<<nblk(12ll * g.nb, 256), 256, 0, s>>>(g, alpha));
  if (g.nv == 0) return;
  KLAUNCH(K_PROJECT, s, k_project<<<nblk(g.nv, 256), 256, 0, s>>>(g, which, vb, cl));
  prof_work(K_PROJECT, g.nv, 48.0 * g.nv);  // rest read + world write per vertex
}

}  // namespace

int narrow_step_of(int mode, int variant) { return kNarrowStep[mode == 2 ? 1 : 0][variant]; }

void launch_project(const Geo& g, int which, double alpha, cudaStream_t s) {
  project_boxes(g, which, alpha, nullptr, nullptr, s);
}

static BinClusters bin_clusters(const Geo& g, CullScratch& cs) {
  const size_t nv = (g.nv + 31) / 32, ne = (g.ne + 31) / 32, nf = (g.nf + 31) / 32;
  cs.cbox.ensure(6 * (nv + ne + nf + g.nb) + 6);
  return {cs.cbox.p, cs.cbox.p + 6 * nv, cs.cbox.p + 6 * (nv + ne), cs.cbox.p + 6 * (nv + ne + nf)};
}

// Float boxes of the edges and faces from those of the vertices (in cs.vbox), and of their clusters
// when the lists are binned from them.
static void edge_face_boxes(const Geo& g, bool clusters, CullScratch& cs, cudaStream_t s) {
  BinClusters cl{};
  if (clusters) cl = bin_clusters(g, cs);
  cs.ebox.ensure(6 * (size_t)g.ne + 6);
  cs.fbox.ensure(6 * (size_t)g.nf + 6);
  if (g.ne + g.nf > 0) {
    KLAUNCH(K_PRIM_BOXES, s, k_prim_boxes<<<nblk((long long)g.ne + g.nf + 31, 256), 256, 0, s>>>(
                                 g, cs.vbox.p, cs.ebox.p, cs.fbox.p, cl));
  }
}

void prim_boxes(const Geo& g, CullScratch& cs, cudaStream_t s) {
  cs.vbox.ensure(6 * (size_t)g.nv + 6);
  if (g.nv > 0) KLAUNCH(K_PRIM_BOXES, s, k_vert_boxes<<<nblk(g.nv, 256), 256, 0, s>>>(g, cs.vbox.p));
  edge_face_boxes(g, false, cs, s);
}

void traj_floats(const Geo& g, CullScratch& cs, cudaStream_t s) {
  cs.vend.ensure(6 * (size_t)g.nv + 6);
  if (g.nv > 0) KLAUNCH(K_PRIM_BOXES, s, k_traj_floats<<<nblk(g.nv, 256), 256, 0, s>>>(g, cs.vend.p));
}

// Narrow phase of a pair cull over binned (and refined, ordered) lists of nov overlaps:
// candidates (grown and repeated when the staging overflows), their FP64 tests, per-overlap
// counts and offsets, one host read of the totals (pt, ee, vg, staged of both kinds),
// then the ordered write of the pairs into S.
static void narrow_pairs(const Geo& g, const Params& P, float ds_f, int nov, const int* ovI, const int* ovJ,
                         CullScratch& cs, PairSet& S, int& npt, int& nee, cudaStream_t s) {
  int* d_tot = cs.tmp_int.p;
  cs.blk_a.ensure(nov + 1);
  cs.blk_b.ensure(nov + 1);
  cs.blk_a_off.ensure(nov + 1);
  cs.blk_b_off.ensure(nov + 1);
  cs.stage_seg.ensure(nov + 1);
  // room for 32 candidates an overlap (piles and columns of spheres: 11 to 19), 64 k at least,
  // 256 M entries at most before the count is known
  size_t want = std::max({cs.stage_key.cap, (size_t)1 << 16, std::min((size_t)32 * nov, (size_t)1 << 28)});
  StageOut so{};
  for (int attempt = 0; attempt < 4; ++attempt) {
    cs.stage_key.ensure(want);
    cs.stage_ty.ensure(cs.stage_key.cap);
    cs.stage_ov.ensure(cs.stage_key.cap);
    so = StageOut{cs.stage_key.p, cs.stage_ov.p, cs.stage_ty.p, cs.stage_seg.p, d_tot + 6, (int)cs.stage_key.cap};
    narrow_smem_attr();
    NarrowLaunch a{g, P, ds_f, ovI, ovJ, cs.bin_cnt.p, cs.bin_off.p, cs.lst.p, cs.vbox.p, cs.ebox.p, cs.fbox.p,
                   nullptr, so, Order{cs.order.p, cs.order_cnt.p, nov}, ToiCand{}};
    narrow_phase(0, nov, a, cs, d_tot + 6, s);
    KLAUNCH(K_NARROW_SCAN, s, k_narrow_exact<<<1216, 128, 0, s>>>(g, P, ovI, ovJ, cs.bin_cnt.p, cs.bin_off.p,
                                                                  cs.lst.p, so));
    // per-overlap pair counts and their offsets, read together with the staged total
    KLAUNCH(K_NARROW_WRITE, s, k_narrow_tally<<<nov, NW, 0, s>>>(g, P, ds_f, ovI, ovJ, cs.bin_cnt.p, cs.bin_off.p,
                                                                 cs.lst.p, cs.vbox.p, cs.ebox.p, cs.fbox.p, so,
                                                                 cs.blk_a.p, cs.blk_b.p));
    scan_exclusive_int2(cs.blk_a.p, cs.blk_a_off.p, d_tot + 3, cs.blk_b.p, cs.blk_b_off.p, d_tot + 4, nov, s,
                        cs.vflag_cnt);
    CK(cudaMemcpyAsync(cs.h_small + 3, d_tot + 3, 5 * sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const size_t staged = (size_t)cs.h_small[6] + cs.h_small[7];
    if (staged <= cs.stage_key.cap) break;
    // staging overflowed: grow to the reported total and repeat
    want = staged + (staged >> 2) + 1024;
  }
  npt = cs.h_small[3];
  nee = cs.h_small[4];
  prof_work(K_NARROW_SCAN, nov, 24.0 * g.nv + 20.0 * ((double)npt + nee));
  S.pt.ensure(4 * (size_t)npt + 4);
  S.pt_ty.ensure(npt + 1);
  S.pt_ov.ensure(npt + 1);
  S.ee.ensure(4 * (size_t)nee + 4);
  S.ee_ty.ensure(nee + 1);
  S.ee_ov.ensure(nee + 1);
  NarrowOut no{S.pt.p, S.pt_ov.p, S.ee.p, S.ee_ov.p, S.pt_ty.p, S.ee_ty.p};
  if (npt + nee > 0)
    KLAUNCH(K_NARROW_WRITE, s, k_narrow_write<<<nov, NW, 0, s>>>(g, P, ds_f, ovI, ovJ, cs.bin_cnt.p, cs.bin_off.p,
                                                                 cs.lst.p, cs.vbox.p, cs.ebox.p, cs.fbox.p, so,
                                                                 cs.blk_a.p, cs.blk_a_off.p, cs.blk_b_off.p, no));
}

void cull(const Geo& g_in, const Params& P, int vtn, double alpha, CullScratch& cs, PairSet& out, double* toi_p,
          double* toi_g, cudaStream_t s) {
  Geo g = g_in;
  if (vtn != 2) g.alpha_s = nullptr;  // per-scene steps apply to trial positions only
  const bool traj = vtn == 3;
  const int nb = g.nb;
  if (!cs.h_small) {
    CK(cudaMallocHost(&cs.h_small, 64 * sizeof(int)));
  }
  // 1. projection
  cs.vbox.ensure(6 * (size_t)g.nv + 6);
  float* vb_cl = bin_clusters(g, cs).v;
  if (vtn == 1) {
    project_boxes(g, 1, 0.0, cs.vbox.p, vb_cl, s);
  } else {
    project_boxes(g, 2, alpha, traj ? nullptr : cs.vbox.p, traj ? nullptr : vb_cl, s);
    if (traj) project_boxes(g, 3, 0.0, cs.vbox.p, vb_cl, s);
  }
  // 2-3. body boxes and overlaps
  cs.bbox.ensure(6 * (size_t)nb);
  cs.bbox_f.ensure(6 * (size_t)nb);
  cs.cnt_all.ensure(nb + 1);
  cs.cnt_up.ensure(nb + 1);
  cs.up_ptr.ensure(nb + 1);
  PairSet& S = out;
  S.row_ptr.ensure(nb + 1);
  KLAUNCH(K_BODY_BOXES, s, k_body_boxes<<<nblk(nb, 128), 128, 0, s>>>(g, vtn, alpha, cs.bbox.p, cs.bbox_f.p));
  KLAUNCH(K_OV_COUNT, s, k_ov_count<<<nblk((long long)nb * 32, 256), 256, 0, s>>>(g, cs.bbox.p, cs.bbox_f.p, cs.cnt_all.p,
                                                                                  cs.cnt_up.p));
  cs.tmp_int.ensure(64);
  int* d_tot = cs.tmp_int.p;  // [0] nnz, [1] nov, [2] list entries, [3] PT, [4] EE, [5] VG, staged
                              // PT and EE ([6], [7])
  scan_exclusive_int2(cs.cnt_all.p, S.row_ptr.p, d_tot, cs.cnt_up.p, cs.up_ptr.p, d_tot + 1, nb, s, cs.vflag_cnt);
  // the vertex-ground pairs need only the positions: counted now, read with the overlaps
  if (!traj) vg_count(g, P, cs, s);
  CK(cudaMemcpyAsync(cs.h_small, d_tot, 6 * sizeof(int), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  int nnz = cs.h_small[0], nov = cs.h_small[1];
  const int nvg = traj ? 0 : cs.h_small[5];
  CK(cudaMemcpyAsync(S.row_ptr.p + nb, d_tot, sizeof(int), cudaMemcpyDeviceToDevice, s));
  S.nnz = nnz;
  S.nov = nov;
  S.col.ensure(nnz + 1);
  S.upidx.ensure(nnz + 1);
  cs.rowid.ensure(nnz + 1);
  S.ovI.ensure(nov + 1);
  S.ovJ.ensure(nov + 1);
  cs.ovcull.ensure(6 * (size_t)nov + 6);
  cs.ovcull_f.ensure(6 * (size_t)nov + 6);
  KLAUNCH(K_OV_FILL, s, k_ov_fill<<<nblk((long long)nb * 32, 256), 256, 0, s>>>(g, cs.bbox.p, cs.bbox_f.p, S.row_ptr.p, cs.up_ptr.p, S.col.p,
                                                          cs.rowid.p, S.upidx.p, S.ovI.p, S.ovJ.p, cs.ovcull.p,
                                                          cs.ovcull_f.p));
  if (nnz) {
    KLAUNCH(K_OV_LOWER, s, k_ov_lower<<<nblk(nnz, 256), 256, 0, s>>>(nnz, S.row_ptr.p, S.col.p, cs.rowid.p, S.upidx.p));
  }
  // 4. primitive boxes and binning
  const float ds_f = float_round_up(P.d_sqrt);
  edge_face_boxes(g, true, cs, s);
  int nlst = 0;
  if (nov > 0) {
    cs.bin_cnt.ensure(6 * (size_t)nov + 6);
    cs.bin_off.ensure(6 * (size_t)nov + 6);
    int nw = 2 * nov;
    const BinClusters cl = bin_clusters(g, cs);
    // list capacity = the primitive counts of both bodies of every overlap; when it fits
    // (at most 2^28 entries) one binning pass writes the lists in place
    bool once = 2ll * nov * g.max_prims < (1ll << 28);
    KLAUNCH(K_BIN, s, k_bin_caps<<<nblk(std::max(6ll * nov, 32ll * g.nb), 256), 256, 0, s>>>(
                          g, nov, S.ovI.p, S.ovJ.p, cs.vbox.p, cl.v, once ? cs.bin_cnt.p : nullptr, cl.tight));
    if (!once) {
      KLAUNCH(K_BIN, s, k_bin<<<nblk((long long)nw * 32, 256), 256, 0, s>>>(g, ds_f, nov, BIN_COUNT, traj, S.ovI.p, S.ovJ.p,
                                                          cs.ovcull.p, cs.ovcull_f.p, cs.vbox.p, cs.ebox.p,
                                                          cs.fbox.p, cl, cl.tight, cs.bin_cnt.p, nullptr, nullptr));
    }
    scan_exclusive_int(cs.bin_cnt.p, cs.bin_off.p, 6 * nov, d_tot + 2, s, cs.vflag_cnt);
    if (once) {
      // the capacities sum to at most both bodies' primitive counts per overlap
      nlst = (int)(2ll * nov * g.max_prims);
    } else {
      CK(cudaMemcpyAsync(cs.h_small + 2, d_tot + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      nlst = cs.h_small[2];
    }
    cs.lst.ensure((size_t)nlst + 1);
    KLAUNCH(K_BIN, s, k_bin<<<nblk((long long)nw * 32, 256), 256, 0, s>>>(g, ds_f, nov, once ? BIN_ONCE : BIN_WRITE, traj,
                                                        S.ovI.p, S.ovJ.p, cs.ovcull.p, cs.ovcull_f.p, cs.vbox.p,
                                                        cs.ebox.p, cs.fbox.p, cl, cl.tight, cs.bin_cnt.p, cs.bin_off.p, cs.lst.p));
  }
  if (traj) {
    const int nk = 2 * g.ns;  // then the number of candidates, read with the keys
    cs.toi_key.ensure(nk + 1);
    if (cs.h_toi_cap < nk + 1) {
      if (cs.h_toi) CK(cudaFreeHost(cs.h_toi));
      CK(cudaMallocHost(&cs.h_toi, (nk + 1) * sizeof(unsigned long long)));
      cs.h_toi_cap = nk + 1;
    }
    unsigned cap = 0;
    double o = 1.0;
    unsigned long long b;
    memcpy(&b, &o, sizeof(b));
    KLAUNCH(K_VG_TOI, s, k_fill_u64<<<nblk(nk, 256), 256, 0, s>>>(cs.toi_key.p, nk, b | 0x8000000000000000ull));
    if (nov > 0) {
      prof_work(K_NARROW_TOI, nov, 48.0 * g.nv);  // positions at q and q + dq
      // refined with the A boxes inflated by sqrt(dhat): a little looser than the TOI
      // needs (its box phase is not inflated, so the TOIs are unchanged), and the lists
      // then hold every candidate of every configuration on the trajectory, which the
      // line-search culls of this step reuse (cull_trial)
      KLAUNCH(K_NARROW_TOI, s, k_refine<true><<<nblk(3ll * nov * 32, 256), 256, 0, s>>>(g, ds_f, nov, S.ovI.p,
                                                                                         S.ovJ.p, cs.bin_cnt.p,
                                                                                         cs.bin_off.p, cs.lst.p,
                                                                                         cs.vbox.p, cs.ebox.p,
                                                                                         cs.fbox.p));
      order_overlaps(nov, cs, s, K_NARROW_TOI);
      narrow_smem_attr();
      traj_floats(g, cs, s);  // allocates cs.vend: before its address is taken
      cs.toi_cand.ensure(std::min(std::max((unsigned)nlst, kToiCandMin), kToiCandMax));
      cap = (unsigned)std::min(cs.toi_cand.cap, (size_t)kToiCandMax);
      unsigned* d_n = reinterpret_cast<unsigned*>(cs.toi_key.p + nk);
      NarrowLaunch a{g, P, ds_f, S.ovI.p, S.ovJ.p, cs.bin_cnt.p, cs.bin_off.p, cs.lst.p, cs.vbox.p, cs.ebox.p,
                     cs.fbox.p, cs.toi_key.p, StageOut{}, Order{cs.order.p, cs.order_cnt.p, nov},
                     ToiCand{cs.vend.p, cs.toi_cand.p, d_n, cap}};
      narrow_phase(2, nov, a, cs, reinterpret_cast<int*>(d_n), s);
      KLAUNCH(K_NARROW_TOI, s, k_toi_list<<<1216, 128, 0, s>>>(g, a.tc, cs.toi_key.p));
    }
    if (P.ground && g.nv) {
      KLAUNCH(K_VG_TOI, s, k_vg_toi<<<nblk(g.nv, 256), 256, 0, s>>>(g, P, cs.toi_key.p + 1));
    }
    CK(cudaMemcpyAsync(cs.h_toi, cs.toi_key.p, (nk + 1) * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (nov > 0) {
      const unsigned found = (unsigned)cs.h_toi[nk];
      if (found > cap) cs.toi_cand.ensure(std::min(found, kToiCandMax));
    }
    for (int sc = 0; sc < g.ns; ++sc) {
      if (toi_p) toi_p[sc] = key_to_double(cs.h_toi[2 * sc]);
      if (toi_g) toi_g[sc] = key_to_double(cs.h_toi[2 * sc + 1]);
    }
    return;
  }
  // 5. narrow phase per overlap: counts, scan, ordered write
  int npt = 0, nee = 0;
  if (nov > 0) {
    KLAUNCH(K_NARROW_SCAN, s, k_refine<true><<<nblk(3ll * nov * 32, 256), 256, 0, s>>>(g, ds_f, nov, S.ovI.p,
                                                                                       S.ovJ.p, cs.bin_cnt.p,
                                                                                       cs.bin_off.p, cs.lst.p,
                                                                                       cs.vbox.p, cs.ebox.p, cs.fbox.p));
    order_overlaps(nov, cs, s, K_NARROW_SCAN);
    narrow_pairs(g, P, ds_f, nov, S.ovI.p, S.ovJ.p, cs, S, npt, nee, s);
  }
  S.npt = npt;
  S.nee = nee;
  // 6. vertex-ground pairs (counted before the overlaps were read)
  vg_write(g, P, cs, S, nvg, s);
}

// Line-search cull at q + alpha dq over the broad phase of this step's trajectory cull H
// (its overlaps, and its lists binned with trajectory boxes and refined with the A boxes
// inflated by sqrt(dhat)): every configuration on the trajectory has its body overlaps
// among H's and its candidates among H's lists, and the lists keep primitive order, so
// the narrow phase at the trial configuration yields the pair set, in the order, that a
// full cull would (overlaps without pairs are extra, empty ones).
void cull_trial(const Geo& g_in, const Params& P, double alpha, CullScratch& cs, const PairSet& H, PairSet& out,
                cudaStream_t s) {
  Geo g = g_in;
  const int nb = g.nb, nov = H.nov, nnz = H.nnz;
  cs.vbox.ensure(6 * (size_t)g.nv + 6);
  project_boxes(g, 2, alpha, cs.vbox.p, nullptr, s);
  vg_count(g, P, cs, s);
  PairSet& S = out;
  S.row_ptr.ensure(nb + 1);
  S.col.ensure(nnz + 1);
  S.upidx.ensure(nnz + 1);
  S.ovI.ensure(nov + 1);
  S.ovJ.ensure(nov + 1);
  CK(cudaMemcpyAsync(S.row_ptr.p, H.row_ptr.p, (nb + 1) * sizeof(int), cudaMemcpyDeviceToDevice, s));
  if (nnz) {
    CK(cudaMemcpyAsync(S.col.p, H.col.p, nnz * sizeof(int), cudaMemcpyDeviceToDevice, s));
    CK(cudaMemcpyAsync(S.upidx.p, H.upidx.p, nnz * sizeof(int), cudaMemcpyDeviceToDevice, s));
  }
  if (nov) {
    CK(cudaMemcpyAsync(S.ovI.p, H.ovI.p, nov * sizeof(int), cudaMemcpyDeviceToDevice, s));
    CK(cudaMemcpyAsync(S.ovJ.p, H.ovJ.p, nov * sizeof(int), cudaMemcpyDeviceToDevice, s));
  }
  S.nnz = nnz;
  S.nov = nov;
  edge_face_boxes(g, false, cs, s);
  int npt = 0, nee = 0, nvg = 0;
  if (nov > 0) {
    narrow_pairs(g, P, float_round_up(P.d_sqrt), nov, S.ovI.p, S.ovJ.p, cs, S, npt, nee, s);
    nvg = cs.h_small[5];
  } else {
    CK(cudaMemcpyAsync(cs.h_small + 5, cs.tmp_int.p + 5, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    nvg = cs.h_small[5];
  }
  S.npt = npt;
  S.nee = nee;
  vg_write(g, P, cs, S, nvg, s);
}

// Vertex-ground pairs in two halves around the host's read of their count (d_tot[5]):
// vg_count launches the per-block counts and their scan, vg_write the ordered write and
// the per-body segments.
void vg_count(const Geo& g, const Params& P, CullScratch& cs, cudaStream_t s) {
  cs.tmp_int.ensure(64);
  int* d_tot = cs.tmp_int.p;
  if (P.ground && g.nv) {
    int nbv = nblk(g.nv, 256);
    cs.vflag_off.ensure(nbv + 1);
    cs.vg_cnt.ensure(nbv + 1);
    KLAUNCH(K_VG, s, k_vg_count<<<nbv, 256, 0, s>>>(g, P, cs.vg_cnt.p));
    scan_exclusive_int(cs.vg_cnt.p, cs.vflag_off.p, nbv, d_tot + 5, s, cs.vflag_cnt);
  } else {
    CK(cudaMemsetAsync(d_tot + 5, 0, sizeof(int), s));
  }
}

void vg_write(const Geo& g, const Params& P, CullScratch& cs, PairSet& S, int nvg, cudaStream_t s) {
  const int nb = g.nb;
  S.vg_seg.ensure(nb + 2);
  if (P.ground && g.nv) {
    S.vg.ensure(2 * (size_t)nvg + 2);
    KLAUNCH(K_VG, s, k_vg_write<<<nblk(g.nv, 256), 256, 0, s>>>(g, P, cs.vflag_off.p, S.vg.p));
  } else {
    nvg = 0;
  }
  S.nvg = nvg;
  S.vg.ensure(2);
  KLAUNCH(K_VG, s, k_vg_seg<<<nblk(nb + 1, 256), 256, 0, s>>>(nb, nvg, S.vg.p, S.vg_seg.p));
}

void vg_pairs(const Geo& g, const Params& P, CullScratch& cs, PairSet& S, cudaStream_t s) {
  if (!cs.h_small) {
    CK(cudaMallocHost(&cs.h_small, 64 * sizeof(int)));
  }
  vg_count(g, P, cs, s);
  CK(cudaMemcpyAsync(cs.h_small + 5, cs.tmp_int.p + 5, sizeof(int), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  vg_write(g, P, cs, S, cs.h_small[5], s);
}

void launch_vg_toi(const Geo& g, const Params& P, unsigned long long* toi_key, cudaStream_t s) {
  if (!g.nv) return;
  KLAUNCH(K_VG_TOI, s, k_vg_toi<<<nblk(g.nv, 256), 256, 0, s>>>(g, P, toi_key + 1));
}

}  // namespace abd
