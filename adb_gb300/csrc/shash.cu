// Spatial-hash broad phase (the reference's iaabb-even path): gen_collision_set
// (model/col_set.cpp:20-339, global point / edge / triangle lists) and
// step_size_upper_bound (model/upper_bound.cpp:16-277) over the hash grid of
// model/spatial_hashing.cpp:11-211.
//
// Grid: a point x lies in cell int(max(x - min_xyz, 0) / dx) per axis; a cell's bucket
// keeps the low xyz_bits bits of each coordinate (spatial_hashing.cpp:11-21), so cells
// that agree modulo 2^xyz_bits share a bucket. A registered primitive is a candidate of a
// query when one of the query's cells has a bucket that holds it (the reference gathers,
// sorts and de-duplicates per query).
//
// How the candidates are found. Registration counts each bucket's entries, gives every used
// bucket a segment and writes (primitive, body) into it; the order inside a bucket is free,
// because pairs are sorted by key afterwards and times of impact are min-reduced. One warp
// per query primitive then walks the buckets of its cells, an entry per lane. With the
// reference's default cell (0.8) a bucket holds hundreds to thousands of primitives and
// nearly all of them are far away, so the walk runs in FP32 only: an outward-rounded box
// test for the culls, the certificates of abd_ccd_filter.cuh for the trajectories. What
// is left is appended to a list that a second kernel evaluates in FP64, a pair per thread.
// (One thread per query used to walk the buckets, with six FP64 divisions per entry for
// its cell range, count and write passes for the culls and a sort of all entries. A frame of
// 33 icospheres, 3 culls and 2 bounds: 489 -> 4.6 ms, of which the queries take 1.5 and the
// rest of the hash 0.9.)
//
// Distance culling keeps the pairs of different bodies with squared distance below
// dhat * safe_factor^2 (PT: vertex of any body against a triangle; EE: edges of bodies
// I < J) and orders them as the overlap-based path does (body pair, then vertex-on-I,
// vertex-on-J, edge-edge, each by primitive ids), building the body-pair CSR the
// assembly walks. The reference appends its threads' pairs in scheduling order, so only
// the set is defined there. The trajectory bound takes the exact time of impact of every
// candidate that shares a bucket (edge trajectories registered by their start position
// unless the fix flag is set, as upper_bound.cpp:151 does), or the d_sqrt / |dq|_1
// bound lowered by the current pairs' times of impact.
#include <algorithm>
#include <cstring>
#include <stdexcept>

#include "abd_ccd_filter.cuh"
#include "abd_engine.h"
#include "abd_exact.cuh"

namespace abd {

namespace {

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

// Order-preserving key of a double for atomicMin on unsigned 64-bit.
__device__ __forceinline__ unsigned long long dkey(double x) {
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ d3 ldX(const double* X, int nv, int v) { return mk(X[v], X[nv + v], X[2 * nv + v]); }

struct ShGrid {
  double mn, dx;
  int bits;
};

__device__ __forceinline__ int sh_cell(double x, const ShGrid& G) {
  double t = XS(x, G.mn);
  t = t < 0.0 ? 0.0 : t;
  return (int)XD(t, G.dx);
}
__device__ __forceinline__ void sh_cells(const d3& p, const ShGrid& G, int* c) {
  c[0] = sh_cell(p.x, G);
  c[1] = sh_cell(p.y, G);
  c[2] = sh_cell(p.z, G);
}
__device__ __forceinline__ unsigned sh_hash(int i, int j, int k, int bits) {
  unsigned m = (1u << bits) - 1u;
  return ((((unsigned)i & m) << bits | ((unsigned)j & m)) << bits) | ((unsigned)k & m);
}
__device__ __forceinline__ d3 dmin3(const d3& a, const d3& b) { return mk(dmin(a.x, b.x), dmin(a.y, b.y), dmin(a.z, b.z)); }
__device__ __forceinline__ d3 dmax3(const d3& a, const d3& b) { return mk(dmax(a.x, b.x), dmax(a.y, b.y), dmax(a.z, b.z)); }

// First cell coordinate a >= l whose bucket residue lies in the residues of [rl, ru].
__device__ __forceinline__ int first_hit(int l, int rl, int ru, int bits) {
  const int M = 1 << bits, m = M - 1;
  int L = ru - rl + 1;
  if (L >= M) return l;
  int off = ((l & m) - (rl & m)) & m;
  return off < L ? l : l + (M - off);
}

// Registered box of a primitive. kind 0: vertex (point, or q -> target segment when
// traj); kind 1: edge (segment at the target, or at q when traj, widened to the target
// positions when fix_edge).
__device__ __forceinline__ void reg_box(const Geo& g, int kind, int id, int traj, int fix_edge, d3& lo, d3& hi) {
  if (kind == 0) {
    d3 p = ldX(g.X, g.nv, id);
    if (traj) {
      d3 p0 = ldX(g.Xq, g.nv, id);
      lo = dmin3(p0, p);
      hi = dmax3(p0, p);
    } else {
      lo = hi = p;
    }
    return;
  }
  int a = g.ev[2 * id], b = g.ev[2 * id + 1];
  const double* P = traj ? g.Xq : g.X;
  d3 a0 = ldX(P, g.nv, a), a1 = ldX(P, g.nv, b);
  lo = dmin3(a0, a1);
  hi = dmax3(a0, a1);
  if (traj && fix_edge) {
    d3 b0 = ldX(g.X, g.nv, a), b1 = ldX(g.X, g.nv, b);
    lo = dmin3(lo, dmin3(b0, b1));
    hi = dmax3(hi, dmax3(b0, b1));
  }
}

// Cells of the registered primitives (kind 0: vertices, 1: edges) and the number of cells
// they cover in all.
__global__ void k_reg_cells(Geo g, ShGrid G, int kind, int n, int traj, int fix_edge, ShCells* cells,
                            unsigned long long* total) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long c = 0;
  if (id < n) {
    d3 lo, hi;
    reg_box(g, kind, id, traj, fix_edge, lo, hi);
    ShCells r;
    sh_cells(lo, G, r.l);
    sh_cells(hi, G, r.u);
    cells[id] = r;
    // capped where it is too many anyway: the product of three counts can wrap around (2^22 by
    // 2^21 by 2^21 cells would count as none, and the entries go past a list of no length)
    c = 1;
    for (int a = 0; a < 3; ++a) c = min(c * ((unsigned long long)((unsigned)r.u[a] - (unsigned)r.l[a]) + 1ull), 1ull << 31);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(total, c);
}

// Cells l .. u of an axis that differ in their bucket: those 2^bits apart share one.
__device__ __forceinline__ int cell_count(int l, int u, int bits) {
  return (int)min((unsigned)u - (unsigned)l, (1u << bits) - 1u) + 1;
}
// The buckets of a cell range, each once (f(bucket)).
template <typename F>
__device__ __forceinline__ void for_buckets(const ShCells& r, int bits, F&& f) {
  const int n0 = cell_count(r.l[0], r.u[0], bits), n1 = cell_count(r.l[1], r.u[1], bits),
            n2 = cell_count(r.l[2], r.u[2], bits);
  for (int i = 0; i < n0; ++i)
    for (int j = 0; j < n1; ++j)
      for (int k = 0; k < n2; ++k) f(sh_hash(r.l[0] + i, r.l[1] + j, r.l[2] + k, bits));
}

// Table build: empty the buckets used last (cnt is zero outside them), count, give each
// used bucket its segment, fill. ctl: [0] used buckets, [1] entries.
__global__ void k_bucket_clear(const int* ctl, const int* used, int* cnt) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ctl[0]; i += gridDim.x * blockDim.x) cnt[used[i]] = 0;
}
__global__ void k_bucket_count(ShGrid G, int n, const ShCells* cells, int* cnt, int* used, int* ctl) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= n) return;
  for_buckets(cells[id], G.bits, [&](unsigned b) {
    if (atomicAdd(&cnt[b], 1) == 0) used[atomicAdd(&ctl[0], 1)] = (int)b;
  });
}
__global__ void k_bucket_alloc(int* ctl, const int* used, const int* cnt, int* cur) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ctl[0]) return;
  const int b = used[i];
  cur[b] = atomicAdd(&ctl[1], cnt[b]);
}
__global__ void k_bucket_fill(Geo g, ShGrid G, int kind, int n, const ShCells* cells, int* cur, int2* ent) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= n) return;
  const int body = g.vbody[kind ? g.ev[2 * id] : id];
  for_buckets(cells[id], G.bits, [&](unsigned b) { ent[atomicAdd(&cur[b], 1)] = make_int2(id, body); });
}

struct ShQuery {
  ShGrid G;
  const ShCells *rcells, *qcells;   // of the registered and of the query primitives
  const int *cnt, *end;             // buckets: entries, end of the segment
  const int2* ent;                  // (primitive, body)
  double qd;     // query box growth (d_sqrt * safe_factor); 0 for trajectories
  float qd_f;    // the same, rounded up past every rounding of the FP64 distance
  double thr;    // squared-distance threshold (dhat * safe_factor^2)
  const float *vb, *eb, *fb;        // float boxes of the primitives (culls)
  const float* vend;                // float positions of the vertices at q and at the target (trajectories)
  int2* cand;                       // candidates: (query primitive, registered primitive)
  unsigned long long cand_cap;
  unsigned long long* n;            // [0] candidates, [1] accepted pairs
};

// Cells of the query primitives (kind 0: triangles, 1: edges): the box at the target, grown
// by qd, or of the whole trajectory.
__global__ void k_query_cells(Geo g, ShGrid G, int kind, int nq, int traj, double qd, ShCells* cells) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= nq) return;
  const int nvtx = kind ? 2 : 3;
  const int* vid = kind ? g.ev + 2 * id : g.fv + 3 * id;
  d3 lo = ldX(g.X, g.nv, vid[0]), hi = lo;
  for (int k = 1; k < nvtx; ++k) {
    const d3 p = ldX(g.X, g.nv, vid[k]);
    lo = dmin3(lo, p);
    hi = dmax3(hi, p);
  }
  if (traj) {
    for (int k = 0; k < nvtx; ++k) {
      const d3 p = ldX(g.Xq, g.nv, vid[k]);
      lo = dmin3(lo, p);
      hi = dmax3(hi, p);
    }
  } else {
    lo = mk(XA(lo.x, -qd), XA(lo.y, -qd), XA(lo.z, -qd));
    hi = mk(XA(hi.x, qd), XA(hi.y, qd), XA(hi.z, qd));
  }
  ShCells r;
  sh_cells(lo, G, r.l);
  sh_cells(hi, G, r.u);
  cells[id] = r;
}

__device__ __forceinline__ unsigned long long pair_key(int A, int a, int B, int b, int sub) {
  unsigned long long lo = A < B ? A : B, hi = A < B ? B : A;
  return (lo << 47) | (hi << 32) | ((unsigned long long)sub << 30) | ((unsigned long long)a << 15) |
         (unsigned long long)b;
}

__device__ __forceinline__ f3 ldf3(const float* p) { return f3{p[0], p[1], p[2]}; }

// Candidates of the query primitives [qbeg, qend), one warp each. KIND 0: triangles against vertices of
// other bodies; 1: edges against the edges of lower bodies (of the same scene both). An entry
// in several of the query's buckets is taken in the first cell that holds it, as by its cell
// range (the test every entry used to pay for, here only for those the FP32 test leaves).
template <int KIND, bool TRAJ>
__global__ void __launch_bounds__(128) k_sh_query(Geo g, ShQuery Q, int qbeg, int qend) {
  const int q = qbeg + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (q >= qend) return;
  constexpr int NV = KIND ? 2 : 3;
  const int* qv = KIND ? g.ev + 2 * q : g.fv + 3 * q;
  const int J = g.vbody[qv[0]], sc = g.bscene[J];
  if (!scene_on(g, J)) return;
  f3 q0[NV], q1[NV];
  float qb[6];
  if (TRAJ) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const float* p = Q.vend + 6 * (size_t)qv[k];
      q0[k] = ldf3(p);
      q1[k] = ldf3(p + 3);
    }
  } else {
    const float* p = (KIND ? Q.eb : Q.fb) + 6 * (size_t)q;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      qb[c] = __fsub_rd(p[c], Q.qd_f);
      qb[c + 3] = __fadd_ru(p[c + 3], Q.qd_f);
    }
  }
  const ShCells r = Q.qcells[q];
  // Cells are counted: a coordinate past 2^31 cells is in the last one an int holds, and a loop
  // up to that cell would not end.
  const int n0 = cell_count(r.l[0], r.u[0], Q.G.bits), n1 = cell_count(r.l[1], r.u[1], Q.G.bits),
            n2 = cell_count(r.l[2], r.u[2], Q.G.bits);
  for (int di = 0; di < n0; ++di)
    for (int dj = 0; dj < n1; ++dj)
      for (int dk = 0; dk < n2; ++dk) {
        const int i = r.l[0] + di, j = r.l[1] + dj, k = r.l[2] + dk;
        const unsigned b = sh_hash(i, j, k, Q.G.bits);
        const int n = Q.cnt[b];
        if (n == 0) continue;  // an unused bucket has no segment
        const int2* ent = Q.ent + (Q.end[b] - n);
        for (int t0 = 0; t0 < n; t0 += 32) {
          bool take = false;
          int id = 0;
          if (t0 + lane < n) {
            const int2 e = ent[t0 + lane];
            id = e.x;
            if ((KIND ? e.y < J : e.y != J) && g.bscene[e.y] == sc) {
              if (TRAJ) {
                if (KIND) {
                  const float *pa = Q.vend + 6 * (size_t)g.ev[2 * id], *pb = Q.vend + 6 * (size_t)g.ev[2 * id + 1];
                  const f3 a0[2] = {ldf3(pa), ldf3(pb)}, a1[2] = {ldf3(pa + 3), ldf3(pb + 3)};
                  take = !f_ee_miss(a0, a1, q0, q1);
                } else {
                  const float* p = Q.vend + 6 * (size_t)id;
                  take = !f_pt_miss(ldf3(p), ldf3(p + 3), q0, q1);
                }
              } else {
                const float* p = (KIND ? Q.eb : Q.vb) + 6 * (size_t)id;
                take = p[0] <= qb[3] && p[3] >= qb[0] && p[1] <= qb[4] && p[4] >= qb[1] && p[2] <= qb[5] &&
                       p[5] >= qb[2];
              }
              if (take) {
                const ShCells c = Q.rcells[id];
                take = i == first_hit(r.l[0], c.l[0], c.u[0], Q.G.bits) &&
                       j == first_hit(r.l[1], c.l[1], c.u[1], Q.G.bits) &&
                       k == first_hit(r.l[2], c.l[2], c.u[2], Q.G.bits);
              }
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, take);
          if (m) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(&Q.n[0], (unsigned long long)__popc(m));
            base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
            if (take && base < Q.cand_cap) Q.cand[base] = make_int2(q, id);
          }
        }
      }
}

// Candidates in FP64: the pairs with squared distance below thr, as keys.
template <int KIND>
__global__ void __launch_bounds__(128) k_sh_exact(Geo g, ShQuery Q, unsigned long long* keys,
                                                  unsigned long long key_cap) {
  const int n = (int)min(Q.n[0], Q.cand_cap);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int2 c = Q.cand[t];
    const int q = c.x, e = c.y;
    unsigned long long key;
    if (KIND == 0) {
      const int i0 = g.fv[3 * q], I = g.vbody[e], J = g.vbody[i0];
      const d3 p = ldX(g.X, g.nv, e), t0 = ldX(g.X, g.nv, i0), t1 = ldX(g.X, g.nv, g.fv[3 * q + 1]),
               t2 = ldX(g.X, g.nv, g.fv[3 * q + 2]);
      if (!(pt_dist(p, t0, t1, t2, pt_type(p, t0, t1, t2)) < Q.thr)) continue;
      key = pair_key(I, e - g.v_off[I], J, q - g.f_off[J], I < J ? 0 : 1);
    } else {
      const int ia = g.ev[2 * e], ib = g.ev[2 * q], I = g.vbody[ia], J = g.vbody[ib];
      const d3 a0 = ldX(g.X, g.nv, ia), a1 = ldX(g.X, g.nv, g.ev[2 * e + 1]), b0 = ldX(g.X, g.nv, ib),
               b1 = ldX(g.X, g.nv, g.ev[2 * q + 1]);
      if (!(ee_dist(a0, a1, b0, b1, ee_type(a0, a1, b0, b1)) < Q.thr)) continue;
      key = pair_key(I, e - g.e_off[I], J, q - g.e_off[J], 2);
    }
    const unsigned long long o = atomicAdd(&Q.n[1], 1ull);
    if (o < key_cap) keys[o] = key;
  }
}

// Candidates in FP64: the earliest time of impact per scene.
template <int KIND>
__global__ void __launch_bounds__(128) k_sh_toi(Geo g, ShQuery Q, unsigned long long* toi_key) {
  const int n = (int)min(Q.n[0], Q.cand_cap);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int q = Q.cand[t].x, e = Q.cand[t].y;
    int vid[4];
    if (KIND == 0) {
      vid[0] = e;
      for (int k = 0; k < 3; ++k) vid[1 + k] = g.fv[3 * q + k];
    } else {
      for (int k = 0; k < 2; ++k) {
        vid[k] = g.ev[2 * e + k];
        vid[2 + k] = g.ev[2 * q + k];
      }
    }
    const int J = g.vbody[vid[3]];
    d3 p0[4], p1[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      p0[k] = ldX(g.Xq, g.nv, vid[k]);
      p1[k] = ldX(g.X, g.nv, vid[k]);
    }
    const double tc = toi_fast<KIND>(p0, p1);
    if (tc < 1.0) atomicMin(toi_key + 2 * g.bscene[J], dkey(tc));
  }
}

// Sorted pair keys -> tuples, distance types (recomputed, as in the query) and the
// body-pair key of each pair.
__global__ void k_decode_pt(Geo g, int n, const unsigned long long* keys, int* pt, int8_t* ty, unsigned* bp) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  unsigned long long k = keys[p];
  int lo = (int)(k >> 47), hi = (int)((k >> 32) & 0x7fff), sub = (int)((k >> 30) & 3);
  int a = (int)((k >> 15) & 0x7fff), b = (int)(k & 0x7fff);
  int A = sub == 0 ? lo : hi, B = sub == 0 ? hi : lo;
  pt[4 * p] = A; pt[4 * p + 1] = a; pt[4 * p + 2] = B; pt[4 * p + 3] = b;
  int f = g.f_off[B] + b;
  d3 x = ldX(g.X, g.nv, g.v_off[A] + a);
  d3 t0 = ldX(g.X, g.nv, g.fv[3 * f]), t1 = ldX(g.X, g.nv, g.fv[3 * f + 1]), t2 = ldX(g.X, g.nv, g.fv[3 * f + 2]);
  ty[p] = (int8_t)pt_type(x, t0, t1, t2);
  bp[p] = (unsigned)(k >> 32);
}
__global__ void k_decode_ee(Geo g, int n, const unsigned long long* keys, int* ee, int8_t* ty, unsigned* bp) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  unsigned long long k = keys[p];
  int A = (int)(k >> 47), B = (int)((k >> 32) & 0x7fff);
  int a = (int)((k >> 15) & 0x7fff), b = (int)(k & 0x7fff);
  ee[4 * p] = A; ee[4 * p + 1] = a; ee[4 * p + 2] = B; ee[4 * p + 3] = b;
  int ea = g.e_off[A] + a, eb = g.e_off[B] + b;
  d3 a0 = ldX(g.X, g.nv, g.ev[2 * ea]), a1 = ldX(g.X, g.nv, g.ev[2 * ea + 1]);
  d3 b0 = ldX(g.X, g.nv, g.ev[2 * eb]), b1 = ldX(g.X, g.nv, g.ev[2 * eb + 1]);
  ty[p] = (int8_t)ee_type(a0, a1, b0, b1);
  bp[p] = (unsigned)(k >> 32);
}

// Body-pair keys (I << 15 | J) of both lists as 64-bit sort keys.
__global__ void k_bp_keys(int npt, const unsigned* bpt, int nee, const unsigned* bee, unsigned long long* out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < npt) out[i] = bpt[i];
  else if (i < npt + nee) out[i] = bee[i - npt];
}
__global__ void k_unique_flags(long long n, const unsigned long long* k, int* flag) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flag[i] = (i == 0 || k[i] != k[i - 1]) ? 1 : 0;
}
__global__ void k_unique_write(long long n, const unsigned long long* k, const int* flag, const int* pos, int* ovI,
                               int* ovJ, unsigned long long* tkeys) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !flag[i]) return;
  int u = pos[i];
  int I = (int)(k[i] >> 15), J = (int)(k[i] & 0x7fff);
  ovI[u] = I;
  ovJ[u] = J;
  tkeys[u] = ((unsigned long long)J << 32) | (unsigned)u;  // transposed: row J, lower entry
}

__device__ __forceinline__ int lb_ov(const int* ovI, int nov, int r) {
  int lo = 0, hi = nov;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (ovI[mid] < r) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ int lb_t(const unsigned long long* t, int nov, int r) {
  int lo = 0, hi = nov;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if ((int)(t[mid] >> 32) < r) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Row r of the symmetric CSR: lower entries (overlaps (I, r), I ascending) then upper
// entries (overlaps (r, J), J ascending); upidx is the overlap of each entry.
__global__ void k_csr_count(int nb, int nov, const int* ovI, const unsigned long long* tkeys, int* cnt) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nb) return;
  cnt[r] = (lb_t(tkeys, nov, r + 1) - lb_t(tkeys, nov, r)) + (lb_ov(ovI, nov, r + 1) - lb_ov(ovI, nov, r));
}
__global__ void k_csr_fill(int nb, int nov, const int* ovI, const int* ovJ, const unsigned long long* tkeys,
                           const int* row_ptr, int* col, int* upidx) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nb) return;
  int e = row_ptr[r];
  for (int t = lb_t(tkeys, nov, r), t1 = lb_t(tkeys, nov, r + 1); t < t1; ++t) {
    int u = (int)(tkeys[t] & 0xffffffffull);
    col[e] = ovI[u];
    upidx[e++] = u;
  }
  for (int u = lb_ov(ovI, nov, r), u1 = lb_ov(ovI, nov, r + 1); u < u1; ++u) {
    col[e] = ovJ[u];
    upidx[e++] = u;
  }
}

// Overlap of every pair (binary search of its body-pair key in the unique list).
__global__ void k_pair_ov(int n, const unsigned* bp, int nov, const int* ovI, const int* ovJ, int* pov) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  unsigned key = bp[p];
  int lo = 0, hi = nov;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    unsigned km = ((unsigned)ovI[mid] << 15) | (unsigned)ovJ[mid];
    if (km < key) lo = mid + 1;
    else hi = mid;
  }
  pov[p] = lo;
}

// step_size_upper_bound without full_ccd: per scene, d_sqrt / 2 / max_I |dq_I|_1 * sf,
// capped at 1 (upper_bound.cpp:232-233).
__global__ void __launch_bounds__(256) k_norm1_bound(const int* sc_beg, const int* sc_end, const double* dq,
                                                    double half_ds, double sf, unsigned long long* toi_key) {
  __shared__ double sh[8];
  int s = blockIdx.x;
  double m = 0.0;
  for (int b = sc_beg[s] + (int)threadIdx.x; b < sc_end[s]; b += blockDim.x) {
    double a = 0.0;
    for (int i = 0; i < 12; ++i) a += fabs(dq[12 * b + i]);
    m = dmax(m, a);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = dmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = dmax(m, sh[w]);
    double t = XM(XD(half_ds, m), sf);
    t = t < 1.0 ? t : 1.0;
    atomicMin(toi_key + 2 * s, dkey(t));
  }
}

// ... lowered by the times of impact of the current pairs.
__global__ void k_pair_toi(Geo g, int npt, const int* pt, int nee, const int* ee, unsigned long long* toi_key) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  double t = 1.0;
  int A;
  if (p < npt) {
    A = pt[4 * p];
    int v = g.v_off[A] + pt[4 * p + 1], B = pt[4 * p + 2], f = g.f_off[B] + pt[4 * p + 3];
    int i0 = g.fv[3 * f], i1 = g.fv[3 * f + 1], i2 = g.fv[3 * f + 2];
    d3 f0[3] = {ldX(g.Xq, g.nv, i0), ldX(g.Xq, g.nv, i1), ldX(g.Xq, g.nv, i2)};
    d3 f1[3] = {ldX(g.X, g.nv, i0), ldX(g.X, g.nv, i1), ldX(g.X, g.nv, i2)};
    t = pt_collision_time(ldX(g.Xq, g.nv, v), f0, ldX(g.X, g.nv, v), f1);
  } else if (p < npt + nee) {
    int q = p - npt;
    A = ee[4 * q];
    int ea = g.e_off[A] + ee[4 * q + 1], B = ee[4 * q + 2], eb = g.e_off[B] + ee[4 * q + 3];
    d3 a0[2] = {ldX(g.Xq, g.nv, g.ev[2 * ea]), ldX(g.Xq, g.nv, g.ev[2 * ea + 1])};
    d3 a1[2] = {ldX(g.X, g.nv, g.ev[2 * ea]), ldX(g.X, g.nv, g.ev[2 * ea + 1])};
    d3 b0[2] = {ldX(g.Xq, g.nv, g.ev[2 * eb]), ldX(g.Xq, g.nv, g.ev[2 * eb + 1])};
    d3 b1[2] = {ldX(g.X, g.nv, g.ev[2 * eb]), ldX(g.X, g.nv, g.ev[2 * eb + 1])};
    t = ee_collision_time(a0, b0, a1, b1);
  } else {
    return;
  }
  if (t < 1.0) atomicMin(toi_key + 2 * g.bscene[A], dkey(t));
}
__global__ void k_vg_pair_toi(Geo g, Params P, int nvg, const int* vg, unsigned long long* toi_key) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nvg) return;
  int b = vg[2 * k], v = g.v_off[b] + vg[2 * k + 1];
  double d2 = XA(g.X[g.nv + v], P.ground_offset);
  if (!(d2 < 0)) return;
  double d1 = XA(g.Xq[g.nv + v], P.ground_offset);
  double t = XD(d1, XS(d1, d2));
  if (t < 1.0) atomicMin(toi_key + 2 * g.bscene[b], dkey(t));
}

__global__ void k_fill_key(unsigned long long* p, int n, unsigned long long v) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

double key_to_double_h(unsigned long long k) {
  unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  double d;
  memcpy(&d, &b, sizeof(d));
  return d;
}

ShGrid grid_of(const ShParams& H) { return ShGrid{H.min_xyz, H.dx, H.bits}; }

}  // namespace

void ShScratch::release() {
  tab.cells.release(); tab.cnt.release(); tab.cur.release(); tab.used.release(); tab.ctl.release();
  tab.ent.release(); qcells.release(); cand.release(); n.release(); scan_i.release(); flag.release(); pos.release();
  pt_keys.release(); ee_keys.release(); bp_all.release(); tkeys.release(); bp_pt.release(); bp_ee.release();
  if (h_int) cudaFreeHost(h_int);
  if (h_n) cudaFreeHost(h_n);
  if (h_toi) cudaFreeHost(h_toi);
  h_int = nullptr;
  h_n = nullptr;
  h_toi = nullptr;
  h_toi_cap = 0;
}

// Registers `n` primitives of `kind` and builds the bucket table in `T`.
static void sh_register(const Geo& g, const ShParams& H, int kind, int n, int traj, ShTable& T, cudaStream_t s) {
  ShGrid G = grid_of(H);
  const size_t nbuckets = (size_t)1 << (3 * H.bits);
  T.ctl.ensure(4);
  if (T.cnt.cap < nbuckets) {
    T.cnt.ensure(nbuckets);
    T.cur.ensure(nbuckets);
    CK(cudaMemsetAsync(T.cnt.p, 0, T.cnt.cap * sizeof(int), s));
  } else {
    KLAUNCH(K_SH, s, k_bucket_clear<<<152, 256, 0, s>>>(T.ctl.p, T.used.p, T.cnt.p));
  }
  CK(cudaMemsetAsync(T.ctl.p, 0, 4 * sizeof(int), s));
  if (n == 0) return;
  T.cells.ensure(n);
  unsigned long long* d_tot = reinterpret_cast<unsigned long long*>(T.ctl.p + 2);
  KLAUNCH(K_SH, s, k_reg_cells<<<nblk(n, 256), 256, 0, s>>>(g, G, kind, n, traj, H.fix_edge, T.cells.p, d_tot));
  CK(cudaMemcpyAsync(&T.h_tot, d_tot, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const unsigned long long tot = T.h_tot;
  if (tot > (1ull << 31) - 1) throw std::invalid_argument("spatial hash: too many cell registrations (dx too small)");
  T.used.ensure(std::min((size_t)tot, nbuckets));
  T.ent.ensure((size_t)tot);
  KLAUNCH(K_SH, s, k_bucket_count<<<nblk(n, 256), 256, 0, s>>>(G, n, T.cells.p, T.cnt.p, T.used.p, T.ctl.p));
  const long long most = (long long)std::min((size_t)tot, nbuckets);
  KLAUNCH(K_SH, s, k_bucket_alloc<<<nblk(most, 256), 256, 0, s>>>(T.ctl.p, T.used.p, T.cnt.p, T.cur.p));
  KLAUNCH(K_SH, s, k_bucket_fill<<<nblk(n, 256), 256, 0, s>>>(g, G, kind, n, T.cells.p, T.cur.p, T.ent.p));
}

// Candidates kept at a time: 32 an edge or face, 16 k at least, 16 MB at most. The list grows to what
// a run of queries leaves; past 16 MB the queries are taken in parts.
constexpr size_t kCandMin = 1u << 14, kCandMax = 1u << 21;

// Registers the primitives that the queries of `kind` run against, computes the queries' cells
// and fills Q (list and counters included).
static void sh_prepare(const Geo& g, const ShParams& H, int kind, int traj, ShScratch& W, CullScratch& cs, ShQuery& Q,
                       cudaStream_t s) {
  sh_register(g, H, kind, kind ? g.ne : g.nv, traj, W.tab, s);
  const int nq = kind ? g.ne : g.nf;
  W.qcells.ensure(nq);
  KLAUNCH(K_SH, s, k_query_cells<<<nblk(nq, 256), 256, 0, s>>>(g, Q.G, kind, nq, traj, Q.qd, W.qcells.p));
  Q.rcells = W.tab.cells.p;
  Q.qcells = W.qcells.p;
  Q.cnt = W.tab.cnt.p;
  Q.end = W.tab.cur.p;  // once filled
  Q.ent = W.tab.ent.p;
  Q.vb = cs.vbox.p;
  Q.eb = cs.ebox.p;
  Q.fb = cs.fbox.p;
  Q.vend = cs.vend.p;
  W.n.ensure(2);
  Q.n = W.n.p;
  W.cand.ensure(std::min(std::max((size_t)32 * std::max(g.ne, g.nf), kCandMin), kCandMax));  // once, for both kinds
  if (!W.h_n) CK(cudaMallocHost(&W.h_n, 2 * sizeof(unsigned long long)));
}

// Runs the query over all primitives of a kind, `eval` on each list and `done` on its two
// counters (false: the same queries again). The queries are taken all at once unless they
// leave more candidates than the largest list holds; then in runs of half as many, down to single
// queries, for which the list grows further (a query has at most as many as there are
// primitives), and of twice as many after a run that fills at most half of it.
template <int KIND, bool TRAJ, typename Eval, typename Done>
static void sh_run(const Geo& g, ShQuery& Q, ShScratch& W, cudaStream_t s, Eval&& eval, Done&& done) {
  const int nq = KIND ? g.ne : g.nf;
  int step = nq;
  for (int q0 = 0; q0 < nq;) {
    const int m = std::min(step, nq - q0);
    Q.cand = W.cand.p;
    Q.cand_cap = std::min<size_t>(W.cand.cap, (1ull << 31) - 1);
    CK(cudaMemsetAsync(Q.n, 0, 2 * sizeof(unsigned long long), s));
    KLAUNCH(K_SH, s, k_sh_query<KIND, TRAJ><<<nblk(32ll * m, 128), 128, 0, s>>>(g, Q, q0, q0 + m));
    eval();
    CK(cudaMemcpyAsync(W.h_n, Q.n, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const size_t found = (size_t)W.h_n[0];
    if (found > Q.cand_cap) {
      if (found <= kCandMax || m == 1) W.cand.ensure(found);
      else step = std::max(1, m / 2);
      continue;
    }
    if (done()) {
      q0 += m;
      // past a dense part of the scene the runs become longer again
      if (2 * found <= Q.cand_cap) step = m <= nq / 2 ? 2 * m : nq;
    }
  }
}

// The pairs of one kind into `keys`, sorted; returns how many. The keys grow to the counted
// total when they overflow.
template <int KIND>
static int sh_pairs(const Geo& g, const ShParams& H, ShQuery& Q, ShScratch& W, CullScratch& cs,
                    DBuf<unsigned long long>& keys, cudaStream_t s) {
  sh_prepare(g, H, KIND, 0, W, cs, Q, s);
  keys.ensure(1u << 15);
  size_t np = 0, lim = 0;
  sh_run<KIND, false>(
      g, Q, W, s,
      [&]() {
        lim = sort_padded_size(1);  // most keys that the sort can pad inside the buffer
        while (2 * lim <= keys.cap) lim *= 2;
        KLAUNCH(K_SH, s, k_sh_exact<KIND><<<608, 128, 0, s>>>(g, Q, keys.p + np, lim - np));
      },
      [&]() {
        const size_t all = np + (size_t)W.h_n[1];
        if (all > lim) {
          keys.ensure(sort_padded_size(all), true, np);
          return false;
        }
        np = all;
        return true;
      });
  if (np) sort_u64(keys.p, np, keys.cap, s);
  return (int)np;
}

void sh_cull(const Geo& g, const Params& P, const ShParams& H, int vtn, double alpha, ShScratch& W, CullScratch& cs,
             PairSet& S, cudaStream_t s) {
  const int nb = g.nb;
  launch_project(g, vtn == 1 ? 1 : 2, alpha, s);
  const double sf = H.safe_factor;
  ShQuery Q{};
  Q.G = grid_of(H);
  Q.qd = P.d_sqrt * sf;
  // 1e-5 past qd: a box further apart than that has an FP64 squared distance above thr
  Q.qd_f = nextafterf((float)(Q.qd * (1.0 + 1e-5)), INFINITY);
  Q.thr = P.dhat * (sf * sf);
  if (!W.h_int) CK(cudaMallocHost(&W.h_int, 8 * sizeof(int)));
  const bool do_pt = P.pt && g.nv && g.nf, do_ee = P.ee && g.ne;
  if (do_pt || do_ee) prim_boxes(g, cs, s);
  // PT: vertices registered, triangles query; EE: edges registered, edges of the higher body
  // query
  const int npt = do_pt ? sh_pairs<0>(g, H, Q, W, cs, W.pt_keys, s) : 0;
  const int nee = do_ee ? sh_pairs<1>(g, H, Q, W, cs, W.ee_keys, s) : 0;
  // tuples, types and body-pair keys
  S.npt = npt;
  S.nee = nee;
  S.pt.ensure(4 * (size_t)npt + 4);
  S.pt_ty.ensure((size_t)npt + 1);
  S.pt_ov.ensure((size_t)npt + 1);
  S.ee.ensure(4 * (size_t)nee + 4);
  S.ee_ty.ensure((size_t)nee + 1);
  S.ee_ov.ensure((size_t)nee + 1);
  W.bp_pt.ensure((size_t)npt + 1);
  W.bp_ee.ensure((size_t)nee + 1);
  if (npt) KLAUNCH(K_SH, s, k_decode_pt<<<nblk(npt, 256), 256, 0, s>>>(g, npt, W.pt_keys.p, S.pt.p, S.pt_ty.p, W.bp_pt.p));
  if (nee) KLAUNCH(K_SH, s, k_decode_ee<<<nblk(nee, 256), 256, 0, s>>>(g, nee, W.ee_keys.p, S.ee.p, S.ee_ty.p, W.bp_ee.p));
  // unique body pairs -> overlaps and the symmetric CSR
  long long nbp = (long long)npt + nee;
  int nov = 0;
  W.bp_all.ensure(sort_padded_size(nbp));
  W.flag.ensure((size_t)nbp + 1);
  W.pos.ensure((size_t)nbp + 1);
  if (nbp) {
    KLAUNCH(K_SH, s, k_bp_keys<<<nblk(nbp, 256), 256, 0, s>>>(npt, W.bp_pt.p, nee, W.bp_ee.p, W.bp_all.p));
    sort_u64(W.bp_all.p, nbp, W.bp_all.cap, s);
    KLAUNCH(K_SH, s, k_unique_flags<<<nblk(nbp, 256), 256, 0, s>>>(nbp, W.bp_all.p, W.flag.p));
    scan_exclusive_int(W.flag.p, W.pos.p, (int)nbp, W.pos.p + nbp, s, W.scan_i);
    CK(cudaMemcpyAsync(W.h_int, W.pos.p + nbp, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    nov = W.h_int[0];
  }
  S.nov = nov;
  S.ovI.ensure(nov + 1);
  S.ovJ.ensure(nov + 1);
  W.tkeys.ensure(sort_padded_size(nov));
  if (nov) {
    KLAUNCH(K_SH, s, k_unique_write<<<nblk(nbp, 256), 256, 0, s>>>(nbp, W.bp_all.p, W.flag.p, W.pos.p, S.ovI.p, S.ovJ.p,
                                                                  W.tkeys.p));
    sort_u64(W.tkeys.p, nov, W.tkeys.cap, s);
  }
  S.row_ptr.ensure(nb + 1);
  cs.cnt_all.ensure(nb + 1);
  KLAUNCH(K_SH, s, k_csr_count<<<nblk(nb, 256), 256, 0, s>>>(nb, nov, S.ovI.p, W.tkeys.p, cs.cnt_all.p));
  scan_exclusive_int(cs.cnt_all.p, S.row_ptr.p, nb, S.row_ptr.p + nb, s, W.scan_i);
  S.nnz = 2 * nov;
  S.col.ensure(S.nnz + 1);
  S.upidx.ensure(S.nnz + 1);
  KLAUNCH(K_SH, s, k_csr_fill<<<nblk(nb, 256), 256, 0, s>>>(nb, nov, S.ovI.p, S.ovJ.p, W.tkeys.p, S.row_ptr.p, S.col.p,
                                                            S.upidx.p));
  if (npt) KLAUNCH(K_SH, s, k_pair_ov<<<nblk(npt, 256), 256, 0, s>>>(npt, W.bp_pt.p, nov, S.ovI.p, S.ovJ.p, S.pt_ov.p));
  if (nee) KLAUNCH(K_SH, s, k_pair_ov<<<nblk(nee, 256), 256, 0, s>>>(nee, W.bp_ee.p, nov, S.ovI.p, S.ovJ.p, S.ee_ov.p));
  // vertex-ground pairs with the scaled threshold (col_set.cpp:49-63)
  Params Pg = P;
  Pg.dhat = Q.thr;
  vg_pairs(g, Pg, cs, S, s);
  CK(cudaStreamSynchronize(s));
}

// Lowers the per-scene keys to the earliest time of impact of the candidates of one kind.
template <int KIND>
static void sh_toi(const Geo& g, const ShParams& H, ShQuery& Q, ShScratch& W, CullScratch& cs, cudaStream_t s) {
  sh_prepare(g, H, KIND, 1, W, cs, Q, s);
  sh_run<KIND, true>(
      g, Q, W, s, [&]() { KLAUNCH(K_SH, s, k_sh_toi<KIND><<<1216, 128, 0, s>>>(g, Q, cs.toi_key.p)); },
      []() { return true; });
}

void sh_bound(const Geo& g, const Params& P, const ShParams& H, const PairSet& cur, ShScratch& W, CullScratch& cs,
              double* toi, cudaStream_t s) {
  launch_project(g, 2, 1.0, s);
  launch_project(g, 3, 0.0, s);
  const int nk = 2 * g.ns;
  cs.toi_key.ensure(nk);
  double one = 1.0;
  unsigned long long b1;
  memcpy(&b1, &one, sizeof(b1));
  KLAUNCH(K_SH, s, k_fill_key<<<nblk(nk, 256), 256, 0, s>>>(cs.toi_key.p, nk, b1 | 0x8000000000000000ull));
  if (H.full_ccd) {
    if (P.ground && g.nv) launch_vg_toi(g, P, cs.toi_key.p, s);
    ShQuery Q{};
    Q.G = grid_of(H);
    const bool do_pt = P.pt && g.nv && g.nf, do_ee = P.ee && g.ne;
    if (do_pt || do_ee) traj_floats(g, cs, s);
    if (do_pt) sh_toi<0>(g, H, Q, W, cs, s);
    if (do_ee) sh_toi<1>(g, H, Q, W, cs, s);
  } else {
    KLAUNCH(K_SH, s, k_norm1_bound<<<g.ns, 256, 0, s>>>(g.sc_beg, g.sc_end, g.dq, P.d_sqrt / 2.0, H.safe_factor,
                                                        cs.toi_key.p));
    if (cur.nvg) KLAUNCH(K_SH, s, k_vg_pair_toi<<<nblk(cur.nvg, 256), 256, 0, s>>>(g, P, cur.nvg, cur.vg.p, cs.toi_key.p + 1));
    long long np = (long long)cur.npt + cur.nee;
    if (np) KLAUNCH(K_SH, s, k_pair_toi<<<nblk(np, 128), 128, 0, s>>>(g, cur.npt, cur.pt.p, cur.nee, cur.ee.p, cs.toi_key.p));
  }
  if (!W.h_toi_cap || W.h_toi_cap < nk) {
    if (W.h_toi) CK(cudaFreeHost(W.h_toi));
    CK(cudaMallocHost(&W.h_toi, nk * sizeof(unsigned long long)));
    W.h_toi_cap = nk;
  }
  CK(cudaMemcpyAsync(W.h_toi, cs.toi_key.p, nk * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  for (int sc = 0; sc < g.ns; ++sc)
    toi[sc] = std::min(key_to_double_h(W.h_toi[2 * sc]), key_to_double_h(W.h_toi[2 * sc + 1]));
}

}  // namespace abd
