// Device parts of the adjoint of a converged frame that the Newton system does not
// already hold: the Jacobian of each point-triangle / edge-edge friction force through
// its tangent frame and multiplier (abd_fric_adj.cuh), its transposed product in body
// coordinates, and the vector kernels of the GMRES solve. Every reduction runs in a
// fixed order.
#include <cmath>

#include "abd_engine.h"
#include "abd_fric_adj.cuh"

namespace abd {
namespace {

inline int nblk_a(long long n, int t) { return (int)((n + t - 1) / t); }

__device__ __forceinline__ d3 ldXa(const double* X, int nv, int v) { return mk(X[v], X[nv + v], X[2 * nv + v]); }

__device__ __forceinline__ void pair_vids(const Geo& g, int kind, const int* tup, int p, int (&vid)[4], int& A,
                                          int& B) {
  A = tup[4 * p];
  B = tup[4 * p + 2];
  const int a = tup[4 * p + 1], b = tup[4 * p + 3];
  if (kind == 0) {
    vid[0] = g.v_off[A] + a;
    const int f = g.f_off[B] + b;
    vid[1] = g.fv[3 * f];
    vid[2] = g.fv[3 * f + 1];
    vid[3] = g.fv[3 * f + 2];
  } else {
    const int ea = g.e_off[A] + a, eb = g.e_off[B] + b;
    vid[0] = g.ev[2 * ea];
    vid[1] = g.ev[2 * ea + 1];
    vid[2] = g.ev[2 * eb];
    vid[3] = g.ev[2 * eb + 1];
  }
}

// Per pair: the 12 x 12 vertex-space Jacobian of its friction force through the frame
// and multiplier, row-major (J[12 r + c] = d g_r / d x_c); 0 for inactive pairs. A thread per
// column: a column is a chain of some 1000 dual-number operations, and a warp holds the columns
// of three pairs, so at most three distance types (the twelve columns of a pair one after the
// other by a thread, and the two kinds one after the other: 1757 us for 2 k pairs; now 89 us).
constexpr int JAC_T = 96;  // threads of k_fric_frame_jac, 8 pairs
__global__ void __launch_bounds__(JAC_T) k_fric_frame_jac(Geo g, Params P, int npt, int nee, const int* pt,
                                                          const int8_t* pt_ty, const int* ee, const int8_t* ee_ty,
                                                          double* Jpt, double* Jee) {
  const int cpt = (npt + JAC_T / 12 - 1) / (JAC_T / 12);  // CTAs of the point-triangle pairs
  const int kind = (int)blockIdx.x < cpt ? 0 : 1;
  const int p = ((int)blockIdx.x - (kind ? cpt : 0)) * (JAC_T / 12) + threadIdx.x / 12, c = threadIdx.x % 12;
  if (p >= (kind ? nee : npt)) return;
  double* Jp = (kind ? Jee : Jpt) + 144 * (size_t)p;
  int vid[4], A, B;
  pair_vids(g, kind, kind ? ee : pt, p, vid, A, B);
  d3 X[4], du[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    X[i] = ldXa(g.X, g.nv, vid[i]);
    du[i] = fsub(X[i], ldXa(g.X0, g.nv, vid[i]));
  }
  const int ty = (kind ? ee_ty : pt_ty)[p];
  const double d = kind == 0 ? pt_dist(X[0], X[1], X[2], X[3], ty) : ee_dist(X[0], X[1], X[2], X[3], ty);
  const bool on = d < P.dhat && P.mu > 0.0 && (kind == 0 ? (P.pt && P.pt_fric) : (P.ee && P.ee_fric));
  double col[12];
  if (on) {
    fadj::frame_jacobian_column(kind, ty, X, du, P.dhat, P.kappa, P.mu, P.epsv, c, col);
  } else {
#pragma unroll
    for (int r = 0; r < 12; ++r) col[r] = 0.0;
  }
#pragma unroll
  for (int r = 0; r < 12; ++r) Jp[12 * r + c] = col[r];
}

// Transpose of the ground-friction multiplier coupling: the lagged multiplier lam(y) =
// -2 b'(d) (y + off) of each vertex-ground pair moves with the vertex height at the solution,
// which adds C = (r_f / lam) (dlam/dy J_y)^T to the Jacobian of the gradient. Per pair, the two
// factors of the vertex's tangential displacement in C^T w (the same for every w); 0 where
// there is no coupling.
__global__ void k_vg_lag_coef(Geo g, Params P, int n, const int* vg, double2* coef) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int v = g.v_off[vg[2 * t]] + vg[2 * t + 1];
  const double y = g.X[g.nv + v] + P.ground_offset, dd = y * y;
  double2 o = make_double2(0.0, 0.0);
  if (dd < P.dhat) {
    BarrierP bp{P.dhat, P.kappa};
    const double b1 = barrier_b1(dd, bp), b2 = barrier_b2(dd, bp);
    const double lam = -b1 * 2 * y;
    if (lam != 0.0) {
      const double dlam = -2.0 * (2.0 * b2 * dd + b1);
      const double uk[2] = {g.X[v] - g.X0[v], g.X[2 * g.nv + v] - g.X0[2 * g.nv + v]};
      double gs = 0.0, M[2][2];
      friction_2x2(uk, lam, FrictionP{P.mu, P.epsv, P.max_uk}, gs, M);
      const double f = dlam * (gs / lam);
      o = make_double2(f * uk[0], f * uk[1]);
    }
  }
  coef[t] = o;
}

// Per pair: y = J^T (Jx w) in vertex space, returned in body space as the pair's
// contributions to its two bodies (12 each: p, a1, a2, a3 rows of Jx^T y). Vertices of
// static bodies do not move: their entries of Jx w are 0, and so are their bodies' rows.
// Twelve threads a pair, one per coordinate (a thread a pair, both kinds: 48 us for 2 k pairs,
// a chain of 300 operations; now 7 us).
constexpr int FFA_P = 16;  // pairs per CTA of k_fric_frame_apply
__global__ void __launch_bounds__(12 * FFA_P) k_fric_frame_apply(Geo g, int npt, int nee, const int* pt,
                                                                 const int* ee, const double* Jpt, const double* Jee,
                                                                 const double* w, double* cpt, double* cee) {
  __shared__ double sv[FFA_P][12], sy[FFA_P][12], sx[FFA_P][4][4];
  const int npc = (npt + FFA_P - 1) / FFA_P;  // CTAs of the point-triangle pairs
  const int kind = (int)blockIdx.x < npc ? 0 : 1, na = kind == 0 ? 1 : 2;
  const int q = threadIdx.x / 12, c = threadIdx.x % 12, i = c / 3, r = c % 3;
  const int p = ((int)blockIdx.x - (kind ? npc : 0)) * FFA_P + q;
  const bool in = p < (kind ? nee : npt);
  if (in) {
    int vid[4], A, B;
    pair_vids(g, kind, kind ? ee : pt, p, vid, A, B);
    const int b = i < na ? A : B, v = i == 0 ? vid[0] : (i == 1 ? vid[1] : (i == 2 ? vid[2] : vid[3]));
    double x[4] = {1.0, g.rest[3 * v], g.rest[3 * v + 1], g.rest[3 * v + 2]}, s = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s += x[k] * w[12 * b + 3 * k + r];
      if (r == 0) sx[q][i][k] = x[k];
    }
    sv[q][c] = g.mass[b] > 0.0 ? s : 0.0;
  }
  __syncthreads();
  if (in) {
    const double* Jp = (kind ? Jee : Jpt) + 144 * (size_t)p;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 12; ++k) s += Jp[12 * k + c] * sv[q][k];
    sy[q][c] = s;
  }
  __syncthreads();
  if (in) {
    double* out = (kind ? cee : cpt) + 24 * (size_t)p;  // row c = 3 i + r of either body
    double o[2] = {0.0, 0.0};
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j < na ? 0 : 1] += sx[q][j][i] * sy[q][3 * j + r];
    out[c] = o[0];
    out[12 + c] = o[1];
  }
}

// out = J^T z, a CTA per body and a warp per row: the body's diagonal block and the blocks of its
// overlaps (lanes over overlaps), the pairs' friction contributions (lanes over the pairs of one
// overlap after the other) and the vertex-ground coupling (lanes over the pairs; coef null: none).
// With threads over rows the loops over overlaps and pairs were chains of dependent loads: the
// product, the coupling, the gather and the additions of the parts 121 us for 64 bodies, now 16 us.
struct AdjApply {
  const int *row_ptr, *col, *upidx, *has;
  const double *ovr, *D;
  const int *pt_seg, *ee_seg, *pt, *ee;
  const double *cpt, *cee;
  const int *vg, *vg_seg;
  const double2* coef;
};
__global__ void __launch_bounds__(384) k_adj_apply(Geo g, AdjApply a, const double* z, double* out) {
  const int b = blockIdx.x, k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool dyn = g.mass[b] > 0.0;
  const double* zb = z + 12 * b;
  double s = lane < 12 ? a.D[144 * b + 12 * k + lane] * zb[lane] : 0.0;
  const int end = a.row_ptr[b + 1];
  for (int e0 = a.row_ptr[b]; e0 < end; e0 += 32) {
    const int e = e0 + lane, u = e < end ? a.upidx[e] : -1;
    int p0 = 0, p1 = 0, q0 = 0, q1 = 0;
    if (u >= 0 && dyn) {
      p0 = a.pt_seg[u];
      p1 = a.pt_seg[u + 1];
      q0 = a.ee_seg[u];
      q1 = a.ee_seg[u + 1];
    }
    if (u >= 0 && a.has[u]) {
      const int cb = a.col[e];
      const double* Bk = a.ovr + (size_t)u * CONTRIB + 288;
      const double* vc = z + 12 * cb;
      const int st = cb > b ? 1 : 12, at = cb > b ? 12 * k : k;
#pragma unroll
      for (int c = 0; c < 12; ++c) s += Bk[at + st * c] * vc[c];
    }
    unsigned m = __ballot_sync(0xffffffffu, p1 > p0 || q1 > q0);
    while (m) {
      const int l = __ffs(m) - 1;
      m &= m - 1;
      const int a0 = __shfl_sync(0xffffffffu, p0, l), a1 = __shfl_sync(0xffffffffu, p1, l);
      const int b0 = __shfl_sync(0xffffffffu, q0, l), b1 = __shfl_sync(0xffffffffu, q1, l);
      for (int p = a0 + lane; p < a1; p += 32) s += a.cpt[24 * (size_t)p + (a.pt[4 * p] == b ? 0 : 12) + k];
      for (int p = b0 + lane; p < b1; p += 32) s += a.cee[24 * (size_t)p + (a.ee[4 * p] == b ? 0 : 12) + k];
    }
  }
  if (a.coef && dyn && k % 3 == 1) {
    for (int j = a.vg_seg[b] + lane; j < a.vg_seg[b + 1]; j += 32) {
      const int v = g.v_off[b] + a.vg[2 * j + 1];
      const double xt[4] = {1.0, g.rest[3 * v], g.rest[3 * v + 1], g.rest[3 * v + 2]};
      double wx = 0.0, wz = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        wx += xt[i] * zb[3 * i];
        wz += xt[i] * zb[3 * i + 2];
      }
      const double2 f = a.coef[j];
      s += (k == 1 ? xt[0] : (k == 4 ? xt[1] : (k == 7 ? xt[2] : xt[3]))) * (f.x * wx + f.y * wz);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[12 * b + k] = s;
}

// Dot product by one CTA: thread t adds entries t, t + 1024, ... in order, then a fixed
// tree over the threads.
__global__ void __launch_bounds__(1024) k_dot(int n, const double* a, const double* b, double* out) {
  __shared__ double sh[1024];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 1024) s += a[i] * b[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = 512; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// Modified Gram-Schmidt of V_{k+1} against V_0 .. V_k by one CTA, the vector in registers:
// h[i] = V_{k+1} . V_i, subtracted before the next, h[k + 1] = the norm of the rest, by which it
// is divided. A dot, its host read and a subtraction a vector took some 25 us each; here a
// vector costs a reduction of 1.8 us (768 entries), and the host reads once. Eight warps while they hold
// the vector: one SM issues an FP64 instruction of a warp in 16 cycles, so the reductions of 24
// warps took 5 us a vector.
constexpr int MGS_R = 12;  // entries per thread, at most
__global__ void __launch_bounds__(1024) k_mgs(int n, int k, double* V, double* h) {
  __shared__ double sh[2][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nt = blockDim.x, nw = nt >> 5;
  double* vn = V + (size_t)(k + 1) * n;
  double v[MGS_R];
#pragma unroll
  for (int j = 0; j < MGS_R; ++j) {
    const int i = threadIdx.x + j * nt;
    v[j] = i < n ? vn[i] : 0.0;
  }
  int par = 0;
  auto total = [&](double s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) sh[par][w] = s;
    __syncthreads();
    s = sh[par][lane & (nw - 1)];  // nw: 8 or 32
    for (int o = nw >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    par ^= 1;  // read before the barrier of the next total
    return s;
  };
  for (int q = 0; q <= k; ++q) {
    const double* vq = V + (size_t)q * n;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < MGS_R; ++j) {
      if (j * nt >= n) break;
      const int i = threadIdx.x + j * nt;
      if (i < n) s += v[j] * vq[i];
    }
    s = total(s);
    if (threadIdx.x == 0) h[q] = s;
#pragma unroll
    for (int j = 0; j < MGS_R; ++j) {
      if (j * nt >= n) break;
      const int i = threadIdx.x + j * nt;
      if (i < n) v[j] -= s * vq[i];
    }
  }
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < MGS_R; ++j) {
    if (j * nt >= n) break;
    s += v[j] * v[j];
  }
  const double hn = sqrt(total(s)), f = hn > 0.0 ? 1.0 / hn : 1.0;
  if (threadIdx.x == 0) h[k + 1] = hn;
#pragma unroll
  for (int j = 0; j < MGS_R; ++j) {
    const int i = threadIdx.x + j * nt;
    if (i < n) vn[i] = v[j] * f;
  }
}

// y = a x + b y
__global__ void k_axpby(int n, double a, const double* x, double b, double* y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = a * x[i] + b * y[i];
}

}  // namespace

void adj_terms(const Geo& g, const Params& P, PairSet& S, NewtonBufs& B, bool vg_coupling, cudaStream_t s) {
  B.fj_pt.ensure(144 * (size_t)S.npt + 1);
  B.fj_ee.ensure(144 * (size_t)S.nee + 1);
  if (S.npt + S.nee)
    KLAUNCH(K_PAIR_TERMS, s, k_fric_frame_jac<<<nblk_a(S.npt, JAC_T / 12) + nblk_a(S.nee, JAC_T / 12), JAC_T, 0, s>>>(
                                 g, P, S.npt, S.nee, S.pt.p, S.pt_ty.p, S.ee.p, S.ee_ty.p, B.fj_pt.p, B.fj_ee.p));
  if (vg_coupling) {
    B.vg_coef.ensure(S.nvg);
    KLAUNCH(K_BODY_SYSTEM, s, k_vg_lag_coef<<<nblk_a(S.nvg, 64), 64, 0, s>>>(g, P, S.nvg, S.vg.p, B.vg_coef.p));
  }
}

void adj_apply(const Geo& g, PairSet& S, NewtonBufs& B, bool vg_coupling, const double* z, double* out,
               cudaStream_t s) {
  B.fc_pt.ensure(24 * (size_t)S.npt + 1);
  B.fc_ee.ensure(24 * (size_t)S.nee + 1);
  if (S.npt + S.nee)
    KLAUNCH(K_VEC, s, k_fric_frame_apply<<<nblk_a(S.npt, FFA_P) + nblk_a(S.nee, FFA_P), 12 * FFA_P, 0, s>>>(
                          g, S.npt, S.nee, S.pt.p, S.ee.p, B.fj_pt.p, B.fj_ee.p, z, B.fc_pt.p, B.fc_ee.p));
  AdjApply a{S.row_ptr.p, S.col.p,  S.upidx.p, B.has_ex.p, B.ovr_ex.p, B.D_ex.p, B.pt_seg.p, B.ee_seg.p, S.pt.p,
             S.ee.p,      B.fc_pt.p, B.fc_ee.p, S.vg.p,     S.vg_seg.p, vg_coupling ? B.vg_coef.p : nullptr};
  KLAUNCH(K_PCG, s, k_adj_apply<<<g.nb, 384, 0, s>>>(g, a, z, out));
}

static void pinned_h(NewtonBufs& B) {
  if (!B.h_dot) CK(cudaMallocHost(&B.h_dot, 64 * sizeof(double)));
}

void orthogonalize(int n, int k, double* V, double* h, NewtonBufs& B, cudaStream_t s) {
  if (n <= 1024 * MGS_R && k + 2 <= 64) {
    B.adj_h.ensure(64);
    pinned_h(B);
    const int nt = n <= 256 * MGS_R ? 256 : 1024;
    KLAUNCH(K_DOTS, s, k_mgs<<<1, nt, 0, s>>>(n, k, V, B.adj_h.p));
    CK(cudaMemcpyAsync(B.h_dot, B.adj_h.p, (k + 2) * sizeof(double), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    for (int i = 0; i < k + 2; ++i) h[i] = B.h_dot[i];
    return;
  }
  double* vn = V + (size_t)(k + 1) * n;
  for (int i = 0; i <= k; ++i) {
    h[i] = dev_dot(n, vn, V + (size_t)i * n, B, s);
    dev_axpby(n, -h[i], V + (size_t)i * n, 1.0, vn, s);
  }
  h[k + 1] = std::sqrt(dev_dot(n, vn, vn, B, s));
  if (h[k + 1] > 0.0) dev_axpby(n, 0.0, vn, 1.0 / h[k + 1], vn, s);
}

double dev_dot(int n, const double* a, const double* b, NewtonBufs& B, cudaStream_t s) {
  B.e_out.ensure(1);
  pinned_h(B);
  KLAUNCH(K_DOTS, s, k_dot<<<1, 1024, 0, s>>>(n, a, b, B.e_out.p));
  CK(cudaMemcpyAsync(B.h_dot, B.e_out.p, sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return *B.h_dot;
}

void dev_axpby(int n, double a, const double* x, double b, double* y, cudaStream_t s) {
  if (n > 0) KLAUNCH(K_VEC, s, k_axpby<<<nblk_a(n, 256), 256, 0, s>>>(n, a, x, b, y));
}

}  // namespace abd
