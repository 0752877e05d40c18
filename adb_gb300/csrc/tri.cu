// Direct solve of block-tridiagonal scenes (chains, stacks): the Newton matrix of a scene
// whose contacts only join consecutive bodies is block-tridiagonal in body order. The
// reference solves every Newton system with a sparse direct factorization (Pardiso LLT,
// model/abd.cpp:233-264); here it is a block Cholesky in odd-even (cyclic reduction) order.
// With i the body's place in its scene, counted from 1, the bodies whose i has l trailing
// zero bits are eliminated at level l, all of them at once: their neighbours still present
// are i - 2^l and i + 2^l. With the couplings U_- and U_+ to those,
//
//   S = D - sum over the neighbours eliminated at levels m < l of W^T W,   S = L L^T,
//   W_- = L^-1 U_-,  W_+ = L^-1 U_+,  y = L^-1 (b - sum of W^T y),
//
// a level l > 0 coupling being -W_-^T W_+ of the body half-way, and from the last level back
//   x = L^-T (y - W_- x_- - W_+ x_+).
//
// What bounds it: the dependent FP64 chain of one 12 x 12 factorization and the chain of
// loads before it. In body order a chain of n links is n of them, one after the other on one
// SM; by levels it is log2 n, at about twice the operations. Measured per solve, in body
// order and by levels: 200 links in contact 2.49 -> 0.17 ms, 256 columns (8212 bodies in all)
// 1.83 -> 0.42 ms, a stack of ten 0.117 -> 0.069 ms.
// Couplings that are absent (runs broken by missing contacts) are flagged and cost nothing.
// Every sum runs in a fixed order, and a body's arithmetic depends only on its own scene and
// its place there, so a scene gets the same solution in a batch as alone.
#include <cooperative_groups.h>

#include <vector>

#include "abd_engine.h"

namespace cg = cooperative_groups;

namespace abd {
namespace {

constexpr int TNT = 192;  // threads per body
constexpr int TWARPS = TNT / 32;

inline int nblk_t(long long n, int t) { return (int)((n + t - 1) / t); }

// Marks in bad[scene] the scenes with a block between bodies that are not consecutive, from
// the row-block copy of the system (k_pcg_rows: per body its diagonal block, then the
// neighbour blocks that hold a contribution).
__global__ void k_tri_mark(int nb, const int* row_ptr, const int* rcol, const int* rn, const int* bscene, int* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb) return;
  const int base = i + row_ptr[i], n = rn[i];
  bool far = false;
  for (int j = 1; j < n; ++j) {
    const int c = rcol[base + j];
    far |= c != i + 1 && c != i - 1;
  }
  if (far) atomicOr(&bad[bscene[i]], 1);
}

// Per scene: solved directly (tri_on) or by the CG (pcg_on); cnt[0] / cnt[1] count them.
__global__ void k_tri_masks(int ns, int enable, const int* sc_on, const int* bad, int* tri_on, int* pcg_on, int* cnt) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ns) return;
  const int on = sc_on[k] != 0;
  const int t = enable && on && !bad[k];
  tri_on[k] = t;
  pcg_on[k] = on && !t;
  if (t) atomicAdd(&cnt[1], 1);
  if (on && !t) atomicAdd(&cnt[0], 1);
}

struct TriArgs {
  const int *row_ptr, *rcol, *rn;
  const double* Hrow;
  const int *bscene, *sc_end, *sc_on, *tri_on;
  const double* b;
  double *Li, *W, *y;  // per body: inverse of the factor's diagonal block, the two coupling blocks
                       // (towards lower and higher bodies), forward solution
  double *x, *dq;
  int* fl;             // per body: bit 0 / 1 = coupled to a lower / higher body when eliminated
  const int *lv_body, *lv_off;  // bodies by level (lv_off: nlev + 1)
  int nlev;
  int* status;
};

// Pivot of a right-looking Cholesky: r = 1 / sqrt(a), d = r^2. A non-positive pivot sets
// ABD_ERR_NOT_SPD and is replaced by 1e-300, as the block-Jacobi preconditioner does.
__device__ __forceinline__ void tri_pivot(double a, double* r, double* d, int* status) {
  if (!(a > 0)) {
    atomicExch(status, (int)ABD_ERR_NOT_SPD);
    a = 1e-300;
  }
  const double q = rsqrt(a);
  *r = q;
  *d = q * q;
}

// acc += sum over r of P[r][i] Q[r], Q read with stride qs (a column of a 12 x 12 block: 12,
// a vector: 1).
__device__ __forceinline__ double tri_dot_t(const double* P, int i, const double* Q, int qs, double acc) {
#pragma unroll
  for (int r = 0; r < 12; ++r) acc += P[12 * r + i] * Q[qs * r];
  return acc;
}

// One cooperative launch: the levels of the elimination in order with a grid barrier after
// each, then the back substitution from the last level to the first. A CTA eliminates one
// body at a time.
//
// An FP64 instruction of a warp takes 64 cycles of its quarter of the SM however many lanes
// are active, so the 12 x 12 work is laid out for few warp instructions: six warps, the
// lower triangles packed. Warps 0-2: the 78 entries of the body's Schur complement and the
// right-hand side, then the right-looking factor, an entry kept in its thread's register and
// put in shared memory when its column is next (the thread that updates the next pivot takes
// its reciprocal square root). Warps 3-5: the two coupling blocks, then L^-1, row c formed one
// column behind the factor from the rows above (T holds I minus their contributions). Then
// each warp forms two rows of L^-1 [U_lower U_upper b], a short and a long one. A batch of
// columns (128 bodies in the deepest) 622 -> 418 us, a chain of 200 256 -> 174 us against
// five warps with a thread per entry of the square.
__global__ void __launch_bounds__(TNT, 5) k_tri_solve(TriArgs a) {
  cg::grid_group grid = cg::this_grid();
  __shared__ double sA[12][13], sL[12][13], sT[12][13], sLi[12][13], sU[2][12][13];
  __shared__ double st[12], sR[12], sD[12];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const bool fac = t < 96;               // else: couplings and L^-1
  const int q = fac ? t : t - 96;        // entry (ei, ej) of a lower triangle; 78..89: rhs
  int ei = 0;
  while ((ei + 1) * (ei + 2) / 2 <= q) ++ei;
  const int ej = q - ei * (ei + 1) / 2;
  const bool ent = q < 78, rhs = fac && q >= 78 && q < 90;
  const int ri = q - 78;                 // row of the right-hand side
  for (int l = 0; l < a.nlev; ++l) {
    const int h = 1 << l, hh = h >> 1;
    for (int it = a.lv_off[l] + blockIdx.x; it < a.lv_off[l + 1]; it += gridDim.x) {
      const int k = a.lv_body[it];
      const int sc = a.bscene[k];
      if (!a.sc_on[sc] || !a.tri_on[sc]) continue;
      const int end = a.sc_end[sc];
      const int base = k + a.row_ptr[k];
      // the two couplings: blocks of the matrix at level 0, else minus the product of the
      // two coupling blocks of the body half-way (eliminated one level earlier)
      int cl = 0, cr = 0;  // coupled; at level 0 the slot of the block in k's row list
      if (l == 0) {
        const int n = a.rn[k];
        for (int j = 1; j < n; ++j) {
          const int c = a.rcol[base + j];
          if (c == k - 1) cl = base + j;
          if (c == k + 1) cr = base + j;
        }
      } else {
        cl = a.fl[k - hh] == 3;
        cr = k + hh < end && a.fl[k + hh] == 3;
      }
      double v = 0.0, u[3] = {0.0, 0.0, 0.0};
      if (fac) {
        // the Schur complement: the bodies eliminated next to this one at the earlier levels
        if (ent || rhs) {
          const double* Hd = a.Hrow + (size_t)base * 144;
          v = ent ? 0.5 * (Hd[12 * ei + ej] + Hd[12 * ej + ei]) : a.b[12 * k + ri];
          const int i = ent ? ei : ri;
          double accl = 0.0, accr = 0.0;
          for (int m = 0; m < l; ++m) {
            const int kl = k - (1 << m), kr = k + (1 << m);
            if (a.fl[kl] & 2) {
              const double* Wr = a.W + (size_t)288 * kl + 144;
              accl = tri_dot_t(Wr, i, ent ? Wr + ej : a.y + 12 * kl, ent ? 12 : 1, accl);
            }
            if (kr < end && (a.fl[kr] & 1)) {
              const double* Wl = a.W + (size_t)288 * kr;
              accr = tri_dot_t(Wl, i, ent ? Wl + ej : a.y + 12 * kr, ent ? 12 : 1, accr);
            }
          }
          v -= accl + accr;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int e = q + 96 * j, side = e / 144, x = e - 144 * side;
          const int c = side ? cr : cl;
          if (!c) continue;
          if (l == 0) {
            u[j] = a.Hrow[(size_t)c * 144 + x];
          } else {
            const double* Wm = a.W + (size_t)288 * (side ? k + hh : k - hh);
            u[j] = -tri_dot_t(Wm + (side ? 0 : 144), x / 12, Wm + (side ? 144 : 0) + x % 12, 12, 0.0);
          }
        }
      }
      __syncthreads();  // the previous body's shared blocks are no longer read
      if (fac) {
        if (ent && ej == 0) sA[ei][0] = v;
        if (rhs) st[ri] = v;
        if (t == 0) tri_pivot(v, &sR[0], &sD[0], a.status);
      } else {
        if (ent) sT[ei][ej] = ei == ej ? 1.0 : 0.0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int e = q + 96 * j, side = e / 144, x = e - 144 * side;
          sU[side][x / 12][x % 12] = u[j];
        }
        v = ei == ej ? 1.0 : 0.0;  // this thread's entry of T
      }
      __syncthreads();
      for (int c = 0; c <= 12; ++c) {
        if (ent && fac) {
          if (c < 12 && ej >= c) {
            if (ej == c) {
              if (ei > c) sL[ei][c] = v * sR[c];
            } else {
              v -= (sA[ei][c] * sD[c]) * sA[ej][c];
              if (ej == c + 1) sA[ei][ej] = v;
              if (ei == c + 1 && ej == c + 1) tri_pivot(v, &sR[c + 1], &sD[c + 1], a.status);
            }
          }
        } else if (ent && c >= 1 && ej < c && ei >= c - 1) {
          const int rw = c - 1;
          const double li = sT[rw][ej] * sR[rw];
          if (ei == rw) {
            sLi[rw][ej] = li;
            a.Li[(size_t)144 * k + 12 * rw + ej] = li;
          } else {
            v -= sL[ei][rw] * li;
            if (ei == c) sT[ei][ej] = v;
          }
        }
        __syncthreads();
      }
      // y = L^-1 rhs, W = L^-1 U for both couplings (L^-1 lower triangular): rows w and 11 - w
      if (lane < 25 && (lane == 24 || (lane < 12 ? cl : cr))) {
        const int side = lane / 12, col = lane - 12 * side;  // lane 24: the right-hand side
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const int row = z ? 11 - w : w;
          double s = 0.0;
          for (int m = 0; m <= row; ++m) s += sLi[row][m] * (lane == 24 ? st[m] : sU[side][m][col]);
          if (lane == 24) a.y[12 * k + row] = s;
          else a.W[(size_t)288 * k + 144 * side + 12 * row + col] = s;
        }
      }
      if (fac && ent && ei > ej) a.Li[(size_t)144 * k + 12 * ej + ei] = 0.0;
      if (t == 0) a.fl[k] = (cl ? 1 : 0) | (cr ? 2 : 0);
    }
    grid.sync();
  }
  // back substitution, one warp per body: lanes 0..11 the rows' lower coupling, lanes
  // 16..27 the upper one, then x = L^-T v with the even terms on the low half, the odd ones
  // on the high half. Bodies of scenes that take no step get x = 0, dq = -0.
  const int row = lane & 15, side = lane >> 4;
  const bool rl = row < 12;
  for (int l = a.nlev - 1; l >= 0; --l) {
    const int h = 1 << l;
    for (int it = a.lv_off[l] + blockIdx.x * TWARPS + w; it < a.lv_off[l + 1]; it += gridDim.x * TWARPS) {
      const int k = a.lv_body[it];
      const int sc = a.bscene[k];
      if (!a.sc_on[sc]) {
        if (lane < 12) {
          a.x[12 * k + lane] = 0.0;
          a.dq[12 * k + lane] = -0.0;
        }
        continue;
      }
      if (!a.tri_on[sc]) continue;
      double v = rl && side == 0 ? a.y[12 * k + row] : 0.0;
      const int f = a.fl[k];
      if (rl && (f & (1 << side))) {
        const double* W = a.W + (size_t)288 * k + 144 * side + 12 * row;
        const double* xn = a.x + 12 * (side ? k + h : k - h);
#pragma unroll
        for (int m = 0; m < 12; ++m) v -= W[m] * xn[m];
      }
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      const double* Li = a.Li + (size_t)144 * k;
      double xv = 0.0;
#pragma unroll
      for (int m = 0; m < 12; m += 2) {
        const double vm = __shfl_sync(0xffffffffu, v, m + side);
        if (rl) xv += Li[12 * (m + side) + row] * vm;
      }
      xv += __shfl_xor_sync(0xffffffffu, xv, 16);
      if (lane < 12) {
        a.x[12 * k + lane] = xv;
        a.dq[12 * k + lane] = -xv;
      }
    }
    if (l > 0) grid.sync();
  }
}

}  // namespace

void tri_classify(const Geo& g, PairSet& S, NewtonBufs& B, int enable, const int* sc_on, cudaStream_t s,
                  int* n_pcg, int* n_tri) {
  const int nb = g.nb, ns = g.ns;
  B.tri_bad.ensure(ns);
  B.tri_on.ensure(ns);
  B.pcg_on.ensure(ns);
  B.tri_cnt.ensure(2);
  CK(cudaMemsetAsync(B.tri_bad.p, 0, ns * sizeof(int), s));
  CK(cudaMemsetAsync(B.tri_cnt.p, 0, 2 * sizeof(int), s));
  KLAUNCH(K_BLOCK_INVERSE, s, k_tri_mark<<<nblk_t(nb, 256), 256, 0, s>>>(nb, S.row_ptr.p, B.rcol.p, B.rn.p, g.bscene,
                                                                       B.tri_bad.p));
  KLAUNCH(K_BLOCK_INVERSE, s, k_tri_masks<<<nblk_t(ns, 256), 256, 0, s>>>(ns, enable, sc_on, B.tri_bad.p, B.tri_on.p,
                                                                        B.pcg_on.p, B.tri_cnt.p));
  CK(cudaMemcpyAsync(B.h_int + 8, B.tri_cnt.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  *n_pcg = B.h_int[8];
  *n_tri = B.h_int[9];
}

void tri_levels(const std::vector<int>& sc_beg, const std::vector<int>& sc_end, NewtonBufs& B, cudaStream_t s) {
  std::vector<std::vector<int>> lv;
  for (size_t k = 0; k < sc_beg.size(); ++k)
    for (int b = sc_beg[k]; b < sc_end[k]; ++b) {
      size_t l = 0;
      for (unsigned i = (unsigned)(b - sc_beg[k]) + 1u; !(i & 1u); i >>= 1) ++l;
      if (lv.size() <= l) lv.resize(l + 1);
      lv[l].push_back(b);
    }
  std::vector<int> body, off{0};
  for (auto& v : lv) {
    body.insert(body.end(), v.begin(), v.end());
    off.push_back((int)body.size());
  }
  B.tri_nlev = (int)lv.size();
  B.tri_width = lv.empty() ? 0 : (int)lv[0].size();
  B.tri_lv_body.ensure(body.size() + 1);
  B.tri_lv_off.ensure(off.size());
  if (!body.empty())
    CK(cudaMemcpyAsync(B.tri_lv_body.p, body.data(), body.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(B.tri_lv_off.p, off.data(), off.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  CK(cudaStreamSynchronize(s));
}

void tri_solve(const Geo& g, PairSet& S, NewtonBufs& B, const int* sc_on, double* dq, cudaStream_t s) {
  const int nb = g.nb;
  B.tri_Li.ensure(144 * (size_t)nb);
  B.tri_W.ensure(288 * (size_t)nb);
  B.tri_y.ensure(12 * (size_t)nb);
  B.tri_fl.ensure(nb);
  static int max_blocks = 0;
  if (!max_blocks) {
    int dev, sms, per;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_tri_solve, TNT, 0));
    max_blocks = sms * (per > 0 ? per : 1);
  }
  TriArgs a{S.row_ptr.p, B.rcol.p,   B.rn.p,  B.Hrow.p,        g.bscene,       g.sc_end,
            sc_on,       B.tri_on.p, B.grad.p, B.tri_Li.p,     B.tri_W.p,      B.tri_y.p,  B.x.p,
            dq,          B.tri_fl.p, B.tri_lv_body.p, B.tri_lv_off.p, B.tri_nlev, B.status.p};
  void* args[] = {&a};
  const int grid = B.tri_width < max_blocks ? B.tri_width : max_blocks;
  KLAUNCH(K_PCG, s, CK(cudaLaunchCooperativeKernel((void*)k_tri_solve, dim3(grid), dim3(TNT), args, 0, s)));
  // per body: its diagonal and coupling blocks read, the factor's blocks written and read
  // back (6 x 1152 B), the right-hand side, y and x
  prof_work(K_PCG, 1, 8.0 * 1152.0 * nb);
}

}  // namespace abd
