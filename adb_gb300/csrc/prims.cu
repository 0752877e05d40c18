// Batched per-primitive entry points mirroring the reference's python module `abdtk`
// (python/bindings.cpp:42-83: ipc_hess_pt_12x12, ipc_hess_ee_12x12, pt_collision_time,
// ee_collision_time), evaluated on the GPU with the same device code as the step, and
// the FP64 throughput probe used as the roofline denominator of FP64-bound kernels.
#include <algorithm>
#include <vector>

#include "abd_ccd_filter.cuh"
#include "abd_engine.h"
#include "abd_ipc.cuh"
#include "batch_pool.h"

namespace abd {
namespace {

__device__ __forceinline__ d3 ld12(const double* x, int i) { return mk(x[3 * i], x[3 * i + 1], x[3 * i + 2]); }

__global__ void k_distance(int kind, int n, const double* x, int* type, double* dist) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* p = x + 12 * i;
  d3 a = ld12(p, 0), b = ld12(p, 1), c = ld12(p, 2), d = ld12(p, 3);
  int ty = kind == 0 ? pt_type(a, b, c, d) : ee_type(a, b, c, d);
  type[i] = ty;
  dist[i] = kind == 0 ? pt_dist(a, b, c, d, ty) : ee_dist(a, b, c, d, ty);
}

// Vertex-space Hessians H = (Q (x) I) S (Q (x) I)^T and gradients of n stencils, `per` to a CTA.
// The stencils of a CTA are taken by parameter count (0, 1, 2: the size of their projection),
// each count from a warp's first lane on, so that a warp runs one of the three; mollified
// edge-edge stencils (a 9 x 9 projection) wait in a list and take a warp each afterwards.
// Bound by FP64 issue. 20011 edge-edge stencils, one in twenty mollified: 2.62 ms a launch
// with a thread each (every warp waited for a serial 9 x 9 Jacobi in local memory, and H took
// 27 products an entry instead of 6) -> 0.50 ms. (One queue of chunks and mollified stencils per CTA
// was slower, 0.58: the warps then wait for the longest item twice.)
constexpr int HESS_BT = 128, HESS_PER = 128;  // threads, most stencils of a CTA
struct HessArgs {
  int n, per, psd;
  const double* x;
  const int* type;
  const double* dist;
  BarrierP bp;
  double eps_x;
  double *H, *g, *moll;
};
template <int KIND>
__device__ __forceinline__ void hess_load(const HessArgs& a, int i, d3 (&X)[4], int& ty, double& d) {
  const double* p = a.x + 12 * (size_t)i;
#pragma unroll
  for (int k = 0; k < 4; ++k) X[k] = ld12(p, k);
  ty = a.type ? a.type[i] : -1;
  const bool given = a.dist && ty >= 0;
  if (ty < 0) ty = KIND == 0 ? pt_type(X[0], X[1], X[2], X[3]) : ee_type(X[0], X[1], X[2], X[3]);
  d = given ? a.dist[i] : (KIND == 0 ? pt_dist(X[0], X[1], X[2], X[3], ty) : ee_dist(X[0], X[1], X[2], X[3], ty));
}
__device__ __forceinline__ void hess_gradient(const HessArgs& a, int i, const d3* gv) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    a.g[12 * (size_t)i + 3 * k] = gv[k].x;
    a.g[12 * (size_t)i + 3 * k + 1] = gv[k].y;
    a.g[12 * (size_t)i + 3 * k + 2] = gv[k].z;
  }
}
template <int KIND>
__global__ void __launch_bounds__(HESS_BT) k_hess(HessArgs a) {
  __shared__ int s_cnt[3], s_list[3][HESS_PER], s_moll[HESS_PER], s_nm;
  __shared__ Jac9 sj[KIND ? HESS_BT / 32 : 1];
  __shared__ MollData smd[KIND ? HESS_BT / 32 : 1];
  const int beg = blockIdx.x * a.per, end = min(a.n, beg + a.per);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 3) s_cnt[threadIdx.x] = 0;
  if (threadIdx.x == 3) s_nm = 0;
  __syncthreads();
  for (int i = beg + threadIdx.x; i < end; i += HESS_BT) {
    d3 X[4];
    int ty = a.type ? a.type[i] : -1;
    if (ty < 0) {
      double d;
      hess_load<KIND>(a, i, X, ty, d);
    }
    const int m = KIND == 0 ? (ty < P_E0 ? 0 : (ty < P_T ? 1 : 2)) : (ty < EA_EB0 ? 0 : (ty < EA_EB ? 1 : 2));
    s_list[m][atomicAdd(&s_cnt[m], 1)] = i;
  }
  __syncthreads();
  // slots: the three lists, each padded to whole warps
  const int w0 = (s_cnt[0] + 31) >> 5, w1 = (s_cnt[1] + 31) >> 5, w2 = (s_cnt[2] + 31) >> 5;
  for (int c = warp; c < w0 + w1 + w2; c += HESS_BT / 32) {
    const int m = c < w2 ? 2 : (c < w2 + w1 ? 1 : 0);  // the largest projections first
    const int at = 32 * (c - (m == 2 ? 0 : (m == 1 ? w2 : w2 + w1))) + lane;
    if (at < s_cnt[m]) {
      const int i = s_list[m][at];
      d3 X[4], gv[4];
      int ty;
      double d;
      hess_load<KIND>(a, i, X, ty, d);
      Stencil st;
      d3 w, W[2], gu, gw;
      double Gi[2][2];
      MollData md;
      if (pair_setup(KIND, ty, X, d, a.bp, a.eps_x, st, w, W, Gi, md, gu, gw)) {
        s_moll[atomicAdd(&s_nm, 1)] = i;
      } else {
        S9Reg S;
        if (m == 2) reduced_project<2, true>(st, w, W, Gi, md.B1, md.B2, a.psd != 0, S);
        else if (m == 1) reduced_project<1, true>(st, w, W, Gi, md.B1, md.B2, a.psd != 0, S);
        else reduced_project<0, true>(st, w, W, Gi, md.B1, md.B2, a.psd != 0, S);
        double* H = a.H + 144 * (size_t)i;
#pragma unroll
        for (int e = 0; e < 144; ++e) {
          const int row = e / 12, col = e % 12;
          if (row > col) continue;
          const double v =
              vertex_entry(row / 3, col / 3, row % 3, col % 3, [&](int p, int q) { return s9_get(S, p, q); });
          H[12 * row + col] = v;
          if (row != col) H[12 * col + row] = v;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) gv[k] = fscl(md.B1 * 2 * st.c[k], w);
        hess_gradient(a, i, gv);
        if (KIND && a.moll) a.moll[i] = 1.0;
      }
    }
  }
  if (KIND == 0) return;
  __syncthreads();
  for (int t = warp; t < s_nm; t += HESS_BT / 32) {
    const int i = s_moll[t];
    d3 X[4], gv[4];
    int ty;
    double d;
    hess_load<KIND>(a, i, X, ty, d);
    Stencil st;
    d3 w, W[2], gu, gw;
    double Gi[2][2];
    MollData md;
    const bool moll = pair_setup(1, ty, X, d, a.bp, a.eps_x, st, w, W, Gi, md, gu, gw);
    Jac9& w9 = sj[KIND ? warp : 0];
    __syncwarp();
    if (lane == 0) {
      smd[KIND ? warp : 0] = md;
      if (!moll) {  // compiled apart, the two tests could differ at the very edge
        double S[9][9];
        if (st.m == 0) reduced_project<0, true>(st, w, W, Gi, md.B1, md.B2, a.psd != 0, S);
        else if (st.m == 1) reduced_project<1, true>(st, w, W, Gi, md.B1, md.B2, a.psd != 0, S);
        else reduced_project<2, true>(st, w, W, Gi, md.B1, md.B2, a.psd != 0, S);
        for (int e = 0; e < 81; ++e) w9.S[e / 9][e % 9] = S[e / 9][e % 9];
      }
    }
    __syncwarp();
    bool neg = false;
    int cur = 0;
    if (moll) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int e = lane + 32 * j;
        if (e < 81) {
          const int p = e / 9, q = e % 9;
          w9.S[p][q] = moll_entry(smd[KIND ? warp : 0], p <= q ? p : q, p <= q ? q : p);
        }
      }
      __syncwarp();
      if (a.psd) {
        cur = jac9_project(w9, neg);
        if (neg) {
          double v[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            if (k == 1 && lane >= 13) continue;
            int p, q;
            jac9_tri(lane + 32 * k, p, q);
            v[k] = jac9_entry(w9, cur, neg, p, q);
          }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            if (k == 1 && lane >= 13) continue;
            int p, q;
            jac9_tri(lane + 32 * k, p, q);
            w9.S[p][q] = v[k];
            w9.S[q][p] = v[k];
          }
        }
      }
      __syncwarp();
    }
    for (int e = lane; e < 144; e += 32) {
      const int row = e / 12, col = e % 12;
      a.H[144 * (size_t)i + e] =
          vertex_entry(row / 3, col / 3, row % 3, col % 3, [&](int p, int q) { return w9.S[p][q]; });
    }
    if (lane == 0) {
      pair_gradient(st, w, md, gu, gw, gv);
      hess_gradient(a, i, gv);
      if (a.moll) a.moll[i] = md.mol;
    }
    __syncwarp();
  }
}

constexpr int TOI_THREADS = 128;
template <int KIND>
__global__ void __launch_bounds__(TOI_THREADS, 3) k_toi(int n, const double* x, double* toi) {
  __shared__ int queue[TOI_THREADS / 32][64];
  toi_stream<KIND>(n, x, toi, queue[threadIdx.x >> 5], [](double) {});
}

// Independent FMA chains; result stored per thread so nothing is optimised away.
__global__ void k_fma64(double* out, int iters, double a, double b) {
  int tid = blockIdx.x * blockDim.x + threadIdx.x;
  double x0 = tid * 1e-7, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  out[tid] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}

template <typename T>
struct DevArr {
  BatchBuf b;
  T* p;
  bool done = false;  // the call's work on it has ended
  explicit DevArr(size_t n) : b(batch_take((n ? n : 1) * sizeof(T))), p(static_cast<T*>(b.p)) {}
  DevArr(const DevArr&) = delete;
  DevArr& operator=(const DevArr&) = delete;
  ~DevArr() { batch_give(b, done); }
};

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

std::string g_prim_err;

template <typename F>
int guard(F&& f) {
  try {
    f();
    return ABD_OK;
  } catch (const CudaError& e) {
    g_prim_err = std::string(e.where) + ": " + cudaGetErrorString(e.code);
    return ABD_ERR_CUDA;
  }
}

int hess_batch(int kind, int n, const double* x, const int* type, const double* dist, double dhat, double kappa,
               double eps_x, int psd, double* H, double* g, double* moll) {
  if (n < 0 || !x || !H || !g) return ABD_ERR_INVALID;
  if (n == 0) return ABD_OK;
  return guard([&]() {
    // one allocation: x, H, g, dist, mollifier, then the types
    const size_t N = n;
    DevArr<double> buf((12 + 144 + 12 + 2) * N + (N + 1) / 2);
    double *dx = buf.p, *dH = dx + 12 * N, *dg = dH + 144 * N, *dd = dg + 12 * N, *dm = dd + N;
    int* dt = reinterpret_cast<int*>(dm + N);
    CK(cudaMemcpy(dx, x, 12 * N * sizeof(double), cudaMemcpyHostToDevice));
    if (type) CK(cudaMemcpy(dt, type, N * sizeof(int), cudaMemcpyHostToDevice));
    if (dist) CK(cudaMemcpy(dd, dist, N * sizeof(double), cudaMemcpyHostToDevice));
    HessArgs a{n, 0, psd, dx, type ? dt : nullptr, dist ? dd : nullptr, BarrierP{dhat, kappa}, eps_x, dH, dg,
               moll ? dm : nullptr};
    // two CTAs an SM while that leaves a warp of stencils each, then fuller ones
    a.per = std::min(HESS_PER, std::max(32, nblk(n, 2 * 152)));
    if (kind == 0) k_hess<0><<<nblk(n, a.per), HESS_BT>>>(a);
    else k_hess<1><<<nblk(n, a.per), HESS_BT>>>(a);
    CK(cudaGetLastError());
    CK(cudaMemcpy(H, dH, 144 * N * sizeof(double), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(g, dg, 12 * N * sizeof(double), cudaMemcpyDeviceToHost));
    if (moll) CK(cudaMemcpy(moll, dm, N * sizeof(double), cudaMemcpyDeviceToHost));
    buf.done = true;
  });
}

int toi_batch(int kind, int n, const double* x, double* toi) {
  if (n < 0 || !x || !toi) return ABD_ERR_INVALID;
  if (n == 0) return ABD_OK;
  return guard([&]() {
    DevArr<double> dx(24 * (size_t)n), dt(n);
    CK(cudaMemcpy(dx.p, x, 24 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
    const int blocks = toi_blocks(n, TOI_THREADS, 3);
    if (kind == 0) k_toi<0><<<blocks, TOI_THREADS>>>(n, dx.p, dt.p);
    else k_toi<1><<<blocks, TOI_THREADS>>>(n, dx.p, dt.p);
    CK(cudaGetLastError());
    CK(cudaMemcpy(toi, dt.p, n * sizeof(double), cudaMemcpyDeviceToHost));
    dx.done = dt.done = true;
  });
}

int dist_batch(int kind, int n, const double* x, int* type, double* dist) {
  if (n < 0 || !x || !type || !dist) return ABD_ERR_INVALID;
  if (n == 0) return ABD_OK;
  return guard([&]() {
    DevArr<double> dx(12 * (size_t)n), dd(n);
    DevArr<int> dt(n);
    CK(cudaMemcpy(dx.p, x, 12 * (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
    k_distance<<<nblk(n, 128), 128>>>(kind, n, dx.p, dt.p, dd.p);
    CK(cudaGetLastError());
    CK(cudaMemcpy(type, dt.p, n * sizeof(int), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(dist, dd.p, n * sizeof(double), cudaMemcpyDeviceToHost));
    dx.done = dd.done = dt.done = true;
  });
}

}  // namespace

double measure_fp64_gflops() {
  int dev, sms;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int blocks = sms * 8, threads = 256, n = blocks * threads, iters = 2048;
  DevArr<double> out(n);
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  float best = 1e30f;
  for (int rep = 0; rep < 4; ++rep) {
    CK(cudaEventRecord(e0));
    k_fma64<<<blocks, threads>>>(out.p, iters, 0.999999, 1e-9);
    CK(cudaEventRecord(e1));
    CK(cudaEventSynchronize(e1));
    float ms;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    if (rep > 0 && ms < best) best = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return 2.0 * 8.0 * iters * (double)n / (best * 1e-3) / 1e9;
}

}  // namespace abd

extern "C" {

int abd_ipc_hess_pt_batch(int n, const double* x, const int* type, const double* dist, double dhat, double kappa,
                          int psd, double* H, double* g) {
  return abd::hess_batch(0, n, x, type, dist, dhat, kappa, 0.0, psd, H, g, nullptr);
}
int abd_ipc_hess_ee_batch(int n, const double* x, const int* type, const double* dist, double dhat, double kappa,
                          double eps_x, int psd, double* H, double* g, double* mollifier) {
  return abd::hess_batch(1, n, x, type, dist, dhat, kappa, eps_x, psd, H, g, mollifier);
}
int abd_pt_collision_time_batch(int n, const double* x, double* toi) { return abd::toi_batch(0, n, x, toi); }
int abd_ee_collision_time_batch(int n, const double* x, double* toi) { return abd::toi_batch(1, n, x, toi); }
int abd_pt_distance_batch(int n, const double* x, int* type, double* dist) {
  return abd::dist_batch(0, n, x, type, dist);
}
int abd_ee_distance_batch(int n, const double* x, int* type, double* dist) {
  return abd::dist_batch(1, n, x, type, dist);
}
double abd_measure_fp64_gflops(void) {
  try {
    return abd::measure_fp64_gflops();
  } catch (...) {
    return -1.0;
  }
}

}  // extern "C"
