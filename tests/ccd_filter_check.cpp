// CPU check of the FP32 certificates (abd_ccd_filter.cuh) against the FP64 test: a certified
// candidate has a time of impact of exactly 1, and the test whose roots are verified in FP32
// where that is certain gives the same time. Prints the number of contradictions and the
// share certified, per kind of configuration.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../adb_gb300/csrc/abd_ccd_filter.cuh"
using namespace abd;

static f3 tf(d3 a) { return f3{(float)a.x, (float)a.y, (float)a.z}; }

int main(int argc, char** argv) {
  std::mt19937_64 g(argc > 1 ? atoi(argv[1]) : 1);
  std::uniform_real_distribution<double> U(-1, 1);
  std::normal_distribution<double> N;
  // primitive size, distance, motion, distance from the origin
  const double forms[][4] = {{0.08, 0.1, 0.01, 10},  {0.08, 0.02, 0.01, 10}, {0.08, 0.5, 0.01, 10}, {0.08, 0.1, 0.2, 10},
                             {0.08, 0.02, 0.2, 0},   {1.0, 0.5, 0.5, 1},     {0.08, 0.1, 0.01, 300}, {1e-3, 1e-3, 1e-3, 1},
                             {30.0, 20.0, 5.0, 1000}};
  long bad = 0;
  for (auto& f : forms) {
    const double L = f[0], D = f[1], mv = f[2], off = f[3];
    long cert[2] = {0, 0}, hit[2] = {0, 0};
    const long n = 60000;
    for (long i = 0; i < n; ++i) {
      const d3 o = mk(off * U(g), off * U(g), off * U(g));
      const int form = i % 6;  // 0-2 general, 3 lattice, 4 planar lattice, 5 slivers
      d3 q[4], dd = mk(D * U(g), D * U(g), D * U(g));
      if (form == 3 || form == 4) dd = mk(D * std::round(2 * U(g)), form == 4 ? 0.0 : D * std::round(2 * U(g)), 0.0);
      for (int k = 0; k < 4; ++k) {
        q[k] = mk(o.x + L * U(g), o.y + L * U(g), o.z + L * U(g));
        if (form == 3) q[k] = mk(o.x + L * std::round(2 * U(g)), o.y + L * std::round(2 * U(g)), o.z + L * std::round(U(g)));
        if (form == 4) q[k] = mk(o.x + L * std::round(2 * U(g)), o.y, o.z + L * std::round(2 * U(g)));
        if (form == 5) q[k] = mk(o.x + L * U(g), o.y + 1e-5 * L * U(g), o.z + 1e-5 * L * U(g));
      }
      const d3 m1 = mk(mv * N(g), mv * N(g), mv * N(g)), m2 = i % 4 == 0 ? mk(0, 0, 0) : mk(mv * N(g), mv * N(g), mv * N(g));
      for (int kind = 0; kind < 2; ++kind) {
        d3 a[4], b[4];
        f3 fa[4], fb[4];
        for (int k = 0; k < 4; ++k) {
          const bool second = kind ? k >= 2 : k == 0;
          a[k] = second ? add(q[k], dd) : q[k];
          b[k] = add(a[k], second ? m1 : m2);
          if (i & 1) b[k] = add(b[k], mk(0.2 * mv * N(g), 0.2 * mv * N(g), 0.2 * mv * N(g)));
          fa[k] = tf(a[k]);
          fb[k] = tf(b[k]);
        }
        const double t = kind ? ee_collision_time(a, a + 2, b, b + 2) : pt_collision_time(a[0], a + 1, b[0], b + 1);
        const bool c = kind ? f_ee_miss(fa, fb, fa + 2, fb + 2) : f_pt_miss(fa[0], fb[0], fa + 1, fb + 1);
        hit[kind] += t < 1.0;
        cert[kind] += c;
        if (c && t != 1.0) ++bad;
        if ((kind ? toi_fast<1>(a, b) : toi_fast<0>(a, b)) != t) ++bad;
      }
    }
    printf("size %g distance %g motion %g offset %g: hits %.4f %.4f certified %.4f %.4f\n", L, D, mv, off,
           hit[0] / (double)n, hit[1] / (double)n, cert[0] / (double)n, cert[1] / (double)n);
  }
  // values that certify nothing
  const float bigs[] = {1e30f, INFINITY, NAN};
  for (float v : bigs) {
    const f3 p{v, 0, 0}, z{0, 0, 0}, x{1, 0, 0}, y{0, 1, 0};
    const f3 t[3] = {z, x, y}, e[2] = {z, x}, h[2] = {p, y};
    if (f_pt_miss(p, p, t, t) || f_ee_miss(e, e, h, h)) ++bad;
  }
  printf("contradictions %ld\n", bad);
  return bad != 0;
}
