// CPU check of the error bounds of the FP32 vectors behind the trajectory certificates and the
// FP32 root verification (abd_ccd_filter.cuh): the difference of two points along a step, formed
// from their rounded ends, against the same in FP64. Coordinates just past a power of two, where
// every rounding is largest, and motions from none to edges that reverse; among random values
// of a coordinate the one of largest error is taken, so that the three errors add up. Prints the
// largest error as a share of the stated bound.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../adb_gb300/csrc/abd_ccd_filter.cuh"
using namespace abd;

struct Coord {
  double p0, p1, q0, q1;  // two points at the start and at the end
  float a0() const { return (float)p1 - (float)p0; }
  float a1() const { return (float)q1 - (float)q0; }
  double at(double t) const { return (p1 - p0) + t * ((q1 - q0) - (p1 - p0)); }
};
static double norm3(const double* x) { return std::sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]); }

int main(int argc, char** argv) {
  std::mt19937_64 g(argc > 1 ? atoi(argv[1]) : 1);
  std::uniform_real_distribution<double> U(0, 1);
  double worst = 0.0;
  for (int trial = 0; trial < 300; ++trial) {
    const int form = trial % 3;  // the edge reverses, stays, or turns up from nothing
    const double t = trial % 2 ? 1.0 - 0.5 * U(g) : U(g);
    auto draw = [&]() {
      auto v = [&]() { return 1.0 + U(g) * (1.0 / 1024); };
      const double p1 = v(), p0 = -v();
      if (form == 0) return Coord{p0, p1, v(), -v()};
      if (form == 1) return Coord{p0, p1, p0 + 2.4e-7 * U(g), p1 + 2.4e-7 * U(g)};
      return Coord{v(), v(), -v(), v()};
    };
    Coord best[3];
    for (Coord& b : best) {
      double most = -1.0;
      for (int k = 0; k < 3000; ++k) {
        const Coord c = draw();
        const f3m r = f3m_at(f3{c.a0(), 0, 0}, f3{c.a1(), 0, 0}, (float)t, 0.f);
        const double e = r.c.x - c.at(t);
        if (e > most) {
          most = e;
          b = c;
        }
      }
    }
    float m = 0.f;
    for (const Coord& c : best)
      m = fmaxf(m, fmaxf(fmaxf(fabsf((float)c.p0), fabsf((float)c.p1)), fmaxf(fabsf((float)c.q0), fabsf((float)c.q1))));
    const float E = 4.5e-7f * m + 1e-30f;
    const f3 a0{best[0].a0(), best[1].a0(), best[2].a0()}, a1{best[0].a1(), best[1].a1(), best[2].a1()};
    const f3m r = f3m_at(a0, a1, (float)t, E);
    const double d[3] = {r.c.x - best[0].at(t), r.c.y - best[1].at(t), r.c.z - best[2].at(t)};
    worst = fmax(worst, norm3(d) / r.dev);
  }
  printf("at a time: %.3f of the bound\n", worst);
  // half-way value of long edges that hardly change: what the change leaves of the bound
  double worst_mid = 0.0;
  for (int trial = 0; trial < 200; ++trial) {
    const double t = trial % 2;
    Coord best[3];
    for (Coord& b : best) {
      double most = -1.0;
      for (int k = 0; k < 20000; ++k) {
        auto v = [&]() { return 1.0 + 1e-5 * U(g); };
        Coord c{-v(), v(), 0.0, 0.0};
        c.q0 = c.p0 + (U(g) - 0.5) * 5e-7 * (k % 3);
        c.q1 = c.p1 + (U(g) - 0.5) * 5e-7 * (k % 3);
        const double e = f3m_of(f3{c.a0(), 0, 0}, f3{c.a1(), 0, 0}, 0.f).c.x - c.at(t) - 0.5 * std::fabs((double)c.a1() - c.a0());
        if (e > most) {
          most = e;
          b = c;
        }
      }
    }
    float m = 0.f;
    for (const Coord& c : best)
      m = fmaxf(m, fmaxf(fmaxf(fabsf((float)c.p0), fabsf((float)c.p1)), fmaxf(fabsf((float)c.q0), fabsf((float)c.q1))));
    const f3m r = f3m_of(f3{best[0].a0(), best[1].a0(), best[2].a0()}, f3{best[0].a1(), best[1].a1(), best[2].a1()},
                         4.5e-7f * m + 1e-30f);
    const double d[3] = {r.c.x - best[0].at(t), r.c.y - best[1].at(t), r.c.z - best[2].at(t)};
    worst_mid = fmax(worst_mid, norm3(d) / r.dev);
  }
  printf("half-way: %.4f of the bound\n", worst_mid);
  return worst > 1.0 || worst_mid > 1.0;
}
