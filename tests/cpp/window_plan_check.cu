// The plans of 2D steps (fdtd_b200/csrc/window_plan.h), checked on the host:
// * for every kind of grid, extents around the windows' and up to 5000 cells and
//   stretches of 2 to 64 steps: an even number of launches that share the steps,
//   none longer than a window of those rows holds exact, rows that the kind has;
// * for the calls measured below (B200, us a call in windows and in launches per
//   half step, of either precision, with and without poles, planes and DFT
//   regions, short and long), the faster form.
// Exit status 1 on the first violation.
#include <cstdio>

#include "../../fdtd_b200/csrc/window_plan.h"

using namespace fdtdb;

struct Measured {
  bool f32, te;
  int nx, ny, poles;
  double share32, share64;
  int planes, gathers, n;
  double windows_us, half_us;
};

const Measured kMeasured[] = {
    {true, true, 64, 2500, 0, 0.000, 0.000, 0, 0, 8, 23, 66},
    {true, true, 480, 700, 0, 0.000, 0.000, 4, 1, 8, 63, 175},
    {true, true, 600, 450, 1, 0.107, 0.113, 4, 0, 8, 59, 144},
    {true, false, 2900, 70, 1, 0.014, 0.011, 0, 0, 8, 31, 66},
    {true, true, 64, 2500, 1, 0.025, 0.025, 0, 0, 2, 27, 18},
    {true, true, 333, 333, 1, 0.167, 0.222, 0, 1, 2, 31, 27},
    {true, true, 2000, 2000, 2, 1.000, 1.000, 0, 1, 64, 4664, 5315},
    {true, true, 400, 300, 2, 1.000, 1.000, 0, 1, 64, 292, 604},
    {true, true, 600, 450, 2, 1.000, 1.000, 0, 0, 2, 41, 23},
    {true, true, 128, 128, 2, 1.000, 1.000, 0, 0, 2, 33, 18},
    {true, false, 110, 200, 3, 1.000, 1.000, 0, 0, 16, 60, 120},
    {true, true, 64, 2500, 3, 1.000, 1.000, 0, 1, 64, 505, 656},
    {true, false, 1700, 1100, 3, 1.000, 1.000, 0, 0, 8, 347, 268},
    {true, false, 800, 800, 3, 1.000, 1.000, 0, 0, 2, 75, 35},
    {false, true, 256, 256, 0, 0.000, 0.000, 0, 1, 64, 233, 472},
    {false, false, 256, 256, 0, 0.000, 0.000, 4, 0, 64, 388, 684},
    {false, false, 480, 700, 0, 0.000, 0.000, 0, 0, 2, 43, 34},
    {false, false, 499, 1917, 0, 0.000, 0.000, 0, 0, 2, 92, 88},
    {false, true, 1200, 300, 0, 0.000, 0.000, 0, 0, 2, 43, 35},
    {false, false, 2000, 2000, 1, 0.100, 0.103, 4, 1, 16, 1227, 3154},
    {false, false, 2500, 2500, 1, 0.095, 0.098, 4, 1, 2, 547, 637},
    {false, true, 400, 300, 1, 0.114, 0.171, 0, 1, 2, 49, 35},
    {false, false, 110, 200, 1, 0.286, 0.250, 4, 1, 2, 58, 43},
    {false, false, 256, 256, 2, 1.000, 1.000, 0, 1, 8, 72, 90},
    {false, true, 90, 60, 2, 1.000, 1.000, 0, 1, 16, 144, 172},
    {false, true, 2000, 2000, 2, 1.000, 1.000, 0, 1, 2, 749, 454},
    {false, true, 70, 70, 2, 1.000, 1.000, 0, 0, 64, 509, 369},
    {false, false, 333, 333, 3, 1.000, 1.000, 0, 0, 16, 132, 154},
    {false, false, 333, 333, 3, 1.000, 1.000, 0, 1, 8, 88, 116},
    {false, false, 1000, 700, 3, 1.000, 1.000, 0, 0, 64, 2422, 2104},
    {false, false, 1000, 700, 3, 1.000, 1.000, 0, 0, 2, 150, 70},
};

int main() {
  long checked = 0;
  for (int kind = 0; kind < 16; kind++)
    for (int nx : {3, 33, 64, 65, 70, 107, 256, 500, 1300, 5000})
      for (int ny : {3, 20, 32, 33, 64, 65, 97, 600, 2047, 5000})
        for (int n = 2; n <= 64; n++)
          for (int more = 0; more < 4; more++) {
            WindowCase c;
            c.f32 = kind & 1;
            c.te = kind >> 1 & 1;
            c.poles = kind >> 2;
            if (!c.f32 && c.te && c.poles == 3) continue;  // more than an FP64 TE window holds
            c.nx = nx;
            c.ny = ny;
            c.pole_share[0] = c.pole_share[1] = c.poles ? 0.25 + 0.25 * more : 0.0;
            c.planes = more & 1 ? 4 : 0;
            c.gathers = more >> 1;
            c.graph = n == 64;
            const WindowPlan p = window_plan(c, n);
            const int longest = p.launches > 0 ? (n + p.launches - 1) / p.launches : 0;
            const bool rows_ok = p.rows == 32 || (p.rows == 64 && c.f32 && c.poles < 2);
            if (p.launches < 2 || p.launches % 2 || p.launches > n || !rows_ok || longest > kWinMaxSteps ||
                p.rows - 2 * longest < 8 || kWinCols - 2 * ((longest + 1) & ~1) < 8 || !(p.us > 0.0) || !(p.half_us > 0.0)) {
              printf("kind %d %d x %d n %d: %d launches of %d rows, %g us\n", kind, nx, ny, n, p.launches, p.rows, p.us);
              return 1;
            }
            checked++;
          }
  for (const Measured& m : kMeasured) {
    WindowCase c;
    c.f32 = m.f32;
    c.te = m.te;
    c.nx = m.nx;
    c.ny = m.ny;
    c.poles = m.poles;
    c.pole_share[0] = m.share32;
    c.pole_share[1] = m.share64;
    c.planes = m.planes;
    c.gathers = m.gathers;
    c.graph = m.n == 64;
    const WindowPlan p = window_plan(c, m.n);
    if (p.windows != (m.windows_us < m.half_us)) {
      printf("%d x %d n %d: %g us in windows, %g per half step, modelled %g and %g\n", m.nx, m.ny, m.n, m.windows_us, m.half_us, p.us, p.half_us);
      return 1;
    }
  }
  printf("%ld plans checked\n", checked);
  return 0;
}
