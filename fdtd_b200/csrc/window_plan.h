// Whether a stretch of steps of a 2D grid goes out in windows (kernels_window.cu,
// kernels_window64.cu) or in launches per half step, and in which windows: the
// form with the least modelled time. Host code, checked on the CPU
// (tests/cpp/window_plan_check.cu).
//
// A launch of windows lasts as long as its first window, first + step * T us for
// T steps, and more + more_step * T us for each further window of an SM (from
// 0.7 windows per SM on where two share one). The
// launches per half step take, per step, the latency of their kernels or the
// time of their cells, whichever is longer, and each kernel beside the two sweeps
// what it adds to the chain. All constants are fitted to B200 measurements of 64
// steps on 70 x 70 to 2000 x 2000 cells, windows of 2 to 16 steps (rms error 2
// to 5% without poles or with poles everywhere, 7 to 14% with a Drude disk).
// They matter most where the two forms are close. FP64 without poles, 256 x 256:
// a call of 2 steps takes 14.4 us per half step and 29.0 in windows, of 8 steps
// 50.5 and 44.5, of 64 steps 346 and 227. A Lorentz pole in every cell, FP64 TE,
// 64 steps: 256 x 256 392 and 500 us, 400 x 300 599 and 529, 600 x 450 1004 and
// 1104, 2000 x 2000 13.7 and 12.8 ms. FP32 takes windows from 4 steps on without
// poles (256 x 256: 29.7 and 18.5 us).
#pragma once
#include <algorithm>
#include <cmath>

#include "internal.h"

namespace fdtdb {

// what the choice depends on
struct WindowCase {
  bool f32 = false, te = false;
  int nx = 0, ny = 0;
  int poles = 0;  // 0 none, 1 Drude alone, 2 one Lorentz pole at most, 3 two
  // share of the 64 x 32 and of the 64 x 64 cell blocks that hold poles
  double pole_share[2] = {0.0, 0.0};
  int planes = 0, gathers = 0, boxes = 0;  // TFSF planes, phases with DFT regions, box sources
  bool graph = false;                      // the stretch is replayed from a graph
  int sms = 148;
};

struct WindowPlan {
  bool windows = false;
  int launches = 0, rows = 0;  // an even number of launches, rows of a window
  double us = 0.0, half_us = 0.0;  // modelled: in windows, in launches per half step
};

struct WindowCost {
  double first, step, more, more_step;
  bool pairs;  // two windows share an SM, so that the second costs less
};
// [poles]
constexpr WindowCost kWin64Te[3] = {{9.8, 2.8, 7.0, 0.84, false}, {12.4, 5.4, 17.2, 3.8, false}, {14.7, 6.4, 18.7, 4.8, false}};
constexpr WindowCost kWin64Tm[4] = {
    {9.8, 2.8, 7.0, 0.84, false}, {12.0, 3.6, 16.1, 2.4, false}, {13.2, 4.3, 15.2, 3.0, false}, {14.7, 6.2, 18.7, 4.6, false}};
constexpr WindowCost kWin32Te[4] = {
    {5.1, 0.99, 1.48, 0.12, true}, {8.7, 1.69, 9.4, 0.43, true}, {13.3, 2.0, 7.2, 1.03, true}, {16.2, 2.5, 17.0, 1.7, false}};
constexpr WindowCost kWin32Tm[4] = {
    {5.1, 0.99, 1.48, 0.12, true}, {7.1, 1.51, 8.8, 0.43, true}, {10.1, 1.66, 5.7, 0.68, true}, {10.8, 2.0, 11.0, 1.3, false}};
constexpr WindowCost kWin32TallTe[2] = {{9.4, 1.48, 2.65, 0.17, true}, {15.1, 2.9, 27.0, 1.9, false}};
constexpr WindowCost kWin32TallTm[2] = {{9.4, 1.48, 2.65, 0.17, true}, {11.7, 2.6, 27.0, 1.65, false}};

// launches per half step, us a step: at least `least`, else base + cells *
// (per million cells, and more for each of those beyond the L2 cache), the
// latter two higher by pole and pole_far where poles are
struct HalfCost {
  double least, base, cells, far, pole, pole_far;
};
constexpr HalfCost kHalf64Te[4] = {
    {5.3, 3.4, 35.0, 10.0, 0, 0}, {5.55, 3.6, 35.0, 10.0, 10.0, 2.0}, {5.8, 3.4, 35.0, 10.0, 10.0, 2.0}, {6.0, 3.3, 35.0, 10.0, 17.0, 4.0}};
constexpr HalfCost kHalf64Tm[4] = {
    {5.3, 3.4, 35.0, 10.0, 0, 0}, {5.4, 3.4, 35.0, 10.0, 0.0, 2.0}, {5.6, 4.1, 33.0, 10.0, 0.0, 3.0}, {5.7, 3.4, 35.0, 10.0, 8.5, 3.0}};
constexpr HalfCost kHalf32Te[4] = {
    {5.8, 4.9, 10.8, 0, 0, 0}, {6.0, 4.9, 10.8, 0, 2.5, 2.4}, {6.9, 5.3, 10.8, 0, 5.0, 4.8}, {7.75, 5.7, 10.8, 0, 8.8, 12.7}};
constexpr HalfCost kHalf32Tm[4] = {
    {5.8, 4.9, 10.8, 0, 0, 0}, {5.7, 5.1, 10.8, 0, 0.9, 0}, {6.4, 5.1, 10.8, 0, 1.8, 0}, {6.4, 5.7, 10.8, 0, 3.0, 6.0}};

// most steps of a launch of windows of `rows` rows: the inner cells stay a
// quarter of a window's rows at least
constexpr int window_most_steps(int rows) { return std::min(kWinMaxSteps, (rows + 16) / 4); }

// us of a launch of T steps in windows of `rows` rows
inline double window_launch_us(const WindowCase& c, int rows, int T) {
  const bool tall = rows == 64;
  const WindowCost* const t = !c.f32 ? (c.te ? kWin64Te : kWin64Tm)
                              : tall ? (c.te ? kWin32TallTe : kWin32TallTm)
                                     : (c.te ? kWin32Te : kWin32Tm);
  const double share = c.pole_share[tall];
  const WindowCost &p = t[c.poles], &n = t[0];
  const int windows = c.f32 ? window_count(c.nx, c.ny, rows, T) : window64_count(c.nx, c.ny, T);
  double one = share > 0.0 ? p.first + p.step * T : n.first + n.step * T;
  // the corrections of a plane: a chain of loads per step
  if (c.planes > 0) one = std::max(one, n.first + (n.step + (tall ? 2.8 : 1.75)) * T);
  const double next = share * (p.more + p.more_step * T) + (1.0 - share) * (n.more + n.more_step * T);
  const double rounds = p.pairs ? std::max(0.0, windows / static_cast<double>(c.sms) - 0.7) : (windows + c.sms - 1) / c.sms - 1;
  return one + rounds * next;
}

// us of n steps in launches per half step
inline double half_steps_us(const WindowCase& c, int n) {
  const HalfCost& h = (c.f32 ? (c.te ? kHalf32Te : kHalf32Tm) : (c.te ? kHalf64Te : kHalf64Tm))[c.poles];
  const double share = c.pole_share[0], cells = 1e-6 * c.nx * c.ny;
  const double bulk = h.base + (h.cells + share * h.pole) * cells + (h.far + share * h.pole_far) * std::max(0.0, cells - 1.5);
  // launched one by one a kernel takes longer than in a graph
  const double step = c.graph ? std::max(h.least, bulk) : std::max(1.2 * h.least, 1.05 * bulk);
  // (FP64 gathers wait for the sweep before them to end)
  const double gather = c.graph ? 2.2 : c.f32 ? 2.3 : 4.4;
  const double plane = c.f32 ? (c.graph ? 6.2 : 7.9) : (c.graph ? 4.8 : 5.8), box = c.f32 ? 4.6 : 2.3;
  return n * (step + gather * c.gathers + (c.planes > 0 ? plane : 0.0) + box * c.boxes);
}

// The plan of a stretch of n steps. The launches, even in number, share the steps
// as equally as they come.
inline WindowPlan window_plan(const WindowCase& c, int n) {
  WindowPlan best;
  best.us = 1e30;
  best.half_us = half_steps_us(c, n);
  for (int rows : {32, 64}) {
    // FP64 windows have 32 rows; with Lorentz poles a window of 64 is more than
    // an SM's shared memory
    if (rows == 64 && (!c.f32 || c.poles > 1)) continue;
    for (int L = 2; L <= n; L += 2) {
      const int T = n / L, longer = n - T * L;
      if (T + (longer > 0) > window_most_steps(rows)) continue;
      double us = (L - longer) * window_launch_us(c, rows, T);
      if (longer > 0) us += longer * window_launch_us(c, rows, T + 1);
      us += (c.planes > 0 ? 10.0 : 0.0) + (c.graph ? 0.0 : 2.0) + n * (0.1 * c.gathers + 0.2 * c.boxes);
      if (us >= best.us) continue;
      best.us = us;
      best.launches = L;
      best.rows = rows;
    }
  }
  // (windows where the two come out alike: over 6156 measured calls the choice is
  // 0.3% slower than the better of the two, and more than 4% slower in 2.5%)
  best.windows = best.launches > 0 && best.us <= 1.03 * best.half_us;
  // FP64 windows of one step move the state as often as the sweeps do, and their
  // halo besides: they gain by the planes, samples and boxes alone (the model has
  // no term for it: 499 x 1917, 2 steps 88 us per half step and 92 in windows)
  if (!c.f32 && n == 2 && c.planes + c.gathers + c.boxes == 0) best.windows = false;
  return best;
}

// Steps per launch and rows per window of the adjoint's reversed steps, fitted to
// the FP32 windows without poles: a launch takes from its predecessor's end about
// 4 us + 1.05 us a step with windows of 32 rows, 8 us + 1.5 us a step with 64
// (317 x 233), each further round of windows (two per SM) 5 and 11.5 us + 0.1 us
// a step (3001 x 2047).
inline int adjoint_window_steps(int nx, int ny, int sms, int* rows) {
  int best = 8;
  double least = 1e30;
  for (int R : {32, 64})
    for (int L : {16, 12, 8, 6, 4}) {
      const int T = (64 + L - 1) / L;
      if (T > window_most_steps(R)) continue;
      const double rounds = window_count(nx, ny, R, T) / (2.0 * sms);
      const double one = R == 32 ? 4.0 + 1.05 * T : 8.0 + 1.5 * T;
      const double more = (R == 32 ? 5.0 : 11.5) + 0.1 * T;
      const double t = (one + std::max(0.0, rounds - 1.0) * more) * L;
      if (t < least) {
        least = t;
        best = T;
        *rows = R;
      }
    }
  return best;
}

}  // namespace fdtdb
