// Temporal blocking of the 2D FP64 grids: several whole steps per launch, in
// windows of 64 x 32 cells (as kernels_window.cu takes the FP32 ones, whose
// opening comment has the scheme: overlapping windows, two copies of the state,
// an even number of launches).
//
// What bounded a small FP64 grid was the chain of launches (256 x 256: 7 us per
// step in four launches); what bounds a window is the chain of a step through
// shared memory and two barriers (a scheduler issues on 46% of cycles; waits on
// shared memory 3.3, fixed latencies 2.5, barriers 2.0 cycles per issue) and its
// instructions, the reference's IEEE divisions among them. A thread holds two neighbouring columns
// of one row, so that the loop stays within the instruction cache (two rows per
// thread, with every division in line, stalled 3.5 cycles per issue on it); 32
// warps at 64 registers take one window per SM. The CPML integrators and the P and J of dispersive cells
// stay in shared memory, where only the cells that have them touch them.
//
// Per cell the operations and their order are plain_e_cell's and
// plain_h_cell's (kernels_plain.cu); this file too is compiled with
// -fmad=false, so every result is the same bit for bit.
#include <algorithm>

#include "plain_tfsf.cuh"
#include "quotient.cuh"

namespace fdtdb {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kRows = kWin64Rows;  // a warp per row
constexpr int kCells = kWinCols * kRows;

// what acts on cells of the window besides the update: a source (its values
// per step in `put`), or a TFSF plane's correction of one component (its
// values per step and cell in memory)
struct Act {
  int comp, lo[2], hi[2];  // window coordinates, clipped to the window
  int ex;                  // plane: cells per row of its box
  const double* at;        // plane: the value of window cell (0, 0) at the launch's first step
};
constexpr int kMaxActs = 32;
struct Region64 {
  int comp, lo[2], hi[2], ex;
  double* out;
};

// sets of acts (bit masks), in the order a half step applies them
enum { kPlanes = 0, kFlux = 1, kSoft = 2, kBox = 3, kKinds = 4 };

struct alignas(16) Shared64 {
  double edge_e[kRows + 1][kWinCols];
  double edge_h[kRows + 1][kWinCols];
  double xp[2][4][kWinCols];  // F, B, C, G of the columns
  double yp[2][4][kRows];
  int ys[kRows];
  Act act[kMaxActs];
  double put[kMaxActs][kWinMaxSteps];
  unsigned sets[2][kKinds];
  Region64 reg[2][kWinMaxRegions];
  int nact, nreg[2];
};

struct Span {
  int x0, y0, ox0, ox1, oy0, oy1;
};

__device__ __forceinline__ double table_value(const double* vals, int nvals, long long t) {
  return t >= 0 && t < nvals ? vals[t] : 0.0;
}

// Lists what acts inside the window: one warp, its lanes in the order planes
// (two components each), sources, boxes, taken 32 at a time
__device__ __forceinline__ void list_acts(const Win64Args& a, Shared64& sh, const Span& sp, int s, int lane) {
  const int total = 4 * a.nplanes + a.nsrc + a.nbox;
  int n = 0;
  if (lane < 2 * kKinds) sh.sets[lane / kKinds][lane % kKinds] = 0;
  __syncwarp();
  for (int base = 0; base < total; base += 32) {
    const int q = base + lane;
    Act t{};
    int half = 0, kind = 0;
    bool in = false;
    if (q < 4 * a.nplanes) {
      const PlaneDev& p = a.planes[q >> 2];
      half = q >> 1 & 1;
      kind = kPlanes;
      // the components the half step's planes correct: those of the mode tangential to the plane
      int comp = -1;
      for (int I = 0, c = q & 1; I < 3; I++) {
        const bool has = half == 0 ? hasE(a.mode, I) && hasH(a.mode, third(I, p.axis)) && I != p.axis
                                   : hasH(a.mode, I) && hasE(a.mode, third(I, p.axis)) && I != p.axis;
        if (has && c-- == 0) comp = I;
      }
      t.comp = comp;
      for (int d = 0; d < 2; d++) {
        t.lo[d] = p.lo[d];
        t.hi[d] = p.hi[d];
      }
      t.ex = p.hi[0] - p.lo[0] + 1;
      in = comp >= 0;
      t.at = a.tfsf + (static_cast<long long>(s) * 2 + half) * a.tfsf_cells * 3 +
             3 * (p.off + static_cast<long long>(sp.y0 - p.lo[1]) * t.ex + (sp.x0 - p.lo[0])) + (comp < 0 ? 0 : comp);
    } else if (q < 4 * a.nplanes + a.nsrc) {
      const SourceDev& r = a.src[q - 4 * a.nplanes];
      half = r.target < 2 ? 0 : 1;
      kind = r.target == 1 || r.target == 3 ? kFlux : kSoft;
      t.comp = r.comp;
      t.lo[0] = t.hi[0] = r.i;
      t.lo[1] = t.hi[1] = r.j;
      in = true;
    } else if (q < total) {
      const WinBox& b = a.box[q - 4 * a.nplanes - a.nsrc];
      half = b.target == 0 ? 0 : 1;
      kind = kBox;
      t.comp = b.comp;
      for (int d = 0; d < 2; d++) {
        t.lo[d] = b.lo[d];
        t.hi[d] = b.hi[d];
      }
      in = true;
    }
    t.lo[0] = max(t.lo[0] - sp.x0, 0);
    t.lo[1] = max(t.lo[1] - sp.y0, 0);
    t.hi[0] = min(t.hi[0] - sp.x0, kWinCols - 1);
    t.hi[1] = min(t.hi[1] - sp.y0, kRows - 1);
    in = in && t.lo[0] <= t.hi[0] && t.lo[1] <= t.hi[1];
    const unsigned set = __ballot_sync(kAll, in);
    const int at = n + __popc(set & ((1u << lane) - 1));
    if (in && at < kMaxActs) {
      sh.act[at] = t;
      atomicOr(&sh.sets[half][kind], 1u << at);
      // which source the act is, for its values
      sh.act[at].ex = kind == kPlanes ? t.ex : q - 4 * a.nplanes;
    }
    n = min(n + __popc(set), kMaxActs);
  }
  if (lane == 0) sh.nact = n;
}

__device__ __forceinline__ void act_values(const Win64Args& a, Shared64& sh, int T, long long t0) {
  const unsigned planes = sh.sets[0][kPlanes] | sh.sets[1][kPlanes];
  for (int w = threadIdx.x; w < sh.nact * T; w += blockDim.x) {
    const int k = w / T, st = w % T;
    if (planes >> k & 1) continue;
    const int q = sh.act[k].ex;
    sh.put[k][st] = q < a.nsrc ? table_value(a.src[q].vals, a.src[q].nvals, t0 + st)
                               : table_value(a.box[q - a.nsrc].vals, a.box[q - a.nsrc].nvals, t0 + st);
  }
}

// v with the acts of `set` on component comp added, for the two columns of a
// lane in window row `row` (out of line: few warps come here)
__device__ __noinline__ double2 with_acts(const Shared64& sh, unsigned set, long long plane_step, int comp, int row,
                                          int lane, int st, double2 v) {
#pragma unroll 1
  for (; set; set &= set - 1) {
    const int k = __ffs(set) - 1;
    const Act& t = sh.act[k];
    if (t.comp != comp || row < t.lo[1] || row > t.hi[1]) continue;
    const int c = 2 * lane;
    double x, y;
    if (plane_step) {
      const double* p = t.at + st * plane_step + 3 * (row * t.ex + c);
      x = c >= t.lo[0] && c <= t.hi[0] ? p[0] : 0.0;
      y = c + 1 >= t.lo[0] && c + 1 <= t.hi[0] ? p[3] : 0.0;
    } else {
      x = y = sh.put[k][st];
    }
    if (c >= t.lo[0] && c <= t.hi[0]) v.x += x;
    if (c + 1 >= t.lo[0] && c + 1 <= t.hi[0]) v.y += y;
  }
  return v;
}

__device__ __forceinline__ void apply(const Win64Args& a, const Shared64& sh, unsigned set, bool plane, int comp, int row,
                                      int lane, int st, double (&v)[2]) {
  if (!set) return;
  const double2 r = with_acts(sh, set, plane ? a.tfsf_cells * 6 : 0, comp, row, lane, st, make_double2(v[0], v[1]));
  v[0] = r.x;
  v[1] = r.y;
}

// the samples of the window's own cells in the DFT regions of `set`, out of line as with_acts
__device__ __noinline__ void sample(const Region64* reg, unsigned set, long long at, int row, int lane, double2 fa, int ca,
                                    double2 fb) {
#pragma unroll 1
  for (; set; set &= set - 1) {
    const Region64& g = reg[__ffs(set) - 1];
    const int c = 2 * lane;
    if (row < g.lo[1] || row > g.hi[1]) continue;
    const double2 f = g.comp == ca ? fa : fb;
    double* o = g.out + at + static_cast<long long>(row) * g.ex + c;
    if (c >= g.lo[0] && c <= g.hi[0]) o[0] = f.x;
    if (c + 1 >= g.lo[0] && c + 1 <= g.hi[0]) o[1] = f.y;
  }
}

// E of one cell with poles from its flux, out of line as with_acts (drude:: and lorentz::
// implicit_update, DispersiveMaterials.hpp:979-998, :710-735); P and J in
// shared memory, `stride` doubles between arrays: P, J of the first pole, ..
__device__ __noinline__ double pole_update(const MatF64& m, double D, double dt, double* pj, int stride) {
  if (m.kind == 2) {
    double P = pj[0], J = pj[stride];
    P += dt * J;
    const double E = (D - P) / m.den_e;
    pj[0] = P;
    pj[stride] = J * m.c1[0] / m.c2[0] + m.c3[0] * E;
    return E;
  }
  double num = D;
  for (int q = 0; q < m.npoles; q++) {
    const double P = pj[2 * q * stride] + dt * pj[(2 * q + 1) * stride];
    pj[2 * q * stride] = P;
    num = num - P;
  }
  const double E = num / m.den_e;
  for (int q = 0; q < m.npoles; q++) {
    double* J = pj + (2 * q + 1) * stride;
    *J = m.c1[q] * *J + m.c2[q] * E - m.c3[q] * pj[2 * q * stride];
  }
  return E;
}

}  // namespace

template <int MODE, bool GEN>
__device__ __forceinline__ void window64_run(const Win64Args& a, Shared64& sh, double* psi, const Span& sp, int T,
                                             int from, int slot, const int (&mid)[2]) {
  constexpr bool TE = MODE == kTE;
  constexpr int NE = TE ? 2 : 1, NH = TE ? 1 : 2;
  const int row = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = sp.x0 + 2 * lane, j = sp.y0 + row;
  const long long nx = a.nx;
  const double dt = a.dt;
  double D[NE][2], B[NH][2], E[NE][2], H[NH][2];
  // arrays of the window in shared memory: the integrators, the divisors and
  // their reciprocals, P and J of each (component, pole)
  double* const psi_at = psi + row * kWinCols + 2 * lane;
  double* const den_at = psi_at + 4 * kCells;
  double* const pj_at = psi_at + 6 * kCells;
  bool in[2] = {true, true};  // an interior cell
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const bool here = !GEN || (c0 + c < a.nx && j < a.ny);
    if (GEN) in[c] = c0 + c >= 1 && c0 + c <= a.nx - 2 && j >= 1 && j <= a.ny - 2;
    const long long at = j * nx + c0 + c;
#pragma unroll
    for (int q = 0; q < NE; q++) {
      D[q][c] = here ? __ldcg(a.D[from][q] + at) : 0.0;
      // the coming E half forms E; a ring cell keeps the stored one
      E[q][c] = GEN && here && !in[c] ? __ldcg(a.E[from][q] + at) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < NH; q++) {
      B[q][c] = here ? __ldcg(a.B[from][q] + at) : 0.0;
      H[q][c] = here ? __ldcg(a.H[from][q] + at) : 0.0;
    }
    const double den = a.den ? (here ? a.den[at] : 1.0) : a.den0;
    den_at[c] = den;
    den_at[c + kCells] = a.den ? quotient_reciprocal(den) : a.rden0;
  }
  const bool has_poles = GEN && __any_sync(kAll, (mid[0] | mid[1]) != 0);
  int xs[2] = {-1, -1}, ys = -1;
  unsigned mine = 0, reg_e = 0, reg_h = 0;
  if (GEN) {
    ys = sh.ys[row];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      if (in[c] && a.pml[0]) xs[c] = slab_index(a.slab[0], c0 + c);
      double p[4] = {0.0, 0.0, 0.0, 0.0};
      if (ys >= 0 && in[c]) {
        p[0] = __ldcg(a.psi[from][0] + ys * nx + c0 + c);
        p[2] = __ldcg(a.psi[from][2] + ys * nx + c0 + c);
      }
      if (xs[c] >= 0) {
        p[1] = __ldcg(a.psi[from][1] + static_cast<long long>(j) * a.slab[0].W + xs[c]);
        p[3] = __ldcg(a.psi[from][3] + static_cast<long long>(j) * a.slab[0].W + xs[c]);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) psi_at[c + q * kCells] = p[q];
      if (mid[c])
        for (int q = 0; q < 2 * a.np * NE; q++) pj_at[c + q * kCells] = __ldcg(a.pj[from][q] + j * nx + c0 + c);
    }
    for (int k = 0; k < sh.nact; k++)
      if (sh.act[k].hi[1] >= row && sh.act[k].lo[1] <= row) mine |= 1u << k;
    for (int k = 0; k < sh.nreg[0]; k++)
      if (sh.reg[0][k].hi[1] >= row && sh.reg[0][k].lo[1] <= row) reg_e |= 1u << k;
    for (int k = 0; k < sh.nreg[1]; k++)
      if (sh.reg[1][k].hi[1] >= row && sh.reg[1][k].lo[1] <= row) reg_h |= 1u << k;
  }
  const bool has_x = GEN && __any_sync(kAll, xs[0] >= 0 || xs[1] >= 0), has_y = GEN && ys >= 0;
#pragma unroll
  for (int c = 0; c < 2; c++) sh.edge_h[row + 1][2 * lane + c] = H[0][c];
  __syncthreads();

  // the integrators of array q: the flux gains fs*psi*G, psi becomes
  // B*psi + C*diff; cells outside the slab keep both
  auto pml_x = [&](int q, int h, double fs, double sign, const double (&diff)[2], double (&f)[2]) {
#pragma unroll
    for (int c = 0; c < 2; c++) {
      if (xs[c] < 0) continue;
      double* p = psi_at + c + q * kCells;
      const double v = *p;
      f[c] += fs * v * sh.xp[h][3][2 * lane + c];
      *p = sh.xp[h][1][2 * lane + c] * v + sign * sh.xp[h][2][2 * lane + c] * diff[c];
    }
  };
  auto pml_y = [&](int q, int h, double fs, double sign, const double (&diff)[2], double (&f)[2]) {
    const double Bc = sh.yp[h][1][row], C = sign * sh.yp[h][2][row], G = sh.yp[h][3][row];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      double* p = psi_at + c + q * kCells;
      const double v = *p, now = f[c] + fs * v * G;
      f[c] = in[c] ? now : f[c];
      if (in[c]) *p = Bc * v + C * diff[c];
    }
  };

#pragma unroll 1
  for (int st = 0; st < T; st++) {
    // ---- E half: Hz (TE) or Hy (TM) is differenced along x, Hz or Hx along y
    {
      const double fx0 = sh.xp[0][0][2 * lane], fx1 = sh.xp[0][0][2 * lane + 1], fy = sh.yp[0][0][row];
      const double2 below = *reinterpret_cast<const double2*>(&sh.edge_h[row][2 * lane]);
      const double (&hx)[2] = H[NH - 1];
      const double left = __shfl_up_sync(kAll, hx[1], 1);
      const double dfx[2] = {hx[0] - left, hx[1] - hx[0]}, dfy[2] = {H[0][0] - below.x, H[0][1] - below.y};
      double d[NE][2];
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const double fx = c ? fx1 : fx0;
        // (+ 0.0: the term of the absent component, which turns -0 into +0)
        if (TE) {
          d[0][c] = D[0][c] + dt * (fy * dfy[c] + 0.0);
          d[NE - 1][c] = D[NE - 1][c] + dt * (-fx * dfx[c] + 0.0);
        } else {
          d[0][c] = D[0][c] + dt * (fx * dfx[c] + -fy * dfy[c]);
        }
      }
      if (GEN) {
        if (__builtin_expect(mine != 0, 0)) {
#pragma unroll
          for (int q = 0; q < NE; q++) {
            apply(a, sh, mine & sh.sets[0][kPlanes], true, TE ? q : 2, row, lane, st, d[q]);
            apply(a, sh, mine & sh.sets[0][kFlux], false, TE ? q : 2, row, lane, st, d[q]);
          }
        }
        // UpdatePML X, then Y
        if (has_x) pml_x(1, 0, dt, TE ? -1.0 : 1.0, dfx, d[NE - 1]);
        if (has_y) pml_y(0, 0, dt, TE ? 1.0 : -1.0, dfy, d[0]);
      }
      const double2 den = *reinterpret_cast<const double2*>(den_at), rden = *reinterpret_cast<const double2*>(den_at + kCells);
      bool easy = quotient_by(rden.x) && quotient_by(rden.y);
#pragma unroll
      for (int q = 0; q < NE; q++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
          D[q][c] = in[c] ? d[q][c] : D[q][c];
          const double e = quotient_of(D[q][c], c ? den.y : den.x, c ? rden.y : rden.x);
          E[q][c] = in[c] ? e : E[q][c];
          easy = easy && quotient_in_range(D[q][c]);
        }
      if (__builtin_expect(!easy, 0)) {
#pragma unroll
        for (int q = 0; q < NE; q++)
#pragma unroll
          for (int c = 0; c < 2; c++)
            if (in[c]) E[q][c] = plain_quotient(D[q][c], den_at[c]);
      }
      if (GEN && has_poles) {
#pragma unroll
        for (int q = 0; q < NE; q++)
#pragma unroll
          for (int c = 0; c < 2; c++)
            if (mid[c] && in[c])
              E[q][c] = pole_update(a.mats[mid[c] - 1], D[q][c], dt, pj_at + c + 2 * a.np * q * kCells, kCells);
      }
      if (GEN && __builtin_expect(mine != 0, 0)) {
#pragma unroll
        for (int q = 0; q < NE; q++) {
          apply(a, sh, mine & sh.sets[0][kSoft], false, TE ? q : 2, row, lane, st, E[q]);
          apply(a, sh, mine & sh.sets[0][kBox], false, TE ? q : 2, row, lane, st, E[q]);
        }
      }
    }
    *reinterpret_cast<double2*>(&sh.edge_e[row][2 * lane]) = make_double2(E[0][0], E[0][1]);
    if (GEN && __builtin_expect(reg_e != 0, 0))
      sample(sh.reg[0], reg_e, (slot + st) * a.dft_pts[0], row, lane, make_double2(E[0][0], E[0][1]), TE ? 0 : 2,
             make_double2(E[NE - 1][0], E[NE - 1][1]));
    __syncthreads();
    // ---- H half: Ey (TE) or Ez (TM) is differenced along x, Ex or Ez along y
    {
      const double fx0 = sh.xp[1][0][2 * lane], fx1 = sh.xp[1][0][2 * lane + 1], fy = sh.yp[1][0][row];
      const double2 above = *reinterpret_cast<const double2*>(&sh.edge_e[row + 1][2 * lane]);
      const double (&ey)[2] = E[NE - 1];
      const double right = __shfl_down_sync(kAll, ey[0], 1);
      const double dfx[2] = {ey[1] - ey[0], right - ey[1]}, dfy[2] = {above.x - E[0][0], above.y - E[0][1]};
      double b[NH][2];
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const double fx = c ? fx1 : fx0;
        if (TE) {
          b[0][c] = B[0][c] + -dt * (fx * dfx[c] + -fy * dfy[c]);
        } else {
          b[0][c] = B[0][c] + -dt * (fy * dfy[c] + 0.0);
          b[NH - 1][c] = B[NH - 1][c] + -dt * (-fx * dfx[c] + 0.0);
        }
      }
      if (GEN) {
        if (__builtin_expect(mine != 0, 0)) {
#pragma unroll
          for (int q = 0; q < NH; q++) {
            apply(a, sh, mine & sh.sets[1][kPlanes], true, TE ? 2 : q, row, lane, st, b[q]);
            apply(a, sh, mine & sh.sets[1][kFlux], false, TE ? 2 : q, row, lane, st, b[q]);
          }
        }
        if (has_x) pml_x(3, 1, -dt, TE ? 1.0 : -1.0, dfx, b[NH - 1]);
        if (has_y) pml_y(2, 1, -dt, TE ? -1.0 : 1.0, dfy, b[0]);
      }
      bool easy = quotient_by(a.rden_h);
#pragma unroll
      for (int q = 0; q < NH; q++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
          B[q][c] = in[c] ? b[q][c] : B[q][c];
          const double h = quotient_of(B[q][c], a.den_h, a.rden_h);
          H[q][c] = in[c] ? h : H[q][c];
          easy = easy && quotient_in_range(B[q][c]);
        }
      if (__builtin_expect(!easy, 0)) {
#pragma unroll
        for (int q = 0; q < NH; q++)
#pragma unroll
          for (int c = 0; c < 2; c++)
            if (in[c]) H[q][c] = plain_quotient(B[q][c], a.den_h);
      }
      if (GEN && __builtin_expect(mine != 0, 0)) {
#pragma unroll
        for (int q = 0; q < NH; q++) {
          apply(a, sh, mine & sh.sets[1][kSoft], false, TE ? 2 : q, row, lane, st, H[q]);
          apply(a, sh, mine & sh.sets[1][kBox], false, TE ? 2 : q, row, lane, st, H[q]);
        }
      }
    }
    *reinterpret_cast<double2*>(&sh.edge_h[row + 1][2 * lane]) = make_double2(H[0][0], H[0][1]);
    if (GEN && __builtin_expect(reg_h != 0, 0))
      sample(sh.reg[1], reg_h, (slot + st) * a.dft_pts[1], row, lane, make_double2(H[0][0], H[0][1]), TE ? 2 : 0,
             make_double2(H[NH - 1][0], H[NH - 1][1]));
    __syncthreads();
  }

  const int to = 1 - from;
  if (j < sp.oy0 || j >= sp.oy1) return;
#pragma unroll
  for (int c = 0; c < 2; c++) {
    if (c0 + c < sp.ox0 || c0 + c >= sp.ox1) continue;
    const long long at = j * nx + c0 + c;
#pragma unroll
    for (int q = 0; q < NE; q++) {
      a.D[to][q][at] = D[q][c];
      a.E[to][q][at] = E[q][c];
    }
#pragma unroll
    for (int q = 0; q < NH; q++) {
      a.B[to][q][at] = B[q][c];
      a.H[to][q][at] = H[q][c];
    }
    if (!GEN || !in[c]) continue;
    const double* p = psi_at + c;
    if (ys >= 0) {
      a.psi[to][0][ys * nx + c0 + c] = p[0];
      a.psi[to][2][ys * nx + c0 + c] = p[2 * kCells];
    }
    if (xs[c] >= 0) {
      a.psi[to][1][static_cast<long long>(j) * a.slab[0].W + xs[c]] = p[kCells];
      a.psi[to][3][static_cast<long long>(j) * a.slab[0].W + xs[c]] = p[3 * kCells];
    }
    if (mid[c])
      for (int q = 0; q < 2 * a.np * NE; q++) a.pj[to][q][at] = pj_at[c + q * kCells];
  }
}

template <int MODE>
__global__ void __launch_bounds__(32 * kRows, 1) window64_kernel(const __grid_constant__ Win64Args a, int T, int s, int from,
                                                               int slot) {
  extern __shared__ __align__(16) double psi64[];
  __shared__ Shared64 sh;
  let_next_launch_start();
  Span sp;
  {
    const int ow = kWinCols - 2 * T, oh = kRows - 2 * T;
    const int tiles_x = window_tiles(a.nx, kWinCols, ow);
    const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
    sp.x0 = tx * ow;
    sp.y0 = ty * oh;
    sp.ox0 = tx == 0 ? 0 : sp.x0 + T;
    sp.oy0 = ty == 0 ? 0 : sp.y0 + T;
    sp.ox1 = sp.x0 + kWinCols >= a.nx ? a.nx : sp.x0 + kWinCols - T;
    sp.oy1 = sp.y0 + kRows >= a.ny ? a.ny : sp.y0 + kRows - T;
  }
  const int tid = threadIdx.x;
  // what no earlier launch writes: profiles, sources, regions, materials
  if (tid < kRows) {
    const int j = sp.y0 + tid;
    const bool rin = j >= 1 && j <= a.ny - 2;
    const int ys = rin && a.pml[1] ? slab_index(a.slab[1], j) : -1;
    sh.ys[tid] = ys;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      sh.yp[h][0][tid] = rin ? a.prof[h][1].F[j] : 0.0;
      sh.yp[h][1][tid] = ys >= 0 ? a.prof[h][1].B[j] : 0.0;
      sh.yp[h][2][tid] = ys >= 0 ? a.prof[h][1].C[j] : 0.0;
      sh.yp[h][3][tid] = ys >= 0 ? a.prof[h][1].G[j] : 0.0;
    }
  } else if (tid >= 64 && tid < 128) {
    const int l = tid - 64, c = sp.x0 + l;
    const bool in = c < a.nx;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      sh.xp[h][0][l] = in ? a.prof[h][0].F[c] : 0.0;
      sh.xp[h][1][l] = in ? a.prof[h][0].B[c] : 0.0;
      sh.xp[h][2][l] = in ? a.prof[h][0].C[c] : 0.0;
      sh.xp[h][3][l] = in ? a.prof[h][0].G[c] : 0.0;
    }
    sh.edge_h[0][l] = 0.0;
    sh.edge_e[kRows][l] = 0.0;
  } else if (tid >= 128 && tid < 160) {
    list_acts(a, sh, sp, s, tid & 31);
  } else if (tid >= 160 && tid < 224) {
    const int h = tid < 192 ? 0 : 1, lane = tid & 31;
    Region64 o{};
    bool in = false;
    if (lane < a.nreg[h]) {
      const DftRegionDev& g = a.reg[h][lane];
      const int lo0 = max(g.lo[0], sp.ox0), hi0 = min(g.lo[0] + g.ext[0], sp.ox1) - 1;
      const int lo1 = max(g.lo[1], sp.oy0), hi1 = min(g.lo[1] + g.ext[1], sp.oy1) - 1;
      in = lo0 <= hi0 && lo1 <= hi1;
      o.comp = g.comp;
      o.lo[0] = lo0 - sp.x0;
      o.hi[0] = hi0 - sp.x0;
      o.lo[1] = lo1 - sp.y0;
      o.hi[1] = hi1 - sp.y0;
      o.ex = g.ext[0];
      o.out = a.dft_buf[h] + g.pt_off + static_cast<long long>(sp.y0 - g.lo[1]) * g.ext[0] + (sp.x0 - g.lo[0]);
    }
    const unsigned set = __ballot_sync(kAll, in);
    if (in) sh.reg[h][__popc(set & ((1u << lane) - 1))] = o;
    if (lane == 0) sh.nreg[h] = __popc(set);
  }
  // the cells' materials with poles: 1 + the material's number, or 0
  int mid[2] = {0, 0};
  if (a.np > 0) {
    const int c0 = sp.x0 + 2 * (tid & 31), j = sp.y0 + (tid >> 5);
#pragma unroll
    for (int c = 0; c < 2; c++)
      if (c0 + c < a.nx && j < a.ny) mid[c] = a.disp[j * static_cast<long long>(a.nx) + c0 + c];
  }
  after_previous_launch();
  const long long t0 = a.ctrl->t + s;
  const bool poles = __syncthreads_or((mid[0] | mid[1]) != 0);
  act_values(a, sh, T, t0);
  __syncthreads();
  const bool plain = sp.x0 >= a.plain[0][0] && sp.x0 + kWinCols - 1 <= a.plain[0][1] && sp.y0 >= a.plain[1][0] &&
                     sp.y0 + kRows - 1 <= a.plain[1][1] && sh.nact + sh.nreg[0] + sh.nreg[1] == 0 && !poles;
  if (plain) window64_run<MODE, false>(a, sh, psi64, sp, T, from, slot, mid);
  else window64_run<MODE, true>(a, sh, psi64, sp, T, from, slot, mid);
}

namespace {

// The TFSF corrections of every plane cell for nsteps steps from the counter
// on: tfsf_pre_kernel's (kernels_plain.cu), [step][half][cell][component]
template <int MODE>
__global__ void __launch_bounds__(128) tfsf_table_kernel(const __grid_constant__ PlainArgs a, double* out) {
  const PlaneDev& p = a.planes[blockIdx.y];
  const long long ex = p.hi[0] - p.lo[0] + 1, cells = ex * (p.hi[1] - p.lo[1] + 1);
  const long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q >= cells) return;
  const int idx[3] = {p.lo[0] + static_cast<int>(q % ex), p.lo[1] + static_cast<int>(q / ex), 0};
  const int s = blockIdx.z;
  for (int ft = 0; ft < 2; ft++) {
    const long long row = a.ctrl->t + s - a.ctrl->t0 + ft;
    double* o = out + ((static_cast<long long>(s) * 2 + ft) * a.tfsf_cells + p.off + q) * 3;
#pragma unroll
    for (int I = 2; I >= 0; I--) {
      if (ft == 0 ? !hasE(MODE, I) : !hasH(MODE, I)) continue;
      o[I] = tfsf_correction<MODE>(a, p, row, ft, I, idx);
    }
  }
}

// the flux-to-field divisor of every cell without poles, and the materials
// with poles
__global__ void window64_cells_kernel(const __grid_constant__ PlainArgs a, double* den, unsigned short* disp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.nx || j >= a.ny) return;
  const long long c = static_cast<long long>(j) * a.nx + i;
  int mid = 0;
  if (a.ids) mid = a.ids[c];
  else if (a.bids) mid = a.bids[(j >> a.bshift) * a.nbx + (i >> a.bshift)];
  const MatF64& m = a.mats[mid];
  const double eps = a.eps_map ? a.eps_map[c] : 0.0;
  if (den) den[c] = m.kind >= 2 ? 1.0 : (a.eps_map && eps > 0.0) ? eps * kEps0 : m.den_e;
  if (disp) disp[c] = m.kind >= 2 ? static_cast<unsigned short>(1 + mid) : 0;
}

template <int MODE>
void window64_go(const Win64Args& a, int n, int T, int s, int from, int slot, cudaStream_t st) {
  auto fn = window64_kernel<MODE>;
  constexpr int NE = MODE == kTE ? 2 : 1;
  const size_t bytes = (6 + 2 * static_cast<size_t>(a.np) * NE) * kCells * sizeof(double);
  once_per_device(reinterpret_cast<const void*>(fn), [&] {
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (6 + 2 * kWin64Poles) * kCells * static_cast<int>(sizeof(double)));
  });
  launch_chained(fn, dim3(n), dim3(32 * kRows), bytes, st, a, T, s, from, slot);
}

}  // namespace

int launch_window64(int mode, const Win64Args& a, int T, int s, int from, int slot, cudaStream_t st) {
  const int n = window64_count(a.nx, a.ny, T);
  if (mode == kTE) window64_go<kTE>(a, n, T, s, from, slot, st);
  else window64_go<kTM>(a, n, T, s, from, slot, st);
  return 1;
}

int launch_tfsf_table(int mode, const PlainArgs& a, int nsteps, double* out, cudaStream_t s) {
  if (a.nplanes == 0) return 0;
  long long most = 1;
  for (int q = 0; q < a.nplanes; q++) {
    const PlaneDev& p = a.planes[q];
    most = std::max(most, static_cast<long long>(p.hi[0] - p.lo[0] + 1) * (p.hi[1] - p.lo[1] + 1));
  }
  const dim3 grid(static_cast<unsigned>((most + 127) / 128), a.nplanes, nsteps);
  if (mode == kTE) tfsf_table_kernel<kTE><<<grid, 128, 0, s>>>(a, out);
  else tfsf_table_kernel<kTM><<<grid, 128, 0, s>>>(a, out);
  return 1;
}

int launch_window64_cells(const PlainArgs& a, double* den, unsigned short* disp, cudaStream_t s) {
  const dim3 block(32, 8), grid((a.nx + 31) / 32, (a.ny + 7) / 8);
  window64_cells_kernel<<<grid, block, 0, s>>>(a, den, disp);
  return 1;
}

}  // namespace fdtdb
