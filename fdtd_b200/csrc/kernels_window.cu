// Temporal blocking of the 2D FP32 grids: several whole steps per launch.
//
// A small 2D grid's step is a chain of launches that each last as long as a
// few dependent L2 round trips; a large one moves its whole state through
// memory twice per step. Both costs are per launch, so one launch here takes
// T steps. A CTA holds a window of 64 x (R NW) cells of one grid in registers
// (each lane two neighbouring columns, each of its NW warps R rows: 64 rows in
// all with R = 4, 32 with R = 2),
// advances it T steps and writes back the inner cells that T steps leave
// exact: a step's dependence reaches one cell each way (E from H at i-1, j-1;
// H from E at i+1, j+1), so values within T cells of a window edge inside the
// grid go stale while the rest stay exact. Windows overlap, so a launch reads
// one copy of the state and writes the other (the grid or batch keeps a
// second copy); an even number of launches ends on the grid's own arrays.
//
// Why this shape: the two columns of a lane are one packed FP32 pair, so a
// pair's update is packed instructions plus one shuffle per half step for the
// x neighbour across lanes; y neighbours are the thread's own rows, except at
// a warp's first and last row, which pass through shared memory with one
// barrier per half step. Four rows keep the loop body within the instruction
// cache and the thread within 64 registers. Windows that touch the CPML, the
// outer ring, a source or a DFT region take the same update with the ring
// masked, profile values per row and column and the CPML integrators in
// shared memory.
//
// The per-cell arithmetic, and so every result, is that of the launches per
// half step: fused_e/h_kernel (XFIRST: the CPML terms of x before those of y)
// for a grid stepped alone, e/h_group_2d (y before x) for a batch. Products
// and sums are explicit operations, so that no other contraction can be
// chosen here.
#include <type_traits>

#include "pairs.cuh"

namespace fdtdb {

namespace {

using namespace pairs;

// what a source adds in this launch: a box, one soft source cell (or several
// on the same cell, summed as the sweeps sum them), or one flux source
struct Entry {
  int half, comp, kind;      // half 0 E, 1 H; kind 0 box, 1 soft point, 2 flux point
  int lo[2], hi[2];          // window coordinates, clipped to the window
};
constexpr int kMaxEntries = kMaxSources + kWinMaxBoxes;  // <= 32: entry sets are bit masks

struct Region {
  int comp, lo[2], hi[2];    // window coordinates, clipped to the cells the window owns
  int ex;
  float* out;                // sample of window cell (0, 0) in slot 0 (may lie outside the buffer)
};

// NW warps of R rows each
template <int NW, int R>
struct Shared {
  static constexpr int kRows = NW * R;
  pair_t edge_e[NW + 1][32];    // first row of each warp's E (the warp below reads it)
  pair_t edge_h[NW + 1][32];    // last row of each warp's H, one place up (the warp above reads it)
  pair_t xp[2][4][32];          // F, B, C, G of the columns
  pair_t yp[2][4][kRows];       // the same of the rows, each value twice
  int ys[kRows];                // the row's place in the y slab, or -1
  Entry entry[kMaxEntries];
  int holder[kMaxEntries];      // the lane that listed the entry
  float undo[kMaxEntries][kWinMaxSteps], put[kMaxEntries][kWinMaxSteps];
  unsigned kinds[2][3];         // the entries of each half and kind
  Region reg[2][kWinMaxRegions];
  int nentry, nreg[2];
};

__device__ __forceinline__ double table_value(const double* vals, int nvals, long long t) {
  return t >= 0 && t < nvals ? vals[t] : 0.0;
}

// The sources that act inside the window, in the order the sweeps apply them
// (boxes before points), listed by one warp: lane b < nbox holds box b, lane
// kWinMaxBoxes + q source q.
template <int NW, int R>
__device__ __forceinline__ void list_entries(const WinArgs& a, Shared<NW, R>& sh, int x0, int y0, int lane) {
  constexpr int rows = Shared<NW, R>::kRows;
  Entry e{};
  bool in = false;
  if (lane < a.nbox) {
    const WinBox& x = a.box[lane];
    e = Entry{x.target == 0 ? 0 : 1, x.comp, 0, {max(x.lo[0] - x0, 0), max(x.lo[1] - y0, 0)},
              {min(x.hi[0] - x0, kWinCols - 1), min(x.hi[1] - y0, rows - 1)}};
    in = e.lo[0] <= e.hi[0] && e.lo[1] <= e.hi[1];
  }
  const int q = lane - kWinMaxBoxes;
  if (q >= 0 && q < a.nsrc) {
    const SourceDev& s = a.src[q];
    const int lx = s.i - x0, ly = s.j - y0;
    in = lx >= 0 && lx < kWinCols && ly >= 0 && ly < rows;
    const bool flux = s.target == 1 || s.target == 3;
    if (in && !flux)  // soft sources on one cell are one entry
      for (int p = 0; p < q; p++) {
        const SourceDev& o = a.src[p];
        if (o.target == s.target && o.comp == s.comp && o.i == s.i && o.j == s.j) in = false;
      }
    e = Entry{s.target < 2 ? 0 : 1, s.comp, flux ? 2 : 1, {lx, ly}, {lx, ly}};
  }
  const unsigned set = __ballot_sync(kAll, in);
  const int at = __popc(set & ((1u << lane) - 1));
  if (in) {
    sh.entry[at] = e;
    sh.holder[at] = lane;
  }
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const unsigned of = __ballot_sync(kAll, in && e.half == k / 3 && e.kind == k % 3);
    // lanes to entry numbers
    unsigned m = 0;
    for (unsigned b = of; b; b &= b - 1) m |= 1u << __popc(set & ((1u << (__ffs(b) - 1)) - 1));
    if (lane == 0) sh.kinds[k / 3][k % 3] = m;
  }
  if (lane == 0) sh.nentry = __popc(set);
}

// the entries' values for the launch's steps, one thread per (entry, step)
template <int NW, int R>
__device__ __forceinline__ void entry_values(const WinArgs& a, Shared<NW, R>& sh, int T, long long t0, int from) {
  for (int w = threadIdx.x; w < sh.nentry * T; w += blockDim.x) {
    const int k = w / T, st = w % T, lane = sh.holder[k];
    const long long t = t0 + st;
    float u = 0.f, p = 0.f;
    if (lane < kWinMaxBoxes) {
      const WinBox& x = a.box[lane];
      const double scale = x.target == 0 ? 1.0 : a.eta;
      u = static_cast<float>(-scale * table_value(x.vals, x.nvals, t - 1));
      p = static_cast<float>(scale * table_value(x.vals, x.nvals, t));
    } else {
      const SourceDev& s = a.src[lane - kWinMaxBoxes];
      if (s.target == 1) p = static_cast<float>(table_value(s.vals, s.nvals, t) * a.src_scale_d);
      else if (s.target == 3) p = -static_cast<float>(table_value(s.vals, s.nvals, t) * a.src_scale_b);
      else
        for (int q = lane - kWinMaxBoxes; q < a.nsrc; q++) {
          const SourceDev& o = a.src[q];
          if (o.target != s.target || o.comp != s.comp || o.i != s.i || o.j != s.j) continue;
          const double v = table_value(o.vals, o.nvals, t);
          const double last = st == 0 ? a.src_last[from][q] : table_value(o.vals, o.nvals, t - 1);
          u = __fadd_rn(u, s.target == 2 ? static_cast<float>(last * a.src_scale_h) : static_cast<float>(last));
          p = __fadd_rn(p, s.target == 2 ? static_cast<float>(v * a.src_scale_h) : static_cast<float>(v));
        }
      u = -u;  // taken back
    }
    sh.undo[k][st] = u;
    sh.put[k][st] = p;
  }
}

// adds its value of step st to the cells of every entry in `set`; the warp's
// rows are row0 .. row0 + R - 1, fa and fb the (one or) two components
template <int R>
__device__ __forceinline__ void apply_entries(const Entry* entry, unsigned set, const float (*vals)[kWinMaxSteps], int st,
                                              int row0, int lane, pair_t (&fa)[R], int ca, pair_t (&fb)[R]) {
#pragma unroll 1
  for (; set; set &= set - 1) {
    const int k = __ffs(set) - 1;
    const Entry& e = entry[k];
    const Cols c(2 * lane, e.lo[0], e.hi[0]);
    const pair_t v = masked(vals[k][st], c.k0, c.k1);
    const int lo = e.lo[1] - row0, hi = e.hi[1] - row0;
    const bool first = e.comp == ca;
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r < lo || r > hi) continue;
      if (first) fa[r] = add2(fa[r], v);
      else fb[r] = add2(fb[r], v);
    }
  }
}

// the samples of the window's own cells in the DFT regions of `set`
template <int R>
__device__ __forceinline__ void sample_regions(const Region* reg, unsigned set, long long at, int row0, int lane,
                                               const pair_t (&fa)[R], int ca, const pair_t (&fb)[R]) {
#pragma unroll 1
  for (; set; set &= set - 1) {
    const Region& g = reg[__ffs(set) - 1];
    const Cols c(2 * lane, g.lo[0], g.hi[0]);
    const int lo = g.lo[1] - row0, hi = g.hi[1] - row0;
    const bool first = g.comp == ca;
    float* o = g.out + at + static_cast<long long>(row0) * g.ex + 2 * lane;
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r >= lo && r <= hi) {
        const float2 f = unpack(first ? fa[r] : fb[r]);
        if (c.k0) o[0] = f.x;
        if (c.k1) o[1] = f.y;
      }
      o += g.ex;
    }
  }
}

// Writes the launch's T samples of the thread's cells on the outer ring again,
// from the ring's values in memory, which it keeps: their registers became NaN
// next to a cell that is not finite. Out of line and at the kernel's end, where
// nothing else is live: next to no thread comes here.
template <bool TE, int R, class Sh>
__device__ __noinline__ void sample_ring(const WinArgs& a, const Sh& sh, int x0, int y0, int T, int from, int slot) {
  const int lane = threadIdx.x & 31, row0 = (threadIdx.x >> 5) * R;
  for (int h = 0; h < 2; h++)
    for (int k = 0; k < sh.nreg[h]; k++) {
      const Region& g = sh.reg[h][k];
      // the components' places in a.f: TE Ex, Ey, Hz, TM Ez, Hx, Hy
      const float* f = a.f[from][h == 0 ? (TE ? g.comp : 0) : (TE ? 2 : 1 + g.comp)];
      for (int w = max(g.lo[1], row0); w <= min(g.hi[1], row0 + R - 1); w++)
        for (int l = max(g.lo[0], 2 * lane); l <= min(g.hi[0], 2 * lane + 1); l++) {
          const int i = x0 + l, j = y0 + w;
          if (i > 0 && i < a.nx - 1 && j > 0 && j < a.ny - 1) continue;
          const float v = __ldcg(f + j * static_cast<long long>(a.pitch) + i);
          for (int st = 0; st < T; st++) g.out[(slot + st) * a.dft_pts[h] + static_cast<long long>(w) * g.ex + l] = v;
        }
    }
}

// Grids with poles or TFSF planes (EXT, kernels of their own, so that the others
// keep their registers). What bounded them was, as for the rest, the chain of
// launches: 9.9 us a step at 160 x 96 TE with Drude cells, 18.3 with TFSF planes
// too, now 2.3 and 4.7; 3000 x 2000 78, 88 and (a Lorentz pole in most cells)
// 140 us, now 22, 35 and 108. J, P and the poles' coefficients of every cell lie
// in shared memory, where the rows of a warp that hold poles take them as packed
// pairs (looked up per cell through the material table, a Lorentz pole's 3000 x
// 2000 took 168 us: slower than the launches per half step). The corrections of
// the planes come from a table of the stretch's steps, formed by one launch
// ahead of its windows: they need only the auxiliary grids.
struct PlaneAct {
  int comp, lo[2], hi[2], ex;
  const float* at;  // value of window cell (0, 0) at the launch's first step
};
struct ExtShared {
  PlaneAct plane[2][kMaxPlanes];
  int nplane[2];
};

// one warp: lane 2 q + half
__device__ __forceinline__ void list_planes(const WinExt& x, ExtShared& es, int mode, int x0, int y0, int rows, int s, int lane) {
  const int q = lane >> 1, h = lane & 1;
  PlaneAct t{};
  bool in = false;
  if (q < x.nplanes) {
    const WinPlane& p = x.plane[q];
    const bool te = mode == kTE;
    // the component that a plane of this normal corrects
    if (h == 0) t.comp = te ? 1 - p.axis : 2;
    else t.comp = te ? 2 : 1 - p.axis;
    for (int d = 0; d < 2; d++) {
      t.lo[d] = max(p.lo[d] - (d ? y0 : x0), 0);
      t.hi[d] = min(p.hi[d] - (d ? y0 : x0), (d ? rows : kWinCols) - 1);
    }
    t.ex = p.hi[0] - p.lo[0] + 1;
    t.at = x.tfsf + (static_cast<long long>(s) * 2 + h) * x.tfsf_cells + p.off + static_cast<long long>(y0 - p.lo[1]) * t.ex + (x0 - p.lo[0]);
    in = p.axis < 2 && t.lo[0] <= t.hi[0] && t.lo[1] <= t.hi[1];
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const unsigned set = __ballot_sync(kAll, in && h == k);
    if (in && h == k) es.plane[k][__popc(set & ((1u << lane) - 1))] = t;
    if (lane == 0) es.nplane[k] = __popc(set);
  }
}

// a cell's entry in WinExt::disp: its poles, its material
__device__ __forceinline__ int poles_of(unsigned mid) { return mid >> 14; }
__device__ __forceinline__ const MatF32& material_of(const WinExt& x, unsigned mid) { return x.mats[mid & 0x3fffu]; }

// a correction v of E moves every pole's current by b * v
__device__ __noinline__ void kick_poles(const WinExt& x, float* at, int n, unsigned mids, pair_t v) {
  const float2 d = unpack(v);
#pragma unroll 1
  for (int c = 0; c < 2; c++) {
    const unsigned mid = c ? mids >> 16 : mids & 0xffffu;
    const int np = poles_of(mid);
    for (int q = 0; q < np; q++) {
      float* j = at + c + q * x.per * n;
      *j = __fmaf_rn(material_of(x, mid).b[q], c ? d.y : d.x, *j);
    }
  }
}

struct NoExt {};

// arrays of the window's cells in shared memory: the integrators, J and P, the
// coefficients
__host__ __device__ __forceinline__ int ext_arrays(int mode, const WinExt& x) {
  return 4 + (mode == kTE ? 2 : 1) * x.np * x.per + x.np * (1 + x.per);
}

}  // namespace

struct WinSpan {
  int x0, y0;                // first cell of the window
  int ox0, ox1, oy0, oy1;    // the cells it owns
};

// One window, T steps. GEN: the window touches the outer ring, the CPML, a
// source or a DFT region; otherwise every cell is interior with the plain
// coefficients and nothing else acts on it. True where a thread's samples of the
// outer ring are lost (sample_ring).
template <int MODE, bool XFIRST, bool GEN, bool CAP, int NW, int R, class Ext>
__device__ __forceinline__ bool window_run(const WinArgs& a, [[maybe_unused]] const Ext& x, [[maybe_unused]] const ExtShared* es,
                                           Shared<NW, R>& sh, float* psi, const WinSpan& sp, int T,
                                           int from, int slot, long long t0, pair_t (&f0)[R], pair_t (&f1)[R], pair_t (&f2)[R],
                                           pair_t (&ie)[R]) {
  constexpr bool TE = MODE == kTE;
  constexpr bool EXT = GEN && std::is_same<Ext, WinExt>::value;
  constexpr int N = kWinCols * Shared<NW, R>::kRows;  // cells of the window: one integrator array
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = w * R, c0 = sp.x0 + 2 * lane, j0 = sp.y0 + row0;
  const long long pitch = a.pitch;
  const bool col_in = c0 < a.nx;
  pair_t fxc[2], fyc[2];  // the plain coefficients
#pragma unroll
  for (int h = 0; h < 2; h++) {
    fxc[h] = fyc[h] = 0ull;
    if (!GEN) {
      fxc[h] = both(a.prof[h][0].F[sp.x0]);
      fyc[h] = both(a.prof[h][1].F[sp.y0]);
    }
  }
  // GEN. A cell of the outer ring (or beyond the grid) keeps its value: its
  // 1/eps is zero in the E half and its factor of the H half too; rows
  // outside the interior skip the H half. (A ring cell next to a non-finite
  // one becomes NaN here; it is sampled and written back as it was, and the
  // interior cells that see it are non-finite already.)
  const bool ok0 = !GEN || (c0 >= 1 && c0 <= a.nx - 2), ok1 = !GEN || c0 + 1 <= a.nx - 2;
  const pair_t minus = GEN ? pack(ok0 ? -1.f : 0.f, ok1 ? -1.f : 0.f) : both(-1.f);
  int xs = -1;  // the columns' place in the aligned x slab rows, or -1
  unsigned rows_in = 0, rows_y = 0;         // the warp's rows in the interior, in the y slab
  unsigned mine = 0, reg_e = 0, reg_h = 0;  // the entries and regions in the warp's rows
  float* const psi_at = psi + row0 * kWinCols + 2 * lane;  // [y of E, x of E, y of H, x of H][row][column]
  if (GEN) {
    if (col_in && a.pml[0]) {
      const int g4 = slab_group4(a.slab[0], c0 & ~3);
      if (g4 >= 0) xs = g4 + (c0 & 3);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int j = j0 + r;
      const int ys = sh.ys[row0 + r];
      const bool in = j >= 1 && j <= a.ny - 2;
      const float2 e = unpack(ie[r]);
      ie[r] = pack(in && ok0 ? e.x : 0.f, in && ok1 ? e.y : 0.f);
      // zero outside the slabs, whose coefficients are zero too
      pair_t p[4] = {0, 0, 0, 0};
      if (ys >= 0 && col_in) {
        p[0] = load_l2(a.psi[from][0] + ys * pitch + c0);
        p[2] = load_l2(a.psi[from][2] + ys * pitch + c0);
      }
      if (in && xs >= 0) {
        p[1] = load_l2(a.psi[from][1] + static_cast<long long>(j) * a.slab[0].W4 + xs);
        p[3] = load_l2(a.psi[from][3] + static_cast<long long>(j) * a.slab[0].W4 + xs);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) store_pair(psi_at + r * kWinCols + q * N, p[q]);
      if (ys >= 0) rows_y |= 1u << r;
      if (in) rows_in |= 1u << r;
    }
    for (int k = 0; k < sh.nentry; k++)
      if (sh.entry[k].hi[1] >= row0 && sh.entry[k].lo[1] < row0 + R) mine |= 1u << k;
    for (int k = 0; k < sh.nreg[0]; k++)
      if (sh.reg[0][k].hi[1] >= row0 && sh.reg[0][k].lo[1] < row0 + R) reg_e |= 1u << k;
    for (int k = 0; k < sh.nreg[1]; k++)
      if (sh.reg[1][k].hi[1] >= row0 && sh.reg[1][k].lo[1] < row0 + R) reg_h |= 1u << k;
  }
  // EXT: the warp's rows with poles, its planes; J and P follow the integrators,
  // then the poles' coefficients a, b (and c) in every cell, zero without poles
  unsigned rows_p = 0, mine_p[2] = {0, 0};
  int npj = 0, per_comp = 0;  // arrays of a component
  const unsigned* mids = nullptr;
  float* const pj_at = psi_at + 4 * N;
  [[maybe_unused]] float* co_at = nullptr;
  if constexpr (EXT) {
    per_comp = x.np * x.per;
    npj = (TE ? 2 : 1) * per_comp;
    const int nco = (1 + x.per) * x.np;
    co_at = pj_at + npj * N;
    unsigned* const mid_at = reinterpret_cast<unsigned*>(psi + (4 + npj + nco) * N) + row0 * 32 + lane;
    mids = mid_at;
    if (x.np > 0) {
#pragma unroll 1
      for (int r = 0; r < R; r++) {
        unsigned m = mid_at[r * 32];  // both cells; none of the ring
        if (!(rows_in >> r & 1)) m = 0;
        if (!ok0) m &= 0xffff0000u;
        if (!ok1) m &= 0xffffu;
        mid_at[r * 32] = m;
        if (!__any_sync(kAll, m != 0)) continue;
        rows_p |= 1u << r;
        const int n0 = poles_of(m & 0xffffu), n1 = poles_of(m >> 16);
        for (int k = 0; k < npj; k++) {
          const int q = k % per_comp / x.per;
          float2 v = make_float2(0.f, 0.f);
          if (m) v = unpack(load_l2(x.pj[from][k] + static_cast<long long>(j0 + r) * pitch + c0));
          store_pair(pj_at + r * kWinCols + k * N, pack(q < n0 ? v.x : 0.f, q < n1 ? v.y : 0.f));
        }
        for (int q = 0; q < x.np; q++) {
          const MatF32* const m0 = q < n0 ? &material_of(x, m) : nullptr;
          const MatF32* const m1 = q < n1 ? &material_of(x, m >> 16) : nullptr;
          float* co = co_at + r * kWinCols + q * (1 + x.per) * N;
          store_pair(co, pack(m0 ? m0->a[q] : 0.f, m1 ? m1->a[q] : 0.f));
          store_pair(co + N, pack(m0 ? m0->b[q] : 0.f, m1 ? m1->b[q] : 0.f));
          if (x.per == 2) store_pair(co + 2 * N, pack(m0 ? -m0->c[q] : 0.f, m1 ? -m1->c[q] : 0.f));
        }
      }
    }
    for (int h = 0; h < 2; h++)
      for (int k = 0; k < es->nplane[h]; k++)
        if (es->plane[h][k].hi[1] >= row0 && es->plane[h][k].lo[1] < row0 + R) mine_p[h] |= 1u << k;
  }
  // sum of the currents of component q's poles in row r, and their update
  auto currents = [&](int q, int r) {
    pair_t s = 0;
    if constexpr (EXT) {
      const float* p = pj_at + q * per_comp * N + r * kWinCols;
      s = load_pair(p);
      if (x.np > 1) s = add2(s, load_pair(p + x.per * N));
    }
    return s;
  };
  // drude_current and lorentz_current (a Drude pole's c is zero; its P is not
  // written back); a cell without the pole keeps its zero whatever E is
  auto advance = [&](int comp, int r, pair_t e) {
    if constexpr (EXT) {
#pragma unroll 1
      for (int q = 0; q < x.np; q++) {
        float* const j = pj_at + (comp * per_comp + q * x.per) * N + r * kWinCols;
        const float* const co = co_at + q * (1 + x.per) * N + r * kWinCols;
        const pair_t jt = load_pair(j);
        pair_t v = fma2(load_pair(co), jt, mul2(load_pair(co + N), e));
        if (x.per == 2) {
          const pair_t pn = add2(load_pair(j + N), jt);
          store_pair(j + N, pn);
          v = fma2(load_pair(co + 2 * N), pn, v);
        }
        const float2 now = unpack(v);
        const unsigned m = mids[r * 32];
        store_pair(j, pack(q < poles_of(m & 0xffffu) ? now.x : 0.f, q < poles_of(m >> 16) ? now.y : 0.f));
      }
    }
  };
  // the planes' corrections of half h; fa and fb the (one or) two components
  auto planes = [&](int h, int st, pair_t (&fa)[R], int ca, pair_t (&fb)[R]) {
    if constexpr (EXT) {
#pragma unroll 1
      for (unsigned m = mine_p[h]; m; m &= m - 1) {
        const PlaneAct& t = es->plane[h][__ffs(m) - 1];
        const Cols c(2 * lane, t.lo[0], t.hi[0]);
        const int lo = t.lo[1] - row0, hi = t.hi[1] - row0;
        const bool first = t.comp == ca;
        const float* p = t.at + st * 2 * x.tfsf_cells + static_cast<long long>(row0) * t.ex + 2 * lane;
        if (!__any_sync(kAll, c.k0 || c.k1)) continue;
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (r < lo || r > hi) continue;
          const pair_t v = pack(c.k0 ? __ldcg(p + static_cast<long long>(r) * t.ex) : 0.f,
                                c.k1 ? __ldcg(p + static_cast<long long>(r) * t.ex + 1) : 0.f);
          if (first) fa[r] = add2(fa[r], v);
          else fb[r] = add2(fb[r], v);
          if (h == 0 && (rows_p >> r & 1)) kick_poles(x, pj_at + (first ? 0 : 1) * per_comp * N + r * kWinCols, N, mids[r * 32], v);
        }
      }
    }
  };
  // which terms the warp's update has, alike for its lanes: x slab, y slab,
  // flux sources (the update is instantiated for each, free of branches)
  const bool has_x = GEN && __any_sync(kAll, xs >= 0), has_y = GEN && rows_y != 0;
  const bool has_flux = GEN && (mine & (sh.kinds[0][2] | sh.kinds[1][2]));
  sh.edge_h[w + 1][lane] = TE ? f2[R - 1] : f1[R - 1];
  __syncthreads();

  // CAP: the curl term d of the owned design cells goes out every step
  unsigned cap_rows = 0;
  Cols cap_cols(c0, max(a.dlo[0], sp.ox0), min(a.dhi[0], sp.ox1 - 1));
  const int cap_w = a.dhi[0] - a.dlo[0] + 1;
  const long long cap_step = static_cast<long long>(cap_w) * (a.dhi[1] - a.dlo[1] + 1);
  float* cap = nullptr;
  if (CAP) {
    cap = a.cap + t0 * cap_step + static_cast<long long>(j0 - a.dlo[1]) * cap_w + (c0 - a.dlo[0]);
#pragma unroll
    for (int r = 0; r < R; r++)
      if (j0 + r >= max(a.dlo[1], sp.oy0) && j0 + r <= min(a.dhi[1], sp.oy1 - 1)) cap_rows |= 1u << r;
  }
  auto flux = [&](int h, int comp, int r, int st, pair_t& d) {
#pragma unroll 1
    for (unsigned m = mine & sh.kinds[h][2]; m; m &= m - 1) {
      const int k = __ffs(m) - 1;
      const Entry& e = sh.entry[k];
      if (e.comp != comp || e.lo[1] != row0 + r) continue;
      const Cols c(2 * lane, e.lo[0], e.lo[0]);
      if (c.k0 || c.k1) d = add2(d, masked(sh.put[k][st], c.k0, c.k1));
    }
  };
  // One half step of the rows r0 .. r1 - 1. X, Y: the curl terms gain psi*G
  // and psi becomes B*psi + C*raw, the x slab by columns, the y slab by rows
  auto e_rows = [&](auto X, auto Y, auto FL, auto PO, int r0, int r1, pair_t below0, int st) {
    const pair_t fx = GEN ? sh.xp[0][0][lane] : fxc[0];
    pair_t bx = 0, cx = 0, gx = 0;
    if (X.value) {
      bx = sh.xp[0][1][lane];
      cx = sh.xp[0][2][lane];
      gx = sh.xp[0][3][lane];
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r < r0 || r >= r1) continue;
      const pair_t below = r == 0 ? below0 : (TE ? f2[r > 0 ? r - 1 : 0] : f1[r > 0 ? r - 1 : 0]);
      // the x neighbours: own first column and the last of the lane before
      const float2 h = unpack(f2[r]);
      const pair_t left = pack(__shfl_up_sync(kAll, h.y, 1), h.x);
      const pair_t fy = GEN ? sh.yp[0][0][row0 + r] : fyc[0];
      float* const py = psi_at + r * kWinCols;
      float* const px = py + N;
      if (TE) {
        const pair_t rxy = sub2(f2[r], below), ryx = sub2(left, f2[r]);
        pair_t dx = mul2(fy, rxy), dy = mul2(fx, ryx);
        if (Y.value) {
          const pair_t p = load_pair(py);
          dx = fma2(p, sh.yp[0][3][row0 + r], dx);
          store_pair(py, dot2(sh.yp[0][1][row0 + r], p, sh.yp[0][2][row0 + r], rxy));
        }
        if (X.value) {
          const pair_t p = load_pair(px);
          dy = fma2(p, gx, dy);
          store_pair(px, dot2(bx, p, cx, ryx));
        }
        if (FL.value) {
          flux(0, 0, r, st, dx);
          flux(0, 1, r, st, dy);
        }
        const bool poles = PO.value && (rows_p >> r & 1);
        if (poles) {
          dx = sub2(dx, currents(0, r));
          dy = sub2(dy, currents(1, r));
        }
        f0[r] = fma2(ie[r], dx, f0[r]);
        f1[r] = fma2(ie[r], dy, f1[r]);
        if (poles) {
          advance(0, r, f0[r]);
          advance(1, r, f1[r]);
        }
      } else {
        const pair_t rzx = sub2(f2[r], left), rzy = sub2(below, f1[r]);
        pair_t dz = dot2(fx, rzx, fy, rzy);
        if (CAP && (cap_rows >> r & 1)) {
          const float2 d = unpack(dz);
          if (cap_cols.k0) cap[r * cap_w] = d.x;
          if (cap_cols.k1) cap[r * cap_w + 1] = d.y;
        }
        auto xterm = [&] {
          const pair_t p = load_pair(px);
          dz = fma2(p, gx, dz);
          store_pair(px, dot2(bx, p, cx, rzx));
        };
        if (X.value && XFIRST) xterm();
        if (Y.value) {
          const pair_t p = load_pair(py);
          dz = fma2(p, sh.yp[0][3][row0 + r], dz);
          store_pair(py, dot2(sh.yp[0][1][row0 + r], p, sh.yp[0][2][row0 + r], rzy));
        }
        if (X.value && !XFIRST) xterm();
        if (FL.value) flux(0, 2, r, st, dz);
        const bool poles = PO.value && (rows_p >> r & 1);
        if (poles) dz = sub2(dz, currents(0, r));
        f0[r] = fma2(ie[r], dz, f0[r]);
        if (poles) advance(0, r, f0[r]);
      }
    }
  };
  auto h_rows = [&](auto X, auto Y, auto FL, int r0, int r1, pair_t top, int st) {
    const pair_t fx = GEN ? sh.xp[1][0][lane] : fxc[1];
    pair_t bx = 0, cx = 0, gx = 0;
    if (X.value) {
      bx = sh.xp[1][1][lane];
      cx = sh.xp[1][2][lane];
      gx = sh.xp[1][3][lane];
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r < r0 || r >= r1) continue;
      const pair_t above = r < R - 1 ? f0[r < R - 1 ? r + 1 : r] : top;
      // the x neighbours: own second column and the first of the lane after
      const pair_t ey = TE ? f1[r] : f0[r];
      const float2 e = unpack(ey);
      const pair_t right = pack(e.y, __shfl_down_sync(kAll, e.x, 1));
      const pair_t fy = GEN ? sh.yp[1][0][row0 + r] : fyc[1];
      const bool in = !GEN || (rows_in >> r & 1);
      float* const py = psi_at + r * kWinCols + 2 * N;
      float* const px = py + N;
      if (TE) {
        const pair_t rzx = sub2(right, ey), rzy = sub2(f0[r], above);
        pair_t dz = dot2(fx, rzx, fy, rzy);
        auto xterm = [&] {
          const pair_t p = load_pair(px);
          dz = fma2(p, gx, dz);
          store_pair(px, dot2(bx, p, cx, rzx));
        };
        if (X.value && XFIRST) xterm();
        if (Y.value) {
          const pair_t p = load_pair(py);
          dz = fma2(p, sh.yp[1][3][row0 + r], dz);
          store_pair(py, dot2(sh.yp[1][1][row0 + r], p, sh.yp[1][2][row0 + r], rzy));
        }
        if (X.value && !XFIRST) xterm();
        if (FL.value) flux(1, 2, r, st, dz);
        if (in) f2[r] = fma2(dz, minus, f2[r]);
      } else {
        const pair_t rxy = sub2(above, ey), ryx = sub2(ey, right);
        pair_t dx = mul2(fy, rxy), dy = mul2(fx, ryx);
        if (Y.value) {
          const pair_t p = load_pair(py);
          dx = fma2(p, sh.yp[1][3][row0 + r], dx);
          store_pair(py, dot2(sh.yp[1][1][row0 + r], p, sh.yp[1][2][row0 + r], rxy));
        }
        if (X.value) {
          const pair_t p = load_pair(px);
          dy = fma2(p, gx, dy);
          store_pair(px, dot2(bx, p, cx, ryx));
        }
        if (FL.value) {
          flux(1, 0, r, st, dx);
          flux(1, 1, r, st, dy);
        }
        if (in) {
          f1[r] = fma2(dx, minus, f1[r]);
          f2[r] = fma2(dy, minus, f2[r]);
        }
      }
    }
  };
  using Yes = std::true_type;
  using No = std::false_type;
  auto e_half = [&](auto X, auto Y, auto FL, int st) { e_rows(X, Y, FL, No(), 0, R, sh.edge_h[w][lane], st); };
  // warps with poles: with and without the other terms
  auto e_half_poles = [&](auto all, int st) { e_rows(all, all, all, Yes(), 0, R, sh.edge_h[w][lane], st); };
  auto h_half = [&](auto X, auto Y, auto FL, int st) { h_rows(X, Y, FL, 0, R, sh.edge_e[w + 1][lane], st); };

#pragma unroll 1
  for (int st = 0; st < T; st++) {
    // ---- E half
    if (GEN && __builtin_expect(mine != 0, 0))
      apply_entries(sh.entry, mine & (sh.kinds[0][0] | sh.kinds[0][1]), sh.undo, st, row0, lane, f0, TE ? 0 : 2, f1);
    bool done = false;
    if constexpr (EXT) {
      if (rows_p) {
        done = true;
        if (has_x || has_y || has_flux) e_half_poles(Yes(), st);
        else e_half_poles(No(), st);
      }
    }
    if (EXT && done) {
    } else if constexpr (!GEN) e_half(No(), No(), No(), st);
    else if (__builtin_expect(has_flux, 0)) e_half(Yes(), Yes(), Yes(), st);
    else if (has_x && has_y) e_half(Yes(), Yes(), No(), st);
    else if (has_x) e_half(Yes(), No(), No(), st);
    else if (has_y) e_half(No(), Yes(), No(), st);
    else e_half(No(), No(), No(), st);
    if (GEN && __builtin_expect(mine != 0, 0))
      apply_entries(sh.entry, mine & sh.kinds[0][1], sh.put, st, row0, lane, f0, TE ? 0 : 2, f1);
    if (EXT && __builtin_expect(mine_p[0] != 0, 0)) planes(0, st, f0, TE ? 0 : 2, f1);
    if (GEN && __builtin_expect(mine != 0, 0))
      apply_entries(sh.entry, mine & sh.kinds[0][0], sh.put, st, row0, lane, f0, TE ? 0 : 2, f1);
    sh.edge_e[w][lane] = f0[0];
    if (GEN && __builtin_expect(reg_e != 0, 0))
      sample_regions(sh.reg[0], reg_e, (slot + st) * a.dft_pts[0], row0, lane, f0, TE ? 0 : 2, f1);
    if (CAP) cap += cap_step;
    __syncthreads();
    // ---- H half
    if (GEN && __builtin_expect(mine != 0, 0)) {
      const unsigned set = mine & (sh.kinds[1][0] | sh.kinds[1][1]);
      if (TE) apply_entries(sh.entry, set, sh.undo, st, row0, lane, f2, 2, f2);
      else apply_entries(sh.entry, set, sh.undo, st, row0, lane, f1, 0, f2);
    }
    if constexpr (!GEN) h_half(No(), No(), No(), st);
    else if (__builtin_expect(has_flux, 0)) h_half(Yes(), Yes(), Yes(), st);
    else if (has_x && has_y) h_half(Yes(), Yes(), No(), st);
    else if (has_x) h_half(Yes(), No(), No(), st);
    else if (has_y) h_half(No(), Yes(), No(), st);
    else h_half(No(), No(), No(), st);
    if (GEN && __builtin_expect((EXT ? mine | mine_p[1] : mine) != 0, 0)) {
      for (int kind = 1; kind >= 0; kind--) {
        if (TE) apply_entries(sh.entry, mine & sh.kinds[1][kind], sh.put, st, row0, lane, f2, 2, f2);
        else apply_entries(sh.entry, mine & sh.kinds[1][kind], sh.put, st, row0, lane, f1, 0, f2);
        if (EXT && kind == 1 && mine_p[1]) {
          if (TE) planes(1, st, f2, 2, f2);
          else planes(1, st, f1, 0, f2);
        }
      }
    }
    sh.edge_h[w + 1][lane] = TE ? f2[R - 1] : f1[R - 1];
    if (GEN && __builtin_expect(reg_h != 0, 0)) {
      if (TE) sample_regions(sh.reg[1], reg_h, (slot + st) * a.dft_pts[1], row0, lane, f2, 2, f2);
      else sample_regions(sh.reg[1], reg_h, (slot + st) * a.dft_pts[1], row0, lane, f1, 0, f2);
    }
    __syncthreads();
  }

  // a sampled cell of the ring once NaN stays so for the launch (a batch samples
  // nothing; the adjoint's forward and EXT have launch_window_ring: the check cost
  // their kernels 4%)
  bool lost = false;
  if (GEN && XFIRST && !CAP && !EXT && __builtin_expect((reg_e | reg_h) != 0, 0)) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const float2 u[3] = {unpack(f0[r]), unpack(f1[r]), unpack(f2[r])};
      const bool row = rows_in >> r & 1;
#pragma unroll
      for (int q = 0; q < 3; q++) lost = lost || (!(row && ok0) && isnan(u[q].x)) || (!(row && ok1) && isnan(u[q].y));
    }
  }

  // the exact cells, into the other copy of the state
  if (c0 < sp.ox0 || c0 >= sp.ox1) return lost;
  const int to = 1 - from;
  // a pair with the halves that hold no interior cell as they were
  auto put = [&](const float* was, float* now, long long at, pair_t v, bool row_ok) {
    if (GEN && !(row_ok && ok0 && ok1)) {
      const float2 o = unpack(load_l2(was + at)), n = unpack(v);
      v = pack(row_ok && ok0 ? n.x : o.x, row_ok && ok1 ? n.y : o.y);
    }
    store_pair(now + at, v);
  };
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int j = j0 + r;
    if (j < sp.oy0 || j >= sp.oy1) continue;
    const long long c = j * pitch + c0;
    const bool in = !GEN || (rows_in >> r & 1);
    put(a.f[from][0], a.f[to][0], c, f0[r], in);
    put(a.f[from][1], a.f[to][1], c, f1[r], in);
    put(a.f[from][2], a.f[to][2], c, f2[r], in);
  }
  if (!GEN) return lost;
#pragma unroll 1
  for (int r = 0; r < R; r++) {
    const int j = j0 + r;
    if (j < sp.oy0 || j >= sp.oy1 || !(rows_in >> r & 1)) continue;
    if (rows_y >> r & 1) {
      const long long p = sh.ys[row0 + r] * pitch + c0;
      put(a.psi[from][0], a.psi[to][0], p, load_pair(psi_at + r * kWinCols), true);
      put(a.psi[from][2], a.psi[to][2], p, load_pair(psi_at + r * kWinCols + 2 * N), true);
    }
    if (xs >= 0) {
      const long long p = static_cast<long long>(j) * a.slab[0].W4 + xs;
      put(a.psi[from][1], a.psi[to][1], p, load_pair(psi_at + r * kWinCols + N), true);
      put(a.psi[from][3], a.psi[to][3], p, load_pair(psi_at + r * kWinCols + 3 * N), true);
    }
    if constexpr (EXT) {
      if (!(rows_p >> r & 1)) continue;
      const unsigned m = mids[r * 32];
      const long long p = j * pitch + c0;
#pragma unroll 1
      for (int c = 0; c < 2; c++) {
        const unsigned mid = c ? m >> 16 : m & 0xffffu;
        if (!mid) continue;
        const int n = material_of(x, mid).npoles;
        for (int k = 0; k < npj; k++) {
          const int kk = k % per_comp;
          if (kk / x.per < (n < 0 ? 1 : n) && !(n < 0 && kk % x.per)) x.pj[to][k][p + c] = pj_at[r * kWinCols + k * N + c];
        }
      }
    }
  }
  return lost;
}

// The window of tile `tile` of a grid: first cell, owned cells, what acts in
// it; then the steps.
template <int MODE, bool XFIRST, bool CAP, int NW, int R, class Ext>
__device__ __forceinline__ void window_tile(const WinArgs& a, const Ext& x, ExtShared* es, Shared<NW, R>& sh, float* psi, int tile, int T, int s, int from,
                                            int slot) {
  constexpr int rows = Shared<NW, R>::kRows;
  constexpr bool EXT = std::is_same<Ext, WinExt>::value;
  const int hx = (T + 1) & ~1;  // columns of a lane come in pairs: an even halo keeps them aligned
  const int ow = kWinCols - 2 * hx, oh = rows - 2 * T;
  const int tiles_x = window_tiles(a.nx, kWinCols, ow);
  const int tx = tile % tiles_x, ty = tile / tiles_x;
  WinSpan sp;
  sp.x0 = tx * ow;
  sp.y0 = ty * oh;
  sp.ox0 = tx == 0 ? 0 : sp.x0 + hx;
  sp.oy0 = ty == 0 ? 0 : sp.y0 + T;
  sp.ox1 = sp.x0 + kWinCols >= a.nx ? a.nx : sp.x0 + kWinCols - hx;
  sp.oy1 = sp.y0 + rows >= a.ny ? a.ny : sp.y0 + rows - T;
  const int tid = threadIdx.x;

  // what no earlier launch writes: profiles, sources, regions, 1/eps
  if (tid < rows) {
    const int j = sp.y0 + tid;
    const bool rin = j >= 1 && j <= a.ny - 2;
    const int ys = rin && a.pml[1] ? slab_index(a.slab[1], j) : -1;
    sh.ys[tid] = ys;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      sh.yp[h][0][tid] = both(rin ? a.prof[h][1].F[j] : 0.f);
      sh.yp[h][1][tid] = both(ys >= 0 ? a.prof[h][1].B[j] : 0.f);
      sh.yp[h][2][tid] = both(ys >= 0 ? a.prof[h][1].C[j] : 0.f);
      sh.yp[h][3][tid] = both(ys >= 0 ? a.prof[h][1].G[j] : 0.f);
    }
  } else if (tid >= 64 && tid < 96) {
    const int l = tid - 64, c0 = sp.x0 + 2 * l;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const bool in = c0 < a.nx;
      sh.xp[h][0][l] = in ? load_pair(a.prof[h][0].F + c0) : 0ull;
      sh.xp[h][1][l] = in ? load_pair(a.prof[h][0].B + c0) : 0ull;
      sh.xp[h][2][l] = in ? load_pair(a.prof[h][0].C + c0) : 0ull;
      sh.xp[h][3][l] = in ? load_pair(a.prof[h][0].G + c0) : 0ull;
    }
    // no warp writes these: the rows beyond the window's first and last
    sh.edge_h[0][l] = 0ull;
    sh.edge_e[NW][l] = 0ull;
  } else if (tid >= 96 && tid < 128) {
    list_entries<NW, R>(a, sh, sp.x0, sp.y0, tid & 31);
  } else if (tid >= 128 && tid < 192) {
    // the DFT regions with cells that the window owns
    const int h = tid < 160 ? 0 : 1, lane = tid & 31;
    Region o{};
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
  } else if (tid >= 192 && tid < 224) {
    if constexpr (EXT) list_planes(x, *es, MODE, sp.x0, sp.y0, rows, s, tid & 31);
  }
  // TE: Ex, Ey, Hz; TM: Ez, Hx, Hy
  pair_t f0[R], f1[R], f2[R], ie[R];
  const int c0 = sp.x0 + 2 * (tid & 31), j0 = sp.y0 + (tid >> 5) * R;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const bool in = c0 < a.nx && j0 + r < a.ny;
    ie[r] = both(a.ie0);
    if (a.ie) ie[r] = in ? load_pair(a.ie + (j0 + r) * static_cast<long long>(a.pitch) + c0) : 0ull;
  }
  bool poles = false;
  if constexpr (EXT) {
    if (x.np > 0) {
      unsigned* const mids = reinterpret_cast<unsigned*>(psi + ext_arrays(MODE, x) * kWinCols * rows);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const bool in = c0 < a.nx && j0 + r < a.ny;
        const unsigned m = in ? *reinterpret_cast<const unsigned*>(x.disp + (j0 + r) * static_cast<long long>(a.pitch) + c0) : 0u;
        mids[((tid >> 5) * R + r) * 32 + (tid & 31)] = m;
        poles = poles || m != 0;
      }
    }
  }
  after_previous_launch();
  const long long t0 = a.ctrl->t + s;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const bool in = c0 < a.nx && j0 + r < a.ny;
    const long long c = (j0 + r) * static_cast<long long>(a.pitch) + c0;
    f0[r] = in ? load_l2(a.f[from][0] + c) : 0ull;
    f1[r] = in ? load_l2(a.f[from][1] + c) : 0ull;
    f2[r] = in ? load_l2(a.f[from][2] + c) : 0ull;
  }
  if (EXT) poles = __syncthreads_or(poles);
  else __syncthreads();
  entry_values<NW, R>(a, sh, T, t0, from);
  bool plain = sp.x0 >= a.plain[0][0] && sp.x0 + kWinCols - 1 <= a.plain[0][1] && sp.y0 >= a.plain[1][0] &&
                     sp.y0 + rows - 1 <= a.plain[1][1] && sh.nentry + sh.nreg[0] + sh.nreg[1] == 0;
  if constexpr (EXT) plain = plain && !poles && es->nplane[0] + es->nplane[1] == 0;
  bool lost = false;
  if (plain) window_run<MODE, XFIRST, false, CAP, NW, R>(a, x, es, sh, psi, sp, T, from, slot, t0, f0, f1, f2, ie);
  else lost = window_run<MODE, XFIRST, true, CAP, NW, R>(a, x, es, sh, psi, sp, T, from, slot, t0, f0, f1, f2, ie);
  // the soft sources' last values, by the window that owns the source cell
  if (tid < a.nsrc) {
    const SourceDev& q = a.src[tid];
    if ((q.target == 0 || q.target == 2) && q.i >= sp.ox0 && q.i < sp.ox1 && q.j >= sp.oy0 && q.j < sp.oy1)
      a.src_last[1 - from][tid] = table_value(q.vals, q.nvals, t0 + T - 1);
  }
  if (XFIRST && !CAP && !EXT && __builtin_expect(lost, 0)) sample_ring<MODE == kTE, R>(a, sh, sp.x0, sp.y0, T, from, slot);
}

template <int MODE, bool CAP, int NW, int R>
__global__ void __launch_bounds__(32 * NW, 2) window_kernel(const __grid_constant__ WinArgs a, int T, int s, int from,
                                                            int slot) {
  extern __shared__ __align__(16) float psi[];
  __shared__ Shared<NW, R> sh;
  let_next_launch_start();
  window_tile<MODE, true, CAP, NW, R>(a, NoExt{}, nullptr, sh, psi, blockIdx.x, T, s, from, slot);
}

template <int MODE, int NW, int R>
__global__ void __launch_bounds__(32 * NW, 2) window_ext_kernel(const __grid_constant__ WinArgs a, const __grid_constant__ WinExt x,
                                                                int T, int s, int from, int slot) {
  extern __shared__ __align__(16) float psi[];
  __shared__ Shared<NW, R> sh;
  __shared__ ExtShared es;
  let_next_launch_start();
  window_tile<MODE, true, false, NW, R>(a, x, &es, sh, psi, blockIdx.x, T, s, from, slot);
}

// a batch: item = (grid index << 24) | tile; the grid's arguments are copied
// into shared memory first (one round trip instead of one per member)
template <int MODE, int NW, int R>
__global__ void __launch_bounds__(32 * NW, 2) window_batch_kernel(const WinArgs* __restrict__ grids,
                                                                  const unsigned* __restrict__ items, int T, int s,
                                                                  int from) {
  extern __shared__ __align__(16) float psi[];
  __shared__ Shared<NW, R> sh;
  __shared__ __align__(16) char raw[sizeof(WinArgs)];
  let_next_launch_start();
  const unsigned w = items[blockIdx.x];
  const int4* src = reinterpret_cast<const int4*>(grids + (w >> 24));
  for (int q = threadIdx.x; q < static_cast<int>(sizeof(WinArgs) / 16); q += blockDim.x)
    reinterpret_cast<int4*>(raw)[q] = src[q];
  __syncthreads();
  window_tile<MODE, false, false, NW, R>(*reinterpret_cast<const WinArgs*>(raw), NoExt{}, nullptr, sh, psi, static_cast<int>(w & 0xffffffu), T, s,
                                  from, 0);
}

namespace {

template <int NW, int R, typename F, typename... A>
void window_go(F fn, int n, cudaStream_t st, A... args) {
  constexpr size_t bytes = 4 * kWinCols * NW * R * sizeof(float);
  once_per_device(reinterpret_cast<const void*>(fn), [&] {
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  });
  launch_chained(fn, dim3(n), dim3(32 * NW), bytes, st, args...);
}

}  // namespace

namespace {

__global__ void window_cells_kernel(const __grid_constant__ FusedArgs a, unsigned short* disp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.pitch || j >= a.ny) return;
  const long long c = static_cast<long long>(j) * a.pitch + i;
  int mid = 0;
  if (i < a.nx && a.ids) mid = a.ids[c];
  else if (i < a.nx && a.bids) mid = a.bids[(j >> a.bshift) * a.nbx + (i >> a.bshift)];
  const int n = i < a.nx ? a.mats[mid].npoles : 0;
  disp[c] = static_cast<unsigned short>(n == 0 ? 0 : (n < 0 ? 1 : n) << 14 | mid);
}

// A 64 x 64 cell block per CTA, its halves of 32 rows one after another
__device__ __forceinline__ bool has_poles(const MatF32& m) { return m.npoles != 0; }
__device__ __forceinline__ bool has_poles(const MatF64& m) { return m.kind >= 2; }
template <class Args, class Mat>
__global__ void __launch_bounds__(256) pole_blocks_kernel(const __grid_constant__ Args a, const Mat* mats, int pitch, unsigned* counts) {
  int found[2];
  for (int h = 0; h < 2; h++) {
    int any = 0;
    for (int q = threadIdx.x; q < 64 * 32; q += 256) {
      const int i = blockIdx.x * 64 + q % 64, j = blockIdx.y * 64 + h * 32 + q / 64;
      if (i >= a.nx || j >= a.ny) continue;
      int mid = 0;
      if (a.ids) mid = a.ids[static_cast<long long>(j) * pitch + i];
      else if (a.bids) mid = a.bids[(j >> a.bshift) * a.nbx + (i >> a.bshift)];
      any |= has_poles(mats[mid]);
    }
    found[h] = __syncthreads_or(any) != 0;
  }
  if (threadIdx.x != 0 || found[0] + found[1] == 0) return;
  atomicAdd(counts, found[0] + found[1]);
  atomicAdd(counts + 1, 1);
}

// the samples of the outer ring's cells in slots slot .. slot + n - 1, one region
// per blockIdx.y, a thread per point
__global__ void __launch_bounds__(256) window_ring_kernel(const __grid_constant__ WinArgs a, int mode, int h, int slot, int n) {
  const DftRegionDev& g = a.reg[h][blockIdx.y];
  const int q = blockIdx.x * 256 + threadIdx.x;
  if (q >= g.npts) return;
  const int i = g.lo[0] + q % g.ext[0], j = g.lo[1] + q / g.ext[0];
  if (i > 0 && i < a.nx - 1 && j > 0 && j < a.ny - 1) return;
  const bool te = mode == kTE;
  const float* f = a.f[0][h == 0 ? (te ? g.comp : 0) : (te ? 2 : 1 + g.comp)];
  const float v = f[j * static_cast<long long>(a.pitch) + i];
  for (int s = slot; s < slot + n; s++) a.dft_buf[h][s * a.dft_pts[h] + g.pt_off + q] = v;
}

size_t ext_bytes(int mode, const WinExt& x, int rows) {
  const size_t cells = static_cast<size_t>(kWinCols) * rows;
  return ext_arrays(mode, x) * cells * sizeof(float) + (x.np > 0 ? cells * sizeof(unsigned short) : 0);
}

template <int NW, int R, typename F>
void window_ext_go(F fn, int mode, int n, cudaStream_t st, const WinArgs& a, const WinExt& x, int T, int s, int from, int slot) {
  once_per_device(reinterpret_cast<const void*>(fn), [&] {
    WinExt most{};
    // (windows of 64 rows hold one Drude pole at most)
    most.np = most.per = NW * R == 64 ? 1 : 2;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ext_bytes(mode, most, NW * R)));
  });
  launch_chained(fn, dim3(n), dim3(32 * NW), ext_bytes(mode, x, NW * R), st, a, x, T, s, from, slot);
}

}  // namespace

int launch_window_cells(const FusedArgs& a, unsigned short* disp, cudaStream_t s) {
  window_cells_kernel<<<dim3((a.pitch + 31) / 32, (a.ny + 7) / 8), dim3(32, 8), 0, s>>>(a, disp);
  return 1;
}

int launch_pole_blocks(const FusedArgs& a, unsigned* counts, cudaStream_t s) {
  pole_blocks_kernel<<<dim3((a.nx + 63) / 64, (a.ny + 63) / 64), 256, 0, s>>>(a, a.mats, a.pitch, counts);
  return 1;
}

int launch_pole_blocks(const PlainArgs& a, unsigned* counts, cudaStream_t s) {
  pole_blocks_kernel<<<dim3((a.nx + 63) / 64, (a.ny + 63) / 64), 256, 0, s>>>(a, a.mats, a.nx, counts);
  return 1;
}

int launch_window_ring(int mode, const WinArgs& a, const long long (&max_pts)[2], int slot, int n, cudaStream_t s) {
  int launches = 0;
  for (int h = 0; h < 2; h++) {
    if (a.nreg[h] == 0) continue;
    window_ring_kernel<<<dim3(static_cast<unsigned>((max_pts[h] + 255) / 256), a.nreg[h]), 256, 0, s>>>(a, mode, h, slot, n);
    launches++;
  }
  return launches;
}

int launch_window(int mode, const WinArgs& a, const WinExt* x, int rows, int T, int s, int from, int slot, cudaStream_t st) {
  const int n = window_count(a.nx, a.ny, rows, T);
  if (x) {
    auto ext = [&](auto small, auto large) {
      if (rows == 32) window_ext_go<16, 2>(small, mode, n, st, a, *x, T, s, from, slot);
      else window_ext_go<16, 4>(large, mode, n, st, a, *x, T, s, from, slot);
    };
    if (mode == kTE) ext(window_ext_kernel<kTE, 16, 2>, window_ext_kernel<kTE, 16, 4>);
    else ext(window_ext_kernel<kTM, 16, 2>, window_ext_kernel<kTM, 16, 4>);
    return 1;
  }
  auto go = [&](auto small, auto large) {
    if (rows == 32) window_go<16, 2>(small, n, st, a, T, s, from, slot);
    else window_go<16, 4>(large, n, st, a, T, s, from, slot);
  };
  if (mode == kTE) go(window_kernel<kTE, false, 16, 2>, window_kernel<kTE, false, 16, 4>);
  else if (a.cap) go(window_kernel<kTM, true, 16, 2>, window_kernel<kTM, true, 16, 4>);
  else go(window_kernel<kTM, false, 16, 2>, window_kernel<kTM, false, 16, 4>);
  return 1;
}

int launch_window_batch(int mode, const WinArgs* grids, const unsigned* items, int nitems, int T, int s, int from,
                        cudaStream_t st) {
  if (nitems <= 0) return 0;
  if (mode == kTE) window_go<16, 4>(window_batch_kernel<kTE, 16, 4>, nitems, st, grids, items, T, s, from);
  else window_go<16, 4>(window_batch_kernel<kTM, 16, 4>, nitems, st, grids, items, T, s, from);
  return 1;
}

}  // namespace fdtdb
