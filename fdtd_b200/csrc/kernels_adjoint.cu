// Discrete adjoint of the FP32 fused 2D TM step, for d(objective)/d(eps_r).
//
// Forward step t (kernels_fused.cu, TM, non-dispersive, design cells outside
// the CPML):
//   E:  Ez' = Ez + ie (Fx r_zx + Fy r_zy + Gx psi_zx + Gy psi_zy)
//       psi_zx' = Bx psi_zx + Cx r_zx,  r_zx = Hy - Hy[i-1]
//       psi_zy' = By psi_zy + Cy r_zy,  r_zy = -(Hx - Hx[j-1])
//   H:  Hx' = Hx - (Fy r_xy + Gy psi_xy),  psi_xy' = By psi_xy + Cy r_xy,  r_xy = Ez'[j+1] - Ez'
//       Hy' = Hy - (Fx r_yx + Gx psi_yx),  psi_yx' = Bx psi_yx + Cx r_yx,  r_yx = -(Ez'[i+1] - Ez')
// (E coefficients for the E half, H coefficients for the H half; sources are
// affine in the state and drop out). Reversing step t, given the adjoints
// (a*) of the state after it, is four per-cell gathers:
//   A1  H cell: rb_xy = -Fy aHx + Cy apsi_xy,  apsi_xy <- By apsi_xy - Gy aHx   (Hy likewise)
//   A2  E cell: aEz += rb_xy[j-1] - rb_xy - rb_yx[i-1] + rb_yx  (+ objective)
//   A3  E cell: db = ie aEz;  rb_zx = Fx db + Cx apsi_zx,  apsi_zx <- Bx apsi_zx + Gx db  (zy likewise);
//               grad += -aEz ie^2 d_t,  d_t = Fx r_zx + Fy r_zy of the forward step
//   A4  H cell: aHy += rb_zx - rb_zx[i+1];  aHx += -rb_zy + rb_zy[j+1]
// A1 and A4 read only the cell's own adjoints besides the rb arrays of the
// other half, so the reverse of step t runs as two launches: the H kernel
// (A4 of step t+1, then A1 of step t) and the E kernel (A2, A3 of step t).
// The objective J = sum_p |X_p|^2, X_p the DFT of Ez at the probe cells
// (sample n = t+1 after the E half of step t), adds
// dJ/dEz_p(n) = 2 Re(X_p e^{2 pi i f n}) to aEz at the probes.
// The gradient accumulates in FP64.
#include <type_traits>

#include "pairs.cuh"

namespace fdtdb {

namespace {

__device__ __forceinline__ bool interior(const AdjArgs& a, int i, int j) {
  return i >= 1 && i <= a.nx - 2 && j >= 1 && j <= a.ny - 2;
}

// 1/eps per cell as the E sweep takes it (material row, or the eps map)
__global__ void adj_inv_eps_kernel(const __grid_constant__ FusedArgs a, float* ie) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.nx || j >= a.ny) return;
  const long long c = static_cast<long long>(j) * a.pitch + i;
  int mid = 0;
  if (a.ids) mid = a.ids[c];
  else if (a.bids) mid = a.bids[(j >> a.bshift) * a.nbx + (i >> a.bshift)];
  const MatF32& m = a.mats[mid];
  float v = m.inv_eps;
  if (a.inv_eps_map && m.npoles == 0) {
    const float u = a.inv_eps_map[c];
    if (u > 0.f) v = u;
  }
  ie[c] = v;
}

// d_t of every design cell from the state at the start of step t
__global__ void adj_capture_kernel(const AdjArgs a, const float* __restrict__ hx, const float* __restrict__ hy,
                                   float* __restrict__ slot) {
  const int dw = a.dhi[0] - a.dlo[0] + 1;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= a.ndesign) return;
  const int i = a.dlo[0] + q % dw, j = a.dlo[1] + q / dw;
  const long long c = static_cast<long long>(j) * a.pitch + i;
  const float r_zx = hy[c] - hy[c - 1];
  const float r_zy = -(hx[c] - hx[c - a.pitch]);
  slot[q] = a.prof[0][0].F[i] * r_zx + a.prof[0][1].F[j] * r_zy;
}

__global__ void __launch_bounds__(256) adj_h_kernel(const AdjArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (!interior(a, i, j)) return;
  const long long c = static_cast<long long>(j) * a.pitch + i;
  // A4 of step t+1 (the rb_z arrays are zero before the first reversed step)
  const float ahx = a.ahx[c] + (-a.rzy[c] + a.rzy[c + a.pitch]);
  const float ahy = a.ahy[c] + (a.rzx[c] - a.rzx[c + 1]);
  a.ahx[c] = ahx;
  a.ahy[c] = ahy;
  // A1 of step t: Hx (curl along y), Hy (curl along x)
  float rxy = -a.prof[1][1].F[j] * ahx;
  const int sy = a.pml_axis[1] ? slab_index(a.slab[1], j) : -1;
  if (sy >= 0) {
    const long long p = static_cast<long long>(sy) * a.pitch + i;
    const float ps = a.apxy[p];
    rxy += a.prof[1][1].C[j] * ps;
    a.apxy[p] = a.prof[1][1].B[j] * ps - a.prof[1][1].G[j] * ahx;
  }
  float ryx = -a.prof[1][0].F[i] * ahy;
  const int sx = a.pml_axis[0] ? slab_index(a.slab[0], i) : -1;
  if (sx >= 0) {
    const long long p = static_cast<long long>(j) * a.slab[0].W + sx;
    const float ps = a.apyx[p];
    ryx += a.prof[1][0].C[i] * ps;
    a.apyx[p] = a.prof[1][0].B[i] * ps - a.prof[1][0].G[i] * ahy;
  }
  a.rxy[c] = rxy;
  a.ryx[c] = ryx;
}

// `back` counts the steps between this one and the last of the recomputed
// segment, whose end the step counter holds: n = t + 1 = ctrl->t - back
__global__ void __launch_bounds__(256) adj_e_kernel(const AdjArgs a, int back, const float* __restrict__ dslot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (!interior(a, i, j)) return;
  const long long c = static_cast<long long>(j) * a.pitch + i;
  const long long n = a.ctrl->t - back;
  // A2
  float v = a.rxy[c - a.pitch] - a.rxy[c] - a.ryx[c - 1] + a.ryx[c];
  if (i >= a.plo[0] && i <= a.phi[0] && j >= a.plo[1] && j <= a.phi[1]) {
    const long long q = static_cast<long long>(j - a.plo[1]) * (a.phi[0] - a.plo[0] + 1) + (i - a.plo[0]);
    double sn, cs;
    sincospi(2.0 * a.freq * static_cast<double>(n), &sn, &cs);
    v += static_cast<float>(2.0 * (a.X[2 * q] * cs - a.X[2 * q + 1] * sn));
  }
  const float ae = a.aez[c] + v;
  a.aez[c] = ae;
  // A3
  const float ie = a.ie[c];
  const float db = ie * ae;
  if (i >= a.dlo[0] && i <= a.dhi[0] && j >= a.dlo[1] && j <= a.dhi[1]) {
    const int q = (j - a.dlo[1]) * (a.dhi[0] - a.dlo[0] + 1) + (i - a.dlo[0]);
    const double die = ie;
    a.grad[q] += -static_cast<double>(ae) * die * die * static_cast<double>(dslot[q]);
  }
  float rx = a.prof[0][0].F[i] * db, ry = a.prof[0][1].F[j] * db;
  const int sx = a.pml_axis[0] ? slab_index(a.slab[0], i) : -1;
  if (sx >= 0) {
    const long long p = static_cast<long long>(j) * a.slab[0].W + sx;
    const float ps = a.apzx[p];
    rx += a.prof[0][0].C[i] * ps;
    a.apzx[p] = a.prof[0][0].B[i] * ps + a.prof[0][0].G[i] * db;
  }
  const int sy = a.pml_axis[1] ? slab_index(a.slab[1], j) : -1;
  if (sy >= 0) {
    const long long p = static_cast<long long>(sy) * a.pitch + i;
    const float ps = a.apzy[p];
    ry += a.prof[0][1].C[j] * ps;
    a.apzy[p] = a.prof[0][1].B[j] * ps + a.prof[0][1].G[j] * db;
  }
  a.rzx[c] = rx;
  a.rzy[c] = ry;
}

}  // namespace

// ---------------------------------------------------------------------------
// The reversed steps in windows: T steps per launch, as kernels_window.cu takes
// the forward ones (two columns per lane in packed pairs, R rows per warp, two
// copies of the state), with A1, A2, A3 and A4 of a step in one pass over the
// thread's rows. A step reads its neighbours' rb_xy (row below), rb_yx (column
// before), rb_zx (column after) and rb_zy (row above): the column ones are
// shuffles, the row ones pass through shared memory at a warp's edge rows
// (`edge_r`, `edge_y`), one barrier each. The forward's d_t of the owned design
// cells are read from memory a step ahead; their gradients are summed in
// shared memory in FP64, step by step as the launches per step do.
namespace {

using namespace pairs;

template <int NW, int R>
struct AdjShared {
  static constexpr int kRows = NW * R;
  pair_t edge_r[NW + 1][32];  // rb_xy of each warp's last row, one place up
  pair_t edge_y[NW + 1][32];  // rb_zy of each warp's first row
  pair_t xp[2][4][32];        // F, B, C, G of the columns (H, E half as 1, 0)
  pair_t yp[2][4][kRows];
};

template <bool GEN, int NW, int R>
__device__ __forceinline__ void adjoint_run(const AdjWinArgs& a, AdjShared<NW, R>& sh, float* psi, double* acc,
                                            int x0, int y0, int ox0, int ox1, int oy0, int oy1, int T, int t, int from) {
  constexpr int N = kWinCols * NW * R;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = w * R, c0 = x0 + 2 * lane, j0 = y0 + row0;
  const long long pitch = a.pitch;
  const bool col_in = c0 < a.nx;
  pair_t ez[R], hx[R], hy[R], ie[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const bool in = col_in && j0 + r < a.ny;
    const long long c = (j0 + r) * pitch + c0;
    ie[r] = in ? load_pair(a.ie + c) : 0ull;
    ez[r] = in ? load_l2(a.f[from][0] + c) : 0ull;
    hx[r] = in ? load_l2(a.f[from][1] + c) : 0ull;
    hy[r] = in ? load_l2(a.f[from][2] + c) : 0ull;
  }
  // GEN: the ring's adjoints stay zero (factor 0), rows outside the interior too
  const bool ok0 = !GEN || (c0 >= 1 && c0 <= a.nx - 2), ok1 = !GEN || c0 + 1 <= a.nx - 2;
  const pair_t one = pack(ok0 ? 1.f : 0.f, ok1 ? 1.f : 0.f);
  unsigned rows_in = ~0u, rows_y = 0;
  int xs = -1, ys[R];
  float* const psi_at = psi + row0 * kWinCols + 2 * lane;
  if (GEN) {
    if (col_in && a.pml[0]) {
      const int g4 = slab_group4(a.slab[0], c0 & ~3);
      if (g4 >= 0) xs = g4 + (c0 & 3);
    }
    rows_in = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int j = j0 + r;
      const bool in = j >= 1 && j <= a.ny - 2;
      ys[r] = in && a.pml[1] ? slab_index(a.slab[1], j) : -1;
      pair_t p[4] = {0, 0, 0, 0};
      if (ys[r] >= 0 && col_in) {
        p[0] = load_l2(a.psi[from][0] + ys[r] * pitch + c0);
        p[3] = load_l2(a.psi[from][3] + ys[r] * pitch + c0);
      }
      if (in && xs >= 0) {
        const long long at = static_cast<long long>(j) * a.slab[0].W4 + xs;
        p[1] = load_l2(a.psi[from][1] + at);
        p[2] = load_l2(a.psi[from][2] + at);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) store_pair(psi_at + r * kWinCols + q * N, p[q]);
      if (ys[r] >= 0) rows_y |= 1u << r;
      if (in) rows_in |= 1u << r;
    }
  }
  const bool has_x = GEN && __any_sync(kAll, xs >= 0), has_y = GEN && rows_y != 0;
  // the owned design cells and the probe cells of the thread
  const int dw = a.dhi[0] - a.dlo[0] + 1, pw = a.phi[0] - a.plo[0] + 1;
  const long long nd = static_cast<long long>(dw) * (a.dhi[1] - a.dlo[1] + 1);
  const long long np = static_cast<long long>(pw) * (a.phi[1] - a.plo[1] + 1);
  const Cols dc(c0, max(a.dlo[0], ox0), min(a.dhi[0], ox1 - 1)), pc(c0, a.plo[0], a.phi[0]);
  unsigned drows = 0, prows = 0;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int j = j0 + r;
    if (j >= max(a.dlo[1], oy0) && j <= min(a.dhi[1], oy1 - 1)) drows |= 1u << r;
    if (j >= a.plo[1] && j <= a.phi[1]) prows |= 1u << r;
  }
  const bool has_d = __any_sync(kAll, drows && (dc.k0 || dc.k1)), has_p = __any_sync(kAll, prows && (pc.k0 || pc.k1));
  const long long d_at = static_cast<long long>(j0 - a.dlo[1]) * dw + (c0 - a.dlo[0]);
  double* const acc_at = acc + row0 * kWinCols + 2 * lane;
  pair_t next[R];  // d of the step to come
  auto fetch = [&](int step) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      float x = 0.f, y = 0.f;
      if (drows >> r & 1) {
        const float* p = a.store + step * nd + d_at + r * dw;
        if (dc.k0) x = p[0];
        if (dc.k1) y = p[1];
      }
      next[r] = pack(x, y);
    }
  };
  if (has_d) {
    fetch(t);
#pragma unroll
    for (int r = 0; r < R; r++)
      if (drows >> r & 1) {
        if (dc.k0) acc_at[r * kWinCols] = a.grad[d_at + r * dw];
        if (dc.k1) acc_at[r * kWinCols + 1] = a.grad[d_at + r * dw + 1];
      }
  }
  pair_t fxc[2] = {0, 0}, fyc[2] = {0, 0};
  if (!GEN)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      fxc[h] = both(a.prof[h][0].F[x0]);
      fyc[h] = both(a.prof[h][1].F[y0]);
    }
  // A1 of one row: rb_xy (curl along y), the integrator's adjoint stepped back
  auto a1_xy = [&](auto Y, int r) {
    const pair_t fy = GEN ? sh.yp[1][0][row0 + r] : fyc[1];
    const pair_t minus_h = mul2(hx[r], both(-1.f));
    pair_t rxy = mul2(fy, minus_h);
    if (Y.value) {
      float* at = psi_at + r * kWinCols;
      const pair_t p = load_pair(at);
      rxy = fma2(sh.yp[1][2][row0 + r], p, rxy);
      store_pair(at, dot2(sh.yp[1][1][row0 + r], p, sh.yp[1][3][row0 + r], minus_h));
    }
    return rxy;
  };
  auto rows = [&](auto X, auto Y, auto D, auto PR, int step, pair_t top_rxy) {
    const pair_t fx_h = GEN ? sh.xp[1][0][lane] : fxc[1], fx_e = GEN ? sh.xp[0][0][lane] : fxc[0];
    pair_t below = sh.edge_r[w][lane], ry_before = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const pair_t rxy = r == R - 1 ? top_rxy : a1_xy(Y, r);
      const pair_t minus_h = mul2(hy[r], both(-1.f));
      pair_t ryx = mul2(fx_h, minus_h);
      if (X.value) {
        float* at = psi_at + r * kWinCols + N;
        const pair_t p = load_pair(at);
        ryx = fma2(sh.xp[1][2][lane], p, ryx);
        store_pair(at, dot2(sh.xp[1][1][lane], p, sh.xp[1][3][lane], minus_h));
      }
      // A2
      const float2 q = unpack(ryx);
      const pair_t left = pack(__shfl_up_sync(kAll, q.y, 1), q.x);
      pair_t v = add2(sub2(sub2(below, rxy), left), ryx);
      if (PR.value && (prows >> r & 1)) {
        const float* p = a.force + step * np + static_cast<long long>(j0 + r - a.plo[1]) * pw + (c0 - a.plo[0]);
        v = add2(v, pack(pc.k0 ? p[0] : 0.f, pc.k1 ? p[1] : 0.f));
      }
      ez[r] = fma2(v, rows_in >> r & 1 ? one : 0ull, ez[r]);
      below = rxy;
      // A3
      const pair_t db = mul2(ie[r], ez[r]);
      if (D.value && (drows >> r & 1)) {
        const float2 e = unpack(ez[r]), i = unpack(ie[r]), d = unpack(next[r]);
        if (dc.k0)
          acc_at[r * kWinCols] += -static_cast<double>(e.x) * static_cast<double>(i.x) * static_cast<double>(i.x) *
                                  static_cast<double>(d.x);
        if (dc.k1)
          acc_at[r * kWinCols + 1] += -static_cast<double>(e.y) * static_cast<double>(i.y) *
                                      static_cast<double>(i.y) * static_cast<double>(d.y);
      }
      const pair_t fy_e = GEN ? sh.yp[0][0][row0 + r] : fyc[0];
      pair_t rx = mul2(fx_e, db), ry = mul2(fy_e, db);
      if (X.value) {
        float* at = psi_at + r * kWinCols + 2 * N;
        const pair_t p = load_pair(at);
        rx = fma2(sh.xp[0][2][lane], p, rx);
        store_pair(at, dot2(sh.xp[0][1][lane], p, sh.xp[0][3][lane], db));
      }
      if (Y.value) {
        float* at = psi_at + r * kWinCols + 3 * N;
        const pair_t p = load_pair(at);
        ry = fma2(sh.yp[0][2][row0 + r], p, ry);
        store_pair(at, dot2(sh.yp[0][1][row0 + r], p, sh.yp[0][3][row0 + r], db));
      }
      if (r == 0) sh.edge_y[w][lane] = ry;
      // A4 of this row's Hy and of the row below's Hx
      const float2 x = unpack(rx);
      const pair_t right = pack(x.y, __shfl_down_sync(kAll, x.x, 1));
      hy[r] = fma2(sub2(rx, right), rows_in >> r & 1 ? one : 0ull, hy[r]);
      if (r > 0) hx[r > 0 ? r - 1 : 0] = fma2(sub2(ry, ry_before), rows_in >> (r - 1) & 1 ? one : 0ull, hx[r > 0 ? r - 1 : 0]);
      ry_before = ry;
    }
    return ry_before;
  };
  using Yes = std::true_type;
  using No = std::false_type;
  pair_t top_rxy = has_y ? a1_xy(Yes(), R - 1) : a1_xy(No(), R - 1);
  sh.edge_r[w + 1][lane] = top_rxy;
  __syncthreads();
#pragma unroll 1
  for (int st = 0; st < T; st++) {
    const int step = t - st;
    pair_t ry;
    if constexpr (GEN) {
      if (__builtin_expect(has_d || has_p, 0)) ry = rows(Yes(), Yes(), Yes(), Yes(), step, top_rxy);
      else if (has_x && has_y) ry = rows(Yes(), Yes(), No(), No(), step, top_rxy);
      else if (has_x) ry = rows(Yes(), No(), No(), No(), step, top_rxy);
      else if (has_y) ry = rows(No(), Yes(), No(), No(), step, top_rxy);
      else ry = rows(No(), No(), No(), No(), step, top_rxy);
    } else {
      if (has_p) ry = rows(No(), No(), Yes(), Yes(), step, top_rxy);
      else if (has_d) ry = rows(No(), No(), Yes(), No(), step, top_rxy);
      else ry = rows(No(), No(), No(), No(), step, top_rxy);
    }
    if (has_d && st + 1 < T) fetch(step - 1);
    __syncthreads();
    hx[R - 1] = fma2(sub2(sh.edge_y[w + 1][lane], ry), rows_in >> (R - 1) & 1 ? one : 0ull, hx[R - 1]);
    if (st + 1 < T) {
      top_rxy = has_y || (GEN && (has_d || has_p)) ? a1_xy(Yes(), R - 1) : a1_xy(No(), R - 1);
      sh.edge_r[w + 1][lane] = top_rxy;
      __syncthreads();
    }
  }
  if (has_d) {
#pragma unroll
    for (int r = 0; r < R; r++)
      if (drows >> r & 1) {
        if (dc.k0) a.grad[d_at + r * dw] = acc_at[r * kWinCols];
        if (dc.k1) a.grad[d_at + r * dw + 1] = acc_at[r * kWinCols + 1];
      }
  }
  if (c0 < ox0 || c0 >= ox1) return;
  const int to = 1 - from;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int j = j0 + r;
    if (j < oy0 || j >= oy1) continue;
    const long long c = j * pitch + c0;
    store_pair(a.f[to][0] + c, ez[r]);
    store_pair(a.f[to][1] + c, hx[r]);
    store_pair(a.f[to][2] + c, hy[r]);
    if (!GEN) continue;
    if (ys[r] >= 0) {
      store_pair(a.psi[to][0] + ys[r] * pitch + c0, load_pair(psi_at + r * kWinCols));
      store_pair(a.psi[to][3] + ys[r] * pitch + c0, load_pair(psi_at + r * kWinCols + 3 * N));
    }
    if (xs >= 0 && (rows_in >> r & 1)) {
      const long long at = static_cast<long long>(j) * a.slab[0].W4 + xs;
      store_pair(a.psi[to][1] + at, load_pair(psi_at + r * kWinCols + N));
      store_pair(a.psi[to][2] + at, load_pair(psi_at + r * kWinCols + 2 * N));
    }
  }
}

template <int NW, int R>
__global__ void __launch_bounds__(32 * NW, R == 2 ? 2 : 1) adjoint_window_kernel(const __grid_constant__ AdjWinArgs a, int T, int t,
                                                                    int from) {
  constexpr int rows = NW * R;
  extern __shared__ __align__(16) float psi[];
  __shared__ AdjShared<NW, R> sh;
  double* acc = reinterpret_cast<double*>(psi + 4 * kWinCols * rows);
  let_next_launch_start();
  const int hx = (T + 1) & ~1;
  const int ow = kWinCols - 2 * hx, oh = rows - 2 * T;
  const int tiles_x = window_tiles(a.nx, kWinCols, ow);
  const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
  const int x0 = tx * ow, y0 = ty * oh;
  const int ox0 = tx == 0 ? 0 : x0 + hx, oy0 = ty == 0 ? 0 : y0 + T;
  const int ox1 = x0 + kWinCols >= a.nx ? a.nx : x0 + kWinCols - hx;
  const int oy1 = y0 + rows >= a.ny ? a.ny : y0 + rows - T;
  const int tid = threadIdx.x;
  if (tid < rows) {
    const int j = y0 + tid;
    const bool rin = j >= 1 && j <= a.ny - 2, slab = rin && a.pml[1] && slab_index(a.slab[1], j) >= 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      sh.yp[h][0][tid] = both(rin ? a.prof[h][1].F[j] : 0.f);
      sh.yp[h][1][tid] = both(slab ? a.prof[h][1].B[j] : 0.f);
      sh.yp[h][2][tid] = both(slab ? a.prof[h][1].C[j] : 0.f);
      sh.yp[h][3][tid] = both(slab ? a.prof[h][1].G[j] : 0.f);
    }
  } else if (tid >= 64 && tid < 96) {
    const int l = tid - 64, c = x0 + 2 * l;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const bool in = c < a.nx;
      sh.xp[h][0][l] = in ? load_pair(a.prof[h][0].F + c) : 0ull;
      sh.xp[h][1][l] = in ? load_pair(a.prof[h][0].B + c) : 0ull;
      sh.xp[h][2][l] = in ? load_pair(a.prof[h][0].C + c) : 0ull;
      sh.xp[h][3][l] = in ? load_pair(a.prof[h][0].G + c) : 0ull;
    }
    sh.edge_r[0][l] = 0ull;
    sh.edge_y[NW][l] = 0ull;
  }
  after_previous_launch();
  __syncthreads();
  const bool plain = x0 >= a.plain[0][0] && x0 + kWinCols - 1 <= a.plain[0][1] && y0 >= a.plain[1][0] &&
                     y0 + rows - 1 <= a.plain[1][1];
  if (plain) adjoint_run<false, NW, R>(a, sh, psi, acc, x0, y0, ox0, ox1, oy0, oy1, T, t, from);
  else adjoint_run<true, NW, R>(a, sh, psi, acc, x0, y0, ox0, ox1, oy0, oy1, T, t, from);
}

__global__ void __launch_bounds__(256) adj_force_kernel(const double* __restrict__ X, double freq, int nprobe,
                                                        int nsteps, float* __restrict__ force) {
  const int t = blockIdx.x * 8 + threadIdx.x / 32;
  if (t >= nsteps) return;
  double sn, cs;
  sincospi(2.0 * freq * static_cast<double>(t + 1), &sn, &cs);
  for (int q = threadIdx.x % 32; q < nprobe; q += 32)
    force[static_cast<long long>(t) * nprobe + q] = static_cast<float>(2.0 * (X[2 * q] * cs - X[2 * q + 1] * sn));
}

template <int NW, int R>
void adjoint_window_go(const AdjWinArgs& a, int T, int t, int from, cudaStream_t s) {
  constexpr size_t bytes = kWinCols * NW * R * (4 * sizeof(float) + sizeof(double));
  auto fn = adjoint_window_kernel<NW, R>;
  once_per_device(reinterpret_cast<const void*>(fn), [&] {
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  });
  launch_chained(fn, dim3(window_count(a.nx, a.ny, NW * R, T)), dim3(32 * NW), bytes, s, a, T, t, from);
}

}  // namespace

int launch_adjoint_window(const AdjWinArgs& a, int rows, int T, int t, int from, cudaStream_t s) {
  if (rows == 32) adjoint_window_go<16, 2>(a, T, t, from, s);
  else adjoint_window_go<16, 4>(a, T, t, from, s);
  return 1;
}

int launch_adjoint_force(const double* X, double freq, int nprobe, int nsteps, float* force, cudaStream_t s) {
  adj_force_kernel<<<(nsteps + 7) / 8, 256, 0, s>>>(X, freq, nprobe, nsteps, force);
  return 1;
}

int launch_adjoint_inv_eps(const FusedArgs& fa, float* ie, cudaStream_t s) {
  dim3 block(32, 8), grid((fa.nx + 31) / 32, (fa.ny + 7) / 8);
  adj_inv_eps_kernel<<<grid, block, 0, s>>>(fa, ie);
  return 1;
}

int launch_adjoint_capture(const AdjArgs& a, const float* hx, const float* hy, float* slot, cudaStream_t s) {
  adj_capture_kernel<<<(a.ndesign + 255) / 256, 256, 0, s>>>(a, hx, hy, slot);
  return 1;
}

// the reverse of the step `back` steps before the one that ends at the
// device step counter
int launch_adjoint_step(const AdjArgs& a, int back, const float* dslot, cudaStream_t s) {
  dim3 block(32, 8), grid((a.nx + 31) / 32, (a.ny + 7) / 8);
  adj_h_kernel<<<grid, block, 0, s>>>(a);
  adj_e_kernel<<<grid, block, 0, s>>>(a, back, dslot);
  return 2;
}

}  // namespace fdtdb
