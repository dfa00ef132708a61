// The TFSF corrections of the FP64 plain method (TFSFPlane::updateD / updateB,
// include/Source.hpp:442-619), for sources compiled with -fmad=false.
#pragma once
#include "internal.h"

namespace fdtdb {

__device__ __forceinline__ double interp_aux(const double* row, int L, double loc, double dx, double shift) {
  // Aux1D::interpolateE / interpolateH (include/Source.hpp:442-458); the host
  // checked that every plane cell lands in 0 <= n <= L-2.
  double nd = static_cast<double>(L) / 2.0 + loc / dx - shift;
  unsigned long long n = static_cast<unsigned long long>(nd);
  double frac = nd - static_cast<double>(n);
  return (1.0 - frac) * row[n] + frac * row[n + 1];
}

// TFSFPlane::field_update::dir_update (Source.hpp:506-531) for flux I of type
// ft at cell idx, summed over d1, d2 as in field_update::get (:542-553).
template <int MODE>
__device__ __forceinline__ double tfsf_term(const PlaneDev& p, const AuxTab& aux, long long row, int ft, int I,
                                            const int (&idx)[3],
                            const Prof<double> (&prof)[2][3], double dx) {
  constexpr int dim = MODE == kThreeD ? 3 : 2;
  const int d1 = dir1(I);
  const int ds[2] = {d1, third(I, d1)};
  double terms[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int J = ds[q], K = third(I, J);
    const bool present = ft == 0 ? hasH(MODE, K) : hasE(MODE, K);
    if (!present) {
      terms[q] = 0.0;
      continue;
    }
    // CurlField offsets (FDTDConstants.hpp:680-744): H_K sits at -0.5 along K
    // only, E_K at -0.5 along the two axes other than K.
    double src[3];
#pragma unroll
    for (int d = 0; d < dim; d++) {
      const double off = ft == 0 ? (d == K ? -0.5 : 0.0) : (d == K ? 0.0 : -0.5);
      const double center = (static_cast<double>(idx[d]) - p.origin[d]) * dx;
      src[d] = center + off * dx;
    }
    double proj = 0;
#pragma unroll
    for (int d = 0; d < dim; d++) proj += p.k[d] * src[d];
    const double sv = ft == 0 ? interp_aux(aux.Htab + row * aux.L, aux.L, proj, dx, 0.5)
                              : interp_aux(aux.Etab + row * aux.L, aux.L, proj, dx, 0.0);
    const double Fdx = prof[ft][J].F[idx[J]];
    const double* pol = ft == 0 ? p.pol_h : p.pol_e;
    terms[q] = (levi(I, J, K) == 1 ? Fdx : -Fdx) * p.normal[J] * sv * pol[K];
  }
  return terms[0] + terms[1];
}

// what half step ft adds to flux I of cell idx for plane p: ft 0 (cc*dt) *
// TFSFPlane::updateD's term, ft 1 (-cc*dt) * updateB's term
template <int MODE>
__device__ __forceinline__ double tfsf_correction(const PlainArgs& a, const PlaneDev& p, long long row, int ft, int I,
                                                  const int (&idx)[3]) {
  const double dt = a.dt;
  const AuxTab& ax = a.aux[p.aux];
  return ft == 0 ? a.cc * dt * tfsf_term<MODE>(p, ax, row, 0, I, idx, a.prof, a.dx)
                 : -a.cc * dt * tfsf_term<MODE>(p, ax, row, 1, I, idx, a.prof, a.dx);
}

}  // namespace fdtdb
