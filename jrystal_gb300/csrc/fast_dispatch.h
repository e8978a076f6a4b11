// Dispatch into the register-resident slab kernels of k_fft_fast.cu.
#pragma once
#include "plan.h"

namespace jrg {
namespace fast {
enum Op { OP_PLANE_INV = 0, OP_LINE_DENSITY, OP_LINE_APPLY_V, OP_PLANE_FWD };
struct Args {
  const void* in;
  void* out;
  const void* aux;      // coefficients (plane fwd) or V(r) (apply_v)
  const double* w;
  double wscale;        // density weight scale, or the FFT scale of plane fwd
  int band0, nbands, bands_per_group;
  double* gscale;       // density: per band group, the FP64 factor of its partial
  const int* bad;       // density, column kernels: nbad flags per band group (group_weights)
  int nbad;
};
// 1: launched, 0: grid not covered (use the generic kernels), <0: -status
template <typename R> int dispatch(const jrg_plan* P, int op, const Args& a, cudaStream_t st);
// dense batched 3-D transform of cubic grids (same return convention)
template <typename R>
int dispatch_dense(const FftAxis* ax, const C_t<R>* tw, int batch, int dir, bool real_in,
                   const void* in, C_t<R>* scratch, C_t<R>* out, double scale, cudaStream_t st);
// V_H(r) and the E_H partials of a density, cubic grids (same return convention)
template <typename R>
int dispatch_hartree(const jrg_plan* P, const void* rho, C_t<R>* mid, C_t<R>* rhog, double* slot_h, int nslots,
                     double pref, double inv_n, const ChargeFix& cf, cudaStream_t st);
}  // namespace fast
namespace cols {
// column-first kernels of k_fft_cols.cu (same return convention); used when
// active(P), for every operation of a call
template <typename R> int dispatch(const jrg_plan* P, int op, const fast::Args& a, cudaStream_t st);
// whether the column-first kernels take the plan's grid (inside: the sphere lies in
// the window |i| < N/4 of all axes; pruned: the plane-first kernels leave out the
// known zeros of all axes)
bool covers(int prec, int nx, int ny, int nz, int nb, bool inside, bool pruned);
bool active(const jrg_plan* P);
}  // namespace cols
}  // namespace jrg
