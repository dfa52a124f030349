// jk_dd.cu -- double-float (dd) J/K kernels, per class: the accurate tier of
// the SF_PREC_MIXED_DF / SF_PREC_DF modes.  Lanes per quartet as the FP64
// kernels (same register footprint per value); the tdd_wide instantiations
// for builds too small to fill the GPU are in jk_dd_wide.cu.
#include "classes.h"
#include "launch.h"

namespace sf {

template <int LA, int LB, int LC, int LD, int T>
static cudaError_t run_jk_dd(const KParams &kp, const ClassWork *w, int nw, const dd *D, double *Jh, double *Kh,
                             cudaStream_t st) {
  ClassMulti m;
  m.n = 0;
  for (int k = 0; k < nw; ++k)
    if (w[k].n > 0 && !add_segment(m, w[k], T)) return cudaErrorInvalidValue;
  if (m.n == 0) return cudaSuccess;
  constexpr size_t smem = jk_smem<LA, LB, LC, LD, dd, T>();
  jk_kernel<LA, LB, LC, LD, dd, T><<<(unsigned)m.cta0[m.n], kBlock, smem, st>>>(kp, m, D, Jh, Kh);
  return cudaGetLastError();
}

// wide (the same for all segments) selects the tdd_wide lanes per quartet
// (compiled in jk_dd_wide.cu), else the FP64 lanes
cudaError_t launch_jk_dd(int cls, const KParams &kp, const ClassWork *w, int nw, const dd *D, double *Jh, double *Kh,
                         cudaStream_t st) {
  if (nw > 0 && w[0].wide) return launch_jk_dd_wide(cls, kp, w, nw, D, Jh, Kh, st);
  switch (cls) {
#define SF_CASE(id, la, lb, lc, ld, t64, t32) \
  case id: return run_jk_dd<la, lb, lc, ld, t64>(kp, w, nw, D, Jh, Kh, st);
    SF_CLASS_LIST(SF_CASE)
#undef SF_CASE
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t prepare_jk_dd() {
  cudaError_t e = cudaSuccess;
#define SF_PREP(id, la, lb, lc, ld, t64, t32)                                                           \
  if (e == cudaSuccess) e = prep_smem(jk_kernel<la, lb, lc, ld, dd, t64>, jk_smem<la, lb, lc, ld, dd, t64>());
  SF_CLASS_LIST(SF_PREP)
#undef SF_PREP
  if (e == cudaSuccess) e = prepare_jk_dd_wide();
  return e;
}

}  // namespace sf
