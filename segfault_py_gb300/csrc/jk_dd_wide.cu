// jk_dd_wide.cu -- double-float J/K kernels with tdd_wide lanes per quartet
// (classes.h): builds too small to fill the GPU, whose long quartets run
// latency-bound with the FP64 lane count.  Its own translation unit so that
// the build compiles it beside jk_dd.cu.
#include "classes.h"
#include "launch.h"

namespace sf {

template <int LA, int LB, int LC, int LD, int T>
static cudaError_t run_jk_dd_wide(const KParams &kp, const ClassWork *w, int nw, const dd *D, double *Jh, double *Kh,
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

cudaError_t launch_jk_dd_wide(int cls, const KParams &kp, const ClassWork *w, int nw, const dd *D, double *Jh, double *Kh,
                              cudaStream_t st) {
  switch (cls) {
#define SF_CASE(id, la, lb, lc, ld, t64, t32) \
  case id: return run_jk_dd_wide<la, lb, lc, ld, tdd_wide(la, lb, lc, ld, t64)>(kp, w, nw, D, Jh, Kh, st);
    SF_CLASS_LIST(SF_CASE)
#undef SF_CASE
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t prepare_jk_dd_wide() {
  cudaError_t e = cudaSuccess;
#define SF_PREP(id, la, lb, lc, ld, t64, t32)                                       \
  if (e == cudaSuccess)                                                             \
    e = prep_smem(jk_kernel<la, lb, lc, ld, dd, tdd_wide(la, lb, lc, ld, t64)>,     \
                  jk_smem<la, lb, lc, ld, dd, tdd_wide(la, lb, lc, ld, t64)>());
  SF_CLASS_LIST(SF_PREP)
#undef SF_PREP
  return e;
}

}  // namespace sf
