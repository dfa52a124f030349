// grad_f32.cu -- FP32 two-electron gradient kernels (FP64 accumulation), one per class.
#include <algorithm>

#include "classes.h"
#include "grad.cuh"
#include "launch.h"

namespace sf {

template <int LA, int LB, int LC, int LD>
static cudaError_t run_grad32(const KParams &kp, const ClassWork *w, int nw, const float *D, double *grad, cudaStream_t st) {
  constexpr int T = tgrad_r<float>(QC<LA, LB, LC, LD>::NABCD);
  ClassMulti m;
  if (!grad_segments(m, w, nw, T)) return cudaErrorInvalidValue;
  if (m.n == 0) return cudaSuccess;
  constexpr size_t smem = grad_smem<LA, LB, LC, LD, float>();
  grad_kernel<LA, LB, LC, LD, float, T><<<(unsigned)m.cta0[m.n], kBlock, smem, st>>>(kp, m, D, grad);
  return cudaGetLastError();
}

cudaError_t launch_grad_f32(int cls, const KParams &kp, const ClassWork *w, int nw, const float *D, double *grad,
                            cudaStream_t st) {
  switch (cls) {
#define SF_CASE(id, la, lb, lc, ld, t64, t32) \
  case id: return run_grad32<la, lb, lc, ld>(kp, w, nw, D, grad, st);
    SF_CLASS_LIST(SF_CASE)
#undef SF_CASE
    default: return cudaErrorInvalidValue;
  }
}

// work tables of every class for the FP64 / double-float and the FP32 lanes
void grad_tables(std::vector<uint2> &tab, std::vector<int2> &hdr) {
  tab.clear();
  hdr.assign(2 * kNumClass * 3, make_int2(0, 0));
#define SF_TAB(id, la, lb, lc, ld, t64, t32)                                     \
  for (int f = 0; f < 2; ++f) {                                                  \
    constexpr int N = QC<la, lb, lc, ld>::NABCD;                                 \
    const int T = f ? tgrad_r<float>(N) : tgrad(N);                              \
    int2 h[3];                                                                   \
    if (T > 1) {                                                                 \
      grad_table<la, lb, lc, ld>(T, tab, h);                                     \
      for (int d = 0; d < 3; ++d) hdr[(2 * id + f) * 3 + d] = h[d];              \
    }                                                                            \
  }
  SF_CLASS_LIST(SF_TAB)
#undef SF_TAB
}

cudaError_t prepare_grad_f32() {
  cudaError_t e = cudaSuccess;
#define SF_PREP(id, la, lb, lc, ld, t64, t32)                                                               \
  if (e == cudaSuccess)                                                                                     \
    e = prep_smem(grad_kernel<la, lb, lc, ld, float, tgrad_r<float>(QC<la, lb, lc, ld>::NABCD)>,                    \
                  grad_smem<la, lb, lc, ld, float>());
  SF_CLASS_LIST(SF_PREP)
#undef SF_PREP
  return e;
}

}  // namespace sf
