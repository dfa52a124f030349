// launch.h -- host-side launchers implemented in the kernel translation units.
#pragma once
#include <vector>

#include "quartet.cuh"

namespace sf {
// J/K digestion kernels of class cls (0..20) over nw <= kMaxSegs segments, one launch
cudaError_t launch_jk_f64(int cls, const KParams &kp, const ClassWork *w, int nw, const double *D, double *Jh, double *Kh,
                          cudaStream_t st);
cudaError_t launch_jk_f32(int cls, const KParams &kp, const ClassWork *w, int nw, const float *D, double *Jh, double *Kh,
                          cudaStream_t st);
cudaError_t launch_jk_dd(int cls, const KParams &kp, const ClassWork *w, int nw, const dd *D, double *Jh, double *Kh,
                         cudaStream_t st);
// the same with tdd_wide lanes per quartet (jk_dd_wide.cu)
cudaError_t launch_jk_dd_wide(int cls, const KParams &kp, const ClassWork *w, int nw, const dd *D, double *Jh, double *Kh,
                              cudaStream_t st);
cudaError_t prepare_jk_dd_wide();
// persistent multi-class FP32 J/K kernels (jk_persist.cu): one launch per
// register tier runs the tiles of every list of the tier's classes, taken
// from a device work queue
constexpr int kPersistTiers = 4;
struct PersistWork {
  const ClassWork *works;   // the tier's lists
  const int *cls;           // class of each list
  const int2 *tiles;        // (list, tile index in the list), heaviest first
  int ntiles;
  unsigned *next;           // queue counter (zeroed by the launcher)
};
// tier of a class whose FP32 kernel runs in the register path, else -1
int persist_tier_of(int cls);
cudaError_t persist_blocks_per_sm(int tier, int *blocks);
cudaError_t launch_jk_persist_f32(int tier, const KParams &kp, const PersistWork &pw, int grid, const float *D,
                                  double *Jh, double *Kh, cudaStream_t st);
// raw integrals of one class (fp32: FP32 evaluation, else FP64)
cudaError_t launch_eri(int cls, int fp32, const KParams &kp, const EriWork &w, cudaStream_t st);
cudaError_t launch_eri_dd(int cls, const KParams &kp, const EriWork &w, cudaStream_t st);
// raw integrals of one class by McMurchie-Davidson (FP64)
cudaError_t launch_md_eri(int cls, const KParams &kp, const EriWork &w, cudaStream_t st);
cudaError_t prepare_md();
// the same with the bra E contraction on the tensor cores (FP32 MD, 3-pass TF32)
cudaError_t launch_md_tc(int cls, const KParams &kp, const EriWork &w, int nsm, cudaStream_t st);
cudaError_t prepare_md_tc();
// polls of md_tc's bounded MMA waits (0: out before the first poll, < 0: the
// default); a test hook
void md_tc_set_wait_limit(int iterations);
// Schwarz bounds of pair class pc (0..5) over pairs [p0, p0+n)
cudaError_t launch_schwarz(int pc, const KParams &kp, int p0, int n, double *qout, cudaStream_t st);

cudaError_t launch_grad_f64(int cls, const KParams &kp, const ClassWork *w, int nw, const double *D, double *grad,
                            cudaStream_t st);
cudaError_t launch_grad_f32(int cls, const KParams &kp, const ClassWork *w, int nw, const float *D, double *grad,
                            cudaStream_t st);
cudaError_t launch_grad_dd(int cls, const KParams &kp, const ClassWork *w, int nw, const dd *D, double *grad,
                           cudaStream_t st);
void grad_tables(std::vector<uint2> &tab, std::vector<int2> &hdr);
cudaError_t prepare_grad_f64();
cudaError_t prepare_grad_dd();
cudaError_t prepare_grad_f32();
cudaError_t prepare_jk_f64();
cudaError_t prepare_jk_f32();
cudaError_t prepare_jk_dd();
cudaError_t prepare_eri_dd();
cudaError_t prepare_eri();

// one-electron kernel parameters (oneint.cu)
struct OneParams {
  DevShells sh;
  int nao;
  const double *atom_xyz, *charges;
  int natom;
  double *S, *T, *V;
  DevPairs pr;                  // canonical shell pairs, class c at [cstart[c], cstart[c + 1])
  const double *rec;            // their primitive-pair records
  int cstart[kNumPairClass + 1];
  const double *boys;           // Boys functions (sf_internal.h)
};

cudaError_t launch_one_electron(const OneParams &P, cudaStream_t st);
// gradient of sum_ij D_ij (T+V)_ij - W_ij S_ij (derivatives of the basis
// centres and, for V, of the nuclei), accumulated into grad[3*natom]
cudaError_t launch_one_electron_grad(const OneParams &P, const double *D, const double *W, double *grad, int nsm,
                                     cudaStream_t st);
cudaError_t prepare_one_electron();

// smem bytes of a group kernel
template <int LA, int LB, int LC, int LD, typename R, int T>
constexpr size_t grp_smem() {
  return T == 1 ? 0 : (size_t)(kBlock / T) * Grp<LA, LB, LC, LD, R, T>::BUFN * sizeof(R);
}

// of an FP64 or double-float J/K kernel (one-lane classes: the integrals of the
// quartets that kCoopLanes or more lanes digest)
template <int LA, int LB, int LC, int LD, typename R, int T>
constexpr size_t jk_smem() {
  return T == 1 ? (size_t)(kBlock / kCoopLanes) * QC<LA, LB, LC, LD>::NABCD * sizeof(R)
                : grp_smem<LA, LB, LC, LD, R, T>();
}

// a raw-integral launch of `quartets` CTA trips, w.cluster CTAs (one cluster) each
template <typename K>
inline cudaError_t launch_eri_kernel(K kern, int64_t quartets, size_t smem, const KParams &kp, const EriWork &w,
                                     cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(quartets * w.cluster));
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)w.cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = w.cluster > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, kp, w);
}

template <typename K>
inline cudaError_t prep_smem(K kern, size_t smem) {
  if (smem > 48 * 1024) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return cudaSuccess;
}
}  // namespace sf
