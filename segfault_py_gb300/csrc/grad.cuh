// grad.cuh -- two-electron part of the analytic RHF nuclear gradient.
//
// The reference has no gradients.  With E2 = 1/2 sum (pq|rs) [D_pq D_rs -
// 1/2 D_pr D_qs] the derivative with respect to a nuclear coordinate, at fixed
// density (the Pulay term -sum W dS is added by the one-electron part), is
//
//   dE2/dR = sum_{canonical shell quartets} m(ab,cd) sum_{ijkl} G_ijkl d(ij|kl)/dR
//   G_ijkl = 1/2 D_ij D_kl - 1/8 (D_ik D_jl + D_il D_jk),
//
// m = 8 / 2^(d_ab + d_cd + d_(ab,cd)) the number of index permutations of the
// quartet.  A Cartesian Gaussian on centre A obeys
// d phi_a / dA_x = 2 alpha phi_{a+1x} - a_x phi_{a-1x}, so in the Rys
// factorisation only the x 2-D integral changes:
//   dIx/dA_x = 2 alpha Ix(a_x+1, ...) - a_x Ix(a_x-1, ...).
// The 2-D tables are therefore built for the class extended by one unit on A,
// B and C ((la+1 lb+1 | lc+1 ld), same recurrences as the energy kernels, one
// more root when the total angular momentum becomes odd).  Per root and direction
// the outputs are contracted in two steps, because many share their exponents in
// that direction: with e the exponents (a_x, b_x, c_x, d_x),
//   F_e = sum_{o: e(o) = e} G_o Iy Iz,
//   g_A,x += sum_e F_e [2 alpha Ix(e +A) - a_x Ix(e -A)], likewise B and C,
// three products per output instead of a derivative term per output, centre and
// direction ((11|11): 81 outputs but 16 e; (22|22): 1296 and 81).  Centre D
// follows from translational invariance, g_D = -(g_A + g_B + g_C).
// (H2O)8 6-31G* forces, FP32 + double-float: 6.4 -> 5.3 ms; (H2O)2, FP64: 1.47 -> 1.20 ms.
#pragma once
#include <algorithm>
#include <vector>

#include "quartet.cuh"

namespace sf {

template <int LA, int LB, int LC, int LD>
struct QG {
  using Q = QC<LA, LB, LC, LD>;
  static constexpr int SZE = (LA + 2) * (LB + 2) * (LC + 2) * (LD + 1);   // extended 2-D table
  static constexpr int NRG = (Q::L + 1) / 2 + 1;                          // roots for degree L+1
  static constexpr int NX = (LA + 1) * (LB + 1) * (LC + 1) * (LD + 1);     // exponents of one direction (QC::toff)
  static constexpr int SA = (LB + 2) * (LC + 2) * (LD + 1), SB = (LC + 2) * (LD + 1), SC = LD + 1;
  __host__ __device__ static constexpr int eoff(int o, int d) {
    return ((cart_e(LA, Q::ca(o), d) * (LB + 2) + cart_e(LB, Q::cb(o), d)) * (LC + 2) + cart_e(LC, Q::cc(o), d)) *
               (LD + 1) +
           cart_e(LD, Q::cd(o), d);
  }
  // exponents e = toff of one direction: those of centre c, and the offset in the extended table
  __host__ __device__ static constexpr int ex(int e, int c) {
    return c == 0 ? e / ((LB + 1) * (LC + 1) * (LD + 1))
         : c == 1 ? e / ((LC + 1) * (LD + 1)) % (LB + 1)
         : c == 2 ? e / (LD + 1) % (LC + 1)
                  : e % (LD + 1);
  }
  __host__ __device__ static constexpr int xoff(int e) {
    return ((ex(e, 0) * (LB + 2) + ex(e, 1)) * (LC + 2) + ex(e, 2)) * (LD + 1) + ex(e, 3);
  }
};

// lanes per quartet of the gradient kernels (bigger tables than the energy);
// T = 1 keeps everything in registers
__host__ __device__ constexpr int tgrad(int nabcd) {
  return nabcd <= 18 ? 1 : nabcd <= 27 ? 4 : nabcd <= 81 ? 8 : nabcd <= 216 ? 16 : 32;
}

// per arithmetic: FP32 values take half the registers, so the FP32 kernels
// keep quartets of up to 27 outputs in one lane (measured: faster up to 27,
// slower with fewer lanes beyond)
template <typename R>
__host__ __device__ constexpr int tgrad_r(int nabcd) {
  if constexpr (sizeof(R) == sizeof(float)) return nabcd <= 27 ? 1 : tgrad(nabcd);
  else return tgrad(nabcd);
}

template <int LA, int LB, int LC, int LD, typename R, int T>
struct GGrp {
  using Q = QC<LA, LB, LC, LD>;
  using G = QG<LA, LB, LC, LD>;
  static constexpr int TABN = 3 * G::NRG * G::SZE;
  static constexpr int ROOTS = TABN;
  static constexpr int GAM = ROOTS + 2 * G::NRG;             // G_o
  static constexpr int FB = GAM + Q::NABCD;                  // F_e of one direction, per root
  static constexpr int BUFN = (FB + G::NX * G::NRG) | 1;
};

// Work table of a group kernel (built by grad_table): per
// direction the outputs of the lanes, lane t's k-th at k T + t, those with equal
// exponents e in a row and whole on one lane, the lanes balanced by length.
//   x = o | (offset in direction d+1) << 11 | (in d+2) << 19 | last of its e << 31
//   (~0: none), y = e.

// index of a class's work table: 2 class + (FP32 lanes)
template <int LA, int LB, int LC, int LD, typename R>
__host__ __device__ constexpr int grad_tab_index() {
  constexpr int X = LA * (LA + 1) / 2 + LB, Y = LC * (LC + 1) / 2 + LD;
  return 2 * (X * (X + 1) / 2 + Y) + (std::is_same<R, float>::value ? 1 : 0);
}

// the work table of one class for T lanes: entries and {offset, steps} of the
// three directions.  Outputs grouped by exponents e, the largest groups first
// to the lane with the least work.
template <int LA, int LB, int LC, int LD>
void grad_table(int T, std::vector<uint2> &tab, int2 (&hdr)[3]) {
  using Q = QC<LA, LB, LC, LD>;
  using G = QG<LA, LB, LC, LD>;
  static_assert(Q::NABCD <= 2048 && G::SZE <= 256, "packed work entries");
  for (int d = 0; d < 3; ++d) {
    std::vector<std::vector<int>> of(G::NX);
    for (int o = 0; o < Q::NABCD; ++o) of[Q::toff(o, d)].push_back(o);
    std::vector<int> order(G::NX);
    for (int e = 0; e < G::NX; ++e) order[e] = e;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return of[a].size() > of[b].size(); });
    std::vector<std::vector<uint2>> lane(T);
    for (int e : order) {
      if (of[e].empty()) continue;
      int best = 0;
      for (int t = 1; t < T; ++t)
        if (lane[t].size() < lane[best].size()) best = t;
      for (size_t k = 0; k < of[e].size(); ++k) {
        const int o = of[e][k];
        uint2 w;
        w.x = (unsigned)o | (unsigned)G::eoff(o, (d + 1) % 3) << 11 | (unsigned)G::eoff(o, (d + 2) % 3) << 19 |
              (k + 1 == of[e].size() ? 1u << 31 : 0u);
        w.y = (unsigned)e;
        lane[best].push_back(w);
      }
    }
    size_t steps = 0;
    for (const auto &l : lane) steps = std::max(steps, l.size());
    hdr[d] = make_int2((int)tab.size(), (int)steps);
    for (size_t k = 0; k < steps; ++k)
      for (int t = 0; t < T; ++t) tab.push_back(k < lane[t].size() ? lane[t][k] : make_uint2(~0u, 0u));
  }
}

template <typename R>
__device__ __forceinline__ void load_exps(const KParams &kp, int prim, R &e0, R &e1) {
  const R *rec = prims_of<R>(kp).rec + (size_t)prim * kPrimRec + 6;
  e0 = ldg_r(rec);
  e1 = ldg_r(rec + 1);
}

// products and sums of the contraction; dd sums stay unnormalised (dd_acc)
// until grad_fin
template <typename R>
__device__ __forceinline__ R grad_mul(R a, R b) {
  if constexpr (std::is_same<R, dd>::value) return dd_mul_raw(a, b);
  else return a * b;
}
template <typename R>
__device__ __forceinline__ void grad_acc(R &s, R a, R b) {
  if constexpr (std::is_same<R, dd>::value) dd_acc(s, a, b);
  else s += a * b;
}
template <typename R>
__device__ __forceinline__ R grad_fin(R s) {
  if constexpr (std::is_same<R, dd>::value) return dd_norm(s);
  else return s;
}
template <typename R>
__device__ __forceinline__ R grad_times(int k, R a) {
  if constexpr (std::is_same<R, dd>::value) return dd_times(k, a);
  else return (R)k * a;
}
__device__ __forceinline__ dd grad_sum(dd a, dd b, dd c) {   // 2 alpha sp - sm
  return dd_fma(dd(2.0f * a.hi, 2.0f * a.lo), dd_norm(b), -dd_norm(c));
}

// T == 1: one lane per quartet, every table in registers, compile-time indices
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void grad_t1(const KParams &kp, const QGeom<R> &g, const R (&gam)[QC<LA, LB, LC, LD>::NABCD],
                                        int p, int P, R (&gA)[3], R (&gB)[3], R (&gC)[3]) {
  using Q = QC<LA, LB, LC, LD>;
  using G = QG<LA, LB, LC, LD>;
  constexpr int NR = G::NRG, SZ = G::SZE;
  const int nprim = g.ab_n * g.cd_n;
  int cur = -1;
  PQ<R> s;
  R pp, px, py, pz, kab, al = 0, be = 0;
  for (int idx = p; idx < nprim; idx += P) {
    const int ip = idx / g.cd_n, iq = idx - ip * g.cd_n;
    if (ip != cur) {
      load_prim_ab<R>(kp, g, ip, s, pp, px, py, pz, kab);
      load_exps<R>(kp, g.ab_off + ip, al, be);
      cur = ip;
    }
    load_prim_cd<R>(kp, g, iq, s, pp, px, py, pz, kab);
    R ga, gd;
    load_exps<R>(kp, g.cd_off + iq, ga, gd);
    R u[NR], wr[NR];
    rys_roots_all<NR, R>(kp, s.x, u, wr);
    R sp[3][3], sm[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int d = 0; d < 3; ++d) sp[c][d] = sm[c][d] = (R)0;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      R I[3][SZ];
      if constexpr (std::is_same<R, dd>::value) {
        const RootDD c(s, u[r]);
        rys_2d_dd<LA + 1, LB + 1, LC + 1, LD, true>(dd(1.0f), dd_fma(-c.tq, s.pqx, s.pax), dd_fma(c.tp, s.pqx, s.qcx),
                                                    c.b00, c.b10, c.b01, g.ABx, g.CDx, I[0]);
        rys_2d_dd<LA + 1, LB + 1, LC + 1, LD, true>(dd(1.0f), dd_fma(-c.tq, s.pqy, s.pay), dd_fma(c.tp, s.pqy, s.qcy),
                                                    c.b00, c.b10, c.b01, g.ABy, g.CDy, I[1]);
        rys_2d_dd<LA + 1, LB + 1, LC + 1, LD, false>(s.pref * wr[r], dd_fma(-c.tq, s.pqz, s.paz),
                                                     dd_fma(c.tp, s.pqz, s.qcz), c.b00, c.b10, c.b01, g.ABz, g.CDz,
                                                     I[2]);
      } else {
        const R uu = u[r];
        const R b00 = (R)0.5 * s.r2 * uu;
        const R b10 = s.i2p * ((R)1 - s.aq * uu);
        const R b01 = s.i2q * ((R)1 - s.ap * uu);
        const R tq = s.aq * uu, tp = s.ap * uu;
        rys_2d<LA + 1, LB + 1, LC + 1, LD, R>((R)1, s.pax - tq * s.pqx, s.qcx + tp * s.pqx, b00, b10, b01, g.ABx,
                                              g.CDx, I[0]);
        rys_2d<LA + 1, LB + 1, LC + 1, LD, R>((R)1, s.pay - tq * s.pqy, s.qcy + tp * s.pqy, b00, b10, b01, g.ABy,
                                              g.CDy, I[1]);
        rys_2d<LA + 1, LB + 1, LC + 1, LD, R>(s.pref * wr[r], s.paz - tq * s.pqz, s.qcz + tp * s.pqz, b00, b10, b01,
                                              g.ABz, g.CDz, I[2]);
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        R F[G::NX];
#pragma unroll
        for (int e = 0; e < G::NX; ++e) F[e] = (R)0;
#pragma unroll
        for (int o = 0; o < Q::NABCD; ++o) {
          const R i1 = I[(d + 1) % 3][G::eoff(o, (d + 1) % 3)], i2 = I[(d + 2) % 3][G::eoff(o, (d + 2) % 3)];
          grad_acc(F[Q::toff(o, d)], grad_mul(gam[o], i1), i2);
        }
#pragma unroll
        for (int e = 0; e < G::NX; ++e) {
          const R f = grad_fin(F[e]);
          const int x = G::xoff(e), ea = G::ex(e, 0), eb = G::ex(e, 1), ec = G::ex(e, 2);
          grad_acc(sp[0][d], f, I[d][x + G::SA]);
          grad_acc(sp[1][d], f, I[d][x + G::SB]);
          grad_acc(sp[2][d], f, I[d][x + G::SC]);
          if (ea) grad_acc(sm[0][d], grad_times(ea, f), I[d][x - G::SA]);
          if (eb) grad_acc(sm[1][d], grad_times(eb, f), I[d][x - G::SB]);
          if (ec) grad_acc(sm[2][d], grad_times(ec, f), I[d][x - G::SC]);
        }
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if constexpr (std::is_same<R, dd>::value) {
        gA[d] += grad_sum(al, sp[0][d], sm[0][d]);
        gB[d] += grad_sum(be, sp[1][d], sm[1][d]);
        gC[d] += grad_sum(ga, sp[2][d], sm[2][d]);
      } else {
        gA[d] += (R)2 * al * sp[0][d] - sm[0][d];
        gB[d] += (R)2 * be * sp[1][d] - sm[1][d];
        gC[d] += (R)2 * ga * sp[2][d] - sm[2][d];
      }
    }
  }
}

template <int LA, int LB, int LC, int LD, typename R, int T, typename A>
__device__ __forceinline__ void grad_quartet(const KParams &kp, const ClassWork &w, int64_t cta,
                                             const R *__restrict__ D, A *grad);

// Gradient contributions of a CTA are summed in shared memory (3 slots per
// atom) and written with one atomic per slot at the end: all quartets add
// into the same 3*natom words, so per-quartet global atomics serialise.
constexpr int kGradSmemAtoms = 512;   // larger molecules add to global memory directly

// Per-CTA sums: FP32 for the FP32 kernels (shared-memory FP32 atomic adds are
// native; FP64 ones are compare-and-swap loops whose FP64 adds, retried on
// every collision of the lanes' atoms, kept the 1/64-rate FP64 pipe a third
// to half busy), FP64 for the FP64 and double-float kernels.
template <typename R>
using GradAcc = typename std::conditional<std::is_same<R, float>::value, float, double>::type;

__device__ __forceinline__ double acc_to_f64(float v) { return f2d_alu(v); }
__device__ __forceinline__ double acc_to_f64(double v) { return v; }
__device__ __forceinline__ float acc_value(float v, float) { return v; }
template <typename V>
__device__ __forceinline__ double acc_value(V v, double) { return to_f64(v); }

// one-lane classes: primitive sub-groups per quartet from which they share its G_o
// (2 / 4 / 8: forces of (H2O)8 FP32 + double-float 4.231 / 4.236 / 4.243 ms, (H2O)4 FP64
// 4.046 / 4.048 / 4.059)
constexpr int kGradCoop = 4;
// shared memory before the CTA's sums: the groups' buffers, or the G_o of the
// quartets of a one-lane class with kGradCoop or more lanes each
template <int LA, int LB, int LC, int LD, typename R, int T>
__host__ __device__ constexpr size_t grad_buf_bytes() {
  const size_t n = T == 1 ? (size_t)(kBlock / kGradCoop) * QC<LA, LB, LC, LD>::NABCD
                          : (size_t)(kBlock / T) * GGrp<LA, LB, LC, LD, R, T>::BUFN;
  return (n * sizeof(R) + 7) / 8 * 8;
}

template <int LA, int LB, int LC, int LD, typename R, int T>
__global__ void __launch_bounds__(kBlock) grad_kernel(KParams kp, const __grid_constant__ ClassMulti m,
                                                      const R *__restrict__ D, double *grad) {
  const int sg = m.find(blockIdx.x);
  const ClassWork w = m.seg[sg];
  const int64_t cta = (int)blockIdx.x - m.cta0[sg];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using A = GradAcc<R>;
  const bool cta_sum = kp.natom <= kGradSmemAtoms;
  A *sgrad = reinterpret_cast<A *>(smem_raw + grad_buf_bytes<LA, LB, LC, LD, R, T>());
  const int TP0 = T * w.psplit;
  const int64_t nq = work_count(w);
  const int64_t qfirst = (cta * (kBlock / TP0)) / w.wsplit;
  if (qfirst >= nq) return;   // the whole CTA is past the end of the list
  if (cta_sum) {
    for (int i = threadIdx.x; i < 3 * kp.natom; i += blockDim.x) sgrad[i] = (A)0;
    __syncthreads();
  }
  const int64_t q0 = (cta * (kBlock / TP0) + threadIdx.x / TP0) / w.wsplit;
  if (q0 < nq) {
    if (cta_sum) grad_quartet<LA, LB, LC, LD, R, T, A>(kp, w, cta, D, sgrad);
    else grad_quartet<LA, LB, LC, LD, R, T, double>(kp, w, cta, D, grad);
  }
  if (cta_sum) {
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * kp.natom; i += blockDim.x)
      if (sgrad[i] != (A)0) atomicAdd(grad + i, acc_to_f64(sgrad[i]));
  }
}

template <int LA, int LB, int LC, int LD, typename R, int T, typename A>
__device__ __forceinline__ void grad_quartet(const KParams &kp, const ClassWork &w, int64_t cta,
                                             const R *__restrict__ D, A *grad) {
  using Q = QC<LA, LB, LC, LD>;
  using G = QG<LA, LB, LC, LD>;
  using GP = GGrp<LA, LB, LC, LD, R, T>;
  constexpr int NR = G::NRG, SZ = G::SZE;
  const int P = w.psplit, W = w.wsplit;
  const int TP = T * P;
  const int grp = threadIdx.x / TP, t = threadIdx.x % T;
  const int64_t gid = cta * (kBlock / TP) + grp;
  const int64_t q = gid / W;
  const int pl = (threadIdx.x / T) % P;
  const int sub = (int)(gid - q * W) * P + pl;   // primitive sub-group of the W*P
  const int2 ij = __ldg(w.list + q);
  const int pab = w.x0 + ij.x, pcd = w.y0 + ij.y;
  const QGeom<R> g = make_geom<R>(kp, pab, pcd, false, false);
  R scale = (R)8;
  if (g.a == g.b) scale *= (R)0.5;
  if (g.c == g.d) scale *= (R)0.5;
  if (w.same && ij.x == ij.y) scale *= (R)0.5;
  const int lane = threadIdx.x & 31;
  const unsigned qmask = (TP == 32) ? 0xffffffffu : (((1u << TP) - 1u) << (lane & ~(TP - 1)));
  const unsigned gmask = (T == 32) ? 0xffffffffu : (((1u << T) - 1u) << (lane & ~(T - 1)));
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R *tab = reinterpret_cast<R *>(smem_raw) + (threadIdx.x / T) * GP::BUFN;

  // G_o (normalised, permutation count folded in).  The primitive sub-groups of a
  // quartet share them: each of the TP lanes evaluates outputs TP apart into the
  // buffer of the first group (six density elements and nine operations each, per
  // lane of every sub-group as much as one primitive quartet's contraction);
  // T == 1 then keeps them in registers.  Forces of (H2O)4 6-31G* double-float
  // 2.20 -> 2.17 ms.
  const int n = kp.nao;
  const int a0 = g.a0, b0 = g.b0, c0 = g.c0, d0 = g.d0;
  auto gamma = [&](int o) {
    const int i = a0 + Q::ca(o), j = b0 + Q::cb(o), kk = c0 + Q::cc(o), l = d0 + Q::cd(o);
    const R Dij = ldg_r(D + i * n + j), Dkl = ldg_r(D + kk * n + l), Dik = ldg_r(D + i * n + kk);
    const R Djl = ldg_r(D + j * n + l), Dil = ldg_r(D + i * n + l), Djk = ldg_r(D + j * n + kk);
    return scale * Q::template norm_r<R>(o) * ((R)0.5 * Dij * Dkl - (R)0.125 * (Dik * Djl + Dil * Djk));
  };
  R gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0}, gC[3] = {0, 0, 0};
  if constexpr (T == 1) {
    R gam[Q::NABCD];
    if (P >= kGradCoop) {
      R *sg = reinterpret_cast<R *>(smem_raw) + (threadIdx.x / P) * Q::NABCD;
      for (int o = pl; o < Q::NABCD; o += P) sg[o] = gamma(o);
      __syncwarp(qmask);
#pragma unroll
      for (int o = 0; o < Q::NABCD; ++o) gam[o] = sg[o];
    } else {
#pragma unroll
      for (int o = 0; o < Q::NABCD; ++o) gam[o] = gamma(o);
    }
    grad_t1<LA, LB, LC, LD, R>(kp, g, gam, sub, W * P, gA, gB, gC);
  } else {
  R *gam = reinterpret_cast<R *>(smem_raw) + (threadIdx.x / TP) * P * GP::BUFN + GP::GAM;
  for (int o = (int)threadIdx.x % TP; o < Q::NABCD; o += TP) gam[o] = gamma(o);
  __syncwarp(qmask);
  const int2 *hdr = kp.grad_hdr + grad_tab_index<LA, LB, LC, LD, R>() * 3;   // {offset, steps} per direction
  const int nprim = g.ab_n * g.cd_n;
  int cur = -1;
  PQ<R> s;
  R pp, px, py, pz, kab, al = 0, be = 0;
  for (int idx = sub; idx < nprim; idx += W * P) {
    const int ip = idx / g.cd_n, iq = idx - ip * g.cd_n;
    if (ip != cur) {
      load_prim_ab<R>(kp, g, ip, s, pp, px, py, pz, kab);
      load_exps<R>(kp, g.ab_off + ip, al, be);
      cur = ip;
    }
    load_prim_cd<R>(kp, g, iq, s, pp, px, py, pz, kab);
    R ga, gd;
    load_exps<R>(kp, g.cd_off + iq, ga, gd);
    for (int r = t; r < NR; r += T) {
      R uu, ww;
      rys_root_one<NR, R>(kp, s.x, r, uu, ww);
      tab[GP::ROOTS + r] = uu;
      tab[GP::ROOTS + NR + r] = ww;
    }
    __syncwarp(gmask);
    for (int task = t; task < 3 * NR; task += T) {
      const int r = task % NR, d = task / NR;
      const R uu = tab[GP::ROOTS + r], ww = tab[GP::ROOTS + NR + r];
      const R pa = d == 0 ? s.pax : d == 1 ? s.pay : s.paz;
      const R qc = d == 0 ? s.qcx : d == 1 ? s.qcy : s.qcz;
      const R pq = d == 0 ? s.pqx : d == 1 ? s.pqy : s.pqz;
      const R ab = d == 0 ? g.ABx : d == 1 ? g.ABy : g.ABz;
      const R cd = d == 0 ? g.CDx : d == 1 ? g.CDy : g.CDz;
      const R g0 = d == 2 ? s.pref * ww : (R)1;
      if constexpr (std::is_same<R, dd>::value) {
        const RootDD c(s, uu);
        rys_2d_dd<LA + 1, LB + 1, LC + 1, LD, false>(g0, dd_fma(-c.tq, pq, pa), dd_fma(c.tp, pq, qc), c.b00, c.b10, c.b01,
                                                     ab, cd, tab + (d * NR + r) * SZ);
      } else {
        const R b00 = (R)0.5 * s.r2 * uu;
        const R b10 = s.i2p * ((R)1 - s.aq * uu);
        const R b01 = s.i2q * ((R)1 - s.ap * uu);
        const R tq = s.aq * uu, tp = s.ap * uu;
        rys_2d<LA + 1, LB + 1, LC + 1, LD, R>(g0, pa - tq * pq, qc + tp * pq, b00, b10, b01, ab, cd,
                                              tab + (d * NR + r) * SZ);
      }
    }
    __syncwarp(gmask);
    R sp[3][3], sm[3][3];   // [centre A,B,C][direction]: + and - shift sums
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int d = 0; d < 3; ++d) sp[c][d] = sm[c][d] = (R)0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int2 h = __ldg(hdr + d);
      const uint2 *work = kp.grad_tab + h.x + t;
      const R *t1 = tab + (d + 1) % 3 * NR * SZ, *t2 = tab + (d + 2) % 3 * NR * SZ;
      R F[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) F[r] = (R)0;
      for (int k = 0; k < h.y; ++k) {
        const uint2 e = __ldg(work + k * T);
        if (e.x == ~0u) break;
        const R gm = gam[e.x & 2047u];
        const R *p1 = t1 + ((e.x >> 11) & 255u), *p2 = t2 + ((e.x >> 19) & 255u);
#pragma unroll
        for (int r = 0; r < NR; ++r) grad_acc(F[r], grad_mul(gm, p1[r * SZ]), p2[r * SZ]);
        if (e.x >> 31) {
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            tab[GP::FB + e.y * NR + r] = grad_fin(F[r]);
            F[r] = (R)0;
          }
        }
      }
      __syncwarp(gmask);
      for (int i = t; i < G::NX * NR; i += T) {
        const int e = i / NR, r = i % NR;
        const R f = tab[GP::FB + i];
        const R *td = tab + (d * NR + r) * SZ + G::xoff(e);
        const int ea = G::ex(e, 0), eb = G::ex(e, 1), ec = G::ex(e, 2);
        grad_acc(sp[0][d], f, td[G::SA]);
        grad_acc(sp[1][d], f, td[G::SB]);
        grad_acc(sp[2][d], f, td[G::SC]);
        if (ea) grad_acc(sm[0][d], grad_times(ea, f), td[-G::SA]);
        if (eb) grad_acc(sm[1][d], grad_times(eb, f), td[-G::SB]);
        if (ec) grad_acc(sm[2][d], grad_times(ec, f), td[-G::SC]);
      }
      __syncwarp(gmask);   // the F_e are read before the next direction's are written
    }
    __syncwarp(gmask);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if constexpr (std::is_same<R, dd>::value) {
        gA[d] += grad_sum(al, sp[0][d], sm[0][d]);
        gB[d] += grad_sum(be, sp[1][d], sm[1][d]);
        gC[d] += grad_sum(ga, sp[2][d], sm[2][d]);
      } else {
        gA[d] += (R)2 * al * sp[0][d] - sm[0][d];
        gB[d] += (R)2 * be * sp[1][d] - sm[1][d];
        gC[d] += (R)2 * ga * sp[2][d] - sm[2][d];
      }
    }
  }
  }
  // sum over the T x P lanes of the quartet.  Eight or more lanes halve the values
  // with every exchange (12 -> 6 -> 3 -> 2 -> 1, a lane adds up the ones that it keeps: 13
  // additions and 6 for centre D, instead of 45 and 6) and the lanes that hold
  // the totals add them to the forces side by side.  Forces of (H2O)8 6-31G* FP32 +
  // double-float 4.82 -> 4.67 ms, (H2O)2 FP64 1.14 -> 1.11.
  if (TP >= 8) {
    R v[12];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      v[d] = gA[d];
      v[3 + d] = gB[d];
      v[6 + d] = gC[d];
      v[9 + d] = -(gA[d] + gB[d] + gC[d]);
    }
    const bool h1 = lane & 1, h2 = lane & 2, h4 = lane & 4, h8 = lane & 8;
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = (h1 ? v[6 + k] : v[k]) + shfl_xor_r(qmask, h1 ? v[k] : v[6 + k], 1);
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = (h2 ? v[3 + k] : v[k]) + shfl_xor_r(qmask, h2 ? v[k] : v[3 + k], 2);
    const R x0 = shfl_xor_r(qmask, h4 ? v[0] : v[2], 4), x1 = shfl_xor_r(qmask, v[1], 4);
    v[0] = (h4 ? v[2] : v[0]) + x0;   // values 0, 1 of three, or value 2
    v[1] = v[1] + x1;
    int i = (h1 ? 6 : 0) + (h2 ? 3 : 0) + (h4 ? 2 : 0), nv = h4 ? 1 : 2;
    if (TP >= 16) {
      const R x = shfl_xor_r(qmask, h8 ? v[0] : v[1], 8);
      v[0] = (h8 ? v[1] : v[0]) + x;
      nv = h8 && h4 ? 0 : 1;
      i += h8;
    }
    if (TP == 32) {
      v[0] = v[0] + shfl_xor_r(qmask, v[0], 16);
      if (lane & 16) nv = 0;
    }
    for (int k = 0; k < nv; ++k, ++i) {
      const int at = kp.sh.atom[i < 3 ? g.a : i < 6 ? g.b : i < 9 ? g.c : g.d];
      atomicAdd(grad + 3 * at + i % 3, acc_value(k ? v[1] : v[0], A()));
    }
    return;
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
    for (int sft = 1; sft < TP; sft <<= 1) {
      gA[d] += shfl_xor_r(qmask, gA[d], sft);
      gB[d] += shfl_xor_r(qmask, gB[d], sft);
      gC[d] += shfl_xor_r(qmask, gC[d], sft);
    }
  if (t == 0 && pl == 0) {
    const int at_a = kp.sh.atom[g.a], at_b = kp.sh.atom[g.b], at_c = kp.sh.atom[g.c], at_d = kp.sh.atom[g.d];
    R gD[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      gD[d] = -(gA[d] + gB[d] + gC[d]);
      atomicAdd(grad + 3 * at_c + d, acc_value(gC[d], A()));
      atomicAdd(grad + 3 * at_d + d, acc_value(gD[d], A()));
    }
    // centres a, b: with one quartet per lane, the lanes sharing the bra pair
    // (consecutive in the cost-sorted list) add their forces first
    R gab[6] = {gA[0], gA[1], gA[2], gB[0], gB[1], gB[2]};
    const bool write = TP > 1 ? true : run_sums<R, 6>(ij.x, gab);
    if (write) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        atomicAdd(grad + 3 * at_a + d, acc_value(gab[d], A()));
        atomicAdd(grad + 3 * at_b + d, acc_value(gab[3 + d], A()));
      }
    }
  }
}

// Primitive split of one gradient segment: the Fock list's S = P*W, re-cut for
// this kernel's T (as many sub-groups as fit in T*P <= 32 lanes, the rest as
// separate groups), and doubled while a sub-group's estimated work is above a
// quarter of the average load of the lanes that fill the GPU (rel_load: the Fock
// kernels' estimate, a derivative quartet costs several times that), until the
// costliest quartet has a sub-group per primitive quartet (with one to two each:
// (H2O)2 6-31G* forces in FP64 0.99 ms against 0.93 here).  Filling the GPU with every
// segment by itself instead: (H2O)8 6-31G* forces in FP64 17.3 ms against 15.2
// here, FP32 + double-float 5.6 against 4.9, nonane 6-31G** 19.5 against 18.3.
inline ClassWork grad_work(const ClassWork &w, int T) {
  int S = (w.psplit < 1 ? 1 : w.psplit) * (w.wsplit < 1 ? 1 : w.wsplit);
  while (S < w.max_cost && 4.0f * (float)w.max_cost * w.rel_load > (float)S * T && 2 * S <= (32 / T) * kMaxWsplit) S *= 2;
  int P = S;
  while (T * P > 32) P >>= 1;
  ClassWork w2 = w;
  w2.psplit = P;
  w2.wsplit = S / P < kMaxWsplit ? S / P : kMaxWsplit;
  return w2;
}

// the segments of one gradient launch
inline bool grad_segments(ClassMulti &m, const ClassWork *w, int nw, int T) {
  m.n = 0;
  for (int k = 0; k < nw; ++k)
    if (w[k].n > 0 && !add_segment(m, grad_work(w[k], T), T)) return false;
  return true;
}

template <int LA, int LB, int LC, int LD, typename R>
constexpr size_t grad_smem() {
  constexpr int T = tgrad_r<R>(QC<LA, LB, LC, LD>::NABCD);
  return grad_buf_bytes<LA, LB, LC, LD, R, T>() + 3 * kGradSmemAtoms * sizeof(double);
}

}  // namespace sf
