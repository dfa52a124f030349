// oneint.cu -- one-electron matrices S, T, V on the GPU.
//
// Reference: src/hf/mmd2.py:14-84 (Fortran E coefficients per primitive pair)
// and src/hf/mmd.py:13-141, called per AO pair and per nucleus at
// src/hf/hf.py:266-274.  Here one warp evaluates the whole Cartesian block of
// one canonical shell pair and writes it and its transpose:
//   E^{ij}_t  Hermite expansion coefficients (McMurchie-Davidson), built by
//             the two-term recursions in i and j (mmd.py:13-30 in closed form:
//             E^{i+1,j}_t = E^{ij}_{t-1}/(2p) + X_PA E^{ij}_t + (t+1) E^{ij}_{t+1})
//   S = E0 E0 E0 (pi/p)^{3/2}                       (mmd.py:32-39)
//   T = b(2 lb + 3) S - 2 b^2 sum S(lb+2) - 1/2 sum lb(lb-1) S(lb-2) (mmd.py:49-60)
//   V = -Z sum_tuv E_t E_u E_v R_tuv(p, P-C) 2 pi / p  (mmd.py:110-133)
// R_tuv by the Hermite Coulomb recursion of mmd.py:70-108 / core.f90:64-97,
// evaluated bottom-up, with the Boys function F_n(T) from a polynomial table
// (T < 64) or its asymptotic form with upward recursion (large T).
#include <cmath>

#include "launch.h"

namespace sf {


// F_0 .. F_M of T from the handle's table (rys_table.cpp: F_m and e^-T as
// degree-7 polynomials on intervals of 1/8 below T = 64): the highest order and
// e^-T by Horner, the others by the downward recursion
// F_m = (2T F_{m+1} + e^-T) / (2m+1), M = 0 and 1 directly.  Above 64,
// F_0 = sqrt(pi/T)/2 and F_{m+1} = (2m+1)/(2T) F_m (e^-T is below 2e-28).
// 7 to 24 FP64 instructions; the power series it replaces took up to 200
// terms with an FP64 division each, and every FP64 instruction of a warp holds
// its sub-partition's FP64 unit for 64 cycles.
__device__ __forceinline__ double boys_horner(const double *row, double s) {
  const double2 *c = reinterpret_cast<const double2 *>(row);   // k = 7 .. 0
  const double2 a = __ldg(c), b = __ldg(c + 1), d = __ldg(c + 2), e = __ldg(c + 3);
  return ((((((a.x * s + a.y) * s + b.x) * s + b.y) * s + d.x) * s + d.y) * s + e.x) * s + e.y;
}
template <int M>
__device__ __forceinline__ void boys_table(const double *tab, double T, double (&F)[M + 1]) {
  static_assert(M <= kBoysMax, "orders in the table");
  if (!(T < kTabXmax)) {   // NaN too: it has no table row
    const double y = rsqrt_nr(T), h = 0.5 * y * y;
    F[0] = 0.886226925452758014 * y;   // sqrt(pi) / 2
#pragma unroll
    for (int m = 0; m < M; ++m) F[m + 1] = (2 * m + 1) * h * F[m];
    return;
  }
  const int j = (int)(T * (double)kTabHF);
  const double s = T * (double)(2 * kTabHF) - (double)(2 * j + 1);
  const double *row = tab + (size_t)j * (kTabDegF + 1);
  constexpr size_t kFn = (size_t)kTabNintF * (kTabDegF + 1);   // doubles per function
  F[M] = boys_horner(row + M * kFn, s);
  if constexpr (M == 1) F[0] = boys_horner(row, s);
  if constexpr (M > 1) {
    const double e = boys_horner(row + (kBoysMax + 1) * kFn, s), t2 = 2.0 * T;
#pragma unroll
    for (int m = M - 1; m >= 0; --m) F[m] = (t2 * F[m + 1] + e) * (1.0 / (2 * m + 1));
  }
}

// E[i][j][t] for i <= LI, j <= LJ, t <= i+j along one direction, from h = 1/(2p)
// with E^00_0 = 1 (the product Gaussian kept apart)
template <int LI, int LJ>
__device__ __forceinline__ void hermite_e(double h, double xpa, double xpb, double (&E)[LI + 1][LJ + 1][LI + LJ + 1]) {
#pragma unroll
  for (int i = 0; i <= LI; ++i)
#pragma unroll
    for (int j = 0; j <= LJ; ++j)
#pragma unroll
      for (int t = 0; t <= LI + LJ; ++t) E[i][j][t] = 0.0;
  E[0][0][0] = 1.0;
#pragma unroll
  for (int i = 0; i < LI; ++i)
#pragma unroll
    for (int t = 0; t <= i + 1; ++t)
      E[i + 1][0][t] = (t > 0 ? h * E[i][0][t - 1] : 0.0) + xpa * E[i][0][t] + (t + 1 <= i ? (t + 1) * E[i][0][t + 1] : 0.0);
#pragma unroll
  for (int i = 0; i <= LI; ++i)
#pragma unroll
    for (int j = 0; j < LJ; ++j)
#pragma unroll
      for (int t = 0; t <= i + j + 1; ++t)
        E[i][j + 1][t] = (t > 0 ? h * E[i][j][t - 1] : 0.0) + xpb * E[i][j][t] +
                         (t + 1 <= i + j ? (t + 1) * E[i][j][t + 1] : 0.0);
}

// R_tuv, t+u+v <= L, from the Boys values: level m overwrites
// t+u+w = L-m .. 1 from the top down (each entry needs level m+1 at
// t+u+w-1 and -2, not yet overwritten), then R^m_000 = (-2p)^m F_m
template <int L>
__device__ __forceinline__ void hermite_r(double p, const double (&pc)[3], const double (&F)[L + 1],
                                          double (&R)[L + 1][L + 1][L + 1]) {
  double fm2p[L + 1];
  fm2p[0] = 1.0;
#pragma unroll
  for (int m = 1; m <= L; ++m) fm2p[m] = fm2p[m - 1] * (-2.0 * p);
  R[0][0][0] = F[L] * fm2p[L];
#pragma unroll
  for (int m = L - 1; m >= 0; --m) {
#pragma unroll
    for (int sl = L - m; sl >= 1; --sl)
#pragma unroll
      for (int t = 0; t <= sl; ++t)
#pragma unroll
        for (int u = 0; u <= sl - t; ++u) {
          const int w = sl - t - u;
          double r;
          if (t > 0) r = (t > 1 ? (t - 1) * R[t - 2][u][w] : 0.0) + pc[0] * R[t - 1][u][w];
          else if (u > 0) r = (u > 1 ? (u - 1) * R[t][u - 2][w] : 0.0) + pc[1] * R[t][u - 1][w];
          else r = (w > 1 ? (w - 1) * R[t][u][w - 2] : 0.0) + pc[2] * R[t][u][w - 1];
          R[t][u][w] = r;
        }
    R[0][0][0] = F[m] * fm2p[m];
  }
}

// Hermite triples t+u+v <= L, enumerated t, then u, then v ascending
__host__ __device__ constexpr int ntuv(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
__host__ __device__ constexpr int tuv_index(int L, int t, int u, int v) {
  int k = 0;
  for (int t2 = 0; t2 < t; ++t2) k += (L - t2 + 1) * (L - t2 + 2) / 2;
  for (int u2 = 0; u2 < u; ++u2) k += L - t - u2 + 1;
  return k + v;
}

// Growth of a kinetic integral over its overlap: T = 1/2 sum_d <d_d a | d_d b>, where a
// derivative of x_A^la exp(-alpha x_A^2) brings la / x_A - 2 alpha x_A, and alpha |x_A|
// reaches mu |AB| + alpha / sqrt(p) around P (mu = alpha beta / p; likewise at B)
__device__ __forceinline__ float kinetic_bound(int la, int lb, float al, float be, float p, float R) {
  const float r = rsqrtf(p), mr = al * r * (be * r) * R;
  return 1.5f * (la + 2.0f * (mr + al * r)) * (lb + 2.0f * (mr + be * r));
}

// S, T, V: one warp per canonical shell pair of the handle's pair table
// (a, b), l_a >= l_b, reading the primitive-pair records of the two-electron
// kernels, so that p, P and the product Gaussian cost nothing here.  What
// bounds it is the number of FP64 warp instructions (64 cycles each on a
// sub-partition, whatever the number of active lanes), so every stage keeps
// the lanes full: the warp is cut into 32/G groups of G lanes (G = 8, 16 or 32
// by the number of primitive pairs and nuclei), a group takes every (32/G)-th
// primitive pair and its lanes
//  * build the E coefficients, one direction per lane, into shared memory;
//  * take nuclei C = l, l+G, ...: Boys values, R_tuv by the Hermite Coulomb
//    recursion in place (level n overwrites t+u+v = L-n .. 1 from the top
//    down, then R^n_000), S_tuv += -Z_C R_tuv (V is linear in R), then the
//    group's sum of S_tuv by shuffles;
//  * take Cartesian entries o = l, l+G, ... of the block: overlap, kinetic and
//    V = 2 pi / p c_i c_j sum_tuv E E E S_tuv, summed over the warp's groups at
//    the end; one lane writes the entry and its transpose.
// Primitive pairs whose contributions all stay below 1e-17 are skipped (the
// product Gaussian c_i c_j exp(-mu |AB|^2) (pi/p)^3/2 bounds the overlap, E
// coefficients grow at most as (|AB| + 1/sqrt(p) + 1)^L, kinetic terms as
// kinetic_bound and attraction as 2 sqrt(p/pi) times the summed charge; the
// bound itself in FP32).
// (H2O)16 6-31G* (48 nuclei, 68 k primitive pairs): 0.30 ms; one CTA of 64 threads
// per pair, with the power series, exp and pow per primitive pair and three
// threads building E, took 3.8 ms.
constexpr int kOneWarps = 4;

template <int LA, int LB>
constexpr int one_e_size() { return (LA + 1) * (LB + 3) * (LA + LB + 1); }   // E_t of one direction, t <= LA + LB
// doubles of one group: E in three directions, S_tuv
template <int LA, int LB>
constexpr int one_group() { return 3 * one_e_size<LA, LB>() + ntuv(LA + LB); }
constexpr int kOneSmem = kOneWarps * 4 * one_group<2, 2>();   // four groups of 8 lanes at most

template <int LA, int LB>
__device__ __forceinline__ void one_pair(const OneParams &P, int pair, double *smem, double zs, int lane) {
  constexpr int NA = ncart(LA), NB = ncart(LB), L = LA + LB, NT = ntuv(L), TE = LA + LB + 1;
  constexpr int KO = (NA * NB + 7) / 8;      // entries per lane at G = 8
  constexpr int ES = one_e_size<LA, LB>();
  const int a = P.pr.a[pair], b = P.pr.b[pair], np = P.pr.np[pair];
  const double *rec0 = P.rec + (size_t)P.pr.poff[pair] * kPrimRec;
  // lanes per primitive pair: all 32 for a lone one; else 8 lanes when that
  // many nuclei are there to share, never fewer
  const int G = np >= 3 ? 8 : np == 2 ? 16 : 32;
  const int sub = lane / G, l = lane % G, ngrp = 32 / G;
  double *E = smem + sub * one_group<LA, LB>(), *St = E + 3 * ES;
#define SF_E(d, i, j, t) E[(d) * ES + ((i) * (LB + 3) + (j)) * TE + (t)]
  const double A[3] = {P.sh.cx[a], P.sh.cy[a], P.sh.cz[a]};
  const double B[3] = {P.sh.cx[b], P.sh.cy[b], P.sh.cz[b]};
  const float R1 = sqrtf((float)((A[0] - B[0]) * (A[0] - B[0]) + (A[1] - B[1]) * (A[1] - B[1]) +
                                 (A[2] - B[2]) * (A[2] - B[2])));
  double sa[KO], ta[KO], va[KO];
#pragma unroll
  for (int k = 0; k < KO; ++k) sa[k] = ta[k] = va[k] = 0.0;
  for (int i0 = 0; i0 < np; i0 += ngrp) {
    const int ip = i0 + sub;
    bool on = ip < np;
    const double *rec = rec0 + (size_t)(on ? ip : 0) * kPrimRec;
    const double p = rec[0], Pc[3] = {rec[1], rec[2], rec[3]}, kt = rec[4], hp = rec[5], al = rec[6], be = rec[7];
    {
      // kt = c_i c_j exp(-mu R^2) sqrt(2) pi^(5/4) / p
      const float pf = (float)p, g = fabsf((float)kt) * 0.9414f * rsqrtf(pf);   // overlap bound
      const float x = R1 + rsqrtf(pf) + 1.0f;
      float e = 1.0f;
#pragma unroll
      for (int k = 0; k < L; ++k) e *= x;
      const float f = 1.0f + 1.1284f * sqrtf(pf) * (float)zs + kinetic_bound(LA, LB, (float)al, (float)be, pf, R1);
      if (g * e * f < 1e-17f) on = false;   // not on NaN: it has to reach the matrix it belongs to
    }
    if (!__any_sync(0xffffffffu, on)) continue;
    __syncwarp();   // the previous pass is done with E and St
    if (on && l < 3) {
      const double pa = l == 0 ? Pc[0] - A[0] : l == 1 ? Pc[1] - A[1] : Pc[2] - A[2];
      const double pb = l == 0 ? Pc[0] - B[0] : l == 1 ? Pc[1] - B[1] : Pc[2] - B[2];
      double Et[LA + 1][LB + 3][LA + LB + 3];
      hermite_e<LA, LB + 2>(hp, pa, pb, Et);
#pragma unroll
      for (int i = 0; i <= LA; ++i)
#pragma unroll
        for (int j = 0; j <= LB + 2; ++j)
#pragma unroll
          for (int t = 0; t < TE; ++t) SF_E(l, i, j, t) = Et[i][j][t];
    }
    __syncwarp();
    if (P.V) {
      double st[NT];
#pragma unroll
      for (int k = 0; k < NT; ++k) st[k] = 0.0;
      for (int at = on ? l : P.natom; at < P.natom; at += G) {
        const double pc[3] = {Pc[0] - P.atom_xyz[3 * at], Pc[1] - P.atom_xyz[3 * at + 1],
                              Pc[2] - P.atom_xyz[3 * at + 2]};
        double F[L + 1];
        boys_table<L>(P.boys, p * (pc[0] * pc[0] + pc[1] * pc[1] + pc[2] * pc[2]), F);
        double R[L + 1][L + 1][L + 1];
        hermite_r<L>(p, pc, F, R);
        const double z = -P.charges[at];
#pragma unroll
        for (int t = 0; t <= L; ++t)
#pragma unroll
          for (int u = 0; u <= L - t; ++u)
#pragma unroll
            for (int w = 0; w <= L - t - u; ++w) st[tuv_index(L, t, u, w)] += z * R[t][u][w];
      }
      __syncwarp();
      for (int off = 1; off < G; off <<= 1) {
#pragma unroll
        for (int k = 0; k < NT; ++k) st[k] += __shfl_xor_sync(0xffffffffu, st[k], off);
      }
      if (l == 0) {
#pragma unroll
        for (int k = 0; k < NT; ++k) St[k] = st[k];
      }
      __syncwarp();
    }
    if (on) {
      // sp = c_i c_j exp(-mu R^2) (pi/p)^(3/2), vp = the same with 2 pi / p
      const double sp = kt * 0.941396263776714813 * rsqrt_nr(p), vp = kt * 1.06225193202719693;
#pragma unroll
      for (int k = 0; k < KO; ++k) {
        const int o = l + k * G;
        if (o >= NA * NB) break;
        const int i = o / NB, j = o % NB;
        const int ax = cart_e(LA, i, 0), ay = cart_e(LA, i, 1), az = cart_e(LA, i, 2);
        const int bx = cart_e(LB, j, 0), by = cart_e(LB, j, 1), bz = cart_e(LB, j, 2);
        const double sx = SF_E(0, ax, bx, 0), sy = SF_E(1, ay, by, 0), sz = SF_E(2, az, bz, 0);
        const double s0 = sx * sy * sz;
        double x2 = SF_E(0, ax, bx + 2, 0) * sy * sz + sx * SF_E(1, ay, by + 2, 0) * sz + sx * sy * SF_E(2, az, bz + 2, 0);
        double t = be * ((2 * LB + 3) * s0 - 2.0 * be * x2);
        if (bx >= 2) t -= SF_E(0, ax, 0, 0) * sy * sz;   // l_x (l_x - 1) / 2 = 1 for l_x = 2
        if (by >= 2) t -= sx * SF_E(1, ay, 0, 0) * sz;
        if (bz >= 2) t -= sx * sy * SF_E(2, az, 0, 0);
        sa[k] += sp * s0;
        ta[k] += sp * t;
        if (P.V) {
          double acc = 0.0;
          for (int tt = 0; tt <= ax + bx; ++tt) {
            double au = 0.0;
            for (int u = 0; u <= ay + by; ++u) {
              double aw = 0.0;
              for (int w = 0; w <= az + bz; ++w) aw += SF_E(2, az, bz, w) * St[tuv_index(L, tt, u, w)];
              au += SF_E(1, ay, by, u) * aw;
            }
            acc += SF_E(0, ax, bx, tt) * au;
          }
          va[k] += vp * acc;
        }
      }
    }
  }
#undef SF_E
  __syncwarp();
  for (int off = G; off < 32; off <<= 1) {
#pragma unroll
    for (int k = 0; k < KO; ++k) {
      sa[k] += __shfl_xor_sync(0xffffffffu, sa[k], off);
      ta[k] += __shfl_xor_sync(0xffffffffu, ta[k], off);
      if (P.V) va[k] += __shfl_xor_sync(0xffffffffu, va[k], off);
    }
  }
  if (sub != 0) return;
  const int a0 = P.sh.ao[a], b0 = P.sh.ao[b], n = P.nao;
#pragma unroll
  for (int k = 0; k < KO; ++k) {
    const int o = l + k * G;
    if (o >= NA * NB) break;
    const int i = o / NB, j = o % NB;
    const double nrm = cart_norm(LA, i) * cart_norm(LB, j);
    const size_t ij = (size_t)(a0 + i) * n + b0 + j, ji = (size_t)(b0 + j) * n + a0 + i;
    if (P.S) P.S[ij] = P.S[ji] = sa[k] * nrm;
    if (P.T) P.T[ij] = P.T[ji] = ta[k] * nrm;
    if (P.V) P.V[ij] = P.V[ji] = va[k] * nrm;
  }
}

// kOneWarps pairs of one pair class per CTA; the classes' CTAs in the order
// dd, dp, ds, pp, ps, ss (the long ones first)
__global__ void __launch_bounds__(kOneWarps * 32, 2) one_electron_kernel(OneParams P) {
  __shared__ __align__(16) double smem[kOneSmem];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int cls = kNumPairClass - 1, blk = blockIdx.x;
  for (; cls > 0; --cls) {
    const int nb = (P.cstart[cls + 1] - P.cstart[cls] + kOneWarps - 1) / kOneWarps;
    if (blk < nb) break;
    blk -= nb;
  }
  const int pair = P.cstart[cls] + blk * kOneWarps + warp;
  if (pair >= P.cstart[cls + 1]) return;
  double zs = 0.0;   // summed nuclear charge, for the primitive bound
  if (P.V) {
    float z = 0.0f;
    for (int k = lane; k < P.natom; k += 32) z += fabsf((float)P.charges[k]);
    for (int off = 16; off > 0; off >>= 1) z += __shfl_xor_sync(0xffffffffu, z, off);
    zs = z;
  }
  double *sm = smem + warp * (kOneSmem / kOneWarps);
  switch (cls) {
    case 0: one_pair<0, 0>(P, pair, sm, zs, lane); break;
    case 1: one_pair<1, 0>(P, pair, sm, zs, lane); break;
    case 2: one_pair<1, 1>(P, pair, sm, zs, lane); break;
    case 3: one_pair<2, 0>(P, pair, sm, zs, lane); break;
    case 4: one_pair<2, 1>(P, pair, sm, zs, lane); break;
    default: one_pair<2, 2>(P, pair, sm, zs, lane); break;
  }
}

cudaError_t launch_one_electron(const OneParams &P, cudaStream_t st) {
  int n = 0;
  for (int c = 0; c < kNumPairClass; ++c) n += (P.cstart[c + 1] - P.cstart[c] + kOneWarps - 1) / kOneWarps;
  if (n == 0) return cudaSuccess;
  one_electron_kernel<<<n, kOneWarps * 32, 0, st>>>(P);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Gradient of E1 = sum_ij D_ij (T_ij + V_ij) - W_ij S_ij.  Per canonical pair
// (a, b) and primitive pair, with P fixed or X = A - B fixed:
//  * a derivative with respect to A is alpha/p d/dP + d/dX, to B
//    beta/p d/dP - d/dX;
//  * d/dP raises a Hermite function, so with H_tuv = sum_ij D_ij E E E the force
//    on nucleus C is Z sum_tuv H_tuv R_{t+1,u,v} (x direction) and d/dP is minus
//    the sum of these over the nuclei;
//  * d/dX acts on the E coefficients, with dphi/dA = 2 alpha phi_{+1} - a phi_{-1}:
//    dE_t/dX = 2 alpha E^{i+1,j}_t - i E^{i-1,j}_t - alpha/p E^{ij}_{t-1}, contracted
//    with S_tuv = sum_C -Z_C R_tuv once per primitive pair;
//  * S and T (two-centre): the bra derivative from one-dimensional overlap and
//    kinetic tables and their derivatives, the ket one is minus it.
// Lanes as in one_electron_kernel: groups of G lanes per primitive pair, lanes
// over nuclei, then over the block's entries.  A warp strides over the pairs
// and keeps the forces in its own shared-memory copy (one per group, so no
// atomics), flushed once at the end: every pair adds to all 3 natom words.
// Primitive pairs whose contributions all stay below 1e-15 are skipped (bounds
// as in one_electron_kernel with one more power on either side, times the block
// maximum of |D|, |W| and the growth of a derivative, 2 max(alpha, beta) + L).
// Forces of (H2O)8 6-31G*, FP32 + double-float, 7.6 -> 6.4 ms (before: a CTA per pair,
// bra and ket Hermite coefficients per primitive pair, one global atomic per nucleus and
// direction).
constexpr int kOneGradWarps = 2;
constexpr int kOneGradAtoms = 128;   // larger molecules add to global memory directly

template <int LA, int LB>
struct OneGrad {
  static constexpr int L = LA + LB, IJ = (LA + 1) * (LB + 1);
  static constexpr int NT = ntuv(L);
  static constexpr int ES = IJ * (L + 1);                      // E_t of one direction
  // doubles of a group: E, dE/dX (3 directions), s, k, ds, dk (3), S_tuv, H_tuv
  static constexpr int GROUP = 6 * ES + 12 * IJ + 2 * NT;
  static constexpr int WARP = 4 * GROUP + 2 * ncart(LA) * ncart(LB);   // four groups, D and W blocks
};
constexpr int kOneGradWarp = OneGrad<2, 2>::WARP;   // the largest

template <int LA, int LB>
__device__ __forceinline__ void one_pair_grad(const OneParams &P, const double *Dm, const double *Wm, double *frc,
                                              int fstride, double *grad, int pair, double *smem, float zs, int lane) {
  using O = OneGrad<LA, LB>;
  constexpr int NA = ncart(LA), NB = ncart(LB), L = O::L, L1 = L + 1, IJ = O::IJ, NT = O::NT, ES = O::ES;
  const int a = P.pr.a[pair], b = P.pr.b[pair], np = P.pr.np[pair];
  const double *rec0 = P.rec + (size_t)P.pr.poff[pair] * kPrimRec;
  const int G = np >= 3 ? 8 : np == 2 ? 16 : 32;
  const int sub = lane / G, l = lane % G, ngrp = 32 / G;
  double *E = smem + sub * O::GROUP, *X = E + 3 * ES, *s1 = X + 3 * ES, *k1 = s1 + 3 * IJ, *ds = k1 + 3 * IJ,
         *dk = ds + 3 * IJ, *St = dk + 3 * IJ, *Ht = St + NT;
  double *Db = smem + 4 * O::GROUP, *Wb = Db + NA * NB;
#define SF_IJ(d, i, j) ((d) * IJ + (i) * (LB + 1) + (j))
#define SF_ET(d, i, j, t) (SF_IJ(d, i, j) * (L + 1) + (t))
  const double A[3] = {P.sh.cx[a], P.sh.cy[a], P.sh.cz[a]};
  const double B[3] = {P.sh.cx[b], P.sh.cy[b], P.sh.cz[b]};
  const int a0 = P.sh.ao[a], b0 = P.sh.ao[b], n = P.nao;
  const double mult = a == b ? 1.0 : 2.0;   // (i, j) and (j, i)
  float dw = 0.0f;
  __syncwarp();
  for (int k = lane; k < NA * NB; k += 32) {
    const double nrm = mult * cart_norm(LA, k / NB) * cart_norm(LB, k % NB);
    const size_t at = (size_t)(a0 + k / NB) * n + b0 + k % NB;
    Db[k] = Dm[at] * nrm;
    Wb[k] = Wm[at] * nrm;
    dw = fmaxf(dw, fmaxf(fabsf((float)Db[k]), fabsf((float)Wb[k])));
  }
  for (int off = 16; off > 0; off >>= 1) dw = fmaxf(dw, __shfl_xor_sync(0xffffffffu, dw, off));
  const float R1 = sqrtf((float)((A[0] - B[0]) * (A[0] - B[0]) + (A[1] - B[1]) * (A[1] - B[1]) +
                                 (A[2] - B[2]) * (A[2] - B[2])));
  double gst[3] = {0.0, 0.0, 0.0}, gva[3] = {0.0, 0.0, 0.0}, gvp[3] = {0.0, 0.0, 0.0};
  for (int i0 = 0; i0 < np; i0 += ngrp) {
    const int ip = i0 + sub;
    bool on = ip < np;
    const double *rec = rec0 + (size_t)(on ? ip : 0) * kPrimRec;
    const double p = rec[0], Pc[3] = {rec[1], rec[2], rec[3]}, kt = rec[4], hp = rec[5], al = rec[6], be = rec[7];
    {
      const float pf = (float)p, g = fabsf((float)kt) * 0.9414f * rsqrtf(pf) * dw;
      const float x = R1 + rsqrtf(pf) + 1.0f, mx = (float)fmax(al, be);
      float e = x;
#pragma unroll
      for (int k = 0; k < L; ++k) e *= x;
      const float f = (2.0f * mx + L1) * (1.0f + 1.1284f * sqrtf(pf) * zs +
                                          kinetic_bound(LA + 1, LB + 1, (float)al, (float)be, pf, R1));
      if (g * e * f < 1e-15f) on = false;   // not on NaN: it has to reach the forces
    }
    if (!__any_sync(0xffffffffu, on)) continue;
    __syncwarp();   // the previous pass is done with the tables
    const double ap = 2.0 * al * hp;   // alpha / p
    if (on && l < 3) {
      const double pa = l == 0 ? Pc[0] - A[0] : l == 1 ? Pc[1] - A[1] : Pc[2] - A[2];
      const double pb = l == 0 ? Pc[0] - B[0] : l == 1 ? Pc[1] - B[1] : Pc[2] - B[2];
      double Et[LA + 2][LB + 3][LA + LB + 4];
      hermite_e<LA + 1, LB + 2>(hp, pa, pb, Et);
      double kin[LA + 2][LB + 1];   // one-dimensional kinetic energy
#pragma unroll
      for (int i = 0; i <= LA + 1; ++i)
#pragma unroll
        for (int j = 0; j <= LB; ++j) {
          double t = be * ((2 * j + 1) * Et[i][j][0] - 2.0 * be * Et[i][j + 2][0]);
          if (j >= 2) t -= 0.5 * j * (j - 1) * Et[i][j - 2][0];
          kin[i][j] = t;
        }
#pragma unroll
      for (int i = 0; i <= LA; ++i)
#pragma unroll
        for (int j = 0; j <= LB; ++j) {
          s1[SF_IJ(l, i, j)] = Et[i][j][0];
          k1[SF_IJ(l, i, j)] = kin[i][j];
          ds[SF_IJ(l, i, j)] = 2.0 * al * Et[i + 1][j][0] - (i > 0 ? i * Et[i - 1][j][0] : 0.0);
          dk[SF_IJ(l, i, j)] = 2.0 * al * kin[i + 1][j] - (i > 0 ? i * kin[i - 1][j] : 0.0);
#pragma unroll
          for (int t = 0; t <= L; ++t) {
            E[SF_ET(l, i, j, t)] = Et[i][j][t];
            X[SF_ET(l, i, j, t)] = 2.0 * al * Et[i + 1][j][t] - (i > 0 ? i * Et[i - 1][j][t] : 0.0) -
                                   (t > 0 ? ap * Et[i][j][t - 1] : 0.0);
          }
        }
    }
    __syncwarp();
    const double sp = kt * 0.941396263776714813 * rsqrt_nr(p), vp = kt * 1.06225193202719693;
    if (on) {
      // density-contracted Hermite coefficients, Hermite triples over the lanes
      int k = 0;
#pragma unroll 1
      for (int t = 0; t <= L; ++t)
#pragma unroll 1
        for (int u = 0; u <= L - t; ++u)
#pragma unroll 1
          for (int v = 0; v <= L - t - u; ++v, ++k) {
            if (k % G != l) continue;
            double h = 0.0;
            for (int o = 0; o < NA * NB; ++o) {
              const int i = o / NB, j = o % NB;
              const int ax = cart_e(LA, i, 0), ay = cart_e(LA, i, 1), az = cart_e(LA, i, 2);
              const int bx = cart_e(LB, j, 0), by = cart_e(LB, j, 1), bz = cart_e(LB, j, 2);
              if (t <= ax + bx && u <= ay + by && v <= az + bz)
                h += Db[o] * E[SF_ET(0, ax, bx, t)] * (E[SF_ET(1, ay, by, u)] * E[SF_ET(2, az, bz, v)]);
            }
            Ht[k] = vp * h;
          }
      // overlap and kinetic bra derivatives, entries over the lanes
      for (int o = l; o < NA * NB; o += G) {
        const int i = o / NB, j = o % NB;
        const int x = SF_IJ(0, cart_e(LA, i, 0), cart_e(LB, j, 0)), y = SF_IJ(1, cart_e(LA, i, 1), cart_e(LB, j, 1)),
                  z = SF_IJ(2, cart_e(LA, i, 2), cart_e(LB, j, 2));
        const double d = sp * Db[o], w = sp * Wb[o];
        const double sx = s1[x], sy = s1[y], sz = s1[z], kx = k1[x], ky = k1[y], kz = k1[z];
        // D (k' s s + s' k s + s' s k) - W s' s s
        const double dx = ds[x], dy = ds[y], dz = ds[z];
        gst[0] += d * (dk[x] * sy * sz + dx * (ky * sz + sy * kz)) - w * dx * sy * sz;
        gst[1] += d * (dk[y] * sx * sz + dy * (kx * sz + sx * kz)) - w * dy * sx * sz;
        gst[2] += d * (dk[z] * sx * sy + dz * (kx * sy + sx * ky)) - w * dz * sx * sy;
      }
    }
    __syncwarp();
    double st[NT], gp[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < NT; ++k) st[k] = 0.0;
    for (int at = on ? l : P.natom; at < P.natom; at += G) {
      const double pc[3] = {Pc[0] - P.atom_xyz[3 * at], Pc[1] - P.atom_xyz[3 * at + 1], Pc[2] - P.atom_xyz[3 * at + 2]};
      double F[L1 + 1];
      boys_table<L1>(P.boys, p * (pc[0] * pc[0] + pc[1] * pc[1] + pc[2] * pc[2]), F);
      double R[L1 + 1][L1 + 1][L1 + 1];
      hermite_r<L1>(p, pc, F, R);
      double q[3] = {0.0, 0.0, 0.0};
      const double z = P.charges[at];
#pragma unroll
      for (int t = 0; t <= L; ++t)
#pragma unroll
        for (int u = 0; u <= L - t; ++u)
#pragma unroll
          for (int v = 0; v <= L - t - u; ++v) {
            const int k = tuv_index(L, t, u, v);
            const double h = Ht[k];
            q[0] += h * R[t + 1][u][v];
            q[1] += h * R[t][u + 1][v];
            q[2] += h * R[t][u][v + 1];
            st[k] -= z * R[t][u][v];
          }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        q[d] *= z;
        gp[d] -= q[d];
        if (frc) frc[sub * fstride + 3 * at + d] += q[d];
        else atomicAdd(grad + 3 * at + d, q[d]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      gvp[d] += gp[d];
      gva[d] += ap * gp[d];
    }
    for (int off = 1; off < G; off <<= 1) {
#pragma unroll
      for (int k = 0; k < NT; ++k) st[k] += __shfl_xor_sync(0xffffffffu, st[k], off);
    }
    if (l == 0) {
#pragma unroll
      for (int k = 0; k < NT; ++k) St[k] = vp * st[k];
    }
    __syncwarp();
    if (on) {
      for (int o = l; o < NA * NB; o += G) {
        const int i = o / NB, j = o % NB;
        const int ax = cart_e(LA, i, 0), ay = cart_e(LA, i, 1), az = cart_e(LA, i, 2);
        const int bx = cart_e(LB, j, 0), by = cart_e(LB, j, 1), bz = cart_e(LB, j, 2);
        const double *ex = E + SF_ET(0, ax, bx, 0), *ey = E + SF_ET(1, ay, by, 0), *ez = E + SF_ET(2, az, bz, 0);
        const double *xx = X + SF_ET(0, ax, bx, 0), *xy = X + SF_ET(1, ay, by, 0), *xz = X + SF_ET(2, az, bz, 0);
        double vx = 0.0, vy = 0.0, vz = 0.0;
        for (int t = 0; t <= ax + bx; ++t) {
          double e0 = 0.0, ey1 = 0.0, ez1 = 0.0;   // E_u E_v S, dE_u E_v S, E_u dE_v S
          for (int u = 0; u <= ay + by; ++u) {
            double c = 0.0, cz = 0.0;
            for (int v = 0; v <= az + bz; ++v) {
              const double sv = St[tuv_index(L, t, u, v)];
              c += ez[v] * sv;
              cz += xz[v] * sv;
            }
            e0 += ey[u] * c;
            ey1 += xy[u] * c;
            ez1 += ey[u] * cz;
          }
          vx += xx[t] * e0;
          vy += ex[t] * ey1;
          vz += ex[t] * ez1;
        }
        gva[0] += Db[o] * vx;
        gva[1] += Db[o] * vy;
        gva[2] += Db[o] * vz;
      }
    }
  }
#undef SF_IJ
#undef SF_ET
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      gst[d] += __shfl_xor_sync(0xffffffffu, gst[d], off);
      gva[d] += __shfl_xor_sync(0xffffffffu, gva[d], off);
      gvp[d] += __shfl_xor_sync(0xffffffffu, gvp[d], off);
    }
  }
  __syncwarp();
  if (lane < 3) {
    const double s = lane == 0 ? gst[0] : lane == 1 ? gst[1] : gst[2];
    const double va = lane == 0 ? gva[0] : lane == 1 ? gva[1] : gva[2];
    const double vp = lane == 0 ? gvp[0] : lane == 1 ? gvp[1] : gvp[2];
    const int ia = 3 * P.sh.atom[a] + lane, ib = 3 * P.sh.atom[b] + lane;
    if (frc) {
      frc[ia] += s + va;
      frc[ib] += vp - va - s;
    } else {
      atomicAdd(grad + ia, s + va);
      atomicAdd(grad + ib, vp - va - s);
    }
  }
  __syncwarp();
}

// warps stride over the pairs in the order dd, dp, ds, pp, ps, ss (the long
// ones first)
__global__ void __launch_bounds__(kOneGradWarps * 32, 4) one_electron_grad_kernel(OneParams P, const double *D,
                                                                                 const double *W, double *grad) {
  extern __shared__ __align__(16) double sm_grad[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *tab = sm_grad + warp * kOneGradWarp;
  const int fstride = 3 * P.natom;
  double *frc = P.natom <= kOneGradAtoms ? sm_grad + kOneGradWarps * kOneGradWarp + warp * 4 * fstride : nullptr;
  if (frc)
    for (int k = lane; k < 4 * fstride; k += 32) frc[k] = 0.0;
  float zs = 0.0f;
  for (int k = lane; k < P.natom; k += 32) zs += fabsf((float)P.charges[k]);
  for (int off = 16; off > 0; off >>= 1) zs += __shfl_xor_sync(0xffffffffu, zs, off);
  __syncwarp();
  const int npair = P.cstart[kNumPairClass];
  for (int k = blockIdx.x * kOneGradWarps + warp; k < npair; k += gridDim.x * kOneGradWarps) {
    const int pair = npair - 1 - k;
    int cls = 0;
    while (pair >= P.cstart[cls + 1]) ++cls;
    switch (cls) {
      case 0: one_pair_grad<0, 0>(P, D, W, frc, fstride, grad, pair, tab, zs, lane); break;
      case 1: one_pair_grad<1, 0>(P, D, W, frc, fstride, grad, pair, tab, zs, lane); break;
      case 2: one_pair_grad<1, 1>(P, D, W, frc, fstride, grad, pair, tab, zs, lane); break;
      case 3: one_pair_grad<2, 0>(P, D, W, frc, fstride, grad, pair, tab, zs, lane); break;
      case 4: one_pair_grad<2, 1>(P, D, W, frc, fstride, grad, pair, tab, zs, lane); break;
      default: one_pair_grad<2, 2>(P, D, W, frc, fstride, grad, pair, tab, zs, lane); break;
    }
  }
  if (!frc) return;
  __syncthreads();
  // the CTA's warps and groups, one atomic per word
  const double *f = sm_grad + kOneGradWarps * kOneGradWarp;
  for (int k = threadIdx.x; k < fstride; k += blockDim.x) {
    double s = 0.0;
#pragma unroll
    for (int g = 0; g < 4 * kOneGradWarps; ++g) s += f[g * fstride + k];
    if (s != 0.0) atomicAdd(grad + k, s);
  }
}

static size_t one_grad_smem(int natom) {
  const size_t f = natom <= kOneGradAtoms ? (size_t)kOneGradWarps * 4 * 3 * natom : 0;
  return (kOneGradWarps * (size_t)kOneGradWarp + f) * sizeof(double);
}

cudaError_t prepare_one_electron() {
  return cudaFuncSetAttribute(one_electron_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)one_grad_smem(kOneGradAtoms));
}

cudaError_t launch_one_electron_grad(const OneParams &P, const double *D, const double *W, double *grad, int nsm,
                                     cudaStream_t st) {
  const int npair = P.cstart[kNumPairClass];
  if (npair == 0) return cudaSuccess;
  const int ctas = (npair + kOneGradWarps - 1) / kOneGradWarps, most = (nsm < 1 ? 1 : nsm) * 4;
  one_electron_grad_kernel<<<ctas < most ? ctas : most, kOneGradWarps * 32, one_grad_smem(P.natom), st>>>(P, D, W, grad);
  return cudaGetLastError();
}

}  // namespace sf
