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
  if (T >= kTabXmax) {
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

// E[i][j][t] for i <= LI, j <= LJ, t <= i+j along one direction
template <int LI, int LJ>
__device__ __forceinline__ void hermite_e(double p, double xpa, double xpb, double e0,
                                          double (&E)[LI + 1][LJ + 1][LI + LJ + 1]) {
#pragma unroll
  for (int i = 0; i <= LI; ++i)
#pragma unroll
    for (int j = 0; j <= LJ; ++j)
#pragma unroll
      for (int t = 0; t <= LI + LJ; ++t) E[i][j][t] = 0.0;
  const double h = 0.5 / p;
  E[0][0][0] = e0;
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


// the same from 1/(2p) with E^00_0 = 1 (the product Gaussian kept apart)
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
// 3 beta (LB + 2) and attraction as 2 sqrt(p/pi) times the summed charge; the
// bound itself in FP32).
// (H2O)16 6-31G* (48 nuclei, 68 k primitive pairs): 0.32 ms; one CTA of 64 threads
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
    const double p = rec[0], Pc[3] = {rec[1], rec[2], rec[3]}, kt = rec[4], hp = rec[5], be = rec[7];
    {
      // kt = c_i c_j exp(-mu R^2) sqrt(2) pi^(5/4) / p
      const float pf = (float)p, g = fabsf((float)kt) * 0.9414f * rsqrtf(pf);   // overlap bound
      const float x = R1 + rsqrtf(pf) + 1.0f;
      float e = 1.0f;
#pragma unroll
      for (int k = 0; k < L; ++k) e *= x;
      const float f = 1.0f + 1.1284f * sqrtf(pf) * (float)zs + 3.0f * (float)be * (LB + 2);
      if (!(g * e * f >= 1e-17f)) on = false;
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
// Gradient of E1 = sum_ij D_ij (T_ij + V_ij) - W_ij S_ij.  With D, W and the
// operators symmetric, d/dR sum_ij D_ij O_ij = 2 sum_ij D_ij <d phi_i/dR|O|phi_j>
// over ordered shell pairs; per canonical pair (a >= b) both the bra and the
// ket derivative are taken, d phi/dA = 2 alpha phi_{+1} - a phi_{-1}:
//  * S and T (two-centre): the ket derivative is minus the bra one;
//  * V: the bra and ket derivative share R_tuv(p, P - C) of each nucleus C,
//    which receives minus their sum (translational invariance of
//    <a|1/r_C|b>).
// CTA per canonical pair (a, b), 64 threads.  For every primitive pair whose
// bound (product Gaussian x block max of |D|, |W| x derivative, kinetic and
// attraction factors) is not below 1e-15:
//  * E coefficients (bra to LA+1, ket to LB+2) into shared memory;
//  * the S and T bra-derivative terms, one (i, j, direction) per thread;
//  * the density-contracted Hermite coefficients of the bra and the ket
//    derivative, M^d_tuv = 2pi/p c_i c_j sum_{i in a, j in b} D_ij sum_+- f
//    E.. E.. E.. (nucleus independent), cooperatively into shared memory;
//  * every thread takes nuclei C = t, t+64, ...: Boys values F_m(p |P-C|^2)
//    = sum_i w_i u_i^m from the FP64 Rys rule of floor(L/2)+1 points (exact
//    for m <= L), R_tuv by the Hermite Coulomb recursion, and
//    dV/dX_d = -Z_C sum_tuv M^d_tuv R_tuv.
constexpr int kOneGradThreads = 64;

// shared-memory doubles of one_pair_grad2<LA, LB>: E coefficients, the bra and
// ket Hermite coefficients MA, MB, the density block and the reduction rows
template <int LA, int LB>
constexpr int one_grad_smem() {
  return 3 * (LA + 2) * (LB + 3) * (LA + LB + 4) + 6 * (LA + LB + 2) * (LA + LB + 2) * (LA + LB + 2) +
         ncart(LA) * ncart(LB) + 6 * kOneGradThreads;
}
constexpr int kOneGradSmem = one_grad_smem<2, 2>();   // the largest

template <int LA, int LB>
__device__ void one_pair_grad2(const OneParams &P, const double *Dm, const double *Wm, double *grad, int a, int b,
                               double *smem) {
  constexpr int NA = ncart(LA), NB = ncart(LB);
  constexpr int LE = LA + 1, L = LA + LB + 1, NH = (L + 1) * (L + 1) * (L + 1);
  constexpr int NRT = L / 2 + 1;   // Rys points whose rule is exact for F_0 .. F_L
  constexpr int EN = (LE + 1) * (LB + 3) * (LE + LB + 3);
  const double pi = 3.14159265358979323846;
  // carved from the kernel's one shared buffer (each instantiation declaring
  // its own arrays made the kernel hold all nine sets, 79.5 KB)
  using EArr = double[LE + 1][LB + 3][LE + LB + 3];
  EArr *E = reinterpret_cast<EArr *>(smem);
  double(*MA)[NH] = reinterpret_cast<double(*)[NH]>(smem + 3 * EN);
  double(*MB)[NH] = MA + 3;
  double(*Dab)[NB] = reinterpret_cast<double(*)[NB]>(smem + 3 * EN + 6 * NH);
  double(*red)[6] = reinterpret_cast<double(*)[6]>(smem + 3 * EN + 6 * NH + NA * NB);
  static_assert(3 * EN + 6 * NH + NA * NB + 6 * kOneGradThreads == one_grad_smem<LA, LB>(), "smem layout");
  const int tid = threadIdx.x;
  const bool two = a != b;   // canonical pair with a distinct ket: ket derivative too
  const double A[3] = {P.sh.cx[a], P.sh.cy[a], P.sh.cz[a]};
  const double B[3] = {P.sh.cx[b], P.sh.cy[b], P.sh.cz[b]};
  const int a0 = P.sh.ao[a], b0 = P.sh.ao[b], n = P.nao;
  // block maximum of |D| and |W| and the summed nuclear charge: the scale of
  // everything this pair adds, for the primitive-pair screening below
  double dw = 0.0, zs = 0.0;
  for (int k = tid; k < NA * NB; k += blockDim.x) {
    const int i = k / NB, j = k % NB;
    const double nrm = cart_norm(LA, i) * cart_norm(LB, j);
    Dab[i][j] = Dm[(a0 + i) * n + b0 + j] * nrm;
    dw = fmax(dw, fmax(fabs(Dab[i][j]), fabs(Wm[(a0 + i) * n + b0 + j] * nrm)));
  }
  for (int k = tid; k < P.natom; k += blockDim.x) zs += fabs(P.charges[k]);
  for (int off = 16; off > 0; off >>= 1) {
    dw = fmax(dw, __shfl_xor_sync(0xffffffffu, dw, off));
    zs += __shfl_xor_sync(0xffffffffu, zs, off);
  }
  if ((tid & 31) == 0) {
    red[tid >> 5][0] = dw;
    red[tid >> 5][1] = zs;
  }
  __syncthreads();
  dw = 0.0;
  zs = 0.0;
  for (int w = 0; w < (int)blockDim.x / 32; ++w) {
    dw = fmax(dw, red[w][0]);
    zs += red[w][1];
  }
  __syncthreads();   // red is written again by the final reduction
  double R2 = 0.0;
  for (int d = 0; d < 3; ++d) R2 += (A[d] - B[d]) * (A[d] - B[d]);
  double gST[3] = {0.0, 0.0, 0.0}, gVA[3] = {0.0, 0.0, 0.0}, gVB[3] = {0.0, 0.0, 0.0};
  for (int ia = P.poff[a]; ia < P.poff[a + 1]; ++ia)
    for (int ib = P.poff[b]; ib < P.poff[b + 1]; ++ib) {
      const double al = P.exps[ia], be = P.exps[ib], p = al + be, mu = al * be / p;
      const double cc = P.coefs[ia] * P.coefs[ib];
      // primitive pairs whose contributions all stay below 1e-15 are skipped
      // (the same on every thread, so the barriers below stay uniform): the
      // product Gaussian c_i c_j exp(-mu |AB|^2) (pi/p)^3/2 bounds the
      // overlap; E coefficients grow at most as (|AB| + 1/sqrt(p) + 1)^(L+1),
      // derivatives as 2 max(alpha, beta) + L, kinetic terms as
      // 3 beta (LB + 2), attraction as 2 sqrt(p/pi) times the summed charge
      {
        const double g = fabs(cc) * exp(-mu * R2) * pow(pi / p, 1.5) * dw;
        const double e = pow(sqrt(R2) + rsqrt(p) + 1.0, (double)(L + 1));
        const double f = (2.0 * fmax(al, be) + L) * (1.0 + 2.0 * sqrt(p / pi) * zs + 3.0 * fmax(al, be) * (LB + 2));
        if (g * e * f < 1e-15) continue;
      }
      double Pc[3];
      for (int d = 0; d < 3; ++d) Pc[d] = (al * A[d] + be * B[d]) / p;
      __syncthreads();   // previous iteration done with E, M
      if (tid < 3) {
        const int d = tid;
        const double X = A[d] - B[d];
        double Et[LE + 1][LB + 3][LE + LB + 3];
        hermite_e<LE, LB + 2>(p, Pc[d] - A[d], Pc[d] - B[d], exp(-mu * X * X), Et);
        for (int i = 0; i <= LE; ++i)
          for (int j = 0; j <= LB + 2; ++j)
            for (int t = 0; t <= LE + LB + 2; ++t) E[d][i][j][t] = Et[i][j][t];
      }
      __syncthreads();
      // overlap / kinetic bra derivatives (Pulay -W dS, D dT), one (i, j, d)
      // per thread (gST is summed over the CTA at the end)
      {
        const double sp = pow(pi / p, 1.5);
        for (int task = tid; task < NA * NB * 3; task += blockDim.x) {
            const int i = task / (NB * 3), j = (task / 3) % NB, d = task % 3;
            const double nrm = cart_norm(LA, i) * cart_norm(LB, j);
            const double Dij = Dab[i][j], Wij = Wm[(a0 + i) * n + b0 + j] * nrm;
            const int bx[3] = {cart_e(LB, j, 0), cart_e(LB, j, 1), cart_e(LB, j, 2)};
            {
              double dS = 0.0, dT = 0.0;
              for (int sgn = 0; sgn < 2; ++sgn) {
                int ax[3] = {cart_e(LA, i, 0), cart_e(LA, i, 1), cart_e(LA, i, 2)};
                const int ad = ax[d];
                if (sgn == 1 && ad == 0) continue;
                ax[d] += sgn == 0 ? 1 : -1;
                const double f = sgn == 0 ? 2.0 * al : -(double)ad;
                const double sx = E[0][ax[0]][bx[0]][0], sy = E[1][ax[1]][bx[1]][0], sz = E[2][ax[2]][bx[2]][0];
                const double s0 = sx * sy * sz * sp;
                double t = be * (2 * (bx[0] + bx[1] + bx[2]) + 3) * s0;
                t -= 2.0 * be * be * sp *
                     (E[0][ax[0]][bx[0] + 2][0] * sy * sz + sx * E[1][ax[1]][bx[1] + 2][0] * sz +
                      sx * sy * E[2][ax[2]][bx[2] + 2][0]);
                if (bx[0] >= 2) t -= 0.5 * bx[0] * (bx[0] - 1) * sp * E[0][ax[0]][bx[0] - 2][0] * sy * sz;
                if (bx[1] >= 2) t -= 0.5 * bx[1] * (bx[1] - 1) * sp * sx * E[1][ax[1]][bx[1] - 2][0] * sz;
                if (bx[2] >= 2) t -= 0.5 * bx[2] * (bx[2] - 1) * sp * sx * sy * E[2][ax[2]][bx[2] - 2][0];
                dS += f * s0;
                dT += f * t;
              }
              gST[d] += cc * (Dij * dT - Wij * dS);
            }
          }
      }
      // density-contracted Hermite coefficients of the bra (MA) and ket (MB) derivatives
      const double pre = 2.0 * pi / p * cc;
      for (int k = tid; k < 3 * NH; k += blockDim.x) {
        const int d = k / NH, h = k % NH;
        const int t = h / ((L + 1) * (L + 1)), u = (h / (L + 1)) % (L + 1), v = h % (L + 1);
        double ma = 0.0, mb = 0.0;
        if (t + u + v <= L) {
          for (int i = 0; i < NA; ++i)
            for (int j = 0; j < NB; ++j) {
              const int ax0[3] = {cart_e(LA, i, 0), cart_e(LA, i, 1), cart_e(LA, i, 2)};
              const int bx0[3] = {cart_e(LB, j, 0), cart_e(LB, j, 1), cart_e(LB, j, 2)};
              double acca = 0.0, accb = 0.0;
              for (int sgn = 0; sgn < 2; ++sgn) {
                {
                  int ax[3] = {ax0[0], ax0[1], ax0[2]};
                  const int ad = ax[d];
                  if (!(sgn == 1 && ad == 0)) {
                    ax[d] += sgn == 0 ? 1 : -1;
                    if (t <= ax[0] + bx0[0] && u <= ax[1] + bx0[1] && v <= ax[2] + bx0[2]) {
                      const double f = sgn == 0 ? 2.0 * al : -(double)ad;
                      acca += f * E[0][ax[0]][bx0[0]][t] * E[1][ax[1]][bx0[1]][u] * E[2][ax[2]][bx0[2]][v];
                    }
                  }
                }
                if (two) {
                  int bx[3] = {bx0[0], bx0[1], bx0[2]};
                  const int bd = bx[d];
                  if (!(sgn == 1 && bd == 0)) {
                    bx[d] += sgn == 0 ? 1 : -1;
                    if (t <= ax0[0] + bx[0] && u <= ax0[1] + bx[1] && v <= ax0[2] + bx[2]) {
                      const double f = sgn == 0 ? 2.0 * be : -(double)bd;
                      accb += f * E[0][ax0[0]][bx[0]][t] * E[1][ax0[1]][bx[1]][u] * E[2][ax0[2]][bx[2]][v];
                    }
                  }
                }
              }
              ma += Dab[i][j] * acca;
              mb += Dab[i][j] * accb;
            }
        }
        MA[d][h] = pre * ma;
        MB[d][h] = pre * mb;
      }
      __syncthreads();
      for (int at = tid; at < P.natom; at += blockDim.x) {
        const double pc[3] = {Pc[0] - P.atom_xyz[3 * at], Pc[1] - P.atom_xyz[3 * at + 1],
                              Pc[2] - P.atom_xyz[3 * at + 2]};
        double F[L + 1];
        {
          double ur[NRT], wr[NRT];
          rys_roots_f64_tab<NRT>(P.tab64, P.asym, p * (pc[0] * pc[0] + pc[1] * pc[1] + pc[2] * pc[2]), ur, wr);
          double pw[NRT];
#pragma unroll
          for (int r = 0; r < NRT; ++r) pw[r] = wr[r];
#pragma unroll
          for (int m = 0; m <= L; ++m) {
            double f = 0.0;
#pragma unroll
            for (int r = 0; r < NRT; ++r) {
              f += pw[r];
              pw[r] *= ur[r];
            }
            F[m] = f;
          }
        }
        // R^m_tuv by the Hermite Coulomb recursion, in place: level m
        // overwrites t+u+w = L-m .. 1 from the top down (each entry needs
        // level m+1 at t+u+w-1 and -2, not yet overwritten), then R^m_000
        double R[L + 1][L + 1][L + 1];
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
        double da[3] = {0.0, 0.0, 0.0}, db[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int t = 0; t <= L; ++t)
#pragma unroll
          for (int u = 0; u <= L - t; ++u)
#pragma unroll
            for (int w = 0; w <= L - t - u; ++w) {
              const int h = (t * (L + 1) + u) * (L + 1) + w;
              const double rr = R[t][u][w];
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                da[d] += MA[d][h] * rr;
                db[d] += MB[d][h] * rr;
              }
            }
        const double z = -P.charges[at];
        for (int d = 0; d < 3; ++d) {
          gVA[d] += z * da[d];
          gVB[d] += z * db[d];
          atomicAdd(grad + 3 * at + d, -2.0 * z * (da[d] + db[d]));
        }
      }
    }
  // reduce over the CTA, one atomic per centre and direction
  for (int d = 0; d < 3; ++d) {
    red[tid][d] = gVA[d] + gST[d];
    red[tid][3 + d] = gVB[d] - gST[d];
  }
  __syncthreads();
  if (tid < 6) {
    double sacc = 0.0;
    for (int k = 0; k < (int)blockDim.x; ++k) sacc += red[k][tid];
    if (tid < 3) atomicAdd(grad + 3 * P.sh.atom[a] + tid, 2.0 * sacc);
    else if (two) atomicAdd(grad + 3 * P.sh.atom[b] + tid - 3, 2.0 * sacc);
  }
}

// one CTA per canonical pair (a >= b): block k = a (a + 1) / 2 + b
__global__ void __launch_bounds__(kOneGradThreads) one_electron_grad_kernel(OneParams P, const double *D,
                                                                            const double *W, double *grad) {
  const int k = blockIdx.x;
  int a = (int)((sqrt(8.0 * k + 1.0) - 1.0) * 0.5);
  while (a * (a + 1) / 2 > k) --a;
  while ((a + 1) * (a + 2) / 2 <= k) ++a;
  const int b = k - a * (a + 1) / 2;
  __shared__ __align__(16) double smem[kOneGradSmem];
  switch (P.sh.l[a] * 3 + P.sh.l[b]) {
    case 0: one_pair_grad2<0, 0>(P, D, W, grad, a, b, smem); break;
    case 1: one_pair_grad2<0, 1>(P, D, W, grad, a, b, smem); break;
    case 2: one_pair_grad2<0, 2>(P, D, W, grad, a, b, smem); break;
    case 3: one_pair_grad2<1, 0>(P, D, W, grad, a, b, smem); break;
    case 4: one_pair_grad2<1, 1>(P, D, W, grad, a, b, smem); break;
    case 5: one_pair_grad2<1, 2>(P, D, W, grad, a, b, smem); break;
    case 6: one_pair_grad2<2, 0>(P, D, W, grad, a, b, smem); break;
    case 7: one_pair_grad2<2, 1>(P, D, W, grad, a, b, smem); break;
    case 8: one_pair_grad2<2, 2>(P, D, W, grad, a, b, smem); break;
    default: break;
  }
}

cudaError_t launch_one_electron_grad(const OneParams &P, const double *D, const double *W, double *grad,
                                     cudaStream_t st) {
  const int n = P.nshell * (P.nshell + 1) / 2;
  if (n == 0) return cudaSuccess;
  one_electron_grad_kernel<<<n, kOneGradThreads, 0, st>>>(P, D, W, grad);
  return cudaGetLastError();
}

}  // namespace sf
