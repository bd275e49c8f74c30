// Closed-form Hellmann-Feynman gradient at fixed converged densities (pm3-rs
// src/gradient.rs:306-599 and src/repulsion.rs:30-49), one thread per atom pair over the pairs
// of every molecule of a batch. Each pair's force is added to atom b and subtracted from atom a with
// FP64 atomics.
//
// A pair's energy is worked out in its own frame, where the 100 two-electron integrals are 34 that do not vanish and
// 22 values, the overlaps five and the attractions four: the density blocks are turned into the frame instead of the
// integrals out of it. Along the axis the integrals change: dual numbers in the distance. Across it only the frame turns:
// with A = dE/dP the derivative by the turning angle is <A, [G, P]>, G mixing sigma with one pi. (The energy does not change when
// the frame turns about the axis.) With every integral a dual number of three partials in the molecular frame a heavy pair was
// 100 rotations of four-fold products: 1000 organics of 10-35 atoms took 3.01 ms (pairs by kind included), 0.47 now, 24 atoms
// 0.22 of 3.9 ms of a call, 0.11 now. Bound by instruction
// fetch (half of the cycles between a warp's instructions: a heavy pair is one long straight run of code) and one thread's chain.
#pragma once
#include "pm3_integrals.cuh"

namespace pm3gpu {

constexpr int kGradThreads = 64;

struct GradMol {
  int atom0, natom, nao, uhf;
  int nh, pad;         // atoms with p orbitals
  long long pair0;     // first global pair index of this molecule
  long long dens_off;  // P_tot [, P_alpha, P_beta] in the density buffer
};

struct GradArgs {
  const ElemDev* elem;
  const PairDev* pairs;
  const int* z;
  const double* xyz;
  const int* ao_off;   // first AO of each atom within its molecule
  const int* order;    // per molecule its atoms (indices within it), those with p orbitals first
  const GradMol* mols;
  int nmol;
  long long npairs;
  const double* dens;
  double* grad;        // [3 * total atoms], zeroed by the host
};

// The two-electron integrals of the local frame that do not vanish: packed orbital pairs of a and of b
// (order s, sigma, pi1, pi2) and the index of their value in local22.
struct LocalInt {
  int p, q, i;
};
__device__ constexpr LocalInt kLocalInts[34] = {
    {0, 0, 0},  {1, 0, 1},  {2, 0, 2},  {5, 0, 3},  {9, 0, 3},  // the first five: all of a heavy atom with a light one
    {0, 1, 4},  {1, 1, 5},  {3, 3, 6},  {6, 6, 6},  {2, 1, 7},  {5, 1, 8},  {9, 1, 8},  {4, 3, 9},  {7, 6, 9},
    {0, 2, 10}, {0, 5, 11}, {0, 9, 11}, {1, 2, 12}, {1, 5, 13}, {1, 9, 13}, {3, 4, 14}, {6, 7, 14},
    {2, 2, 15}, {5, 2, 16}, {9, 2, 16}, {2, 5, 17}, {2, 9, 17}, {5, 5, 18}, {9, 9, 18}, {4, 4, 19}, {7, 7, 19},
    {5, 9, 20}, {9, 5, 20}, {8, 8, 21}};

__device__ __forceinline__ constexpr int hi_of(int p) { return p >= 6 ? 3 : p >= 3 ? 2 : p >= 1 ? 1 : 0; }
__device__ __forceinline__ constexpr int lo_of(int p) { return p - hi_of(p) * (hi_of(p) + 1) / 2; }

// One atom's density block in the frame, packed. E: rows = axes of the frame.
template <int N>
__device__ __forceinline__ void local_diag(const double* P, int o, int n, const double (&E)[9], double (&out)[10]) {
  const double* base = P + (size_t)o * n + o;
  out[0] = base[0];
  if constexpr (N == 4) {
    double t[3][3];
  #pragma unroll
    for (int i = 0; i < 3; ++i) {
      double d = 0.0;
  #pragma unroll
      for (int k = 0; k < 3; ++k) d = fma(E[3 * i + k], base[(size_t)(1 + k) * n], d);
      out[(i + 1) * (i + 2) / 2] = d;
  #pragma unroll
      for (int c = 0; c < 3; ++c) {
        double x = 0.0;
  #pragma unroll
        for (int k = 0; k < 3; ++k) x = fma(E[3 * i + k], base[(size_t)(1 + k) * n + 1 + c], x);
        t[i][c] = x;
      }
    }
  #pragma unroll
    for (int i = 0; i < 3; ++i)
  #pragma unroll
      for (int j = 0; j <= i; ++j)
        out[(i + 1) * (i + 2) / 2 + j + 1] = fma(t[i][2], E[3 * j + 2], fma(t[i][1], E[3 * j + 1], t[i][0] * E[3 * j]));
  }
}

// The block between the two atoms.
template <int NA, int NB>
__device__ __forceinline__ void local_pair(const double* P, int oa, int ob, int n, const double (&E)[9], double (&X)[4][4]) {
  const double* base = P + (size_t)oa * n + ob;
  double y[NA][NB];
#pragma unroll
  for (int i = 0; i < NA; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) y[i][j] = base[(size_t)i * n + j];
  double t[NA][NB];  // rows turned
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    t[0][j] = y[0][j];
#pragma unroll
    for (int i = 1; i < NA; ++i) {
      double x = 0.0;
#pragma unroll
      for (int k = 1; k < NA; ++k) x = fma(E[3 * (i - 1) + k - 1], y[k][j], x);
      t[i][j] = x;
    }
  }
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    X[i][0] = t[i][0];
#pragma unroll
    for (int j = 1; j < NB; ++j) {
      double x = 0.0;
#pragma unroll
      for (int k = 1; k < NB; ++k) x = fma(E[3 * (j - 1) + k - 1], t[i][k], x);
      X[i][j] = x;
    }
  }
}

// <A, [G, P]> of a packed block for G mixing sigma with pi1 (T[0]) and with pi2 (T[1]); A = dE/dP per packed element.
__device__ __forceinline__ void turn_diag(const double (&A)[10], const double (&P)[10], double (&T)[2]) {
  T[0] += A[1] * P[3] - A[3] * P[1] + 2.0 * P[4] * (A[2] - A[5]) + A[4] * (P[5] - P[2]) + A[7] * P[8] - A[8] * P[7];
  T[1] += A[1] * P[6] - A[6] * P[1] + 2.0 * P[7] * (A[2] - A[9]) + A[7] * (P[9] - P[2]) + A[4] * P[8] - A[8] * P[4];
}

// dE/d(R_b - R_a) of one ordered pair (a heavy-first), eV/Bohr; NA, NB: orbitals of the atoms (1 or 4).
template <int NA, int NB>
__device__ __noinline__ void pair_force(const ElemDev& ea, const ElemDev& eb, const PairDev& pp, const double* ra,
                                        const double* rb, int oa, int ob, int n, const double* Pt, bool uhf, double f[3]) {
  const double dv[3] = {rb[0] - ra[0], rb[1] - ra[1], rb[2] - ra[2]};
  const double dist = sqrt(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]), ir = 1.0 / dist;
  const D1 r{dist, 1.0};
  double E[9];  // the frame: row 0 from b to a
  frame(-(dv[0] * ir), -(dv[1] * ir), -(dv[2] * ir), E);
  double de = core_core(ea, eb, pp, r).g;  // dE/dr; first the core-core repulsion
  double T[2] = {0.0, 0.0};                // dE by the angles of row 0 towards rows 1 and 2

  constexpr int kInts = NB == 4 ? 34 : NA == 4 ? 5 : 1;
  D1 ri[22];
  if (NB == 4) {
    local22(ee_pole(ea), ee_pole(eb), r, ri);
  } else if (NA == 4) {
    local4(ee_pole(ea), eb.rho0, r, ri);
  } else {
    const double sr = ea.rho0 + eb.rho0;
    ri[0] = rsq(r * r + sr * sr) * kEv;
  }
  {  // Coulomb terms and the attraction of each atom's electrons by the other's core
    double Pa[10], Pb[10], Aa[10], Ab[10];
    local_diag<NA>(Pt, oa, n, E, Pa);
    local_diag<NB>(Pt, ob, n, E, Pb);
#pragma unroll
    for (int p = 0; p < 10; ++p) Aa[p] = Ab[p] = 0.0;
    auto attraction = [&](const ElemDev& orb, const ElemDev& cor, bool heavy, double sign, const double (&P)[10], double (&A)[10]) {
      const double c = (orb.po1 + cor.po9) * (orb.po1 + cor.po9);
      D1 li[4];
      if (heavy && orb.z >= 3) {
        local4(core_pole(orb), cor.po9, r, li);
        A[1] = -2.0 * sign * cor.core * li[1].v;
        A[2] = -cor.core * li[2].v;
        A[5] = A[9] = -cor.core * li[3].v;
        de -= cor.core * (li[0].g * P[0] + 2.0 * sign * li[1].g * P[1] + li[2].g * P[2] + li[3].g * (P[5] + P[9]));
      } else {
        li[0] = rsq(r * r + c) * kEv;
        de -= cor.core * li[0].g * P[0];
      }
      A[0] = -cor.core * li[0].v;
    };
    attraction(ea, eb, NA == 4, 1.0, Pa, Aa);
    attraction(eb, ea, NB == 4, -1.0, Pb, Ab);  // seen from b the axis points the other way
#pragma unroll
    for (int e = 0; e < kInts; ++e) {
      constexpr auto& tab = kLocalInts;
      const int p = tab[e].p, q = tab[e].q, i = tab[e].i;
      const double m = (hi_of(p) == lo_of(p) ? 1.0 : 2.0) * (hi_of(q) == lo_of(q) ? 1.0 : 2.0);
      Aa[p] = fma(m * ri[i].v, Pb[q], Aa[p]);
      Ab[q] = fma(m * ri[i].v, Pa[p], Ab[q]);
      de = fma(ri[i].g, m * Pa[p] * Pb[q], de);
    }
    if (NA == 4) turn_diag(Aa, Pa, T);
    if (NB == 4) turn_diag(Ab, Pb, T);
  }
  const size_t nn = (size_t)n * n;
  for (int blk = 0; blk < (uhf ? 3 : 1); ++blk) {  // total density: resonance (and exchange when closed-shell); spin densities: exchange
    double X[4][4], A[4][4];
    local_pair<NA, NB>(Pt + blk * nn, oa, ob, n, E, X);
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) A[i][j] = 0.0;
    if (blk == 0) {  // P_ab (beta_i + beta_j) S_ab, both off-diagonal blocks
      const bool swap = ea.npq < eb.npq;
      D1 o[5];
      if (dist >= 1.0e-8 && overlap_local(swap ? eb : ea, swap ? ea : eb, r, o)) {  // constant below, as in overlap_block
        const double ss = ea.bs + eb.bs, ps = ea.bp + eb.bs, sp = ea.bs + eb.bp, p2 = ea.bp + eb.bp;
        A[0][0] = ss * o[0].v;
        de = fma(ss * o[0].g, X[0][0], de);
        if (NA == 4) {
          const D1 x = -(swap ? o[2] : o[1]);
          A[1 % NA][0] = ps * x.v;
          de = fma(ps * x.g, X[1][0], de);
        }
        if (NB == 4) {
          const D1 x = swap ? o[1] : o[2];
          A[0][1 % NB] = sp * x.v;
          de = fma(sp * x.g, X[0][1], de);
        }
        if (NA == 4 && NB == 4) {
          A[1][1] = -p2 * o[3].v;
          A[2][2] = A[3][3] = p2 * o[4].v;
          de += p2 * (o[4].g * (X[2][2] + X[3][3]) - o[3].g * X[1][1]);
        }
      }
    }
    if (blk != 0 || !uhf) {
      const double fx = uhf ? -0.5 : -0.25;
#pragma unroll
      for (int e = 0; e < kInts; ++e) {
        constexpr auto& tab = kLocalInts;
        const int ph = hi_of(tab[e].p), pl = lo_of(tab[e].p), qh = hi_of(tab[e].q), ql = lo_of(tab[e].q), i = tab[e].i;
        const double m = fx * (ph == pl ? 1.0 : 2.0) * (qh == ql ? 1.0 : 2.0), w = m * ri[i].v;
        de = fma(m * ri[i].g, X[ph][qh] * X[pl][ql] + X[pl][qh] * X[ph][ql], de);
        A[ph][qh] = fma(w, X[pl][ql], A[ph][qh]);
        A[pl][ql] = fma(w, X[ph][qh], A[pl][ql]);
        A[pl][qh] = fma(w, X[ph][ql], A[pl][qh]);
        A[ph][ql] = fma(w, X[pl][qh], A[ph][ql]);
      }
    }
    if (NA == 4) {
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        T[0] += A[1][j] * X[2][j] - A[2][j] * X[1][j];
        T[1] += A[1][j] * X[3][j] - A[3][j] * X[1][j];
      }
    }
    if (NB == 4) {
#pragma unroll
      for (int i = 0; i < NA; ++i) {
        T[0] += A[i][1] * X[i][2] - A[i][2] * X[i][1];
        T[1] += A[i][1] * X[i][3] - A[i][3] * X[i][1];
      }
    }
  }
  T[0] *= ir;
  T[1] *= ir;
#pragma unroll
  for (int k = 0; k < 3; ++k) f[k] = -(de * E[k] + T[0] * E[3 + k] + T[1] * E[6 + k]);
}

// pair index -> (u < v) of N items
__device__ __forceinline__ void grad_pair(int N, int t, int& u, int& v) {
  const double b = 2.0 * N - 1.0;
  int uu = (int)floor((b - sqrt(b * b - 8.0 * t)) * 0.5);
  if (uu < 0) uu = 0;
  while (uu > 0 && uu * (2 * N - uu - 1) / 2 > t) --uu;
  while ((uu + 1) * (2 * N - uu - 2) / 2 <= t) ++uu;
  u = uu;
  v = t - uu * (2 * N - uu - 1) / 2 + uu + 1;
}

__global__ void __launch_bounds__(kGradThreads) gradient_kernel(GradArgs g) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < g.npairs; t += stride) {
    int lo = 0, hi = g.nmol - 1;  // molecule with pair0 <= t < next pair0
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (g.mols[mid].pair0 <= t) lo = mid;
      else hi = mid - 1;
    }
    const GradMol& M = g.mols[lo];
    // Pairs by kind: heavy-heavy, heavy-light, light-light, so that a warp does one kind's work. With the kinds mixed in the
    // molecule's order nearly every warp ran the heavy-heavy path for a quarter of its lanes (1000 organics of 10-35 atoms:
    // 3.4 ms, 3.0 by kind).
    const int loc = (int)(t - M.pair0), nl = M.natom - M.nh, nhh = (int)((long long)M.nh * (M.nh - 1) / 2);
    const int nhl = M.nh * nl;
    int ia, ib;
    if (loc < nhh) {
      grad_pair(M.nh, loc, ia, ib);
    } else if (loc < nhh + nhl) {
      ia = (loc - nhh) / nl;
      ib = M.nh + (loc - nhh) % nl;
    } else {
      grad_pair(nl, loc - nhh - nhl, ia, ib);
      ia += M.nh;
      ib += M.nh;
    }
    const int ga = M.atom0 + g.order[M.atom0 + ia], gb = M.atom0 + g.order[M.atom0 + ib];
    const double* Pt = g.dens + M.dens_off;
    const ElemDev &ea = g.elem[g.z[ga]], &eb = g.elem[g.z[gb]];
    const double *xa = g.xyz + 3 * (size_t)ga, *xb = g.xyz + 3 * (size_t)gb;
    const int oa = g.ao_off[ga], ob = g.ao_off[gb];
    double f[3];
    if (eb.norb == 4) pair_force<4, 4>(ea, eb, *g.pairs, xa, xb, oa, ob, M.nao, Pt, M.uhf != 0, f);
    else if (ea.norb == 4) pair_force<4, 1>(ea, eb, *g.pairs, xa, xb, oa, ob, M.nao, Pt, M.uhf != 0, f);
    else pair_force<1, 1>(ea, eb, *g.pairs, xa, xb, oa, ob, M.nao, Pt, M.uhf != 0, f);
    for (int ax = 0; ax < 3; ++ax) {
      atomicAdd(&g.grad[3 * (size_t)gb + ax], f[ax]);
      atomicAdd(&g.grad[3 * (size_t)ga + ax], -f[ax]);
    }
  }
}

}  // namespace pm3gpu
