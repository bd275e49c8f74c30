// Persistent batched PM3 SCF: every CTA repeatedly takes the next job (one SCF solve of one
// molecule) from a global work queue and runs the whole calculation for it -- pair
// integrals, H_core, the SCF loop (Fock build, commutator, Pulay CDIIS / A-DIIS, eigensolve,
// density) and the properties of the converged state. Jobs are queued largest first, so the
// tail of the launch is a small molecule.
//
// The per-molecule algorithm is the reference's (pm3-rs src/hamiltonian.rs:191-344,
// src/fock.rs:93-332, src/scf.rs:1039-1693); the stability-search driver that decides
// which jobs to run lives on the host.
#pragma once
#include <cstdint>

#include "cta_blas.cuh"
#include "cta_eigen.cuh"
#include "pm3_integrals.cuh"

namespace pm3gpu {

constexpr int kMaxDepth = 8;  // deepest accelerator history (scf.rs:300)
// Phases of one job, timed with clock64 by thread 0 when profiling is on.
enum Phase : int {
  kPhCore = 0, kPhFock, kPhCommutator, kPhDiisSolve, kPhPack, kPhTridiag, kPhEigval, kPhEigvec, kPhBack,
  kPhDensity, kPhFinal, kPhGradient, kPhases
};

enum JobFlags : int {
  kJobUhf = 1,        // unrestricted iteration
  kJobKeepDens = 2,   // A-DIIS density history
  kJobGrad = 4,       // export the densities the gradient kernel needs (P, and Pa/Pb for UHF)
  kJobDensity = 8,    // export the total density
  kJobEps = 16,       // export all MO energies of the last iteration
  kJobCoreOnly = 32,  // stop after H_core: export H (build_core)
  kJobFockOnly = 64,  // H_core, then F(P) for a given density (build_fock_spin)
};

struct JobDesc {
  int atom0, natom, nao;
  int n_alpha, n_beta;
  int flags;
  int mol;     // molecule index (host bookkeeping)
  int rung0, nrung;  // stability-search jobs of this molecule in the rung table (first pass only)
  int stab;    // 0 no search, 1 search when the frontier gap < 6 eV, 2 always (first pass only)
  int backup;  // rung-table job that repeats this pass from the standard guess if it fails (-1: none)
  int guess;   // 1 SAD, 2 core Hamiltonian, 3 symmetry-broken SAD, 4 given density (learned guess)
  int accel;   // 0 none, 1 CDIIS, 2 A-DIIS -> CDIIS (already combined with use_diis)
  int depth;   // accelerator history length
  int max_scf;
  double e_tol, p_tol, adiis_switch, shift, damping;
  long long charge_off;   // into charges[] (natom values)
  long long dens_off;     // into densities[] (nao^2), when kJobDensity
  long long guess_off;    // into guess_dens[] (nao^2), when guess == 4 (learned initial density)
  long long eps_off;      // into eps[] (2 nao: alpha then beta), when kJobEps
};

struct JobOut {
  int status;        // 0 ok, 4 not converged, 5 linear algebra, 8 unsupported
  int converged, iterations, pad;
  double electronic, core, last_change;
  double homo, lumo;       // frontier over both spins (scf.rs:804-822)
  int has_homo, has_lumo;
  double homo_a, lumo_a;   // alpha-only frontier (a spin-pure UHF rung collapsed to RHF)
  int has_homo_a, has_lumo_a;
  double gap;              // frontier gap used by the stability trigger (scf.rs:106-124)
  double spin_max;         // max |P_alpha - P_beta| (unrestricted jobs)
  double dipole[3];        // Debye
};

// Byte offsets of the dynamic shared-memory carve-up (computed on the host).
struct SmemLayout {
  int amax;      // atoms per molecule this launch supports
  int nsm;       // size up to which the eigensolver's matrix is certain to stay on chip (make_layout)
  int uni;       // doubles in the union of the phases' scratch
  int off_int, off_dbl, off_eig, off_union;
  int bytes;
};

struct KernelArgs {
  const ElemDev* elem;
  const PairDev* pairs;
  const int* z;          // [total atoms]
  const double* xyz;     // [3 * total atoms], Bohr
  const JobDesc* jobs;   // first-pass jobs, largest first
  int njobs;
  JobOut* out;
  const JobDesc* rjobs;  // stability-search rung table (all candidates)
  int nrjobs;
  JobOut* rout;          // status stays -1 for rungs that were never enqueued
  int* rlist;            // [nrjobs] rung queue entries (rung table indices)
  int* rready;           // [nrjobs] 1 once rlist[i] is published
  double* charges;
  double* densities;
  const double* guess_dens;  // initial densities of guess-4 jobs
  double* grads;
  double* eps;
  double* work;          // per-CTA slots
  long long slot;        // doubles per slot
  int nmax;              // largest nao of the launch (slot dimension)
  long long wcap;        // doubles reserved for the pair table
  int* queue;            // [0] next first-pass job, [1] rung queue tail, [2] rung queue head, [3] error,
                         // [4] finished first passes, [5] CTAs waiting for late work, [6] jobs paired
  unsigned long long* prof;  // [kPhases] SM cycles per phase, summed over CTAs (null = off)
  SmemLayout sm;
  struct HelpRec* help;  // [grid] per CTA: its unrestricted job's offer of the beta spin (null = off)
  unsigned long long* tjob;  // [njobs + 1] global-timer ns when each first pass ended, [njobs] the start (null = off)
  int max_waiters;       // CTAs that may stay, once the first passes are all taken, for work still to come
};

// One CTA's offer of the beta spin of its unrestricted job to an idle CTA (a "helper"). `sg`
// packs a generation (bits 3..) and a state (bits 0-2): 0 idle, 1 open, 2 taken by a helper,
// 3 active (the two CTAs run the iterations from `go` on together), 4 stop. Each new offer takes a
// new generation, so a helper of an older offer never acts on a newer one.
struct HelpRec {
  int sg;
  int kind, idx;   // the job: 0 first-pass table, 1 rung table
  int go;          // iteration the helper may run next (the leader published its densities for it)
  int cur;         // current density buffer of iteration `go`
  int hdone;       // last iteration the helper has finished
  int pad[2];
  double part_b[2], sq_b[2];  // helper's energy part sum P_beta F_beta and squared density change, by iteration parity
};

// ---------------------------------------------------------------------------- helpers
__device__ __forceinline__ double oc_integral(const ElemDev& e, int a, int b, int c, int d) {
  // One-centre (ab|cd) from Gss..Hsp (fock.rs:244-282).
  if (a == b && c == d) {
    if (a == 0 && c == 0) return e.gss;
    if (a == 0 || c == 0) return e.gsp;
    return a == c ? e.gpp : e.gp2;
  }
  const int ba = min(a, b), bb = max(a, b), kc = min(c, d), kd = max(c, d);
  if (ba == 0 && bb != 0 && kc == 0 && kd != 0 && bb == kd) return e.hsp;
  if (ba != 0 && bb != 0 && ba != bb && ba == kc && bb == kd) return 0.5 * (e.gpp - e.gp2);
  return 0.0;
}

// Per-job context: shared-memory views and global buffers of this CTA's slot.
struct Ctx {
  const KernelArgs* A;
  JobDesc job;
  JobOut* out;
  int n, N;             // AOs, atoms
  // shared
  int* sz;              // [amax] Z of each atom
  int* soff;            // [amax] first AO
  int* order;           // [amax] atoms with p orbitals first, then the others, each in the molecule's order
  int *sprow, *sroff;   // scf_tight_kernel: [amax + 1] prefix of packed sizes, [amax] pair-table row offsets
  int nh;               // atoms with p orbitals
  double* sxyz;         // [3 amax]
  double* red;          // reduction scratch
  double* misc;         // broadcast scalars
  double* bg;           // [8*8] <E_i,E_j>
  double* mg;           // [8*8] <D_i,F_j>
  double* coef;         // [kMaxDepth+1]
  int* iv;              // small ints
  double *dpk, *jacc;   // scf_tight_kernel: [10 amax] packed densities, [10 amax] Coulomb accumulators (in the union)
  double* tile;         // the union: GEMM tiles, the Fock build's packed rows, the eigensolver's scratch
  EigenScratch es;
  unsigned long long* ph;  // [kPhases] shared accumulators
  long long tmark;
  // global (slot)
  double *H, *P[2], *Q[2], *F, *G, *Vt, *Vb, *Ag, *tf, *hist, *W, *Wg, *tri_a, *tri_b;  // W: the pair table, in Wg or in shared memory
  int cur;              // which P/Q buffer is current
};

__device__ __forceinline__ void mark(Ctx& c, int phase) {
  if (c.A->prof && threadIdx.x == 0) {
    const long long now = clock64();
    c.ph[phase] += (unsigned long long)(now - c.tmark);
    c.tmark = now;
  }
}

__device__ __forceinline__ bool heavy(const Ctx& c, int a) { return c.A->elem[c.sz[a]].norb == 4; }
// pair index t -> (u < v)
__device__ __forceinline__ void pair_uv(int N, int t, int& u, int& v) {
  const double b = 2.0 * N - 1.0;
  int uu = (int)floor((b - sqrt(b * b - 8.0 * t)) * 0.5);
  if (uu < 0) uu = 0;
  while (uu > 0 && uu * (2 * N - uu - 1) / 2 > t) --uu;
  while ((uu + 1) * (2 * N - uu - 2) / 2 <= t) ++uu;
  u = uu;
  v = t - uu * (2 * N - uu - 1) / 2 + uu + 1;
}

// The same for one molecule's short lists, in single precision with the integer correction.
__device__ __forceinline__ void pair_uv_short(int N, int t, int& u, int& v) {
  const float b = 2.0f * N - 1.0f;
  int uu = max(0, min(N - 2, (int)((b - sqrtf(fmaxf(b * b - 8.0f * t, 0.0f))) * 0.5f)));
  while (uu > 0 && uu * (2 * N - uu - 1) / 2 > t) --uu;
  while ((uu + 1) * (2 * N - uu - 2) / 2 <= t) ++uu;
  u = uu;
  v = t - uu * (2 * N - uu - 1) / 2 + uu + 1;
}

// A molecule's atom pairs by kind, so that the threads of a warp do the same work: both atoms with p orbitals
// (heavy, nhh pairs), one of them (nhl), none (nll). The pair table W holds the integrals of a kind
// with the pair index fastest (100, 10 and 1 rows of nhh, nhl and nll values), so that a warp reads
// consecutive addresses. Rows of packed densities and Coulomb sums: 10 per heavy atom, then 1 per light one.
struct PairKinds {
  int nh, nl, nhh, nhl, nll, rows;
  __device__ __forceinline__ PairKinds(int nh_, int N)
      : nh(nh_), nl(N - nh_), nhh(nh_ * (nh_ - 1) / 2), nhl(nh_ * (N - nh_)), nll((N - nh_) * (N - nh_ - 1) / 2),
        rows(10 * nh_ + (N - nh_)) {}
  __device__ __forceinline__ int row(int i) const { return i < nh ? 10 * i : 10 * nh + (i - nh); }
};

// Doubles of the union that the phases of an n-function molecule use beside a pair table kept there.
__host__ __device__ constexpr int union_keep(int n) {
  const int a = lower_scratch(n, true) > 2080 ? lower_scratch(n, true) : 2080, b = tri_scratch(n), c = back_scratch(n), d = 25 * n;
  const int m = a > b ? a : b, k = c > d ? c : d;
  return m > k ? m : k;
}

// ------------------------------------------------------------------ job setup + H_core
__device__ void setup_job(Ctx& c) {
  const KernelArgs& A = *c.A;
  const int tid = threadIdx.x;
  for (int a = tid; a < c.N; a += kThreads) {
    c.sz[a] = A.z[c.job.atom0 + a];
    for (int k = 0; k < 3; ++k) c.sxyz[3 * a + k] = A.xyz[3 * (size_t)(c.job.atom0 + a) + k];
  }
  __syncthreads();
  // first AO of every atom and the heavy-first order, by counting the heavy atoms before each
  for (int a = tid; a < c.N; a += kThreads) {
    int hv = 0;
    for (int k = 0; k < a; ++k) hv += heavy(c, k) ? 1 : 0;
    c.soff[a] = a + 3 * hv;
    c.iv[0] = 0;
    if (a == c.N - 1) c.iv[1] = hv + (heavy(c, a) ? 1 : 0);
  }
  __syncthreads();
  c.nh = c.iv[1];
  for (int a = tid; a < c.N; a += kThreads) {
    const int hv = (c.soff[a] - a) / 3;  // heavy atoms before a
    c.order[heavy(c, a) ? hv : c.nh + (a - hv)] = a;
  }
  // A small molecule keeps its pair table at the end of the union (n = 60 and 12 + 12 atoms: 63 KB); with
  // helpers another CTA may have to read it, from global memory.
  const PairKinds K(c.nh, c.N);
  const int wsize = 100 * K.nhh + 10 * K.nhl + K.nll;
  const bool near = A.help == nullptr && max(union_keep(c.n), tri_resident(c.n)) + wsize <= A.sm.uni;
  c.W = near ? c.tile + (A.sm.uni - wsize) : c.Wg;
  c.es.sh_doubles = near ? A.sm.uni - wsize : A.sm.uni;
  __syncthreads();
}

// One atom pair of H_core (hamiltonian.rs:191-344): both atoms' electron-core attraction blocks
// (stored to hacc_a, hacc_b; kAdd: added to them atomically), the pair table block W in (a, b) orientation (a
// the atom with more orbitals; consecutive integrals ws apart), and the resonance block H_ab = (beta_i + beta_j)/2 S_ij written to
// both triangles of H (row stride n). Returns the pair's core-core energy (repulsion.rs:57-120),
// evaluated with the atoms in the caller's (u, v) order.
template <bool kAdd = false>
__device__ __forceinline__ double core_pair(const ElemDev& ea, const ElemDev& eb, const ElemDev& eu, const ElemDev& ev,
                                            const PairDev& pp, const double* xa, const double* xb, int oa, int ob,
                                            size_t n, double* hacc_a, double* hacc_b, double* w, int ws,
                                            double* H) {
  const double d[3] = {xb[0] - xa[0], xb[1] - xa[1], xb[2] - xa[2]};
  const double r = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
  const double dv[3] = {d[0] / r * r, d[1] / r * r, d[2] / r * r};
  const double mdv[3] = {-dv[0], -dv[1], -dv[2]};
  if (hacc_a) {  // null: the caller adds the electron-core blocks per atom itself
    double blk[10];
    core_attraction(ea, eb, dv, blk);
    for (int k = 0; k < (ea.norb == 4 ? 10 : 1); ++k) {
      if (kAdd) atomicAdd(&hacc_a[k], blk[k]);
      else hacc_a[k] = blk[k];
    }
    core_attraction(eb, ea, mdv, blk);
    for (int k = 0; k < (eb.norb == 4 ? 10 : 1); ++k) {
      if (kAdd) atomicAdd(&hacc_b[k], blk[k]);
      else hacc_b[k] = blk[k];
    }
  }
  const double ir = 1.0 / r;
  double R[9];
  frame(-(dv[0] * ir), -(dv[1] * ir), -(dv[2] * ir), R);
  const double rv = sqrt(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]);
  if (ea.norb == 1) {
    const double s = ea.rho0 + eb.rho0;
    w[0] = rsq(rv * rv + s * s) * kEv;
  } else if (eb.norb == 1) {
    double ri[4];
    local4(ee_pole(ea), eb.rho0, rv, ri);
    for (int kk = 0; kk < 4; ++kk)
      for (int ll = 0; ll <= kk; ++ll) w[(size_t)pk(kk, ll) * ws] = w4(ri, R, kk, ll);
  } else {
    double ri[22];
    local22(ee_pole(ea), ee_pole(eb), rv, ri);
    for (int kk = 0; kk < 4; ++kk)
      for (int ll = 0; ll <= kk; ++ll)
        for (int mm = 0; mm < 4; ++mm)
          for (int nn = 0; nn <= mm; ++nn) w[(size_t)(pk(kk, ll) * 10 + pk(mm, nn)) * ws] = w22(ri, R, kk, ll, mm, nn);
  }
  double s[16];
  overlap_block(ea, eb, d, s);
  for (int i = 0; i < ea.norb; ++i) {
    const double bi = i == 0 ? ea.bs : ea.bp;
    for (int j = 0; j < eb.norb; ++j) {
      const double bj = j == 0 ? eb.bs : eb.bp;
      const double h = 0.5 * (bi + bj) * s[i * 4 + j];
      H[(size_t)(oa + i) * n + ob + j] = h;
      H[(size_t)(ob + j) * n + oa + i] = h;
    }
  }
  const double dd = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
  return core_core(eu, ev, pp, dd);
}

// Item t of the pair kinds in turn: atoms (positions in the heavy-first order), table entry and its stride.
__device__ __forceinline__ void pair_item(const PairKinds& K, int t, int& ia, int& ib, size_t& w0, int& ws) {
  if (t < K.nhh) {
    pair_uv_short(K.nh, t, ia, ib);
    w0 = t;
    ws = K.nhh;
  } else if (t < K.nhh + K.nhl) {
    const int q = t - K.nhh;
    ia = q / K.nl;
    ib = K.nh + q - ia * K.nl;
    w0 = (size_t)100 * K.nhh + q;
    ws = K.nhl;
  } else {
    const int q = t - K.nhh - K.nhl;
    pair_uv_short(K.nl, q, ia, ib);
    ia += K.nh;
    ib += K.nh;
    w0 = (size_t)100 * K.nhh + (size_t)10 * K.nhl + q;
    ws = K.nll;
  }
}

// Sums every packed row r over the partner atoms, in their order: S[y rows + r] holds partner y's part. With few rows
// the partners are split over 2 or 4 groups of threads; out[g rows + r] gets group g's sum, and the number of groups is returned.
__device__ __forceinline__ int gather_rows(const PairKinds& K, int N, const double* __restrict__ S, double* out) {
  const int groups = K.rows <= 64 ? 4 : (K.rows <= 128 ? 2 : 1), per = kThreads / groups;
  const int g = threadIdx.x / per, y0 = N * g / groups, y1 = N * (g + 1) / groups;
  for (int r = threadIdx.x % per; r < K.rows; r += per) {
    const int self = r < 10 * K.nh ? r / 10 : K.nh + (r - 10 * K.nh);
    double acc = 0.0;
    for (int y = y0; y < y1; y += 8) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = y + u < y1 && y + u != self ? S[(size_t)(y + u) * K.rows + r] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) acc += x[u];
    }
    out[g * K.rows + r] = acc;
  }
  return groups;
}

// H_core (hamiltonian.rs:191-344) and the pair table W; returns the core-core energy
// (repulsion.rs:13-27) to every thread. Each pair writes its two electron-core blocks to its own place
// in scratch and every element of an atom's block is summed over the partners in order: sums of the shared accumulators
// with atomics took most of the time (5.8M of 6M cycles at n = 148, 61 atoms).
__device__ __noinline__ double build_core(Ctx& c) {
  const KernelArgs& A = *c.A;
  const int n = c.n, N = c.N, tid = threadIdx.x;
  const PairKinds K(c.nh, N);
  double* S = c.hist;  // [N][rows]
  double ecc = 0.0;
  for (int t = tid; t < K.nhh + K.nhl + K.nll; t += kThreads) {
    int ia, ib, ws;
    size_t w0;
    pair_item(K, t, ia, ib, w0, ws);
    const int a = c.order[ia], b = c.order[ib], u = min(a, b), v = max(a, b);
    ecc += core_pair(A.elem[c.sz[a]], A.elem[c.sz[b]], A.elem[c.sz[u]], A.elem[c.sz[v]], *A.pairs, c.sxyz + 3 * a,
                     c.sxyz + 3 * b, c.soff[a], c.soff[b], (size_t)n, S + (size_t)ib * K.rows + K.row(ia),
                     S + (size_t)ia * K.rows + K.row(ib), c.W + w0, ws, c.H);
  }
  __syncthreads();
  double* sums = in_shared(c.tile);
  const int groups = gather_rows(K, N, S, sums);
  __syncthreads();
  // diagonal blocks: U + sum of electron-core attractions
  for (int k = tid; k < N * 16; k += kThreads) {
    const int i = k >> 4, mu = (k >> 2) & 3, nu = k & 3, a = c.order[i];
    const ElemDev& e = A.elem[c.sz[a]];
    if (mu >= e.norb || nu >= e.norb) continue;
    double h = mu == nu ? (mu == 0 ? e.uss : e.upp) : 0.0;
    for (int g = 0; g < groups; ++g) h += sums[g * K.rows + K.row(i) + pk(mu, nu)];
    c.H[(size_t)(c.soff[a] + mu) * n + c.soff[a] + nu] = h;
  }
  __syncthreads();
  return block_sum(ecc, c.red);
}

// ------------------------------------------------------------------------ Fock build
// Exchange block of one atom pair on the whole-GPU path (fock.rs:106-193): F_ab = H_ab - K_ab, written to both
// triangles. NA / NB are the orbital counts of atom a (the heavier one) and b, so every loop has a fixed trip
// count. W is the pair's (PA x PB) row-major integral block.
template <int NA, int NB, bool UHF>
__device__ __forceinline__ void fock_pair(int n, int oa, int ob, const double* __restrict__ H,
                                          const double* __restrict__ w, const double* Pt, const double* Pa,
                                          const double* Pb, double* F, double* G) {
  constexpr int PB = NB == 4 ? 10 : 1;
  // exchange: K[mu][la] = sum_{nu, si} X[nu][si] (mu nu | la si), one spin at a time
#pragma unroll
  for (int spin = 0; spin < (UHF ? 2 : 1); ++spin) {
    const double* X = UHF ? (spin == 0 ? Pa : Pb) : Pt;
    const double xs = UHF ? 1.0 : 0.5;
    double* out = spin == 0 ? F : G;
    double x[NA * NB];
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) x[i * NB + j] = xs * X[(size_t)(oa + i) * n + ob + j];
#pragma unroll
    for (int mu = 0; mu < NA; ++mu)
#pragma unroll
      for (int la = 0; la < NB; ++la) {
        double k = 0.0;
#pragma unroll
        for (int nu = 0; nu < NA; ++nu)
#pragma unroll
          for (int si = 0; si < NB; ++si) k = fma(x[nu * NB + si], w[pk(mu, nu) * PB + pk(la, si)], k);
        const double f = H[(size_t)(oa + mu) * n + ob + la] - k;
        out[(size_t)(oa + mu) * n + ob + la] = f;
        out[(size_t)(ob + la) * n + oa + mu] = f;
      }
  }
}

// One pair with at most one heavy atom a (NA = 4 or 1) and a light atom b of the per-CTA Fock build, for one spin density X (times
// xs): the exchange block F_ab = H_ab - K_ab to both triangles and, with kJ, the pair's Coulomb parts J_a[p] = W[p] d_b and
// J_b = sum_p d_a[p] W[p] to sa and sb. Returns the pair's part of sum P (H + F), both triangles.
template <int NA, bool kJ>
__device__ __forceinline__ double light_item(int n, int oa, int ob, const double* __restrict__ w, int ws, const double* da,
                                             double db, double* __restrict__ sa, double* __restrict__ sb,
                                             const double* __restrict__ H, const double* __restrict__ X, double xs,
                                             double* __restrict__ F) {
  constexpr int PA = NA == 4 ? 10 : 1;
  const int ab = oa * n + ob, ba = ob * n + oa;
  double wv[PA], x[NA], h[NA];
#pragma unroll
  for (int p = 0; p < PA; ++p) wv[p] = w[p * ws];
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    x[i] = xs * X[ab + i * n];
    h[i] = H[ab + i * n];
  }
  if (kJ) {
    double jb = 0.0;
#pragma unroll
    for (int p = 0; p < PA; ++p) {
      sa[p] = wv[p] * db;
      jb = fma(da[p], wv[p], jb);
    }
    *sb = jb;
  }
  double en = 0.0;
#pragma unroll
  for (int mu = 0; mu < NA; ++mu) {
    double k = 0.0;
#pragma unroll
    for (int nu = 0; nu < NA; ++nu) k = fma(x[nu], wv[pk(mu, nu)], k);
    const double f = h[mu] - k;
    F[ab + mu * n] = f;
    F[ba + mu] = f;
    en = fma(x[mu], h[mu] + f, en);
  }
  return 2.0 * en / xs;
}

// Row mu of a pair of heavy atoms, one of the four lanes that share the pair: the exchange elements F_mu,la and, with kJ, the
// Coulomb parts of the table rows (mu, nu <= mu), J_b summed over the four lanes. A lane reads 40 of the 100 integrals. (With the whole
// pair on one lane the few pairs of a small molecule were one warp's chain of 1500 instructions: 18k of the 35k cycles
// of a Fock build at 11 atoms.) Whole warps call, with `on` false past the last pair.
template <bool kJ>
__device__ __forceinline__ double heavy_item(bool on, int n, int oa, int ob, int mu, const double* __restrict__ w, int ws,
                                             const double* da, const double* db, double* __restrict__ sa,
                                             double* __restrict__ sb, const double* __restrict__ H,
                                             const double* __restrict__ X, double xs, double* __restrict__ F) {
  const int ab = oa * n + ob;
  double x[4][4], k[4] = {0.0, 0.0, 0.0, 0.0}, jb[12], d[10];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) x[i][j] = on ? X[ab + i * n + j] : 0.0;
  if (kJ) {
#pragma unroll
    for (int q = 0; q < 12; ++q) jb[q] = 0.0;
#pragma unroll
    for (int q = 0; q < 10; ++q) d[q] = db[q];
  }
#pragma unroll
  for (int nu = 0; nu < 4; ++nu) {
    const int p = mu >= nu ? mu * (mu + 1) / 2 + nu : nu * (nu + 1) / 2 + mu;
    const double* wr = w + p * 10 * ws;
    double wv[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) wv[q] = wr[q * ws];
#pragma unroll
    for (int la = 0; la < 4; ++la)
#pragma unroll
      for (int si = 0; si <= la; ++si) {
        const double e = wv[pk(la, si)];
        k[la] = fma(x[nu][si], e, k[la]);
        if (la != si) k[si] = fma(x[nu][la], e, k[si]);
      }
    if (kJ) {
      const bool mine = on && nu <= mu;
      const double dp = mine ? da[p] : 0.0;
      double a0 = 0.0, a1 = 0.0;
#pragma unroll
      for (int q = 0; q < 10; q += 2) {
        a0 = fma(d[q], wv[q], a0);
        a1 = fma(d[q + 1], wv[q + 1], a1);
        jb[q] = fma(dp, wv[q], jb[q]);
        jb[q + 1] = fma(dp, wv[q + 1], jb[q + 1]);
      }
      if (mine) sa[p] = a0 + a1;
    }
  }
  if (kJ) {  // twelve places over four lanes: three sums each
    const bool b1 = mu & 2, b0 = mu & 1;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const double send = b1 ? jb[q] : jb[q + 6], keep = b1 ? jb[q + 6] : jb[q];
      jb[q] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double send = b0 ? jb[q] : jb[q + 3], keep = b0 ? jb[q + 3] : jb[q];
      const double t = keep + __shfl_xor_sync(0xffffffffu, send, 1);
      const int at = (b1 ? 6 : 0) + (b0 ? 3 : 0) + q;
      if (on && at < 10) sb[at] = t;
    }
  }
  if (!on) return 0.0;
  double en = 0.0;
  const int row = ab + mu * n, colm = ob * n + oa + mu;
#pragma unroll
  for (int la = 0; la < 4; ++la) {
    const double h = H[row + la], f = fma(-xs, k[la], h);
    F[row + la] = f;
    F[colm + la * n] = f;
    const double xm = mu == 0 ? x[0][la] : (mu == 1 ? x[1][la] : (mu == 2 ? x[2][la] : x[3][la]));
    en = fma(xm, h + f, en);
  }
  return 2.0 * en;
}

// The off-diagonal blocks of one spin's Fock matrix over all pairs of the molecule; with kJ also every pair's Coulomb
// parts to S (gather_rows' layout). Returns this thread's part of sum P (H + F).
template <bool kJ>
__device__ __noinline__ double fock_pairs(const Ctx& c, const double* dpk_, double* S, const double* X, double xs, double* F) {
  const PairKinds K(c.nh, c.N);
  const int n = c.n, tid = threadIdx.x;
  const int* soff = in_shared(c.soff);
  const int* order = in_shared(c.order);
  const double* dpk = in_shared(dpk_);
  const double* __restrict__ W = c.W;
  const double* __restrict__ H = c.H;
  double en = 0.0;
  const int mu = tid & 3;
#pragma unroll 1
  for (int t0 = 0; t0 < 4 * K.nhh; t0 += kThreads) {
    const int t = (t0 + tid) >> 2;
    const bool on = t < K.nhh;
    int ia, ib;
    pair_uv_short(K.nh, on ? t : 0, ia, ib);
    en += heavy_item<kJ>(on, n, soff[order[ia]], soff[order[ib]], mu, W + (on ? t : 0), K.nhh, dpk + 10 * ia, dpk + 10 * ib,
                         S + ib * K.rows + 10 * ia, S + ia * K.rows + 10 * ib, H, X, xs, F);
  }
  // the other kinds from the last thread on: the warps that had one heavy pair less begin first
  const double* Wl = W + (size_t)100 * K.nhh;
#pragma unroll 1
  for (int t = kThreads - 1 - tid; t < K.nhl; t += kThreads) {
    const int ia = t / K.nl, ib = K.nh + t - ia * K.nl, rb = K.row(ib);
    en += light_item<4, kJ>(n, soff[order[ia]], soff[order[ib]], Wl + t, K.nhl, dpk + 10 * ia, dpk[rb], S + ib * K.rows + 10 * ia,
                            S + ia * K.rows + rb, H, X, xs, F);
  }
  Wl += (size_t)10 * K.nhl;
#pragma unroll 1
  for (int t = kThreads - 1 - tid; t < K.nll; t += kThreads) {
    int ia, ib;
    pair_uv_short(K.nl, t, ia, ib);
    ia += K.nh;
    ib += K.nh;
    const int ra = K.row(ia), rb = K.row(ib);
    en += light_item<1, kJ>(n, soff[order[ia]], soff[order[ib]], Wl + t, K.nll, dpk + ra, dpk[rb], S + ib * K.rows + ra,
                            S + ia * K.rows + rb, H, X, xs, F);
  }
  return en;
}

// F = H + J(Pt) - K(Ps) (fock.rs:285-332), and the sum over the built spins of Ps (H + F) to all threads. Pt = total
// density (null: Pa + Pb). RHF: Pa null, Ps = Pt / 2. UHF: two spin Focks F (from Pa) and G (from Pb).
// With Pa and Pb given and G null, the spin of Pa alone.
// Every Coulomb part goes to its own place in scratch and is summed per packed row in a fixed order, so
// repeated solves agree bit for bit (atomics on the atoms' accumulators, 32 lanes at one address, took
// most of the build: 680k cycles at n = 148, 61 atoms).
__device__ __noinline__ double build_fock(Ctx& c, const double* Pt, const double* Pa, const double* Pb, double* F, double* G) {
  const KernelArgs& A = *c.A;
  const int n = c.n, N = c.N, tid = threadIdx.x;
  const PairKinds K(c.nh, N);
  double* dpk = in_shared(c.tile);  // [rows] packed densities (fock.rs:93-100)
  double* sums = dpk + K.rows;      // [groups][rows] Coulomb sums
  const int* soff = in_shared(c.soff);
  const int* order = in_shared(c.order);
  for (int r = tid; r < K.rows; r += kThreads) {
    const int i = r < 10 * K.nh ? r / 10 : K.nh + (r - 10 * K.nh);
    int hi, lo;
    unpk(r - K.row(i), hi, lo);
    const int o = soff[order[i]];
    const size_t ix = (size_t)(o + hi) * n + o + lo;
    const double v = Pt ? Pt[ix] : Pa[ix] + Pb[ix];
    dpk[r] = hi != lo ? 2.0 * v : v;
  }
  __syncthreads();
  double* S = c.tf;  // [N][rows]
  double en = fock_pairs<true>(c, dpk, S, Pa ? Pa : Pt, Pa ? 1.0 : 0.5, F);
  if (G) en += fock_pairs<false>(c, dpk, S, Pb, 1.0, G);
  __syncthreads();
  const int groups = gather_rows(K, N, S, sums);
  __syncthreads();
  // atom-diagonal blocks: H + one-centre J - K (fock.rs:244-282) + two-centre J
  for (int k = tid; k < 16 * K.nh + K.nl; k += kThreads) {
    const bool hv = k < 16 * K.nh;
    const int i = hv ? k >> 4 : K.nh + (k - 16 * K.nh), mu = hv ? (k >> 2) & 3 : 0, nu = hv ? k & 3 : 0;
    const int a = order[i], o = soff[a];
    const ElemDev& e = A.elem[c.sz[a]];
    const double hpp = 0.5 * (e.gpp - e.gp2);
    auto tot = [&](int x, int y) {
      const size_t ix = (size_t)(o + x) * n + o + y;
      return Pt ? Pt[ix] : Pa[ix] + Pb[ix];
    };
    double j = 0.0;
    for (int g = 0; g < groups; ++g) j += sums[g * K.rows + K.row(i) + pk(mu, nu)];
    // integrals (mu mu | x x) and (mu x | mu x) of the atom
    auto gm = [&](int x, int y) { return x == y ? (x == 0 ? e.gss : e.gpp) : (x == 0 || y == 0 ? e.gsp : e.gp2); };
    auto hm = [&](int x, int y) { return x == y ? (x == 0 ? e.gss : e.gpp) : (x == 0 || y == 0 ? e.hsp : hpp); };
    if (mu == nu) {
      for (int x = 0; x < (hv ? 4 : 1); ++x) j = fma(tot(x, x), gm(mu, x), j);
    } else {
      j = fma(hm(mu, nu), tot(mu, nu) + tot(nu, mu), j);
    }
    const size_t ix = (size_t)(o + mu) * n + o + nu;
    const double h = c.H[ix];
#pragma unroll
    for (int spin = 0; spin < 2; ++spin) {
      if (spin == 1 && !G) break;
      const double* P = spin == 1 ? Pb : (Pa ? Pa : Pt);
      const double xs = Pa ? 1.0 : 0.5;
      auto den = [&](int x, int y) { return P[(size_t)(o + x) * n + o + y]; };
      double ex = 0.0;
      if (mu == nu) {
        for (int x = 0; x < (hv ? 4 : 1); ++x) ex = fma(den(x, x), hm(mu, x), ex);
      } else {
        ex = fma(gm(mu, nu), den(mu, nu), hm(mu, nu) * den(nu, mu));
      }
      const double f = h + j - xs * ex;
      (spin == 1 ? G : F)[ix] = f;
      en = fma(P[ix], h + f, en);
    }
  }
  return block_sum(en, c.red);  // its barriers also publish F
}

// The lower triangle of E = F P - P F (scf.rs:1039-1054), which is antisymmetric: nothing reads the other half. The
// transposed subtraction of a full product F P cost as much as the product (n = 148: 550k cycles before, 180k now, FP64
// issue).
__device__ __noinline__ void commutator(Ctx& c, const double* Fm, const double* Pm, double* E) {
  const int n = c.n;
  lower_product<true>(n, n, Fm, Pm, in_shared(c.tile),
                      [&](int i, int j, double v) { E[(size_t)i * n + j] = i == j ? 0.0 : v; });
}

// ------------------------------------------------------------ small dense solves
// Pulay coefficients from the Gram matrix (scf.rs:1544-1630), on one thread; false = singular / unusable.
__host__ __device__ inline bool cdiis_coeffs(int m, const double* gram, double* x) {
  if (m < 2) return false;
  double scale = 0.0;
  for (int i = 0; i < m * m; ++i) scale = fmax(scale, fabs(gram[(i / m) * kMaxDepth + i % m]));
  if (!(scale > 0.0) || !isfinite(scale)) return false;
  const int dim = m + 1;
  double B[(kMaxDepth + 1) * (kMaxDepth + 1)], rhs[kMaxDepth + 1];
  for (int i = 0; i < dim; ++i) {
    rhs[i] = 0.0;
    for (int j = 0; j < dim; ++j) B[i * dim + j] = 0.0;
  }
  for (int i = 0; i < m; ++i) {
    for (int j = 0; j < m; ++j) B[i * dim + j] = gram[i * kMaxDepth + j] / scale;
    B[i * dim + m] = -1.0;
    B[m * dim + i] = -1.0;
  }
  rhs[m] = -1.0;
  for (int col = 0; col < dim; ++col) {
    int piv = col;
    double best = fabs(B[col * dim + col]);
    for (int r = col + 1; r < dim; ++r)
      if (fabs(B[r * dim + col]) > best) {
        best = fabs(B[r * dim + col]);
        piv = r;
      }
    if (best < 1.0e-12) return false;
    if (piv != col) {
      for (int j = 0; j < dim; ++j) {
        const double t = B[col * dim + j];
        B[col * dim + j] = B[piv * dim + j];
        B[piv * dim + j] = t;
      }
      const double t = rhs[col];
      rhs[col] = rhs[piv];
      rhs[piv] = t;
    }
    for (int r = col + 1; r < dim; ++r) {
      const double f = B[r * dim + col] / B[col * dim + col];
      if (f == 0.0) continue;
      for (int j = col; j < dim; ++j) B[r * dim + j] -= f * B[col * dim + j];
      rhs[r] -= f * rhs[col];
    }
  }
  for (int col = dim - 1; col >= 0; --col) {
    double sum = rhs[col];
    for (int j = col + 1; j < dim; ++j) sum -= B[col * dim + j] * x[j];
    x[col] = sum / B[col * dim + col];
  }
  return true;
}

// The same on one warp: lane r holds row r of the scaled bordered matrix (and its right-hand side), the pivot rows
// come round by shuffles. Coefficients to x; false = singular / unusable. `gram` and x in shared memory.
__device__ __forceinline__ bool cdiis_coeffs_warp(int m, const double* gram, double* x) {
  constexpr int D = kMaxDepth + 1;
  constexpr unsigned full = 0xffffffffu;
  if (m < 2) return false;
  const int lane = threadIdx.x & 31, dim = m + 1;
  double scale = 0.0;
  for (int i = lane; i < m * m; i += 32) scale = fmax(scale, fabs(gram[(i / m) * kMaxDepth + i % m]));
  scale = warp_max(scale);
  if (!(scale > 0.0) || !isfinite(scale)) return false;
  double B[D], rhs = lane == m ? -1.0 : 0.0;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    double v = 0.0;
    if (lane < m && j < m) v = gram[lane * kMaxDepth + j] / scale;
    else if ((lane < m && j == m) || (lane == m && j < m)) v = -1.0;
    B[j] = v;
  }
  bool done = lane >= dim;  // rows that have been pivots (or are not there)
  int mine = -1;            // the column this row was the pivot of
#pragma unroll
  for (int col = 0; col < D; ++col) {
    if (col >= dim) break;
    // largest element of the column among the rows left
    double best = done ? -1.0 : fabs(B[col]);
    int piv = lane;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(full, best, o);
      const int op = __shfl_xor_sync(full, piv, o);
      if (ob > best || (ob == best && op < piv)) {
        best = ob;
        piv = op;
      }
    }
    best = __shfl_sync(full, best, 0);  // the first 16 lanes hold all rows
    piv = __shfl_sync(full, piv, 0);
    if (best < 1.0e-12) return false;
    const double pv = __shfl_sync(full, B[col], piv);
    const double f = done || lane == piv ? 0.0 : B[col] / pv;
    if (lane == piv) {
      done = true;
      mine = col;
    }
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (j >= col) B[j] -= f * __shfl_sync(full, B[j], piv);
    rhs -= f * __shfl_sync(full, rhs, piv);
  }
#pragma unroll
  for (int col = D - 1; col >= 0; --col) {
    if (col >= dim) continue;
    const int src = __ffs(__ballot_sync(full, mine == col)) - 1;
    const double xc = __shfl_sync(full, rhs / B[col], src);
    if (lane == 0) x[col] = xc;
    rhs -= B[col] * xc;
  }
  __syncwarp();
  return true;
}

// A-DIIS weights on the simplex by projected gradient (scf.rs:1152-1172, 1637-1693), one warp:
// lane k owns row k of the gradient's matrix; all lanes hold the whole trial point and weights. The Euclidean projection onto
// the simplex subtracts the theta for which the positive parts sum to 1; the set of positive entries rarely
// changes between steps, so theta is first formed from the previous set and accepted when the set reproduces itself
// (which makes it the projection), else the set is rebuilt from all entries, dropping those below theta until none
// is. A step is one chain of about 300 cycles, up to 400 steps (1300 when every lane sorted the trial point and
// scanned it as the reference does).
__device__ __forceinline__ void adiis_coeffs_warp(int m, const double* mg, double* out) {
  constexpr int K = kMaxDepth;
  constexpr unsigned full = 0xffffffffu;
  const int k = threadIdx.x & 31, last = m - 1, row = k < m ? k : 0;
  const double mnn = mg[last * K + last];
  // S = mg - (last row and column), T = S + S^T: the gradient is 2 d + T c
  auto S = [&](int i, int j) { return mg[i * K + j] - mg[i * K + last] - mg[last * K + j] + mnn; };
  const double d2 = 2.0 * (mg[row * K + last] - mnn);
  double T[K], c[K], own = row == last && k < m ? 1.0 : 0.0, rs = 0.0;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    T[j] = j < m ? S(row, j) + S(j, row) : 0.0;
    rs += fabs(T[j]);
    c[j] = j == last ? 1.0 : 0.0;
  }
  const double lr = 1.0 / fmax(1.0e-12, warp_max(rs));
  unsigned set = (1u << m) - 1u;
  for (int it = 0; it < 400; ++it) {
    const double g = d2 + (((T[0] * c[0] + T[1] * c[1]) + (T[2] * c[2] + T[3] * c[3])) +
                           ((T[4] * c[4] + T[5] * c[5]) + (T[6] * c[6] + T[7] * c[7])));
    const double mine = own - lr * g;
    double t[K];
#pragma unroll
    for (int j = 0; j < K; ++j) t[j] = __shfl_sync(full, mine, j);
    double theta = 0.0;
    unsigned cur = set;
    for (int tries = 0; tries < 2 * K + 2; ++tries) {
      double v[K];
#pragma unroll
      for (int j = 0; j < K; ++j) v[j] = (cur >> j) & 1u ? t[j] : 0.0;
      const double sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
      // 1 / count for 1 .. 8
      const int q = __popc(cur);
      const double inv = q <= 2 ? (q == 1 ? 1.0 : 0.5) : q <= 4 ? (q == 3 ? 1.0 / 3.0 : 0.25)
                         : q <= 6 ? (q == 5 ? 0.2 : 1.0 / 6.0) : (q == 7 ? 1.0 / 7.0 : 0.125);
      theta = (sum - 1.0) * inv;
      unsigned nx = 0;
#pragma unroll
      for (int j = 0; j < K; ++j) nx |= j < m && t[j] > theta ? 1u << j : 0u;
      if (nx == cur) break;
      // first the whole set, then only shrinking ones
      cur = tries == 0 ? (1u << m) - 1u : (cur & nx ? cur & nx : cur);
    }
    set = cur;
    double dl[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const double pj = j < m ? fmax(t[j] - theta, 0.0) : 0.0;
      dl[j] = fabs(pj - c[j]);
      c[j] = pj;
    }
    own = fmax(mine - theta, 0.0);
    if (((dl[0] + dl[1]) + (dl[2] + dl[3])) + ((dl[4] + dl[5]) + (dl[6] + dl[7])) < 1.0e-12) break;
  }
  if (k < m) out[k] = own;
  __syncwarp();
}

// ------------------------------------------------------------------- eigensolve + density
// The eigen input X [+ shift (I - Pproj)].
__device__ __forceinline__ SymInput sym_input(const double* X, const double* Pproj, double shift) {
  return SymInput{X, nullptr, nullptr, 0, 0, 1, 0, Pproj, shift};
}

// Diagonalise the matrix: kval lowest eigenvalues into lam_out, kvec eigenvectors
// into Y (rows). The tridiagonal (d, e) is saved to `tri_save` (2n) for the final MO energies.
// With `warm`, lam_out holds the same eigenvalues from the previous SCF iteration and `dlam`
// their last change; both seed the eigenvalue search and are updated. Without it dlam is reset.
__device__ void eigensolve(Ctx& c, const SymInput& in, int kval, int kvec, double* Y, double* lam_out, double* tri_save,
                           bool warm = false, double* dlam = nullptr) {
  const int n = c.n;
  mark(c, kPhPack);
  tridiagonalize(n, in, c.Ag, c.tf, c.es);
  if (tri_save)
    for (int i = threadIdx.x; i < n; i += kThreads) {
      tri_save[i] = c.es.d[i];
      tri_save[n + i] = c.es.e[i];
    }
  __syncthreads();  // the splitting of T writes e
  mark(c, kPhTridiag);
  const bool seeded = warm && dlam != nullptr;
  tridiag_eigenvalues(n, kval, c.es, seeded ? lam_out : nullptr, seeded ? dlam : nullptr);
  for (int j = threadIdx.x; j < kval; j += kThreads) {
    if (dlam) dlam[j] = seeded ? c.es.lam[j] - lam_out[j] : 1.0e30;
    lam_out[j] = c.es.lam[j];
  }
  mark(c, kPhEigval);
  if (kvec > 0) {
    const double* Yt = tridiag_vectors(n, kvec, c.tf, c.es);
    mark(c, kPhEigvec);
    back_transform(n, kvec, c.Ag, Yt, Y, c.es);
  }
  __syncthreads();
  mark(c, kPhBack);
}

// Pnew = w Y^T Y (first k rows of Y); returns sum (Pnew - Pold)^2 to all threads. With
// damping lam > 0 the stored value is (1-lam) Pnew + lam Pold (scf.rs:1440-1448); the RMS
// uses the undamped Pnew, as the reference does.
__device__ __noinline__ double density(Ctx& c, const double* Y, int k, double w, const double* Pold, double* Pnew, double damp) {
  const int n = c.n;
  double sq = 0.0;
  if (k == 0) {
    for (int q = threadIdx.x; q < n * n; q += kThreads) {
      const double o = Pold[q];
      sq += o * o;
      Pnew[q] = damp > 0.0 ? damp * o : 0.0;
    }
    __syncthreads();
    return block_sum(sq, c.red);
  }
  lower_product<false>(n, k, Y, nullptr, in_shared(c.tile), [&](int i, int j, double y) {
    const double v = w * y;
    const size_t ij = (size_t)i * n + j, ji = (size_t)j * n + i;
    const double o = Pold[ij];
    const double dlt = v - o;
    sq += (i == j ? 1.0 : 2.0) * dlt * dlt;
    const double st = damp > 0.0 ? (1.0 - damp) * v + damp * o : v;
    Pnew[ij] = st;
    Pnew[ji] = st;
  });
  return block_sum(sq, c.red);
}

// --------------------------------------------------------------------------- guesses
__device__ void sad_guess(Ctx& c, double* P, double scale, bool tilt) {
  const KernelArgs& A = *c.A;
  const int n = c.n;
  for (size_t k = threadIdx.x; k < (size_t)n * n; k += kThreads) P[k] = 0.0;
  __syncthreads();
  for (int a = threadIdx.x; a < c.N; a += kThreads) {
    const ElemDev& e = A.elem[c.sz[a]];
    const int o = c.soff[a];
    P[(size_t)o * n + o] = e.occ_s * scale;
    if (e.norb == 4)
      for (int k = 1; k < 4; ++k) P[(size_t)(o + k) * n + o + k] = (e.occ_p / 3.0) * scale;
  }
  __syncthreads();
  if (tilt && threadIdx.x == 0) {  // scf.rs:894-916: move 0.2 e from pz to px on the most p-rich atom
    int target = -1;
    double best = 0.0;
    for (int a = 0; a < c.N; ++a) {
      const ElemDev& e = A.elem[c.sz[a]];
      if (e.norb == 4 && e.occ_p > best) {
        best = e.occ_p;
        target = a;
      }
    }
    if (target >= 0) {
      const int o = c.soff[target];
      // the unscaled SAD entries are tilted, then the spin split scales them (scf.rs:951-977)
      const double pz = A.elem[c.sz[target]].occ_p / 3.0;
      const double t = fmin(0.2, pz);
      P[(size_t)(o + 3) * n + o + 3] = (pz - t) * scale;
      P[(size_t)(o + 1) * n + o + 1] = (pz + t) * scale;
    }
  }
  __syncthreads();
}

// ------------------------------------------------------------------------- properties
__device__ void properties(Ctx& c, const double* Pt, JobOut& o) {
  const KernelArgs& A = *c.A;
  const int n = c.n;
  double* q = A.charges + c.job.charge_off;
  for (int a = threadIdx.x; a < c.N; a += kThreads) {
    const ElemDev& e = A.elem[c.sz[a]];
    double pop = 0.0;
    for (int k = 0; k < e.norb; ++k) pop += Pt[(size_t)(c.soff[a] + k) * n + c.soff[a] + k];
    q[a] = e.core - pop;
  }
  // dipole about the centre of mass (dipole.rs:64-144)
  double v[4] = {0, 0, 0, 0};
  for (int a = threadIdx.x; a < c.N; a += kThreads) {
    const double m = A.elem[c.sz[a]].mass;
    v[0] += m;
    for (int k = 0; k < 3; ++k) v[1 + k] += m * c.sxyz[3 * a + k];
  }
  block_sums<4>(v, c.red, c.misc);
  const double mt = c.misc[0];
  double com[3];
  for (int k = 0; k < 3; ++k) com[k] = mt > 0.0 ? c.misc[1 + k] / mt : 0.0;
  double mu[3] = {0, 0, 0};
  for (int a = threadIdx.x; a < c.N; a += kThreads) {
    const ElemDev& e = A.elem[c.sz[a]];
    const int o = c.soff[a];
    double pop = 0.0;
    for (int k = 0; k < e.norb; ++k) pop += Pt[(size_t)(o + k) * n + o + k];
    for (int ax = 0; ax < 3; ++ax) {
      const double disp = c.sxyz[3 * a + ax] - com[ax];
      double el = pop * disp;
      if (e.norb == 4) el += 2.0 * Pt[(size_t)o * n + o + ax + 1] * e.dd;
      mu[ax] += disp * e.core - el;
    }
  }
  block_sums<3>(mu, c.red, c.misc);
  for (int ax = 0; ax < 3; ++ax) o.dipole[ax] = c.misc[ax] * kAuDipoleToDebye;
}

}  // namespace pm3gpu
