// Device kernels of libwedg: one RHS stage of the EDG scheme for the
// Westervelt equation on sm_103a, in FP64 and 64-bit fixed point.
//
// Design (GB300): the path is bound by arithmetic, not by HBM, and the FP64
// pipe is slow (about 1.2 TFLOP/s on GB300, 1/58 of FP32; one operation holds
// a scheduler's pipe for 64 cycles) while the integer pipes stand idle beside
// it. So the contractions over modes and points, which are most of the work,
// run in 64-bit fixed point with one exponent per element (wedg_fixed.cuh:
// three integer multiply-adds of 2 cycles for an FP64 one), and
// the fluxes, sources, inner products and updates in FP64. A team of threads
// shares an element: thread r has column or row r of its modal blocks or point
// r of its sides, and blocks change hands through shared memory. That spreads
// small meshes over the chip and keeps the registers low enough for 20 to 48
// warps an SM.
//
// One RHS evaluation is three kernels:
//   k_prep   traces of the stage state on the four sides of every element
//            (src/rhs.jl:384-410), the weight check of the boundary points
//            (src/rhs.jl:105-110, 729-757), G = 2βv at the high-order points
//            and the Chebyshev interval data (src/rhs.jl:889-907), so that every
//            error of the stage is known before the next kernel starts;
//            Its first blocks, or k_bnd, take the flux slots of the physical sides
//            (src/rhs.jl:65-103), projected on the face modes;
//   k_stage  face fluxes of the element's own interior sides (src/rhs.jl:611-700),
//            lifts (:412-473), volume terms (:309-333), source
//            (:335-350) and u-equation (:352-382) with the u part of the RK4
//            stage update (src/solver.jl:299-321); it leaves the right-hand
//            side of the mass system in HBM;
//   k_cheb   the Chebyshev mass solve (:920-939) and the v part of the RK4
//            update. Elements are visited in decreasing order of their Chebyshev
//            step counts (k_prep lists them by count), so the longest solves start
//            first;
//   k_cg     the same with conjugate gradients (:821-853).
// Interior faces are evaluated by both neighbours, each writing only its own
// slots, so no element writes another element's data.
//
// Device layouts (element index e = j + N k fastest everywhere):
//   state       x[e + E (a + n b)]                 (the reference's own layout)
//   traces      tr[((fam*4 + side)*NQ + i)*E + e]  fam du, v, dv; side B, T, L, R
//   Cw, Aw      [(r + NQ s) E + e]
//   Ainv        [row E + e]                        packed upper triangle by columns
//   h-faces     [jf + (N+1)(k + N i)]              face row jf, column k, point i
//   v-faces     [j + N (kf + (N+1) i)]
//   bnd data    [m + N i]
//   Pi, srcP    [(a + NV b) E + e]
//   2β, G       [(r + QH s) E + e]                 G as integers, its exponents in rows QH² and QH² + 1
//   bslots      [(q*4 + side) N + m]               q over the face modes of A, D, F
//   mass rhs    [(a + NV b) E + e]
#pragma once
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include "wedg_fixed.cuh"

namespace wedg {

constexpr unsigned long long ERR_NONE = ~0ull;
constexpr int ERR_CLASS_SHIFT = 56;   // class 0: boundary weight, 1: mass matrix not PD, 3: stopped (non-finite)
constexpr int NBIN = 48;              // Chebyshev-count bins of the mass kernel (the last holds n ≥ NBIN)
constexpr int CHEB_THREADS = 128;    // threads per block of the mass-solve kernels

__host__ __device__ constexpr int qhigh(int nu, int nv) {
  // q_high = max(ceil(3 q_v / 2) + 1, q_u + 1), src/solver.jl:483
  return ((3 * (nv - 1) + 1) / 2 + 1) > nu ? ((3 * (nv - 1) + 1) / 2 + 1) : nu;
}

// k_stage: a team of NU threads per element in blocks of 128
constexpr int STAGE_THREADS = 128;
__host__ __device__ constexpr int stage_tile(int nu) { return (32 / nu) * (STAGE_THREADS / 32); }   // elements per block

template <int NU, int NV>
struct Basis {
  static constexpr int NQ = NU;
  static constexpr int QH = qhigh(NU, NV);
  double w[NQ];
  double P[NQ][NU], S[NQ][NU];   // P[i][d] = P_u[i, d], S likewise; the v-basis is d < NV
  double Pw[NQ][NU];             // w[i] P[i][d]
  double El[NU], E1l[NU];        // the modes and their derivatives at the low end; at the high end (-1)^a El[a], -(-1)^a E1l[a]
  double E1F[NU];                // -E1l, the lift factor of the u-slots (the v-slots' factors
                                 // (2/h) El and (4/h²) E1l take the mesh size from Fields)
  double Ph[QH][NV];             // P_h_v[r, d]
  double PhW[QH][NV];            // w_h[r] P_h_v[r, d], with W2d_h = w_h w_h^T
  double wh[QH];                 // w_h
  double K1[NU][NU];             // 1D stiffness S^T diag(w) S
  // fixed-point forms (wedg_fixed.cuh): Ph, PhW; for the constant-coefficient kernels the end values,
  // K1[a][c] 2^-kK1[c], K1's eigenvectors Q (Q[row][col]; Q[.][0] = e_0), L = 1 / (λ_i + λ_j) (0 at
  // (0, 0)) and the pairs QE[i] L[i][j], QE[j] L[i][j] (QE = Q^T E1F: the u-slots' lift factor in the
  // eigenbasis)
  FxC fPh[QH][NV], fPhW[QH][NV], fEl[NU], fE1[NU], fK1[NU][NU], fQ[NU][NU], fL[NU][NU], fM[NU][NU][2];
  int gPh, gPhW, gEl, gE1, gK1, gQ, gL, gM;   // their exponents
  int kK1[NU];
  int nrow;                      // bits that the grid rows of team_K_fx have room for in every case
  int cPh[NV];                   // 2^8 max|Ph[.][a]|, rounded up
};

struct Fields {
  int N, E;
  const double *Cw, *Aw, *Ainv, *ic2e, *c2e, *ae;
  const double *hc2, *haf, *hcf, *hbf, *hc2m, *hafm, *hJC;
  const double *vc2, *vaf, *vcf, *vbf, *vc2m, *vafm, *vJC;
  // with modal traces and one-sided faces: the jump terms' projections Σ_i w_i P[i][b] JC_i on the
  // face modes b, in the layouts of hJC, vJC with mode b in the slot of point b (null: no jump term)
  const double *hJCm, *vJCm;
  const double *bsp[4], *bspn[4];
  const double *PiSP, *PiBSP2, *PiCdiv, *PiDdiv, *srcP;
  const double *beta2;        // 2β at the high-order points, [(r + QH s) E + e]
  // G = 2βv at the high-order points, as integers of one exponent per element, which row QH² holds with
  // a normalising shift (GPack).
  // Row QH² + 1: the largest high words of U and V beside the constant mode (k_stage's exponents)
  double *tr, *G, *th, *de;
  // the flux slots of the physical sides projected on the face modes: [(q 4 + s) N + m], q over the
  // modes of A, D and F, m along side s
  double *bslots;
  double *mrhs;               // right-hand side of the mass system, [(a + NV b) E + e]
  int *nst;
  int *nmax;                  // largest Chebyshev count: [parity] of a stage (the common count of
                              // src/rhs.jl:911-918), [2] of the whole call (statistics)
  int *bins, *bin_count;      // elements by Chebyshev count: bins[b E + i], two count buffers of NBIN
  unsigned long long *nsum;   // Σ of the per-element Chebyshev step counts
  unsigned long long *err;    // [0] the error recorded, [1] the same once later kernels stop for it
  unsigned int *cg_nfail, *nonfinite;
  double theta, tau, lu, lv, omega, two_h, four_hh, mass_tol, Lcheb;
  int one_sided, mms_on, src_on, cg, cheb_common, sorted;
  // modal traces: tr holds each side's modal end sums (index b < n in place of point i), and the
  // interior slots are projected in that form (every interior face's coefficients are one value
  // along the face; the adjoint kernels read point traces)
  int modal;
  int kind[4];
  double gam[4], eta[4], sig[4], kb[4], kap[4];
};

enum StageMode {
  OUT_RHS = 0, OUT_RK4_STAGE = 1, OUT_RK4_LAST = 2, OUT_RK4_LAST_ACC = 3,
  // adjoint parts of k_stage (both forms are symmetric, so the forward code is its own transpose):
  OUT_ADJ_USOLVE = 4,   // ut = A_e⁻¹ xu (the u-solve alone)
  OUT_ADJ_VOLUME = 5    // vt = R_v, ut = b of the volume terms alone, for the state (xu, xv)
};

struct StageIO {
  const double *xu, *xv;     // stage state
  double ct, st, srct;       // time factors of the stage (src/rhs.jl:509-511)
  double cSP, cB, cC, cD;    // source weights: -ω²ct, -2ω³ st ct, 1 - ct, ω st
  // or, for launches replayed from a CUDA graph, the same seven factors (and one pad) from a
  // host-computed table of tf_n steps: tf[((step mod tf_n)·4 + stage)·8 + f], step = *step (the
  // workspace's device step counter); the host refills the table every tf_n steps
  const double *tf;
  const long long *step;
  long long tf_n;
  int stage;
  int mode, first;
  int parity;                // which bin-count buffer this stage fills (the other is cleared)
  double *ut, *vt;           // OUT_RHS
  const double *u0, *v0;     // RK4 base state
  double *su, *sv;           // next stage state
  double *accu, *accv;       // k1 + 2k2 + 2k3 (+ k4)
  double *uo, *vo;           // in-place target of the last stage
  double c;                  // next-stage factor, or dt/6 on the last stage
};

// The time factors of a stage: from the launch parameters, or from the table of a graph replay
struct TimeF {
  double ct, st, srct, cSP, cB, cC, cD;
};
__device__ __forceinline__ TimeF time_factors(const StageIO &S) {
  if (!S.tf) return TimeF{S.ct, S.st, S.srct, S.cSP, S.cB, S.cC, S.cD};
  long long it = *(volatile const long long *)S.step;
  it = it < 0 ? 0 : it % S.tf_n;
  const double *f = S.tf + (it * 4 + S.stage) * 8;
  return TimeF{f[0], f[1], f[2], f[3], f[4], f[5], f[6]};
}

__device__ __forceinline__ unsigned long long err_word(const Fields &F) {
  return *(volatile unsigned long long *)F.err;
}
// Errors are recorded by k_prep and k_cg (F.err[0], the smallest by atomicMin), and which one is reported must
// not depend on the order of their blocks. So these kernels and k_cheb stop on errors of earlier kernels alone:
// those which the last k_stage or the end of a step found (F.err[1], stage_failed). Between k_cg and the next
// k_prep there may be neither, but with k_cg k_prep records boundary weights only, so any other error is
// an earlier one. One answer for all threads of a warp (several streams may share the words, and a team leaves as a
// whole), before any of them returns: a vote of each team by itself takes 150 to 600 cycles of its warp, one of
// the warp some 20.
__device__ __forceinline__ bool warp_stopped(const Fields &F) {
  return __any_sync(~0u, *(volatile unsigned long long *)(F.err + 1) != ERR_NONE);
}
__device__ __forceinline__ bool prep_stopped(const Fields &F) {
  bool stop = *(volatile unsigned long long *)(F.err + 1) != ERR_NONE;
  if (F.cg) {
    const unsigned long long w = err_word(F);
    stop = stop || (w != ERR_NONE && (w >> ERR_CLASS_SHIFT) > 0);
  }
  return __any_sync(~0u, stop);
}
// k_stage and the adjoint's kernels stop on any error: none is recorded on their stream while they run, but another
// stream's k_prep may record one for the same words (the adjoint's recompute beside its reverse sweep)
__device__ __forceinline__ bool warp_failed(const Fields &F) { return __any_sync(~0u, err_word(F) != ERR_NONE); }
// The same in k_stage, where one thread of a launch (latch) hands the error on to the kernels that stop on earlier
// errors alone, with the word it has read: a read of its own before the block's barrier was 0.4 us of every stage
__device__ __forceinline__ bool stage_failed(const Fields &F, bool latch) {
  const unsigned long long w = err_word(F);
  if (latch && w != ERR_NONE) F.err[1] = w;
  return __any_sync(~0u, w != ERR_NONE);
}

// ----------------------------------------------------------------------------
// Multi-instance launches (the batched form): one launch runs one kernel of a stage for up to
// CAP instances with the same degrees (so the same kernel and the same 1D operators) and
// any mesh sizes. Their arguments travel in the launch's parameter block. The launch covers
// first[n] virtual blocks: virtual block vb belongs to the instance i with first[i] ≤ vb <
// first[i+1] and covers `tile` elements (or element slots of the mass solves' order) of it,
// from (vb - first[i]) tile on. Each block runs the single-instance kernel's
// body on its instance's arguments, so an element's arithmetic is the same as in a launch of its
// instance alone. A grid smaller than first[n] makes the launch
// persistent: block b takes the virtual blocks b, b + gridDim.x, ...
// ----------------------------------------------------------------------------
struct StageArgs {
  Fields F;
  StageIO S;
};

// Where kernels are launched early (launch_after), every thread waits here for the end of the kernel before
// on the stream, and with it of all before that, ahead of the first read or write of memory. Without such
// a launch it does nothing.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class Args, int CAP>
struct Multi {
  static constexpr int cap = CAP;
  int n, tile;
  int first[CAP + 1];
  Args a[CAP];
};

// CAP is what fits the kernel parameter limit (32 764 bytes) beside the largest Basis
using MultiStage = Multi<StageArgs, 22>;

// The instance of virtual block vb. The kernels read that instance's arguments where they lie, in
// the parameter block: the index is the same for the whole block, so the reads are uniform
// constant-bank loads. The barrier keeps a persistent block's next virtual block from reusing
// shared memory that threads of the previous one still read.
template <class Args, int CAP>
__device__ __forceinline__ int multi_begin(const Multi<Args, CAP> &P, int vb) {
  int inst = 0;
  while (inst + 1 < P.n && vb >= P.first[inst + 1]) ++inst;
  __syncthreads();
  return inst;
}

// ----------------------------------------------------------------------------
// Mirror-parity contractions. The points of both quadratures are Gauss-Legendre
// points (mirrored through the element centre) and the basis is the Legendre one,
// so P[n-1-i][d] = (-1)^d P[i][d] for the values and the opposite sign for the
// derivatives (the host makes these exact). A contraction over the modes is then
// done on the first half of the points only: its even-mode and odd-mode parts give
// the point and its mirror as a sum and a difference.
// ----------------------------------------------------------------------------

// Y[s] = Σ_b T[b] Ph[s][b] at all QH points
template <int QH, int NV>
__device__ __forceinline__ void ph_to_points(const double (&Ph)[QH][NV], const double (&T)[NV], double (&Y)[QH]) {
#pragma unroll
  for (int s = 0; s < QH / 2; ++s) {
    double ev = 0.0, od = 0.0;
#pragma unroll
    for (int b = 0; b < NV; b += 2) ev = fma(T[b], Ph[s][b], ev);
#pragma unroll
    for (int b = 1; b < NV; b += 2) od = fma(T[b], Ph[s][b], od);
    Y[s] = ev + od;
    Y[QH - 1 - s] = ev - od;
  }
  if constexpr ((QH & 1) != 0) {
    double ev = 0.0;
#pragma unroll
    for (int b = 0; b < NV; b += 2) ev = fma(T[b], Ph[QH / 2][b], ev);
    Y[QH / 2] = ev;
  }
}

// ----------------------------------------------------------------------------
// k_prep: traces, boundary weight check, Chebyshev interval data
// ----------------------------------------------------------------------------

// Row QH² of G: the exponent sG of the element's integers G (G = integer 2^sG) and the shift ng that
// takes their largest to [2^59, 2^60)
struct GPack {
  static constexpr int BAD = INT_MIN;                    // sG where V or β is not finite
  int sG, ng;
  __device__ GPack(int s, i64 lo, i64 hi) : sG(s) {
    const i64 top = max(hi, -lo);
    ng = top > 0 ? __clzll(top) - 4 : 0;
  }
  __device__ explicit GPack(i64 w) : sG((int)(w >> 32)), ng((int)w) {}
  __device__ i64 word() const { return (i64)sG << 32 | (unsigned)ng; }
};

// ----------------------------------------------------------------------------
// k_stage helpers
// ----------------------------------------------------------------------------

// Coefficients of an interior face point: the one-sided values of c² and α on the "-" and "+"
// sides and the jump term K (one-sided faces), or the face values c², α (continuous faces)
struct FaceCoef {
  double c2m, c2p, afm, afp, K;
};
__device__ __forceinline__ FaceCoef face_coef(const Fields &F, const double *c2p_a, const double *afp_a,
                                              const double *c2m_a, const double *afm_a, const double *jc_a,
                                              size_t fi) {
  if (F.one_sided) return FaceCoef{c2m_a[fi], c2p_a[fi], afm_a[fi], afp_a[fi], jc_a[fi]};
  return FaceCoef{0.0, c2p_a[fi], 0.0, afp_a[fi], 0.0};
}

// The flux slots of the "+" (plus) or "-" element at an interior face point from the traces of
// both elements (src/rhs.jl:620-700): affine in (dum, dup, vm, vp, dvm, dvp)
__device__ __forceinline__ void interior_flux(const Fields &F, const FaceCoef &cf, bool plus, double dum,
                                              double dup, double vm, double vp, double dvm, double dvp,
                                              double &A, double &D, double &Fs) {
  const double th = F.theta, tau = F.tau, two_h = F.two_h;
  if (F.one_sided) {
    const double c2m = cf.c2m, c2p = cf.c2p, afm = cf.afm, afp = cf.afp, K = cf.K;
    const double J = two_h * (c2m * dum - c2p * dup + afm * dvm - afp * dvp) + K;
    const double G = two_h * ((1 - th) * (c2m * dum + afm * dvm) + th * (c2p * dup + afp * dvp));
    const double pen = (0.5 * (c2m + c2p)) * F.lu + (0.5 * (afm + afp)) * F.lv;
    const double sj = vm - vp;
    if (plus) {
      const double dvsp = th * sj - tau * J;
      A = pen * sj - G - (1 - th) * K; D = -afp * dvsp; Fs = c2p * dvsp;
    } else {
      const double dvsm = (1 - th) * (vp - vm) - tau * J;
      A = G - pen * sj - th * K; D = afm * dvsm; Fs = -c2m * dvsm;
    }
  } else {
    const double c2 = cf.c2p, af = cf.afp;
    const double gs = two_h * (c2 * (th * dup + (1 - th) * dum) + af * (th * dvp + (1 - th) * dvm));
    const double Jt = c2 * (two_h * (dum - dup)) + af * (two_h * (dvm - dvp));
    const double pen = c2 * F.lu + af * F.lv;
    if (plus) {
      A = pen * (vm - vp) - gs;
      D = -af * (th * (vm - vp) - tau * Jt);
      Fs = c2 * (th * (vm - vp) - tau * Jt);
    } else {
      A = gs - pen * (vm - vp);
      D = af * ((1 - th) * (vp - vm) - tau * Jt);
      Fs = -c2 * ((1 - th) * (vp - vm) - tau * Jt);
    }
  }
}

// Numerical flux slots A, D, F at point i of physical side s of the element (src/rhs.jl:65-103, 738-763)
template <int NU, int NV>
__device__ __forceinline__ void boundary_point(const Fields &F, const TimeF &S, int s, int j,
                                               int k, int i, double du, double v_fp, double dv_fp, double &A,
                                               double &D, double &Fs) {
  const int N = F.N;
  const int m = s < 2 ? k : j;
  const double sgn = (s == 0 || s == 2) ? -1.0 : 1.0;
  size_t fi;
  const double *c2a, *afa, *cfa, *bfa;
  if (s < 2) { fi = (s == 0 ? 0 : N) + (size_t)(N + 1) * (k + (size_t)N * i); c2a = F.hc2; afa = F.haf; cfa = F.hcf; bfa = F.hbf; }
  else { fi = j + (size_t)N * ((s == 2 ? 0 : N) + (size_t)(N + 1) * i); c2a = F.vc2; afa = F.vaf; cfa = F.vcf; bfa = F.vbf; }
  const double c2f = c2a[fi], af = afa[fi], cf = cfa[fi];
  const double gun = sgn * (F.two_h * du), gvn = sgn * (F.two_h * dv_fp);
  const double spn = F.bspn[s][m + (size_t)N * i], sp = F.bsp[s][m + (size_t)N * i];
  const double gu_ex = sgn * (S.ct * spn - spn);
  const double gv_ex = sgn * (-F.omega * S.st * spn);
  const double v_ex = -F.omega * S.st * sp;
  double F1, dv;
  if (F.kind[s] == 3) {
    const double g2 = c2f * gu_ex + af * gv_ex;
    const double rho_w = c2f * gun + af * gvn - g2;
    dv = -(F.kap[s] / cf) * rho_w;
    F1 = g2;
  } else {
    const double bf = bfa[fi];
    const double g = F.gam[s], et = F.eta[s], sg = F.sig[s], kb = F.kb[s];
    const double sqf = sqrt(1.0 - kb * bf * v_fp);
    const double rho_num = et * (c2f * gun + af * gvn) + g * cf * sqf * v_fp;
    const double rho_ex = et * (c2f * gu_ex + af * gv_ex) + g * cf * sqrt(1.0 - kb * bf * v_ex) * v_ex;
    const double rho = rho_num - rho_ex;
    F1 = c2f * gun + af * gvn - (et + sg * g) * rho;
    dv = -(g - sg * et) / (cf * sqf) * rho;
  }
  A = F1;
  D = sgn * (af * dv);
  Fs = -sgn * (c2f * dv);
}

// Numerical flux slots A, D, F at point i of interior side s of the element (src/rhs.jl:620-700)
template <int NU, int NV>
__device__ __forceinline__ void side_point(const Fields &F, int s, int j, int k, int e, int i, double &A, double &D,
                                           double &Fs) {
  constexpr int NQ = NU;
  const int N = F.N, E = F.E;
  const double *tr = F.tr;
  auto T = [&](int fam, int side, int el) { return tr[((fam * 4 + side) * NQ + i) * (size_t)E + el]; };
  // interior: the element is "+" on its B and L sides, "-" on T and R
  const bool plus = (s == 0 || s == 2);
  const int nb = s == 0 ? e - 1 : s == 1 ? e + 1 : s == 2 ? e - N : e + N;
  const int sm = s < 2 ? 1 : 3, spp = s < 2 ? 0 : 2;      // trace sides of the "-" and "+" elements
  const int em = plus ? nb : e, ep = plus ? e : nb;
  size_t fi;
  const double *c2p_a, *afp_a, *c2m_a, *afm_a, *jc_a;
  if (s < 2) {
    fi = (s == 0 ? j : j + 1) + (size_t)(N + 1) * (k + (size_t)N * i);
    c2p_a = F.hc2; afp_a = F.haf; c2m_a = F.hc2m; afm_a = F.hafm; jc_a = F.hJC;
  } else {
    fi = j + (size_t)N * ((s == 2 ? k : k + 1) + (size_t)(N + 1) * i);
    c2p_a = F.vc2; afp_a = F.vaf; c2m_a = F.vc2m; afm_a = F.vafm; jc_a = F.vJC;
  }
  const double vm = T(1, sm, em), vp = T(1, spp, ep);
  const double dum = T(0, sm, em), dup = T(0, spp, ep);
  const double dvm = T(2, sm, em), dvp = T(2, spp, ep);
  const FaceCoef cf = face_coef(F, c2p_a, afp_a, c2m_a, afm_a, jc_a, fi);
  interior_flux(F, cf, plus, dum, dup, vm, vp, dvm, dvp, A, D, Fs);
}

// The physical sides, a team of NQ lanes per side: lane i takes the side's traces at mode i from the state,
// evaluates the flux slots at point i, then projects them on mode i (Y[b] = Σ_q w_q P[q][b] (.)_q), and k_stage reads the
// projections. A point costs about 150 FP64 operations (two square roots and the divisions); in its
// element's thread of k_stage a side held the 31 others of the warp up for 7 points on end, in every
// fourth warp at N = 256 and in every one below N = 64, and the columns of the left and right sides
// were whole warps of it. With traces of their own (6 NU operations a lane) the sides need nothing of k_prep,
// so a launch of it over all elements has them as its first blocks; after k_prep, as a kernel of their own
// (k_bnd: after a k_prep by ranges of elements, and k_bnd_m), they take 6 to 9 us of a stage: N = 64 31 -> 23 us with
// k_prep, N = 512 445 -> 436.
constexpr int BND_THREADS = 32;
__host__ __device__ constexpr int bnd_tile(int nu) { return BND_THREADS / nu; }
template <int NU, int NV>
__device__ __forceinline__ void bnd_body(const Basis<NU, NV> &B, const Fields &F, const StageIO &S, int side0) {
  constexpr int NQ = NU;
  const int N = F.N, E = F.E, lane = threadIdx.x & 31, tw = lane / NQ, i = lane - tw * NQ;
  const int x = side0 + tw;
  if (tw >= bnd_tile(NU) || x >= 4 * N) return;
  const unsigned mask = ((1u << NQ) - 1u) << (tw * NQ);
  const TimeF tf = time_factors(S);
  const int s = x / N, m = x - s * N;
  const int j = s == 0 ? 0 : s == 1 ? N - 1 : m, k = s == 2 ? 0 : s == 3 ? N - 1 : m, e = j + N * k;
  // the side's traces: the sums over the normal modes at mode i along the side, then at point i
  const size_t Eu = (size_t)E;
  const bool hi = s & 1, along = s < 2, has_v = i < NV;
  double xe = 0, xo = 0, ve = 0, vo = 0, de = 0, dd = 0;
#pragma unroll
  for (int a = 0; a < NU; ++a) {
    const double x = S.xu[e + Eu * (along ? a + NU * i : i + NU * a)];
    if (a & 1) xo = fma(B.E1l[a], x, xo);
    else xe = fma(B.E1l[a], x, xe);
  }
#pragma unroll
  for (int a = 0; a < NV; ++a) {
    const double x = has_v ? S.xv[e + Eu * (along ? a + NV * i : i + NV * a)] : 0.0;
    if (a & 1) { vo = fma(B.El[a], x, vo); dd = fma(B.E1l[a], x, dd); }
    else { ve = fma(B.El[a], x, ve); de = fma(B.E1l[a], x, de); }
  }
  const double mu = hi ? xo - xe : xe + xo, mv = hi ? ve - vo : ve + vo, md = hi ? dd - de : de + dd;
  double du = 0.0, v = 0.0, dv = 0.0;
#pragma unroll
  for (int b = 0; b < NU; ++b) {
    const double p = B.P[i][b];
    du = fma(p, __shfl_sync(mask, mu, tw * NQ + b), du);
    if (b < NV) {
      v = fma(p, __shfl_sync(mask, mv, tw * NQ + b), v);
      dv = fma(p, __shfl_sync(mask, md, tw * NQ + b), dv);
    }
  }
  double A, D, Fs;
  boundary_point<NU, NV>(F, tf, s, j, k, i, du, v, dv, A, D, Fs);
  double ya = 0.0, yd = 0.0, yf = 0.0;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const double p = B.Pw[q][i];
    ya = fma(p, __shfl_sync(mask, A, tw * NQ + q), ya);
    yd = fma(p, __shfl_sync(mask, D, tw * NQ + q), yd);
    yf = fma(p, __shfl_sync(mask, Fs, tw * NQ + q), yf);
  }
  double *o = F.bslots + x;
  const size_t st = (size_t)4 * N;
  if (i < NV) {
    o[i * st] = ya;
    o[(NV + i) * st] = yd;
  }
  o[(2 * NV + i) * st] = yf;
}
template <int NU, int NV>
__global__ void __launch_bounds__(BND_THREADS) k_bnd(const __grid_constant__ Basis<NU, NV> B,
                                                     const __grid_constant__ Fields F,
                                                     const __grid_constant__ StageIO S) {
  after_previous();
  bnd_body<NU, NV>(B, F, S, blockIdx.x * bnd_tile(NU));
}
// tile = bnd_tile(NU) sides per virtual block, of the 4N of an instance
template <int NU, int NV>
__global__ void __launch_bounds__(BND_THREADS) k_bnd_m(const __grid_constant__ Basis<NU, NV> B,
                                                       const __grid_constant__ MultiStage P) {
  for (int vb = blockIdx.x; vb < P.first[P.n]; vb += gridDim.x) {
    const int inst = multi_begin(P, vb);
    bnd_body<NU, NV>(B, P.a[inst].F, P.a[inst].S, (vb - P.first[inst]) * P.tile);
  }
}

// Count of Chebyshev steps for the interval θ ± δ: ceil(L / acosh(θ/δ)), from FP32 where that is not within its
// rounding of a whole number (acosh costs some 100 FP64 operations). FP32's θ/δ is good to 2e-7, acosh of it
// to 1e-5 from 1.01 on; closer to 1 the count is taken in FP64
__device__ __forceinline__ int cheb_count(double L, double th, double de) {
  const float x = (float)L / acoshf((float)th / (float)de), r = rintf(x);
  if (th > 1.01 * de && x < 1e6f && fabsf(x - r) > 1e-4f * x + 1e-4f) return (int)ceilf(x);
  return (int)ceil(L / acosh(th / de));
}

// k_prep: a team of NU threads per element. Thread r takes the sums over the normal modes at mode r of
// the four sides (column r and row r of the blocks), the r-th face point, column r of P_h V and the
// point rows r, r + NU, ... With a thread per element a warp held the chip's FP64 pipes for the
// whole of its 378 trace operations and two blocks of state per thread; the team fills them from more
// warps and spreads small meshes over the chip.
//
// What bounds it: the FP64 pipe (60 %: the traces, and a conversion per entry of V and 2β) and the latency of
// its loads. N = 512, q = 6: 760 us as FP64 code with a thread per element; 526, 488, 458 and 442 us so at four, five,
// six and eight blocks an SM (64 registers), the last with the physical sides 445, and 435 with them in its own blocks.
template <int NU, int NV>
struct PrepTeam {
  static constexpr int QH = qhigh(NU, NV), TPW = 32 / NU;
  static constexpr int S0 = NU * NU + NV * NV, S1 = 12 * NU, S2 = QH * NV;
  static constexpr int SLOT = (S0 > S1 ? (S0 > S2 ? S0 : S2) : S1 > S2 ? S1 : S2) | 1;   // odd: bank conflicts
};
__host__ __device__ constexpr int prep_tile(int nu, int threads) { return (threads / 32) * (32 / nu); }
// Blocks per SM asked of k_prep: eight (64 registers), and twelve up to q_u = 2, where a thread needs fewer (N = 1024,
// q_u = 1: 231 and 208 us)
__host__ __device__ constexpr int prep_blocks(int nu) { return nu <= 3 ? 12 : 8; }

// The block's elements from e0 on (first: the instance's first block, which clears the bin counts)
template <int NU, int NV>
__device__ __forceinline__ void prep_body(const Basis<NU, NV> &B, const Fields &F, const StageIO &S, int e0,
                                          bool first) {
  using T = PrepTeam<NU, NV>;
  constexpr int NQ = NU, QH = T::QH;
  __shared__ double sh[T::TPW * 4 * T::SLOT];
  __shared__ double Ps[NQ * NU];
  const int E = F.E;
  // the bin counts and the largest count of the next stage start at zero: all NBIN bins, whatever
  // the element count
  if (first && F.sorted)
    for (int b = threadIdx.x; b < NBIN; b += blockDim.x) F.bin_count[(1 - S.parity) * NBIN + b] = 0;
  if (first && threadIdx.x == 0) F.nmax[1 - S.parity] = 0;
  for (int i = threadIdx.x; i < NQ * NU; i += blockDim.x) Ps[i] = B.P[i / NU][i % NU];
  __syncthreads();
  if (prep_stopped(F)) return;
  const int lane = threadIdx.x & 31, tw = lane / NU;
  if (tw >= T::TPW) return;
  const int r = lane - tw * NU, slot = (threadIdx.x >> 5) * T::TPW + tw, e = e0 + slot;
  if (e >= E) return;
  const unsigned mask = ((1u << NU) - 1u) << (tw * NU);
  const Team team{mask, tw * NU, r};
  const size_t Eu = (size_t)E;
  const bool has_v = r < NV, modal = F.modal != 0;
  double *Us = sh + slot * T::SLOT, *Vs = Us + NU * NU;
  // ---- traces (src/rhs.jl:388-410): the sums over the normal modes, at mode r: family x (du, v, dv) of the
  //      low and the high side of both axes; El, Er are the values or derivatives of the modes at the
  //      two ends, Er[a] = ±(-1)^a El[a], so both ends come from the even and odd parts of one sum
  double V[NV];
  double lo[3][2], hi[3][2];
  int hu = 0, hv = 0;                                    // the largest high words beside the constant mode
  auto ends = [&](double xe, double xo, bool der, double &l, double &h) {
    l = xe + xo;
    h = der ? xo - xe : xe - xo;
  };
  {
    double U[NU];
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      U[a] = S.xu[e + Eu * (a + NU * r)];
      Us[a + NU * r] = U[a];
      if (a + r > 0) hu = max(hu, fx_abs_hi(U[a]));
    }
#pragma unroll
    for (int a = 0; a < NV; ++a) {
      V[a] = has_v ? S.xv[e + Eu * (a + NV * r)] : 0.0;
      if (has_v) Vs[a + NV * r] = V[a];
      if (a + r > 0) hv = max(hv, fx_abs_hi(V[a]));
    }
    __syncwarp(mask);
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {
      double ue = 0, uo = 0, ve = 0, vo = 0, de = 0, d_o = 0;
#pragma unroll
      for (int a = 0; a < NU; ++a) {
        const double x = ax == 0 ? U[a] : Us[r + NU * a];
        if (a & 1) uo = fma(B.E1l[a], x, uo); else ue = fma(B.E1l[a], x, ue);
        if (a < NV) {
          const double y = ax == 0 ? V[a] : has_v ? Vs[r + NV * a] : 0.0;
          if (a & 1) { vo = fma(B.El[a], y, vo); d_o = fma(B.E1l[a], y, d_o); }
          else { ve = fma(B.El[a], y, ve); de = fma(B.E1l[a], y, de); }
        }
      }
      ends(ue, uo, true, lo[0][ax], hi[0][ax]);
      ends(ve, vo, false, lo[1][ax], hi[1][ax]);
      ends(de, d_o, true, lo[2][ax], hi[2][ax]);
    }
  }
  hu = team_max<NU>(team, hu);
  hv = team_max<NU>(team, hv);
  i64 *Gi = reinterpret_cast<i64 *>(F.G);
  if (r == 0) Gi[(size_t)(QH * QH + 1) * E + e] = (i64)hu << 32 | hv;
  const int N = F.N, j = e % N, k = e / N;
  const bool onb[4] = {j == 0, j == N - 1, k == 0, k == N - 1};
  const bool check = (onb[0] && F.kind[0] != 3) || (onb[1] && F.kind[1] != 3) || (onb[2] && F.kind[2] != 3) ||
                     (onb[3] && F.kind[3] != 3);
  __syncwarp(mask);                                      // U, V in shared memory are spent
  double *ss = Us;                                       // the sums, [(fam 4 + side) NU + mode]
  if (!modal || check) {
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int ax = 0; ax < 2; ++ax) {
        ss[(f * 4 + 2 * ax) * NU + r] = lo[f][ax];
        ss[(f * 4 + 2 * ax + 1) * NU + r] = hi[f][ax];
      }
    __syncwarp(mask);
  }
  // the sum over the face modes at point r
  auto at = [&](int f, int s) {
    double x = 0.0;
#pragma unroll
    for (int b = 0; b < NU; ++b)
      if (f == 0 || b < NV) x = fma(Ps[r * NU + b], ss[(f * 4 + s) * NU + b], x);
    return x;
  };
  if (modal) {             // the end sums themselves, mode r in the slot of point r
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int ax = 0; ax < 2; ++ax)
        if (f == 0 || has_v) {
          F.tr[((f * 4 + 2 * ax) * NQ + r) * Eu + e] = lo[f][ax];
          F.tr[((f * 4 + 2 * ax + 1) * NQ + r) * Eu + e] = hi[f][ax];
        }
  } else {
#pragma unroll 1
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int f = 0; f < 3; ++f) F.tr[((f * 4 + s) * NQ + r) * Eu + e] = at(f, s);
  }
  // weight check 1 - kβv > 0 for the trace and the data on physical sides at point r
  // (src/rhs.jl:109-110, 751-757); key of src/rhs.jl:732
  if (check) {
    const double st = time_factors(S).st;
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
      if (!onb[s] || F.kind[s] == 3) continue;
      const int m = s < 2 ? k : j;
      const double bf = s < 2 ? F.hbf[(s == 0 ? 0 : N) + (size_t)(N + 1) * (k + (size_t)N * r)]
                              : F.vbf[j + (size_t)N * ((s == 2 ? 0 : N) + (size_t)(N + 1) * r)];
      const double v_fp = at(1, s), v_ex = -F.omega * st * F.bsp[s][m + (size_t)N * r];
      const int bad = (1.0 - F.kb[s] * bf * v_fp <= 0.0) ? 1 : (1.0 - F.kb[s] * bf * v_ex <= 0.0) ? 2 : 0;
      if (bad) atomicMin(F.err, 2ull * ((unsigned long long)s * NQ * N + r + (unsigned long long)m * NQ) + bad);
    }
  }

  // ---- Chebyshev interval of the element: v_q = P_h V P_h^T, G = 2βv_q, a± = 1 - extrema(G), in fixed
  //      point (the integers of V and 2β share an exponent over the element)
  int hb = 0;
#pragma unroll 1
  for (int q = r; q < QH; q += NU)
#pragma unroll
    for (int s2 = 0; s2 < QH; ++s2) hb = max(hb, fx_abs_hi(F.beta2[(q + QH * s2) * Eu + e]));
  hb = team_max<NU>(team, hb);
  hv = max(hv, __shfl_sync(mask, fx_abs_hi(V[0]), team.lane0));   // with the constant mode
  const bool nan = !fx_finite(hv) || !fx_finite(hb);
  const int ev = fx_exp(hv), eb = fx_exp(hb) + 2;
  Fx2 x[NV];
  int top = 0;
#pragma unroll
  for (int a = 0; a < NV; ++a) {
    const i64 y = fx_from(V[a], ev);
    x[a] = fx_split(y);
    top += (B.cPh[a] * ((fx_hi(y) >> 12) + 1)) >> 8;
  }
  // the rows T = Ph V go up by nt, the room that Σ_a max|Ph[.][a]| |V[a][b]| leaves in every column, so that
  // v_q has the bits which the levels' headroom for any V would take (top 2^12 bounds the high words
  // of T 2^(61 - gPh))
  const int nt = max(__clz(team_max<NU>(team, top)) - 3 - 12 + (61 - B.gPh), 0);
  const int sG = (ev - FX_BIAS) + 2 * (61 - B.gPh) - nt + (eb - FX_BIAS) + 61;   // G = (integer) 2^sG
  Fx2 *Ts = reinterpret_cast<Fx2 *>(Us);                 // T[q][b] at Ts[q NV + b]
  __syncwarp(mask);                                      // the sums are spent
  if (has_v) {
    auto xa = [&](int a) { return x[a]; };
#pragma unroll
    for (int q = 0; q < (QH + 1) / 2; ++q) {
      auto c = [&](int a) -> const FxC & { return B.fPh[q][a]; };
      const i64 t0 = fx_dot<0, 2, NV>(xa, c), t1 = fx_dot<1, 2, NV>(xa, c);
      Ts[q * NV + r] = fx_split((t0 + t1) << nt);
      if (2 * q + 1 != QH) Ts[(QH - 1 - q) * NV + r] = fx_split((t0 - t1) << nt);
    }
  }
  __syncwarp(mask);
  i64 kmin = LLONG_MAX, kmax = LLONG_MIN;
#pragma unroll 1
  for (int q = r; q < QH; q += NU) {
#pragma unroll
    for (int b = 0; b < NV; ++b) x[b] = Ts[q * NV + b];
    auto tb = [&](int b) { return x[b]; };
    auto point = [&](i64 y, int s2) {
      const size_t gi = (q + QH * s2) * Eu + e;
      const i64 g = fx_mul(fx_split(y), fx_split(fx_from(F.beta2[gi], eb)));
      Gi[gi] = g;
      kmin = min(kmin, g);
      kmax = max(kmax, g);
    };
    // v_q = Σ_b T[b] Ph[s2][b], mirrored columns s2 and QH-1-s2 together
#pragma unroll
    for (int s2 = 0; s2 < QH / 2; ++s2) {
      auto c = [&](int b) -> const FxC & { return B.fPh[s2][b]; };
      const i64 t0 = fx_dot<0, 2, NV>(tb, c), t1 = fx_dot<1, 2, NV>(tb, c);
      point(t0 + t1, s2);
      point(t0 - t1, QH - 1 - s2);
    }
    if constexpr ((QH & 1) != 0)
      point(fx_dot<0, 2, NV>(tb, [&](int b) -> const FxC & { return B.fPh[QH / 2][b]; }), QH / 2);
  }
  kmax = team_max<NU>(team, kmax);
  kmin = team_min<NU>(team, kmin);
  if (r != 0) return;
  Gi[(size_t)QH * QH * E + e] = GPack(nan ? GPack::BAD : sG, kmin, kmax).word();
  if (F.cg) return;                                      // (k_cg finds a matrix that is not positive definite)
  const double gmin = ldexp((double)kmin, sG), gmax = ldexp((double)kmax, sG);
  const double amin = 1.0 - gmax, amax = 1.0 - gmin;
  const double th = 0.5 * (amax + amin);
  const double de = fmax(0.5 * (amax - amin), 1e-15 * th);
  const int n = cheb_count(F.Lcheb, th, de);
  // (no count: θ = δ to the last bit, a matrix that is singular to rounding. The conversion of an infinite
  // count gives INT_MAX, steps for an hour)
  if (nan || !(amin > 0.0) || n == INT_MAX) {
    atomicMin(F.err, (1ull << ERR_CLASS_SHIFT) | (unsigned long long)(e + 1));
    return;
  }
  F.th[e] = th;
  F.de[e] = de;
  F.nst[e] = n;
  // largest count and the sum of the counts: one atomic each per warp
  const unsigned am = __activemask();
  const int nw = __reduce_max_sync(am, n);
  const unsigned ns = __reduce_add_sync(am, (unsigned)n);
  if (lane == __ffs(am) - 1) {
    atomicMax(&F.nmax[S.parity], nw);
    atomicMax(&F.nmax[2], nw);
    atomicAdd(F.nsum, (unsigned long long)ns);
  }
  if (F.sorted) {
    // append e to the list of its count, one atomic per group of lanes with the same count
    const int bin = (n < NBIN ? n : NBIN) - 1;
    const unsigned same = __match_any_sync(am, bin);
    const int leader = __ffs(same) - 1;
    const int rank = __popc(same & ((1u << lane) - 1));
    int first_slot = 0;
    if (lane == leader) first_slot = atomicAdd(&F.bin_count[S.parity * NBIN + bin], __popc(same));
    first_slot = __shfl_sync(same, first_slot, leader);
    F.bins[(size_t)bin * E + first_slot + rank] = e;
  }
}

template <int NU, int NV>
__global__ void __launch_bounds__(128, prep_blocks(NU)) k_prep(const __grid_constant__ Basis<NU, NV> B,
                                              const __grid_constant__ Fields F,
                                              const __grid_constant__ StageIO S, int e0, int nb) {
  after_previous();
  const int vb = (int)blockIdx.x - nb;
  if (vb < 0) {                                          // the first nb blocks take the physical sides
    bnd_body<NU, NV>(B, F, S, (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * bnd_tile(NU));
    return;
  }
  // elements from e0 on: a launch may cover a range of the elements (the first range clears the next
  // stage's counts)
  prep_body<NU, NV>(B, F, S, e0 + vb * prep_tile(NU, blockDim.x), vb == 0 && e0 == 0);
}

// tile = prep_tile(NU, threads) elements per virtual block
template <int NU, int NV>
__global__ void __launch_bounds__(128, prep_blocks(NU)) k_prep_m(const __grid_constant__ Basis<NU, NV> B,
                                                const __grid_constant__ MultiStage P) {
  for (int vb = blockIdx.x; vb < P.first[P.n]; vb += gridDim.x) {
    const int inst = multi_begin(P, vb);
    const int e0 = (vb - P.first[inst]) * P.tile;
    prep_body<NU, NV>(B, P.a[inst].F, P.a[inst].S, e0, e0 == 0);
  }
}

}  // namespace wedg

#include "wedg_stage_fx.cuh"
#include "wedg_stage_gen.cuh"

namespace wedg {

// Blocks per SM asked of k_stage: the constant-coefficient kernels six (80 registers), the general ones
// three (168)
__host__ __device__ constexpr int stage_m_blocks(int, bool fast) { return fast ? 6 : 3; }

template <int NU, int NV, bool FAST>
__global__ void __launch_bounds__(STAGE_THREADS, stage_m_blocks(NU, FAST))
    k_stage(const __grid_constant__ Basis<NU, NV> B, const __grid_constant__ Fields F,
            const __grid_constant__ StageIO S) {
  const int e0 = blockIdx.x * stage_tile(NU);
  if constexpr (FAST) stage_fast_body<NU, NV>(B, F, S, e0);
  else stage_gen_body<NU, NV>(B, F, S, e0);
}


// tile = stage_tile(NU) elements per virtual block
template <int NU, int NV, bool FAST>
__global__ void __launch_bounds__(STAGE_THREADS, stage_m_blocks(NU, FAST))
    k_stage_m(const __grid_constant__ Basis<NU, NV> B, const __grid_constant__ MultiStage P) {
  for (int vb = blockIdx.x; vb < P.first[P.n]; vb += gridDim.x) {
    const int inst = multi_begin(P, vb);
    const int e0 = (vb - P.first[inst]) * P.tile;
    if constexpr (FAST) stage_fast_body<NU, NV>(B, P.a[inst].F, P.a[inst].S, e0);
    else stage_gen_body<NU, NV>(B, P.a[inst].F, P.a[inst].S, e0);
  }
}

// ----------------------------------------------------------------------------
// The mass solve M(v_h) VT = R on every element (src/rhs.jl:778-951) and the v part of the outputs
// ----------------------------------------------------------------------------

// element of thread g: in the order of the Chebyshev step counts, or in mesh order
// (largest counts first: the blocks with the most work start first, and the short ones fill the
// SMs behind them). pref[b] = number of elements in the bins above b.
__device__ __forceinline__ int mass_element(const Fields &F, const StageIO &S, int g, int *pref) {
  if (!F.sorted) return g;
  int lo = NBIN - 1;
#pragma unroll 1
  for (int b = 0; b < NBIN; ++b)
    if (pref[b] <= g) { lo = b; break; }
  return F.bins[(size_t)lo * F.E + (g - pref[lo])];
}

// v outputs of modal entry l = e + E (a + NV b): RK4 as in k_stage (src/solver.jl:299-321)
__device__ __forceinline__ void store_v(const StageIO &S, size_t l, double kk, bool &fin) {
  if (S.mode == OUT_RHS) {
    S.vt[l] = kk;
  } else if (S.mode == OUT_RK4_STAGE) {
    S.accv[l] = S.first ? kk : S.accv[l] + 2.0 * kk;
    S.sv[l] = S.v0[l] + S.c * kk;
  } else if (S.mode == OUT_RK4_LAST) {
    const double x = S.v0[l] + S.c * (S.accv[l] + kk);
    S.vo[l] = x;
    fin = fin && isfinite(x);
  } else {
    S.accv[l] = S.accv[l] + kk;
  }
}

// k_cheb: the Chebyshev mass solve (Saad Alg. 12.1, src/rhs.jl:920-939), a team of QH threads per
// element: thread u takes row u of the point grid and J of the modal entries. Elements are visited in
// decreasing order of their step counts (k_prep lists them by count), so the longest solves start
// first.
//
// The iteration runs in fixed point on the system scaled by the middle θ of the spectral interval,
// (M/θ) X' = R with X' = θX, whose spectrum is 1 ± ε, ε = δ/θ. r, X' and d are integers r 2^nr, X' 2^nX and
// d 2^nd of the exponent of R, each brought to the top of its range by its own shift after every step, so
// that each keeps some 55 bits of its own size or more, however far the residual falls and whatever ε, θ and
// G are. (With one exponent for r and X' over all steps, and the headroom that the solution may need,
// 49 bits were left at ε close to 1, and systems beyond ε = 31/32 took a form in FP64.)
//
// What bounds it: one product with M costs about 1 300 multiply-adds an element at q = 6, three integer
// ones each (2 cycles a warp) and as much again on the ALU, and 18 shared-memory words a thread: both pipes are 57 to
// 60 % busy where every element takes 29 steps. A thread per row keeps 20 to 24 warps an SM
// where a thread per pair of rows (half the exchanges, 16 warps) left the pipes waiting.
// N = 512, q = 6, a front (3.6 steps on average): 2 569 us in FP64, 890 us so (1 004 us with a thread per
// pair of rows). N = 300, q_v = 7, 27 steps: 12 850 us in FP64, 4 620 us so. N = 333, q = 2, 19 steps: 282 us.
template <int NU, int NV>
struct MassTeam {
  static constexpr int QH = qhigh(NU, NV);
  static constexpr int HP = (QH + 1) / 2;               // row pairs (and the middle row)
  static constexpr int TPW = 32 / QH;                   // teams per warp
  static constexpr int TPB = TPW * (CHEB_THREADS / 32); // elements per block
  static constexpr int NE = NV * NV;
  static constexpr int J = (NE + QH - 1) / QH;          // modal entries per thread
  static constexpr int ZR = 2 * HP * NV;                // the sums and differences of row pairs
  static constexpr int SLOT = (2 * NE + ZR + QH * QH) | 1;   // d, X', the rows, G; odd: bank conflicts
};
__host__ __device__ constexpr int mass_tile(int nu, int nv, int threads) {
  return (threads / 32) * (32 / qhigh(nu, nv));
}

// One product with K = P_h^T W G P_h for x in xs (Fx2, below 2^61, complete, after a __syncwarp) and G in
// Gs: use(j, k, y, ey) for the thread's entries k = u + QH j, where K x = y 2^(sG - ng + ey) (GPack) in the
// integers of x. The operators' exponents leave headroom at every level for the largest sums that are
// possible, up to four bits more than sums usually take. So each level's numbers go up to the top of their
// range by what room they have: the thread's row T and its weighted points by nt, the rows of the team by nz.
// Without the second and third shift the error of a product was 2 to 5e-16 of its largest entry from n_v = 4
// on, as in FP64 or twice that, and is 0.3 to 1e-16 so. Up to n_v = 3 (0.5 to 1.6e-16) the rows go up by
// what the norms leave in every case (nrow), and the last level takes the products of the low halves too: the
// shifts would cost a tenth of such a product.
template <int NU, int NV, class Use>
__device__ __forceinline__ void team_K_fx(const Basis<NU, NV> &B, const Fx2 *Gs, const Team &team, const Fx2 *Phs,
                                           const Fx2 *PhWs, const Fx2 *xs, Fx2 *zs, const Use &use) {
  using T = MassTeam<NU, NV>;
  constexpr int QH = T::QH, HP = T::HP, NE = T::NE, J = T::J, NP = (NV + 1) / 2;
  constexpr bool RISE = NV >= 4;
  const int u = team.u;
  const unsigned mask = team.mask;
  const bool high = u >= HP;                             // the mirror of a lower row
  const int low = high ? QH - 1 - u : u, mate = team.lane0 + (QH - 1 - u);
  // row u of P_h d: the thread of the lower row sums the even modes, its mirror the odd ones
  i64 Tv[NV];
  {
    Fx2 p[NP];
    const int o = high ? 1 : 0;
#pragma unroll
    for (int i = 0; i < NP; ++i) p[i] = 2 * i + o < NV ? Phs[low * NV + 2 * i + o] : Fx2{0, 0};
#pragma unroll
    for (int b = 0; b < NV; ++b) {
      i64 m = 1 << 28, h = 0;
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const Fx2 x = xs[(2 * i + o < NV ? 2 * i + o : 0) + NV * b];
        m = fx_mad(x.h, p[i].l, fx_mad(x.l, p[i].h, m));
        h = fx_mad(x.h, p[i].h, h);
      }
      const i64 t = (h << 3) + (m >> 29), q = __shfl_sync(mask, t, mate);
      Tv[b] = 2 * u + 1 == QH ? t : high ? q - t : t + q;   // (the odd modes vanish in the middle row)
    }
  }
  int nt = 0;
#pragma unroll
  for (int b = 0; b < NV; ++b) nt = max(nt, fx_hi(Tv[b]));
  nt = fx_room(nt);
  // the points of the row, weighted, and back to the modes
  i64 Z[NV];
  int nz;
  {
    Fx2 t[NV];
#pragma unroll
    for (int b = 0; b < NV; ++b) t[b] = fx_split(Tv[b] << nt);
    auto tv = [&](int b) { return t[b]; };
    i64 ys[QH / 2 + 1], yd[QH / 2 + 1];
    auto weigh = [&](i64 y0, int s2) {
      const Fx2 y = fx_split(y0), g = Gs[u + QH * s2];
      const i64 m = fx_mad(y.h, g.l, fx_mad(y.l, g.h, 1 << 28));
      return (fx_mad(y.h, g.h, 0) << 3) + (m >> 29);
    };
    int top = 0;
#pragma unroll
    for (int s2 = 0; s2 < QH / 2; ++s2) {
      auto c = [&](int b) -> const FxC & { return B.fPh[s2][b]; };
      const i64 e0 = fx_dot<0, 2, NV>(tv, c), o0 = fx_dot<1, 2, NV>(tv, c);
      const i64 p = weigh(e0 + o0, s2), m = weigh(e0 - o0, QH - 1 - s2);
      ys[s2] = p + m;
      yd[s2] = p - m;
      if constexpr (RISE) top |= fx_hi(p + m) | fx_hi(p - m);
    }
    if constexpr ((QH & 1) != 0) {
      ys[QH / 2] = weigh(fx_dot<0, 2, NV>(tv, [&](int b) -> const FxC & { return B.fPh[QH / 2][b]; }), QH / 2);
      if constexpr (RISE) top |= fx_hi(ys[QH / 2]);
    }
    const int nw = RISE ? fx_room(top) : 0;
    nt += nw;
    int hz = 0;
#pragma unroll
    for (int b = 0; b < NV; ++b) {
      auto c = [&](int s2) -> const FxC & { return B.fPhW[s2][b]; };
      if (b & 1) Z[b] = fx_dot<0, 1, QH / 2>([&](int s2) { return fx_split(yd[s2] << nw); }, c);
      else Z[b] = fx_dot<0, 1, (QH + 1) / 2>([&](int s2) { return fx_split(ys[s2] << nw); }, c);
      hz |= fx_hi(Z[b]);
    }
    // the rows' common exponent, below 2^60 for the sums of pairs
    nz = RISE ? team_min<QH>(team, nt + fx_room(hz)) - 1 : B.nrow;
#pragma unroll
    for (int b = 0; b < NV; ++b) Z[b] = fx_shift(Z[b], nz - nt);
  }
  // the sums (lower row's thread) and differences (its mirror) of the row pairs, [row NV + b] each; the
  // middle row is its own sum, and its difference is not read for anything (P_h's odd modes vanish there)
#pragma unroll
  for (int b = 0; b < NV; ++b) {
    const i64 q = __shfl_sync(mask, Z[b], mate);
    const i64 z = 2 * u + 1 == QH ? Z[b] : high ? q - Z[b] : Z[b] + q;
    zs[((high ? HP : 0) + low) * NV + b] = fx_split(z);
    if (2 * u + 1 == QH) zs[(HP + low) * NV + b] = Fx2{0, 0};
  }
  __syncwarp(mask);
  const int zsh = 2 * (61 - B.gPh) + 2 * (61 - B.gPhW) - nz, ey = RISE ? 61 + zsh : 64;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int k = u + QH * j;
    if (k < NE) {
      const int a = k % NV, b = k / NV;
      const Fx2 *z = zs + ((a & 1) ? HP * NV : 0) + b;
      i64 m = RISE ? 1 << 28 : 0, h = 0;
#pragma unroll
      for (int v = 0; v < HP; ++v) {
        const Fx2 p = PhWs[v * NV + a], y = z[v * NV];
        if constexpr (!RISE) m += fx_mad(y.l, p.l, 0) >> 32;
        m = fx_mad(y.h, p.l, fx_mad(y.l, p.h, m));
        h = fx_mad(y.h, p.h, h);
      }
      use(j, k, RISE ? (h << 3) + (m >> 29) : (h << zsh) + (m >> (32 - zsh)), ey);
    }
  }
}

// 1/D for 1 ≤ D ≤ 2 as integers of 2^-59: FP32's reciprocal and two steps of Newton's method
__device__ __forceinline__ i64 fx_recip(i64 D) {
  const float f = __uint_as_float((unsigned)(D >> 36) - (1u << 23) + (127u << 23));   // D ≥ 2^59: its top 24 bits
  i64 r = (i64)((1.0f / f) * 1073741824.0f) << 29;
  const Fx2 d = fx_split(D);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const Fx2 q = fx_split(r), t = fx_split(((i64)1 << 60) - (fx_mul(d, q) << 2));     // 2 - D r
    r = fx_mul(q, t) << 2;
  }
  return r;
}

// The start of the kernels on MassTeam: the operators' tables; the elements by count (pref[b]: those in the
// bins above b); and the thread's team, row u and slot of elements g, where threads without one return
#define WEDG_MASS_TABLES() \
  using T = MassTeam<NU, NV>; \
  constexpr int QH = T::QH, NE = T::NE, J = T::J, HP = T::HP; \
  __shared__ double sh[T::TPB * T::SLOT]; \
  __shared__ Fx2 Phf[HP * NV], PhWf[HP * NV]; \
  for (int i = threadIdx.x; i < HP * NV; i += blockDim.x) { \
    Phf[i] = Fx2{B.fPh[i / NV][i % NV].h, B.fPh[i / NV][i % NV].l}; \
    PhWf[i] = Fx2{B.fPhW[i / NV][i % NV].h, B.fPhW[i / NV][i % NV].l}; \
  } \
  after_previous();
#define WEDG_MASS_BINS() \
  __shared__ int pref[NBIN]; \
  if (F.sorted && threadIdx.x < 32) { \
    int carry = 0; \
_Pragma("unroll") \
    for (int b0 = 0; b0 < NBIN; b0 += 32) { \
      const int b = NBIN - 1 - b0 - (int)threadIdx.x, own = b >= 0 ? F.bin_count[S.parity * NBIN + b] : 0; \
      int x = own; \
_Pragma("unroll") \
      for (int o = 1; o < 32; o <<= 1) { \
        const int y = __shfl_up_sync(~0u, x, o); \
        if ((int)threadIdx.x >= o) x += y; \
      } \
      if (b >= 0) pref[b] = carry + x - own; \
      carry += __shfl_sync(~0u, x, 31); \
    } \
  }
#define WEDG_MASS_TEAM(g0) \
  __syncthreads(); \
  if (warp_stopped(F)) return; \
  const int lane = threadIdx.x & 31, tw = lane / QH; \
  if (tw >= T::TPW) return; \
  const int u = lane - tw * QH, lane0 = tw * QH, slot = (threadIdx.x >> 5) * T::TPW + tw, g = (g0) + slot; \
  if (g >= F.E) return; \
  const unsigned mask = ((1u << QH) - 1u) << lane0; \
  const Team team{mask, lane0, u}; \
  const size_t Eu = (size_t)F.E;

template <int NU, int NV>
__device__ __forceinline__ void cheb_body(const Basis<NU, NV> &B, const Fields &F, const StageIO &S, int g0) {
  WEDG_MASS_TABLES()
  WEDG_MASS_BINS()
  WEDG_MASS_TEAM(g0)
  const int e = mass_element(F, S, g, pref);
  double *xs = sh + slot * T::SLOT, *X = xs + NE, *zs = X + NE;
  const double th = F.th[e], de = F.de[e];
  const int n = F.cheb_common ? F.nmax[S.parity] : F.nst[e];
  const i64 *G = reinterpret_cast<const i64 *>(F.G) + e;
  const GPack gp(G[(size_t)QH * QH * Eu]);
  double R[J];
  int hr = 0;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int k = u + QH * j;
    R[j] = k < NE ? F.mrhs[k * Eu + e] : 0.0;
    hr = max(hr, fx_abs_hi(R[j]));
  }
  // the thread's row of G 2^ng, just below 2^60
  Fx2 *Gs = reinterpret_cast<Fx2 *>(zs + T::ZR);
  if (n > 1)
#pragma unroll
    for (int s2 = 0; s2 < QH; ++s2) Gs[u + QH * s2] = fx_split(G[(u + QH * s2) * Eu] << gp.ng);
  hr = team_max<QH>(team, hr);
  bool fin = true;
  const double ith = 1.0 / th;
  if (n == 1 || !fx_finite(hr)) {                  // (one step is R/θ)
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int k = u + QH * j;
      if (k < NE) store_v(S, e + Eu * k, n > 1 ? __longlong_as_double(0x7ff8000000000000LL) : R[j] * ith, fin);
    }
  } else {
    const int er = fx_exp(hr);
    // r in registers, X' and d in shared memory
    Fx2 *xf = reinterpret_cast<Fx2 *>(xs);
    i64 *Xf = reinterpret_cast<i64 *>(X);
    i64 rr[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int k = u + QH * j;
      rr[j] = fx_from(R[j], er);
      if (k < NE) {
        Xf[k] = rr[j];
        xf[k] = fx_split(rr[j]);
      }
    }
    __syncwarp(mask);
    // r = rr 2^-nr with room for ur bits more, d = (Xf's thread entries) 2^-nd at the top of its range, X' with
    // high words below bX
    int nr = 0, ur = 0, nX = 0, nd = 0;
    unsigned bX = (1u << 29) + 1;
    // 1/θ = (integer 2^-60) 2^(fi - 1022), the integer in [2^59, 2^60). The entries of (M/θ) d are below
    // (1 + ε) NV times the largest of d (Euclidean norms), that is below 2^LG times it
    constexpr int LG = NV <= 1 ? 1 : NV <= 2 ? 2 : NV <= 4 ? 3 : 4;
    static_assert(2 * NV <= 1 << LG, "the bound of a step");
    const int fi = (__double2hiint(ith) >> 20) & 0x7ff;
    const Fx2 ithf = fx_split(fx_from(ith, fi + 1));
    // the scalars, as integers of 2^-59: with q = ρ θ/δ the recurrence ρ' = 1/(2 θ/δ - ρ) is q' = 1/(2 - ε² q),
    // and d' = ρ'ρ d + 2 (ρ'/δ) r in the scaled system is ε² q q' d + 2 q' r
    const double eps = de * ith;
    const Fx2 e2 = fx_split(fx_scalar(eps * eps, FX_BIAS - 59));
    i64 q = (i64)1 << 59;                          // ρ = δ/θ: q = 1
#pragma unroll 1
    for (int step = 1; step < n; ++step) {
      // r -= (M/θ) d, M d = d - K d, at the exponent n1 that leaves both below 2^60. The difference, times
      // 2^(fi - 1022) for 1/θ, is below 2^61 and is taken modulo 2^64
      const int n1 = min(nr + ur, nd - LG) - 1, sd = fi - 1022 + n1 - nd, sr = n1 - nr;
      // (a half unit of bias a step would add up: r moved down goes toward -∞, and so does what is taken from it)
      const int half_p = sr < 0 ? 0 : 1 << 27;
      int hr1 = 0;
      team_K_fx<NU, NV>(B, Gs, team, Phf, PhWf, xf, reinterpret_cast<Fx2 *>(zs), [&](int j, int k, i64 y, int ey) {
        const int sy = gp.sG - gp.ng + ey + sd;
        const Fx2 t = fx_split((i64)((u64)fx_shift(fx_join(xf[k]), sd) - (u64)fx_shift(y, sy)));
        const i64 m = fx_mad(t.h, ithf.l, fx_mad(t.l, ithf.h, half_p));
        rr[j] = fx_shift(rr[j], sr) - ((fx_mad(t.h, ithf.h, 0) << 4) + (m >> 28));
        hr1 |= fx_hi(rr[j]);
      });
      const i64 eq = fx_mul(fx_split(q), e2) << 2;                       // ε² q
      q = fx_recip(((i64)1 << 60) - eq);
      const Fx2 qs = fx_split(q), c2 = fx_split(2 * q);
      const Fx2 c1 = fx_split(fx_sar(fx_mul(qs, fx_split(eq)) << 2, nd - n1));   // d's part at the exponent n1
      int hd = 0;
      i64 dd[J];
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int k = u + QH * j;
        const Fx2 d = k < NE ? xf[k] : Fx2{0, 0}, r = fx_split(rr[j]);
        const i64 m = fx_mad(d.h, c1.l, fx_mad(d.l, c1.h, fx_mad(r.h, c2.l, fx_mad(r.l, c2.h, 1 << 28))));
        dd[j] = (fx_mad(d.h, c1.h, fx_mad(r.h, c2.h, 0)) << 3) + (m >> 29);
        hd |= fx_hi(dd[j]);
      }
      // the room of both (|r| ≤ 2^61, |d'| < 2^61 at the exponent n1 - 2), as far as 14 bits, from the ors of the
      // high words' upper halves
      const unsigned w = team_or<QH>(team, (unsigned)hd >> 15 | (unsigned)hr1 >> 15 << 16);
      const int ud = max(__clz(w & 0xffff) - 18, 0);
      ur = __clz(w >> 16) - 18;
      nr = n1;
      nd = n1 - 2 + ud;
      // X' += d', to nearest
      int sX = nd - nX;
      if (sX < 0) {
#pragma unroll
        for (int j = 0; j < J; ++j)
          if (u + QH * j < NE) Xf[u + QH * j] = fx_sar(Xf[u + QH * j], -sX);
        bX = (bX >> min(-sX, 31)) + 1;
        nX = nd;
        sX = 0;
      }
      sX = min(sX, 62);
      const i64 half = ((i64)1 << sX) >> 1;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int k = u + QH * j;
        const i64 d = dd[j] << ud;
        if (k < NE) {
          xf[k] = fx_split(d);
          Xf[k] += fx_sar(d + half, sX);
        }
      }
      bX += ((1u << 29) >> min(sX, 31)) + 1;
      if (bX > 0x50000000u) {                      // the next d' may not fit: the actual size, and down by one if needed
        int hX = 0;
#pragma unroll
        for (int j = 0; j < J; ++j)
          if (u + QH * j < NE) hX = max(hX, fx_hi(Xf[u + QH * j]));
        bX = team_max<QH>(team, hX) + 1;
        if (bX > 1u << 29) {
#pragma unroll
          for (int j = 0; j < J; ++j)
            if (u + QH * j < NE) Xf[u + QH * j] >>= 1;
          bX = (bX >> 1) + 1;
          --nX;
        }
      }
      __syncwarp(mask);
    }
    // X = X' / θ; in two factors where 2^kk or the product of both is beyond the normal numbers
    const int kk = er - FX_BIAS - nX, ei = fi - 1023;
    const bool wide = kk > 1023 || abs(kk + ei) > 1000;
    const double sc = wide ? fx_pow2(-ei) * ith : fx_pow2(kk) * ith;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int k = u + QH * j;
      if (k < NE) {
        double x = __dmul_rn((double)Xf[k], sc);
        if (wide) x = ldexp(x, kk + ei);
        store_v(S, e + Eu * k, x, fin);
      }
    }
  }
  if (S.mode == OUT_RK4_LAST && !fin) atomicOr(F.nonfinite, 1u);
}

// Σ over the team's W threads of x, on every one of them: the same tree for each
template <int W>
__device__ __forceinline__ double team_sum(double x, int u, int lane0, unsigned mask) {
  constexpr int top = W > 8 ? 8 : W > 4 ? 4 : W > 2 ? 2 : 1;
#pragma unroll
  for (int o = top; o > 0; o >>= 1) {
    const double y = __shfl_sync(mask, x, lane0 + (u + o < W ? u + o : u));
    if (u < o && u + o < W) x += y;
  }
  return __shfl_sync(mask, x, lane0);
}

// k_cg: the mass solve by conjugate gradients from X = R (src/rhs.jl:821-853), elements in mesh order, on the
// team layout of k_cheb: the products with K in fixed point on p as integers of its own exponent, the
// vectors and inner products in FP64, summed over the team's lanes in a fixed order so that every lane
// takes the same decisions. A chain of products and reductions bounds it, with three blocks an SM to hide
// it. N = 97, q = 5: 405 us with FP64 products of half as many threads, 137 us so (and 11 us for the integers
// of G, which k_prep writes).
template <int NU, int NV>
__device__ __forceinline__ void cg_body(const Basis<NU, NV> &B, const Fields &F, const StageIO &S, int g0) {
  WEDG_MASS_TABLES()
  WEDG_MASS_TEAM(g0)
  const int e = g;
  double *xs = sh + slot * T::SLOT, *zs = xs + 2 * NE;
  Fx2 *xf = reinterpret_cast<Fx2 *>(xs), *Gs = reinterpret_cast<Fx2 *>(zs + T::ZR);
  const i64 *G = reinterpret_cast<const i64 *>(F.G) + e;
  const GPack gp(G[(size_t)QH * QH * Eu]);
  const bool g_ok = gp.sG != GPack::BAD;
#pragma unroll
  for (int s2 = 0; s2 < QH; ++s2) Gs[u + QH * s2] = fx_split(g_ok ? G[(u + QH * s2) * Eu] << gp.ng : 0);
  // y = K x for the threads' entries x[j]; NaN where x or G is not finite
  auto K = [&](const double (&x)[J], double (&y)[J]) {
    int hx = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) hx = max(hx, fx_abs_hi(x[j]));
    hx = team_max<QH>(team, hx);
    const int ex = fx_exp(hx);
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int k = u + QH * j;
      if (k < NE) xf[k] = fx_split(fx_from(x[j], ex));
      y[j] = 0.0;
    }
    __syncwarp(mask);
    const double one = g_ok && fx_finite(hx) ? 1.0 : __longlong_as_double(0x7ff8000000000000LL);
    const int k0 = ex - FX_BIAS + (g_ok ? gp.sG - gp.ng : 0);
    team_K_fx<NU, NV>(B, Gs, team, Phf, PhWf, xf, reinterpret_cast<Fx2 *>(zs),
                      [&](int j, int, i64 v, int ey) { y[j] = fx_scale((double)v * one, k0 + ey); });
    __syncwarp(mask);
  };
  double X[J], r[J], p[J], Ap[J];
  double r0 = 0;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int k = u + QH * j;
    X[j] = k < NE ? F.mrhs[k * Eu + e] : 0.0;
    r0 = fma(X[j], X[j], r0);
  }
  r0 = sqrt(team_sum<QH>(r0, u, lane0, mask));
  K(X, r);                                               // r = R - M X = K R for X = R
  double rr = 0;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    p[j] = r[j];
    rr = fma(r[j], r[j], rr);
  }
  rr = team_sum<QH>(rr, u, lane0, mask);
  const int maxit = NV * NV + 10;
  int it = 0;
  bool bad = false;
  while (sqrt(rr) > F.mass_tol * r0 && it < maxit) {
    ++it;
    K(p, Ap);
    double pAp = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      Ap[j] = __dsub_rn(p[j], Ap[j]);                    // A p = p - K p
      pAp = fma(p[j], Ap[j], pAp);
    }
    pAp = team_sum<QH>(pAp, u, lane0, mask);
    if (!(pAp > 0.0)) { bad = true; break; }
    const double al = rr / pAp;
    double rrn = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      X[j] = fma(al, p[j], X[j]);
      r[j] = fma(-al, Ap[j], r[j]);
      rrn = fma(r[j], r[j], rrn);
    }
    rrn = team_sum<QH>(rrn, u, lane0, mask);
    const double bt = rrn / rr;
#pragma unroll
    for (int j = 0; j < J; ++j) p[j] = fma(bt, p[j], r[j]);
    rr = rrn;
  }
  if (bad) {
    if (u == 0) atomicMin(F.err, (1ull << ERR_CLASS_SHIFT) | (unsigned long long)(e + 1));
    return;
  }
  if (u == 0 && sqrt(rr) > F.mass_tol * r0) atomicAdd(F.cg_nfail, 1u);

  bool fin = true;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int k = u + QH * j;
    if (k < NE) store_v(S, e + Eu * k, X[j], fin);
  }
  if (S.mode == OUT_RK4_LAST && !fin) atomicOr(F.nonfinite, 1u);
}

// Blocks per SM asked of the mass solves. k_cheb: five from n_v = 6 on, where six (80 registers) spill 92 bytes a
// thread and more (a stage's solves at N = 512, q = 6: 935 us at six, 888 at five; N = 300, q = 7 4 690 and 4 636 us), and
// six below (n_v = 5, N = 256: 132 and 138 us; n_v = 3, N = 333: 314 and 322 us). k_cg: three
__host__ __device__ constexpr int mass_blocks(int nv, bool cg) { return cg ? 3 : nv >= 6 ? 5 : 6; }

template <int NU, int NV>
__global__ void __launch_bounds__(CHEB_THREADS, mass_blocks(NV, false))
    k_cheb(const __grid_constant__ Basis<NU, NV> B, const __grid_constant__ Fields F,
           const __grid_constant__ StageIO S) {
  cheb_body<NU, NV>(B, F, S, blockIdx.x * mass_tile(NU, NV, blockDim.x));
}

template <int NU, int NV>
__global__ void __launch_bounds__(CHEB_THREADS, mass_blocks(NV, true))
    k_cg(const __grid_constant__ Basis<NU, NV> B, const __grid_constant__ Fields F,
         const __grid_constant__ StageIO S) {
  cg_body<NU, NV>(B, F, S, blockIdx.x * mass_tile(NU, NV, blockDim.x));
}

// tile = mass_tile elements per virtual block; CG selects k_cg's body
template <int NU, int NV, bool CG>
__global__ void __launch_bounds__(CHEB_THREADS, mass_blocks(NV, CG))
    k_mass_m(const __grid_constant__ Basis<NU, NV> B, const __grid_constant__ MultiStage P) {
  for (int vb = blockIdx.x; vb < P.first[P.n]; vb += gridDim.x) {
    const int inst = multi_begin(P, vb);
    const int g0 = (vb - P.first[inst]) * P.tile;
    if constexpr (CG) cg_body<NU, NV>(B, P.a[inst].F, P.a[inst].S, g0);
    else cheb_body<NU, NV>(B, P.a[inst].F, P.a[inst].S, g0);
  }
}

// Last RK4 update when the last stage may still raise an error inside k_cg
// (CG mode): u += (dt/6) acc unless an error was recorded.
__global__ void k_rk4_final(int n_u, int n_v, double *u, double *v, const double *accu, const double *accv,
                            double c, const unsigned long long *err, unsigned int *nonfinite);

// Device-side step bookkeeping after each RK4 step: counts completed steps and,
// when asked, stops the run after a non-finite result.
__global__ void k_step_done(unsigned long long *err, const unsigned int *nonfinite, int stop_nonfinite,
                            long long *steps_done);

}  // namespace wedg

#include "wedg_adjoint.cuh"

