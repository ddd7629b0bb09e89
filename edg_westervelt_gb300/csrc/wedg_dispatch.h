// Dispatch of the size-templated kernels of libwedg. Each q_u = NU - 1 is
// compiled in its own translation unit (wedg_qN.cu) so that the build runs in
// parallel; this header is the interface between them and wedg_api.cu.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <mutex>
#include <type_traits>

#include "wedg_kernels.cuh"

namespace wedg {

constexpr int MAXN = 8;    // q_u ≤ 7
constexpr int MAXQH = 12;  // q_high for q_v = 7
constexpr int MAX_DEVICES = 64;

// Runtime-sized copy of the 1D operators, packed into Basis<NU, NV> per launch.
struct BasisHost {
  int nu, nv, qh;
  double w[MAXN], P[MAXN][MAXN], S[MAXN][MAXN];
  double Pw[MAXN][MAXN];
  double El[MAXN], Er[MAXN], E1l[MAXN], E1r[MAXN];
  double E1F[MAXN];
  double Ph[MAXQH][MAXN], Wh[MAXQH][MAXQH], wh[MAXQH], PhW[MAXQH][MAXN];
  double K1[MAXN][MAXN], Q[MAXN][MAXN], ilam2[MAXN][MAXN];
};

// A launcher enqueues one kernel; it returns an error only when it could not launch (a launch
// error itself is left to the caller's cudaGetLastError)
typedef cudaError_t (*launch_fn)(const void *basis, const Fields &F, const StageIO &S, int blocks, int threads,
                                 cudaStream_t st);
typedef void (*pack_fn)(const BasisHost &h, void *out);

typedef void (*adj_fn)(const void *basis, const Fields &F, const StageIO &S, const AdjIO &A, cudaStream_t st);

// k_adj_face; with gc2 (and gal, gbe) non-null also the coefficient derivatives
typedef void (*adj_face_fn)(const void *basis, const Fields &F, const StageIO &S, const AdjIO &A, double *gc2,
                            double *gal, double *gbe, cudaStream_t st);

// Multi-instance launches (wedg_kernels.cuh): `grid` blocks (0: one per virtual block) of
// `threads` threads; the caller sets P.tile to the kernel's elements per block (k_prep: prep_tile,
// k_bnd: bnd_tile sides, k_stage: stage_tile, the mass solves: (threads / 32) teams per warp)
typedef cudaError_t (*multi_fn)(const void *basis, const MultiStage &P, int grid, int threads,
                                cudaStream_t st);
typedef cudaError_t (*multi_adj_fn)(const void *basis, const MultiAdj &P, int grid, cudaStream_t st);
enum { MK_PREP = 0, MK_BND = 1, MK_STAGE = 2, MK_MASS = 3 };
// Blocks of `threads` threads of a multi-instance kernel that an SM of the current device holds at once
typedef int (*resident_fn)(int kind, int threads, bool cg);

// k_prep over the elements [e0, e0 + blocks × prep_tile) (clipped to the mesh)
typedef cudaError_t (*prep_fn)(const void *basis, const Fields &F, const StageIO &S, int blocks, int threads,
                               cudaStream_t st, int e0);

struct Launchers {
  prep_fn prep = nullptr;
  launch_fn bnd = nullptr, stage = nullptr, mass = nullptr;
  adj_fn adj_hats = nullptr, adj_mass = nullptr;
  adj_face_fn adj_face = nullptr;
  multi_fn prep_m = nullptr, bnd_m = nullptr, stage_m = nullptr, mass_m = nullptr;
  resident_fn resident = nullptr;
  multi_adj_fn adj_hats_m = nullptr, adj_mass_m = nullptr, adj_face_m = nullptr;
  pack_fn pack = nullptr;
  size_t basis_size = 0;
};

static_assert(sizeof(MultiStage) + sizeof(Basis<MAXN, MAXN>) <= 32764 &&
                  sizeof(MultiAdj) + sizeof(Basis<MAXN, MAXN>) <= 32764,
              "the arguments of a multi-instance launch exceed the kernel parameter limit");

inline int multi_grid(int grid, int total) { return grid > 0 && grid < total ? grid : total; }

template <int NU, int NV>
const Basis<NU, NV> &basis_of(const void *basis) {
  return *static_cast<const Basis<NU, NV> *>(basis);
}

// Launches k after the kernel before it on the stream. With `early` the launch itself is already under way while that
// kernel runs, and k's threads wait for its end on the device (after_previous), which saves most of the gap between
// two kernels, at every size: two RK4 steps at q = 2 and 6, N = 364 2 198 -> 2 141 and 9 360 -> 9 300 us, N = 512 3 950
// -> 3 895 and 17 720 -> 17 662 us; N = 32 2.71 -> 2.40 ms and N = 64 25.1 -> 22.9 ms for their runs. The kernels of
// several instances, which fill the chip, gained nothing.
// (Letting k's blocks onto the SMs as well, before the kernel before it has ended, was better at N = 32 alone:
// they spread unevenly over the SMs that happen to have room; N = 128 adjoint 4 % slower.)
template <class... P, class... A>
cudaError_t launch_after(void (*k)(P...), bool early, int grid, int threads, cudaStream_t st, const A &...a) {
  static_assert((std::is_same<P, A>::value && ...), "the arguments are passed by address");
  void *args[] = {const_cast<void *>(static_cast<const void *>(&a))...};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(threads);
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelExC(&c, reinterpret_cast<const void *>(k), args);
}

template <int NU, int NV>
void pack_basis(const BasisHost &h, void *out) {
  Basis<NU, NV> &b = *static_cast<Basis<NU, NV> *>(out);
  constexpr int NQ = NU, QH = Basis<NU, NV>::QH;
  for (int i = 0; i < NQ; ++i) {
    b.w[i] = h.w[i];
    for (int d = 0; d < NU; ++d) { b.P[i][d] = h.P[i][d]; b.S[i][d] = h.S[i][d]; b.Pw[i][d] = h.Pw[i][d]; }
  }
  for (int d = 0; d < NU; ++d) {
    b.El[d] = h.El[d]; b.E1l[d] = h.E1l[d];
    b.E1F[d] = h.E1F[d];
    for (int c = 0; c < NU; ++c) { b.K1[d][c] = h.K1[d][c]; }
  }
  for (int r = 0; r < QH; ++r) {
    b.wh[r] = h.wh[r];
    for (int d = 0; d < NV; ++d) { b.Ph[r][d] = h.Ph[r][d]; b.PhW[r][d] = h.PhW[r][d]; }
  }
  // fixed-point forms: Ph is contracted over its modes (row sums), PhW over its points (column sums)
  auto big = [](double &m, double x) { m = x > m ? x : m; };
  double sP = 0, bP = 0, sW = 0, bW = 0;
  for (int r = 0; r < QH; ++r) {
    double s = 0;
    for (int d = 0; d < NV; ++d) { s += fabs(b.Ph[r][d]); big(bP, fabs(b.Ph[r][d])); big(bW, fabs(b.PhW[r][d])); }
    big(sP, s);
  }
  for (int d = 0; d < NV; ++d) {
    double s = 0;
    for (int r = 0; r < QH; ++r) s += fabs(b.PhW[r][d]);
    big(sW, s);
  }
  b.gPh = fx_exponent(sP, bP);
  b.gPhW = fx_exponent(sW, bW);
  for (int d = 0; d < NV; ++d) {
    double c = 0;
    for (int r = 0; r < QH; ++r) big(c, fabs(b.Ph[r][d]));
    b.cPh[d] = (int)ceil(ldexp(c, 8));
  }
  {
    // rows of the grid of K d stay below max|G| |d| max_r |Ph[r]| (Euclidean norms)
    double c = 0;
    for (int r = 0; r < QH; ++r) {
      double s = 0;
      for (int d = 0; d < NV; ++d) s += b.Ph[r][d] * b.Ph[r][d];
      big(c, sqrt(s));
    }
    int lg;
    frexp(NV * c, &lg);
    const int up = 2 * (61 - b.gPh) + (61 - b.gPhW) - lg;
    b.nrow = up > 0 ? up : 0;
  }
  // the constant-coefficient kernels' operators: the end values two to a sum (A and D of a side), K1
  // by its rows (columns in one sum with them), Q by rows or columns beside the constant mode
  double eL = 0, e1 = 0, sK = 0, bK = 0, sQ = 0, bQ = 0, bL = 0, bE = 0;
  double QE[NU];
  for (int i = 0; i < NU; ++i) {
    big(eL, fabs(h.El[i]));
    big(e1, fabs(h.E1l[i]));
    double k = 0, r = 0, c = 0;
    QE[i] = 0;
    for (int a = 0; a < NU; ++a) {
      QE[i] += h.Q[a][i] * h.E1F[a];
      k += fabs(ldexp(h.K1[i][a], -k1_bits<NU>(a)));
      big(bK, fabs(ldexp(h.K1[i][a], -k1_bits<NU>(a))));
      if (i == 0 || a == 0) continue;
      r += fabs(h.Q[i][a]);
      c += fabs(h.Q[a][i]);
      big(bQ, fabs(h.Q[i][a]));
    }
    big(sK, 2 * k);
    big(sQ, r);
    big(sQ, c);
    for (int a = 0; a < NU; ++a)
      if (i + a > 0) big(bL, fabs(h.ilam2[i][a]));
  }
  for (int i = 0; i < NU; ++i)
    for (int a = 0; a < NU; ++a)
      if (i + a > 0) big(bE, fabs(QE[i] * h.ilam2[i][a]));
  b.gEl = fx_exponent(2 * eL, eL);
  b.gE1 = fx_exponent(2 * e1, e1);
  b.gK1 = fx_exponent(sK, bK);
  b.gQ = fx_exponent(sQ, bQ);
  b.gL = fx_exponent(bL, bL);
  b.gM = fx_exponent(2 * bE, bE);
  for (int i = 0; i < NU; ++i) {
    b.fEl[i] = fx_const(h.El[i], b.gEl);
    b.fE1[i] = fx_const(h.E1l[i], b.gE1);
    b.kK1[i] = k1_bits<NU>(i);
    for (int a = 0; a < NU; ++a) {
      b.fK1[i][a] = fx_const(ldexp(h.K1[i][a], -k1_bits<NU>(a)), b.gK1);
      b.fQ[i][a] = fx_const(i == 0 || a == 0 ? 0.0 : h.Q[i][a], b.gQ);
      b.fL[i][a] = fx_const(i + a == 0 ? 0.0 : h.ilam2[i][a], b.gL);
      b.fM[i][a][0] = fx_const(i + a == 0 ? 0.0L : (long double)QE[i] * h.ilam2[i][a], b.gM);
      b.fM[i][a][1] = fx_const(i + a == 0 ? 0.0L : (long double)QE[a] * h.ilam2[i][a], b.gM);
    }
  }
  for (int r = 0; r < QH; ++r)
    for (int d = 0; d < NV; ++d) {
      b.fPh[r][d] = fx_const(b.Ph[r][d], b.gPh);
      b.fPhW[r][d] = fx_const(b.PhW[r][d], b.gPhW);
    }
}

template <int NU, int NV>
cudaError_t launch_prep(const void *basis, const Fields &F, const StageIO &S, int blocks, int threads,
                        cudaStream_t st, int e0) {
  // (ranges of elements also wait for their copies to the device, and are launched after those)
  const bool all = blocks * prep_tile(NU, threads) >= F.E;
  const int sides = (threads / 32) * bnd_tile(NU), nb = all ? (4 * F.N + sides - 1) / sides : 0;
  return launch_after(k_prep<NU, NV>, all, nb + blocks, threads, st, basis_of<NU, NV>(basis), F, S,
                      e0, nb);
}

// k_bnd over the 4N physical sides (the grid follows from F.N), after a k_prep by ranges
template <int NU, int NV>
cudaError_t launch_bnd(const void *basis, const Fields &F, const StageIO &S, int, int, cudaStream_t st) {
  return launch_after(k_bnd<NU, NV>, true, (4 * F.N + bnd_tile(NU) - 1) / bnd_tile(NU), BND_THREADS, st,
                      basis_of<NU, NV>(basis), F, S);
}

// k_stage: `blocks` blocks of STAGE_THREADS, stage_tile elements each
template <int NU, int NV, bool FAST>
cudaError_t launch_stage(const void *basis, const Fields &F, const StageIO &S, int blocks, int threads,
                         cudaStream_t st) {
  if (blocks <= 0) return cudaSuccess;
  return launch_after(k_stage<NU, NV, FAST>, true, blocks, threads, st, basis_of<NU, NV>(basis), F, S);
}

// The mass solve: k_cheb or k_cg, a team of threads per element (static shared memory sized
// for CHEB_THREADS). `threads` (32, 64, 96 or 128) sets the warps of a block and with them its
// elements; the grid follows from F.E, `blocks` only says whether to launch.
template <int NU, int NV>
cudaError_t launch_mass(const void *basis, const Fields &F, const StageIO &S, int blocks, int threads,
                        cudaStream_t st) {
  if (blocks <= 0) return cudaSuccess;
  const Basis<NU, NV> &B = *static_cast<const Basis<NU, NV> *>(basis);
  threads = (threads >= 32 && threads <= CHEB_THREADS && threads % 32 == 0) ? threads : CHEB_THREADS;
  const int tpb = mass_tile(NU, NV, threads);
  const int grid = (F.E + tpb - 1) / tpb;
  if (F.cg) return launch_after(k_cg<NU, NV>, true, grid, threads, st, B, F, S);
  return launch_after(k_cheb<NU, NV>, true, grid, threads, st, B, F, S);
}

// The adjoint kernels (wedg_adjoint.cuh)
template <int NU, int NV>
void launch_adj_hats(const void *basis, const Fields &F, const StageIO &, const AdjIO &A, cudaStream_t st) {
  launch_after(k_adj_hats<NU, NV>, true, (F.E + HATS_THREADS - 1) / HATS_THREADS, HATS_THREADS, st,
               basis_of<NU, NV>(basis), F, A);
}
template <int NU, int NV>
void launch_adj_mass(const void *basis, const Fields &F, const StageIO &, const AdjIO &A, cudaStream_t st) {
  constexpr int tpb = mass_tile(NU, NV, CHEB_THREADS);
  launch_after(k_adj_mass<NU, NV>, true, (F.E + tpb - 1) / tpb, CHEB_THREADS, st, basis_of<NU, NV>(basis), F, A);
}
template <int NU, int NV>
void launch_adj_face(const void *basis, const Fields &F, const StageIO &S, const AdjIO &A, double *gc2, double *gal,
                     double *gbe, cudaStream_t st) {
  const Basis<NU, NV> &B = *static_cast<const Basis<NU, NV> *>(basis);
  const int grid = (F.E + adj_tile(NU) - 1) / adj_tile(NU);
  if (gc2) launch_after(k_adj_face<NU, NV, true>, true, grid, ADJ_THREADS, st, B, F, S, A, gc2, gal, gbe);
  else launch_after(k_adj_face<NU, NV, false>, true, grid, ADJ_THREADS, st, B, F, S, A, gc2, gal, gbe);
}

template <int NU, int NV>
cudaError_t launch_prep_m(const void *basis, const MultiStage &P, int grid, int threads, cudaStream_t st) {
  const int total = P.first[P.n];
  if (total <= 0) return cudaSuccess;
  k_prep_m<NU, NV><<<multi_grid(grid, total), threads, 0, st>>>(*static_cast<const Basis<NU, NV> *>(basis), P);
  return cudaSuccess;
}

template <int NU, int NV>
cudaError_t launch_bnd_m(const void *basis, const MultiStage &P, int grid, int, cudaStream_t st) {
  const int total = P.first[P.n];
  if (total <= 0) return cudaSuccess;
  k_bnd_m<NU, NV><<<multi_grid(grid, total), BND_THREADS, 0, st>>>(*static_cast<const Basis<NU, NV> *>(basis), P);
  return cudaSuccess;
}

template <int NU, int NV, bool FAST>
cudaError_t launch_stage_m(const void *basis, const MultiStage &P, int grid, int, cudaStream_t st) {
  const int total = P.first[P.n];
  if (total <= 0) return cudaSuccess;
  k_stage_m<NU, NV, FAST><<<multi_grid(grid, total), STAGE_THREADS, 0, st>>>(
      *static_cast<const Basis<NU, NV> *>(basis), P);
  return cudaSuccess;
}

template <int NU, int NV>
cudaError_t launch_mass_m(const void *basis, const MultiStage &P, int grid, int threads, cudaStream_t st) {
  const int total = P.first[P.n];
  if (total <= 0) return cudaSuccess;
  const Basis<NU, NV> &B = *static_cast<const Basis<NU, NV> *>(basis);
  if (P.a[0].F.cg) k_mass_m<NU, NV, true><<<multi_grid(grid, total), threads, 0, st>>>(B, P);
  else k_mass_m<NU, NV, false><<<multi_grid(grid, total), threads, 0, st>>>(B, P);
  return cudaSuccess;
}

template <int NU, int NV, bool FAST>
int resident_m(int kind, int threads, bool cg) {
  const void *k = kind == MK_PREP    ? (const void *)k_prep_m<NU, NV>
                  : kind == MK_BND   ? (const void *)k_bnd_m<NU, NV>
                  : kind == MK_STAGE ? (const void *)k_stage_m<NU, NV, FAST>
                  : cg               ? (const void *)k_mass_m<NU, NV, true>
                                     : (const void *)k_mass_m<NU, NV, false>;
  int n = 0;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, 0) == cudaSuccess && n > 0 ? n : 1;
}

template <int NU, int NV>
cudaError_t launch_adj_hats_m(const void *basis, const MultiAdj &P, int grid, cudaStream_t st) {
  const int total = P.first[P.n];
  if (total <= 0) return cudaSuccess;
  k_adj_hats_m<NU, NV><<<multi_grid(grid, total), HATS_THREADS, 0, st>>>(*static_cast<const Basis<NU, NV> *>(basis),
                                                                         P);
  return cudaSuccess;
}

template <int NU, int NV>
cudaError_t launch_adj_mass_m(const void *basis, const MultiAdj &P, int grid, cudaStream_t st) {
  const int total = P.first[P.n];
  if (total <= 0) return cudaSuccess;
  k_adj_mass_m<NU, NV><<<multi_grid(grid, total), CHEB_THREADS, 0, st>>>(*static_cast<const Basis<NU, NV> *>(basis),
                                                                          P);
  return cudaSuccess;
}

// PARAMS when the instances pass coefficient gradients (all or none of them)
template <int NU, int NV>
cudaError_t launch_adj_face_m(const void *basis, const MultiAdj &P, int grid, cudaStream_t st) {
  const int total = P.first[P.n];
  if (total <= 0) return cudaSuccess;
  const Basis<NU, NV> &B = *static_cast<const Basis<NU, NV> *>(basis);
  if (P.a[0].gc2) k_adj_face_m<NU, NV, true><<<multi_grid(grid, total), ADJ_THREADS, 0, st>>>(B, P);
  else k_adj_face_m<NU, NV, false><<<multi_grid(grid, total), ADJ_THREADS, 0, st>>>(B, P);
  return cudaSuccess;
}

template <int NU, int NV>
Launchers make_launchers(bool fast) {
  Launchers L;
  L.prep_m = launch_prep_m<NU, NV>;
  L.bnd_m = launch_bnd_m<NU, NV>;
  L.stage_m = fast ? launch_stage_m<NU, NV, true> : launch_stage_m<NU, NV, false>;
  L.mass_m = launch_mass_m<NU, NV>;
  L.resident = fast ? resident_m<NU, NV, true> : resident_m<NU, NV, false>;
  L.adj_hats_m = launch_adj_hats_m<NU, NV>;
  L.adj_mass_m = launch_adj_mass_m<NU, NV>;
  L.adj_face_m = launch_adj_face_m<NU, NV>;
  L.adj_hats = launch_adj_hats<NU, NV>;
  L.adj_mass = launch_adj_mass<NU, NV>;
  L.adj_face = launch_adj_face<NU, NV>;
  L.prep = launch_prep<NU, NV>;
  L.bnd = launch_bnd<NU, NV>;
  L.mass = launch_mass<NU, NV>;
  L.stage = fast ? launch_stage<NU, NV, true> : launch_stage<NU, NV, false>;
  L.pack = pack_basis<NU, NV>;
  L.basis_size = sizeof(Basis<NU, NV>);
  return L;
}

// defined in wedg_q1.cu ... wedg_q7.cu (NU = q_u + 1)
Launchers launchers_q1(int nv, bool fast);
Launchers launchers_q2(int nv, bool fast);
Launchers launchers_q3(int nv, bool fast);
Launchers launchers_q4(int nv, bool fast);
Launchers launchers_q5(int nv, bool fast);
Launchers launchers_q6(int nv, bool fast);
Launchers launchers_q7(int nv, bool fast);

}  // namespace wedg
