// k_stage for elements with constant c² and α (the constant-coefficient kernels): fluxes and lifts,
// volume terms, source and u-equation of an element by a team of NU threads, with every contraction
// over modes in fixed point (wedg_fixed.cuh) and the flux slots, sources and RK4 updates in FP64.
// Thread c of a team takes mode c along the faces, and column or row c of the modal blocks, whichever
// the product at hand leaves on its own; the blocks change hands through shared memory.
//
// What bounds it: as FP64 code with a thread per element these kernels spent about 2 150 FP64
// operations per element at q = 6 and ran the FP64 pipe at 60-70 %. Here the stiffness products (252
// multiply-adds), the lifts (294 + 76) and the u-solve (608) are integer work beside the FP64 pipe,
// which keeps about 700 operations: the slots, one conversion per output and the updates. The team
// keeps the registers low enough for 24 warps an SM and spreads small meshes over the chip.
// N = 512, q = 6: 1 499 us as FP64 code with a thread per element, 1 108 us in fixed point so, 844 us by teams at
// six blocks an SM (980 and 878 at four and five), 852 us with the room taken back in the u-solve; N = 64, q = 4: 87
// and 26 us.
//
// With Cw = c²W, Aw = αW, the 1D stiffness K1 = S^T diag(w) S and the orthonormal basis
//   (c²∇φ_v,∇u_h) + (α∇φ_v,∇v_h) = (K1 W + W K1)[v-block] / (-4/h²),  W = -(4/h²)(c² U + α V),
// and A_e = c² (K1 ⊗ I + I ⊗ K1) + e_0 e_0^T is diagonal in the eigenbasis Q ⊗ Q of K1 (e_0 first,
// λ_0 = 0; the constant mode passes unchanged). K1 and Q couple only modes of equal parity. The
// u-equation's volume part c²(K1 V + V K1), taken to the eigenbasis and divided by c²(λ_i + λ_j), is
// Q^T V Q itself, so UT = Q [Q^T V Q + L ∘ b~] Q^T, L = 1/(λ_i + λ_j) and b~ the lifts of the slots
// F/c² in the eigenbasis: rank-one terms per side, never stored as a block, whose factors M =
// QE[i] L[i][j] (QE = Q^T E1F) are one constant per entry and axis.
#pragma once

namespace wedg {

// 2^k as the unit of integers that become doubles (k outside the normal range only where the
// numbers are)
__device__ __forceinline__ double fx_unit(int k) { return fx_pow2(min(max(k, -1022), 1023)); }

// x 2^-n to nearest (n ≥ 0)
__device__ __forceinline__ i64 fx_down(i64 x, int n) {
  n = min(n, 62);
  return n ? (x + ((i64)1 << (n - 1))) >> n : x;
}

// The size of the entries of K1's column c, as a power of two: K1 is used as fK1 = K1[a][c] 2^-k_c with
// the mode c of the other factor taken 2^k_c times, so that the sums' exponent follows the modes
// that are large (smooth states: the low ones) and not K1's largest entry. K1[a][c] =
// √((2a+1)(2c+1)) m(m+1)/2, m = min(a, c), for modes of equal parity.
template <int NU>
__host__ __device__ constexpr int k1_bits(int c) {
  int k = 0;
  for (int a = 1; a < NU; ++a) {
    if ((a + c) & 1) continue;
    const int m = a < c ? a : c;
    const int n = (2 * a + 1) * (2 * c + 1) * m * m * (m + 1) * (m + 1);   // 4 K1²
    while ((4LL << (2 * k)) < n) ++k;
  }
  return k;
}

template <int NU, int NV>
struct FastTeam {
  static constexpr int TPW = 32 / NU;                    // teams (elements) per warp
  static constexpr int TPB = TPW * (STAGE_THREADS / 32); // elements per block
  static constexpr int X = NU * NU > 12 * NU ? NU * NU : 12 * NU;   // a block (or the slots at the points)
  static constexpr int SLOT = (X + 10 * NU + 40) | 1;    // and vectors along the faces; odd: bank conflicts
};

// The factors of an interior face's slots (the face coefficients are one value along the face), so that
// with q∓ = (2/h)(c² du + α dv) of the "-" and "+" element and s = v⁻ - v⁺ (interior_flux), mode by mode,
//   "+": A = pen s - (1-θ) q⁻ - θ q⁺ - (1-θ) K,  w = θ s - τ (q⁻ - q⁺ + K),       D = -α⁺ w, F = c²⁺ w
//   "-": A = -pen s + (1-θ) q⁻ + θ q⁺ - θ K,     w = -(1-θ) s - τ (q⁻ - q⁺ + K),  D = α⁻ w,  F = -c²⁻ w
// with A times 2/h, D times 4/h² and F over c². (The slots' projections are the same combinations of
// the traces' modes as their point values are of the traces: the face rule integrates the product of
// two modes exactly.)
struct FaceFactors {
  double um, vm, up, vp, pen, am, ap, ak, dD, dF;
};
__device__ __forceinline__ size_t face_index(int N, int s, int j, int k) {
  return s < 2 ? (s == 0 ? j : j + 1) + (size_t)(N + 1) * k : j + (size_t)N * (s == 2 ? k : k + 1);
}
template <int NU>
__device__ __forceinline__ FaceFactors face_factors(const Fields &F, int s, int j, int k, double ic2) {
  const size_t fi = face_index(F.N, s, j, k);              // point 0 of the face
  const FaceCoef cf = s < 2 ? face_coef(F, F.hc2, F.haf, F.hc2m, F.hafm, F.hJC, fi)
                            : face_coef(F, F.vc2, F.vaf, F.vc2m, F.vafm, F.vJC, fi);
  const bool plus = (s == 0 || s == 2);
  const double th = F.theta, two_h = F.two_h, sg = plus ? 1.0 : -1.0;
  const double c2m = F.one_sided ? cf.c2m : cf.c2p, afm = F.one_sided ? cf.afm : cf.afp;
  const double c2p = cf.c2p, afp = cf.afp;
  FaceFactors f;
  if (NU == 2 && !F.one_sided) {
    // a continuous face has one value of c² and α: fewer operations, where the factors serve two modes and are a quarter of
    // k_stage's FP64 work (N = 1024, q_u = 1: 554 and 510 us)
    f.um = f.up = two_h * c2p; f.vm = f.vp = two_h * afp;
    f.pen = (c2p * F.lu + afp * F.lv) * (plus ? two_h : -two_h);
    const double t = th * two_h, o = (1.0 - th) * two_h;
    f.am = plus ? -o : o; f.ap = plus ? -t : t;
    f.ak = plus ? -o : -t;
    f.dD = (plus ? -afp : afm) * F.four_hh; f.dF = (plus ? c2p : -c2m) * ic2;
    return f;
  }
  f.um = two_h * c2m; f.vm = two_h * afm; f.up = two_h * c2p; f.vp = two_h * afp;
  f.pen = ((0.5 * (c2m + c2p)) * F.lu + (0.5 * (afm + afp)) * F.lv) * sg * two_h;
  f.am = -(1.0 - th) * sg * two_h; f.ap = -th * sg * two_h;
  f.ak = (plus ? -(1.0 - th) : -th) * two_h;
  f.dD = (plus ? -afp : afm) * F.four_hh; f.dF = (plus ? c2p : -c2m) * ic2;
  return f;
}

// Mode b of the projected slots of interior side s
template <int NU, int NV>
__device__ __forceinline__ void interior_slot(const Fields &F, const FaceFactors &f, int s, int j, int k, int e, int b,
                                              double &ya, double &yd, double &yf) {
  constexpr int NQ = NU;
  const int N = F.N;
  const size_t E = F.E;
  const bool plus = (s == 0 || s == 2);
  const int nb = s == 0 ? e - 1 : s == 1 ? e + 1 : s == 2 ? e - N : e + N;
  const int sm = s < 2 ? 1 : 3, spp = s < 2 ? 0 : 2;      // trace sides of the "-" and "+" elements
  const int em = plus ? nb : e, ep = plus ? e : nb;
  const double *jcm = s < 2 ? F.hJCm : F.vJCm;
  const double th = F.theta, tau = F.tau;
  const bool minus_side = th != 1.0 || tau != 0.0;        // else q⁻ has no part in this face
  auto T = [&](int fam, int side, int el) { return F.tr[((fam * 4 + side) * NQ + b) * E + el]; };
  double qp = f.up * T(0, spp, ep), qm = 0.0, sj = 0.0;
  if (minus_side) qm = f.um * T(0, sm, em);
  if (b < NV) {
    qp = fma(f.vp, T(2, spp, ep), qp);
    if (minus_side) qm = fma(f.vm, T(2, sm, em), qm);
    sj = T(1, sm, em) - T(1, spp, ep);
  }
  double w = (plus ? th : -(1.0 - th)) * sj;
  const double K = jcm ? jcm[face_index(N, s, j, k) + (size_t)(N + 1) * N * b] : 0.0;
  if (tau != 0.0) w = fma(-tau, (qm - qp) + K, w);
  double a = fma(f.ap, qp, f.pen * sj);
  if (minus_side) a = fma(f.am, qm, a);
  if (jcm) a = fma(f.ak, K, a);
  ya = a;
  yd = f.dD * w;
  yf = f.dF * w;
}

// k_stage's work for the block's elements from e0 on
template <int NU, int NV>
__device__ __forceinline__ void stage_fast_body(const Basis<NU, NV> &B, const Fields &F, const StageIO &S, int e0) {
  using T = FastTeam<NU, NV>;
  constexpr int NQ = NU;
  __shared__ double sh[T::TPB * T::SLOT];
  __shared__ FxC tQ[NU * NU], tM[NU * NU][2], tE[2 * NU]; // per-thread columns and rows of the operators
  __shared__ double Pws[NQ * NU];
  for (int i = threadIdx.x; i < NU * NU; i += blockDim.x) {
    tQ[i] = B.fQ[i / NU][i % NU];
    tM[i][0] = B.fM[i / NU][i % NU][0];
    tM[i][1] = B.fM[i / NU][i % NU][1];
    Pws[i] = B.Pw[i / NU][i % NU];
  }
  if (threadIdx.x < NU) { tE[threadIdx.x] = B.fEl[threadIdx.x]; tE[NU + threadIdx.x] = B.fE1[threadIdx.x]; }
  after_previous();
  __syncthreads();
  if (stage_failed(F, e0 == 0 && threadIdx.x == 0)) return;
  const int lane = threadIdx.x & 31, tw = lane / NU;
  if (tw >= T::TPW) return;
  const int c = lane - tw * NU, slot = (threadIdx.x >> 5) * T::TPW + tw;
  const int e = e0 + slot, E = F.E, N = F.N;
  if (e >= E) return;
  const unsigned mask = ((1u << NU) - 1u) << (tw * NU);
  const Team team{mask, tw * NU, c};
  const size_t Eu = (size_t)E;
  const bool usolve = S.mode == OUT_ADJ_USOLVE, volume = S.mode == OUT_ADJ_VOLUME;
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  double *base = sh + slot * T::SLOT;
  i64 *X = reinterpret_cast<i64 *>(base);                // X(a, b) at X[a + NU b]
  Fx2 *AD = reinterpret_cast<Fx2 *>(base + T::X);        // axis 1: A by parity, D by parity
  Fx2 *Fv = AD + 4 * NU;                                 // F of both axes by parity
  i64 *FQ = reinterpret_cast<i64 *>(Fv + 4 * NU);        // axis 0's F in the eigenbasis, by parity
  FaceFactors *ff = reinterpret_cast<FaceFactors *>(FQ + 2 * NU);
  constexpr bool QI = NU <= 3;                           // one mode beside the constant one of each parity: Q = 1
  const int dQ = QI ? 0 : 61 - B.gQ;
  bool ok = true;
  double x00 = 0.0;                                      // the constant mode, which the u-solve passes
  int sX, sF = 0;                                        // exponents of the integers in X and of F's
  i64 f1[2] = {0, 0};                                    // axis 1's F in the eigenbasis at row c, by parity
  Fx2 x[NU];                                             // a column of the u-solve's input

  // R = K1 W + W K1 on column c (rows a < NU) for the blocks' columns w of the team's threads, whose
  // integers have the exponent s; on return s is R's. Uses X.
  auto stiffness = [&](const i64 (&w)[NU], i64 (&R)[NU], int &s) {
    constexpr int kmax = k1_bits<NU>(NU - 1);
    int top = 0;                                         // the largest |W| 2^(k of its modes - kmax), high words
    const int kc = B.kK1[c];
#pragma unroll
    for (int a = 0; a < NU; ++a) top = max(top, fx_hi(w[a]) >> (kmax - max(k1_bits<NU>(a), kc)));
    const int room = fx_room(team_max<NU>(team, top) + 1);
    s += kmax - room + 61 - B.gK1;
    // the entry of a contraction over its mode m: W 2^(k_m - kmax + room)
    auto scaled = [&](i64 v, int m) {
      const int n = room - (kmax - k1_bits<NU>(m));
      return fx_split((v << max(n, 0)) >> max(-n, 0));
    };
    Fx2 y[NU];
    auto yc = [&](int m) { return y[m]; };
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      X[a + NU * c] = w[a];
      y[a] = scaled(w[a], a);
    }
    R[0] = 0;
#pragma unroll
    for (int a = 1; a < NU; ++a) {                       // K1 W, column c
      auto q = [&](int m) -> const FxC & { return B.fK1[a][m]; };
      R[a] = (a & 1) ? fx_dot<1, 2, NU>(yc, q) : fx_dot<2, 2, NU>(yc, q);
    }
    __syncwarp(mask);
#pragma unroll
    for (int b = 0; b < NU; ++b) y[b] = scaled(X[c + NU * b], b);
    __syncwarp(mask);
#pragma unroll
    for (int b = 1; b < NU; ++b) {                       // W K1, row c, to the columns' threads
      auto q = [&](int m) -> const FxC & { return B.fK1[b][m]; };
      X[c + NU * b] = (b & 1) ? fx_dot<1, 2, NU>(yc, q) : fx_dot<2, 2, NU>(yc, q);
    }
    __syncwarp(mask);
    if (c > 0)
#pragma unroll
      for (int a = 0; a < NU; ++a) R[a] += X[a + NU * c];
    __syncwarp(mask);
  };

  if (usolve) {
    double d[NU];
    int hx = 0;
    x00 = S.xu[e];
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      d[a] = a + c > 0 ? S.xu[e + Eu * (a + NU * c)] : 0.0;
      hx = max(hx, fx_abs_hi(d[a]));
    }
    hx = team_max<NU>(team, hx);
    ok = fx_finite(hx);
    const int ex = fx_exp(hx);
    sX = ex - FX_BIAS;
#pragma unroll
    for (int a = 0; a < NU; ++a) x[a] = fx_split(fx_from(d[a], ex));
  } else {
    // ---- column c of U and V, and their exponents away from the constant mode, which no stiffness
    //      sees: from k_prep, or for the adjoint's volume mode from the input
    const double c2 = F.c2e[e], al = F.ae[e];
    double du[NU], dv[NU];
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      du[a] = a + c > 0 ? S.xu[e + Eu * (a + NU * c)] : 0.0;
      dv[a] = a + c > 0 && a < NV && c < NV ? S.xv[e + Eu * (a + NV * c)] : 0.0;
    }
    int hu = 0, hv = 0;
    if (!volume) {
      const i64 w = reinterpret_cast<const i64 *>(F.G)[(size_t)(Basis<NU, NV>::QH * Basis<NU, NV>::QH + 1) * E + e];
      hu = (int)(w >> 32);
      hv = (int)w;
    } else {
#pragma unroll
      for (int a = 0; a < NU; ++a) { hu = max(hu, fx_abs_hi(du[a])); hv = max(hv, fx_abs_hi(dv[a])); }
      hu = team_max<NU>(team, hu);
      hv = team_max<NU>(team, hv);
    }
    ok = fx_finite(hu) && fx_finite(hv);
    const int eu = fx_exp(hu), ev = fx_exp(hv);
#pragma unroll
    for (int a = 0; a < NU; ++a) x[a] = fx_split(fx_from(dv[a], ev));
    sX = ev - FX_BIAS;

    // ---- volume terms (src/rhs.jl:309-333)
    i64 R[NU];
    int sR;
    {
      const double mc2 = -F.four_hh * c2, mal = -F.four_hh * al;
      auto expo = [](double y) { return (__double2hiint(y) >> 20) & 0x7ff; };
      // |mc2 U|, |mal V| < 2^kU, 2^kV; W below 2^(kW - 1)
      const int kU = expo(mc2) - 1022 + eu - FX_BIAS + 61, kV = expo(mal) - 1022 + ev - FX_BIAS + 61;
      sR = max(kU, kV) + 2 - 61;
      const Fx2 mu = fx_split(fx_scalar(mc2, 2 * FX_BIAS - eu + sR - 61));
      const Fx2 mv = fx_split(fx_scalar(mal, 2 * FX_BIAS - ev + sR - 61));
      i64 w[NU];
#pragma unroll
      for (int a = 0; a < NU; ++a) {
        const Fx2 u = fx_split(fx_from(du[a], eu));
        i64 m = fx_mad(u.h, mu.l, fx_mad(u.l, mu.h, 1 << 28));
        m = fx_mad(x[a].h, mv.l, fx_mad(x[a].l, mv.h, m));
        m = fx_mad(u.h, mu.h << 3, m >> 29);
        w[a] = a + c > 0 ? fx_mad(x[a].h, mv.h << 3, m) : 0;
      }
      stiffness(w, R, sR);
    }

    if (volume) {
      // the volume terms alone: vt = R, ut = b = c²(K1 V + V K1)
      const double ur = ok ? fx_unit(sR) : nan;
      if (c < NV)
#pragma unroll
        for (int a = 0; a < NV; ++a) S.vt[e + Eu * (a + NV * c)] = __dmul_rn((double)R[a], ur);
      i64 w[NU];
#pragma unroll
      for (int a = 0; a < NU; ++a) w[a] = fx_join(x[a]);
      stiffness(w, R, sX);
      const double ub = (ok ? fx_unit(sX) : nan) * c2;
#pragma unroll
      for (int a = 0; a < NU; ++a) S.ut[e + Eu * (a + NU * c)] = __dmul_rn((double)R[a], ub);
      return;
    }

    // ---- faces: mode c of the projected slots of the four sides
    const int j = e % N, k = e / N;
    const TimeF tf = time_factors(S);
    const double ic2 = F.ic2e[e];
    const bool bnd[4] = {j == 0, j == N - 1, k == 0, k == N - 1};
    double A[4], D[4], Fo[4];
    if (F.modal) {
      for (int s = c; s < 4; s += NU)
        if (!bnd[s]) ff[s] = face_factors<NU>(F, s, j, k, ic2);
    } else {
#pragma unroll 1
      for (int s = 0; s < 4; ++s)
        if (!bnd[s])
          side_point<NU, NV>(F, s, j, k, e, c, base[(3 * s) * NQ + c], base[(3 * s + 1) * NQ + c],
                             base[(3 * s + 2) * NQ + c]);
    }
    __syncwarp(mask);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      A[s] = D[s] = Fo[s] = 0.0;
      if (bnd[s] || !F.modal) {
        if (bnd[s]) {
          const double *o = F.bslots + (size_t)s * N + (s < 2 ? k : j);
          const size_t st = (size_t)4 * N;
          if (c < NV) { A[s] = o[c * st]; D[s] = o[(NV + c) * st]; }
          Fo[s] = o[(2 * NV + c) * st];
        } else {
          const double *q = base + 3 * s * NQ;
#pragma unroll 1
          for (int i = 0; i < NQ; ++i) {
            const double p = Pws[i * NU + c];
            A[s] = fma(p, q[i], A[s]);
            D[s] = fma(p, q[NQ + i], D[s]);
            Fo[s] = fma(p, q[2 * NQ + i], Fo[s]);
          }
          if (c >= NV) A[s] = D[s] = 0.0;
        }
        A[s] *= F.two_h; D[s] *= F.four_hh; Fo[s] *= ic2;
      } else {
        interior_slot<NU, NV>(F, ff[s], s, j, k, e, c, A[s], D[s], Fo[s]);
        if (c >= NV) A[s] = D[s] = 0.0;
      }
    }
    int ha = 0, hd = 0, hf = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      ha = max(ha, fx_abs_hi(A[s]));
      hd = max(hd, fx_abs_hi(D[s]));
      hf = max(hf, fx_abs_hi(Fo[s]));
    }
    ha = team_max<NU>(team, ha);
    hd = team_max<NU>(team, hd);
    hf = team_max<NU>(team, hf);
    ok = ok && fx_finite(ha) && fx_finite(hd) && fx_finite(hf);
    const int ea = fx_exp(ha) + 1, ed = fx_exp(hd) + 1, ef = fx_exp(hf) + 1;
    // ---- lifts (src/rhs.jl:421-473). The two sides of an axis are lifted together: with σ_a = (-1)^a the
    //      right-end factors are the left-end ones times ±σ_a, so R += El ⊗ (A_0 + σ A_1) + E1l ⊗ (D_0 -
    //      σ D_1) and b = -E1l ⊗ (F_0 - σ F_1) (bottom/top: the row index carries E; left/right: the
    //      column index). R and the lifts take the largest of their exponents.
    const int sA = ea - FX_BIAS + 61 - B.gEl, sD = ed - FX_BIAS + 61 - B.gE1;
    const int sN = max(sR, max(sA, sD)), nA = sN - sA, nD = sN - sD, nR = sN - sR;
    Fx2 a0[2], d0[2];                                    // axis 0 at column c, by the row's parity
    {
      const i64 p0 = fx_from(A[0], ea), p1 = fx_from(A[1], ea), p2 = fx_from(A[2], ea), p3 = fx_from(A[3], ea);
      const i64 q0 = fx_from(D[0], ed), q1 = fx_from(D[1], ed), q2 = fx_from(D[2], ed), q3 = fx_from(D[3], ed);
      const i64 f0 = fx_from(Fo[0], ef), f1_ = fx_from(Fo[1], ef), f2 = fx_from(Fo[2], ef), f3 = fx_from(Fo[3], ef);
      a0[0] = fx_split(fx_down(p0 + p1, nA)); a0[1] = fx_split(fx_down(p0 - p1, nA));
      d0[0] = fx_split(fx_down(q0 - q1, nD)); d0[1] = fx_split(fx_down(q0 + q1, nD));
      AD[c] = fx_split(fx_down(p2 + p3, nA)); AD[NU + c] = fx_split(fx_down(p2 - p3, nA));
      AD[2 * NU + c] = fx_split(fx_down(q2 - q3, nD)); AD[3 * NU + c] = fx_split(fx_down(q2 + q3, nD));
      Fv[c] = fx_split(f0 - f1_); Fv[NU + c] = fx_split(f0 + f1_);
      Fv[2 * NU + c] = fx_split(f2 - f3); Fv[3 * NU + c] = fx_split(f2 + f3);
    }
    __syncwarp(mask);
    if (c < NV) {
      // column c of R, the source (src/rhs.jl:340-350), and the mass right-hand side to HBM
      const FxC el = tE[c], e1 = tE[NU + c];
      const Fx2 *a1 = AD + (c & 1) * NU, *d1 = a1 + 2 * NU;
      const double ur = ok ? fx_unit(sN) : nan;
#pragma unroll
      for (int a = 0; a < NV; ++a) {
        const Fx2 p = a0[a & 1], q = d0[a & 1], p1 = a1[a], q1 = d1[a];
        i64 m = fx_mad(p.h, B.fEl[a].l, fx_mad(p.l, B.fEl[a].h, 1 << 28));
        m = fx_mad(q.h, B.fE1[a].l, fx_mad(q.l, B.fE1[a].h, m));
        m = fx_mad(p1.h, el.l, fx_mad(p1.l, el.h, m));
        m = fx_mad(q1.h, e1.l, fx_mad(q1.l, e1.h, m));
        m = fx_mad(p.h, B.fEl[a].h8, m >> 29);
        m = fx_mad(q.h, B.fE1[a].h8, m);
        m = fx_mad(p1.h, el.h8, m);
        m = fx_mad(q1.h, e1.h8, m);
        const size_t l = (a + NV * c) * Eu + e;
        double y = (double)(fx_down(R[a], nR) + m);
        if (F.mms_on) {
          y = fma(tf.cSP, F.PiSP[l], __dmul_rn(y, ur));
          y = fma(tf.cB, F.PiBSP2[l], y);
          y = fma(tf.cC, F.PiCdiv[l], y);
          y = fma(tf.cD, F.PiDdiv[l], y);
        } else if (!F.src_on) {
          y = fma(y, ur, F.PiCdiv[l]);
        } else {
          y = __dmul_rn(y, ur);
        }
        if (F.src_on) y = fma(tf.srct, F.srcP[l], y);
        F.mrhs[l] = y;
      }
    }
    // ---- the slots F into the eigenbasis: Q^T F, entry c
    x00 = S.xv[e];
    sF = ef - FX_BIAS + dQ;
    auto q = [&](int a) -> const FxC & { return tQ[a * NU + c]; };
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      auto g0 = [&](int a) { return Fv[p * NU + a]; };
      auto g1 = [&](int a) { return Fv[(2 + p) * NU + a]; };
      i64 y0, y1;
      if (QI || c == 0) {
        y0 = fx_down(fx_join(Fv[p * NU + c]), dQ);
        y1 = fx_down(fx_join(Fv[(2 + p) * NU + c]), dQ);
      } else {                                           // (Q vanishes between modes of unlike parity)
        y0 = fx_dot<1, 1, NU>(g0, q);
        y1 = fx_dot<1, 1, NU>(g1, q);
      }
      FQ[p * NU + c] = y0;
      f1[p] = y1;
    }
  }

  // ---- the u-solve (src/rhs.jl:352-382), four products with Q, columns and rows in turn
  auto xs = [&](int a) { return x[a]; };
  X[NU * c] = fx_down(fx_join(x[0]), dQ);                // Q^T V, column c
#pragma unroll
  for (int i = 1; i < NU; ++i) {
    auto q = [&](int a) -> const FxC & { return B.fQ[a][i]; };
    X[i + NU * c] = QI ? fx_join(x[i]) : (i & 1) ? fx_dot<1, 2, NU>(xs, q) : fx_dot<2, 2, NU>(xs, q);
  }
  __syncwarp(mask);
#pragma unroll
  for (int b = 0; b < NU; ++b) x[b] = fx_split(X[c + NU * b]);
  // row c of X Q, with the eigenvalues: L ∘ X for the solve of a given right-hand side, X + L ∘ b~ for the
  // forward one (b~'s exponent sB, aligned with X's)
  const int sV = sX + 2 * dQ, sB = sF + 61 - B.gM;
  sX = usolve ? sV + 61 - B.gL : max(sV, sB) + 1;
  const int nV = sX - sV, nB = sX - sB;
  const Fx2 g1[2] = {fx_split(f1[0]), fx_split(f1[1])};
  int top = 0;                                           // the largest high word of the row
#pragma unroll
  for (int b = 0; b < NU; ++b) {
    auto q = [&](int m) -> const FxC & { return B.fQ[m][b]; };
    i64 y;
    if (QI || b == 0) y = fx_down(fx_join(x[b]), dQ);
    else y = (b & 1) ? fx_dot<1, 2, NU>(xs, q) : fx_dot<2, 2, NU>(xs, q);
    if (usolve) {
      const FxC l = B.fL[c][b];
      y = fx_mul(fx_split(y), Fx2{l.h, l.l});
    } else {
      const Fx2 f0 = fx_split(FQ[(c & 1) * NU + b]), g = g1[b & 1];
      const FxC c0 = tM[c * NU + b][0], c1 = tM[c * NU + b][1];
      i64 m = fx_mad(f0.h, c0.l, fx_mad(f0.l, c0.h, 1 << 28));
      m = fx_mad(g.h, c1.l, fx_mad(g.l, c1.h, m));
      m = fx_mad(f0.h, c0.h8, m >> 29);
      m = fx_mad(g.h, c1.h8, m);
      y = fx_down(y, nV) + fx_down(m, nB);
    }
    X[c + NU * b] = y;
    top |= fx_hi(y);
  }
  // Each product leaves dQ bits of headroom for sums that an orthonormal Q seldom has: over the four of them eight
  // bits, so that 52 were left. The room there is after two is taken back (2^sX stays far from subnormal)
  const int up = min(fx_room(team_or<NU>(team, top)), max(sX + 960, 0));
  sX -= up;
  __syncwarp(mask);
#pragma unroll
  for (int i = 0; i < NU; ++i) x[i] = fx_split(X[i + NU * c] << up);
  X[NU * c] = fx_down(fx_join(x[0]), dQ);                // Q X, column c
#pragma unroll
  for (int a = 1; a < NU; ++a) {
    auto q = [&](int i) -> const FxC & { return B.fQ[a][i]; };
    X[a + NU * c] = QI ? fx_join(x[a]) : (a & 1) ? fx_dot<1, 2, NU>(xs, q) : fx_dot<2, 2, NU>(xs, q);
  }
  __syncwarp(mask);
  // row c of X Q^T, and the u outputs: RK4 (src/solver.jl:289-321): acc = k1 + 2 k2 + 2 k3 in this
  // order, the next stage state u + c k, the last stage u + (dt/6)(acc + k4) with the finite check
#pragma unroll
  for (int i = 0; i < NU; ++i) x[i] = fx_split(X[c + NU * i]);
  // kk = t f: f the integers' unit, but 1 for the constant mode (thread 0's first entry)
  const double un = (ok ? fx_unit(sX + 2 * dQ) : nan) * (usolve ? F.ic2e[e] : 1.0), u1 = ok ? 1.0 : nan;
  const double un2 = __dmul_rn(2.0, un), unc = __dmul_rn(S.c, un);
  bool fin = true;
#pragma unroll
  for (int b = 0; b < NU; ++b) {
    auto q = [&](int i) -> const FxC & { return B.fQ[b][i]; };
    i64 y;
    if (QI || b == 0) y = fx_down(fx_join(x[b]), dQ);
    else y = (b & 1) ? fx_dot<1, 2, NU>(xs, q) : fx_dot<2, 2, NU>(xs, q);
    const bool first = b == 0 && c == 0;
    const double t = first ? x00 : (double)y, f = first ? u1 : un;
    const size_t l = e + Eu * (c + NU * b);
    if (S.mode == OUT_RHS || usolve) {
      S.ut[l] = __dmul_rn(t, f);
    } else if (S.mode == OUT_RK4_STAGE) {
      S.accu[l] = S.first ? __dmul_rn(t, f) : fma(t, first ? 2.0 * u1 : un2, S.accu[l]);
      S.su[l] = fma(t, first ? S.c * u1 : unc, S.u0[l]);
    } else if (S.mode == OUT_RK4_LAST) {
      // Chebyshev mode only: no error can arise after k_prep, so u is updated in place now
      const double x1 = fma(S.c, fma(t, f, S.accu[l]), S.u0[l]);
      S.uo[l] = x1;
      fin = fin && isfinite(x1);
    } else {
      S.accu[l] = fma(t, f, S.accu[l]);
    }
  }
  if (S.mode == OUT_RK4_LAST && !fin) atomicOr(F.nonfinite, 1u);
}

}  // namespace wedg
