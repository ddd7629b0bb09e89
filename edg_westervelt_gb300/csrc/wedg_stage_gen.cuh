// k_stage for coefficients that vary inside the elements (the general kernels): fluxes and lifts,
// volume terms by quadrature, source and u-equation by the stored inverse, a team of NU threads per
// element. Thread r of the team takes the r-th face point of the four sides, then the r-th mode along
// the faces, then the r-th row of the point grid, then column r of the modal blocks.
//
// What bounds it: about 9 000 FP64 operations an element at q = 6, and the 9.8 KB of its inverse. One
// thread per element left the chip idle below some 150 000 elements (one warp's FP64 operations are
// a chain of 64 cycles each) and held two blocks of state per thread in shared memory; a team
// spreads an element over NU times the warps. The teams of a warp take neighbouring elements, so
// that a load of one entry per thread reads whole 32-byte sectors. N = 201, q = 6: 1 242 us with a thread per
// element, 783 us by teams; N = 32, q = 4: 191 and 41 us; N = 512, q = 6, where a thread per element filled the
// chip: 4 950 and 4 800 us, the FP64 pipe 90 % busy.
#pragma once

namespace wedg {

template <int NU, int NV>
struct GenTeam {
  static constexpr int TPW = 32 / NU;                    // teams (elements) per warp
  static constexpr int THREADS = 128;
  static constexpr int TPB = TPW * (THREADS / 32);       // elements per block
  // U, V; the slots; the volume rows; b
  static constexpr int Z = 2 * NU * NV + 2 * NU * NU > 12 * NU ? 2 * NU * NV + 2 * NU * NU : 12 * NU;
  static constexpr int YS = 2 * NV + NU;                 // a side's projections of A, D and F
  static constexpr int SLOT = (Z + 4 * YS) | 1;          // odd: fewer bank conflicts
};

// Mode b of the projections Y_A, Y_D (b < NV) and Y_F of the slots of interior side s from the traces'
// modal end sums (Fields::modal: every interior face has one value of the coefficients)
template <int NU, int NV>
__device__ __forceinline__ void modal_mode(const Fields &F, int s, int j, int k, int e, int b, double &ya, double &yd,
                                           double &yf) {
  constexpr int NQ = NU;
  const int N = F.N;
  const size_t E = F.E;
  const bool plus = (s == 0 || s == 2);
  const int nb = s == 0 ? e - 1 : s == 1 ? e + 1 : s == 2 ? e - N : e + N;
  const int sm = s < 2 ? 1 : 3, spp = s < 2 ? 0 : 2;      // trace sides of the "-" and "+" elements
  const int em = plus ? nb : e, ep = plus ? e : nb;
  size_t fi;
  const double *c2p_a, *afp_a, *c2m_a, *afm_a, *jc_a, *jcm;
  if (s < 2) {
    fi = (s == 0 ? j : j + 1) + (size_t)(N + 1) * k;
    c2p_a = F.hc2; afp_a = F.haf; c2m_a = F.hc2m; afm_a = F.hafm; jc_a = F.hJC; jcm = F.hJCm;
  } else {
    fi = j + (size_t)N * (s == 2 ? k : k + 1);
    c2p_a = F.vc2; afp_a = F.vaf; c2m_a = F.vc2m; afm_a = F.vafm; jc_a = F.vJC; jcm = F.vJCm;
  }
  FaceCoef cf = face_coef(F, c2p_a, afp_a, c2m_a, afm_a, jc_a, fi);   // point 0 of the face
  // interior_flux on the traces' modes: its slots are linear in them and in the jump term
  if (!F.one_sided) { cf.c2m = cf.c2p; cf.afm = cf.afp; }
  const size_t fstride = (size_t)(N + 1) * N;              // from point (mode) b to b + 1
  auto T = [&](int fam, int side, int el) { return F.tr[((fam * 4 + side) * NQ + b) * E + el]; };
  const double K = jcm ? jcm[fi + fstride * b] : 0.0;
  const double dum = T(0, sm, em), dup = T(0, spp, ep);
  double vm = 0.0, vp = 0.0, dvm = 0.0, dvp = 0.0;
  if (b < NV) { vm = T(1, sm, em); vp = T(1, spp, ep); dvm = T(2, sm, em); dvp = T(2, spp, ep); }
  cf.K = F.one_sided ? K : 0.0;
  interior_flux(F, cf, plus, dum, dup, vm, vp, dvm, dvp, ya, yd, yf);
}

// Row r of the point grid of the n × n block X (S, P: row r of the derivatives and values):
// Σ_b (Σ_a S[r][a] X[a][b]) P[s][b] and Σ_b (Σ_a P[r][a] X[a][b]) S[s][b], mirrored points together
// (P[m][b] = (-1)^b P[s][b], S[m][b] = -(-1)^b S[s][b] at m = NQ-1-s)
template <int NU, int NV, int n>
__device__ __forceinline__ void gen_row(const Basis<NU, NV> &B, const double *X, const double *S, const double *P,
                                        double (&y1)[NU], double (&y2)[NU]) {
  constexpr int NQ = NU;
  double t1[n], t2[n];
#pragma unroll
  for (int b = 0; b < n; ++b) { t1[b] = 0; t2[b] = 0; }
#pragma unroll
  for (int a = 0; a < n; ++a) {
    const double sa = S[a], pa = P[a];
#pragma unroll
    for (int b = 0; b < n; ++b) {
      const double x = X[a + n * b];
      t1[b] = fma(sa, x, t1[b]);
      t2[b] = fma(pa, x, t2[b]);
    }
  }
#pragma unroll
  for (int s = 0; s < (NQ + 1) / 2; ++s) {
    double pe = 0, po = 0, se = 0, so = 0;
#pragma unroll
    for (int b = 0; b < n; ++b) {
      if (b & 1) { po = fma(t1[b], B.P[s][b], po); so = fma(t2[b], B.S[s][b], so); }
      else { pe = fma(t1[b], B.P[s][b], pe); se = fma(t2[b], B.S[s][b], se); }
    }
    y1[s] = pe + po;
    y2[s] = se + so;
    if (2 * s + 1 != NQ) {
      y1[NQ - 1 - s] = pe - po;
      y2[NQ - 1 - s] = so - se;
    }
  }
}

// Back to the modes along the row: Σ_s y1[s] P[s][b], Σ_s y2[s] S[s][b], from the sums and differences of
// mirrored points
template <int NU, int NV, int n>
__device__ __forceinline__ void gen_back(const Basis<NU, NV> &B, double (&y1)[NU], double (&y2)[NU], double sc,
                                         double *o1, double *o2) {
  constexpr int NQ = NU;
#pragma unroll
  for (int s = 0; s < NQ / 2; ++s) {
    const int m = NQ - 1 - s;
    const double p = y1[s] + y1[m], d = y1[s] - y1[m], p2 = y2[s] + y2[m], d2 = y2[s] - y2[m];
    y1[s] = p; y1[m] = d; y2[s] = p2; y2[m] = d2;
  }
#pragma unroll
  for (int b = 0; b < n; ++b) {
    double x1 = 0, x2 = 0;
#pragma unroll
    for (int s = 0; s < NQ / 2; ++s) {
      const int m = NQ - 1 - s;
      x1 = fma((b & 1) ? y1[m] : y1[s], B.P[s][b], x1);
      x2 = fma((b & 1) ? y2[s] : y2[m], B.S[s][b], x2);
    }
    if ((NQ & 1) != 0) {                              // the middle point
      if (!(b & 1)) x1 = fma(y1[NQ / 2], B.P[NQ / 2][b], x1);
      else x2 = fma(y2[NQ / 2], B.S[NQ / 2][b], x2);
    }
    o1[b] = sc * x1;
    o2[b] = sc * x2;
  }
}

// k_stage's work for the block's elements from e0 on
template <int NU, int NV>
__device__ __forceinline__ void stage_gen_body(const Basis<NU, NV> &B, const Fields &F, const StageIO &S, int e0) {
  using T = GenTeam<NU, NV>;
  constexpr int NQ = NU, YS = T::YS;
  __shared__ double sh[T::TPB * T::SLOT];
  __shared__ double Ps[NQ * NU], Ss[NQ * NU], Pws[NQ * NU], ends[4 * NU];
  for (int i = threadIdx.x; i < NQ * NU; i += blockDim.x) {
    Ps[i] = B.P[i / NU][i % NU];
    Ss[i] = B.S[i / NU][i % NU];
    Pws[i] = B.Pw[i / NU][i % NU];
  }
  if (threadIdx.x < NU) {
    const int i = threadIdx.x;
    ends[i] = B.El[i]; ends[NU + i] = B.E1l[i]; ends[2 * NU + i] = B.E1F[i];
  }
  after_previous();
  __syncthreads();
  if (stage_failed(F, e0 == 0 && threadIdx.x == 0)) return;
  const int lane = threadIdx.x & 31, tw = lane / NU;
  if (tw >= T::TPW) return;
  const int r = lane - tw * NU, slot = (threadIdx.x >> 5) * T::TPW + tw;
  const int e = e0 + slot, E = F.E, N = F.N;
  if (e >= E) return;
  const unsigned mask = (NU == 32 ? ~0u : ((1u << NU) - 1u)) << (tw * NU);
  const size_t Eu = (size_t)E;
  const bool adjoint = S.mode >= OUT_ADJ_USOLVE;
  const bool has_v = r < NV;                              // the thread's column of the v-blocks
  const double two_h = F.two_h, four_hh = F.four_hh;
  double *z = sh + slot * T::SLOT, *Y = z + T::Z;
  const TimeF tf = time_factors(S);
  double Rc[NV], bc[NU];                                  // column r of R_v and of b
#pragma unroll
  for (int a = 0; a < NU; ++a) {
    if (a < NV) Rc[a] = 0.0;
    bc[a] = S.mode == OUT_ADJ_USOLVE ? S.xu[e + Eu * (a + NU * r)] : 0.0;
  }

  // ---- faces and lifts (src/rhs.jl:421-473)
  if (!adjoint) {
    const int j = e % N, k = e / N;
    const bool bnd[4] = {j == 0, j == N - 1, k == 0, k == N - 1};
    if (!F.modal) {
#pragma unroll 1
      for (int s = 0; s < 4; ++s)
        if (!bnd[s])
          side_point<NU, NV>(F, s, j, k, e, r, z[(3 * s) * NQ + r], z[(3 * s + 1) * NQ + r],
                             z[(3 * s + 2) * NQ + r]);
      __syncwarp(mask);
    }
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
      double ya = 0.0, yd = 0.0, yf = 0.0;
      if (bnd[s]) {
        const double *o = F.bslots + (size_t)s * N + (s < 2 ? k : j);
        const size_t st = (size_t)4 * N;
        if (has_v) { ya = o[r * st]; yd = o[(NV + r) * st]; }
        yf = o[(2 * NV + r) * st];
      } else if (F.modal) {
        modal_mode<NU, NV>(F, s, j, k, e, r, ya, yd, yf);
      } else {
        const double *q = z + 3 * s * NQ;
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          const double p = Pws[i * NU + r];
          ya = fma(p, q[i], ya);
          yd = fma(p, q[NQ + i], yd);
          yf = fma(p, q[2 * NQ + i], yf);
        }
      }
      if (has_v) { Y[s * YS + r] = ya; Y[s * YS + NV + r] = yd; }
      Y[s * YS + 2 * NV + r] = yf;
    }
    __syncwarp(mask);
    // R = El ⊗ (2/h)(A_0 + σ A_1) + E1l ⊗ (4/h²)(D_0 - σ D_1), b = E1F ⊗ (F_0 - σ F_1), σ_a = (-1)^a
    // (bottom/top: the row index carries E; left/right: the column index)
    const double sg = (r & 1) ? -1.0 : 1.0;
    const double el = two_h * ends[r], ed = four_hh * ends[NU + r], ef = ends[2 * NU + r];
    double ap = 0, am = 0, dp = 0, dm = 0;
    if (has_v) {
      ap = two_h * (Y[r] + Y[YS + r]); am = two_h * (Y[r] - Y[YS + r]);
      dp = four_hh * (Y[NV + r] + Y[YS + NV + r]); dm = four_hh * (Y[NV + r] - Y[YS + NV + r]);
    }
    const double fp = Y[2 * NV + r] + Y[YS + 2 * NV + r], fm = Y[2 * NV + r] - Y[YS + 2 * NV + r];
    const double *Yl = Y + 2 * YS, *Yr = Y + 3 * YS;
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      if (a < NV) {
        Rc[a] = fma(B.E1l[a], (a & 1) ? dp : dm, B.El[a] * ((a & 1) ? am : ap));
        if (has_v)
          Rc[a] = fma(ed, fma(-sg, Yr[NV + a], Yl[NV + a]), fma(el, fma(sg, Yr[a], Yl[a]), Rc[a]));
      }
      bc[a] = fma(ef, fma(-sg, Yr[2 * NV + a], Yl[2 * NV + a]), B.E1F[a] * ((a & 1) ? fp : fm));
    }
    __syncwarp(mask);
  }

  // ---- volume terms (src/rhs.jl:309-333): R += -4/h² [(c²∇φ_v,∇u_h) + (α∇φ_v,∇v_h)], b += (c²∇φ_u, ∇v_h),
  //      thread r on row r of the point grid
  if (S.mode != OUT_ADJ_USOLVE) {
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      z[a + NU * r] = S.xu[e + Eu * (a + NU * r)];
      if (a < NV && has_v) z[NU * NU + a + NV * r] = S.xv[e + Eu * (a + NV * r)];
    }
    __syncwarp(mask);
    const double *U = z, *V = z + NU * NU;
    double g1[NQ], g2[NQ], b1[NQ], b2[NQ];                // the rows at the points: u's and v's derivatives
    gen_row<NU, NV, NU>(B, U, Ss + r * NU, Ps + r * NU, g1, g2);
    gen_row<NU, NV, NV>(B, V, Ss + r * NU, Ps + r * NU, b1, b2);
    // weighted by the coefficients
#pragma unroll
    for (int s = 0; s < NQ; ++s) {
      const size_t ci = (r + NQ * s) * Eu + e;
      const double cw = F.Cw[ci], aw = F.Aw[ci];
      g1[s] = fma(aw, b1[s], cw * g1[s]);
      g2[s] = fma(aw, b2[s], cw * g2[s]);
      b1[s] *= cw;
      b2[s] *= cw;
    }
    __syncwarp(mask);                                     // U, V are spent
    double *z1 = z, *z2 = z + NU * NV, *y1 = z + 2 * NU * NV, *y2 = y1 + NU * NU;
    gen_back<NU, NV, NV>(B, g1, g2, -four_hh, z1 + r * NV, z2 + r * NV);
    gen_back<NU, NV, NU>(B, b1, b2, 1.0, y1 + r * NU, y2 + r * NU);
    __syncwarp(mask);
    // column r: the rows with their weights
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const double p1 = has_v ? z1[i * NV + r] : 0.0, p2 = has_v ? z2[i * NV + r] : 0.0;
      const double q1 = y1[i * NU + r], q2 = y2[i * NU + r];
#pragma unroll
      for (int a = 0; a < NU; ++a) {
        if (a < NV) Rc[a] = fma(B.S[i][a], p1, fma(B.P[i][a], p2, Rc[a]));
        bc[a] = fma(B.S[i][a], q1, fma(B.P[i][a], q2, bc[a]));
      }
    }
    __syncwarp(mask);
  }
  if (S.mode == OUT_ADJ_VOLUME) {
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      if (a < NV && has_v) S.vt[e + Eu * (a + NV * r)] = Rc[a];
      S.ut[e + Eu * (a + NU * r)] = bc[a];
    }
    return;
  }

  // ---- source (src/rhs.jl:340-350), and the mass right-hand side to HBM
  if (!adjoint) {
    if (has_v) {
#pragma unroll
      for (int a = 0; a < NV; ++a) {
        const size_t l = (a + NV * r) * Eu + e;
        double x = Rc[a];
        if (F.mms_on) {
          x = fma(tf.cSP, F.PiSP[l], x);
          x = fma(tf.cB, F.PiBSP2[l], x);
          x = fma(tf.cC, F.PiCdiv[l], x);
          x = fma(tf.cD, F.PiDdiv[l], x);
        } else if (!F.src_on) {
          x += F.PiCdiv[l];
        }
        if (F.src_on) x = fma(tf.srct, F.srcP[l], x);
        F.mrhs[l] = x;
      }
    }
    if (r == 0) bc[0] += S.xv[e];
  }

  // ---- u-equation (src/rhs.jl:352-382): UT = A_e⁻¹ b, A_e U = VB - Fu + e_1 V[0][0]. The packed upper
  //      triangle of the symmetric inverse by columns: entry (i, j), i ≤ j, in row j(j+1)/2 + i; thread r
  //      takes the rows of its column's entries
#pragma unroll
  for (int a = 0; a < NU; ++a) z[a + NU * r] = bc[a];
  __syncwarp(mask);
  double ut[NU];
#pragma unroll
  for (int a = 0; a < NU; ++a) ut[a] = 0.0;
  const double *Ai = F.Ainv + e;
#pragma unroll 1
  for (int c = 0; c < NU; ++c) {                          // block (·, column c): its own triangle for c = r
    double x[NU];
#pragma unroll
    for (int a = 0; a < NU; ++a) x[a] = z[a + NU * c];
#pragma unroll
    for (int a = 0; a < NU; ++a) {
      const int i = a + NU * r;
#pragma unroll
      for (int q = 0; q < NU; ++q) {
        const int jj = q + NU * c, lo = min(i, jj), hi = max(i, jj);
        ut[a] = fma(Ai[(size_t)(hi * (hi + 1) / 2 + lo) * Eu], x[q], ut[a]);
      }
    }
  }

  // ---- u outputs: RK4 (src/solver.jl:289-321): acc = k1 + 2 k2 + 2 k3 in this order, the next
  //      stage state u + c k, the last stage u + (dt/6)(acc + k4) with the finite check
  bool fin = true;
#pragma unroll
  for (int a = 0; a < NU; ++a) {
    const size_t l = e + Eu * (a + NU * r);
    const double kk = ut[a];
    if (S.mode == OUT_RHS || S.mode == OUT_ADJ_USOLVE) {
      S.ut[l] = kk;
    } else if (S.mode == OUT_RK4_STAGE) {
      S.accu[l] = S.first ? kk : S.accu[l] + 2.0 * kk;
      S.su[l] = S.u0[l] + S.c * kk;
    } else if (S.mode == OUT_RK4_LAST) {
      // Chebyshev mode only: no error can arise after k_prep, so u is updated in place now
      const double x = S.u0[l] + S.c * (S.accu[l] + kk);
      S.uo[l] = x;
      fin = fin && isfinite(x);
    } else {
      S.accu[l] = S.accu[l] + kk;
    }
  }
  if (S.mode == OUT_RK4_LAST && !fin) atomicOr(F.nonfinite, 1u);
}

}  // namespace wedg
