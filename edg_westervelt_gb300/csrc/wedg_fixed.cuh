// 64-bit fixed-point arithmetic for the contractions of the stage kernels.
//
// The FP64 pipe of sm_103a issues 2 lanes per clock and SM (628 G DFMA/s measured over the chip: eight chains
// a thread, 64 warps an SM, 2 070 MHz), 64 cycles a warp and scheduler; the integer multiply-add with a 64-bit sum
// (mad.wide.s32) takes 2.04 (19 780 G/s, the same probe), at the same time. A product of two 62-bit
// integers costs three of them, a tenth of an FP64 one; the sums, shifts and splits around it are work of the
// ALU. A block keeps 61 bits of its largest number where doubles keep 53 of each: a number 2^-k of the largest
// has 61 - k.
//
// A block of numbers shares one exponent: x = X 2^s with |X| < 2^61, from the largest number of the
// block (fx_from). Numbers and constants are used in balanced halves, X = h 2^32 + l with l in
// [-2^31, 2^31), so that every partial product is signed. A sum of products drops the products of
// two low halves:
//   Σ X C / 2^61 = Σ h_X (8 h_C) + (Σ (h_X l_C + l_X h_C)) / 2^29.
// With Σ|C| ≤ 2^61, every |C| < 2^60 and at most six terms no partial sum overflows and the result
// is again below 2^61: contractions chain without a check. Its error is about one unit, 2^-61 of the
// largest result the constants allow, against half a unit of 2^-53 of every partial sum in FP64.
#pragma once
#include <cuda_runtime.h>

namespace wedg {

typedef long long i64;
typedef unsigned long long u64;

// A constant C 2^-g of an operator (g stands beside the array): balanced halves and 8 h
struct alignas(16) FxC {
  int h, l, h8;
};

// A number in balanced halves
struct Fx2 {
  int h, l;
};
__host__ __device__ __forceinline__ Fx2 fx_split(i64 x) {
  return Fx2{(int)(x >> 32) + (int)((unsigned)x >> 31), (int)x};
}
__host__ __device__ __forceinline__ i64 fx_join(Fx2 x) { return (i64)x.h * ((i64)1 << 32) + x.l; }

// The exponent field of a block from the largest high word (sign bit cleared) of its numbers. Blocks
// below 2^-895 share that exponent, so that 2^s is a normal double: their numbers keep an absolute
// error of 2^-955.
constexpr int FX_EXP_MIN = 128;
__device__ __forceinline__ int fx_exp(int hmax) { return max(hmax >> 20, FX_EXP_MIN); }
__device__ __forceinline__ bool fx_finite(int hmax) { return hmax < 0x7ff00000; }
__device__ __forceinline__ int fx_abs_hi(double x) { return __double2hiint(x) & 0x7fffffff; }

// x as an integer of the block with exponent field ex: x = X 2^(ex - FX_BIAS), |X| < 2^61 (smaller by
// 2^k for ex raised by k); toward zero
constexpr int FX_BIAS = 1083;
__device__ __forceinline__ i64 fx_from(double x, int ex) {
  const int hi = __double2hiint(x);
  const int sh = ex - ((hi >> 20) & 0x7ff);
  u64 m = ((u64)(unsigned)((hi & 0xfffff) | 0x100000) << 32 | (unsigned)__double2loint(x)) << 8;
  asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(sh));   // 0 from 64 on
  const i64 s = hi >> 31;
  return ((i64)m ^ s) - s;
}

// x as the integer x 2^(FX_BIAS - ex) (a scalar of any size: 0 where that is below 1)
__device__ __forceinline__ i64 fx_scalar(double x, int ex) {
  return (__double2hiint(x) & 0x7ff00000) ? fx_from(x, ex) : 0;
}

// The bits by which a thread's numbers with the largest |high word| h (h ^ (h >> 31)) can go up
__device__ __forceinline__ int fx_room(int h) { return max(__clz(h) - 3, 0); }
__device__ __forceinline__ int fx_hi(i64 x) {
  const int h = (int)(x >> 32);
  return h ^ (h >> 31);
}

// x 2^-n for n ≥ 0 (toward -∞; n from 64 on as 63) and x 2^n for any n, modulo 2^64
__device__ __forceinline__ i64 fx_sar(i64 x, int n) {
  asm("shr.s64 %0, %0, %1;" : "+l"(x) : "r"(n));
  return x;
}
__device__ __forceinline__ i64 fx_shift(i64 x, int n) {
  asm("shl.b64 %0, %0, %1;" : "+l"(x) : "r"(max(n, 0)));     // 0 from 64 on
  return fx_sar(x, max(-n, 0));
}

// 2^k for -1022 ≤ k ≤ 1023, and x 2^k for any k (rounded where that is subnormal)
__device__ __forceinline__ double fx_pow2(int k) { return __hiloint2double((k + 1023) << 20, 0); }
__device__ __forceinline__ double fx_scale(double x, int k) {
  k = min(max(k, -2044), 2046);
  return __dmul_rn(__dmul_rn(x, fx_pow2(k >> 1)), fx_pow2(k - (k >> 1)));
}

__device__ __forceinline__ i64 fx_mad(int a, int b, i64 c) {
  i64 d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// Σ_i x(i) c(i) / 2^61 over i = I0, I0 + ST, ... < N (x: Fx2, c: FxC)
template <int I0, int ST, int N, class X, class C>
__device__ __forceinline__ i64 fx_dot(const X &x, const C &c) {
  i64 m = 1 << 28;                                 // to nearest
#pragma unroll
  for (int i = I0; i < N; i += ST) {
    const Fx2 a = x(i);
    m = fx_mad(a.h, c(i).l, m);
    m = fx_mad(a.l, c(i).h, m);
  }
  m >>= 29;
#pragma unroll
  for (int i = I0; i < N; i += ST) m = fx_mad(x(i).h, c(i).h8, m);
  return m;
}

// x c / 2^61 for |c| < 2^60
__device__ __forceinline__ i64 fx_mul(Fx2 x, Fx2 c) {
  const i64 m = fx_mad(x.h, c.l, fx_mad(x.l, c.h, 1 << 28));
  return fx_mad(x.h, c.h << 3, m >> 29);
}

// The largest or smallest x and the or of the bits of a team of W threads (this one thread u of it, the first at
// lane0), on every one of them, by shuffles around the team: what they gather overlaps, which these operations
// allow. A reduction instruction takes the teams of a warp one by one, 240 to 980 cycles (W = 10 and 3),
// the shuffles 200 to 230.
struct Team {
  unsigned mask;
  int lane0, u;
};
template <int W, class T, class Op>
__device__ __forceinline__ T team_all(const Team &t, T x, const Op &op) {
#pragma unroll
  for (int o = 1; o < W; o *= 2) x = op(x, __shfl_sync(t.mask, x, t.lane0 + (t.u + o < W ? t.u + o : t.u + o - W)));
  return x;
}
template <int W, class T>
__device__ __forceinline__ T team_max(const Team &t, T x) {
  return team_all<W>(t, x, [](T a, T b) { return max(a, b); });
}
template <int W, class T>
__device__ __forceinline__ T team_min(const Team &t, T x) {
  return team_all<W>(t, x, [](T a, T b) { return min(a, b); });
}
template <int W, class T>
__device__ __forceinline__ T team_or(const Team &t, T x) {
  return team_all<W>(t, x, [](T a, T b) { return a | b; });
}

// Host side: the exponent g of an operator whose contractions have sums of magnitudes up to `sum` and
// entries up to `big` (Σ|C| ≤ 2^61, |C| < 2^60), and one entry of it
inline int fx_exponent(double sum, double big) {
  if (!(sum > 0) || !(big > 0)) return 0;
  int a, b;
  frexp(sum, &a);
  frexp(big * (1 + 1e-6), &b);
  return (61 - a < 60 - b) ? 61 - a : 60 - b;
}
inline FxC fx_const(long double x, int g) {
  const Fx2 p = fx_split((i64)llrintl(ldexpl(x, g)));
  return FxC{p.h, p.l, 8 * p.h};
}

}  // namespace wedg
