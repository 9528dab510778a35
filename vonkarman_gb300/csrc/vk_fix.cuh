// FP64-class line transforms on the integer pipes: 64-bit fixed point with one
// block exponent per line.
//
// GB300 issues 2 FP64 operations per clock and SM, but about 100 32-bit
// integer additions, 58 low and 29 high halves of 32 x 32 products (measured:
// DADD 1.9, 64-bit integer add 51, complex multiply below 2.2 per clock and
// SM), so a transform made of integer additions and multiplications runs
// several times faster than one made of DFMAs.
//
// A transform of L points takes two or three stages of in-register DFTs.  A
// line of doubles z becomes integers trunc(z 2^-Q), where 2^(Q + 62) bounds the
// sum of |z| over the inputs of every first-stage butterfly, so that no partial
// sum overflows; the twiddles of the later stages carry a factor 1/G (a power
// of two, at least their radix), which makes room for the stage's growth.
// Rounding then happens at the quantum 2^Q of the inputs (amplified by sqrt(L))
// and at G 2^Q, G^2 2^Q before the later stages (amplified by the square root
// of what follows); the butterfly sums are at most sqrt(R0) ||z||, so the error
// is below one unit in the last place of a double relative to the line's norm
// in the worst case, and a few times smaller for lines whose norm is spread
// out.  An FFT in doubles has the same
// kind of bound with a larger constant (tests/test_fix_cpu.py measures both).
//
// This header holds the arithmetic and the radix kernels (natural-order
// in-register DFTs, untwiddled); they also compile for the host, where the CPU
// tests run them against a reference.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define VK_FIX_HD __host__ __device__ __forceinline__
#else
#define VK_FIX_HD inline
#endif

namespace vk {

struct alignas(16) fx2 { long long x, y; };
// twiddle exp(-i a) = c + i d in the units of fx_growth, each component as
// h 2^32 + l with a signed low word
struct alignas(16) fxtw { int ch, cl, dh, dl; };

VK_FIX_HD long long fx_join(int hi, unsigned lo) { return (long long)(((unsigned long long)(unsigned)hi << 32) | lo); }
// high word of a b, plus c (mod 2^32)
VK_FIX_HD int fx_madhi(int a, int b, int c) {
#ifdef __CUDA_ARCH__
  int d;
  asm("mad.hi.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
#else
  return (int)((unsigned)(int)(((long long)a * b) >> 32) + (unsigned)c);
#endif
}
// a b from its two halves: on this chip IMAD.LO + IMAD.HI issue faster than
// the 64-bit IMAD.WIDE (58 and 29 against 14 to 21 per clock and SM)
VK_FIX_HD long long fx_wide(int a, int b) {
  return fx_join(fx_madhi(a, b, 0), (unsigned)a * (unsigned)b);
}
// v = h 2^32 + l with signed l
struct fxsplit { int h, l; };
VK_FIX_HD fxsplit fx_split(long long v) {
  fxsplit s;
  s.l = (int)v;
  s.h = (int)(v >> 32) - (s.l >> 31);
  return s;
}

VK_FIX_HD fx2 fx_add(fx2 a, fx2 b) { return fx2{a.x + b.x, a.y + b.y}; }
VK_FIX_HD fx2 fx_sub(fx2 a, fx2 b) { return fx2{a.x - b.x, a.y - b.y}; }
// times -i (forward) or +i (inverse)
template <bool INV> VK_FIX_HD fx2 fx_rot(fx2 a) { return INV ? fx2{-a.y, a.x} : fx2{a.y, -a.x}; }
VK_FIX_HD fx2 fx_neg(fx2 a) { return fx2{-a.x, -a.y}; }

// Rounding has no preferred direction and keeps zeros: shifts round to nearest
// even, and of the two cross products of an operand a = h 2^32 + l with a factor
// one is floored and the other rounded up, minus the floor of its negative.
// Their means cancel, and a zero operand adds nothing.  A constant that
// returned the floors' mean instead would turn an exact zero into a few units,
// the same in every line, and these add up over the N^2 lines of a grid.
// a w / 2^64, or a conj(w) / 2^64 for INV, of an |a| < 2^62 (so that the sum of
// the four cross terms stays inside a word); the dropped low x low terms are
// below half a unit, of mean zero.  Which of the two is rounded up differs
// between the terms of x and of y: the short components of quarter and twelfth
// turns (low words of 1, fx_stage_twiddle) leave 1/16 or 1/32 of a unit, whose
// signs so alternate over the turns that one butterfly meets.  The products of
// w = 1 are exact where a is a multiple of the factor 2^growth in the table's units
// (the stage before rounds the outputs that meet it so: all inputs of one
// butterfly of a line do).
template <bool INV> VK_FIX_HD fx2 fx_twiddle(fx2 a, fxtw w) {
  const fxsplit x = fx_split(a.x), y = fx_split(a.y);
  const int nc = -w.ch, nh = -w.dh, nl = -w.dl;
  // y's factor in the real part (p) is minus x's in the imaginary part (q)
  const int ph = INV ? w.dh : nh, pl = INV ? w.dl : nl;
  const int qh = INV ? nh : w.dh, ql = INV ? nl : w.dl;
  const int t = fx_madhi(x.h, w.cl, fx_madhi(y.l, ph, 0)) - fx_madhi(x.l, nc, fx_madhi(y.h, ql, 0));
  const int s = fx_madhi(y.h, w.cl, fx_madhi(x.l, qh, 0)) - fx_madhi(y.l, nc, fx_madhi(x.h, pl, 0));
  return fx2{fx_wide(x.h, w.ch) + fx_wide(y.h, ph) + (long long)t, fx_wide(y.h, w.ch) + fx_wide(x.h, qh) + (long long)s};
}
// v plus what makes a floor to a multiple of 2^B round to nearest even
template <int B> VK_FIX_HD long long fx_bump(long long v) {
  return v + (long long)((1 << (B - 1)) - 1 + ((int)((unsigned)v >> B) & 1));
}
// the nearest multiple of 2^B
template <int B> VK_FIX_HD fx2 fx_multiple(fx2 a) {
  return fx2{fx_bump<B>(a.x) & -(1ll << B), fx_bump<B>(a.y) & -(1ll << B)};
}
// a / 2^B (the untwiddled input beside twiddled ones)
template <int B> VK_FIX_HD fx2 fx_shift(fx2 a) { return fx2{fx_bump<B>(a.x) >> B, fx_bump<B>(a.y) >> B}; }
// Plans.  From 192 points on three stages of small radices (up to 12), whose few
// registers let up to three times the warps of a two-stage plan be resident: the
// integer code is bound by latency, not by its instruction count.  (z pass with
// the cross product, ms: N = 256 {24, 16} 2.90, {8, 8, 6} 2.65; N = 128 {12, 16}
// 0.414, {12, 4, 4} 0.375, {6, 8, 4} 0.355.)  Below, two stages: a third one's
// exchange costs about what it gains (N = 64 {12, 8} 0.055, {3, 8, 4} 0.062;
// {6, 4, 4} 0.047, but with the roundings of that time a mean error of its own).
// The first stage has 2^b or 16 c butterflies, so that groups of lanes keep one
// contiguous line.
VK_FIX_HD constexpr int fx_radix0(int L) {
  return L == 8 ? 2 : L == 12 ? 3 : L == 16 ? 4 : L == 24 ? 6 : L == 32 ? 4 : L == 48 ? 6 : L == 64 ? 8 : L == 96 ? 12
       : L == 128 ? 16 : L == 192 ? 6 : L == 256 ? 8 : L == 384 ? 8 : L == 512 ? 8 : L == 768 ? 12 : 0;
}
VK_FIX_HD constexpr bool fx_supported(int L) { return fx_radix0(L) > 0; }
VK_FIX_HD constexpr int fx_stages(int L) { return L >= 192 ? 3 : 2; }
VK_FIX_HD constexpr int fx_radix1(int L) { return fx_stages(L) == 2 ? L / fx_radix0(L) : 8; }
VK_FIX_HD constexpr int fx_radix(int L, int s) {
  return s == 0 ? fx_radix0(L) : s == 1 ? fx_radix1(L) : L / fx_radix0(L) / fx_radix1(L);
}
// log2 of the factor that the twiddles of a later stage (radix up to 8) divide by;
// their components are held in units of 2^-(64 - growth), which makes
// fx_twiddle's a w / 2^64 the scaled product
constexpr int FX_GROWTH = 3;
VK_FIX_HD constexpr int fx_growth(int) { return FX_GROWTH; }
// sum of the growths of a plan's stages: the outputs' exponent above the quantum
VK_FIX_HD constexpr int fx_total_growth(int L) {
  int g = 0;
  for (int s = 1; s < fx_stages(L); ++s) g += fx_radix(L, s) <= 8 ? FX_GROWTH : 64;
  return g;
}
// W_L^m = c - i s (cosine and sine of 2 pi m / L) in units of 2^-62 (host)
inline fxtw fx_make_twiddle(int m, int L, long double c, long double s) {
  const auto words = [](long double v, int& h, int& l) {
    v *= 4611686018427387904.0L;
    const long long q = (long long)(v < 0 ? v - 0.5L : v + 0.5L);
    l = (int)(unsigned)(unsigned long long)q;
    h = (int)((q - (long long)l) >> 32);
  };
  fxtw w;
  words(c, w.ch, w.cl);
  words(-s, w.dh, w.dl);
  if (4 * (m % L) % L == 0) {   // the zeros of quarter turns exactly
    if (2 * (m % L) % L == 0) w.dh = w.dl = 0;
    else w.ch = w.cl = 0;
  }
  return w;
}
// the table's twiddle in the units of a stage of growth g.  Short components
// (other than of w = 1, whose products are exact) get a low word of 1: the term
// that it adds is -1 for negative operands, which makes the rounding up of the other
// term one away from zero.
VK_FIX_HD fxtw fx_stage_twiddle(fxtw w, int g) {
  const bool one = w.ch > 0 && (w.dh | w.dl) == 0;
  const auto shift = [g, one](int& h, int& l) {
    const long long v = ((long long)h * 4294967296ll + l) >> (g - 2);
    l = (int)(unsigned)(unsigned long long)v;
    h = (int)((v - (long long)l) >> 32);
    if (l == INT32_MIN) ++l;   // fx_twiddle negates it
    if (l == 0 && h != 0 && !one) l = 1;
  };
  shift(w.ch, w.cl);
  shift(w.dh, w.dl);
  return w;
}

// Constants k in (0, 1/2) in units of 2^-64: 1 - cos(pi/8), sin(pi/8),
// 1 - sqrt(1/2), 1 - sqrt(3)/2.  Factors above 1/2 are applied as x - x (1 - k),
// so that the constant's high word stays signed.
struct FxConst {
  static constexpr unsigned long long omc = 0x137ca1866b95cebbull, sn = 0x61f78a9abaa58b47ull;
  static constexpr unsigned long long omr2 = 0x4afb0ccc06219b7cull, omr3 = 0x224c28bd3d9aac62ull;
};
template <unsigned long long K, bool NEG> struct FxWords {
  static constexpr long long v = NEG ? -(long long)K : (long long)K;
  static constexpr int l = (int)(unsigned)(unsigned long long)v;
  static constexpr int h = (int)((v - (long long)l) >> 32);
};
// v k
template <unsigned long long K> VK_FIX_HD long long fx_mulc(long long v) {
  using W = FxWords<K, false>;
  const fxsplit s = fx_split(v);
  return fx_wide(s.h, W::h) + (long long)(fx_madhi(s.h, W::l, 0) - fx_madhi(s.l, -W::h, 0));
}
// a exp(-+ 2 pi i M / 16) (INV: +)
template <int M, bool INV> VK_FIX_HD fx2 fx_w16(fx2 a) {
  constexpr int q = ((M + 2) & 15) / 4;          // quarter turns
  constexpr int m = ((M + 2) & 15) - 2 - 4 * q;  // rest in [-2, 2)
  if constexpr (q == 1) a = fx_rot<INV>(a);
  if constexpr (q == 2) a = fx_neg(a);
  if constexpr (q == 3) a = fx_rot<!INV>(a);
  if constexpr (m == 0) {
    return a;
  } else if constexpr (m == -2) {   // sqrt(1/2) (1 +- i): forward exp(+i pi/4)
    const long long u = INV ? a.x + a.y : a.x - a.y, w = INV ? a.y - a.x : a.y + a.x;
    return fx2{u - fx_mulc<FxConst::omr2>(u), w - fx_mulc<FxConst::omr2>(w)};
  } else {
    constexpr bool pos = (m > 0) != INV;   // re = c x + s y, im = c y - s x with s > 0; else the other signs
    using C = FxWords<FxConst::omc, true>;   // c = 1 + C
    using S = FxWords<FxConst::sn, !pos>;
    using T = FxWords<FxConst::sn, pos>;
    const fxsplit x = fx_split(a.x), y = fx_split(a.y);
    const int t = fx_madhi(x.h, C::l, fx_madhi(y.l, S::h, 0)) - fx_madhi(x.l, -C::h, fx_madhi(y.h, T::l, 0));
    const int s = fx_madhi(y.h, C::l, fx_madhi(x.l, T::h, 0)) - fx_madhi(y.l, -C::h, fx_madhi(x.h, S::l, 0));
    return fx2{fx_wide(x.h, C::h) + fx_wide(y.h, S::h) + (long long)t + a.x,
               fx_wide(y.h, C::h) + fx_wide(x.h, T::h) + (long long)s + a.y};
  }
}

// ---------------------------------------------------------------------------
// In-register DFTs, v[k] <- sum_n v[n] exp(-+ 2 pi i n k / RAD), natural order.
// Inputs that are literal zeros (padding) fold away at compile time.
// ---------------------------------------------------------------------------
template <int RAD, bool INV> struct FxDft;

template <bool INV> struct FxDft<2, INV> {
  static VK_FIX_HD void run(fx2* v) {
    const fx2 p = fx_add(v[0], v[1]);
    v[1] = fx_sub(v[0], v[1]);
    v[0] = p;
  }
};
template <bool INV> struct FxDft<3, INV> {
  static VK_FIX_HD void run(fx2* v) {
    const fx2 t = fx_add(v[1], v[2]), d = fx_sub(v[1], v[2]);
    const fx2 h = fx_shift<1>(t);
    const fx2 m = fx_sub(v[0], h);
    const fx2 e{d.x - fx_mulc<FxConst::omr3>(d.x), d.y - fx_mulc<FxConst::omr3>(d.y)};   // sqrt(3)/2 d
    const fx2 r = fx_rot<INV>(e);
    v[0] = fx_add(v[0], t);
    v[1] = fx_add(m, r);
    v[2] = fx_sub(m, r);
  }
};
template <bool INV> struct FxDft<4, INV> {
  static VK_FIX_HD void run(fx2* v) {
    const fx2 a = fx_add(v[0], v[2]), b = fx_sub(v[0], v[2]);
    const fx2 c = fx_add(v[1], v[3]), d = fx_rot<INV>(fx_sub(v[1], v[3]));
    v[0] = fx_add(a, c);
    v[2] = fx_sub(a, c);
    v[1] = fx_add(b, d);
    v[3] = fx_sub(b, d);
  }
};
template <bool INV> struct FxDft<8, INV> {
  static VK_FIX_HD void run(fx2* v) {
    fx2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    FxDft<4, INV>::run(e);
    FxDft<4, INV>::run(o);
    o[1] = fx_w16<2, INV>(o[1]);
    o[2] = fx_rot<INV>(o[2]);
    o[3] = fx_w16<6, INV>(o[3]);
    for (int k = 0; k < 4; ++k) {
      v[k] = fx_add(e[k], o[k]);
      v[k + 4] = fx_sub(e[k], o[k]);
    }
  }
};
// 4 x 4 (Cooley-Tukey): 4-point DFTs over x[b + 4 a], constant twiddles W16^(b k),
// 4-point DFTs over b; output k + 4 j.
template <bool INV> struct FxDft<16, INV> {
  template <int K> static VK_FIX_HD void column(fx2 (*y)[4], fx2* v) {
    fx2 t[4] = {y[0][K], fx_w16<K, INV>(y[1][K]), fx_w16<2 * K, INV>(y[2][K]), fx_w16<3 * K, INV>(y[3][K])};
    FxDft<4, INV>::run(t);
    for (int j = 0; j < 4; ++j) v[K + 4 * j] = t[j];
  }
  static VK_FIX_HD void run(fx2* v) {
    fx2 y[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
#pragma unroll
      for (int a = 0; a < 4; ++a) y[b][a] = v[b + 4 * a];
      FxDft<4, INV>::run(y[b]);
    }
    column<0>(y, v);
    column<1>(y, v);
    column<2>(y, v);
    column<3>(y, v);
  }
};
// 3 x B with B = 2, 4 (coprime: no twiddles): n = B n1 + 3 n2 mod 3B, and
// k = k1 mod 3 = k2 mod B.
template <int B, bool INV> struct FxDft3 {
  static VK_FIX_HD void run(fx2* v) {
    constexpr int R = 3 * B;
    constexpr int e1 = B * (B % 3 == 1 ? 1 : 2);   // 1 mod 3, 0 mod B
    constexpr int e2 = R + 1 - e1;                 // 0 mod 3, 1 mod B
    fx2 y[3][B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      fx2 t[3] = {v[(3 * n2) % R], v[(B + 3 * n2) % R], v[(2 * B + 3 * n2) % R]};
      FxDft<3, INV>::run(t);
      y[0][n2] = t[0];
      y[1][n2] = t[1];
      y[2][n2] = t[2];
    }
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      FxDft<B, INV>::run(y[k1]);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[(e1 * k1 + e2 * k2) % R] = y[k1][k2];
    }
  }
};
template <bool INV> struct FxDft<6, INV> {
  static VK_FIX_HD void run(fx2* v) { FxDft3<2, INV>::run(v); }
};
template <bool INV> struct FxDft<12, INV> {
  static VK_FIX_HD void run(fx2* v) { FxDft3<4, INV>::run(v); }
};
// ---------------------------------------------------------------------------
// Doubles <-> fixed point
// ---------------------------------------------------------------------------
// trunc(v 2^-Q) for K = Q + 1085 and |v| < 2^(Q + 62): the 53-bit mantissa
// left-aligned at bit 62, shifted right by K - exponent.  Zeros (and
// denormals, far below the quantum of a line of normal range) shift out.
VK_FIX_HD long long fx_from_double(int hi, int lo, int k) {
  // k - exponent, from the sign-cleared high word (its mantissa bits add less than one)
  const unsigned r = (((unsigned)k << 20) + 0xfffffu - ((unsigned)hi & 0x7fffffffu)) >> 20;
  const unsigned mh = ((((unsigned)hi << 10) | ((unsigned)lo >> 22)) & 0x3fffffffu) | 0x40000000u;
  unsigned long long m = ((unsigned long long)mh << 32) | ((unsigned)lo << 10);
#ifdef __CUDA_ARCH__
  asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(m), "r"(r));   // clamps at 64
#else
  m = r > 63 ? 0ull : m >> r;
#endif
  const long long s = (long long)(hi >> 31);
  return ((long long)m ^ s) - s;
}

// Bound of a sum of magnitudes, as an exponent K: sum |z| < 2^(K - 1023).  top is
// the largest high word (sign cleared) of the components, sum the float sum of
// fx_relative(larger high word of each z, top): |z| <= sqrt(2) max(|x|, |y|), and
// the truncated magnitudes and the float sum add less than 2^-10 of it.  Exponents
// stay integers, so the whole range of a double is covered.
VK_FIX_HD float fx_relative(int t, int top) {
  t -= (top & 0x7ff00000) - (127 << 20);
  t = (t > 0 ? t : 0) << 3;
#ifdef __CUDA_ARCH__
  return __int_as_float(t);
#else
  float f;
  memcpy(&f, &t, 4);
  return f;
#endif
}
VK_FIX_HD int fx_bound(int top, float sum) {
  sum *= 1.41602f;
  int b;
#ifdef __CUDA_ARCH__
  b = __float_as_int(sum);
#else
  memcpy(&b, &sum, 4);
#endif
  return (top >> 20) + ((b >> 23) & 0xff) - 127 + 1;
}
// Q = K - 1023 - 62, and eb of fx_from_double = K
VK_FIX_HD constexpr int fx_quantum(int k) { return k - 1085; }

}  // namespace vk
