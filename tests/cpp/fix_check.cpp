// Host check of the fixed-point line transform (vk_fix.cuh): every plan against
// a long double DFT (error relative to the line's norm, next to an FFT in
// doubles), and the mean error of every output over many lines.
#include "vk_fix.cuh"

#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

using namespace vk;
using LD = long double;
using CL = std::complex<LD>;
using CD = std::complex<double>;

static const LD TWO_PI = 6.283185307179586476925286766559005768L;

static std::vector<CL> roots(int L) {
  std::vector<CL> w(L);
  for (int m = 0; m < L; ++m) w[m] = CL(cosl(TWO_PI * m / L), -sinl(TWO_PI * m / L));
  return w;
}

template <int R0, int R1, bool INV> struct Line {
  static constexpr int L = R0 * R1, G = fx_growth(R1);
  std::vector<fxtw> tw;
  Line() : tw(L) {
    const auto w = roots(L);
    for (int m = 0; m < L; ++m) {
      fx_words(w[m].real(), 64 - G, tw[m].ch, tw[m].cl);
      fx_words(w[m].imag(), 64 - G, tw[m].dh, tw[m].dl);
    }
  }
  template <int R> void twiddle(fx2* t, int j) const {
    if constexpr (R < R1) {
      t[R] = fx_twiddle<INV>(t[R], tw[R * j % L], FxSpecial<R0, R1>::template round0<R>(j));
      twiddle<R + 1>(t, j);
    }
  }
  std::vector<fx2> run(const std::vector<fx2>& v) const {
    std::vector<fx2> w(L), o(L);
    for (int j = 0; j < R1; ++j) {
      fx2 t[R0];
      for (int r = 0; r < R0; ++r) t[r] = v[j + r * R1];
      FxDft<R0, INV>::run(t);
      for (int r = 0; r < R0; ++r)
        w[j * R0 + r] = FxSpecial<R0, R1>::output(r) ? fx_multiple<G + 1>(t[r]) : t[r];
    }
    for (int j = 0; j < R0; ++j) {
      fx2 t[R1];
      for (int r = 0; r < R1; ++r) t[r] = w[j + r * R0];
      t[0] = fx_shift<G>(t[0]);
      twiddle<1>(t, j);
      FxDft<R1, INV>::run(t);
      for (int r = 0; r < R1; ++r) o[j + r * R0] = t[r];
    }
    return o;
  }
  // the exponent of a line, as the kernels form it
  static int bound(const std::vector<double>& x) {
    int k = 0;
    for (int j = 0; j < R1; ++j) {
      int top = 0;
      float sum = 0.f;
      auto hi = [&](int p, int c) {
        unsigned long long b;
        memcpy(&b, &x[2 * p + c], 8);
        return (int)(b >> 32) & 0x7fffffff;
      };
      for (int r = 0; r < R0; ++r) top = std::max(top, std::max(hi(j + r * R1, 0), hi(j + r * R1, 1)));
      for (int r = 0; r < R0; ++r) sum += fx_relative(std::max(hi(j + r * R1, 0), hi(j + r * R1, 1)), top);
      k = std::max(k, fx_bound(top, sum));
    }
    return k;
  }
};

static void fft_double(CD* a, int n, int sign) {
  if (n == 1) return;
  const int r = n % 3 == 0 ? 3 : 2, m = n / r;
  std::vector<CD> b(n);
  for (int i = 0; i < n; ++i) b[(i % r) * m + i / r] = a[i];
  for (int q = 0; q < r; ++q) fft_double(&b[q * m], m, sign);
  for (int k = 0; k < n; ++k) {
    CD s = b[k % m];
    for (int q = 1; q < r; ++q) {
      const LD an = sign * TWO_PI * ((long)q * k % n) / n;
      s += b[q * m + k % m] * CD((double)cosl(an), (double)sinl(an));
    }
    a[k] = s;
  }
}

template <int R0, int R1, bool INV> void accuracy() {
  const Line<R0, R1, INV> line;
  constexpr int L = R0 * R1;
  const auto W = roots(L);
  for (int kind = 0; kind < 5; ++kind) {
    std::mt19937_64 g(5 + kind);
    std::normal_distribution<double> n;
    LD fix = 0, dbl = 0, ref = 0;
    for (int rep = 0; rep < 4; ++rep) {
      std::vector<double> x(2 * L);
      const double scale = std::ldexp(1.0, 200 * (rep - 1));
      for (int p = 0; p < L; ++p) {
        const double k = p < L / 2 ? p : L - p;
        const double amp = kind == 0 ? 1 : kind == 1 ? std::pow(1 + k, -3) : kind == 2 ? std::exp(-0.3 * k)
                         : kind == 3 ? (p == 3 ? 1 : 1e-9) : (k < L / 3 ? 1 : 0);
        x[2 * p] = scale * amp * n(g);
        x[2 * p + 1] = scale * amp * n(g);
      }
      const int k = line.bound(x);
      std::vector<fx2> v(L);
      for (int p = 0; p < L; ++p) {
        unsigned long long b[2];
        memcpy(b, &x[2 * p], 16);
        v[p] = fx2{fx_from_double((int)(b[0] >> 32), (int)b[0], k), fx_from_double((int)(b[1] >> 32), (int)b[1], k)};
      }
      const auto o = line.run(v);
      std::vector<CD> d(L);
      for (int p = 0; p < L; ++p) d[p] = CD(x[2 * p], x[2 * p + 1]);
      fft_double(d.data(), L, INV ? 1 : -1);
      const LD inv = 1.0L / scale;
      for (int p = 0; p < L; ++p) {
        CL s = 0;
        for (int q = 0; q < L; ++q) {
          const CL w = W[(long)p * q % L];
          s += CL(x[2 * q], x[2 * q + 1]) * (INV ? std::conj(w) : w);
        }
        const int e = fx_quantum(k) + line.G;
        const CL f((double)std::ldexp((double)o[p].x, e), (double)std::ldexp((double)o[p].y, e));
        fix += std::norm((f - s) * inv);
        dbl += std::norm((CL(d[p].real(), d[p].imag()) - s) * inv);
        ref += std::norm(s * inv);
      }
    }
    std::printf("accuracy %d %d %d %.4Le %.4Le\n", L, (int)INV, kind, std::sqrt(fix / ref), std::sqrt(dbl / ref));
  }
}

// mean error of each output over many lines, in standard errors of that mean
template <int R0, int R1, bool INV> void bias() {
  const Line<R0, R1, INV> line;
  constexpr int L = R0 * R1, NR = 1500;
  const auto W = roots(L);
  std::mt19937_64 g(9);
  std::vector<LD> sx(L, 0), sy(L, 0);
  LD var = 0;
  for (int it = 0; it < NR; ++it) {
    std::vector<fx2> v(L);
    for (auto& q : v) q = fx2{((long long)g() >> 2) / L, ((long long)g() >> 2) / L};
    const auto o = line.run(v);
    std::vector<CL> B(L);
    for (int j = 0; j < R1; ++j)
      for (int k = 0; k < R0; ++k) {
        CL s = 0;
        for (int r = 0; r < R0; ++r) {
          const CL w = W[r * k % R0 * (L / R0)];
          s += CL(v[j + r * R1].x, v[j + r * R1].y) * (INV ? std::conj(w) : w);
        }
        const CL w = W[j * k % L];
        B[j * R0 + k] = s * (INV ? std::conj(w) : w) / (LD)(1 << line.G);
      }
    for (int j = 0; j < R0; ++j)
      for (int k = 0; k < R1; ++k) {
        CL s = 0;
        for (int r = 0; r < R1; ++r) {
          const CL w = W[r * k % R1 * (L / R1)];
          s += B[j + r * R0] * (INV ? std::conj(w) : w);
        }
        const CL e = CL(o[j + k * R0].x, o[j + k * R0].y) - s;
        sx[j + k * R0] += e.real();
        sy[j + k * R0] += e.imag();
        var += std::norm(e) / 2;
      }
  }
  const LD se = std::sqrt(var / ((LD)NR * L) / NR);
  LD worst = 0;
  for (int p = 0; p < L; ++p) worst = std::max(worst, std::max(std::fabs(sx[p]), std::fabs(sy[p])) / NR / se);
  std::printf("bias %d %d %.3Lf\n", L, (int)INV, worst);
}

template <int L> void both() {
  constexpr int R0 = fx_radix(L, 0), R1 = L / R0;
  accuracy<R0, R1, false>();
  accuracy<R0, R1, true>();
  bias<R0, R1, false>();
  bias<R0, R1, true>();
}

int main() {
  both<8>(); both<12>(); both<16>(); both<24>(); both<32>(); both<48>(); both<64>(); both<96>();
  both<128>(); both<192>(); both<256>(); both<384>(); both<512>(); both<768>();
  return 0;
}
