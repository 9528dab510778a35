// Host check of the fixed-point line transform (vk_fix.cuh): every plan against
// a long double DFT (error relative to the line's norm, next to an FFT in
// doubles), and the mean error of every output over many lines.
#include "vk_fix.cuh"

#include <cmath>
#include <complex>
#include <cstdio>
#include <map>
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

// one line through the plan of length L
template <int L, bool INV> struct Line {
  static constexpr int ST = fx_stages(L), SHIFT = fx_total_growth(L);
  static constexpr int R0 = fx_radix(L, 0), NB0 = L / R0;
  std::vector<fxtw> tw;
  Line() : tw(L) {
    for (int m = 0; m < L; ++m) tw[m] = fx_make_twiddle(m, L, cosl(TWO_PI * m / L), sinl(TWO_PI * m / L));
  }
  template <int S, int NS> void stages(std::vector<fx2>& v) const {
    constexpr int R = fx_radix(L, S), NB = L / R, G = fx_growth(R);
    constexpr int GN = S + 1 < ST ? fx_growth(fx_radix(L, S + 1)) : 1;
    std::vector<fx2> o(L);
    for (int j = 0; j < NB; ++j) {
      const int k = j % NS;
      fx2 t[R];
      for (int r = 0; r < R; ++r) {
        t[r] = v[j + r * NB];
        if (S > 0) t[r] = r == 0 ? fx_shift<G>(t[r]) : fx_twiddle<INV>(t[r], fx_stage_twiddle(tw[r * k * (L / (NS * R))], G));
      }
      FxDft<R, INV>::run(t);
      if (S + 1 < ST) t[0] = fx_multiple<GN>(t[0]);
      for (int r = 0; r < R; ++r) o[(j - k) * R + k + r * NS] = t[r];
    }
    v = o;
    if constexpr (S + 1 < ST) stages<S + 1, NS * R>(v);
  }
  std::vector<fx2> run(std::vector<fx2> v) const {
    stages<0, 1>(v);
    return v;
  }
  // the exponent of a line, as the kernels form it
  static int bound(const std::vector<double>& x) {
    int k = 0;
    for (int j = 0; j < NB0; ++j) {
      int top = 0;
      float sum = 0.f;
      auto hi = [&](int p, int c) {
        unsigned long long b;
        memcpy(&b, &x[2 * p + c], 8);
        return (int)(b >> 32) & 0x7fffffff;
      };
      for (int r = 0; r < R0; ++r) top = std::max(top, std::max(hi(j + r * NB0, 0), hi(j + r * NB0, 1)));
      for (int r = 0; r < R0; ++r) sum += fx_relative(std::max(hi(j + r * NB0, 0), hi(j + r * NB0, 1)), top);
      k = std::max(k, fx_bound(top, sum));
    }
    return k;
  }
};

template <typename F> void fft(std::complex<F>* a, int n, int sign) {
  if (n == 1) return;
  const int r = n % 3 == 0 ? 3 : 2, m = n / r;
  std::vector<std::complex<F>> b(n);
  for (int i = 0; i < n; ++i) b[(i % r) * m + i / r] = a[i];
  for (int q = 0; q < r; ++q) fft(&b[q * m], m, sign);
  static std::map<int, std::vector<CL>> tables;
  std::vector<CL>& w = tables[n];
  if (w.empty()) w = roots(n);
  for (int k = 0; k < n; ++k) {
    std::complex<F> s = b[k % m];
    for (int q = 1; q < r; ++q) {
      const CL c = w[(long)q * k % n];
      s += b[q * m + k % m] * std::complex<F>((F)c.real(), (F)(sign < 0 ? c.imag() : -c.imag()));
    }
    a[k] = s;
  }
}

template <int L, bool INV> void accuracy() {
  const Line<L, INV> line;
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
      fft<double>(d.data(), L, INV ? 1 : -1);
      const LD inv = 1.0L / scale;
      for (int p = 0; p < L; ++p) {
        CL s = 0;
        for (int q = 0; q < L; ++q) {
          const CL w = W[(long)p * q % L];
          s += CL(x[2 * q], x[2 * q + 1]) * (INV ? std::conj(w) : w);
        }
        const int e = fx_quantum(k) + line.SHIFT;
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
template <int L, bool INV> void bias() {
  const Line<L, INV> line;
  constexpr int NR = 1500;
  std::mt19937_64 g(9);
  std::vector<LD> sx(L, 0), sy(L, 0);
  LD var = 0;
  for (int it = 0; it < NR; ++it) {
    std::vector<fx2> v(L);
    for (auto& q : v) q = fx2{((long long)g() >> 2) / line.R0, ((long long)g() >> 2) / line.R0};
    const auto o = line.run(v);
    std::vector<CL> d(L);
    for (int p = 0; p < L; ++p) d[p] = CL(v[p].x, v[p].y);
    fft<LD>(d.data(), L, INV ? 1 : -1);
    for (int p = 0; p < L; ++p) {
      const CL e = CL(o[p].x, o[p].y) - d[p] / (LD)(1 << line.SHIFT);
      sx[p] += e.real();
      sy[p] += e.imag();
      var += std::norm(e) / 2;
    }
  }
  const LD sd = std::sqrt(var / ((LD)NR * L)), noise = sd / std::sqrt((LD)NR);
  LD worst = 0;
  for (int p = 0; p < L; ++p) worst = std::max(worst, std::max(std::fabs(sx[p]), std::fabs(sy[p])) / NR);
  std::printf("bias %d %d %.4Lf %.4Lf\n", L, (int)INV, worst, noise);
}

template <int L> void both() {
  accuracy<L, false>();
  accuracy<L, true>();
  bias<L, false>();
  bias<L, true>();
}

int main() {
  both<8>(); both<12>(); both<16>(); both<24>(); both<32>(); both<48>(); both<64>(); both<96>();
  both<128>(); both<192>(); both<256>(); both<384>(); both<512>(); both<768>();
  return 0;
}
