// Host check of what the fixed-point line transform (vk_fix.cuh) does with zeros
// and constants, and of the mean of its rounding errors: every plan, forward and
// inverse, against long double arithmetic.
#include "vk_fix.cuh"

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

using namespace vk;
using LD = long double;
using CL = std::complex<LD>;

static const LD TWO_PI = 6.283185307179586476925286766559005768L;

// one line through the plan of length L
template <int L, bool INV> struct Line {
  static constexpr int ST = fx_stages(L), SHIFT = fx_total_growth(L);
  static constexpr int R0 = fx_radix(L, 0), NB0 = L / R0;
  std::vector<fxtw> tab[3];   // twiddles of a stage, (r, k) at r NS + k
  Line() {
    int ns = 1;
    for (int s = 0; s < ST; ++s) {
      const int rad = fx_radix(L, s);
      for (int i = 0; s > 0 && i < rad * ns; ++i) {
        const int m = (i / ns) * (i % ns) * (L / (ns * rad));
        const LD a = TWO_PI * m / L;
        tab[s].push_back(fx_stage_twiddle(fx_make_twiddle(m, L, cosl(a), sinl(a)), fx_growth(rad)));
      }
      ns *= rad;
    }
  }
  template <int S, int NS> void stages(std::vector<fx2>& v, std::vector<fx2>& o) const {
    constexpr int R = fx_radix(L, S), NB = L / R, G = fx_growth(R);
    constexpr int GN = S + 1 < ST ? fx_growth(fx_radix(L, S + 1)) : 1;
    for (int j = 0; j < NB; ++j) {
      const int k = j % NS;
      fx2 t[R];
      for (int r = 0; r < R; ++r) {
        t[r] = v[j + r * NB];
        if (S > 0) t[r] = r == 0 ? fx_shift<G>(t[r]) : fx_twiddle<INV>(t[r], tab[S][r * NS + k]);
      }
      FxDft<R, INV>::run(t);
      if (S + 1 < ST) t[0] = fx_multiple<GN>(t[0]);
      for (int r = 0; r < R; ++r) o[(j - k) * R + k + r * NS] = t[r];
    }
    v.swap(o);
    if constexpr (S + 1 < ST) stages<S + 1, NS * R>(v, o);
  }
  std::vector<fx2> run(std::vector<fx2> v) const {
    std::vector<fx2> o(L);
    stages<0, 1>(v, o);
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
      k = std::max(k, top == 0 ? 0 : fx_bound(top, sum));
    }
    return k == 0 ? 1023 : k;   // (a line of zeros)
  }
  // doubles to doubles
  std::vector<double> transform(const std::vector<double>& x) const {
    const int k = bound(x), e = fx_quantum(k) + SHIFT;
    std::vector<fx2> v(L);
    for (int p = 0; p < L; ++p) {
      unsigned long long b[2];
      memcpy(b, &x[2 * p], 16);
      v[p] = fx2{fx_from_double((int)(b[0] >> 32), (int)b[0], k), fx_from_double((int)(b[1] >> 32), (int)b[1], k)};
    }
    v = run(v);
    std::vector<double> o(2 * L);
    for (int p = 0; p < L; ++p) {
      o[2 * p] = std::ldexp((double)v[p].x, e);
      o[2 * p + 1] = std::ldexp((double)v[p].y, e);
    }
    return o;
  }
};

static std::vector<CL> dft(const std::vector<CL>& x, bool inv) {
  const int n = (int)x.size();
  std::vector<CL> w(n), o(n);
  for (int m = 0; m < n; ++m) w[m] = CL(cosl(TWO_PI * m / n), (inv ? 1 : -1) * sinl(TWO_PI * m / n));
  for (int p = 0; p < n; ++p)
    for (int q = 0; q < n; ++q) o[p] += x[q] * w[(long)p * q % n];
  return o;
}

// "zeros L INV kind n": outputs that are not what exact arithmetic gives, for
// lines on which no rounding is needed
template <int L, bool INV> void zeros(const Line<L, INV>& line) {
  for (int part = 0; part < 2; ++part) {
    std::vector<double> x(2 * L);
    int bad = 0;
    x[part] = 1.0;   // one entry: every output is that entry
    auto o = line.transform(x);
    for (int p = 0; p < L; ++p) bad += o[2 * p + part] != 1.0 || o[2 * p + 1 - part] != 0.0;
    std::printf("zeros %d %d single%d %d\n", L, (int)INV, part, bad);
    bad = 0;
    for (int p = 0; p < L; ++p) x[2 * p + part] = 1.0;   // a constant: its sum
    o = line.transform(x);
    for (int p = 0; p < L; ++p) bad += o[2 * p + part] != (p == 0 ? (double)L : 0.0) || o[2 * p + 1 - part] != 0.0;
    std::printf("zeros %d %d constant%d %d\n", L, (int)INV, part, bad);
  }
  int bad = 0;
  for (double v : line.transform(std::vector<double>(2 * L))) bad += v != 0.0;
  std::printf("zeros %d %d none %d\n", L, (int)INV, bad);
}

// "sparse L INV kind e": error relative to the norm
template <int L, bool INV> void sparse(const Line<L, INV>& line) {
  for (int kind = 0; kind < 4; ++kind) {
    std::mt19937_64 g(11 + kind);
    std::normal_distribution<double> n;
    LD err = 0, ref = 0;
    for (int rep = 0; rep < 8; ++rep) {
      std::vector<double> x(2 * L);
      const int at = (int)(g() % L);
      for (int p = 0; p < L; ++p) {
        if (kind == 0) x[2 * p] = p == at ? n(g) : 0.0;                       // one real entry
        if (kind == 1) x[2 * p] = n(g);                                       // real
        if (kind == 2) x[2 * p] = 1.0 / 3.0, x[2 * p + 1] = 1e-10 / 3.0;      // constants of two sizes
        if (kind == 3) x[2 * p] = 1.0 / 3.0 + 1e-10 * n(g), x[2 * p + 1] = 1e-10 * n(g);   // a constant and a disturbance
      }
      const auto o = line.transform(x);
      std::vector<CL> c(L);
      for (int p = 0; p < L; ++p) c[p] = CL(x[2 * p], x[2 * p + 1]);
      c = dft(c, INV);
      for (int p = 0; p < L; ++p) {
        err += std::norm(CL(o[2 * p], o[2 * p + 1]) - c[p]);
        ref += std::norm(c[p]);
      }
    }
    std::printf("sparse %d %d %d %.4Le\n", L, (int)INV, kind, std::sqrt(err / ref));
  }
}

// "mean L INV zero worst": mean error of output 0 and the largest of the others
// over many lines, in units of the output.  The transform is linear, so the sum
// of the outputs is compared with the transform of the sum of the lines.
template <int L, bool INV> void mean(const Line<L, INV>& line, int lines) {
  std::mt19937_64 g(9);
  std::vector<__int128> in(2 * L), out(2 * L);
  for (int it = 0; it < lines; ++it) {
    std::vector<fx2> v(L);
    for (auto& q : v) q = fx2{((long long)g() >> 2) / line.R0, ((long long)g() >> 2) / line.R0};
    for (int p = 0; p < L; ++p) in[2 * p] += v[p].x, in[2 * p + 1] += v[p].y;
    v = line.run(v);
    for (int p = 0; p < L; ++p) out[2 * p] += v[p].x, out[2 * p + 1] += v[p].y;
  }
  std::vector<CL> c(L);
  for (int p = 0; p < L; ++p) c[p] = CL((LD)in[2 * p], (LD)in[2 * p + 1]);
  c = dft(c, INV);
  LD zero = 0, worst = 0;
  for (int p = 0; p < L; ++p) {
    const LD u = (LD)(1 << line.SHIFT);
    const LD e = std::max(std::fabs((LD)out[2 * p] - c[p].real() / u), std::fabs((LD)out[2 * p + 1] - c[p].imag() / u));
    (p == 0 ? zero : worst) = std::max(p == 0 ? zero : worst, e / lines);
  }
  std::printf("mean %d %d %.4Lf %.4Lf\n", L, (int)INV, zero, worst);
}

template <int L, bool INV> void one() {
  const Line<L, INV> line;
  zeros(line);
  sparse(line);
  mean(line, 40000);
}
template <int L> void both() {
  one<L, false>();
  one<L, true>();
}

int main() {
  both<8>(); both<12>(); both<16>(); both<24>(); both<32>(); both<48>(); both<64>(); both<96>();
  both<128>(); both<192>(); both<256>(); both<384>(); both<512>(); both<768>();
  return 0;
}
