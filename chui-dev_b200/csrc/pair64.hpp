// FP64 kernel of a direct pair, K(r) = (r^2 + eps^2)^(-3/2) - H(t) / (8 r_s^3),
// t = r^2 / (4 r_s^2), with the long-range coefficient
//   H(t) = [erf(q) - 2 q e^-t / sqrt(pi)] / q^3, q = sqrt(t)
//        = (4 / sqrt(pi)) int_0^1 x^2 e^(-t x^2) dx
// as a fitted polynomial: no erf, exp or division per pair. Plain C++ apart
// from the device's approximate rsqrt, so that its accuracy is tested on the host.
#pragma once

#include <cmath>
#include <cstring>
#include <vector>

#ifdef __CUDACC__
#define CHUI_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define CHUI_HOST_DEVICE inline
#endif

namespace chui {

// Terms of the fit: 22 leave less than 1e-16 of H(t_cut) for r_cut / r_s up to
// 5.5 (2e-17 at 5; 20 terms: 3e-16). terms 0: no such fit, the pairs take the
// closed form.
constexpr int kPoly64Terms = 22;
struct PolyH64 {
  int terms = 0;
  double scale = 0.0;             // s = 1 - r^2 scale, in [0, 1] inside r_cut
  double c[kPoly64Terms] = {};    // H(t) / (8 r_s^3) in powers of s
};

// H is a mean of decaying exponentials: in powers of its distance from the far
// end of the interval, s = 1 at r = 0 and 0 beyond r_cut, its terms are
// positive and nothing cancels, so the polynomial's rounding is relative to H
// at every distance. (In powers of r^2 about the middle of the interval it is an
// absolute 1e-16 of H(0), which near r_cut is 2 to 4 times the closed form's.)
// Chebyshev interpolation in long double; accepted when the coefficients left
// out sum to less than 1.5e-16 of H(t_cut).
inline PolyH64 fitPoly64(double rs, double cutoff) {
  constexpr int m = kPoly64Terms, nodes = 32;
  const long double pi = 3.141592653589793238462643383279502884L;
  PolyH64 p;
  p.scale = static_cast<double>(1.0L / (static_cast<long double>(cutoff) * cutoff * (1.0L + 1.0e-5L)));
  const long double k8 = 0.125L / (static_cast<long double>(rs) * rs * rs);
  if (!std::isnormal(p.scale) || !std::isnormal(static_cast<double>(k8))) return PolyH64();
  // H(t) = (4/sqrt(pi)) e^-t sum_k (2t)^k / (3 5 ... (2k+3)): positive terms
  auto exactH = [&](long double t) {
    long double sum = 0.0L, term = 1.0L / 3.0L;
    for (int k = 1; k < 400 && term > 1e-22L * sum; ++k) {
      sum += term;
      term *= 2.0L * t / (2.0L * k + 3.0L);
    }
    return 4.0L / std::sqrt(pi) * std::exp(-t) * sum;
  };
  long double f[nodes], cheb[nodes], cosine[4 * nodes];
  for (int i = 0; i < 4 * nodes; ++i) cosine[i] = std::cos(pi * i / (2.0L * nodes));
  for (int k = 0; k < nodes; ++k) {
    const long double s = 0.5L * (cosine[2 * k + 1] + 1.0L);
    f[k] = k8 * exactH((1.0L - s) / p.scale / (4.0L * static_cast<long double>(rs) * rs));
  }
  for (int j = 0; j < nodes; ++j) {
    long double sum = 0.0L;
    for (int k = 0; k < nodes; ++k) sum += f[k] * cosine[j * (2 * k + 1) % (4 * nodes)];
    cheb[j] = (j == 0 ? 1.0L : 2.0L) * sum / nodes;
  }
  long double left_out = 0.0L;
  for (int j = m; j < nodes; ++j) left_out += std::fabs(cheb[j]);
  const long double end = k8 * exactH(1.0L / p.scale / (4.0L * static_cast<long double>(rs) * rs));
  if (!(left_out <= 1.5e-16L * end) || !std::isnormal(static_cast<double>(end))) return PolyH64();
  // shifted Chebyshev polynomials T_j(2 s - 1) in powers of s
  std::vector<long double> before(m, 0.0L), now(m, 0.0L), next(m, 0.0L), sum(m, 0.0L);
  before[0] = 1.0L;
  now[0] = -1.0L;
  now[1] = 2.0L;
  for (int i = 0; i < m; ++i) sum[i] = cheb[0] * before[i] + cheb[1] * now[i];
  for (int j = 2; j < m; ++j) {
    for (int i = 0; i < m; ++i) next[i] = (i > 0 ? 4.0L * now[i - 1] : 0.0L) - 2.0L * now[i] - before[i];
    before = now;
    now = next;
    for (int i = 0; i < m; ++i) sum[i] += cheb[j] * now[i];
  }
  for (int i = 0; i < m; ++i) p.c[i] = static_cast<double>(sum[i]);
  p.terms = m;
  return p;
}

// 1/sqrt(d) to about 20 bits, the low half of its mantissa zero (its square is exact).
CHUI_HOST_DEVICE double shortRsqrt(double d) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  return y;
#else
  unsigned long long bits;
  const double y = 1.0 / std::sqrt(d);
  std::memcpy(&bits, &y, 8);
  bits &= 0xFFFFFFFF00000000ull;
  double out;
  std::memcpy(&out, &bits, 8);
  return out;
#endif
}

// The short rsqrt and the series take 10 FP64 operations, where rsqrt of a
// double with a residual of its own took about 19 (262 k particles: 4.27 against
// 4.79 ms a solve; 4.35 with one Newton step, whose cube is 1.8 times as far off).
// (r^2 + eps^2)^(-3/2) - H(t) / (8 r_s^3), d = r^2 + eps^2 > 0. From y near d^(-1/2)
// with y^2 and so e = 1 - d y^2 exact, d^(-3/2) = y^3 (1 - e)^(-3/2) is the binomial
// series 1 + 3/2 e + 15/8 e^2 + 35/16 e^3 + ... (e below 2^-17: the rest is below
// 2^-66); y^3 in two parts, and the sum with -H rounded at its end.
CHUI_HOST_DEVICE double softMinusLong64(double r2, double eps, double scale, const double* c) {
  const double s = fma(-r2, scale, 1.0);
  double h = c[kPoly64Terms - 1];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int j = kPoly64Terms - 2; j >= 0; --j) h = fma(h, s, c[j]);
  const double d = fma(eps, eps, r2);
  const double y = shortRsqrt(d);
  const double y2 = y * y;
#ifdef __CUDA_ARCH__
  const double y3 = __dmul_rn(y2, y);  // rounded: never fused into the sum
#else
  const double y3 = y2 * y;
#endif
  const double y3_lo = fma(y2, y, -y3);
  const double e = fma(-d, y2, 1.0);
  const double more = e * fma(e, fma(e, 2.1875, 1.875), 1.5);
  return y3 + (fma(y3, more, y3_lo) - h);
}

}  // namespace chui
