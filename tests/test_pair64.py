"""The FP64 pair kernel's polynomial form (csrc/pair64.hpp, compiled for the host)
against the closed form with erf and exp that it stands in for: each one's rms
error against long double, over the distances inside r_cut."""
import os
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "pair64.hpp"
using LD = long double;
static const LD kPi = 3.141592653589793238462643383279502884L;
static LD longRange(LD r2, LD rs) {
  LD t = r2 / (4 * rs * rs), sum = 0, term = 1.0L / 3;
  for (int k = 1; k < 400; ++k) { sum += term; term *= 2 * t / (2 * k + 3.0L); }
  return 4 / std::sqrt(kPi) * std::exp(-t) * sum / (8 * rs * rs * rs);
}
// the closed form: series below q = 1/8, else erf and exp
static double closed(double r2, double eps, double rs) {
  const double s2 = std::fma(eps, eps, r2), r = std::sqrt(r2), q = 0.5 * r / rs, t = q * q;
  const double series = 2.25675833419102514779231780624309034 *
      (1.0 / 3 + t * (-1.0 / 5 + t * (1.0 / 14 + t * (-1.0 / 54 + t * (1.0 / 264 + t * (-1.0 / 1560 + t * (1.0 / 10800 - t / 85680)))))));
  const double k = q < 0.125 ? ((0.125 * series / rs) / rs) / rs
      : (((std::erf(q) - 2.0 * 0.564189583547756286948079451560772586 * q * std::exp(-q * q)) / r) / r) / r;
  return 1.0 / (s2 * std::sqrt(s2)) - k;
}
int main(int argc, char** argv) {
  const double rs = std::atof(argv[1]), ratio = std::atof(argv[2]), eps = std::atof(argv[3]) * rs, cut = ratio * rs;
  const chui::PolyH64 p = chui::fitPoly64(rs, cut);
  std::printf("%d\n", p.terms);
  if (p.terms == 0) return 0;
  unsigned long long state = 12345;
  const int bands = 24, each = 2000;
  for (int b = 0; b < bands; ++b) {
    const double lo = cut * std::pow(0.005, (bands - b) / (double)bands), hi = cut * std::pow(0.005, (bands - b - 1) / (double)bands);
    LD ec = 0, ep = 0;
    for (int i = 0; i < each; ++i) {
      state = state * 6364136223846793005ull + 1442695040888963407ull;
      const double r = lo + (hi - lo) * (double)(state >> 11) / 9007199254740992.0, r2 = r * r;
      const LD d = (LD)eps * eps + r2, truth = 1 / (d * std::sqrt(d)) - longRange(r2, rs);
      const LD c = closed(r2, eps, rs) - truth, q = chui::softMinusLong64(r2, eps, p.scale, p.c) - truth;
      ec += c * c; ep += q * q;
    }
    std::printf("%.6g %.6g %.6g\n", hi / rs, (double)std::sqrt(ec / each), (double)std::sqrt(ep / each));
  }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair64")
    (d / "pair64_test.cpp").write_text(SOURCE)
    exe = d / "pair64_test"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{os.path.join(ROOT, 'chui-dev_b200', 'csrc')}",
                    str(d / "pair64_test.cpp"), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("ratio", [1.0, 3.0, 4.5, 5.0, 5.5])
@pytest.mark.parametrize("eps", [0.0, 0.01, 0.1, 0.5, 1.0])
@pytest.mark.parametrize("rs", [1.0, 0.0137])
def test_no_further_off_than_the_closed_form(program, ratio, eps, rs):
    """In every band of distances, softenings up to r_s."""
    lines = subprocess.run([program, str(rs), str(ratio), str(eps)], check=True, capture_output=True, text=True).stdout.split("\n")
    assert int(lines[0]) == 22
    for line in lines[1:-1]:
        r, closed, poly = (float(v) for v in line.split())
        assert poly <= closed, (r, closed, poly)


@pytest.mark.parametrize("rs,ratio", [(1.0, 7.0), (1.0, 14.0), (1.0, 1e6), (1e-120, 5.0), (1e120, 5.0), (1.0, 1e200)])
def test_closed_form_where_no_fit_holds(program, rs, ratio):
    out = subprocess.run([program, str(rs), str(ratio), "0.1"], check=True, capture_output=True, text=True).stdout
    assert int(out.split("\n")[0]) == 0
