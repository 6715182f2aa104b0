"""Arithmetic that the kernels share with a host program built from the same
headers: the vertical modes of the wavemaker potential by rotations (modes.h), the
division by an order (division.h)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hos-nwt_gb300", "csrc")
INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def _run(tmp_path, program):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(program)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", INC,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout


MODES = r"""
#include <cmath>
#include <cstdio>
#include "modes.h"
static const long double kPi = 3.14159265358979323846264338327950288L;
int main() {
  // runs of 32 of up to 512 modes, elevations of +-0.16 depths
  const int N = 512, P = 2000;
  auto f = [](double x, double* s, double* c) {
    *s = (double)sinl(kPi * (long double)x);
    *c = (double)cosl(kPi * (long double)x);
  };
  const int b[] = {0, 4, 8, 16, 32, 64, 128, 512};
  long double rot[7] = {}, direct[7] = {}, most = 0;
  unsigned long long seed = 1;
  for (int p = 0; p < P; ++p) {
    seed = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    const double e = 1.0 + 0.32 * ((double)(seed >> 11) / 9007199254740992.0 - 0.5);
    double s = 0, c = 0, s2, c2;
    hos::mode_start(0.5, e, f, s2, c2);
    for (int i = 0, q = 0; i < N; ++i) {
      if (i % 32 == 0) hos::mode_start((2 * i + 1) * 0.25, e, f, s, c);
      else hos::mode_next(s2, c2, s, c);
      if (i == b[q + 1]) ++q;
      const long double a = (2 * i + 1) * (kPi / 4) * (long double)e;
      const double x = (2 * (i + 1) - 1) * (3.141592653589793 / 4.0) * e;
      const long double ds = s - sinl(a), dc = c - cosl(a), xs = std::sin(x) - sinl(a), xc = std::cos(x) - cosl(a);
      rot[q] += ds * ds + dc * dc;
      direct[q] += xs * xs + xc * xc;
      most = fmaxl(most, fmaxl(fabsl(ds), fabsl(dc)));
    }
  }
  bool ok = most < 1.6e-14L;
  for (int q = 0; q < 7; ++q) {
    const long double n = 2.0L * P * (b[q + 1] - b[q]);
    std::printf("modes %d to %d: rotations %.2Le, direct %.2Le\n", b[q], b[q + 1], sqrtl(rot[q] / n), sqrtl(direct[q] / n));
    ok = ok && rot[q] <= direct[q];
  }
  std::printf("largest %.2Le\n", most);
  return ok ? 0 : 1;
}
"""


def test_modes_by_rotations(tmp_path):
    """No block of modes is further from the series, in the mean square, than the
    direct cos(kx_add e) is; and no mode by more than 32 rotations can err (two
    rounded factors and three roundings of 2^-53 each, 5e-16: 1.6e-14)."""
    _run(tmp_path, MODES)


DIVISION = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "division.h"
static double bits(unsigned long long b) {
  double v;
  std::memcpy(&v, &b, 8);
  return v;
}
int main() {
  unsigned long long bad = 0, n = 0, seed = 7;
  auto look = [&](double v, double d) {
    const double a = hos::div_by(v, d, 1.0 / d), b = v / d;
    bad += std::memcmp(&a, &b, 8) != 0 && !(a != a && b != b);
    ++n;
  };
  for (int d = 1; d <= 17; ++d) {
    // exponents on both sides of the limit, the ends of the range, what is not finite
    for (unsigned long long e : {0ULL, 1ULL, 2ULL, 53ULL, 62ULL, 63ULL, 64ULL, 65ULL, 1000ULL, 1022ULL, 1023ULL, 1500ULL, 2045ULL, 2046ULL, 2047ULL})
      for (int k = 0; k < 4000; ++k) {
        seed = seed * 6364136223846793005ULL + 1442695040888963407ULL;
        const unsigned long long m = k == 0 ? 0 : (k == 1 ? 0xfffffffffffffULL : seed >> 12);
        look(bits((e << 52) | m), d);
        look(bits((1ULL << 63) | (e << 52) | m), d);
      }
    // quotients next to the middle of two doubles, and exact ones
    for (int k = 0; k < 20000; ++k) {
      seed = seed * 6364136223846793005ULL + 1442695040888963407ULL;
      const double q = bits((1023ULL << 52) | (seed >> 12));
      const double v = q * d, w = std::fma(q, (double)d, 0x1p-53 * d);
      for (double x : {v, w, std::nextafter(v, 0.0), std::nextafter(v, 99.0), std::nextafter(w, 0.0), std::nextafter(w, 99.0)}) look(x, d);
    }
  }
  std::printf("%llu of %llu differ\n", bad, n);
  return bad != 0;
}
"""


def test_division_by_an_order(tmp_path):
    """The bits of v / d for d = 1 to 17."""
    _run(tmp_path, DIVISION)
