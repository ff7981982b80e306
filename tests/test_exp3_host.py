"""The SU(3) exponential on the host, both sides of the norm that separates its two series,
against a long-double Taylor series: 3e-16 per entry (a few roundings of numbers of order 1)."""
import os
import subprocess

SRC = r'''
#include <complex>
#include <cstdio>
#include <random>
#include "gh_math.cuh"
using namespace ghm;
typedef std::complex<long double> cl;
int main() {
  std::mt19937_64 g(3);
  std::normal_distribution<double> n;
  const double norms[] = {0.0, 1e-6, 0.0625, 0.15, 0.1999, 0.2001, 0.3, 0.49};
  double worst = 0;
  for (int t = 0; t < 40000; ++t) {
    double v[8], m = 0;
    for (double& x : v) { x = n(g); m += x * x; }
    for (double& x : v) x *= norms[t % 8] * std::sqrt(2 / m);      // ||sum v_a T^a||_F = |v| / sqrt 2
    const Mat<3, double> H = alg_to_mat<3, double>(v), E = expi<3, double>(H);
    cl A[9], T[9], S[9];
    for (int i = 0; i < 9; ++i) { A[i] = cl(-H.e[i].im, H.e[i].re); T[i] = S[i] = i % 4 == 0; }
    for (int k = 1; k < 30; ++k) {
      cl N[9];
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
          cl z = 0;
          for (int q = 0; q < 3; ++q) z += T[i * 3 + q] * A[q * 3 + j];
          N[i * 3 + j] = z / (long double)k;
        }
      for (int i = 0; i < 9; ++i) { T[i] = N[i]; S[i] += N[i]; }
    }
    for (int i = 0; i < 9; ++i) worst = std::max(worst, (double)std::abs(S[i] - cl(E.e[i].re, E.e[i].im)));
  }
  std::printf("%.3e\n", worst);
}
'''


def test_exponential(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + os.path.join(root, "gauge_higgs_b200", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    assert float(subprocess.run([exe], capture_output=True, text=True, check=True).stdout) < 3e-16
