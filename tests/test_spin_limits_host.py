"""Shared memory of k_gen_spin on the host: for every n it accepts, the force's partial sums (3
doubles per warp and lane) lie inside the entries of D, which is read by then, and n = 4 to 17
(the largest a context builds) are accepted."""
import os
import shutil
import subprocess

SRC = r'''
#include <cstdio>
#include "gh_kernels.cuh"
using namespace ghk;
int main() {
  for (int n = 1; n < 40; ++n)
    std::printf("%d %d %zu %d %zu\n", n, (int)spin_fits(n), sizeof(double) * 3 * SPIN_WARPS * 32, spin_entries(n) * 32 * 16, spin_smem(n));
}
'''


def test_partial_sums_stay_inside_d(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    (tmp_path / "t.cu").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-I" + os.path.join(root, "gauge_higgs_b200", "csrc"), str(tmp_path / "t.cu"), "-o", exe],
                   check=True, capture_output=True)
    rows = [[int(x) for x in line.split()] for line in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    for n, fits, sums, entries, total in rows:
        assert not fits or (sums <= entries and total <= 227 * 1024)
    assert [n for n, fits, *_ in rows if fits][:14] == list(range(4, 18))
