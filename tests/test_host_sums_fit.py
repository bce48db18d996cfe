"""The products that keep a row's four slice sums as one 64-bit integer do so only where no sum can
leave it: a genotype count is at most 2, a panel value at most 2^40 in units of its last slice."""
import os
import subprocess

from eig_gb300 import build as B

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "gp_geno_tc.h"
int main(int n, char **k)
{
  for (int i = 1; i < n; ++i) printf("%d\n", (int)gp_tc_sums_fit(atoll(k[i])));
}
"""


def test_sums_fit(tmp_path):
    (tmp_path / "fit.cu").write_text(SOURCE)
    exe = str(tmp_path / "fit")
    subprocess.run([B._nvcc(), "-std=c++17", "-I", os.path.join(B.ROOT, "include"), "-I", B.CSRC,
                    "-o", exe, str(tmp_path / "fit.cu")], check=True)
    # a block; the benchmark's panel twice (counts and masks); whole genomes; the largest SNP count
    ks = [64, 2 * 600_000, 1 << 21, 1 << 22, 8_400_000, 1 << 24, 84_000_000, 2 ** 31 - 1]
    out = subprocess.run([exe] + [str(k) for k in ks], check=True, capture_output=True, text=True)
    fits = [int(x) for x in out.stdout.split()]
    assert fits[:2] == [1, 1]
    for k, f in zip(ks, fits):
        assert not f or 2 * 2 ** 40 * k < 2 ** 63, k
