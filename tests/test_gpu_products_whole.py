"""Products of a code operand with so many row tiles that none is split along k: the kernel writes
them itself, from one chunk of sums or from several (above 8,192 samples), for a last row tile and
a last column group only partly used.  SNP weights against numpy on every 50th SNP.

Tolerance per SNP and vector: 10 fancy x (allele counts and mean, both <= 2) x n samples x the
slices' 2^-41 of the vector's largest entry, twice for the two products; FP64 rounding below it."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,k", [(300, 130000, 3), (300, 130049, 5), (1200, 120001, 4),
                                   (8300, 60000, 2)])
def test_weights(gpu, n, m, k):
    rec, pop = native.synth_records(m, [n // 2, n - n // 2], [0.02, 0.03], miss=0.01, seed=n + k,
                                    nthreads=4)
    gpu.load_genotypes(rec, n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(m, dtype=np.int32))
    gpu.xtx(precision=native.GP_PREC_SPLIT_FP16, want_xtx=False)
    _, V = gpu.eigvecs(k)
    ff = gpu.snp_weights(k)[0]
    sub = np.arange(0, m, 50)
    g = O.unpack(rec[sub], n).astype(np.float64)
    seen = (g >= 0) & (g != 3)
    cnt = np.where(seen, g, 0).sum(1)
    mean = cnt / np.maximum(seen.sum(1), 1)
    p = mean / 2
    fancy = np.where(p * (1 - p) > 0, 1 / np.sqrt(np.where(p * (1 - p) > 0, p * (1 - p), 1)), 0)
    X = np.where(seen, g - mean[:, None], 0) * fancy[:, None]
    want = 10 * V @ X.T
    tol = 10 * fancy * 2 * n * 2 * 2.0**-41 * np.max(np.abs(V), axis=1)[:, None] + 1e-12
    assert np.all(np.abs(ff[:, sub] - want) <= tol)
