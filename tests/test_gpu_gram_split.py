"""The split Gram where its last wave of tiles is cut along the SNPs: against the FP64 Gram.

Tolerance of an entry, relative to sqrt(G_ii G_jj) >= sum |x_i x_j|: lo lo is left out (2^-22 of a
product with fp16, 2^-16 with bf16), and an FP32 accumulator takes 24 truncated sums per 128 SNPs
(2^-23 of the running value each); everything above is summed in 48 bits or more."""
import numpy as np
import pytest

from eig_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,lolo", [(native.GP_PREC_SPLIT_FP16, 2.0**-22),
                                       (native.GP_PREC_SPLIT_BF16, 2.0**-16)])
@pytest.mark.parametrize("n,m", [
    (100, 8192),     # one tile, two parts
    (129, 8191),     # just too few SNPs for parts
    (257, 40961),    # six tiles, ten parts, the last fold one SNP
    (1000, 16500),   # 36 tiles in four parts
    (2200, 9000),    # 152 whole tiles, then 19 in two parts
])
def test_split_gram_parts(gpu, n, m, prec, lolo, monkeypatch):
    r = np.random.default_rng(n + m)
    f = r.uniform(0.05, 0.95, m)
    g = r.binomial(2, f[:, None], (m, n)).astype(np.uint8)
    g[r.random((m, n)) < 0.02] = 3
    rec = np.full((m, (n + 3) // 4 * 4), 3, np.uint8)
    rec[:, :n] = g
    rec = (rec[:, 0::4] << 6) | (rec[:, 1::4] << 4) | (rec[:, 2::4] << 2) | rec[:, 3::4]
    gpu.load_genotypes(rec, n)
    gpu.set_samples(np.arange(n))
    gpu.set_snps(np.arange(m))
    want = gpu.xtx(precision=native.GP_PREC_FP64)["XTX"]
    d = np.sqrt(np.diag(want))
    tol = lolo + 24 * 2.0**-23
    got = gpu.xtx(precision=prec)["XTX"]
    assert np.max(np.abs(got - want) / np.outer(d, d)) <= tol
    assert np.array_equal(got, got.T)
    assert np.array_equal(got, gpu.xtx(precision=prec)["XTX"])
    # super-chunks: parts of a second pass added to the first's
    monkeypatch.setenv("GP_BF16_BUDGET_BYTES", str((n + 127) // 128 * 128 * 4 * 8320))
    got = gpu.xtx(precision=prec)["XTX"]
    assert np.max(np.abs(got - want) / np.outer(d, d)) <= tol
