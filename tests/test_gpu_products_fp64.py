"""Weights, scores and lsqproject of the FP64 precision: the products with 12-bit slices at the
edges of their tiles, column groups and k ranges, against the oracle on the same vectors."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def panel(n, m, miss, seed):
    r = np.random.default_rng(seed)
    p = r.uniform(0.05, 0.95, m)
    g = (r.random((m, n)) < p[:, None]).astype(np.int8) + (r.random((m, n)) < p[:, None])
    g[r.random((m, n)) < miss] = -1
    return O.pack(g)


# K = 25: 126 slice columns; 26: 130, two tiles; lsqproject's panel has K (K + 1) / 2 + 1 columns:
# K = 22 gives 254, 23 gives 277 (two groups of 256), 64 gives 2,081 (nine)
@pytest.mark.parametrize("n,m,K,subset", [(40, 63, 1, False), (127, 400, 6, True),
                                          (128, 1024, 22, False), (129, 1100, 23, True),
                                          (130, 4097, 25, False), (257, 900, 26, True),
                                          (200, 2500, 64, True)])
def test_products(gpu, n, m, K, subset):
    rec = panel(n, m, 0.04, n + m)
    rows = np.arange(n, dtype=np.int32)
    if subset:
        rows = rows[rows % 7 != 2]
    cols = np.arange(m, dtype=np.int32)
    gpu.load_genotypes(rec, n)
    gpu.set_samples(rows)
    gpu.set_snps(cols)
    gpu.xtx()
    _, V = gpu.eigvecs(K)
    ff, fx, sc = gpu.snp_weights(K)
    s = O.pass_columns(rec, cols, rows)
    off, ofx, osc = O.weights(s, V, K)
    u = 2.0 ** -53
    nr = len(rows)
    tab = s.tab.reshape(-1, 4)
    code = O.unpack(rec, n)
    v = np.take_along_axis(tab, np.where(code < 0, 3, code)[:, rows], axis=1)
    # ff = f (G W) - xmean (O W), |W| = 10: FP64 sums of nr terms on one side; on the other a few
    # roundings of the two products, |G W| <= 20 sqrt(nr), and of the slices
    tff = (2 * nr * u * 10 * np.sqrt((v * v).sum(1))
           + 16 * u * 20 * np.sqrt(nr) * (np.abs(s.xfancy) + np.abs(s.xmean)))
    assert np.all(np.abs(ff - off) <= tff[None, :])
    # fx: sums over m SNPs of x ff, x within 3 / sqrt(p (1-p)); plus the difference of the ff
    x = np.abs(s.xfancy) * 2 + np.abs(s.xmean)
    tfx = 2 * m * u * (x[None, :] * np.abs(off)).sum(1) + (x * tff).sum()
    assert np.all(np.abs(fx - ofx) <= tfx[:, None])
    proj = np.arange(n, dtype=np.int32)
    a, b, nobs, st = gpu.lsqproj(K, proj)
    oa, ob, onobs, ost = O.lsqproj(s, ff, sc, K, proj)
    assert np.array_equal(nobs, onobs)
    E = ff * sc[:, None] * (s.killed == 0)
    tb = 4 * m * u * (x[None, :] * np.abs(E)).sum(1)
    ok = st == 0
    assert np.all(np.abs(b - ob)[:, ok] <= tb[:, None])
    # each solution's residual in the oracle's normal equations: the sums' and the Cholesky
    # solve's backward errors
    for q in np.flatnonzero(ok)[:: max(1, n // 16)]:
        co = (E * (code[:, q] >= 0)) @ E.T
        size = np.trace(co)
        res = co @ a[:, q] - ob[:, q]
        assert np.max(np.abs(res)) <= (np.max(tb)
                                       + (2 * m + 4 * K * K) * u * size * np.linalg.norm(a[:, q]))
    assert np.mean(st == ost) > 0.99 and ok.any()
