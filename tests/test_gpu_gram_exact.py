"""The FP64 Gram's exact tensor-core sums at the edges of their tiles, blocks and chunks."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def panel(n, m, miss, rare, seed):
    """packed records with a share of missing calls; rare: allele frequencies down to 1/(2n)"""
    r = np.random.default_rng(seed)
    p = 0.5 * (1.0 / n) ** r.random(m) if rare else r.uniform(0.05, 0.95, m)
    g = (r.random((m, n)) < p[:, None]).astype(np.int8) + (r.random((m, n)) < p[:, None])
    g[r.random((m, n)) < miss] = -1
    return O.pack(g)


def check(gpu, rec, rows, cols, nind, alt=1):
    gpu.load_genotypes(rec, nind)
    gpu.set_samples(rows)
    gpu.set_snps(cols)
    r = gpu.xtx(altnormstyle=alt)
    s = O.pass_columns(rec, cols, rows, altnormstyle=alt)
    tab = s.tab.reshape(-1, 4)
    code = O.unpack(rec[cols], nind)[:, rows]
    v = np.take_along_axis(tab, np.where(code < 0, 3, code), axis=1)
    X = v.T @ v
    # the FP64 dot products' own bound, the rounding of R1 = f v and R2 = T1 v (two operations
    # each, coefficients of at most 1), and their 2^-60 of the power of two above the largest
    m = len(cols)
    keep = s.killed == 0
    assert r["nused"] == int(keep.sum())
    f = np.maximum(np.abs(s.xfancy), np.abs(tab[:, 1])) * keep
    big = np.max(f[:, None] * np.abs(tab), initial=0.0)
    d = np.sqrt(np.diag(X))
    tol = (m * 2.0 ** -53 * np.outer(d, d) + 2.0 ** -50 * np.sqrt(np.sum(f * f)) * d[None, :]
           + m * 2.0 ** -58 * big)
    assert np.all(np.abs(r["XTX"] - X) <= np.maximum(tol, tol.T))
    assert np.array_equal(r["XTX"], r["XTX"].T)
    assert abs(r["trace"] - np.trace(X)) <= np.sum(np.diag(tol)) + 2.0 ** -50 * np.trace(X)
    return r["XTX"]


@pytest.mark.parametrize("n,m", [(2, 3), (47, 64), (48, 65), (49, 63), (128, 200), (129, 130),
                                 (255, 4096), (256, 4097), (257, 300), (305, 8300), (600, 513)])
@pytest.mark.parametrize("rare", [False, True])
def test_tile_edges(gpu, n, m, rare):
    rec = panel(n, m, 0.05, rare, n * 7 + m)
    # one SNP that is surely kept, whatever the small panels drew
    g = np.zeros(n, np.int8)
    g[::2] = 1
    rec[0] = O.pack(g[None])[0]
    check(gpu, rec, np.arange(n, dtype=np.int32), np.arange(m, dtype=np.int32), n)


@pytest.mark.parametrize("alt", [0, 1])
def test_row_and_column_subsets(gpu, alt):
    """gaps in the rows, columns in another order and twice, no missing calls at all"""
    r = np.random.default_rng(5)
    rec = panel(500, 900, 0.0, False, 6)
    rows = np.sort(r.choice(500, 333, replace=False)).astype(np.int32)
    cols = np.concatenate([r.permutation(900)[:700], [3, 3, 4]]).astype(np.int32)
    check(gpu, rec, rows, cols, 500, alt)


def test_passes_give_the_same_bits(gpu, monkeypatch):
    """several passes over the SNPs (a small operand budget) add up to the same integers"""
    n, m = 310, 5000
    rec = panel(n, m, 0.1, True, 9)
    rows, cols = np.arange(n, dtype=np.int32), np.arange(m, dtype=np.int32)
    one = check(gpu, rec, rows, cols, n)
    monkeypatch.setenv("GP_EXACT_BUDGET_BYTES", str(5 * 7 * 61440))
    assert np.array_equal(check(gpu, rec, rows, cols, n), one)


def values(rec, n, alt=1):
    """(tables [m][4], codes [m][n], kept) by the oracle"""
    m = len(rec)
    s = O.pass_columns(rec, np.arange(m, dtype=np.int32), np.arange(n, dtype=np.int32),
                       altnormstyle=alt)
    code = O.unpack(rec, n)
    return s.tab.reshape(-1, 4), np.where(code < 0, 3, code), s.killed == 0, s.xfancy


# panels whose rarest allele is seen once and that take six digits: edges of the 40-column tiles, of
# the 64-SNP blocks and of a chunk of 4,096 SNPs; a cohort of several thousand samples
@pytest.mark.parametrize("n,m", [(39, 60), (40, 63), (41, 50), (81, 65), (255, 64), (257, 130),
                                 (601, 4160), (5003, 600)])
def test_rare_variants(gpu, n, m, monkeypatch):
    r = np.random.default_rng(n + m)
    p = 0.5 * (1.0 / n) ** r.random(m)
    p = np.where(r.random(m) < 0.5, p, 1 - p)
    g = (r.random((m, n)) < p[:, None]).astype(np.int8) + (r.random((m, n)) < p[:, None])
    g[r.random((m, n)) < 0.03] = -1
    g[0], g[0, n // 2], g[1], g[1, n // 3] = 0, 1, 2, 1
    g[2, ::2], g[2, 1::2] = 0, 1
    rec = O.pack(g)
    gpu.load_genotypes(rec, n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(m, dtype=np.int32))
    got = gpu.xtx(altnormstyle=1)["XTX"]
    tab, code, keep, fancy = values(rec, n)
    v = np.take_along_axis(tab, code, axis=1)
    # some rows against all samples, in long double
    q = np.unique(np.r_[0, n // 3, n // 2, n - 1, r.choice(n, min(n, 36), replace=False)])
    X = np.zeros((len(q), n), np.longdouble)
    for a in range(0, m, 64):
        X += v[a:a + 64, q].T.astype(np.longdouble) @ v[a:a + 64].astype(np.longdouble)
    X = X.astype(float)
    # the value of the more frequent homozygote (T0 or T2) enters as it is, the others as it plus or
    # minus f: two roundings of their own and one of its; 72 bits below the scale for each term; the
    # combination and the rounding of the result
    base = np.where(np.abs(tab[:, 0]) <= np.abs(tab[:, 2]), 0, 2)
    other = (code != base[:, None]) & (code != 3) & keep[:, None]
    a = np.where(other, 2 * np.abs(v) + np.abs(tab[np.arange(m), base])[:, None], 0.0)
    u = 2.0 ** -53
    f = np.maximum(np.abs(fancy), np.abs(tab[:, 1])) * keep
    scale = 2.0 * np.max(f[:, None] * np.abs(tab))
    tol = (u * (a[:, q].T @ np.abs(v) + np.abs(v[:, q]).T @ a) + 4 * u * np.abs(X)
           + 2 * m * 2.0 ** -72 * scale)
    assert np.all(np.abs(got[q] - X) <= tol)
    assert np.array_equal(got, got.T)
    monkeypatch.setenv("GP_EXACT_BUDGET_BYTES", str(((n + 39) // 40) * 61440))
    assert np.array_equal(gpu.xtx(altnormstyle=1)["XTX"], got)
