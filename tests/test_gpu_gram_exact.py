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
