"""The tiled tridiagonalisation's packed steps at the edges of tiles, column units and warps'
shares (to the last column, and handing over to the shared-memory steps), against LAPACK with
test_gpu_tridiag's tolerances, and at an order near its limit, where a CTA's shared memory is
nearly full."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O
from tests.test_gpu_tridiag import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("switch", ["1", "70"])
@pytest.mark.parametrize("n", [73, 127, 128, 129, 191, 400, 1153])
def test_tile_edges(gpu, monkeypatch, n, switch):
    monkeypatch.setenv("GP_TRIDIAG_SWITCH", switch)
    solve(gpu, n, 2 * n + 7, n)


@pytest.mark.parametrize("n", [400, 1153])
def test_rank_deficient(gpu, monkeypatch, n):
    """reflectors of columns that are zero to rounding"""
    monkeypatch.setenv("GP_TRIDIAG_SWITCH", "1")
    w = solve(gpu, n, 60, 5)
    assert np.max(np.abs(w[60:])) <= 1e-11 * w[0]


def test_whole_columns_give_the_same(gpu, monkeypatch):
    monkeypatch.setenv("GP_TRIDIAG_SMEM", "100")
    w = solve(gpu, 500, 900, 3)
    monkeypatch.setenv("GP_TRIDIAG_TILED", "0")
    # two float-float reductions, each within solve()'s bound
    assert np.max(np.abs(w - solve(gpu, 500, 900, 3))) <= 2 * (4 * np.sqrt(500) * 2.0**-44 +
                                                               1e-12) * w[0]


def test_near_the_largest_order(gpu):
    n, m, k = 7600, 7700, 3
    r = np.random.default_rng(9)
    p = r.uniform(0.05, 0.95, m)
    pop = np.arange(n) % 3
    q = np.clip(p[:, None] + 0.2 * r.standard_normal((m, 3)), 0.02, 0.98)
    g = r.binomial(2, q[:, pop]).astype(np.int8)
    gpu.load_genotypes(O.pack(g), n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(m, dtype=np.int32))
    x = gpu.xtx(native.GP_PREC_FP64)
    w, V = gpu.eigvecs(k)
    A = x["XTX"] * ((n - 1) / x["trace"])
    tol = (4 * np.sqrt(n) * 2.0**-44 + 1e-12) * w[0]
    assert abs(np.sum(w) - (n - 1)) <= n * tol  # the trace
    assert np.max(np.abs(V @ V.T - np.eye(k))) <= 1e-9
    R = A @ V[:2].T - V[:2].T * w[:2]
    assert np.max(np.linalg.norm(R, axis=0)) <= 8 * tol
