"""The tridiagonalisation's shared-memory steps (alone and after steps in L2) against LAPACK,
at the edges of the blocks' column counts and on rank-deficient matrices."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def solve(gpu, n, m, seed):
    r = np.random.default_rng(seed)
    p = r.uniform(0.05, 0.95, m)
    g = (r.random((m, n)) < p[:, None]).astype(np.int8) + (r.random((m, n)) < p[:, None])
    g[0, : n // 2] = 0  # at least one SNP that varies
    g[0, n // 2:] = 1
    gpu.load_genotypes(O.pack(g), n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(m, dtype=np.int32))
    x = gpu.xtx()
    k = min(n, 4)
    w, V = gpu.eigvecs(k)
    A = x["XTX"] * ((n - 1) / x["trace"])
    ref = np.linalg.eigvalsh(A)[::-1]
    # float-float steps: n reflections of relative error 2^-44 each, accumulating as sqrt(n);
    # the eigenvalues' own brackets end at 1e-13 of the norm
    tol = (4 * np.sqrt(n) * 2.0 ** -44 + 1e-12) * ref[0]
    assert np.max(np.abs(w - ref)) <= tol
    assert np.max(np.abs(V @ V.T - np.eye(k))) <= 1e-9
    # a vector's residual, well above the eigenvalue's error for an order of 1,000
    assert np.max(np.abs(A @ V.T - V.T * w[:k])) <= 8 * tol
    return w


@pytest.mark.parametrize("n", [2, 3, 16, 17, 31, 33, 64, 65, 180, 557, 560, 1023, 1026])
def test_block_counts(gpu, n):
    """from one block to all, one and two rows per thread"""
    solve(gpu, n, 4 * n + 20, n)


@pytest.mark.parametrize("n,limit", [(300, "1"), (300, "2"), (300, "152"), (301, "200"),
                                     (900, "899"), (1800, ""), (2600, "")])
def test_from_l2_to_shared_memory(gpu, monkeypatch, n, limit):
    """the trailing orders at which the matrix moves into shared memory, among them the last
    column alone; 2,600: after tiled steps"""
    if limit:
        monkeypatch.setenv("GP_TRIDIAG_SMEM", limit)
    solve(gpu, n, 2 * n, n + 1)


def test_tiled_straight_to_shared_memory(gpu, monkeypatch):
    monkeypatch.setenv("GP_TRIDIAG_SWITCH", "400")
    solve(gpu, 700, 1500, 3)


@pytest.mark.parametrize("n,m", [(200, 30), (700, 100)])
def test_rank_deficient(gpu, n, m):
    """reflectors of columns that are zero to rounding"""
    w = solve(gpu, n, m, 5)
    assert np.max(np.abs(w[m:])) <= 1e-11 * w[0]


def test_repeated_eigenvalues(gpu):
    """every sample carries one allele of its own: a multiple of I - 11'/n, whose vectors come
    out of inverse iteration far from orthogonal"""
    n = 40
    gpu.load_genotypes(O.pack(np.eye(n, dtype=np.int8)), n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(n, dtype=np.int32))
    x = gpu.xtx()
    w, V = gpu.eigvecs(5)
    A = x["XTX"] * ((n - 1) / x["trace"])
    assert np.max(np.abs(w[:-1] - 1.0)) <= 1e-12 and abs(w[-1]) <= 1e-12
    assert np.max(np.abs(V @ V.T - np.eye(5))) <= 1e-12
    assert np.max(np.abs(A @ V.T - V.T * w[:5])) <= 1e-11


def test_more_vectors_than_the_joint_orthonormalisation_takes(gpu):
    r = np.random.default_rng(8)
    n, m, k = 120, 900, 70
    g = r.integers(0, 3, (m, n)).astype(np.int8)
    gpu.load_genotypes(O.pack(g), n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(m, dtype=np.int32))
    x = gpu.xtx()
    w, V = gpu.eigvecs(k)
    A = x["XTX"] * ((n - 1) / x["trace"])
    assert np.max(np.abs(V @ V.T - np.eye(k))) <= 1e-9
    assert np.max(np.abs(A @ V.T - V.T * w[:k])) <= 1e-10 * w[0]
