"""fastmode at block widths and counts where its packed triangles, even tiles and two-block first
projection can go wrong (odd L, L = 2 and 64, one to many blocks, few independent directions):
the Ritz pairs of the last block's full reorthogonalisation against a dense Rayleigh-Ritz.

Tolerance: the Krylov space of at least as many columns as the panel's rank holds every
eigenvector, so the Ritz values are the eigenvalues to the products' 2^-41 (split) or 2^-52 (FP64)
times the number of products; 1e-9 as in the long Krylov test."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [native.GP_PREC_FP64, native.GP_PREC_SPLIT_FP16])
@pytest.mark.parametrize("n,m,K,L,I", [(90, 700, 1, 2, 60), (97, 701, 3, 5, 30), (120, 64, 4, 21, 6),
                                       (150, 900, 10, 33, 5), (200, 500, 20, 64, 3),
                                       (61, 1300, 5, 64, 1)])
def test_blocks(gpu, n, m, K, L, I, prec):
    r = np.random.default_rng(n + L)
    f = r.uniform(0.1, 0.9, (m, 1)) + 0.25 * r.standard_normal((m, 6))[:, np.arange(n) % 6]
    g = r.binomial(2, np.clip(f, 0.02, 0.98)).astype(np.int8)
    rec = O.pack(g)
    gpu.load_genotypes(rec, n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(m, dtype=np.int32))
    ev, V = gpu.fastpca(K, L, I, seed=3, precision=prec)
    s = O.pass_columns(rec, np.arange(m, dtype=np.int32), np.arange(n, dtype=np.int32),
                       minallelecnt=0, maxmissing=2 ** 31 - 1)
    w, U = np.linalg.eigh(O.gram(s) / (2.0 * m))
    w, U = w[::-1][:K], U[:, ::-1][:, :K].T
    assert np.max(np.abs(ev - w) / w) <= 1e-9, (ev, w)
    # V's rows are eigenvectors: residuals, so that close eigenvalues need no matching
    G = O.gram(s) / (2.0 * m)
    V = V / np.linalg.norm(V, axis=1)[:, None]
    assert np.max(np.linalg.norm(V @ G - ev[:, None] * V, axis=1)) <= 1e-8 * w[0]
    assert np.max(np.abs(V @ V.T - np.eye(K))) <= 1e-8
