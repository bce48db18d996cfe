"""The eigenvalues' error where one warp has several of them: half of the widest last bracket,
1.5e-14 of the norm, over all of them in the mean square (a midpoint's error is at most half of its
bracket, and the tridiagonal's float-float arithmetic and the FP64 counts leave less)."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# six, four and three points a step; 6,080 is the last order with three
@pytest.mark.parametrize("n", [2500, 3700, 4900])
def test_mean_square_error(gpu, n):
    r = np.random.default_rng(n)
    m = n + 500
    p = r.uniform(0.05, 0.95, (m, 1)) + 0.1 * r.standard_normal((m, 2))[:, np.arange(n) % 2]
    gpu.load_genotypes(O.pack(r.binomial(2, np.clip(p, 0.02, 0.98)).astype(np.int8)), n)
    gpu.set_samples(np.arange(n, dtype=np.int32))
    gpu.set_snps(np.arange(m, dtype=np.int32))
    x = gpu.xtx()
    w, _ = gpu.eigvecs(4)
    ref = np.linalg.eigvalsh(x["XTX"] * ((n - 1) / x["trace"]))[::-1]
    assert np.sqrt(np.mean((w - ref) ** 2)) <= 1.5e-14 * ref[0]
