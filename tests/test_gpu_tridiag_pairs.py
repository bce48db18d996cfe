"""The shared-memory tridiagonalisation's pairs of rows at the edges of its variants (2, 4 and 8
rows a thread), odd and even orders and first steps, against LAPACK with test_gpu_tridiag's
tolerances."""
import pytest

from tests.test_gpu_tridiag import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 5, 8, 63, 319, 320, 321, 1024, 1025, 1706, 1707])
def test_orders(gpu, n):
    solve(gpu, n, n + 40, n)


@pytest.mark.parametrize("n,limit", [(400, 321), (401, 321), (400, 320), (401, 320), (1300, 1025)])
def test_handed_over(gpu, monkeypatch, n, limit):
    monkeypatch.setenv("GP_TRIDIAG_SMEM", str(limit))
    solve(gpu, n, n + 40, n)
