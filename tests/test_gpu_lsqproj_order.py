"""lsqproject of sample lists in any order: each listed sample's result is the one it has in the
ascending list of all samples, to the bit (the products are exact sums, the solve is a sample's own).

Lists that start past their end, whose middle lies outside their first and last sample, that
repeat, that fill one block of 128 rows or more, near (within 64 record bytes) and far apart."""
import numpy as np
import pytest

from eig_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N, M, K = 1100, 1500, 4


def lists():
    r = np.random.default_rng(8)
    every = np.arange(N)
    ends = np.stack([every, every[::-1]], 1).ravel()[:N]
    return dict(descending=every[::-1], permuted=r.permutation(N), ends=ends,
                repeated=np.repeat(every[::2], 2), one_over_and_over=np.full(130, 777),
                near_descending=np.arange(400, 200, -1), near_outlier=np.r_[100:200, 1099, 200:227],
                far_in_the_middle=np.r_[8, 1099, 0, 9], last=np.array([N - 1]),
                few_permuted=r.permutation(N)[:129])


@pytest.fixture(scope="module", params=[native.GP_PREC_FP64, native.GP_PREC_SPLIT_FP16],
                ids=["fp64", "fp16"])
def ascending(gpu, request):
    r = np.random.default_rng(7)
    f = r.uniform(0.05, 0.95, (M, 1)) + 0.1 * r.standard_normal((M, 6))[:, np.arange(N) % 6]
    g = r.binomial(2, np.clip(f, 0.02, 0.98)).astype(np.int8)
    g[r.random((M, N)) < 0.05] = -1
    gpu.load_genotypes(O.pack(g), N)
    gpu.set_samples(np.arange(0, N, 2, dtype=np.int32))
    gpu.set_snps(np.arange(M, dtype=np.int32))
    gpu.xtx(precision=request.param)
    gpu.eigvecs(K)
    gpu.snp_weights(K)
    return gpu, gpu.lsqproj(K, np.arange(N, dtype=np.int32))


@pytest.mark.parametrize("name", list(lists()))
def test_list_order(ascending, name):
    gpu, (a, b, nobs, st) = ascending
    q = lists()[name].astype(np.int32)
    a2, b2, nobs2, st2 = gpu.lsqproj(K, q)
    assert np.array_equal(nobs2, nobs[q]) and np.array_equal(st2, st[q])
    assert np.array_equal(b2, b[:, q])
    assert np.array_equal(a2, a[:, q])
