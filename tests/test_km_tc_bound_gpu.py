"""The tensor-core k-means screen (NaiveKMA::ComputeMSEAndCorrect, Clust/
KMAlgorithm.cpp:205-255) on data with a narrow part to decide in: far from the
origin, one column far away, single rows far out.  Labels and counts
against the FP64 oracle."""
import numpy as np
import pytest

from fastem_gb300 import CudaKMA

pytestmark = pytest.mark.gpu


def data(n, k, gap, offset=0.0, column=0.0, outlier=0.0, seed=0):
    """Unit blobs around centres `gap` apart, and those centres."""
    rng = np.random.default_rng(seed)
    C = rng.normal(0.0, gap, (k, 32)) + offset
    C[:, 5] += column
    X = (C[rng.integers(0, k, n)] + rng.standard_normal((n, 32))).astype(np.float32)
    if outlier:
        X[n // 3, 7] = outlier
    return X, C.astype(np.float32).astype(np.float64)


CASES = [dict(offset=300.0), dict(offset=1000.0), dict(offset=3000.0), dict(offset=2e4), dict(offset=1e5),
         dict(column=2000.0), dict(outlier=2000.0), dict(outlier=1e5), dict(column=-2000.0, outlier=3e4)]


@pytest.mark.parametrize("gap", [0.1, 0.3, 1.0])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "_".join("%s%g" % i for i in c.items()))
def test_labels_are_the_fp64_argmin(gpu_lib, oracle, case, gap):
    n, k = 20000, 256
    X, C = data(n, k, gap, seed=int(100 * gap), **case)
    with CudaKMA(32, n, k, precision="mixed", repair=False) as km:
        km.SetDataset(X)
        fo, _, co, lo = oracle.km_iterate(X, C, repair=False)
        _, cg = km.ComputeMSEAndCorrectCounts(C.copy())
        assert np.array_equal(km.Assignment(), lo)
        assert np.array_equal(cg, co)


@pytest.mark.parametrize("case", [{}] + CASES + [dict(outlier=1e7)], ids=lambda c: "_".join("%s%g" % i for i in c.items()))
def test_an_offset_or_an_outlier_opens_few_rows(gpu_lib, oracle, case):
    """The screen decides nearly every row whatever the data's offset, and
    whatever one row or one centroid far out does to the largest value."""
    n, k = 20000, 256
    X, C = data(n, k, 1.0, **case)
    for far in (0.0, 1e4):
        C[9, :] += far
        with CudaKMA(32, n, k, precision="mixed", repair=False) as km:
            km.SetDataset(X)
            lo = oracle.km_iterate(X, C, repair=False)[3]
            km.ComputeMSEAndCorrect(C.copy())
            assert np.array_equal(km.Assignment(), lo)
            assert km.Stats()["rechecked"] <= n // 100


@pytest.mark.parametrize("shuffled", [False, True])
def test_mostly_equal_rows_open_few(gpu_lib, oracle, shuffled):
    """Four of five rows the same, sorted first or mixed in: the others are
    screened as well."""
    n, k = 30000, 64
    X, C = data(n, k, 5.0, seed=4)
    X[:4 * n // 5] = 0.0
    C[0] = 0.0
    if shuffled:
        X = X[np.random.default_rng(1).permutation(n)]
    with CudaKMA(32, n, k, precision="mixed", repair=False) as km:
        km.SetDataset(X)
        lo = oracle.km_iterate(X, C, repair=False)[3]
        km.ComputeMSEAndCorrect(C.copy())
        assert np.array_equal(km.Assignment(), lo)
        assert km.Stats()["rechecked"] <= n // 100
