"""The FP32 k-means screen (NaiveKMA::ComputeMSEAndCorrect, Clust/KMAlgorithm.cpp:
205-255) with a centroid or a row far out: labels against the FP64 oracle, and
the other rows still decided by the screen."""
import numpy as np
import pytest

from fastem_gb300 import CudaKMA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 16, 64])
@pytest.mark.parametrize("far,outlier", [(30.0, 0.0), (1e3, 0.0), (1e5, 0.0), (1e9, 0.0), (0.0, 1e4), (0.0, 1e9),
                                         (1e4, -1e6)])
def test_one_far_out_does_not_open_the_rest(gpu_lib, oracle, d, far, outlier):
    n, k = 60001, 60
    rng = np.random.default_rng(d)
    C = rng.normal(0.0, 20.0, (k, d)).astype(np.float32)
    X = (C[rng.integers(0, k, n)] + rng.standard_normal((n, d))).astype(np.float32)

    def iterate(X, C):
        with CudaKMA(d, n, k, precision="fp32", repair=False) as km:
            km.SetDataset(X)
            ms = []
            for _ in range(5):
                _, counts = km.ComputeMSEAndCorrectCounts(C.astype(np.float64))
                ms.append(km.Stats()["assign_ms"])
            return km.Assignment(), counts, min(ms)

    clean = iterate(X, C)[2]
    if outlier:
        X[n // 2, d - 1] = outlier
    if far:
        C[7] += far
    _, _, co, lo = oracle.km_iterate(X, C.astype(np.float64), repair=False)
    labels, counts, ms = iterate(X, C)
    assert np.array_equal(labels, lo)
    assert np.array_equal(counts, co)
    # a screen that left every row open took 10 to 70 times as long
    assert ms <= 4.0 * clean


@pytest.mark.parametrize("d,k", [(2, 300), (8, 100), (16, 100), (32, 100), (64, 100)])
def test_close_centroids_far_from_the_middle(gpu_lib, oracle, d, k):
    """Several centroids in each of a few blobs: the product form's bound, which
    grows with the distance from the middle, leaves most rows to the differences."""
    n = 60001
    rng = np.random.default_rng(d + 1)
    apart = rng.normal(0.0, 20.0, (k, d)).astype(np.float32)
    blobs = 100.0 * rng.random((1, d)) * np.arange(5)[:, None]
    close = (blobs[np.arange(k) % 5] + 0.1 * rng.standard_normal((k, d))).astype(np.float32)
    close[k - 1] = close[0]                                    # exact ties
    ms = []
    for centres, C in ((apart, apart), (blobs, close)):
        X = (centres[rng.integers(0, len(centres), n)] + rng.standard_normal((n, d))).astype(np.float32)
        _, _, co, lo = oracle.km_iterate(X, C.astype(np.float64), repair=False)
        with CudaKMA(d, n, k, precision="fp32", repair=False) as km:
            km.SetDataset(X)
            t = []
            for _ in range(5):
                _, counts = km.ComputeMSEAndCorrectCounts(C.astype(np.float64))
                t.append(km.Stats()["assign_ms"])
            assert np.array_equal(km.Assignment(), lo)
            assert np.array_equal(counts, co)
            ms.append(min(t))
    # a difference form for each row beside the screen, not a warp's decision
    assert ms[1] <= 5.0 * ms[0] + 0.05
