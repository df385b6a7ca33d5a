"""The FP32 k-means path (NaiveKMA::ComputeMSEAndCorrect, Clust/KMAlgorithm.cpp:
205-255) at the edges of its kernel, against the FP64 oracle."""
import numpy as np
import pytest

from fastem_gb300 import CudaKMA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,k", [
    (2, 31, 1), (2, 100003, 700), (4, 33, 5), (4, 40001, 1024), (8, 129, 3), (8, 70001, 257), (16, 1, 2),
    (16, 300007, 100), (32, 513, 40), (32, 50021, 480), (64, 65, 2), (64, 30011, 190),
])
def test_km_fp32_screen_matches_oracle(gpu_lib, oracle, d, n, k):
    """The FP32 screen (w = ||c||^2 / 2 - x.c, two smallest, warp-wide decision
    of the rest) at the edges of its row groups and centroid counts: labels,
    counts and centroids of two iterations, far from the origin, with
    duplicated centroids (exact ties) and rows midway between two."""
    rng = np.random.default_rng(d * 1000 + k)
    X = (rng.uniform(-20, 20, (max(2, k // 3), d))[rng.integers(0, max(2, k // 3), n)]
         + rng.standard_normal((n, d)) + 300.0).astype(np.float32)
    C = X[rng.integers(0, n, k)].astype(np.float64)
    if k > 1:
        C[k - 1] = C[0]
        X[n // 2] = (0.5 * (C[0] + C[k // 2])).astype(np.float32)
    with CudaKMA(d, n, k, precision="fp32", repair=False) as km:
        km.SetDataset(X)
        for _ in range(2):
            fo, Co, co, lo = oracle.km_iterate(X, C, repair=False)
            Cg = C.copy()
            fg, cg = km.ComputeMSEAndCorrectCounts(Cg)
            assert np.array_equal(km.Assignment(), lo)
            assert np.array_equal(cg, co)
            live = np.asarray(co) > 0
            np.testing.assert_allclose(Cg[live], np.asarray(Co)[live], rtol=1e-12, atol=1e-12)
            assert np.array_equal(Cg[~live], C[~live])
            C = Cg
