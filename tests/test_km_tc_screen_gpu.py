"""The tensor-core k-means screen (NaiveKMA::ComputeMSEAndCorrect, Clust/
KMAlgorithm.cpp:205-255) where its scaling, exclusion and two-part sums can go
wrong, against the FP64 oracle: data scales, far centroids, padded counts."""
import numpy as np
import pytest

from fastem_gb300 import CudaKMA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,scale,shift,far", [
    (129, 2, 1.0, 0.0, 0),
    (40000, 47, 1e-6, 0.0, 0),        # data far below 1
    (40001, 64, 1e6, 0.0, 0),         # far above FP16's range
    (300001, 256, 1.0, 500.0, 0),     # far from the origin; above the row count of the 32-bit sums
    (300001, 17, 1.0, 0.0, 3),        # centroids parked far outside the data
    (5000, 20, 1.0, 0.0, 20),         # all of them far outside: every centroid a candidate
    (1 << 20, 250, 30.0, 10.0, 1),
])
def test_km_tc_screen_matches_oracle(gpu_lib, oracle, n, k, scale, shift, far):
    rng = np.random.default_rng(n + k)
    blobs = rng.uniform(-20, 20, (max(2, k // 2), 32))
    X = (scale * (blobs[rng.integers(0, len(blobs), n)] + rng.standard_normal((n, 32)) + shift)).astype(np.float32)
    C = X[rng.integers(0, n, k)].astype(np.float64)
    if far:
        C[:far] = scale * rng.uniform(1e5, 2e5, (far, 32))
    elif k > 2:
        C[k - 1] = C[0]                                               # exact ties
        X[n // 2] = (0.5 * (C[0] + C[k // 2])).astype(np.float32)     # a row midway
    with CudaKMA(32, n, k, precision="mixed", repair=False) as km:
        km.SetDataset(X)
        for _ in range(2):
            fo, Co, co, lo = oracle.km_iterate(X, C, repair=False)
            Cg = C.copy()
            fg, cg = km.ComputeMSEAndCorrectCounts(Cg)
            assert np.array_equal(km.Assignment(), lo)
            assert np.array_equal(cg, co)
            live = np.asarray(co) > 0
            # FP64 sums of n rows in another order, of rows rounded to the
            # engine's fixed-point grid (2^-40, or what keeps n max|x| in 62 bits)
            grid = 2.0 ** -min(40, np.floor(61 - np.ceil(np.log2(np.abs(X).max()) + np.log2(n))))
            np.testing.assert_allclose(Cg[live], np.asarray(Co)[live], rtol=1e-12,
                                       atol=0.5 * grid + 1e-12 * scale * (1 + shift))
            assert np.array_equal(Cg[~live], C[~live])
            C = Cg
