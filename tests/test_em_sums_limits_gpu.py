"""The FP32 M-step sums (SimpleMatrixEM::MStep, EM2/MatrixEM.cpp:309-378) of
several point groups: sums beyond FP32's range, and what the groups' addition
rounds."""
import numpy as np
import pytest

from fastem_gb300 import CudaBatchEM, CudaMatrixEM, GaussianMixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 4, 7, 12])
def test_batched_sums_beyond_fp32_are_infinite(gpu_lib, d):
    """(x - mu)^2 above FP32's range gives an infinite variance, no NaN and no
    failed factorisation of the sweep that finds it."""
    n = 3001
    rng = np.random.default_rng(d)
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[:, 0] = 3e19 * np.sign(X[:, 0])
    S = np.eye(d)[None]
    S[0, 0, 0] = 1e39
    with CudaBatchEM([(d, n, 1)], precision="fp32", max_sweeps=1) as b:
        b.CopyDatasets([X])
        b.SetMixture(0, GaussianMixture(np.ones(1), np.zeros((1, d)), S))
        b.TrainNoCopy()
        assert b.GetMixture(0).covs[0, 0, 0] == np.inf


@pytest.mark.parametrize("d", [3, 8, 16])
def test_group_sums_are_added_without_rounding(gpu_lib, d):
    """Values whose products are multiples of 2^-12, few enough per point group
    to add up exactly in FP32 but not over all groups: the covariance is exact."""
    n = 1 << 22
    rng = np.random.default_rng(d)
    half = rng.integers(33, 65, (n // 2, d)) * rng.choice([-1, 1], (n // 2, d))
    U = np.concatenate([half, -half]).astype(np.int64)[rng.permutation(n)]     # means exactly 0
    X = (U / 64.0).astype(np.float32)
    ref = (U.T @ U).astype(np.float64) / 4096.0 / n
    with CudaMatrixEM(d, n, 1, precision="fp32") as em:
        em.CopyDataset(X)
        em.SetMixture(GaussianMixture(np.ones(1), np.zeros((1, d)), np.eye(d)[None]))
        em.InitDensities()
        em.PrecomputeDensityMatrix()
        em.MStep()
        G = em.GetMixture()
    assert np.all(G.means == 0.0)
    assert np.array_equal(G.covs[0], ref)
