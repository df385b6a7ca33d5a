"""The mixed M-step (SimpleMatrixEM::MStep, EM2/MatrixEM.cpp:309-378) on columns
with a wide range: one value far above the rest of its column, which belongs to
a component of its own."""
import numpy as np
import pytest

from fastem_gb300 import CudaMatrixEM, GaussianMixture

pytestmark = pytest.mark.gpu


def one_mstep(X, means, covs):
    n, d = X.shape
    k = len(means)
    with CudaMatrixEM(d, n, k, precision="mixed") as em:
        em.CopyDataset(X)
        em.SetMixture(GaussianMixture(np.full(k, 1.0 / k), means, covs))
        em.InitDensities()
        em.PrecomputeDensityMatrix()
        R = em.Posteriors()
        em.MStep()
        G = em.GetMixture()
    return G.means, G.covs, R


@pytest.mark.parametrize("n,d,k", [
    (32768 + 77, 64, 2),     # components of 16384 rows and more
    (33000, 20, 2),
    (60000, 64, 12),         # small ones: split tensor-core covariances
    (20000, 40, 3),          # and CUDA-core covariances
])
@pytest.mark.parametrize("big", [1000.0, 30000.0])
def test_means_beside_a_large_value(gpu_lib, n, d, k, big):
    """A mean is as exact as its own rows allow.  The values of column 3 lie
    where a part held to 2^-11 of a value is off by all of that, one way."""
    rng = np.random.default_rng(d)
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[:, 3] = np.where(rng.random(n) < 0.5, 0.125, 0.25) * (1.0 + 0.98 * 2.0 ** -11)
    X[n // 2, 3] = big
    means = np.zeros((k, d))
    means[:, 3] = 0.19
    means[k - 1, 3] = big
    covs = np.broadcast_to(np.eye(d), (k, d, d)).copy()
    mu, _, R = one_mstep(X, means, covs)
    X64 = X.astype(np.float64)
    # every MMA cuts its 16 products and the accumulator to 2^-23 of the largest,
    # 12 MMAs per block of 64 rows; the blocks are dealt to 152 CTAs, 64 at most per FP32 sum
    mmas = 12 * min(64, -(-((n + 63) // 64) // 152))
    for j in range(k - 1):
        nj = R[:, j].sum()
        a = R[:, j] @ np.abs(X64) / nj
        tol = (17 * mmas * 2.0 ** -23 + 2.0 ** -21) * a
        assert a[3] < 0.2 and np.all(np.abs(mu[j] - R[:, j] @ X64 / nj) <= tol)
    np.testing.assert_allclose(mu[k - 1, 3], big, rtol=1e-6)
