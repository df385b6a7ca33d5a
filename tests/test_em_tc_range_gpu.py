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


def mixture(n, d, k, spread, offset, skew, seed):
    """Rows of k Gaussians of unit scale, their means and covariances; `skew`: half of them of the first."""
    rng = np.random.default_rng(seed)
    M = rng.normal(0.0, spread, (k, d)) + offset
    L = 0.6 * rng.standard_normal((k, d, d)) / np.sqrt(d) + 0.8 * np.eye(d)
    z = rng.integers(0, k, n)
    if skew:
        z[rng.random(n) < 0.5] = 0
    X = rng.standard_normal((n, d))
    for j in range(k):
        X[z == j] = X[z == j] @ L[j].T + M[j]
    return X.astype(np.float32), M, L @ L.transpose(0, 2, 1)


@pytest.mark.parametrize("n,d,k", [(1 << 18, 64, 128), (60000, 64, 12), (100003, 33, 50)])
@pytest.mark.parametrize("spread,offset,skew,outlier,width", [
    (3.0, 0.0, False, 0.0, 1.0),
    (3.0, 0.0, True, 0.0, 1.0),       # one component with half of the rows
    (10.0, 0.0, False, 0.0, 1.0),     # columns wide against a component
    (100.0, 0.0, False, 0.0, 1.0),
    (3.0, 100.0, False, 0.0, 1.0),    # far from the origin
    (3.0, 0.0, False, 1e4, 1.0),      # one value far out
    (3.0, 0.0, False, 0.0, 1e3),      # a start far wider than the data
    (3.0, 0.0, False, 0.0, 0.2),      # and far narrower
])
def test_split_covariances_are_as_exact_as_fp32_sums(gpu_lib, n, d, k, spread, offset, skew, outlier, width):
    """Small components with d > 32, whatever the columns' range: covariances
    against FP64 sums over the engine's own posteriors, means and weights."""
    X, M, S = mixture(n, d, k, spread, offset, skew, seed=k)
    if outlier:
        X[n // 2, 3] = outlier
    mu, cov, R = one_mstep(X, M, 1.2 * width ** 2 * S)
    X64 = X.astype(np.float64)
    for j in sorted({0, 1, k // 2, k - 1}):
        nj = R[:, j].sum()
        if nj < 50:
            continue
        u = X64 - R[:, j] @ X64 / nj
        # around the engine's mean
        o = R[:, j] @ X64 / nj - mu[j]
        ref = (u * R[:, j:j + 1]).T @ u / nj + np.outer(o, o)
        s = np.sqrt(np.diag(ref))
        e = cov[j] - ref
        # the sum of posteriors that it is divided by has an error of its own
        e -= ref * (np.sum(e * ref) / np.sum(ref * ref))
        e /= np.outer(s, s)
        np.fill_diagonal(e, 0.0)
        # every term of a sum of nj rows is rounded to 2^-24 of it, signs at random
        # (8 for the posteriors' halves, the rounding of x - mu and of the partial
        # sums), and FP32 sums span up to 4096 rows before they reach FP64
        assert np.sqrt(np.mean(e * e)) <= 2.0 ** -24 * (8.0 / np.sqrt(nj) + 1.0 / 16)
