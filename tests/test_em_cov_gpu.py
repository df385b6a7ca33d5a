"""The CUDA-core covariance sums (SimpleMatrixEM::MStep, EM2/MatrixEM.cpp:
53-99,363-375) at the edges of their blocks, unit splits and row tiles: the
covariances of one M-step against the same sums over the engine's own
posteriors in FP64 numpy."""
import numpy as np
import pytest

from fastem_gb300 import CudaMatrixEM, GaussianMixture

pytestmark = pytest.mark.gpu

U32, U64 = 2.0 ** -24, 2.0 ** -53


def one_mstep(X, k, precision, seed, width=1.0):
    """(means, covariances, posteriors) of one M-step from a spread-out mixture."""
    n, d = X.shape
    rng = np.random.default_rng(seed)
    means = X[rng.choice(n, k, replace=n < k)].astype(np.float64)
    G = GaussianMixture(np.full(k, 1.0 / k), means, np.broadcast_to(30.0 * width ** 2 * np.eye(d), (k, d, d)))
    with CudaMatrixEM(d, n, k, precision=precision) as em:
        em.CopyDataset(X)
        em.SetMixture(G)
        em.InitDensities()
        em.PrecomputeDensityMatrix()
        R = em.Posteriors()
        em.MStep()
        G = em.GetMixture()
    return G.means, G.covs, R


def check_covariances(X, mu, cov, R, precision, rows):
    """Every covariance against the sums over R around the engine's means, to
    the rounding of sums over at most `rows` rows per FP32 sum."""
    n = len(X)
    X64, xmax = X.astype(np.float64), float(np.abs(X).max())
    for j in range(R.shape[1]):
        # around the means the engine found: the rounding of the means is its own
        nj = R[:, j].sum()
        u = X64 - mu[j]
        ref = (u * R[:, j:j + 1]).T @ u / nj
        s = np.sqrt(np.diag(ref))
        if precision == "fp64":
            # n-term sums in any order, and the rounding of mu
            tol = U64 * ((n + 16) * np.outer(s, s) + 8 * xmax * (s[:, None] + s[None, :] + xmax))
        else:
            # x - mu rounds to 2^-24 of |x| + |mu| and mu itself to FP32.  mixed:
            # the posteriors' hi + lo halves carry 22 bits
            tol = U32 * ((rows + 16) * np.outer(s, s) + 8 * xmax * (s[:, None] + s[None, :]) + 8 * U32 * xmax ** 2)
        assert np.all(np.abs(cov[j] - ref) <= tol), (j, float(np.max(np.abs(cov[j] - ref) / tol)))
        assert np.array_equal(cov[j], cov[j].T)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("n,d,k", [
    (1, 1, 1),            # one row, one dimension
    (7, 3, 2),            # fewer rows than a tile; 4 x 4 triangle
    (511, 4, 3),
    (1025, 5, 20),        # one triangular 8 x 8 block, many point groups
    (3001, 8, 127),
    (2049, 9, 5),         # two blocks, seven padded dimensions
    (4099, 16, 100),      # units that do not divide by 256
    (1000, 17, 11),
    (5003, 31, 7),
    (2500, 64, 3),
    (40961, 63, 60),      # more than 2048 rows per FP32 sum, one point group
    ((1 << 21) + 5, 32, 8),   # the same with three point groups
])
def test_covariance_sums_match_numpy(gpu_lib, precision, n, d, k):
    if n > 10 ** 6 and precision == "fp64":
        pytest.skip("FP64 sums have no row windows")
    rng = np.random.default_rng(100 * d + k)
    X = (rng.normal(0.0, 3.0, (n, d)) + rng.normal(0.0, 2.0, d)).astype(np.float32)
    mu, cov, R = one_mstep(X, k, precision, seed=d)
    check_covariances(X, mu, cov, R, precision, 2048)


@pytest.mark.parametrize("n,d,k,scale,shift", [
    (4929, 64, 128, 1.0, 2.0),       # one point in the last block, chunks of a few blocks
    (77889, 33, 5, 1.0, 2.0),        # three padded components, 31 padded dimensions
    (10497, 63, 60, 1e-4, 2.0),      # data far below 1: sums are in units of the data
    (10431, 48, 61, 100.0, 50.0),    # data far from the origin
    ((1 << 18) + 3, 64, 128, 1.0, 2.0),   # several FP64 windows per chunk
])
def test_split_covariance_sums_match_numpy(gpu_lib, n, d, k, scale, shift):
    """The mixed path's split tensor-core sums (d > 32, N < 16384 K, enough
    blocks for every SM) reach the CUDA-core form's accuracy."""
    rng = np.random.default_rng(7 * d + k)
    X = (scale * (rng.normal(0.0, 3.0, (n, d)) + rng.normal(0.0, shift, d))).astype(np.float32)
    mu, cov, R = one_mstep(X, k, "mixed", seed=d, width=scale)
    check_covariances(X, mu, cov, R, "mixed", 4096)
