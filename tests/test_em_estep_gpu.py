"""The CUDA-core E-steps (MatrixEMBase::BlockDensities and
PostProcessDensityMatrix, EM2/MatrixEM.cpp:39-51,69-81) at the edges of their
dimension classes, component groups and point tiles, against FP64 numpy."""
import numpy as np
import pytest
from scipy.linalg import cholesky, solve_triangular
from scipy.special import logsumexp

from fastem_gb300 import CudaMatrixEM, GaussianMixture
from fastem_gb300.batch import CudaBatchEM

pytestmark = pytest.mark.gpu

U32, U64 = 2.0 ** -24, 2.0 ** -53


def problem(n, d, k, seed):
    rng = np.random.default_rng(seed)
    mu = rng.normal(0.0, 3.0, (k, d))
    A = rng.normal(0.0, 0.4 / np.sqrt(d), (k, d, d))
    cov = A @ A.transpose(0, 2, 1) + np.eye(d)[None] * rng.uniform(0.5, 2.0, (k, 1, 1))
    w = rng.uniform(0.5, 1.5, k)
    X = (mu[rng.integers(0, k, n)] + 2.0 * rng.normal(0.0, 1.0, (n, d))).astype(np.float32)
    return X, GaussianMixture(w / w.sum(), mu, cov)


def reference(X, G, u):
    """(posteriors, LogL, bound on the error of a log density per point): the
    rounding of the centred values, of the factor, and of sums of d products,
    carried through ||W (x - mu)||^2 at unit roundoff u."""
    X = X.astype(np.float64)
    n, d = X.shape
    k = len(G.weights)
    L, dl = np.empty((n, k)), np.zeros(n)
    for j in range(k):
        ch = cholesky(G.covs[j], lower=True)
        W = solve_triangular(ch, np.eye(d), lower=True)
        t = X - G.means[j]
        y = t @ W.T
        s = np.sum(y * y, axis=1)
        lc = np.log(G.weights[j]) - 0.5 * d * np.log(2 * np.pi) - np.sum(np.log(np.diag(ch)))
        L[:, j] = lc - 0.5 * s
        aW = np.abs(W)
        # W: rounded to u, and its FP64 factorisation
        dw = u + 4 * d * np.linalg.cond(G.covs[j]) * U64
        dy = ((d + 2) * u + dw) * (np.abs(t) @ aW.T) + u * ((np.abs(X) + np.abs(G.means[j])) @ aW.T)
        e = np.sum(np.abs(y) * dy, axis=1) + (d + 4) * u * s + 2 * u * (abs(lc) + np.abs(L[:, j]))
        dl = np.maximum(dl, e)
    lse = logsumexp(L, axis=1)
    return np.exp(L - lse[:, None]), lse, dl + u * np.abs(lse)


SHAPES = [
    (1, 1, 1), (127, 2, 3), (129, 3, 17), (128 * 3 + 1, 4, 16), (1000, 5, 33), (511, 6, 9), (513, 7, 8),
    (640, 8, 25), (300, 9, 5), (300, 10, 8), (300, 12, 4), (300, 13, 7), (300, 14, 9), (301, 16, 17),
    (259, 17, 3), (400, 20, 2), (400, 21, 5), (400, 24, 6), (300, 25, 3), (300, 28, 1), (300, 31, 2),
    (513, 32, 9), (300, 33, 4), (300, 40, 3), (300, 41, 2), (300, 48, 5), (200, 49, 2), (200, 63, 3),
    (200, 64, 2), (200, 65, 2),
    # more than one point per thread
    (160001, 4, 5), (160003, 7, 17), (120001, 11, 5), (117001, 16, 6), (80003, 19, 3), (80001, 24, 3),
    (120007, 27, 3), (120001, 32, 3), (80001, 40, 3), (80001, 47, 3), (80003, 50, 2),
]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,d,k", SHAPES)
def test_posteriors_match_numpy(gpu_lib, precision, n, d, k):
    u = U64 if precision == "fp64" else U32
    X, G = problem(n, d, k, 1000 * d + k)
    with CudaMatrixEM(d, n, k, precision=precision) as em:
        em.CopyDataset(X)
        em.SetMixture(G)
        em.InitDensities()
        logl = em.PrecomputeDensityMatrix()
        R = em.Posteriors()
    ref, lse, dl = reference(X, G, u)
    # each log density off by dl moves a posterior by a factor exp(2 dl); k
    # additions, an exponential and a logarithm or a division on top
    tol = ref * np.expm1(2 * dl + (k + 16) * u)[:, None] + 2.0 ** -126
    assert np.all(np.abs(R - ref) <= tol), float(np.max(np.abs(R - ref) / tol))
    bound = np.sum(dl + (k + 16) * u * (1 + np.abs(lse))) + U64 * n * np.abs(lse).sum()
    assert abs(logl - lse.sum()) <= bound


@pytest.mark.parametrize("d", [1, 15, 16, 17, 32, 33, 48, 49, 64])
def test_mixed_posteriors_match_numpy(gpu_lib, d):
    """the tensor-core E-step at the edges of its 16-wide blocks of dimensions"""
    n, k = 1000, 5
    X, G = problem(n, d, k, 50 + d)
    with CudaMatrixEM(d, n, k, precision="mixed") as em:
        em.CopyDataset(X)
        em.SetMixture(G)
        em.InitDensities()
        em.PrecomputeDensityMatrix()
        R = em.Posteriors()
    # x and W carry 22 bits each without the product of their low halves, and an
    # accumulator is cut to 24 bits up to 12 times: W x to 2^-19 of |W| |x|
    ref, _, _ = reference(X, G, U32)
    X64, dl = X.astype(np.float64), np.zeros(n)
    for j in range(k):
        W = solve_triangular(cholesky(G.covs[j], lower=True), np.eye(d), lower=True)
        y = (X64 - G.means[j]) @ W.T
        dy = 2.0 ** -19 * (np.abs(X64) + np.abs(G.means[j])) @ np.abs(W).T
        e = np.sum(np.abs(y) * dy + 0.5 * dy * dy, axis=1) + (d + 8) * U32 * (np.sum(y * y, axis=1) + d)
        dl = np.maximum(dl, e)
    # FP16 hi + lo posteriors: 22 bits down to FP16's smallest steps
    tol = ref * (np.expm1(2 * dl) + (k + 16) * 2.0 ** -22)[:, None] + 2.0 ** -24
    assert np.all(np.abs(R - ref) <= tol), float(np.max(np.abs(R - ref) / tol))


def test_batch_weights_match_numpy(gpu_lib):
    shapes = [(1, 17, 1), (511, 20, 5), (513, 24, 4), (1025, 23, 13), (512, 25, 3), (700, 32, 9), (600, 16, 9),
              (600, 9, 8), (600, 8, 17), (600, 5, 16), (600, 3, 33)]
    data = [problem(n, d, k, 7 * d + k) for n, d, k in shapes]
    with CudaBatchEM([(d, n, k) for n, d, k in shapes], precision="fp32", max_sweeps=1) as b:
        b.SetParameters(1, 1e-12, 1e300, 0.0)
        b.CopyDatasets([X for X, _ in data])
        for i, (_, G) in enumerate(data):
            b.SetMixture(i, G)
        b.TrainNoCopy()
        got = [b.GetMixture(i) for i in range(len(data))]
    for (X, G), H, (n, d, k) in zip(data, got, shapes):
        ref, _, dl = reference(X, G, U32)
        # posteriors as above, then FP32 sums over at most n rows
        tol = np.mean(ref * np.expm1(2 * dl + (k + 16 + n) * U32)[:, None], axis=0) + 2.0 ** -126
        assert np.all(np.abs(H.weights - ref.mean(axis=0)) <= tol)
