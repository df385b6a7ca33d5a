"""The batched M-step sums (SimpleMatrixEM::MStep, EM2/MatrixEM.cpp:319-375) at
the edges of their dimension classes, unit ranges, point groups and work items:
weights, means and covariances of one sweep against FP64 numpy."""
import numpy as np
import pytest

from fastem_gb300 import GaussianMixture
from fastem_gb300.batch import CudaBatchEM
from test_em_estep_gpu import U32, problem, reference

pytestmark = pytest.mark.gpu

# (n, d, k): fewer rows than a tile; odd rows; one unit, and units that
# do not divide by the threads; the largest k; d at and beside the class edges
SHAPES = [(2, 1, 1), (3, 2, 1), (130, 3, 5), (4097, 4, 64), (1001, 4, 7), (63, 5, 2), (2049, 7, 33), (5000, 8, 64),
          (129, 9, 1), (1025, 12, 21), (3001, 16, 64), (500, 16, 3), (127, 17, 2), (2050, 23, 37), (4099, 24, 64),
          (700, 25, 1), (1500, 31, 9), (9001, 32, 64), (255, 32, 26)]


REG = 0.5   # a covariance of few rows is singular without


@pytest.mark.parametrize("chunk", [256, 2048])
def test_sums_match_numpy(gpu_lib, chunk):
    data = [problem(n, d, k, 31 * d + k) for n, d, k in SHAPES]
    tuning = dict(means_chunk=[chunk] * 4, cov_chunk=[chunk] * 4)
    with CudaBatchEM([(d, n, k) for n, d, k in SHAPES], precision="fp32", max_sweeps=1, tuning=tuning) as b:
        b.SetParameters(1, 1e-12, 1e300, REG)
        b.CopyDatasets([X for X, _ in data])
        for i, (_, G) in enumerate(data):
            b.SetMixture(i, G)
        b.TrainNoCopy()
        got = [b.GetMixture(i) for i in range(len(data))]
    for (X, G), H, (n, d, k) in zip(data, got, SHAPES):
        # the start is regularised as well
        tr = np.trace(G.covs, axis1=1, axis2=2)[:, None, None]
        G = GaussianMixture(G.weights, G.means, (1.0 - REG) * G.covs + REG * tr / d * np.eye(d))
        R, _, dl = reference(X, G, U32)
        X64, xmax = X.astype(np.float64), float(np.abs(X).max())
        # posteriors to their own error; then FP32 sums over at most `rows` rows each
        rows = min(n, chunk)
        dR = R * np.expm1(2 * dl + (k + 16) * U32)[:, None] + 2.0 ** -126
        Nj, dN = R.sum(axis=0), dR.sum(axis=0) + (rows + 16) * U32 * R.sum(axis=0)
        assert np.all(np.abs(H.weights - Nj / n) <= 2 * dN / n)
        for j in range(k):
            if dN[j] > 0.25 * Nj[j]:
                continue                                # a component without rows: nothing to compare
            r, dr = R[:, j], dR[:, j] + (rows + 16) * U32 * R[:, j]
            mu = r @ X64 / Nj[j]
            tol = 2 * (dr @ np.abs(X64) + dN[j] * np.abs(mu)) / Nj[j] + 4 * U32 * xmax
            assert np.all(np.abs(H.means[j] - mu) <= tol), (n, d, k, j)
            u = X64 - H.means[j]
            ref = (u * r[:, None]).T @ u / Nj[j]
            a = np.abs(u)
            s = np.sqrt(np.diag(ref))
            tol = 2 * ((a * dr[:, None]).T @ a + dN[j] * np.abs(ref)) / Nj[j] + U32 * (
                8 * xmax * (s[:, None] + s[None, :]) + 8 * U32 * xmax ** 2 + 16 * np.outer(s, s))
            # S' = (1 - REG) S + REG tr(S) / d I, which keeps the trace
            S = (H.covs[j] - REG * np.trace(H.covs[j]) / d * np.eye(d)) / (1.0 - REG)
            tol = tol + REG / (1.0 - REG) * np.trace(tol) / d * np.eye(d)
            assert np.all(np.abs(S - ref) <= tol), (n, d, k, j)
            assert np.array_equal(H.covs[j], H.covs[j].T)
