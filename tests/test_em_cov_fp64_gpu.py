"""The FP64 covariance sums of more than one block per dimension (SimpleMatrixEM::
MStep, EM2/MatrixEM.cpp:53-99,363-375) at the edges of their blocks, unit splits
and tiles, against FP64 numpy."""
import numpy as np
import pytest

from test_em_cov_gpu import check_covariances, one_mstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [
    (1, 9, 1),              # one row, most point groups
    (2, 12, 300),           # many components, fewer rows than a tile
    (9001, 13, 200),
    (4099, 20, 60),
    (777, 33, 11),
    (513, 64, 85),          # units that do not divide by 256
    (1030, 65, 20),         # three padded dimensions, 4-byte copies
    (640, 130, 4),
    (515, 200, 9),          # 8 x 8 blocks
    (300, 255, 3),
    (301, 256, 30),
    (200003, 10, 2),        # many tiles per chunk
])
def test_fp64_covariances_match_numpy(gpu_lib, n, d, k):
    rng = np.random.default_rng(10 * d + k)
    X = (rng.normal(0.0, 3.0, (n, d)) + rng.normal(0.0, 2.0, d)).astype(np.float32)
    mu, cov, R = one_mstep(X, k, "fp64", seed=d)
    live = R.sum(axis=0) > 1e-200
    check_covariances(X, mu[live], cov[live], R[:, live], "fp64", n)
