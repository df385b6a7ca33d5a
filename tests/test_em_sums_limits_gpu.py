"""The FP32 M-step sums (SimpleMatrixEM::MStep, EM2/MatrixEM.cpp:309-378) of
several point groups: sums beyond FP32's range, and what the groups' addition
rounds."""
import numpy as np
import pytest

from fastem_gb300 import CudaBatchEM, CudaMatrixEM, GaussianMixture
from fastem_gb300 import _capi as C

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
