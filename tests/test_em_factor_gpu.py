"""The per-component FP64 factorisation (NormalDensity::Init, EM2/
NormalDensity.cpp:43-65) at the edges of its forms: L^-1 and log det of random
covariances, and the first non-positive pivot."""
import numpy as np
import pytest

from fastem_gb300 import CudaMatrixEM, GaussianMixture
from fastem_gb300 import _capi as C

pytestmark = pytest.mark.gpu


def covariances(d, k, seed):
    A = np.random.default_rng(seed).standard_normal((k, d, d + 2))
    return A @ A.transpose(0, 2, 1) / d + 0.3 * np.eye(d)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("d", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 118, 119, 128, 160, 186, 187, 256])
def test_factors_match_numpy(gpu_lib, precision, d):
    k, u = 5, 2.0 ** -53
    S = covariances(d, k, seed=d)
    with CudaMatrixEM(d, 64, k, precision=precision) as em:
        em.SetMixture(GaussianMixture(np.full(k, 0.2), np.zeros((k, d)), S))
        em.InitDensities()
        U, logdet = em.Factors()
    for j in range(k):
        W = U[j].T
        assert np.all(np.triu(W, 1) == 0.0)
        L = np.linalg.cholesky(S[j])
        # |L L^T - S| <= (d + 1) u |L||L^T| and |W L - I| <= d u |W||L| componentwise
        B = np.abs(W) @ np.abs(L)
        assert np.all(np.abs(W @ S[j] @ W.T - np.eye(d)) <= 4 * (d + 2) * u * (B @ B.T))
        ref = 2.0 * np.log(np.diag(L)).sum()
        assert abs(logdet[j] - ref) <= 4 * d * (d + 2) * u * np.max(np.diag(B @ B.T))


@pytest.mark.parametrize("d", [1, 32, 64, 100, 119, 200])
def test_first_bad_pivot_is_reported(gpu_lib, d):
    """Eigen's LLT fails on a pivot <= 0: the lowest failing component is named."""
    k = 4
    S = covariances(d, k, seed=d + 1)
    S[2, d - 1, :] = S[2, :, d - 1] = 0.0       # last pivot exactly 0
    S[3, 0, 0] = np.nan
    with CudaMatrixEM(d, 64, k, precision="fp64") as em:
        em.SetMixture(GaussianMixture(np.full(k, 0.25), np.zeros((k, d)), S))
        with pytest.raises(C.FemError) as e:
            em.InitDensities()
        assert e.value.status == C.FEM_ERR_CHOLESKY and "component 2" in str(e.value)
