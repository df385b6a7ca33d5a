"""A covariance that is not positive definite (NormalDensity::Init, EM2/
NormalDensity.cpp:43-65): the non-positive pivot in every part of a panel and
of a warp, the component that is named, and the handle afterwards."""
import ctypes

import numpy as np
import pytest

from fastem_gb300 import CudaBatchEM, CudaMatrixEM, GaussianMixture
from fastem_gb300 import _capi as C
from test_em_factor_gpu import covariances

pytestmark = pytest.mark.gpu


def spoil(S, q):
    """S with pivot q of its Cholesky factorisation below zero, those before it as they were."""
    T = S.copy()
    r = np.linalg.solve(S[:q, :q], S[:q, q]) if q else np.zeros(0)
    T[q, q] = S[q, :q] @ r - 0.5
    return T


@pytest.mark.parametrize("d", [1, 2, 24, 32, 33, 64, 65, 118, 119, 160, 256])
def test_failed_pivot_at_every_place(gpu_lib, d):
    k = 9
    S = covariances(d, k, seed=3 * d)
    with CudaMatrixEM(d, 64, k, precision="fp64") as em:
        def init(covs):
            em.SetMixture(GaussianMixture(np.full(k, 1.0 / k), np.zeros((k, d)), covs))
            failed = ctypes.c_int(-7)
            return gpu_lib.fem_em_init_densities(em.handle, ctypes.byref(failed)), failed.value

        for q in sorted({0, 1, 7, 30, 31, 32, 33, d // 2, 63, 64, 95, 96, d - 2, d - 1}):
            if not 0 <= q < d:
                continue
            T = S.copy()
            T[5], T[8] = spoil(S[5], q), spoil(S[8], d - 1 - q)
            assert init(T) == (C.FEM_ERR_CHOLESKY, 5)
        # every component stops, each at a pivot of its own
        assert init(np.stack([spoil(S[j], j * (d - 1) // (k - 1)) for j in range(k)])) == (C.FEM_ERR_CHOLESKY, 0)
        assert init(S) == (C.FEM_OK, -1)
        U, logdet = em.Factors()
        np.testing.assert_allclose(logdet, np.linalg.slogdet(S)[1], rtol=1e-12, atol=1e-10)


def test_failed_pivot_stops_only_its_fit(gpu_lib):
    shapes = [(d, 500, 3) for d in (1, 4, 7, 16, 31, 32) for _ in range(2)]
    rng = np.random.default_rng(11)
    with CudaBatchEM(shapes, precision="fp32", max_sweeps=2) as b:
        b.CopyDatasets([rng.standard_normal((n, d)).astype(np.float32) for d, n, _ in shapes])
        for i, (d, _, k) in enumerate(shapes):
            S = np.broadcast_to(np.eye(d), (k, d, d)).copy()
            if i % 2:
                S[1] = spoil(covariances(d, 1, seed=i)[0], d - 1 - i % d)
            b.SetMixture(i, GaussianMixture(np.full(k, 1.0 / k), np.zeros((k, d)), S))
        status, _, _ = b.TrainNoCopy()
        assert list(status) == [C.FEM_ERR_CHOLESKY if i % 2 else C.FEM_OK for i in range(len(shapes))]
        assert [b.FailedComponent(i) for i in range(len(shapes))] == [1 if i % 2 else -1 for i in range(len(shapes))]
