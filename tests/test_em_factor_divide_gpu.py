"""The multipliers of the factorisation (NormalDensity::Init, EM2/NormalDensity.cpp:
43-65): divided by pivots of any mantissa and exponent, at both ends of the range
that the corrected reciprocal covers, subnormal and infinite ones."""
from fractions import Fraction

import numpy as np
import pytest

from fastem_gb300 import CudaMatrixEM, GaussianMixture

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def inverse_factors(S):
    k, d = S.shape[:2]
    with CudaMatrixEM(d, 4, k, precision="fp64") as em:
        em.SetMixture(GaussianMixture(np.full(k, 1.0 / k), np.zeros((k, d)), S))
        em.InitDensities()
        return em.Factors()[0].transpose(0, 2, 1)


def exact_root(x):
    """The square root of a fraction to 2^-80 of it, as a fraction."""
    s = 1 << 400
    n = x.numerator * x.denominator * s * s
    r = 1 << ((n.bit_length() + 1) // 2)
    while True:
        t = (r + n // r) // 2
        if t >= r:
            return Fraction(r, x.denominator * s)
        r = t


@pytest.mark.parametrize("exponents", [(-40, 40), (-962, -955), (955, 963), (-1022, -990), (-1060, -1030), (990, 1000)])
def test_multipliers_are_rounded_quotients(gpu_lib, exponents):
    k = 512
    rng = np.random.default_rng(exponents[0] + 2000)
    e = rng.integers(exponents[0], exponents[1], k)
    p = np.ldexp(1.0 + rng.random(k), e)
    p[:4] = np.ldexp([1.0, np.nextafter(2.0, 0.0), np.nextafter(1.0, 2.0), 1.5], int(e[0]))
    # S = [[p, u], [u, 1]] with u^2 / p around 0.1
    u = 0.3 * np.sqrt(p) * (0.5 + rng.random(k)) * rng.choice([-1.0, 1.0], k)
    S = np.empty((k, 2, 2))
    S[:, 0, 0], S[:, 1, 1] = p, 1.0
    S[:, 0, 1] = S[:, 1, 0] = u
    W = inverse_factors(S)
    for j in range(k):
        P, V = Fraction(p[j]), Fraction(u[j])
        d2 = exact_root(1 - V * V / P)
        # W_00 = 1 / sqrt(p), W_10 = -(u / p) / sqrt(1 - u^2 / p), W_11 = 1 / sqrt(1 - u^2 / p): a
        # rounding each for the quotient, u m (0.2 of the pivot at most, taken off 0.8 or more), the
        # root, its reciprocal and the product
        for got, ref, ulps in ((W[j, 0, 0], 1 / exact_root(P), 2), (W[j, 1, 0], -V / P / d2, 5), (W[j, 1, 1], 1 / d2, 3)):
            assert abs(Fraction(got) - ref) <= ulps * Fraction(U) * abs(ref), (j, p[j], u[j], got, float(ref))


def test_an_infinite_pivot_divides_to_zero(gpu_lib):
    S = np.array([[[np.inf, 2.0], [2.0, 4.0]]])
    W = inverse_factors(S)[0]
    assert W[0, 0] == 0.0 and W[1, 0] == 0.0 and W[1, 1] == 0.5
