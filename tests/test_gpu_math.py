"""The refined device arithmetic (physics.cuh) against 80-bit results: square root, the shear
factor 1 - r^M of HLLC on both sides of its series' limits, and the indicator's power, on whose
error the margin of the flags rests."""
import numpy as np
import pytest

import kfvm_abi as abi

pytestmark = pytest.mark.gpu
L = np.longdouble


def test_square_root(gpu, product_lib):
    """The correction by the residual leaves half an ulp and the rounding of the residual's
    product: within one ulp of the rounded root over the whole range that is not taken as 0."""
    rng = np.random.default_rng(1)
    x = 10.0 ** rng.uniform(-289.9, 308.0, 1 << 20)
    x = np.concatenate([x, 1.0 + rng.uniform(-1e-3, 1e-3, 1 << 16), np.arange(1.0, 4096.0) ** 2,
                        [1.7976931348623157e308, 1.0, 4.0, 0.25, 2.0 ** 1000]])
    got, want = product_lib.selftest_math(product_lib.SELFTEST_SQRT, x), np.sqrt(x)
    assert np.abs(got.view(np.int64) - want.view(np.int64)).max() <= 1
    got = product_lib.selftest_math(product_lib.SELFTEST_SQRT, np.array([0.0, 1e-291, -1e-291, 5e-324]))
    assert np.array_equal(got, np.zeros(4))
    assert np.isnan(product_lib.selftest_math(product_lib.SELFTEST_SQRT, np.array([-1.0, -1e-280, np.nan]))).all()


def test_shear_factor(gpu, product_lib):
    """Series (|z| < 0.04, |t| < 1/16): its four roundings of z, six of each series and one each
    of t and the product, relative to the result.  Otherwise exp of M log r, whose exponent's
    rounding of 2^-52 |t| meets the result times e^t, and the cancellation against 1: absolute."""
    rng = np.random.default_rng(2)
    n = 1 << 20
    d = 10.0 ** rng.uniform(-14, 0, n)                     # pMin / pMax = 1 - d
    d[: n // 4] = 0.0769 * (1.0 + 1e-4 * rng.standard_normal(n // 4))   # about |z| = 0.04
    pMax = 10.0 ** rng.uniform(-6, 6, n)
    pMin = pMax * (1.0 - np.minimum(d, 1.0 - 1e-9))
    M = 10.0 ** rng.uniform(-6, 2, n)
    t0 = np.log1p(-np.minimum(d, 1.0 - 1e-9))
    edge = rng.random(n) < 0.25                            # about |t| = 1/16
    M[edge] = np.clip(0.0625 / np.abs(t0[edge]), 1e-6, 1e6) * (1.0 + 1e-3 * rng.standard_normal(edge.sum()))
    got = product_lib.selftest_math(product_lib.SELFTEST_ONE_MINUS_POW, pMin, pMax, M)
    t = L(M) * np.log1p((L(pMin) - L(pMax)) / L(pMax))
    want = -np.expm1(t)
    err = np.abs(L(got) - want)
    z = (pMin - pMax) / (pMin + pMax)
    series = (np.abs(z) < 0.0399) & (np.abs(t) < 0.0624)
    assert series.sum() > n // 10 and (~series).sum() > n // 10
    assert (err[series] / want[series]).max() <= 20 * 2.0 ** -53
    # of the logarithm's argument: two roundings, times M
    bound = 2.0 ** -52 * (2.0 + np.exp(t) * (2.0 * np.abs(t) + 2.0 * M))
    assert (err <= bound).all(), (err / bound).max()


def test_shear_factor_of_equal_pressures(gpu, product_lib):
    p = np.array([0.0, 1e-300, 1.0, 1e300, 0.0, -1.0])
    M = np.array([np.nan, np.nan, 0.5, np.inf, np.inf, np.nan])
    assert np.array_equal(product_lib.selftest_math(product_lib.SELFTEST_ONE_MINUS_POW, p, p, M), np.zeros(6))


@pytest.mark.parametrize("gamma", [abi.stof(1.001), 4.0 / 3.0, abi.stof(1.4), abi.stof(1.66666666666666), 3.0])
def test_power_of_the_indicator(gamma, gpu, product_lib):
    """rho^-gamma to 1e-9, which kWenoRoundEps adds to the rounding to FP32; outside of the
    range where that holds, not a number, which has the flags recomputed."""
    rng = np.random.default_rng(3)
    n = 1 << 20
    rho = 10.0 ** rng.uniform(-80, 80, n)
    rho[: n // 2] = np.exp(rng.uniform(-2, 2, n // 2))
    e = rng.integers(-20, 20, n // 8)
    rho[: n // 8] = np.sqrt(2.0) * 2.0 ** e * (1.0 + 1e-12 * rng.standard_normal(n // 8))   # where the mantissa folds
    rho[n // 8: n // 4] = 2.0 ** rng.integers(-60, 60, n // 8)
    got = product_lib.selftest_math(product_lib.SELFTEST_POWER, np.full(n, gamma), rho)
    t = -L(gamma) * np.log2(L(rho))
    ok = np.abs(t) < 999.0
    assert np.isfinite(got[ok]).all()
    assert np.abs(L(got[ok]) / np.exp2(t[ok]) - 1).max() <= 1e-9
    bad = np.array([0.0, -1.0, np.nan, np.inf, 1e-300, 1e300, 5e-324])
    assert np.isnan(product_lib.selftest_math(product_lib.SELFTEST_POWER, np.full(7, gamma), bad)).all()


@pytest.mark.parametrize("eq,rs", [(abi.KFVM_EQ_HYDRO, abi.KFVM_RS_HLLC), (abi.KFVM_EQ_HYDRO, abi.KFVM_RS_HLL),
                                   (abi.KFVM_EQ_MHD_GLM, abi.KFVM_RS_HLL), (abi.KFVM_EQ_MHD_GLM, abi.KFVM_RS_LLF),
                                   (abi.KFVM_EQ_SRHYDRO, abi.KFVM_RS_HLL)])
@pytest.mark.parametrize("dir", [0, 1, 2])
def test_flux_is_consistent_and_turns_with_the_axes(eq, rs, dir, gpu, product_lib):
    """Between equal states the flux is the physical one, whatever the solver: F(u, u) of one
    solver equals the other's; and the flux in direction d of a state is that in x of the
    state turned by d axes, to rounding."""
    rng = np.random.default_rng(4)
    n = 4096
    nv = 9 if eq == abi.KFVM_EQ_MHD_GLM else 5
    rho, p = rng.uniform(0.1, 2.0, (2, n)), rng.uniform(0.05, 2.0, (2, n))
    v = rng.uniform(-0.5, 0.5, (2, 3, n))
    u = np.zeros((2, nv, n))
    u[:, 0], u[:, 1:4] = rho, rho[:, None] * v
    u[:, 4] = p / 0.4 + 0.5 * rho * (v ** 2).sum(1)
    if eq == abi.KFVM_EQ_SRHYDRO:
        W = 1.0 / np.sqrt(1.0 - (v ** 2).sum(1))
        h = rho + 1.4 / 0.4 * p
        u[:, 0], u[:, 1:4], u[:, 4] = rho * W, (h * W ** 2)[:, None] * v, h * W ** 2 - p
    if nv == 9:
        u[:, 5:8] = rng.uniform(-1, 1, (2, 3, n))
        u[:, 8] = rng.uniform(-0.1, 0.1, (2, n))
        u[:, 4] += 0.5 * (u[:, 5:8] ** 2).sum(1) + 0.5 * u[:, 8] ** 2

    def turned(a):
        b = a.copy()
        for k in range(3):
            b[..., 1 + k, :] = a[..., 1 + (dir + k) % 3, :]
            if nv == 9:
                b[..., 5 + k, :] = a[..., 5 + (dir + k) % 3, :]
        return b

    F, s = product_lib.selftest_flux(eq, rs, 1.4, u[0], u[1], dir=dir, ch=0.7)
    t = turned(u)
    Fx, sx = product_lib.selftest_flux(eq, rs, 1.4, t[0], t[1], dir=0, ch=0.7)
    scale = np.abs(Fx).max()
    # the squares of the components are summed in the order of the axes: one rounding each
    assert np.abs(turned(F) - Fx).max() <= 2e-14 * scale
    assert np.abs(s - sx).max() <= 2e-14 * np.abs(sx).max()
    A, _ = product_lib.selftest_flux(eq, rs, 1.4, u[0], u[0], dir=dir, ch=0.7)
    B, _ = product_lib.selftest_flux(eq, abi.KFVM_RS_LLF, 1.4, u[0], u[0], dir=dir, ch=0.7)
    assert np.abs(A - B).max() <= 2e-14 * np.abs(B).max()
