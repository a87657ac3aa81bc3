"""Riemann fluxes against the oracle where their forms change: pressure ratios and Mach
numbers on both sides of the short series of the HLLC shear factor (|z| = 0.04, |t| = 1/16),
gas at rest, supersonic flow in both directions, equal and unequal states, every direction.

The right-hand side of a cell differences fluxes that agree to about 20 roundings of 2^-53
of their scale, so RHS differences stay below 1e-14 / dx of the flux scale; the cells' own
linear reconstruction adds as much again."""
import numpy as np
import pytest

import kfvm_abi as abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,eq,rs", [(2, abi.KFVM_EQ_HYDRO, abi.KFVM_RS_HLLC), (3, abi.KFVM_EQ_HYDRO, abi.KFVM_RS_HLLC),
                                       (3, abi.KFVM_EQ_HYDRO, abi.KFVM_RS_HLL), (2, abi.KFVM_EQ_MHD_GLM, abi.KFVM_RS_HLL),
                                       (3, abi.KFVM_EQ_MHD_GLM, abi.KFVM_RS_LLF)])
@pytest.mark.parametrize("amp", [0.0, 1e-9, 1e-3, 0.03, 0.12])
@pytest.mark.parametrize("mach", [0.0, 0.05, 1.0, 3.0])
def test_flux_forms(dim, eq, rs, amp, mach, gpu, product_lib, oracle_lib):
    n = (19, 10, 5)[:dim]
    cfg = abi.make_config(dim, eq, *n, rs=rs)
    cfg.indicator = abi.KFVM_IND_NONE
    g, o = product_lib.Solver(cfg), oracle_lib.OracleSolver(cfg)
    g.set_indicator(abi.KFVM_IND_NONE)
    o.set_indicator(abi.KFVM_IND_NONE)
    rng = np.random.default_rng(int(1e6 * (amp + mach)) + dim)
    c = abi.ncells(cfg)
    # bounded noise: Gaussian noise of 0.24 left a cell with a negative pressure, whose
    # fluxes are NaN on both sides
    rho = 1.0 + amp * rng.uniform(-1.5, 1.5, c)
    p = 0.8 * (1.0 + 2.0 * amp * rng.uniform(-1.5, 1.5, c))
    vel = mach * np.array([[0.8], [-0.5], [0.3]]) * (1.0 + amp * rng.standard_normal((3, c)))
    u = np.zeros((g.nv, c))
    u[0], u[1:4] = rho, rho * vel
    u[4] = p / (cfg.gamma - 1.0) + 0.5 * rho * (vel ** 2).sum(0)
    if eq == abi.KFVM_EQ_MHD_GLM:
        b = np.array([[0.4], [0.3], [-0.2]]) * (1.0 + amp * rng.standard_normal((3, c)))
        u[5:8] = b
        u[8] = amp * rng.standard_normal(c)
        u[4] += 0.5 * (b ** 2).sum(0) + 0.5 * u[8] ** 2
    g.set_state(u)
    o.set_state(u)
    rg, vg = g.eval_rhs()
    ro, vo = o.eval_rhs()
    assert abs(vg - vo) <= 1e-13 * abs(vo)
    scale = np.abs(u).max() * vo * max(cfg.nx, cfg.ny, cfg.nz)
    assert np.abs(rg - ro).max() <= 4e-14 * scale, np.abs(rg - ro).max() / scale


def hllc(uL, uR, g):
    """The literal low-Mach / shear-corrected HLLC flux along x (Hydro_Riemann.H:26-187), with
    the shear factor 0 where the pressures are equal."""
    with np.errstate(all="ignore"):
        (rL, vL, pL), (rR, vR, pR) = [(u[0], u[1:4] / u[0], (g - 1.0) * (u[4] - 0.5 * (u[1:4] ** 2).sum() / u[0]))
                                      for u in (uL, uR)]
        aL, aR = np.sqrt(g * pL / rL), np.sqrt(g * pR / rR)
        wL, wR = np.sqrt(rL), np.sqrt(rR)
        v = (wL * vL + wR * vR) / (wL + wR)
        h = (wL * (uL[4] + pL) / rL + wR * (uR[4] + pR) / rR) / (wL + wR)
        a = np.sqrt((g - 1.0) * (h - 0.5 * (v ** 2).sum()))
        sL, sR = min(vL[0] - aL, v[0] - a), max(vR[0] + aR, v[0] + a)
        psL, psR = rL * (sL - vL[0]), rR * (sR - vR[0])
        sS = ((pR - pL) + (psL * vL[0] - psR * vR[0])) / (psL - psR)
        pS = 0.5 * ((pL + pR) + psL * (sS - vL[0]) + psR * (sS - vR[0]))
        left = sL >= 0.0 or sS >= 0.0
        u, w, p, s = (uL, vL, pL, sL) if left else (uR, vR, pR, sR)
        F = w[0] * u
        F[1] += p
        F[4] += w[0] * p
        if not (0.0 <= sL or sR <= 0.0):
            M = np.fmax(np.sqrt((vL ** 2).sum()) / aL, np.sqrt((vR ** 2).sum()) / aR)
            psi = psL * psR / (psR - psL)
            shear = 0.0 if pL == pR else 1.0 - (min(pL, pR) / max(pL, pR)) ** M
            M = np.fmin(M, 1.0)
            fM = M * np.sqrt(4.0 + (1.0 - M * M) ** 2) / (1.0 + M * M)
            d = 1.0 / (s - sS)
            pf = psi * (fM - 1.0) * (vR[0] - vL[0]) + s * pS * d
            sh = psi * shear * s * d * (vR - vL)
            F = sS * d * (s * u - F)
            F += np.array([0.0, pf, sh[1], sh[2], sS * pf])
        return F


@pytest.mark.parametrize("shift", [0.0, 0.25, -0.25])
def test_cold_gas_flux(shift, gpu, product_lib):
    """Zero pressure on both sides of a face, exactly: the Mach number is infinite or not a
    number, the shear factor of equal pressures is 0, and the fluxes stay finite; and the same
    velocities at equal, small and unequal pressures.  Sums of about 20 terms of the flux
    scale (2 here): 20 roundings of 2^-53 each is 5e-15, with the divisor psL - psR >= 1 / 2."""
    rng = np.random.default_rng(3)
    gamma = 1.5
    # all are small binary fractions, so that E - m^2 / (2 rho) is the pressure exactly
    rho = rng.choice([0.5, 1.0, 2.0], (2, 64))
    vel = rng.integers(-4, 5, (2, 3, 64)) / 8.0
    vel[0, 0], vel[1, 0] = 1.0 + shift, -1.0 + shift   # colliding
    for pL, pR in ((0.0, 0.0), (0.25, 0.25), (2.0 ** -30, 2.0 ** -30), (0.5, 0.25)):
        u = np.zeros((2, 5, 64))
        u[:, 0], u[:, 1:4] = rho, rho[:, None] * vel
        u[:, 4] = 0.5 * rho * (vel ** 2).sum(1) + np.array([pL, pR])[:, None] / (gamma - 1.0) * (np.array([pL, pR])[:, None] > 0)
        F, s = product_lib.selftest_flux(abi.KFVM_EQ_HYDRO, abi.KFVM_RS_HLLC, gamma, u[0], u[1])
        want = np.stack([hllc(u[0, :, t], u[1, :, t], gamma) for t in range(64)], 1)
        assert np.isfinite(want).all() and np.isfinite(F).all() and np.isfinite(s).all(), (pL, pR)
        assert np.abs(F - want).max() <= 2e-14 * np.abs(want).max(), (pL, pR)
