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
