"""The parity form of the linear reconstruction (two Gauss points; Euler, Navier-Stokes,
GLM-MHD): the mirror symmetry of the weights that it rests on, on the CPU, and its
face states, flags and limiter against the oracle at the edges of its blocks: rows of 32
cells with remainders, chunks of planes down to one, odd row pitches, the smallest
grid, every kind of boundary.

The bound on the face states: a point's sum has 33 products of weights below 0.8 with
the stencil's values, so either side's rounding stays below 33 x 2^-53 x 0.8 x 33 of the
largest value, which is 1e-13; with the WENO cells' longer sums the suite uses 1e-12.
"""
import numpy as np
import pytest

import kfvm_abi as abi


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("lfac", [2.0, 5.0, 20.0])
def test_weights_are_mirror_images(dim, lfac, product_lib):
    cfg = abi.make_config(dim, abi.KFVM_EQ_MHD_GLM, 24, 17, 11, rs=abi.KFVM_RS_HLL, lfac=lfac)
    st = product_lib.stencil(cfg)
    C = st.n_cells
    off = [tuple(o) for o in np.array(st.off)[:dim, :C].T.tolist()]
    cell = {o: c for c, o in enumerate(off)}
    point = {}  # position, in signs (2: on the face) -> weights
    for f in range(2 * dim):
        ax, side = f // 2, 1 if f % 2 else -1
        rest = [d for d in range(dim) if d != ax]
        for q in range(st.nqf):
            qs = [q] if dim == 2 else [q // 2, q % 2]
            p = [0] * dim
            p[ax] = 2 * side
            for d, b in zip(rest, qs):
                p[d] = 1 if b else -1
            point[tuple(p)] = np.array(st.face_w[0][f][q][:C])
    for q in range(st.nqc):
        b = [q >> (dim - 1 - d) & 1 for d in range(dim)]
        point[tuple(1 if x else -1 for x in b)] = np.array(st.cell_w[0][q][:C])
    assert len(point) == 2 * dim * st.nqf + st.nqc
    for p, w in point.items():
        assert abs(w.sum() - 1.0) < 2e-15
        for d in range(dim):
            mirror = tuple(-x if k == d else x for k, x in enumerate(p))
            perm = [cell[tuple(-x if k == d else x for k, x in enumerate(o))] for o in off]
            assert np.array_equal(w, point[mirror][perm])


GRIDS = [(2, 3, 3, 1), (2, 33, 9, 1), (2, 31, 8, 1), (2, 70, 25, 1), (3, 3, 3, 3), (3, 33, 4, 7), (3, 31, 6, 3),
         (3, 65, 3, 12), (3, 8, 70, 41)]


@pytest.mark.gpu
@pytest.mark.parametrize("eq", [abi.KFVM_EQ_HYDRO, abi.KFVM_EQ_NAVIERSTOKES, abi.KFVM_EQ_MHD_GLM])
@pytest.mark.parametrize("dim,nx,ny,nz", GRIDS)
def test_block_edges_against_oracle(dim, nx, ny, nz, eq, gpu, product_lib, oracle_lib):
    bc = [["periodic"], ["outflow"], ["reflecting", "outflow", "noslip"]][(nx + ny + nz) % 3]
    bc = (bc * 6)[:6]
    cfg = abi.make_config(dim, eq, nx, ny, nz, bc=bc, gamma=5.0 / 3.0, reynolds=100.0,
                          rs=abi.KFVM_RS_HLL if eq == abi.KFVM_EQ_MHD_GLM else abi.KFVM_RS_HLLC)
    g, o = product_lib.Solver(cfg), oracle_lib.OracleSolver(cfg)
    g.init_ic(abi.KFVM_IC_SMOOTH_WAVE)
    u = g.get_state()
    rng = np.random.default_rng(7)
    # a jump in density and pressure across the middle of the grid, and noise
    k = np.arange(u.shape[1])
    half = (k % nx) > nx // 2
    u[0] *= np.where(half, 1.0, 0.3) * (1.0 + 1e-3 * rng.standard_normal(u.shape[1]))
    u[1:4] *= np.where(half, 1.0, 0.3)
    u[4] *= np.where(half, 1.0, 0.4)
    g.set_state(u)
    o.set_state(u)
    o.keep_faces(True)
    for _ in range(2):  # the second evaluation reads the first one's theta
        rg, vg = g.eval_rhs()
        ro, vo = o.eval_rhs()
    assert abs(vg - vo) <= 1e-13 * abs(vo)
    for d in range(dim):
        fg, fo = g.faces(d), o.faces(d)
        scale = np.abs(fo).max(axis=(0, 1, 3), keepdims=True)
        assert np.all(np.abs(fg - fo) <= 1e-12 * np.maximum(scale, 1e-3 * scale.max())), d
    (ag, tg), (ao, to) = g.flags(), o.flags()
    assert np.array_equal(ag, ao)
    assert np.allclose(tg, to, rtol=0, atol=1e-10)
    assert np.abs(rg - ro).max() <= 1e-10 * np.abs(ro).max()


@pytest.mark.gpu
def test_more_rows_than_a_launch_has_in_y(gpu, product_lib, oracle_lib):
    """65600 rows of cells in y, above the 65535 of a launch's second dimension.  The cells are
    1 / 65600 high: fluxes of a few units with 20 roundings of 2^-53 each, and initial values
    one rounding apart, differ by 1e-14, and the right-hand side by that times 65600."""
    cfg = abi.make_config(3, abi.KFVM_EQ_HYDRO, 3, 65600, 3, bc=["periodic"] * 6, gamma=1.4)
    g, o = product_lib.Solver(cfg), oracle_lib.OracleSolver(cfg)
    for s in (g, o):
        s.set_indicator(abi.KFVM_IND_NONE)
        s.init_ic(abi.KFVM_IC_SMOOTH_WAVE)
    rg, vg = g.eval_rhs()
    ro, vo = o.eval_rhs()
    assert abs(vg - vo) <= 1e-12 * abs(vo)
    assert np.abs(rg - ro).max() <= 1e-9 * np.abs(ro).max()
