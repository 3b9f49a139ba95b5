"""The reference path's wavefront Gauss-Seidel (k_gs_tiles, k_gs_planes) and
its one-block solid solves (k_solid_block) against the oracle, bit for bit
with the pressure solve off: rows that fill, just pass and just miss the 8 x 4
tiles, rows shorter than a chunk, more tiles than resident warps, windows on
both sides of the tile form's limit, solid boxes of one cell, of one plane and
around the shared-memory limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["u_star", "v_star", "w_star", "up", "vp", "wp", "p_temp", "t_temp", "ux", "uy", "uz", "p", "t"]


@pytest.mark.parametrize("dims,blocks", [((7, 8, 5), [(3, 4, 3, 4, 2, 3)]), ((9, 9, 9), [(4, 4, 4, 4, 4, 4)]),
                                         ((5, 17, 13), [(2, 4, 4, 10, 5, 5)]), ((33, 16, 12), [(5, 20, 3, 9, 4, 8)]),
                                         ((5, 203, 107), [(2, 4, 30, 60, 20, 40)]),
                                         ((40, 31, 33), [(2, 29, 2, 29, 2, 30), (33, 38, 3, 8, 3, 3)]),
                                         ((40, 36, 36), [(2, 34, 3, 35, 2, 34)])])
@pytest.mark.parametrize("gs_max", [1, 3, 100])
def test_wavefront_sweeps_bit_exact(dims, blocks, gs_max):
    import hsolver_b200
    from hsolver_b200 import cases
    from oracle import oracle
    prm = {"pcg_maxiter": 0, "gs_max": gs_max}
    op = oracle.default_params()
    for k, v in prm.items():
        setattr(op, k, v)
    deck = cases.channel(*dims, blocks)
    g = hsolver_b200.Solver(deck, hsolver_b200.default_params(**prm))
    o = oracle.OracleCase(deck, op)
    g.init()
    o.init()
    for s in range(3):
        st = g.step(1, stats=True)
        o.step(1)
        os_ = o.stats()
        for f in ("sweeps_u", "sweeps_v", "sweeps_w", "sweeps_t"):
            assert st[f] == os_[f], (s, f)
        assert st["sweeps_solid_max"] == max(os_["sweeps_solid"])
        for f in FIELDS:
            assert np.array_equal(g.field(f), o.field(f)), (s, f)
        for r in range(o.nsolid):
            assert np.array_equal(g.solid(r), o.solid(r)), (s, r)
            assert np.array_equal(g.solid(r, "t"), o.solid(r, "t")), (s, r)
