"""The mixed p' solve's run passes (csrc/hs_run.cuh: the V-cycle's levels of a
million cells and more by 16-byte runs) against the per-cell passes
(p_level0 = 1).  Both evaluate every point update in the same order and sum
<r, z> in the same order, so the fields are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["u", "v", "w", "p", "T", "p_prime"]


# odd sizes, a row of one run past the pitch (nx + 2 a multiple of four and one
# more), thin levels, and one with two levels in run passes
@pytest.mark.parametrize("dims,blocks", [((101, 100, 101), [(20, 50, 30, 60, 10, 40)]),
                                         ((62, 127, 129), [(5, 20, 1, 30, 60, 90)]),
                                         ((999, 33, 31), [(400, 500, 10, 20, 5, 25)]),
                                         ((255, 192, 192), [(60, 90, 50, 90, 80, 120), (150, 170, 1, 40, 10, 30)])])
@pytest.mark.parametrize("sweeps", [0, 1])
def test_run_passes_equal_per_cell_passes(dims, blocks, sweeps):
    import hsolver_b200
    from hsolver_b200 import cases
    deck = cases.channel(*dims, blocks)
    out = []
    for form in (0, 1):
        c = hsolver_b200.Channel(deck, re=200.0, precision=hsolver_b200.PREC_MIXED, p_level0=form, p_tol=1e-5,
                                 t_tol=0.5, t_maxiter=1, p_mg_sweeps=sweeps)
        ctype, _ = hsolver_b200.Case(deck).cell_types()
        c.set_solid(np.full(c.nblocks, 50.0), np.where(ctype == 1, 1.0, 0.0))
        c.init()
        st = c.step(2)
        out.append((st["pcg_iters"], {f: c.field(f) for f in FIELDS}))
        c.close()
    assert out[0][0] == out[1][0] > 1
    for f in FIELDS:
        assert np.array_equal(out[0][1][f], out[1][1][f]), f
