"""Channels whose every p' level is handled by block 0 alone: the z-marching
form of the finest level (p_level0 = 2) does not apply there, and the solve is
the grid-wide form's (p_level0 = 1), bit for bit over several CG iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# block 0 takes levels of at most 2048 cells whose x and rhs, with the coarser
# levels', fit in 64 KB: 16x12x10 in FP32 only (67.7 KB in FP64, where the
# z-marching form runs); 4x4x4 has the directly solved level alone
@pytest.mark.parametrize("precision,dims,block", [(0, (13, 11, 9), (4, 6, 2, 5, 3, 7)), (1, (13, 11, 9), (4, 6, 2, 5, 3, 7)),
                                                  (1, (16, 12, 10), (5, 8, 3, 6, 1, 4)),
                                                  (0, (4, 4, 4), (2, 2, 2, 2, 2, 2)), (1, (4, 4, 4), (2, 2, 2, 2, 2, 2))])
def test_z_marching_falls_back_on_small_grids(precision, dims, block):
    import hsolver_b200
    from hsolver_b200 import cases
    deck = cases.channel(*dims, [block])
    ctype, _ = hsolver_b200.Case(deck).cell_types()
    out = []
    for form in (1, 2):
        c = hsolver_b200.Channel(deck, re=100.0, precision=precision, p_level0=form, p_tol=1e-6)
        c.set_solid(np.full(c.nblocks, 50.0), np.where(ctype == 1, 1.0, 0.0))
        c.init()
        its = [c.step(1)["pcg_iters"] for _ in range(3)]
        out.append((its, {f: c.field(f) for f in ("u", "v", "w", "p", "T", "p_prime")}))
        c.close()
    assert out[0][0] == out[1][0]
    if dims[0] > 4:
        assert min(out[0][0]) > 2
    for f in out[0][1]:
        assert np.array_equal(out[0][1][f], out[1][1][f]), f
