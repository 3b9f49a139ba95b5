"""A wait between the tiles of a wavefront sweep that runs out.  A limit of no
polls makes every wait run out at its first call, whatever the other tiles
have done: the kernels still return, and the calls that read report it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HS_ERR_INTERNAL = -8
BLOCKS = [(5, 20, 3, 9, 4, 8)]


def _solver(dims=(33, 16, 12), blocks=BLOCKS, **prm):
    import hsolver_b200
    from hsolver_b200 import cases
    s = hsolver_b200.Solver(cases.channel(*dims, blocks), hsolver_b200.default_params(pcg_maxiter=5, **prm))
    s.init()
    return s


def _fails(call, *args, **kw):
    import hsolver_b200
    with pytest.raises(hsolver_b200.HsError) as e:
        call(*args, **kw)
    assert e.value.code == HS_ERR_INTERNAL and "ran out" in str(e.value)


# one tile, a few, more than the resident warps
@pytest.mark.parametrize("dims,blocks", [((7, 8, 5), [(3, 4, 3, 4, 2, 3)]), ((33, 16, 12), BLOCKS),
                                         ((5, 203, 107), [(2, 4, 30, 60, 20, 40)])])
@pytest.mark.parametrize("gs_max", [1, 3])
def test_a_wait_that_runs_out_is_reported(dims, blocks, gs_max):
    s = _solver(dims, blocks, gs_max=gs_max)
    s.set_wait_limit(0)
    s.step(2)
    _fails(s.sync)
    _fails(s.step, 1, stats=True)
    _fails(s.field, "ux")
    _fails(s.solid, 0)
    s.close()


def test_every_reader_reports_it():
    """The calls that hand out the step's outcome without copying a field:
    counters, phase times, device addresses and the energy solve on the
    engine's velocities."""
    from hsolver_b200.adjoint import ChtProblem
    s = _solver()
    s.profile(True)
    prob = ChtProblem(s, k_fluid=1.0, maxiter=10)
    try:
        k, q = np.full(prob.nreg, 10.0), np.zeros(33 * 16 * 12)
        prob.forward(k, q)
        s.set_wait_limit(0)
        s.step(1)
        _fails(prob.velocities)
        _fails(prob.gradient)
        _fails(prob.forward, k, q)
        _fails(s.counters)
        _fails(s.profile_read)
        _fails(s.device_ptr, "u_star")
    finally:
        prob.__del__()  # before its solver


def test_the_limit_leaves_results_alone():
    a, b = _solver(), _solver()
    b.set_wait_limit(1 << 20)
    for s in (a, b):
        s.step(3)
    for f in ("u_star", "v_star", "w_star", "t_temp", "ux", "p", "t"):
        assert np.array_equal(a.field(f), b.field(f)), f


def test_negative_limit_is_refused():
    import hsolver_b200
    s = _solver()
    with pytest.raises(hsolver_b200.HsError) as e:
        s.set_wait_limit(-1)
    assert e.value.code == -1


# a frozen pressure matrix (the default) is assembled once: also that of an
# abandoned first step must not stay
@pytest.mark.parametrize("good_steps", [0, 2])
def test_init_starts_again_after_a_report(good_steps):
    a, b = _solver(), _solver()
    a.step(good_steps)
    a.set_wait_limit(0)
    a.step(2)
    _fails(a.sync)
    a.set_wait_limit(1 << 21)
    a.init()
    for n in (1, 2):
        a.step(n)
        b.step(n)
        for f in ("u_star", "v_star", "w_star", "p_temp", "t_temp", "up", "vp", "wp", "ux", "uy", "uz", "p", "t", "p_prime"):
            assert np.array_equal(a.field(f), b.field(f)), (n, f)
        for w in ("t_temp", "t"):
            assert np.array_equal(a.solid(0, w), b.solid(0, w)), (n, w)
    assert a.counters()["steps"] == good_steps + 2 + 3


def test_init_does_not_hide_an_abandoned_step():
    s = _solver()
    s.set_wait_limit(0)
    s.step(1)
    _fails(s.init)
    s.set_wait_limit(1 << 21)
    s.init()
    s.step(1, stats=True)
