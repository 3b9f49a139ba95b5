"""The work that users of hsolver_b200 have it do, as measurable cases.

A case is a dict of plain values.  Four kinds, each through the calls a user
makes:

* ``channel``: an outer-iteration loop of the channel conjugate-heat-transfer
  solver (``hsolver_b200.Channel``): start, a number of SIMPLE steps, the five
  fields read back into the program's (pinned) arrays.  Both precisions, the
  three convection schemes, buoyancy, uniform and wall-stretched grids;
* ``adjoint``: one gradient of the heat-sink objective on a frozen flow
  (``Channel.adjoint``: a forward energy solve and the transposed one);
* ``lid``: outer steps of the reference-faithful lid-driven cavity
  (``hsolver_b200.Solver``), then its cell and face results;
* ``pcg``: the stand-alone pressure-correction solve of the C ABI
  (``hs_pcg_solve``) on the caller's device arrays.

Sizes are those of ``hsolver_b200/cases.py``, of the tests and of the bench,
or odd ones between them.
"""
import ctypes
import math
import random

import numpy as np
import torch

import hsolver_b200
from hsolver_b200 import cases as decks

# the bench's inner solves: p' to the reference's rtol, one energy iteration
BENCH = {"p_tol": 1e-5, "t_tol": 0.5, "t_maxiter": 1}
# the library's defaults: p' to 1e-8, the energy residual down by 100
DEFAULT = {"p_tol": 1e-8, "t_tol": 1e-2, "t_maxiter": 200}


def _channel(name, dims, steps, blocks, edges, mixed=False, solver=BENCH, conv=0, ri=0.0, stretched=False, re=400.0):
    c = {"kind": "channel", "nx": dims[0], "ny": dims[1], "nz": dims[2], "steps": steps, "blocks": blocks,
         "edge_lo": edges[0], "edge_hi": edges[1], "mixed": mixed, "conv": conv, "ri": ri, "stretched": stretched,
         "re": re}
    c.update(solver)
    if name:
        c["name"] = name
    return c


def _adjoint(name, dims, blocks, edges, mixed=False, re=400.0):
    c = {"kind": "adjoint", "nx": dims[0], "ny": dims[1], "nz": dims[2], "blocks": blocks, "edge_lo": edges[0],
         "edge_hi": edges[1], "mixed": mixed, "re": re, "tol": 1e-12}
    if name:
        c["name"] = name
    return c


def _lid(name, dims, steps, before, blocks, edges):
    c = {"kind": "lid", "nx": dims[0], "ny": dims[1], "nz": dims[2], "steps": steps, "before": before,
         "blocks": blocks, "edge_lo": edges[0], "edge_hi": edges[1]}
    if name:
        c["name"] = name
    return c


def _pcg(name, dims, tol):
    c = {"kind": "pcg", "nx": dims[0], "ny": dims[1], "nz": dims[2], "tol": tol}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a coarse first look at a geometry, or a test: launches and barriers are all there is
        _channel("channel_small", (24, 12, 12), 20, 1, (3, 4), solver=DEFAULT, re=100.0),
        # the smallest specified channel, run as the library's defaults run it
        _channel("channel_48", (48, 24, 24), 50, 1, (6, 9), solver=DEFAULT, re=100.0),
        # the same channel resolved at the walls (aspect ratio 20), mixed precision
        _channel("channel_stretched_mixed", (48, 24, 24), 50, 1, (6, 9), mixed=True, stretched=True, re=100.0),
        # natural convection with the higher-order scheme, cell counts as a user's geometry gives them
        _channel("channel_ragged_quick", (101, 67, 45), 10, 4, (5, 16), conv=2, ri=1.0),
        # a mid-size study in mixed precision with the hybrid scheme, odd sizes
        _channel("channel_ragged_hybrid_mixed", (203, 75, 110), 10, 6, (8, 24), mixed=True, conv=1),
        # the at-scale channel, both precisions
        _channel("channel_256", (256, 128, 128), 10, 8, (8, 24)),
        _channel("channel_256_mixed", (256, 128, 128), 10, 8, (8, 24), mixed=True),
        # the largest specified channel: the fields no longer fit any cache
        _channel("channel_512_mixed", (512, 256, 256), 4, 32, (8, 48), mixed=True, re=1000.0),
        # one design gradient at the adjoint configuration
        _adjoint("adjoint_128", (128, 64, 64), 4, (8, 24)),
        # the reference's own step: its 50^3 example's size, and at scale
        _lid("lid_50", (50, 50, 50), 5, 20, 2, (8, 16)),
        _lid("lid_256", (256, 128, 128), 2, 20, 8, (8, 24)),
        # the solver alone, for a host program with its own assembly
        _pcg("pcg_128", (128, 128, 128), 1e-12),
    ]


def _dims(rng, lo, hi):
    """A grid of lo..hi cells (log-uniform), its sides within a factor of
    about two of each other or stretched along the channel, odd ones too."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, ay = rng.uniform(1.0, 2.4), rng.uniform(0.7, 1.4)
    nz = (n / (ax * ay)) ** (1.0 / 3.0)
    return tuple(max(10, int(round(v))) for v in (ax * nz, ay * nz, nz))


def draw(rng: random.Random):
    kind = rng.choices(["channel", "adjoint", "lid", "pcg"], [6, 2, 2, 2])[0]
    if kind == "channel":
        dims = _dims(rng, 3500, 16e6)
        n = dims[0] * dims[1] * dims[2]
        steps = 20 if n < 2e5 else 10 if n < 4e6 else 3
        m = min(dims)
        conv = rng.choice([0, 0, 1, 2])
        return _channel(None, dims, steps, rng.randint(1, 4), (max(2, m // 8), max(3, m // 4)), mixed=rng.random() < 0.5,
                        conv=conv, ri=rng.choice([0.0, 1.0]) if conv == 2 else 0.0, stretched=rng.random() < 0.25,
                        re=rng.choice([100.0, 400.0, 1000.0]))
    if kind == "adjoint":
        dims = _dims(rng, 2e4, 4e6)
        m = min(dims)
        return _adjoint(None, dims, rng.randint(1, 4), (max(2, m // 8), max(3, m // 4)), mixed=rng.random() < 0.5)
    if kind == "lid":
        dims = _dims(rng, 2e4, 4e6)
        m = min(dims)
        return _lid(None, dims, 2, 10, rng.randint(1, 4), (max(2, m // 8), max(3, m // 4)))
    return _pcg(None, _dims(rng, 2e4, 4e6), 1e-12)


def _deck(case, seed):
    """The case's deck: a 2 x 1 x 1 domain with seeded, separate solid blocks."""
    dims = (case["nx"], case["ny"], case["nz"])
    boxes = decks.place_blocks(dims, case["blocks"], case["edge_lo"], case["edge_hi"], seed)
    ys = zs = None
    if case.get("stretched"):
        dx = 2.0 / dims[0]
        ys = decks.tanh_clustered(dims[1], 1.0, 20.0, dx)  # largest aspect ratio 20
        zs = decks.tanh_clustered(dims[2], 1.0, 20.0, dx)
    return decks.channel(*dims, boxes, ys=ys, zs=zs)


def _pinned(n):
    return torch.zeros(n, dtype=torch.float64, pin_memory=True)


def _make_channel(case, seed, **kw):
    deck = _deck(case, seed)
    c = hsolver_b200.Channel(deck, re=case["re"], precision=hsolver_b200.PREC_MIXED if case["mixed"] else
                             hsolver_b200.PREC_FP64, **kw)
    ctype, region = hsolver_b200.Case(deck).cell_types()
    rng = np.random.default_rng(seed)
    q = rng.uniform(0.5, 2.0, c.nblocks)
    c.set_solid(rng.uniform(10.0, 1000.0, c.nblocks), np.where(ctype == 1, q[np.maximum(region, 0)], 0.0))
    return c


# the C ABI's stand-alone solve, bound as a host program binds it
def _pcg_api():
    L = hsolver_b200.load()
    vp = ctypes.c_void_p
    L.hs_pcg_create.argtypes = [ctypes.c_int] * 4 + [ctypes.POINTER(vp)]
    L.hs_pcg_solve.argtypes = [vp] * 6 + [ctypes.c_double, ctypes.c_int, vp, ctypes.POINTER(ctypes.c_int),
                                          ctypes.POINTER(ctypes.c_double)]
    L.hs_pcg_destroy.argtypes = [vp]
    return L


class _Pcg:
    """hs_pcg with its device system: constant coefficients per axis on the
    unknowns (a box without one solid block), a random right-hand side."""

    def __init__(self, case, seed):
        self.L = _pcg_api()
        self.h = ctypes.c_void_p()
        self.coef, self.b = _pcg_system(case, seed)
        if self.L.hs_pcg_create(case["nx"], case["ny"], case["nz"], 0, ctypes.byref(self.h)) != 0:
            raise RuntimeError(self.L.hs_last_error(None).decode())
        self.x = torch.empty_like(self.b)
        self.tol = case["tol"]

    def solve(self):
        it, rel = ctypes.c_int(), ctypes.c_double()
        rc = self.L.hs_pcg_solve(self.h, *[t.data_ptr() for t in self.coef], self.b.data_ptr(), self.x.data_ptr(),
                                 self.tol, 20000, None, ctypes.byref(it), ctypes.byref(rel))
        if rc != 0:
            raise RuntimeError(self.L.hs_last_error(None).decode())
        return self.x

    def __del__(self):
        if self.h:
            self.L.hs_pcg_destroy(self.h)
            self.h = None


def _pcg_system(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["nz"] + 2, case["ny"] + 2, case["nx"] + 2)
    rng = random.Random(seed)
    unknown = torch.zeros(shape, dtype=torch.bool, device="cuda")
    unknown[1:-1, 1:-1, 1:-1] = True
    lo = [rng.randrange(1, max(2, s // 2)) for s in shape]
    hi = [a + max(1, s // 6) for a, s in zip(lo, shape)]
    unknown[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = False
    coef = [unknown.to(torch.float64) * rng.uniform(0.5, 2.0) for _ in range(3)]
    b = torch.randn(shape, generator=g, dtype=torch.float64, device="cuda") * unknown
    return coef, b


def prepare(case, seed):
    kind = case["kind"]
    if kind == "channel":
        extra = {"conv": case["conv"], "ri": case["ri"], "g_axis": 1} if case["conv"] or case["ri"] else {}
        c = _make_channel(case, seed, p_tol=case["p_tol"], t_tol=case["t_tol"], t_maxiter=case["t_maxiter"], **extra)
        out = {f: _pinned(c.field_size(f)) for f in ("u", "v", "w", "p", "T")}
        return {"kind": kind, "solver": c, "steps": case["steps"], "out": out}
    if kind == "adjoint":
        c = _make_channel(case, seed, **BENCH)
        c.init()
        c.step(5)  # the flow the gradient is taken on
        return {"kind": kind, "solver": c, "tol": case["tol"]}
    if kind == "lid":
        prm = hsolver_b200.default_params(u_lid=0.1 * random.Random(seed).uniform(0.8, 1.2))
        s = hsolver_b200.Solver(_deck(case, seed), prm)
        s.init()
        s.step(case["before"])  # past the first steps, whose energy sweeps are at their limit
        s.sync()
        out = {f: _pinned(s.field_size(f)) for f in ("ux", "uy", "uz", "p", "t")}
        return {"kind": kind, "solver": s, "steps": case["steps"], "out": out}
    return {"kind": kind, "solver": _Pcg(case, seed)}


def run(state):
    s = state["solver"]
    if state["kind"] == "channel":
        s.init()
        s.step(state["steps"])
    elif state["kind"] == "adjoint":
        J, dq, dk, _ = s.adjoint(tol=state["tol"], maxiter=2000)
        return {"J": J, "dJdq": dq, "dJdk": dk}
    elif state["kind"] == "lid":
        s.step(state["steps"])
    else:
        return s.solve()
    for name, t in state["out"].items():
        s.field(name, out=t.numpy())
    return state["out"]


def work(case):
    """Bytes and operations that a pass cannot do without: the state in and
    out of every step, and per Krylov iteration each vector and coefficient
    once per direction of the V-cycle (FP64 8 B, mixed 4 B a value; the
    coarse levels a seventh of the finest).  Iteration counts are those the
    tolerances take on these systems."""
    n = case["nx"] * case["ny"] * case["nz"]
    side = n ** (1.0 / 3.0)
    kind = case["kind"]
    if kind == "channel":
        w = 4.0 if case["mixed"] else 8.0
        mom = 33.0 + 6 * w                                      # u, v, w, p, mask; u* and d of three faces
        asm = 3 * w + 24.0 + 4 * w                              # d, u*; couplings, rhs
        pit = 7.0 if case["p_tol"] > 1e-6 else 11.0
        pcg = pit * (13 * w + 8.0 / 7.0 * 11 * w)               # CG vectors; x, rhs, three couplings down and up
        cor = 3 * w + 24.0 + w + 40.0                           # d, u*, p'; u, v, w, p
        tit = 1.0 if case["t_maxiter"] == 1 else 4.0
        en = 24.0 + 17.0 + 8 * w + tit * (2 * 8.0 / 7.0 * 17 * w + 30 * w) + 16.0
        per, flops = mom + asm + pcg + cor + en, 300.0 + pit * 130.0 + tit * 300.0
        fields = 2 * 40.0                                       # the start, and the fields read back
        return {"bytes": n * (case["steps"] * per + fields), "flops": n * case["steps"] * flops}
    if kind == "adjoint":
        w, it = (4.0 if case["mixed"] else 8.0), 2 * 30.0 * max(1.0, side / 80.0) ** 0.5
        return {"bytes": n * (it * (2 * 8.0 / 7.0 * 17 * w + 30 * 8.0) + 400.0), "flops": n * it * 300.0}
    if kind == "lid":
        it = 2.0 * side                                         # the unpreconditioned CG
        per = 3 * 49.0 + it * 98.0 + 97.0 + 2 * 41.0            # momentum, CG, correction, energy
        return {"bytes": n * case["steps"] * per, "flops": n * case["steps"] * (300.0 + it * 20.0)}
    it = 4.0 * side
    return {"bytes": n * it * 98.0, "flops": n * it * 20.0}


def exact(case, seed):
    """The stand-alone solve's system solved to round-off with plain torch in
    FP64.  The other kinds return the iterates of a nonlinear outer loop cut
    at the inner solves' tolerances, or gradients on such a flow: they have no
    value of their own."""
    if case["kind"] != "pcg":
        return None
    (cx, cy, cz), b = _pcg_system(case, seed)
    d = 2 * cx + 2 * cy + 2 * cz

    def apply(p):
        s = d * p
        for c, axis in ((cx, 2), (cy, 1), (cz, 0)):
            s -= c * (torch.roll(p, 1, axis) + torch.roll(p, -1, axis))
        return s

    x, r = torch.zeros_like(b), b.clone()
    p, rr, bb = r.clone(), (b * b).sum(), (b * b).sum()
    for it in range(4000):
        s = apply(p)
        alpha = rr / (s * p).sum()
        x += alpha * p
        r -= alpha * s
        new = (r * r).sum()
        p = r + (new / rr) * p
        rr = new
        if it % 50 == 49 and float(rr / bb) < 1e-28:
            break
    return x
