"""Fluid without a boundary link (periodic on every axis): a step is the bulk kernel alone, each launch beginning under
the one before it, so what it reads early must have been written before the call and the rest read after its wait."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cerebrosim_b200 import lbm  # noqa: E402
from oracle import lattice_ref as L  # noqa: E402
from oracle.step_ref import OracleSolver  # noqa: E402

DIMS = (64, 48, 40)
PHI = -np.ones(DIMS, np.float32)
BOX = dict(phi=PHI, origin=[0, 0, 0], dx=1.0, openings=(), periodic=(0, 1, 2))


def waves(coords):
    """Populations of a moving start: a wave per link, its own direction and phase."""
    rng = np.random.default_rng(5)
    k = 2 * np.pi * rng.integers(-2, 3, size=(lbm.Q, 3)) / np.array(DIMS)
    return (0.02 * np.asarray(lbm.W)[:, None] * np.sin(k @ np.asarray(coords, float).T
                                                     + rng.uniform(0, 2 * np.pi, (lbm.Q, 1)))).astype(np.float32)


def start(s, f):
    s.set_force([1e-5, -2e-5, 3e-5])
    s.set_drive([1.0, 0.5, -0.8, 0.3, 0.0], period=9, ramp=6)
    if isinstance(s.f[0], np.ndarray):
        s.f[0][:] = f
    else:
        with torch.cuda.stream(s.stream):
            s.f[0].copy_(torch.as_tensor(f))
    return s


class Stiffening(lbm.Solver):
    """A launch hook that changes the relaxation rates before every step, on the solver's stream."""

    def _launch(self, a):
        with torch.cuda.stream(self.stream):
            self.om.mul_(1.002)
        super()._launch(a)


@pytest.mark.parametrize("model", ["regularised", "trt"])
def test_rates_changed_between_calls(model):
    """The rates that a kernel of the same stream wrote right before a call are the ones its steps use: captured
    graphs and calls one after the other give the fields of steps that are waited for one by one, bit for bit."""
    lat = lbm.build_lattice(**BOX)
    f = waves(lat["coords"])
    runs = []
    for way in ("waited", "calls", "graph"):
        s = start(Stiffening(lat, 0.1, model=model), f)
        assert s.gmax == 0 and s.N == PHI.size
        if way == "waited":
            for _ in range(60):
                s._launch(s.cur)
                s.synchronize()
                s.cur = 1 - s.cur
        else:
            s.run(60, chunk=20 if way == "graph" else 200)
        runs.append(s.fields())
        assert s.om[0].item() == pytest.approx(1.002 ** 60 / s.tau, rel=1e-5)
    assert np.abs(runs[0][1]).max() > 1e-3
    for p, u in runs[1:]:
        assert np.array_equal(p, runs[0][0]) and np.array_equal(u, runs[0][1])


@pytest.mark.parametrize("model", ["regularised", "trt"])
def test_steps_of_one_call(model):
    """One call of many steps, each of them launched under the one before, gives the fields of steps that are waited
    for one by one, bit for bit; both agree with the oracle. Populations of up to 0.006 in magnitude: 61 steps of some
    thirty roundings, each 2^-24 of that, stay below 7e-7 (a drive one step late would move the velocity by 5e-6)."""
    lat = lbm.build_lattice(**BOX)
    f = waves(lat["coords"])
    one, singles = (start(lbm.Solver(lat, 0.1, model=model), f) for _ in range(2))
    one.run(61, chunk=200)
    graph = start(lbm.Solver(lat, 0.1, model=model), f)
    graph.run(61, chunk=20)
    for _ in range(61):
        singles.run(1)
        singles.synchronize()
    ref = start(OracleSolver(L.build_lattice(**BOX), 0.1, model=model), f)
    ref.run(61)
    p, u = one.fields()
    for s in (singles, graph):
        assert np.array_equal(p, s.fields()[0]) and np.array_equal(u, s.fields()[1])
        assert s.tick_value() == 61 and s.drv.item() == one.drv.item()
    pr, ur = ref.fields()
    assert np.abs(ur).max() > 1e-3
    assert np.abs(p - pr).max() <= 7e-7 and np.abs(u - ur).max() <= 7e-7
