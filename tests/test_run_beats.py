"""What the heartbeat loop asks of the solver and the probes it is given (on the host, with stand-ins)."""
import numpy as np
import torch

from cerebrosim_b200 import simulate


class Flow:
    """Another solver: its flows offer numpy(), its pressures are a tensor, and that is all."""

    def __init__(self):
        self.steps, self.n_open = 0, 2
        self.p_out = torch.zeros(3)
        self.Qlast = self

    def numpy(self):
        return np.array([0.5, 0.25]) * self.steps

    def run(self, steps, chunk=200):
        self.steps += steps
        self.p_out += steps

    def ok(self):
        return True


class Scaled(simulate.Probes):
    """Probes whose samples are a measurement of their own."""

    def __init__(self, s):
        self.s, self.taken = s, []

    def sample(self):
        self.taken.append(self.s.steps)
        return np.array([10.0 * self.s.steps]), 0.1 * self.s.steps


def check(series):
    assert series["step"].tolist() == [5, 10, 15, 20]
    assert np.array_equal(series["Q"], [[2.5, 1.25], [5, 2.5], [7.5, 3.75], [10, 5]])
    assert np.array_equal(series["p_open"], [[5, 5], [10, 10], [15, 15], [20, 20]])


def test_another_solver():
    check(simulate.run_beats(Flow(), 10, 2, 5, frames=0)[0])


def test_overridden_sample_is_used():
    s = Flow()
    probes = Scaled(s)
    series, _ = simulate.run_beats(s, 10, 2, 5, probes=probes, frames=0)
    check(series)
    assert probes.taken == [5, 10, 15, 20]
    assert series["p_probe"].ravel().tolist() == [50, 100, 150, 200] and np.allclose(series["umax"], [0.5, 1, 1.5, 2])


def test_sample_set_on_the_object_is_used():
    s = Flow()
    probes = simulate.Probes.__new__(simulate.Probes)
    probes.sample = lambda: (np.array([s.steps]), 0.0)
    series, _ = simulate.run_beats(s, 10, 1, 5, probes=probes, frames=0)
    assert series["p_probe"].ravel().tolist() == [5, 10]
