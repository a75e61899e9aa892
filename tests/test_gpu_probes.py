"""Probes beside the heartbeat loop's own solver."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cerebrosim_b200 import cases, lbm, simulate  # noqa: E402


def test_probes_of_another_solver():
    """A sample is what its own solver's stream has computed, however far that is behind the solver that the loop
    advances."""
    far = lbm.Solver(lbm.build_lattice(**cases.lattice_args(cases.case("open_pipe_R16_L96"))), 0.02)
    near = lbm.Solver(lbm.build_lattice(**cases.lattice_args(cases.case("open_pipe_R8_L40"))), 0.02)
    for s in (far, near):
        s.set_drive([0.03])
        s.run(40)
    idx = np.arange(0, far.N, 7)
    probes = simulate.Probes(far, idx, idx % 3, 3)
    probes.sample()                              # the buffers hold an older sample
    with torch.cuda.stream(torch.cuda.Stream()):     # Solver.run orders itself with the caller's stream only
        far.run(4000)                            # some 30 ms of steps, not waited for
    series, _ = simulate.run_beats(near, 40, 2, 20, probes=probes, frames=0)
    far.synchronize()
    p, umax = probes.sample()
    assert len(series["p_probe"]) == 2 and np.array_equal(series["p_probe"], [p, p])
    assert (series["umax"] == umax).all() and umax > 0


def test_values_wait_for_their_read_back():
    s = lbm.Solver(lbm.build_lattice(**cases.lattice_args(cases.case("open_pipe_R16_L96"))), 0.02)
    s.set_drive([0.03])
    probes = simulate.Probes(s, np.arange(100), np.zeros(100, int), 1)
    s.run(4000)
    probes.enqueue()
    p, umax = probes.values()
    s.synchronize()
    again = probes.sample()
    assert np.array_equal(p, again[0]) and umax == again[1] > 0
