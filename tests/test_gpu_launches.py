"""What a call of the step enqueues: the kernels of its steps and no more."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cerebrosim_b200 import _lib, batch, cases, lbm, simulate  # noqa: E402


def kernels(s, enqueue):
    """Nodes of the graph that `enqueue(stream)` leaves on the stream of solver s."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    st = s.stream.cuda_stream
    s.synchronize()
    err, = rt.cudaStreamBeginCapture(st, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)
    assert int(err) == 0
    rc = enqueue(ctypes.c_void_p(st))
    err, g = rt.cudaStreamEndCapture(st)
    assert rc == 0 and int(err) == 0
    n = rt.cudaGraphGetNodes(g)[-1]
    rt.cudaGraphDestroy(g)
    return n


@pytest.mark.parametrize("steps", [1, 3])
def test_launches_of_a_call(steps):
    lib = _lib.load()
    lat = lbm.build_lattice(**cases.lattice_args(cases.case("open_pipe_R8_L40")))
    box = lbm.build_lattice(-np.ones((16, 12, 8), np.float32), [0, 0, 0], 1.0, periodic=(0, 1, 2))
    plain, periodic = lbm.Solver(lat, 0.02), lbm.Solver(box, 0.02)
    idx = np.arange(50)
    flux = {"idx": idx, "w": np.ones((50, 3), np.float32), "slot": np.zeros(50, np.int64)}
    coupled = simulate.ArterySolver(lat, 0.02, flux, [0.0], 0.0, 0.1)

    def step(s):
        d, x = s._desc(), s._layout()
        return kernels(s, lambda st: lib.cs_step_ex(ctypes.byref(d), ctypes.byref(x), s.cur, steps, st))
    assert step(plain) == 2 * steps            # boundary links, nodes
    assert step(coupled) == 3 * steps          # and the resistances
    assert step(periodic) == 1 + steps         # no boundary kernel that could evaluate the first drive
    b = batch.BatchSolver([plain, lbm.Solver(lat, 0.02)])
    b._refresh()
    assert kernels(b, lambda st: lib.cs_batch_step_ex(ctypes.byref(b.desc), b._layouts, b.cur, steps, st)) == 2 * steps
