"""The step's C interface as callers of cs_step know it: the descriptor ends with beat_acc, and the entry points that take
it alone need nothing else. (The library's own binding passes a cs_step_layout beside it.)"""
import ctypes

import numpy as np
import pytest
import torch

from cerebrosim_b200 import _lib, batch, cases, lbm, simulate


def test_descriptor_keeps_its_size():
    assert _lib.load().cs_abi_sizeof(1) == 456 and _lib.StepDesc.beat_acc.offset == 448
    assert _lib.load().cs_abi_sizeof(4) == ctypes.sizeof(_lib.StepLayout) == 24


def plain_desc():
    """A descriptor of 100 nodes whose pointers are only looked at for being there."""
    d = _lib.StepDesc()
    d.n, d.npad, d.gmax, d.period, d.block, d.model, d.n_out, d.n_irr = 100, 130, 30, 1, 128, 1, 1, 1
    d.gblock = (ctypes.c_int32 * 28)(*[0] * 27, 0)
    for name in ("rho", "lcode", "segdelta", "irr", "gnode", "ginfo", "gq", "uin", "om", "p_out", "tick", "drive", "coef"):
        setattr(d, name, 1 << 20)
    for k in range(2):
        d.f[k] = d.vel[k] = 1 << 20
    return d


def test_descriptor_alone_is_accepted():
    lib, d = _lib.load(), plain_desc()
    assert lib.cs_step_check(ctypes.byref(d)) == _lib.CS_OK, _lib.last_error()


@pytest.mark.parametrize("layout", [(0, 129, 0), (0, 0, 99), (0, 1 << 27, 0), (0, 0, 1 << 30)])
def test_layout_is_checked(layout):
    lib, d, x = _lib.load(), plain_desc(), _lib.StepLayout(*layout)
    assert lib.cs_step_ex(ctypes.byref(d), ctypes.byref(x), 0, 1, None) == _lib.CS_ERR_SIZE
    assert "row strides" in _lib.last_error()


def solvers():
    lat = lbm.build_lattice(**cases.lattice_args(cases.case("open_pipe_R8_L40")))
    box = lbm.build_lattice(-np.ones((16, 12, 8), np.float32), [0, 0, 0], 1.0, periodic=(0, 1, 2))
    empty = lbm.build_lattice(np.ones((4, 4, 4), np.float32), [0, 0, 0], 1.0)
    n = lbm.n_nodes(lat)
    flux = {"idx": np.arange(0, n, 3), "w": np.ones((len(range(0, n, 3)), 3), np.float32),
            "slot": np.zeros(len(range(0, n, 3)), np.int64)}
    out = [lbm.Solver(lat, 0.02, model="regularised"), lbm.Solver(box, 0.02, model="regularised"),
           simulate.ArterySolver(lat, 0.02, flux, [0.0], 0.0, 0.1, model="regularised"),
           lbm.Solver(empty, 0.02, model="regularised")]
    for s in out:
        s.set_drive([0.02, 0.01, -0.005], period=12, ramp=7)
        s.set_force([1e-6, 0, 0])
    return out


def back_to_back(s):
    with torch.cuda.stream(s.stream):
        s.f, s.vel = [f.contiguous() for f in s.f], [v.contiguous() for v in s.vel]
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("way", ["calls", "graph", "batch", "batch graph"])
def test_steps_of_a_descriptor_alone(way):
    """cs_step, cs_graph_capture and the batched pair on a descriptor alone, rows back to back, give what Solver.run
    gives, bit for bit: boundary links, none, resistances, no node."""
    lib = _lib.load()
    ref, own = solvers(), [back_to_back(s) for s in solvers()]
    for s in ref:
        s.run(24, chunk=200)
    st = [ctypes.c_void_p(s.stream.cuda_stream) for s in own]
    if way == "calls":
        for s, p in zip(own, st):
            for k in (1, 1, 2, 20):
                d = s._desc()
                _lib.check(lib.cs_step(ctypes.byref(d), s.cur, k, p))
                s.cur ^= k & 1
    elif way == "graph":
        for s, p in zip(own, st):
            d, g = s._desc(), ctypes.c_void_p()
            _lib.check(lib.cs_graph_capture(ctypes.byref(d), 0, 12, p, ctypes.byref(g)))
            for _ in range(2):
                _lib.check(lib.cs_graph_launch(g, p))
            s.synchronize()
            _lib.check(lib.cs_graph_destroy(g))
    else:
        b = batch.BatchSolver(own)
        b._refresh()
        b._sync_in()
        p = ctypes.c_void_p(b.stream.cuda_stream)
        if way == "batch":
            _lib.check(lib.cs_batch_step(ctypes.byref(b.desc), 0, 24, p))
        else:
            g = ctypes.c_void_p()
            _lib.check(lib.cs_batch_graph_capture(ctypes.byref(b.desc), 0, 12, p, ctypes.byref(g)))
            for _ in range(2):
                _lib.check(lib.cs_graph_launch(g, p))
        b.synchronize()
        if way != "batch":
            _lib.check(lib.cs_graph_destroy(g))
    for r, s in zip(ref, own):
        for a, c in zip(r.fields(), s.fields()):
            assert np.array_equal(a, c)
        assert s.drv.item() == r.drv.item() != 0 and s.tick_value() == r.tick_value() == 24
    assert np.array_equal(ref[2].Qlast.numpy(), own[2].Qlast.numpy()) and ref[2].Qlast.numpy()[0] != 0
    assert ref[0].fields()[1].any()
