"""The step's paths beside its arithmetic, at the sizes where each can go wrong: the drive evaluated a step ahead, the
flux sums over few and many blocks, population rows with and without padding, and an empty lattice's clock."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cerebrosim_b200 import batch, cases, lbm, simulate  # noqa: E402


def pipe(name="open_pipe_R8_L40"):
    return lbm.build_lattice(**cases.lattice_args(cases.case(name)))


def drive(coef, period, ramp, t):
    ph = 2 * np.pi * (t % period) / period
    k = np.arange(1, (len(coef) + 1) // 2)
    v = coef[0] + (coef[1::2] * np.cos(k * ph) + coef[2::2] * np.sin(k * ph)).sum()
    return v * (0.5 - 0.5 * np.cos(np.pi * t / ramp)) if t < ramp else v


@pytest.mark.parametrize("harmonics", [0, 1, 16, 17, 33])
def test_drive_of_every_step(harmonics):
    """The drive stored by each step, over steps taken one by one, in one call and across a change of the drive, against
    64 bits: float32 angles of up to 33 periods and a sum of 67 rounded terms stay within 33 * (2 pi * 33 * 2^-24) +
    67 * 2^-24 < 5e-4 of terms below 1, here 1e-3."""
    rng = np.random.default_rng(harmonics)
    s = lbm.Solver(pipe(), 0.02, model="regularised")
    t = 0
    for coef, period, ramp in ((rng.uniform(-1, 1, 2 * harmonics + 1), 7, 5), (rng.uniform(-1, 1, 2 * harmonics + 1), 40, 0)):
        coef = 1e-3 * coef
        s.set_drive(coef, period=period, ramp=ramp)
        for steps in (1, 1, 2, 5, 8):
            s.run(steps, chunk=4)
            t += steps
            assert s.tick_value() == t
            assert abs(s.drv.item() - drive(coef, period, ramp, t - 1)) < 5e-7


@pytest.mark.parametrize("block", [32, 128, 256])
@pytest.mark.parametrize("share", [0.0, 0.001, 1.0])
def test_flux_sums(block, share):
    """Flux over no cell, a few and every cell (77 k nodes in blocks of 32 are more rows than k_bc holds in flight)
    equals the FP64 sum over the velocity field up to the rounding of 1e5 additions."""
    lat = pipe("open_pipe_R16_L96")
    n = lbm.n_nodes(lat)
    rng = np.random.default_rng(3)
    idx = np.flatnonzero(rng.uniform(size=n) < share)
    flux = {"idx": idx, "w": rng.uniform(-1, 1, size=(len(idx), 3)).astype(np.float32), "slot": rng.integers(0, 1, len(idx))}
    s = simulate.ArterySolver(lat, 0.02, flux, [0.0], 0.0, 0.1, model="regularised", block=block)
    s.set_drive([0.02])
    s.run(7)
    u = s.fields()[1].astype(np.float64)
    terms = (u[idx] * flux["w"]).sum(1)
    assert abs(s.Qlast.numpy()[0] - terms.sum()) <= 1e5 * 2.0 ** -53 * np.abs(terms).sum()
    assert s.p_out64[0].item() == s.drv.item()


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("kw", [{"model": "regularised"}, {"model": "trt"}, {"model": "regularised", "block": 256}])
def test_padded_rows(storage, kw):
    """Rows that start on 128-byte lines and rows back to back give the same fields bit for bit."""
    lat = pipe("open_pipe_R7_L33")
    out = []
    for padded in (True, False):
        s = lbm.Solver(lat, 0.02, storage=storage, **kw)
        assert s.f[0].stride(0) * s.f[0].element_size() % 128 == 0 and s.vel[0].stride(0) % 32 == 0
        if not padded:
            s.f = [f.contiguous() for f in s.f]
            s.vel = [v.contiguous() for v in s.vel]
            assert s.f[0].stride(0) == s.npad and s.vel[0].stride(0) == s.N
        s.set_sponge(5, 0.6)
        s.set_drive([0.03, 0.01, 0.0], period=50, ramp=10)
        s.set_outlet_pressure([0.001])
        s.run(60, chunk=20)
        out.append(s.fields())
    assert np.abs(out[0][1]).max() > 0
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_empty_lattice_keeps_time():
    """A lattice without fluid advances its clock and drive, alone and beside another in a batch."""
    empty = lbm.build_lattice(np.ones((4, 4, 4), np.float32), [0, 0, 0], 1.0)
    s = lbm.Solver(empty, 0.02, model="regularised", block=128)
    s.set_drive([1.0, 0.5, 0.0], period=8)
    s.run(3, chunk=2)
    assert s.tick_value() == 3 and s.drv.item() == pytest.approx(drive(np.array([1.0, 0.5, 0.0]), 8, 0, 2), abs=1e-6)
    other = lbm.Solver(pipe(), 0.02, model="regularised", block=128)
    b = batch.BatchSolver([s, other])
    b.run(5, chunk=2)
    b.synchronize()
    assert s.tick_value() == 8 and other.tick_value() == 5
    assert s.drv.item() == pytest.approx(drive(np.array([1.0, 0.5, 0.0]), 8, 0, 7), abs=1e-6)


@pytest.mark.parametrize("sizes", [(0, 1, 31), (1023, 1024, 1025), (4095, 4097, 9000)])
def test_probe_sizes(sizes):
    """Probes without a cell, below and above a thread's and a block's share, against the fields: the sums in another
    order of FP64, the largest speed to a float32 square root of three products (4 ulp)."""
    lat = pipe("open_pipe_R16_L96")
    s = lbm.Solver(lat, 0.02, model="regularised", order="boundary-first")
    s.set_drive([0.03])
    s.run(20)
    rng = np.random.default_rng(1)
    idx = [rng.integers(0, s.N, size=n) for n in sizes]
    probes = simulate.Probes(s, np.concatenate(idx), np.repeat(np.arange(len(sizes)), sizes), len(sizes))
    p, umax = probes.sample()
    rho, u = s.rho[s.inv].double().cpu().numpy(), s.fields()[1].astype(np.float64)
    for k, c in enumerate(idx):
        if len(c):
            assert p[k] == pytest.approx(rho[c].mean() / 3, rel=0, abs=1e-12)
        else:
            assert np.isnan(p[k])
    assert umax == pytest.approx(np.linalg.norm(u[np.concatenate(idx)], axis=1).max(), rel=4 * 2.0 ** -23)


@pytest.mark.parametrize("block", [32, 128, 256])
@pytest.mark.parametrize("ends", [2, 8])
def test_flux_of_several_ends(ends, block):
    """Every open end's flow and relaxed pressure, with 1 cell in 3 and 1 in 5 measured by an end of its own choice (in
    blocks of 32 more rows than k_bc holds in flight): the FP64 sum over the velocity field up to the rounding of 1e5
    additions, and p' = p + alpha (R Q - pref - p) from it up to a few roundings."""
    lat = pipe("open_pipe_R16_L96")
    lat = dict(lat, n_outlets=max(ends, lat["n_outlets"]))
    n = lbm.n_nodes(lat)
    rng = np.random.default_rng(ends)
    idx = np.concatenate([np.arange(0, n, 3), np.arange(1, n, 5)])
    flux = {"idx": idx, "w": rng.uniform(-1, 1, size=(len(idx), 3)).astype(np.float32), "slot": rng.integers(0, ends, len(idx))}
    R = np.concatenate([[0.0], rng.uniform(0.1, 1.0, ends - 1)]).astype(np.float32)
    s = simulate.ArterySolver(lat, 0.02, flux, R, 0.001, 0.1, model="regularised", block=block)
    s.set_drive([0.02])
    s.run(6)
    before = s.p_out64.cpu().numpy()[:ends]
    s.run(1)
    u = s.fields()[1].astype(np.float64)
    terms = (u[idx] * flux["w"]).sum(1)
    q, after = s.Qlast.numpy(), s.p_out64.cpu().numpy()[:ends]
    assert after[0] == s.drv.item()
    for k in range(ends):
        t = terms[flux["slot"] == k]
        assert abs(q[k] - t.sum()) <= 1e5 * 2.0 ** -53 * np.abs(t).sum()
        if k:
            want = before[k] + 0.1 * (float(R[k]) * q[k] - 0.001 - before[k])
            assert abs(after[k] - want) <= 1e-14 and after[k] != before[k]


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_pulls_past_the_l2(storage):
    """The pulls that go out of the caches first (both buffers within the L2) and the others give the same fields bit for
    bit: rows so far apart that the same lattice counts as larger than the L2 choose the others."""
    lat = pipe("open_pipe_R7_L33")
    out = []
    for stride in (None, 3 << 20):
        s = lbm.Solver(lat, 0.02, model="regularised", storage=storage)
        l2 = torch.cuda.get_device_properties(s.dev).L2_cache_size
        if stride:
            with torch.cuda.stream(s.stream):
                s.f = [torch.zeros((lbm.Q, stride), dtype=f.dtype, device=s.dev)[:, :s.npad] for f in s.f]
        assert (2 * lbm.Q * s.f[0].stride(0) * s.f[0].element_size() > l2) == bool(stride)
        s.set_drive([0.03, 0.01, 0.0], period=50, ramp=10)
        s.set_outlet_pressure([0.001])
        s.run(60, chunk=20)
        out.append(s.fields())
    assert np.abs(out[0][1]).max() > 0
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("persistent", [True, False])
@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_batch_rows(storage, persistent):
    """A batch of members with padded rows and rows back to back, of even and odd parity, gives each member's own run."""
    lats = [pipe("open_pipe_R7_L33"), pipe()]

    def members():
        out = [lbm.Solver(lat, 0.02, model="regularised", storage=storage) for lat in lats]
        for k, s in enumerate(out):
            s.set_drive([0.02 + 0.01 * k, 0.01, 0.0], period=30, ramp=5)
            s.run(3 + k)
        return out
    alone, together = members(), members()
    for s in alone:
        s.run(25, chunk=10)
    with torch.cuda.stream(together[1].stream):
        together[1].f, together[1].vel = ([t.contiguous() for t in ts] for ts in (together[1].f, together[1].vel))
    b = batch.BatchSolver(together, persistent=persistent)
    b.run(25, chunk=10)
    b.synchronize()
    for a, t in zip(alone, together):
        assert all(np.array_equal(x, y) for x, y in zip(a.fields(), t.fields())) and a.fields()[1].any()
