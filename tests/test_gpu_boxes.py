"""The FP32 tiled mover when its particles have left their bricks: boxes cut
to shared memory with particles outside them (2D and 3D, exact charge), and
the reorders pic_step adds before that happens."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = 0.45


def _hot(nx, ny, nz, dims, ppc, seed, spread=0.6):
    from pictor_b200 import Particles

    rng = np.random.Generator(np.random.Philox(key=seed))
    n = ppc * nx * ny * nz
    p = Particles.empty(2 * n)
    for k, m in (("x", nx), ("y", ny), ("z", nz)):
        a = rng.random(n) * m + (3.0 if k != "z" or dims == 3 else 1.0)
        getattr(p, k)[:] = np.concatenate([a, a])
    for k in "uvw":
        getattr(p, k)[:] = rng.normal(scale=spread, size=2 * n)
    p.q[:n], p.q[n:] = 1.0, -1.0
    p.flv[:n], p.flv[n:] = 1, 2
    return p


def _cfg(shape, dims, ppc, period, precision="fp32", **kw):
    from pictor_b200 import PicConfig, init_scale

    sc = init_scale(C, 2.0, ppc)
    n = 2 * ppc * shape[0] * shape[1] * shape[2]
    return PicConfig(nx=shape[0], ny=shape[1], nz=shape[2], dims=dims, c=C, qi=sc["qi"], precision=precision,
                     capacity=int(n * (1.1 if precision == "fp32" else 3)) + 4096, reorder_period=period, **kw), sc


@pytest.mark.parametrize("shape,dims,ppc,steps,kw", [
    ((41, 24, 23), 3, 8, 16, {}),                  # about half the particles outside the cut boxes
    ((24, 24, 24), 3, 2, 9, {"exact_charge": 1}),
    ((24, 41, 13), 3, 1, 3, {"brick": (8, 8, 8)}),
    ((96, 75, 1), 2, 8, 60, {"brick": (8, 8, 1)}),
])
def test_outgrown_boxes_move_like_the_per_particle_form(shape, dims, ppc, steps, kw):
    """After `steps` moves without a reorder the boxes have outgrown shared
    memory.  One more move, tiled, against the per-particle form from the same
    slots and fields: particles bit for bit, the current (through E) to the
    FP32 rounding of its sums (64 contributions of a cell, 2^-24 each, within
    1e-5 of the largest)."""
    from pictor_b200 import Simulation

    cfg, _ = _cfg(shape, dims, ppc, 0, **kw)
    with Simulation(cfg) as a, Simulation(cfg) as b:
        a.load_particles(_hot(*shape, dims, ppc, 5))
        a.reorder()
        a.step(steps)
        b.load_particles(a.fetch_particles())
        b.load_fields(a.fetch_fields())
        a.step(1)
        b.step(1)
        pa, pb = a.fetch_particles(), b.fetch_particles()
        for k in ("x", "y", "u", "v", "w", "q", "flv") + (("z",) if dims == 3 else ()):
            assert np.array_equal(getattr(pa, k), getattr(pb, k)), k
        fa, fb = a.fetch_fields(), b.fetch_fields()
        for k in ("Ex", "Ey", "Ez"):
            ea, eb = getattr(fa, k), getattr(fb, k)
            assert np.abs(ea - eb).max() <= 1e-5 * np.abs(eb).max(), k
        assert a.device_errors() == 0


def test_pic_step_reorders_before_the_boxes_are_outgrown():
    """A hot run is reordered more often than the period, also across calls;
    a cold one is not; the hot run's energies stay the FP64 run's (FP32
    rounding of 40 steps: 1e-4)."""
    from pictor_b200 import Simulation

    shape, ppc = (48, 32, 32), 8

    def run(precision, spread):
        cfg, sc = _cfg(shape, 3, ppc, 20, precision)
        with Simulation(cfg) as s:
            s.load_particles(_hot(*shape, 3, ppc, 7, spread))
            s.reorder()
            s.profile(True)
            s.phase_times()
            for n in (20, 1, 1, 11, 7):
                s.step(n)
            t = s.phase_times()
            d = s.diagnostics(sc["masse"])
        return t["launches"]["reorder"], d

    hot, d32 = run("fp32", 0.6)
    cold, _ = run("fp32", 0.01)
    per = cold // 2
    assert cold == 2 * per and hot >= 4 * per
    _, d64 = run("fp64", 0.6)
    for k in ("B2", "E2"):
        assert abs(d32[k] - d64[k]) <= 1e-4 * d64[k]
    assert np.allclose(d32["kinetic"], d64["kinetic"], rtol=1e-4)


@pytest.mark.parametrize("how", ["load_particles", "init_weibel"])
def test_a_reloaded_run_reorders_as_a_new_one(how):
    """The interval learned from a hot plasma is not applied to the cold one
    loaded after it: the same number of reorders as in a run of its own."""
    from pictor_b200 import Simulation

    shape, ppc = (48, 32, 32), 8
    cfg, sc = _cfg(shape, 3, ppc, 20)

    def load_cold(s):
        if how == "init_weibel":
            s.init_weibel(ppc, 0.5, 0.0, 1e-6, 1e-6)
        else:
            s.load_particles(_hot(*shape, 3, ppc, 8, 0.01))
        s.set_step(0)
        s.reorder()
        s.phase_times()
        s.step(45)
        return s.phase_times()["launches"]["reorder"]

    with Simulation(cfg) as a, Simulation(cfg) as b:
        for s in (a, b):
            s.profile(True)
        a.load_particles(_hot(*shape, 3, ppc, 7))
        a.reorder()
        a.step(30)      # learns a short interval, and leaves a report unread
        a.reorder()
        assert load_cold(a) == load_cold(b)


@pytest.mark.parametrize("form", [{"per_phase": True}, {"persistent": True}])
def test_batched_steps_leave_the_learned_interval_alone(form):
    """A warm run stepped by pic_step, then for two periods and a half by the
    batched or persistent form, then by pic_step again, reorders in the last
    part as often as a run that pic_step stepped throughout (one more or less:
    the phase in which it starts)."""
    from pictor_b200 import Simulation, step_many

    shape, ppc = (48, 32, 32), 8
    cfg, _ = _cfg(shape, 3, ppc, 20)
    counts = []
    with Simulation(cfg) as a, Simulation(cfg) as b:
        for s, batched in ((a, False), (b, True)):
            s.load_particles(_hot(*shape, 3, ppc, 7, 0.15))
            s.reorder()
            s.step(25)
            if batched:
                step_many([s], 50, **form)
            else:
                s.step(50)
            s.profile(True)
            s.phase_times()
            s.step(60)
            counts.append(s.phase_times()["launches"]["reorder"])
            s.profile(False)
    per = 6   # launches of a reorder
    assert abs(counts[0] - counts[1]) <= per, counts
    assert min(counts) >= 3 * per


def test_reorders_captured_from_the_handle_stream():
    """Two reorders captured by the caller from the handle's stream and
    replayed: the steps after them do not wait for what was only captured."""
    import torch

    from pictor_b200 import Simulation

    shape = (24, 24, 24)
    cfg, _ = _cfg(shape, 3, 2, 20)
    with Simulation(cfg) as s:
        s.load_particles(_hot(*shape, 3, 2, 9))
        s.reorder()
        s.step(1)
        n = s.particle_count()
        s.set_sync(False)
        stream = torch.cuda.ExternalStream(s.stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            s.reorder()
            s.reorder()
        with torch.cuda.stream(stream):
            graph.replay()
        s.set_sync(True)
        s.step(25)
        assert s.device_errors() == 0
        assert s.particle_count() == n
