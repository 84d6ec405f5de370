"""Runs that nearly fill the device: arrays that only make a run faster are not
taken, or given back, when what the run needs would not fit beside them.  The
device is filled with a torch tensor that nothing touches."""
import contextlib

import numpy as np
import pytest

from .test_gpu_boxes import _cfg, _hot

pytestmark = pytest.mark.gpu

SLACK = 32 << 20   # allocation granularity, graphs


@contextlib.contextmanager
def _only(room):
    """`room` bytes of device memory free."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - int(room), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del fill
        torch.cuda.empty_cache()


def _used(run):
    """What run() returned and the device memory it held at its end."""
    import torch

    run()   # kernels loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    held = []
    out = run(lambda: held.append(before - torch.cuda.mem_get_info()[0]))
    return out, held[0]


def _particles(kind, shape, n):
    p = _hot(*shape, 3, 1, 3, 0.3)
    for k in p.NAMES:
        setattr(p, k, getattr(p, k)[:n].copy())
    p.flv[:] = 1 + np.arange(n) % 2
    p.q[:] = np.where(p.flv == 1, 1.0, -1.0)
    if kind == "cylindrical":
        p.x[:] = 3.6 + (p.x - 3.0) * (shape[0] - 1) / shape[0]
        p.q[:] *= p.x - 3.0
    return p


@pytest.mark.parametrize("geom,precision,optional,filt", [
    ("cartesian", "fp64", 48, 0), ("cylindrical", "fp64", 48, 0), ("cartesian", "fp32", 24, 0),
    ("cylindrical", "fp32", 24, 0), ("cartesian", "fp32", 24 + 8, 1), ("cartesian", "fp64", 48 + 16, 2)])
def test_a_run_that_fits_without_the_optional_arrays(geom, precision, optional, filt):
    """Room for what a run needs with its outputs, and for part of its optional
    arrays (`optional` bytes a cell), the density arrays left short of 0.6 of
    their size once the optional ones are taken: every call succeeds and gives
    what the run gives with room to spare (particles bit for bit after the
    first move, fields to the rounding of the current's sums)."""
    from pictor_b200 import PicConfig, Simulation

    shape = (128, 8, 2048) if geom == "cylindrical" else (128, 128, 128)
    cells = int(np.prod([n + 5 for n in shape]))
    p = _particles(geom, shape, 200000)
    kw = dict(geom="cylindrical", rmin=-0.5, inc_axis=1) if geom == "cylindrical" else dict(curr_filter=filt)
    cfg = PicConfig(nx=shape[0], ny=shape[1], nz=shape[2], dims=3, c=0.45, qi=0.01, precision=precision,
                    capacity=300000, reorder_period=0, brick=(8, 8, 4), **kw)

    def run(at_end=lambda: None):
        with Simulation(cfg) as s:
            s.load_particles(p)
            s.reorder()
            s.step(1)
            first = s.fetch_particles()
            s.step(2)
            d = s.diagnostics(0.01)
            f = s.fetch_fields(False)
            at_end()
            return first, d, f

    (pa, da, fa), used = _used(run)
    need = used - optional * cells
    with _only(need + optional * cells - 0.6 * 16 * cells):
        pb, db, fb = run()
    with _only(need + SLACK):
        run()
    order = [np.lexsort((q.z, q.y, q.x)) for q in (pa, pb)]   # the FP32 reorder's slots are in any order
    for k in pa.NAMES:
        assert np.array_equal(getattr(pa, k)[order[0]], getattr(pb, k)[order[1]]), k
    tol = 1e-12 if precision == "fp64" else 1e-5
    for k in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
        a, b = getattr(fa, k), getattr(fb, k)
        assert np.abs(a - b).max() <= tol * max(np.abs(fa.Ex).max(), np.abs(a).max()), k
    assert np.allclose(da["kinetic"], db["kinetic"], rtol=1e-6)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_optional_arrays_are_given_back(precision):
    """A run created with room to spare has its optional arrays; when the room
    goes, a later call that allocates (the density of the diagnostics, the
    Gauss solve) takes their place, and the run steps on."""
    from pictor_b200 import Simulation

    shape = (128, 128, 128)
    cfg, sc = _cfg(shape, 3, 1, 0, precision)
    p = _particles("cartesian", shape, 200000)
    with Simulation(cfg) as a, Simulation(cfg) as b:
        for s in (a, b):
            s.load_particles(p)
            s.reorder()
            s.step(1)
        da = a.diagnostics(sc["masse"])
        ga = a.solve_gauss(1e-6)
        with _only(8 << 20):
            db = b.diagnostics(sc["masse"])
        with _only(8 << 20):
            try:
                b.solve_gauss(1e-6)
            except RuntimeError as e:   # 4 doubles a cell: more than what is left to give
                assert "OOM" in str(e)
        gb = b.solve_gauss(1e-6)
        for s in (a, b):
            s.step(3)
        pa, pb = a.fetch_particles(), b.fetch_particles()
    assert abs(da["rho_max"] - db["rho_max"]) <= 1e-12 * da["rho_max"]
    assert ga["iters"] == gb["iters"]
    order = [np.lexsort((q.z, q.y, q.x)) for q in (pa, pb)]
    tol = 1e-9 if precision == "fp64" else 1e-3
    assert np.abs(pa.x[order[0]] - pb.x[order[1]]).max() <= tol


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_optional_arrays_in_a_caller_s_graph_are_kept(precision):
    """The phases of a step captured by the caller and replayed after a call
    that found no room: the call fails instead of taking the arrays that the
    graph uses, and the replay is the step (particles bit for bit: the first
    move gathers from loaded fields)."""
    import torch

    from pictor_b200 import Simulation
    from pictor_b200._capi import PicError

    shape = (128, 128, 128)
    cfg, sc = _cfg(shape, 3, 1, 0, precision)
    p = _particles("cartesian", shape, 200000)
    rng = np.random.default_rng(5)

    def phases(s):
        s.update_b_half()
        s.move_deposit()
        s.exchange_particles()
        s.update_b_half()
        s.update_e()
        s.fold_current()
        s.add_current()
        s.reset_current()

    with Simulation(cfg) as a, Simulation(cfg) as b:
        f = a.fetch_fields(False)
        for k in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
            getattr(f, k)[...] = rng.normal(scale=0.01, size=cfg.shape)
        for s in (a, b):
            s.load_fields(f)
            s.load_particles(p)
            s.reorder()
        a.set_sync(False)
        stream = torch.cuda.ExternalStream(a.stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            phases(a)
        a.set_sync(True)
        with _only(8 << 20), pytest.raises(PicError, match="OOM"):
            a.diagnostics(sc["masse"])
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        phases(b)
        pa, pb = a.fetch_particles(), b.fetch_particles()
        assert a.device_errors() == 0
        assert a.diagnostics(sc["masse"])["rho_max"] > 0
    order = [np.lexsort((q.z, q.y, q.x)) for q in (pa, pb)]
    for k in pa.NAMES:
        assert np.array_equal(getattr(pa, k)[order[0]], getattr(pb, k)[order[1]]), k


def test_outgrown_boxes_are_reported_without_the_node_arrays():
    """A hot run with no room for the node arrays reorders as often as one that
    has them."""
    from pictor_b200 import Simulation

    shape, ppc = (160, 96, 96), 2
    cfg, _ = _cfg(shape, 3, ppc, 20)

    def run(at_end=lambda: None):
        with Simulation(cfg) as s:
            s.init_weibel(ppc, 0.5, 0.0, 0.2, 0.2)
            s.reorder()
            s.profile(True)
            s.phase_times()
            s.step(40)
            at_end()
            t = s.phase_times()["launches"]
            return t["reorder"], t["move"]

    (reorders, moves), used = _used(run)
    with _only(used - 24 * 165 * 101 * 101 + SLACK):
        got, moved = run()
    assert got == reorders
    assert moved == moves      # the counting launch stands where the node pass stood


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_an_adjoint_that_fits_without_the_half_step_tape(precision):
    """Room for the checkpoints and the tape of E and B, not for the tape of
    the B between the half steps: the reverse steps compute it again, and the
    gradient is that of a run with room for it (bit for bit: the same values
    from the same expressions; the particles' sums are of one particle per
    cell at most, in any order)."""
    from pictor_b200 import PicConfig
    from pictor_b200.adjoint import Adjoint

    n, K, size = 1024, 8, 8 if precision == "fp64" else 4
    cfg = PicConfig(nx=n, ny=n, dims=2, c=0.45, qi=0.01, precision=precision, capacity=20000)
    p = _hot(n, n, 1, 2, 1, 3, 0.2)
    for k in p.NAMES:
        setattr(p, k, getattr(p, k)[:20000].copy())
    p.flv[:] = 1 + np.arange(20000) % 2
    p.q[:] = np.where(p.flv == 1, 1.0, -1.0)

    def run(at_end=lambda: None):
        with Adjoint(cfg) as a:
            a.load_particles(p)
            obj = a.forward(2 * K, K)
            g = a.gradient(drift=0.0, temp=(0.0, 0.0))
            at_end()
            return obj, g

    (oa, ga), used = _used(run)
    with _only(used - 3 * K * n * n * size + SLACK):
        ob, gb = run()
    tol = 1e-12 if precision == "fp64" else 1e-4
    assert abs(oa - ob) <= tol * oa
    for k in ("u", "v", "w", "x", "y"):
        assert np.abs(ga[k] - gb[k]).max() <= tol * np.abs(ga[k]).max(), k
