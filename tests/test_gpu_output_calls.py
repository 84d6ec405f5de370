"""What an output call returns, over the routes it can take: the charge density
by bricks (after a reorder, boxes kept, cut or outgrown) against the particles
in any order, the kinetic energy of more flavours than the two kept in
registers, and the fields of small grids (one conversion, one or more copies)
and of grids past the staging buffer."""
import numpy as np
import pytest

from pictor_b200.simulation import Fields

from .test_gpu_boxes import _cfg, _hot

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,dims,ppc,steps", [((24, 20, 17), 3, 6, 0), ((41, 24, 23), 3, 6, 14),
                                                  ((96, 75, 1), 2, 6, 25), ((5, 5, 5), 3, 1, 2)])
def test_density_by_bricks(shape, dims, ppc, steps):
    """The diagnostics of a reordered run and of the same slots loaded into
    one that was not: the density scale and the Gauss residual to the rounding
    of the sums (1e-12 of the largest density), the energies to 1e-12."""
    from pictor_b200 import Simulation

    cfg, sc = _cfg(shape, dims, ppc, 0)
    with Simulation(cfg) as a, Simulation(cfg) as b:
        p = _hot(*shape, dims, ppc, 21)
        p.q *= np.random.default_rng(2).uniform(0.2, 3.0, size=len(p))
        a.load_particles(p)
        a.reorder()
        a.step(steps)
        b.load_particles(a.fetch_particles())
        b.load_fields(a.fetch_fields())
        da, db = a.diagnostics(sc["masse"]), b.diagnostics(sc["masse"])
    assert db["rho_max"] > 0
    for k in ("rho_max", "gauss_linf"):
        assert abs(da[k] - db[k]) <= 1e-12 * db["rho_max"], k
    for k in ("B2", "E2"):
        assert abs(da[k] - db[k]) <= 1e-12 * max(db[k], 1e-300)
    assert np.allclose(da["kinetic"], db["kinetic"], rtol=1e-12)


@pytest.mark.parametrize("shape,dims,ppc,steps,brick", [((24, 20, 17), 3, 6, 0, (3, 3, 3)),
                                                        ((41, 24, 23), 3, 6, 14, (4, 4, 4)),
                                                        ((96, 75, 1), 2, 6, 25, (4, 4, 1)),
                                                        ((96, 75, 1), 2, 40, 1, (4, 4, 1)),
                                                        ((333, 5, 5), 3, 2, 3, (1, 5, 5))])
def test_density_of_many_bricks(shape, dims, ppc, steps, brick):
    """As test_density_by_bricks with at least the two bricks per SM from which
    the density is summed brick by brick."""
    from pictor_b200 import Simulation

    cfg, sc = _cfg(shape, dims, ppc, 0, brick=brick)
    assert np.prod([-(-n // b) for n, b in zip(shape, brick)]) >= 2 * 148
    with Simulation(cfg) as a, Simulation(cfg) as b:
        p = _hot(*shape, dims, ppc, 21)
        p.q *= np.random.default_rng(2).uniform(0.2, 3.0, size=len(p))
        a.load_particles(p)
        a.reorder()
        a.step(steps)
        b.load_particles(a.fetch_particles())
        b.load_fields(a.fetch_fields())
        da, db = a.diagnostics(sc["masse"]), b.diagnostics(sc["masse"])
    assert db["rho_max"] > 0
    for k in ("rho_max", "gauss_linf"):
        assert abs(da[k] - db[k]) <= 1e-12 * db["rho_max"], k


@pytest.mark.parametrize("qi", [0.01, -0.01])
def test_density_by_bricks_keeps_light_particles(qi):
    """Eight particles 2^-47 as heavy as the others, on nodes of their own, in
    a brick of 16384 (the other 319 bricks are empty), with either sign of the
    charge unit.  The others lie in pairs of opposite charge at quarters of a
    cell, so their sums are exact and cancel: the Gauss residual is the density
    of the heaviest light one, the same reordered and not (one product per
    node), and FP32's positions give it to 1e-6."""
    from pictor_b200 import PicConfig, Simulation

    n, light = 32, 2.0 ** -47
    cfg = PicConfig(nx=32 * n, ny=10 * n, dims=2, c=0.45, qi=qi, precision="fp32", capacity=1 << 15, brick=(n, n, 1))
    p = _hot(n, n, 1, 2, 8, 4)
    m = len(p)
    rng = np.random.default_rng(4)
    p.x[:], p.y[:] = 3.0 + rng.integers(0, 4 * n, m) / 4, 3.0 + rng.integers(0, 2 * n, m) / 4
    for k in ("x", "y"):
        getattr(p, k)[9::2] = getattr(p, k)[8:-1:2]
    p.q[8::2], p.q[9::2] = 1.0, -1.0
    p.x[:8], p.y[:8] = 3.3 + np.arange(8) * 4, 3.7 + 0.75 * n
    p.q[:8] = light * np.arange(3, 11)
    p.u[:], p.v[:], p.w[:] = 0.0, 0.0, 0.0
    with Simulation(cfg) as a, Simulation(cfg) as b:
        for s in (a, b):
            s.load_particles(p)
        a.reorder()
        da, db = a.diagnostics(1.0), b.diagnostics(1.0)
    assert da["rho_max"] == pytest.approx(db["rho_max"], rel=1e-12) and db["rho_max"] > 0
    assert da["gauss_linf"] == pytest.approx(db["gauss_linf"], rel=1e-12)
    assert db["gauss_linf"] == pytest.approx(10 * light * abs(qi) * 0.7 * 0.7, rel=1e-6)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_kinetic_energy_of_every_flavour(precision):
    from pictor_b200 import PicConfig, Simulation

    qm = tuple([1.0, -1.0, 0.5, -1.0, 0.25] + [1.0] * 10)
    cfg = PicConfig(nx=12, ny=10, dims=2, c=0.45, qi=0.01, qm=qm, precision=precision, capacity=1 << 14)
    p = _hot(12, 10, 1, 2, 20, 3, 0.3)
    n = len(p)
    p.flv[:] = 1 + np.arange(n) % 15
    p.q[:] = np.where(np.isin(p.flv, (2, 4)), -1.0, 1.0)
    with Simulation(cfg) as s:
        s.load_particles(p)
        got = s.diagnostics(0.02)["kinetic"]
        f = s.fetch_particles()
    gm = np.sqrt(1 + f.u ** 2 + f.v ** 2 + f.w ** 2) - 1
    m = np.where(f.q > 0, f.q * 0.01 / np.array((0.0,) + qm)[f.flv], 0.02) * 0.45 ** 2
    want = np.array([(gm * m)[f.flv == k].sum() for k in range(1, 16)])
    assert np.allclose(got, want, rtol=1e-12)


@pytest.mark.parametrize("nx,ny", [(5, 5), (64, 33), (900, 700)])
@pytest.mark.parametrize("layout", ["separate", "contiguous", "gaps"])
def test_fetched_fields(nx, ny, layout):
    """Loaded fields come back (as FP32 keeps them) into arrays of their own,
    into one block, and into rows with gaps; with and without the current.
    The small grids' arrays fit the staging buffer together, the last one's
    do not."""
    from pictor_b200 import PicConfig, Simulation

    cfg = PicConfig(nx=nx, ny=ny, dims=2, c=0.45, qi=0.01, precision="fp32", capacity=4096)
    n = int(np.prod(cfg.shape))
    rng = np.random.default_rng(nx)
    f = Fields(*(np.asfortranarray(rng.normal(size=cfg.shape)) for _ in range(9)))
    with Simulation(cfg) as s:
        s.load_fields(f)
        s.load_current(f.Jx, f.Jy, f.Jz)
        for with_j in (True, False):
            row = n if layout == "contiguous" else n + 3
            buf = np.full((9, row), 7.0)
            out = None if layout == "separate" else Fields(*(buf[k, :n].reshape(cfg.shape, order="F") for k in range(9)))
            got = s.fetch_fields(with_j, out=out)
            for k in ("Ex", "Ey", "Ez", "Bx", "By", "Bz") + (("Jx", "Jy", "Jz") if with_j else ()):
                assert np.array_equal(getattr(got, k), getattr(f, k).astype(np.float32).astype(np.float64)), k
            if layout == "gaps":
                assert (buf[:, n:] == 7.0).all()
            if not with_j and out is not None:
                assert (buf[6:] == 7.0).all()


@pytest.mark.parametrize("registered", [[(0, 4)], [(3, 6)], [(5, 9)], [(0, 9)], [], [(0, 3), (3, 7)], [(1, 2), (2, 9)]])
def test_fetched_fields_into_partly_registered_memory(registered):
    """Nine host arrays one after the other, of which some lie in one or two
    ranges registered with CUDA (page-aligned: 64 x 64 float64 is 8 pages)."""
    import mmap

    import torch

    from pictor_b200 import PicConfig, Simulation

    cfg = PicConfig(nx=59, ny=59, dims=2, c=0.45, qi=0.01, precision="fp32", capacity=4096)
    n = 64 * 64
    rng = np.random.default_rng(4)
    f = Fields(*(np.asfortranarray(rng.normal(size=cfg.shape)) for _ in range(9)))
    buf = np.frombuffer(mmap.mmap(-1, 9 * n * 8), dtype=np.float64).reshape(9, n)
    buf[:] = 7.0
    out = Fields(*(buf[k].reshape(cfg.shape, order="F") for k in range(9)))
    rt = torch.cuda.cudart()
    with Simulation(cfg) as s:
        s.load_fields(f)
        s.load_current(f.Jx, f.Jy, f.Jz)
        for first, last in registered:
            assert int(rt.cudaHostRegister(buf[first].ctypes.data, (last - first) * n * 8, 0)) == 0
        try:
            s.fetch_fields(out=out)
        finally:
            for first, _ in registered:
                rt.cudaHostUnregister(buf[first].ctypes.data)
    for k in Fields.__dataclass_fields__:
        assert np.array_equal(getattr(out, k), getattr(f, k).astype(np.float32).astype(np.float64)), k
