"""The FP64 tiled mover away from the usual case: particles far outside their
tiles (boxes cut to shared memory, node values from the grid's array),
second segments queued, appended particles moved by the same launch, and the
exchange that looks only at the slots the mover marked."""
import numpy as np
import pytest

from .test_gpu_boxes import C, _hot

pytestmark = pytest.mark.gpu


def _sims(shape, dims, ppc, capacity):
    from pictor_b200 import PicConfig, Simulation, init_scale

    sc = init_scale(C, 2.0, ppc)
    mk = lambda tiles: Simulation(PicConfig(nx=shape[0], ny=shape[1], nz=shape[2], dims=dims, c=C, qi=sc["qi"],  # noqa: E731
                                            precision="fp64", capacity=capacity, reorder_period=0, fp64_tiles=tiles))
    return mk(1), mk(-1)


@pytest.mark.parametrize("shape,dims,ppc,steps,capacity", [
    ((40, 24, 20), 3, 4, 18, 1 << 19),     # boxes cut, most particles outside
    ((5, 5, 5), 3, 3, 4, 1 << 13),         # the smallest grid: one partial tile
    ((130, 7, 1), 2, 9, 12, 1 << 16),      # several tiles per row, every row crossing y
    ((33, 66, 1), 2, 1, 3, 6_000_000),     # counts of the exchange past the one-block scan
])
def test_tiled_steps_keep_the_slots_of_the_per_particle_form(shape, dims, ppc, steps, capacity):
    """Both forms from the same particles: the same holes and appended slots
    after every step (the exchange's order), positions and momenta to 1e-9
    (the current's sums differ in the last bits and the run amplifies them);
    then one step from the tiled form's state, bit for bit."""
    a, b = _sims(shape, dims, ppc, capacity)
    with a, b:
        p = _hot(*shape, dims, ppc, 9)
        for s in (a, b):
            s.load_particles(p)
            s.reorder()
        for _ in range(steps):
            a.step(1)
            b.step(1)
            pa, pb = a.fetch_particles(), b.fetch_particles()
            assert np.array_equal(pa.flv, pb.flv)
            for k in ("x", "y", "z", "u", "v", "w"):
                assert np.abs(getattr(pa, k) - getattr(pb, k)).max() <= 1e-9, k
        b.load_particles(pa)
        b.load_fields(a.fetch_fields())
        a.step(1)
        b.step(1)
        pa, pb = a.fetch_particles(), b.fetch_particles()
        for k in pa.NAMES:
            assert np.array_equal(getattr(pa, k), getattr(pb, k)), k
        fa, fb = a.fetch_fields(), b.fetch_fields()
        for k in ("Ex", "Ey", "Ez"):
            assert np.abs(getattr(fa, k) - getattr(fb, k)).max() <= 1e-12 * np.abs(getattr(fb, k)).max(), k


def test_tiles_on_the_longest_grid():
    """65535 z cells, the most the field phases launch: a sparse run stepped
    after a reorder by either form, bit for bit (particles), ends included."""
    shape = (5, 5, 65535)
    a, b = _sims(shape, 3, 1, 1 << 14)
    p = _hot(5, 5, 40, 3, 2, 3)
    p.z[:] = 3.0 + (p.z - 3.0) / 40 * 65535
    p.z[:200] = 3.0 + np.linspace(0, 2, 200)
    p.z[200:400] = 65538.0 - np.linspace(1e-3, 2, 200)
    with a, b:
        for s in (a, b):
            s.load_particles(p)
            s.reorder()
            s.step(1)
        pa, pb = a.fetch_particles(), b.fetch_particles()
        for k in pa.NAMES:
            assert np.array_equal(getattr(pa, k), getattr(pb, k)), k
        assert a.device_errors() == 0 and len(pa) > len(p)   # some crossed the z ends
