"""The current filter (three axes and components in one launch) against the
oracle's axis-by-axis passes: odd and even pass counts (the result ends in
either buffer), block and plane-chunk remainders, the smallest grid."""
import numpy as np
import pytest

from oracle import oracle as O

from ._util import grid_and_config, to_gpu_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,nx,ny,nz,passes", [(2, 5, 5, 1, 1), (2, 33, 17, 1, 2), (3, 5, 5, 5, 3),
                                                   (3, 34, 9, 17, 1), (3, 31, 16, 8, 2)])
def test_filter_equals_the_oracle(dims, nx, ny, nz, passes):
    """The phase call on a random folded current, bit for bit on the interior,
    and one filtered step (the deposit's atomic order: 1e-12 of the fields)."""
    from pictor_b200 import Simulation

    g, cfg = grid_and_config(dims=dims, nx=nx, ny=ny, nz=nz, curr_filter=passes, qi=0.0016)
    p = O.load_weibel(dims, nx, ny, nz, epc=4, drift=0.4, temp=0.02, seed=11)
    o = O.Oracle(g, p.copy())
    rng = np.random.default_rng(nx)
    for a in (o.f.Jx, o.f.Jy, o.f.Jz):
        a[...] = rng.normal(size=a.shape)
    k = slice(2, -3) if dims == 3 else slice(None)
    with Simulation(cfg) as s:
        s.load_particles(to_gpu_particles(p))
        s.load_current(o.f.Jx, o.f.Jy, o.f.Jz)
        o.fold_current()
        s.fold_current()
        o.filter_current(passes)
        s.filter_current()
        f = s.fetch_fields()
        for n in ("Jx", "Jy", "Jz"):
            assert np.array_equal(getattr(f, n)[2:-3, 2:-3, k], getattr(o.f, n)[2:-3, 2:-3, k]), n
        for t in (1, 2):
            o.step_filtered(t, 0, passes)
            s.step(1)
        f = s.fetch_fields()
        for n in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
            ref = getattr(o.f, n)
            assert np.abs(getattr(f, n) - ref).max() <= 1e-12 * max(np.abs(o.f.Ex).max(), 1e-300), n
        for n in ("Jx", "Jy", "Jz"):
            assert not getattr(f, n).any(), n
