"""The cylindrical E phase of pic_step (E update, fold, AddCurrent and the
zeroing of J in one launch, images included) against the separate phase calls,
at the smallest grid, at remainders of the 32-wide and 8-high blocks and past
one block of theta, on the theta grid and on the modes, FP64 and FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("fp32", 1e-5)])
@pytest.mark.parametrize("modes", [0, 2])
@pytest.mark.parametrize("nx,ny,nz", [(5, 6, 5), (28, 8, 7), (37, 18, 33)])
def test_step_equals_its_phases(nx, ny, nz, modes, precision, tol):
    """Two steps; fields and current (zero) of every cell, ghosts included.
    Only the order of the deposit's atomic sums differs: FP64 1e-13, FP32 1e-5
    of each component's largest value."""
    from pictor_b200 import Particles, PicConfig, Simulation

    rng = np.random.default_rng(nx * 100 + ny)
    n = 6 * nx * ny * nz
    p = Particles.empty(n)
    p.x[:] = 3.0 + nx * rng.random(n) ** 0.5
    p.y[:] = 3.0 + ny * rng.random(n)
    p.z[:] = 3.0 + nz * rng.random(n)
    for k in "uvw":
        getattr(p, k)[:] = rng.normal(scale=0.05, size=n)
    p.q[:] = -(p.x - 3.4)
    p.flv[:] = 2
    cfg = PicConfig(nx=nx, ny=ny, nz=nz, dims=3, c=0.3, qi=0.01, qm=(1.0, -1.0), fdtd="lehe", geom="cylindrical",
                    precision=precision, capacity=4 * n, reorder_period=0, rmin=-0.5, inc_axis=1, cyl_modes=modes)
    with Simulation(cfg) as a, Simulation(cfg) as b:
        for s in (a, b):
            s.load_particles(p)
        for _ in range(2):
            a.step(1)
            b.update_b_half()
            b.move_deposit()
            b.exchange_particles()
            b.update_b_half()
            b.update_e()
            b.fold_current()
            b.add_current()
            b.reset_current()
        fa, fb = a.fetch_fields(), b.fetch_fields()
        for k in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
            va, vb = getattr(fa, k), getattr(fb, k)
            assert np.abs(vb).max() > 0
            assert np.abs(va - vb).max() <= tol * np.abs(vb).max(), k
        for k in ("Jx", "Jy", "Jz"):
            assert not getattr(fa, k).any(), k
