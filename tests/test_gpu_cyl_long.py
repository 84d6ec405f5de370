"""Cylinders of many z cells: every launch of the field phases within the grid
limits for as many planes as the smallest of them allows (65530), and an error
on every step beyond it."""
import numpy as np
import pytest

from pictor_b200.simulation import Fields

pytestmark = pytest.mark.gpu

NR, NT = 5, 6


def _sim(nz, precision, modes):
    from pictor_b200 import PicConfig, Simulation

    return Simulation(PicConfig(nx=NR, ny=NT, nz=nz, dims=3, c=0.3, qi=0.01, qm=(1.0, -1.0), fdtd="yee",
                                geom="cylindrical", precision=precision, capacity=64, reorder_period=0, rmin=-0.5,
                                inc_axis=1, cyl_modes=modes))


def _tile(a, nz, reps, ghosts=1):
    """The interior z planes of a repeated, with the periodic z ghosts (times
    ghosts: a current without any folds to itself)."""
    b = np.tile(a[:, :, 2:2 + nz], (1, 1, reps))
    return np.asfortranarray(np.concatenate([ghosts * b[:, :, -2:], b, ghosts * b[:, :, :3]], axis=2))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("modes", [0, 2])
@pytest.mark.parametrize("nz,reps", [(22, 1000), (10, 6553)])
def test_long_cylinder_repeats_the_short_one(nz, reps, modes, precision):
    """Fields and a current of period nz along z: a step without particles,
    then the separate E phase calls, of a cylinder of reps periods equal those
    of one period, repeated, in every cell bit for bit (no sums by atomics)."""
    rng = np.random.default_rng(nz)
    with _sim(nz, precision, modes) as a, _sim(nz * reps, precision, modes) as b:
        f = Fields(*(np.asfortranarray(rng.normal(size=a.cfg.shape)) for _ in range(9)))
        per = {k: _tile(getattr(f, k), nz, 1) for k in Fields.__dataclass_fields__}
        a.load_fields(Fields(**per))
        b.load_fields(Fields(**{k: _tile(v, nz, reps) for k, v in per.items()}))

        def same():
            fa, fb = a.fetch_fields(False), b.fetch_fields(False)
            for k in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
                want = _tile(getattr(fa, k), nz, reps)
                assert np.abs(want).max() > 0
                bad = np.argwhere(want != getattr(fb, k))
                assert len(bad) == 0, (k, len(bad), bad[:4])

        for s in (a, b):
            s.step(2)
        same()
        for s, r in ((a, 1), (b, reps)):
            s.load_current(*(_tile(per[k], nz, r, 0) for k in ("Jx", "Jy", "Jz")))
            s.update_e()
            s.fold_current()
            s.add_current()
        same()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_step_that_cannot_be_launched_fails_every_time(precision):
    """One z plane more than a launch can index: the step's graph is refused,
    not kept without that launch, so the second call fails as the first does;
    a run of another size on the same device is not disturbed."""
    from pictor_b200._capi import PicError

    with _sim(66000, precision, 0) as s, _sim(12, precision, 0) as t:
        for _ in range(3):
            with pytest.raises(PicError, match="CUDA"):
                s.step(1)
        t.step(1)
        assert t.device_errors() == 0
