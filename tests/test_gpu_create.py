"""What creating a run costs and keeps."""
import statistics
import time

import pytest

pytestmark = pytest.mark.gpu


def test_a_run_created_alone_costs_what_it_costs_beside_another():
    """Creating and destroying a small run pins and frees no memory for the only
    run of a program: the median of 60 takes at most twice what it takes while
    another run is alive (1.8 against 1.2 ms: the driver gives the blocks of
    small device allocations back with the last of them; with a pinned block
    made and freed each time it was 4.2 against 1.1 ms)."""
    from pictor_b200 import PicConfig, Simulation

    cfg = PicConfig(nx=64, ny=64, dims=2, c=0.45, qi=0.01, precision="fp32", capacity=40000)

    def once():
        t = time.perf_counter()
        Simulation(cfg).close()
        return time.perf_counter() - t

    for _ in range(10):
        once()
    best = float("inf")
    for _ in range(3):      # a busy host slows one side or the other
        alone, beside = [], []
        for _ in range(3):
            alone += [once() for _ in range(20)]
            with Simulation(cfg):
                beside += [once() for _ in range(20)]
        best = min(best, statistics.median(alone) / statistics.median(beside))
        if best <= 2.0:
            return
    assert best <= 2.0, best


def test_more_runs_than_shared_slots():
    """Past the 256 slots of the shared pinned block a run pins its own; slots
    given back are taken again; every run's words are its own."""
    from pictor_b200 import PicConfig, Simulation

    cfg = PicConfig(nx=5, ny=5, dims=2, c=0.45, qi=0.01, precision="fp32", capacity=64)
    runs = [Simulation(cfg) for _ in range(260)]
    try:
        for _ in range(2):
            assert all(s.particle_count() == 0 and s.diagnostics()["rho_max"] == 0 for s in runs[::37] + runs[-5:])
            for s in runs[100:258]:
                s.close()
            runs[100:258] = [Simulation(cfg) for _ in range(158)]
    finally:
        for s in runs:
            s.close()
