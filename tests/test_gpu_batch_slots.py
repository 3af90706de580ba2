"""A batch whose slots change filters between runs: a recorded run is relaunched
only for filters of the sizes that it was recorded for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


@pytest.mark.parametrize("tiling", [0, 4])
@pytest.mark.parametrize("first,then", [(30000, 5000), (5000, 30000), (3000, 70000)])
@pytest.mark.parametrize("form", [0, 1])
def test_replaced_filter_after_recorded_runs(capi, form, first, then, tiling):
    T, other = 6, 20000
    ox, oy = capi.cv_simulate(T, obs_seed=3)

    def alone(N, seed, runs):  # (the resampling engine goes on from run to run)
        with capi.CVFilter(N, T, form=form, seed=seed) as f:
            f.set_observations_host(ox, oy)
            for _ in range(runs):
                f.initialize()
                f.iterate(T - 1)
            return f.history()

    with capi.CVBatch(2, form=form) as b:
        # (the tile map has room for every run below: its address stays)
        big = b.admit(100000, T, seed=1)
        b.set_observations([big], [(ox, oy)])
        b.run([big])
        b.release(big)
        b.set_tiling(tiling)
        keep = b.admit(other, T, seed=21)
        for k, (N, seed) in enumerate(((first, 31), (then, 32), (first, 33))):
            slot = b.admit(N, T, seed=seed)
            slots = [keep, slot]
            for _ in range(4):  # two direct runs, one recorded, one relaunched
                b.set_observations(slots, [(ox, oy)] * 2)
                b.initialize(slots)
                b.run(slots)
            for s, want in ((keep, alone(other, 21, 4 * k + 4)), (slot, alone(N, seed, 4))):
                got = b.history(s)
                for q in want:
                    assert np.array_equal(got[q], want[q]), (N, q)
            b.release(slot)
