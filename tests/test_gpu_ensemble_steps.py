"""Ensembles too large for the resident step, as users run them: programmatic
dependent launches, every scenario's time-dependent tags at its own clock, and
launches that shrink as scenarios finish.  Every scenario runs as it does alone,
bit for bit, with the overlap of the step kernels on and off."""
import numpy as np
import pytest

from helpers import bits_equal, gpu_from_scenario

pytestmark = pytest.mark.gpu

FINALS = [12.0, 6.0, 0.4, 3.0]


def _scenarios():
    from anuga_cuda import scenarios
    return [scenarios.tidal_harbour(9500, seed=1),
            scenarios.inflow_harbour(2600, seed=3, peak=300.0, rise=60.0),
            scenarios.small_basin(6, 5, seed=4), scenarios.tidal_harbour(900, seed=5)]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("method", ["euler", "rk2"])
def test_scenarios_run_as_alone(precision, method, swgpu_built):
    from anuga_cuda import DEFAULT
    from anuga_cuda._lib import check, lib
    from anuga_cuda.autotune import get_config, set_config
    from anuga_cuda.ensemble import Ensemble
    scs = _scenarios()
    assert scs[0].N > 8192
    runs = []
    for overlap in (1, 0):
        ens = Ensemble(scs, DEFAULT, precision)
        set_config(ens._h, dict(get_config(ens._h), dependent_launch=overlap))
        check(lib().swgpu_set_timestepping_method(ens._h, {"euler": 1, "rk2": 2}[method]), ens._h)
        ens.set_tracking(0.05)
        states = ens.evolve(FINALS)
        runs.append((states, ens.centroid_values("stage"), ens.centroid_values("xmomentum"),
                     ens.get_tracking()))
    for i, (sc, final) in enumerate(zip(scs, FINALS)):
        d = gpu_from_scenario(sc, DEFAULT, precision)
        d.set_timestepping_method(method)
        d.set_tracking(0.05)
        assert list(d.evolve(yieldstep=final, finaltime=final))[-1] == final
        want = d._state()
        for states, stage, xmom, tracked in runs:
            assert (states[i].time, states[i].total_steps) == (final, want.total_steps), i
            assert bits_equal(stage[i], d.quantities["stage"].centroid_values), i
            assert bits_equal(xmom[i], d.quantities["xmomentum"].centroid_values), i
            for a, b in zip(tracked[i], d.get_tracking()):
                assert np.array_equal(a, b), i
    # the scenarios took different numbers of steps: the launches shrank
    assert len({s.total_steps for s in runs[0][0]}) > 1
