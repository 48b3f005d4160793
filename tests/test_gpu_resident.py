"""The resident step (small mixed meshes: whole steps in one launch, a cluster
per scenario) against the step kernels (dependent_launch off), bit for bit:
sizes at the edges of its blocks and clusters and just past them, every
boundary type, every method, yields, tracking, ensembles of unequal scenarios,
and an error in one block that stops the others."""
import numpy as np
import pytest

from helpers import bits_equal, gpu_from_scenario

pytestmark = pytest.mark.gpu

QS = ("stage", "xmomentum", "ymomentum")


def _set(handle, resident):
    from anuga_cuda.autotune import get_config, set_config
    set_config(handle, dict(get_config(handle), dependent_launch=int(resident)))


def _scene(kind, m, n):
    from anuga_cuda import scenarios
    if kind == "harbour":
        return scenarios.tidal_harbour(m, seed=2)
    if kind == "channel":
        return scenarios.channel_inflow(m, n, seed=2, peak=3.0, rise=0.5)
    return scenarios.small_basin(m, n, seed=3)


# 4 m n triangles: one block short and full (96, 128), two blocks, a cluster of
# 16 blocks of 128, 256 and 512 exactly and by one cell more, past the largest
@pytest.mark.parametrize("kind,m,n", [
    ("basin", 6, 4), ("basin", 8, 4), ("channel", 11, 3), ("channel", 32, 16),
    ("basin", 27, 19), ("basin", 32, 32), ("channel", 41, 25), ("basin", 64, 32),
    ("basin", 683, 3), ("harbour", 1500, 0), ("harbour", 6000, 0)])
def test_resident_equals_step_kernels(kind, m, n, swgpu_built):
    from anuga_cuda import DEFAULT
    sc = _scene(kind, m, n)
    for method, steps in (("euler", 33), ("rk2", 7), ("rk3", 5)):
        runs = []
        for resident in (True, False):
            d = gpu_from_scenario(sc, DEFAULT, "mixed")
            d.set_timestepping_method(method)
            _set(d._h, resident)
            d.set_tracking(0.05)
            st = d.evolve_steps(steps)
            runs.append([st.time, st.timestep, st.total_steps, st.stop_reason] +
                        [d.quantities[q].centroid_values for q in QS] +
                        [d.quantities[q].vertex_values for q in QS] +
                        [d.quantities[q].boundary_values for q in QS] + list(d.get_tracking()))
        for a, b in zip(*runs):
            assert bits_equal(a, b), (method, sc.N)


def test_resident_yields_and_single_steps(swgpu_built):
    from anuga_cuda import DEFAULT
    sc = _scene("channel", 21, 9)
    runs = []
    for resident in (True, False):
        d = gpu_from_scenario(sc, DEFAULT, "mixed")
        _set(d._h, resident)
        times = list(d.evolve(yieldstep=0.3, finaltime=1.0))
        more = []
        e = gpu_from_scenario(sc, DEFAULT, "mixed")
        _set(e._h, resident)
        e.evolve_steps(0)
        for _ in range(5):
            more.append(e.step().time)
        runs.append([times, more, d.quantities["stage"].centroid_values,
                     e.quantities["stage"].centroid_values, d._state().total_steps])
    for a, b in zip(*runs):
        assert bits_equal(np.asarray(a), np.asarray(b))


def test_resident_ensemble(swgpu_built):
    from anuga_cuda import DEFAULT
    from anuga_cuda.ensemble import Ensemble
    scs = [_scene("basin", 9, 7), _scene("channel", 33, 17), _scene("harbour", 2500, 0)]
    runs = []
    for resident in (True, False):
        ens = Ensemble(scs, DEFAULT, "mixed")
        _set(ens._h, resident)
        ens.set_tracking(0.05)
        states = ens.evolve([0.4, 1.5, 20.0])
        runs.append([np.array([[s.time, s.total_steps, s.stop_reason] for s in states])] +
                    ens.centroid_values("stage") + ens.centroid_values("xmomentum") +
                    [x for pair in ens.get_tracking() for x in pair])
    for a, b in zip(*runs):
        assert bits_equal(a, b)


def test_resident_error_stops_every_block(swgpu_built):
    from anuga_cuda import DEFAULT
    from anuga_cuda._lib import SwgpuError
    sc = _scene("basin", 30, 20)
    sc.stage_centroid = sc.stage_centroid.copy()
    sc.stage_centroid[-3] = np.nan   # in the last block
    out = []
    for resident in (True, False):
        d = gpu_from_scenario(sc, DEFAULT, "mixed")
        _set(d._h, resident)
        with pytest.raises(SwgpuError) as e:
            d.evolve_steps(40)
        s = d._state()
        out.append((e.value.status, s.total_steps, s.stop_reason))
    assert out[0] == out[1]
