"""A call that the library refuses leaves no trace: what it was given is neither
reported nor used by the calls after it."""
import ctypes as C

import numpy as np
import pytest

from helpers import bits_equal

pytestmark = pytest.mark.gpu

EINVAL = 1  # SWGPU_EINVAL


def _ensemble(precision):
    from anuga_cuda import DEFAULT, scenarios
    from anuga_cuda.ensemble import Ensemble
    return Ensemble([scenarios.small_basin(9, 7, seed=s) for s in (1, 2, 3)], DEFAULT, precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_refused_finaltimes_are_forgotten(precision, swgpu_built):
    from anuga_cuda import _lib
    from anuga_cuda._lib import f64p, lib
    runs = []
    for refused in (False, True):
        ens = _ensemble(precision)
        ens.evolve(1.0, max_steps=9)
        before = [(s.finaltime, s.time) for s in ens.states()]
        if refused:
            times = np.array([s.time for s in ens.states()])
            bad = np.full(3, 0.5 * (times.max() + 1.0))
            bad[2] = 0.5 * times.min()  # before its scenario's time
            assert lib().swgpu_ensemble_set_finaltimes(ens._h, f64p(bad)) == EINVAL
            assert [(s.finaltime, s.time) for s in ens.states()] == before
        st = _lib.State_t()
        assert lib().swgpu_evolve_run(ens._h, 0, C.byref(st)) == 0
        runs.append([np.array([[s.time, s.finaltime, s.total_steps] for s in ens.states()])] +
                    ens.centroid_values("stage"))
    assert (runs[0][0][:, 0] == 1.0).all()
    for a, b in zip(*runs):
        assert bits_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_refused_run_is_forgotten(precision, swgpu_built):
    """A run past every final time is refused; the clocks stay, and a later final
    time runs on from there."""
    from anuga_cuda import _lib
    from anuga_cuda._lib import f64p, lib
    runs = []
    for refused in (False, True):
        ens = _ensemble(precision)
        before = [(s.time, s.total_steps, s.stop_reason) for s in ens.evolve(0.25)]
        st = _lib.State_t()
        if refused:
            assert lib().swgpu_evolve_run(ens._h, 0, C.byref(st)) == EINVAL
            assert [(s.time, s.total_steps, s.stop_reason) for s in ens.states()] == before
        assert lib().swgpu_ensemble_set_finaltimes(ens._h, f64p(np.full(3, 0.1))) == EINVAL
        assert lib().swgpu_evolve_start(ens._h, 0.0, 0.5, 0.5) == 0
        assert lib().swgpu_evolve_run(ens._h, 0, C.byref(st)) == 0
        runs.append([np.array([[s.time, s.total_steps] for s in ens.states()])] +
                    ens.centroid_values("stage"))
    for a, b in zip(*runs):
        assert bits_equal(a, b)
