"""Manning friction where its comparisons meet a NaN, which fails them: a triangle
without a friction value (NaN) has none, and one whose depth is NaN gets no
term, as in the reference's `if (eta > eps) ... if (h >= eps)`."""
import dataclasses

import numpy as np
import pytest

from helpers import bits_equal, gpu_from_scenario, max_rel, oracle_from_scenario

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sloped", [0, 1])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nan_friction_is_no_friction(precision, sloped, swgpu_built):
    from anuga_cuda import DEFAULT, scenarios
    sc = scenarios.small_basin(16, 12, seed=3)
    p = DEFAULT.replace(use_sloped_mannings=sloped)
    runs = []
    for value in (0.0, np.nan, -np.nan):
        eta = sc.friction.copy()
        eta[::3] = value
        d = gpu_from_scenario(dataclasses.replace(sc, friction=eta), p, precision)
        st = d.evolve_steps(12)
        assert st.status == 0
        runs.append([d.quantities[q].centroid_values for q in ("stage", "xmomentum", "ymomentum")])
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert bits_equal(a, b)


@pytest.mark.parametrize("explicit", [False, True])
def test_nan_depth_and_friction_per_method(explicit, oracle_mod, swgpu_built):
    from anuga_cuda import DEFAULT, scenarios
    sc = scenarios.small_basin(16, 12, seed=3)
    sc.friction = sc.friction.copy()
    sc.friction[::5] = np.nan
    sc.stage_centroid = sc.stage_centroid.copy()
    sc.stage_centroid[1::5] = np.nan
    od = oracle_from_scenario(oracle_mod, sc, DEFAULT)
    d = gpu_from_scenario(sc, DEFAULT)
    if explicit:
        od.manning_friction_explicit()
        d.manning_friction_explicit()
    else:
        od.manning_friction()
        d.compute_forcing_terms()
    for name, pre in (("xmomentum", "xmom"), ("ymomentum", "ymom")):
        q = d.quantities[name]
        got = q.explicit_update if explicit else q.semi_implicit_update
        want = od.arrays[pre + ("_explicit_update" if explicit else "_semi_implicit_update")]
        assert not got[::5].any() and not got[1::5].any() and np.any(got)
        assert max_rel(got, want) <= 1e-13, name  # pow: an ulp of either
