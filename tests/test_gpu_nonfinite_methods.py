"""The FP64 distribute and fluxes on states that are not numbers (NaN and infinities
of either sign in stage and momentum): the comparisons of the limiter, the dry
test, the balance and the flux come out as the reference's C comparisons do, so
that every number is the oracle's bit for bit and NaN stands where the oracle's
does.  In every form that the mesh size picks."""
import numpy as np
import pytest

from helpers import gpu_from_scenario, oracle_from_scenario

pytestmark = pytest.mark.gpu

QS = (("stage", "stage"), ("xmomentum", "xmom"), ("ymomentum", "ymom"))

VARIANTS = {
    "default": {},
    "betas_differ": {"beta_w_dry": 0.2, "beta_uh_dry": 0.1, "beta_vh_dry": 0.3},
    "momentum": {"extrapolate_velocity_second_order": 0},
    "loose_slopes": {"tight_slope_limiters": 0},
    "blended": {"use_centroid_velocities": 0},
    "all_cells": {"optimise_dry_cells": 0},
    "first_order": {"default_order": 1},
    "vertex_limiter": {"optimised_gradient_limiter": 0},
    "tsunami": {"flow_algorithm": 1},
    "tsunami_betas": {"flow_algorithm": 1, "beta_w_dry": 0.2, "beta_uh_dry": 0.1},
}


def _scene(single):
    import torch
    from anuga_cuda import scenarios
    if not single:
        return scenarios.small_basin(31, 23, seed=5)
    line = 160 * torch.cuda.get_device_properties(0).multi_processor_count
    m = int((line / 4) ** 0.5) + 2
    return scenarios.small_basin(m, m, seed=5)


def _same(got, want):
    got, want = np.ravel(got), np.ravel(want)
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(got[~nan], want[~nan])


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("odd", ["nan", "inf"])
@pytest.mark.parametrize("variant", VARIANTS)
def test_distribute_of_odd_states(variant, odd, single, oracle_mod, swgpu_built):
    from anuga_cuda import DEFAULT
    sc = _scene(single)
    rng = np.random.default_rng(11)
    values = [np.nan, -np.nan] if odd == "nan" else [np.inf, -np.inf]
    for name in ("stage_centroid", "xmom_centroid", "ymom_centroid"):
        a = getattr(sc, name).copy()
        at = rng.choice(sc.N, sc.N // 60, replace=False)
        a[at] = rng.choice(values, len(at))
        setattr(sc, name, a)
    p = DEFAULT.replace(**VARIANTS[variant])
    od = oracle_from_scenario(oracle_mod, sc, p)
    d = gpu_from_scenario(sc, p)
    od.distribute_to_vertices_and_edges()
    d.distribute_to_vertices_and_edges()
    for name, pre in QS:
        q = d.quantities[name]
        assert _same(q.centroid_values, od.arrays[pre + "_centroid_values"]), name
        assert _same(q.vertex_values, od.arrays[pre + "_vertex_values"]), name
        assert _same(q.edge_values, od.arrays[pre + "_edge_values"]), name
    od.update_boundary()
    d.update_boundary()
    ft = od.compute_fluxes()
    od.gravity_wb()
    assert _same([d.compute_fluxes()], [ft])
    for name, pre in QS:
        assert _same(d.quantities[name].explicit_update,
                     od.arrays[pre + "_explicit_update"]), name
