"""The FP64 flux where epsilon lies above ten times H0: each side of an edge is
cut to a dry state by its own depth (below both), whatever the other side's
depth is, as the reference's _compute_speed does; bit for bit with the oracle."""
import numpy as np
import pytest

from helpers import bits_equal, gpu_from_scenario, oracle_from_scenario

pytestmark = pytest.mark.gpu

QS = (("stage", "stage"), ("xmomentum", "xmom"), ("ymomentum", "ymom"))


@pytest.mark.parametrize("optimise", [0, 1])
@pytest.mark.parametrize("epsilon", [1.0e-12, 0.009, 0.01, 0.011, 0.05])
def test_flux_cuts_each_side_by_its_own_depth(epsilon, optimise, oracle_mod, swgpu_built):
    from anuga_cuda import DEFAULT, scenarios
    sc = scenarios.small_basin(17, 13, seed=6)
    rng = np.random.default_rng(8)
    sc.elevation_vertex = np.zeros_like(sc.elevation_vertex)
    h = rng.choice([0.0, 0.004, 0.02, 0.2], sc.N) * rng.uniform(0.5, 1.5, sc.N)
    sc.stage_centroid = h
    sc.xmom_centroid = rng.standard_normal(sc.N) * h
    sc.ymom_centroid = rng.standard_normal(sc.N) * h
    # a flat bed and first order: the edges have the depths drawn above
    p = DEFAULT.replace(epsilon=epsilon, H0=1.0e-3, optimise_dry_cells=optimise, default_order=1)
    od = oracle_from_scenario(oracle_mod, sc, p)
    d = gpu_from_scenario(sc, p)
    for x in (od, d):
        x.distribute_to_vertices_and_edges()
        x.update_boundary()
    for name, pre in QS:
        assert bits_equal(d.quantities[name].edge_values.ravel(),
                          od.arrays[pre + "_edge_values"]), name
    ft = od.compute_fluxes()
    od.gravity_wb()
    assert bits_equal([d.compute_fluxes()], [ft])
    for name, pre in QS:
        assert bits_equal(d.quantities[name].explicit_update,
                          od.arrays[pre + "_explicit_update"]), name
