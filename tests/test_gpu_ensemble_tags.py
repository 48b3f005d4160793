"""Time-dependent boundaries of an ensemble in the step kernels of the mixed
path: evaluated once per tag and stage at the time of the tag's scenario, or
edge by edge where scenarios share a tag.  Either way every scenario runs as it
does alone, bit for bit."""
import numpy as np
import pytest

from helpers import bits_equal, gpu_from_scenario

pytestmark = pytest.mark.gpu


def _scenarios(shared):
    from anuga_cuda import scenarios
    if shared:  # the same boundaries, on two meshes
        return [scenarios.tidal_harbour(1500, seed=1), scenarios.tidal_harbour(2600, seed=1)]
    return [scenarios.tidal_harbour(1500, seed=1),
            scenarios.inflow_harbour(2600, seed=3, peak=300.0, rise=60.0),
            scenarios.small_basin(6, 5, seed=4), scenarios.tidal_harbour(900, seed=5)]


@pytest.mark.parametrize("shared", [False, True])
def test_scenarios_keep_their_clocks(shared, swgpu_built):
    from anuga_cuda import DEFAULT
    from anuga_cuda.autotune import get_config, set_config
    from anuga_cuda.ensemble import Ensemble

    class Shared(Ensemble):
        """Every scenario's edges with the tags of the first."""

        def _create(self):
            n = len(self.scenarios[0].mesh.tag_names)
            t = self.arrays["boundary_tag"]
            self.arrays["boundary_tag"] = np.where(t < self.pad_tag, t % n, t)
            super()._create()

    scs = _scenarios(shared)
    if shared:
        assert scs[0].mesh.tag_names == scs[1].mesh.tag_names
    ens = (Shared if shared else Ensemble)(scs, DEFAULT, "mixed")
    # the step kernels, which a mesh of this size does without otherwise
    set_config(ens._h, dict(get_config(ens._h), dependent_launch=0))
    ens.evolve(1.0e6, max_steps=37)
    stages, xmoms = ens.centroid_values("stage"), ens.centroid_values("xmomentum")
    for i, sc in enumerate(scs):
        d = gpu_from_scenario(sc, DEFAULT, "mixed")
        d.evolve_steps(37)
        assert bits_equal(stages[i], d.quantities["stage"].centroid_values), i
        assert bits_equal(xmoms[i], d.quantities["xmomentum"].centroid_values), i
