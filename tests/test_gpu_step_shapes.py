"""The step kernels on both sides of the mesh sizes where their shape changes:
three threads per triangle or one in the FP64 distribute, more or fewer registers
in the FP64 kernels, and where in a kernel (or whether) the next one starts."""
import dataclasses

import numpy as np
import pytest

from helpers import bits_equal, gpu_from_scenario, max_rel, oracle_from_scenario

pytestmark = pytest.mark.gpu

QS = [("stage", "stage"), ("xmomentum", "xmom"), ("ymomentum", "ymom")]


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _scene(triangles, above):
    """The wet/dry beach of about ``triangles`` triangles: at most that many, or
    more."""
    from anuga_cuda import scenarios
    m = int((triangles / 4) ** 0.5)
    n = triangles // (4 * m) + (1 if above else 0)
    assert (4 * m * n > triangles) == above
    return scenarios.wet_dry(m, n)


# The same operations in the same order on both sides, without friction (whose
# power is the math library's own): what is left is the last bits of a few
# products that a compiler may fuse, 1e-16 a step and value.
TOL = 1.0e-12


@pytest.mark.parametrize("flow", [0, 1])
@pytest.mark.parametrize("size", ["one_block", "ragged", "split", "single", "dense"])
def test_fp64_distribute_shapes_match_oracle(size, flow, oracle_mod, swgpu_built):
    from anuga_cuda import DEFAULT, scenarios
    line = 160 * _sms()
    if size == "one_block":
        sc = scenarios.small_basin(3, 2, seed=3)
    elif size == "ragged":
        sc = scenarios.small_basin(41, 23, seed=5)
    else:
        sc = _scene(420 * _sms() if size == "dense" else line, size != "split")
    sc = dataclasses.replace(sc, friction=np.zeros(sc.N))
    p = DEFAULT.replace(flow_algorithm=flow)
    od = oracle_from_scenario(oracle_mod, sc, p)
    od.run_steps(3)
    d = gpu_from_scenario(sc, p)
    st = d.evolve_steps(3)
    assert st.status == 0
    for name, pre in QS:
        q = d.quantities[name]
        assert max_rel(q.centroid_values, od.arrays[pre + "_centroid_values"]) <= TOL, name
        assert max_rel(q.vertex_values, od.arrays[pre + "_vertex_values"].reshape(-1, 3)) <= TOL
        assert max_rel(q.edge_values, od.arrays[pre + "_edge_values"].reshape(-1, 3)) <= TOL


@pytest.mark.parametrize("above", [False, True])
@pytest.mark.parametrize("precision,per_sm", [("fp64", 80), ("fp64", 420), ("mixed", 840),
                                              ("mixed", 1450)])
def test_start_of_the_next_kernel_changes_nothing(precision, per_sm, above, swgpu_built):
    from anuga_cuda import DEFAULT
    from anuga_cuda.autotune import get_config, set_config
    sc = _scene(per_sm * _sms(), above)
    runs = []
    for overlap in (1, 0):
        d = gpu_from_scenario(sc, DEFAULT, precision)
        set_config(d._h, dict(get_config(d._h), dependent_launch=overlap))
        d.evolve_steps(19)
        d.set_timestepping_method("rk2")
        d.evolve_steps(3)
        runs.append([d.get_time()] + [d.quantities[q].centroid_values for q, _ in QS] +
                    [d.quantities[q].edge_values for q, _ in QS])
    for a, b in zip(*runs):
        assert bits_equal(a, b)
