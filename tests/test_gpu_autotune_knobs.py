"""The autotuner times no two shapes that are the same launches: the resident step
reads no block size, the FP64 blocks of a small mesh shrink whatever their upper
bound is, and its distribute has a shape of its own."""
import pytest

from helpers import gpu_from_scenario

pytestmark = pytest.mark.gpu

SHAPE = {"flux_block": 128, "update_block": 256, "distribute_block": 256, "steps_per_graph": 16,
         "flux_pipelined": 0, "dependent_launch": 1}


def _domain(m, precision):
    from anuga_cuda import DEFAULT, scenarios
    return gpu_from_scenario(scenarios.small_basin(m, m, seed=1), DEFAULT, precision)


def test_resolved_shapes(swgpu_built):
    from anuga_cuda._lib import SwgpuError
    from anuga_cuda.autotune import resolve_config
    small, large = _domain(20, "mixed"), _domain(50, "mixed")  # 1,600 and 10,000 triangles
    assert resolve_config(small._h, SHAPE) == dict.fromkeys(SHAPE, 0) | {"dependent_launch": 1}
    kernels = dict(SHAPE, dependent_launch=0)
    assert resolve_config(small._h, kernels) == kernels
    assert resolve_config(large._h, SHAPE) == SHAPE
    d = _domain(20, "fp64")
    one, other = (resolve_config(d._h, dict(SHAPE, flux_block=f, update_block=u, flux_pipelined=p,
                                            distribute_block=u))
                  for f, u, p in ((64, 128, 0), (128, 512, 1)))
    assert one == other and one["flux_block"] == one["update_block"] == 32
    assert one["distribute_block"] == 0 and one["steps_per_graph"] == 16
    with pytest.raises(SwgpuError):
        resolve_config(d._h, dict(SHAPE, update_block=1024))


@pytest.mark.parametrize("precision,m,shapes", [("mixed", 20, 1), ("fp64", 20, 3),
                                                ("mixed", 50, 11)])
def test_same_launches_are_timed_once(precision, m, shapes, monkeypatch, swgpu_built):
    from anuga_cuda import autotune
    d = _domain(m, precision)
    d.evolve_steps(0)
    timed = []
    monkeypatch.setattr(autotune, "_time_shape",
                        lambda h, cfg, steps: timed.append(dict(cfg)) or 1.0)
    rec = autotune.tune_handle(d._h, steps=2)
    # the default, and each shape that differs from all before it: for the small
    # FP64 mesh the graph lengths alone
    assert len(timed) == shapes, timed
    assert rec["config"] == timed[0]
