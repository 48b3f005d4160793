"""The FP64 step kernels' forms by mesh size (three threads per triangle or one
in the distribute, more or fewer registers, the clock by the update or by the
flux's last block) under every parameter that the distribute branches on.  The
form follows an ensemble's total size, so copies of one small scenario, as few
as take the first form and as many as take each of the others, have to stay the
same bits."""
import ctypes as C

import numpy as np
import pytest

from helpers import bits_equal

pytestmark = pytest.mark.gpu

VARIANTS = {
    "default": {},
    "first_order": {"default_order": 1},
    "vertex_limiter": {"optimised_gradient_limiter": 0},
    "edge_limiter": {"use_edge_limiter": 1},
    "betas_differ": {"beta_w_dry": 0.2, "beta_uh": 0.7, "beta_uh_dry": 0.1, "beta_vh_dry": 0.3},
    "momentum": {"extrapolate_velocity_second_order": 0},
    "blended_momentum": {"use_centroid_velocities": 0, "extrapolate_velocity_second_order": 0},
    "loose_slopes": {"tight_slope_limiters": 0},
    "dry_cells": {"optimise_dry_cells": 0},
    "speed_and_slope": {"maximum_allowed_speed": 0.5, "use_sloped_mannings": 1},
    "tsunami": {"flow_algorithm": 1},
    "tsunami_betas": {"flow_algorithm": 1, "beta_w_dry": 0.2, "beta_uh_dry": 0.1},
    "tsunami_momentum": {"flow_algorithm": 1, "extrapolate_velocity_second_order": 0},
}


def _values(ens):
    """Centroid, vertex and edge values of the conserved quantities, per copy."""
    from anuga_cuda import _lib
    from anuga_cuda._lib import check, f64p, lib
    out = []
    for q in (_lib.STAGE, _lib.XMOMENTUM, _lib.YMOMENTUM):
        c, v, e = np.empty(ens.N), np.empty(3 * ens.N), np.empty(3 * ens.N)
        check(lib().swgpu_get_quantity(ens._h, q, f64p(c), f64p(v), f64p(e)), ens._h)
        out += [a.reshape(len(ens), -1) for a in (c, v, e)]
        b = np.empty(ens.Nb)
        check(lib().swgpu_get_boundary_values(ens._h, q, f64p(b)), ens._h)
        out.append(b.reshape(len(ens), -1))
    return out


def _run(sc, copies, params):
    from anuga_cuda._lib import check, lib
    from anuga_cuda.ensemble import Ensemble
    ens = Ensemble([sc] * copies, params, "fp64")
    states = ens.evolve(1.0e6, max_steps=6)
    out = [np.array([[s.time, s.timestep, s.total_steps, s.status] for s in states])]
    out += _values(ens)
    if not params.flow_algorithm:
        check(lib().swgpu_extrapolate_second_order_sw(ens._h), ens._h)
        out += _values(ens)
    return out


@pytest.mark.parametrize("variant", VARIANTS)
def test_every_form_gives_the_same_bits(variant, swgpu_built):
    import torch
    from anuga_cuda import DEFAULT, scenarios
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sc = scenarios.small_basin(9, 7, seed=1)  # 252 triangles, 256 with the padding
    params = DEFAULT.replace(**VARIANTS[variant])
    want = _run(sc, 2, params)
    assert (want[0][:, 3] == 0).all()
    for per_sm in (160, 420, 1500):  # past each of the sizes where a form changes
        copies = per_sm * sms // 256 + 1
        got = _run(sc, copies, params)
        for a, b in zip(want, got):
            assert bits_equal(np.broadcast_to(a[0], b.shape), b), (variant, per_sm)
