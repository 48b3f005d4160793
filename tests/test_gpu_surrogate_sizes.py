"""Inference at the sizes where its tiling can go wrong: single rows, the edges
of a 128-row tile and of the 256 rows that a pair of CTAs works on, one tile of
a pair missing, and one pair more than the GPU has.  The training forward walks
single tiles with other kernels but adds in the same order, so the outputs
agree bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def network():
    import torch
    from anuga_cuda.surrogate import FamilyMesh, Surrogate, sample_params
    fm = FamilyMesh(cells=40)
    need = 2 * 128 * (torch.cuda.get_device_properties(0).multi_processor_count // 2 + 1)
    scen = -(-need // fm.N) + 1
    sg = Surrogate(fm, seed=6)
    sg.set_data(sample_params(scen, seed=9), np.zeros((scen, fm.N, 2), np.float32))
    return sg, scen * fm.N, need


@pytest.mark.parametrize("row0,rows", [
    (0, 1), (5, 127), (0, 128), (77, 129), (1, 255), (0, 256), (3, 257), (9, 383), (2, 385),
    (0, -255), (4, -256), (0, -128), (7, 0), (1, 1)])
def test_predict_at_tile_edges(network, row0, rows):
    """``rows`` at or below zero: that many fewer than one pair of tiles more
    than there are pairs of SMs."""
    import torch
    from anuga_cuda import _lib
    sg, total, most = network
    n = rows if rows > 0 else most + rows
    assert row0 + n <= total
    out = torch.full((n + 8, 3), -7.0, dtype=torch.float32, device="cuda")
    sg._check(_lib.lib().swgpu_mlp_predict(sg._h, row0, n, C.c_void_p(out.data_ptr()), None), sg._h)
    y, _, _ = sg.gradients(np.arange(row0, row0 + n, dtype=np.int64))
    got = out.cpu().numpy()
    assert np.array_equal(got[:n], y)
    assert (got[n:] == -7.0).all()  # nothing past the last row
