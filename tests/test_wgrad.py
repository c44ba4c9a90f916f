"""The weight gradients at the edges of their tiles and chunks: grids that fill no
tile of 32 x 8 x 4 voxels, voxel counts that are no multiple of a chunk or of a
segment, rows shorter than a block of 16 voxels, several segments. Against the
NumPy network in its BF16-emulating mode; the tolerance is what a few values
rounded to the neighbouring BF16 number cost a layer's gradient (3 % at most on
the grids of test_warm_start.py; a tap, row or tile left out costs more)."""

import numpy as np
import pytest

from oracle import unet
from tests.test_warm_start import random_fields, random_parameters, rel


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(8, 16, 72), (20, 12, 40), (36, 8, 16), (12, 20, 100), (24, 28, 8)], ids=lambda s: "x".join(map(str, s[::-1])))
def test_weight_gradients_at_tile_edges(shape, sf, lib, cuda):
    params = random_parameters(7)
    b, p_prev, p_target = random_fields(shape, 8)
    with sf.WarmStartNetwork(seed=0, lib=lib) as net:
        net.set_parameters(params)
        loss, grad = net.gradients(b, p_prev, p_target, 1.0)
        again = net.gradients(b, p_prev, p_target, 1.0)[1]
    ref_loss, ref = unet.UNet(params, bf16=True).loss_and_gradients(b, p_prev, p_target, 1.0)
    assert abs(loss - ref_loss) <= 1e-3 * ref_loss
    got, want = unet.split(grad), unet.split(ref)
    for name, _, _ in unet.LAYERS:
        for k in range(2):
            if np.linalg.norm(want[name][k]) > 0:
                assert rel(got[name][k], want[name][k]) <= 5e-2, (name, k)
    assert rel(again, grad) <= 1e-5  # the order of a few atomic additions
