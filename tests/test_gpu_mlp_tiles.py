"""Training batches of several tiles a block: the next tile is gathered into a
second buffer while the current one is worked on."""
import numpy as np
import pytest

from test_mlp import params_for


@pytest.mark.gpu
@pytest.mark.parametrize("nin,nh,B", [(6, 64, 2049), (6, 64, 4097), (20, 48, 4500), (40, 64, 6200)])
def test_gradient_over_several_tiles(pkg, po, nin, nh, B):
    """2,049 samples over 16 blocks are a full tile of 128 and a second of one row
    each, the last block less than one tile; 4,097 the same with a third tile.
    Tolerance as for one tile: 1e-4 of the largest entry, for the accumulation
    order and activations on a bfloat16 rounding boundary."""
    rng = np.random.default_rng(nin * 1000 + B)
    prm = po.bf16_round(params_for(nin, nh, 11))
    x = rng.normal(size=(B, nin)).astype(np.float32)
    y = rng.normal(size=(B, 2)).astype(np.float32)
    g_dev, L_dev = pkg._handle(0).learn_gradcheck(nin, nh, prm, x, y)
    g_ref, L_ref = po.mlp_forward_backward(nin, nh, prm, x, y, rounding="device")
    assert abs(L_dev - L_ref) <= 1e-4 * abs(L_ref)
    assert np.abs(g_dev - g_ref).max() <= 1e-4 * np.abs(g_ref).max()
