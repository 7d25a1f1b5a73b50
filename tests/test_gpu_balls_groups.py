"""Containing balls on extents around the groups of 2 x 2 x 2 tiles of 8^3 that share a list (one tile, one
voxel into the next, odd tile counts), with few and with more than 8192 groups, the two forms of the
lists' counters. Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (16, 16, 16), (17, 15, 16), (24, 9, 33), (40, 41, 23), (1, 1500, 1501)])
def test_balls_groups(ctx, oracle_mod, shape):
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = (np.random.default_rng(11).random(shape) < 0.04).astype(np.uint8)
    vol[:, :, : shape[2] // 3] = 1  # tiles without a void voxel
    e, most, _ = oracle_mod.edt(vol)
    want = oracle_mod.containing_balls(e, most)
    mask, count = oracle_mod.max_ball_mask(*want[1:])
    edt2 = torch.from_numpy(e.view(np.int32)).cuda()
    got = pma.set_containing_balls(ctx, edt2, most)
    for a, b in zip(got[:4], want):
        assert (a.cpu().numpy().view(np.uint32) == b).all()
    assert (got[4].cpu().numpy() == mask).all() and got[5] == count
