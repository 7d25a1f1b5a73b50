"""Containing balls on extents around the bricks of the kept-centre kernel (32 x 8 x 8) and the tiles of
8^3, and with enough kept centres (2^18) that they are taken by descending radius. Bit-exact
against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 9, 33), (7, 8, 32), (8, 9, 31), (9, 16, 65), (17, 7, 40), (80, 96, 100)]


@pytest.mark.parametrize("fraction", [0.0, 0.01, 0.15])
@pytest.mark.parametrize("shape", SHAPES)
def test_balls_forms(ctx, oracle_mod, shape, fraction):
    import torch
    import porousmediaanalysis_gb300 as pma
    if fraction == 0.0 and shape[0] > 40:
        pytest.skip("balls of the whole box: the oracle's scatter takes minutes")
    vol = (np.random.default_rng(3).random(shape) < fraction).astype(np.uint8)
    e, most, _ = oracle_mod.edt(vol)
    want = oracle_mod.containing_balls(e, most)
    mask, count = oracle_mod.max_ball_mask(*want[1:])
    edt2 = torch.from_numpy(e.view(np.int32)).cuda()
    got = pma.set_containing_balls(ctx, edt2, most)
    for a, b in zip(got[:4], want):
        assert (a.cpu().numpy().view(np.uint32) == b).all()
    assert (got[4].cpu().numpy() == mask).all() and got[5] == count
