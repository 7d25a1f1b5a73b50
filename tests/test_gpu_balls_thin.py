"""Containing balls on wide volumes of one layer of tile groups, whose lists alone are more than the memory
budget of the tiles' lists: the layer is cut into runs of groups. Bit-exact against the oracle where
that takes seconds; device memory where the lists are longest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _specks(shape, fraction):
    return (np.random.default_rng(3).random(shape) < fraction).astype(np.uint8)


@pytest.mark.parametrize("shape", [(16, 400, 500), (1, 1200, 1301), (23, 380, 401)])
def test_runs_of_groups(pma_lib, oracle_mod, shape):
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = _specks(shape, 0.01 if shape[0] > 1 else 0.003)
    e, most, _ = oracle_mod.edt(vol)
    want = oracle_mod.containing_balls(e, most)
    mask, count = oracle_mod.max_ball_mask(*want[1:])
    with pma.Context(0) as ctx:
        ctx.set_timing(True)
        got = pma.set_containing_balls(ctx, torch.from_numpy(e.view(np.int32)).cuda(), most)
        entries, runs = ctx.timing_report()["count.balls.runs"]
    for a, b in zip(got[:4], want):
        assert (a.cpu().numpy().view(np.uint32) == b).all()
    assert (got[4].cpu().numpy() == mask).all() and got[5] == count
    # 64 MB of tile lists, 64 B an entry of a group's list; a layer is cut where it does not fit
    assert runs >= entries / (1 << 20)


def test_memory_of_one_layer(pma_lib):
    """1.3 list entries a voxel in one layer: 8 B each for the groups' lists, 16 B a voxel for the tiles', 13 B a
    voxel for keys, flags and centres, and what the pool holds beside (the tiles' lists of the whole
    layer at once would take 85 B a voxel more)."""
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = torch.from_numpy(_specks((16, 1024, 1024), 0.0003)).cuda()
    with pma.Context(0) as ctx:
        edt2, most, _ = pma.compute_euclidean_distances(ctx, vol)
        before = ctx.scratch_bytes
        pma.set_containing_balls(ctx, edt2, most)
        assert ctx.scratch_bytes - before < 64 * vol.numel()
