"""Containing balls on wide volumes of one layer of tile groups, whose lists alone are more than the memory
budget of the tiles' lists: the layer is cut into runs of groups. And on a volume of few large pores,
whose long lists still go through in one run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _specks(shape, fraction):
    return (np.random.default_rng(3).random(shape) < fraction).astype(np.uint8)


@pytest.mark.parametrize("shape,fraction,times", [((16, 100, 125), 0.01, (10, 10)), ((23, 93, 110), 0.01, (11, 9))])
def test_runs_of_groups(pma_lib, oracle_mod, shape, fraction, times):
    """Copies of one block, solid walls between them (no ball reaches beyond a wall): each is the oracle's block."""
    import torch
    import porousmediaanalysis_gb300 as pma
    block = _specks(shape, fraction)
    block[:, [0, -1], :] = 1
    block[:, :, [0, -1]] = 1
    e, most, _ = oracle_mod.edt(block)
    want = oracle_mod.containing_balls(e, most)
    mask, count = oracle_mod.max_ball_mask(*want[1:])
    with pma.Context(0) as ctx:
        edt2 = torch.from_numpy(np.tile(e, (1,) + times).view(np.int32)).cuda()
        ctx.set_timing(True)
        crad2, cx, cy, cz, got_mask, got_count = pma.set_containing_balls(ctx, edt2, most)
        entries, runs = ctx.timing_report()["count.balls.runs"]
    # 512 MB of tile lists, 64 B an entry of a group's list; a layer is cut where it does not fit
    assert runs >= 2 and runs >= entries / (1 << 23)
    void = want[0] != 0
    as_u32 = lambda t: t.cpu().numpy().view(np.uint32)
    for i in range(times[0]):
        for j in range(times[1]):
            at = np.s_[:, i * shape[1]:(i + 1) * shape[1], j * shape[2]:(j + 1) * shape[2]]
            assert (as_u32(crad2[at].contiguous()) == want[0]).all()
            assert (as_u32(cx[at].contiguous())[void] == want[1][void] + i * shape[1]).all()
            assert (as_u32(cy[at].contiguous())[void] == want[2][void] + j * shape[2]).all()
            assert (as_u32(cz[at].contiguous())[void] == want[3][void]).all()
            assert (got_mask[at].cpu().numpy() == mask).all()
    assert got_count == count * times[0] * times[1]


def test_memory_of_one_layer(pma_lib):
    """1.3 list entries a voxel in one layer: 8 B each for the groups' lists, 16 B a voxel for the tiles', 13 B a
    voxel for keys, flags and centres, and what the pool holds beside (the tiles' lists of the whole
    layer at once would take 85 B a voxel more)."""
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = torch.from_numpy(_specks((16, 2048, 2048), 0.0003)).cuda()
    with pma.Context(0) as ctx:
        edt2, most, _ = pma.compute_euclidean_distances(ctx, vol)
        before = ctx.scratch_bytes
        pma.set_containing_balls(ctx, edt2, most)
        assert ctx.scratch_bytes - before < 64 * vol.numel()


def test_long_lists_in_one_run(pma_lib):
    """Few large pores: 5 M entries on 10^6 voxels, seven layers that would each leave most of the GPU idle."""
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = torch.from_numpy(_specks((100, 100, 100), 0.00001)).cuda()
    with pma.Context(0) as ctx:
        edt2, most, _ = pma.compute_euclidean_distances(ctx, vol)
        ctx.set_timing(True)
        pma.set_containing_balls(ctx, edt2, most)
        entries, runs = ctx.timing_report()["count.balls.runs"]
    assert 1 << 20 < entries <= 1 << 23 and runs == 1
