"""Seed-set unions of every size of the level sweep: a corridor of radius 1 whose side voxels, all of
different larger radii, each start a pore, so that the corridor's plateau unites as many seed sets
as there are side voxels. 31 to 33 edges: a warp's union or the block's; 1024 and 2048: what the
block's hash set holds in a run of small levels and in a level of its own; beyond: merged by
expansion and sort. `others` isolated voxels of radius 1 make the corridor's level a large one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _corridor(count, others):
    """(mask, edt2 = crad2, side voxel positions in order of their radii) for the 6-neighbour stencil."""
    length = 2 * ((count + 3) // 4) + 2
    sy = max(length, 2 * others + 1)
    r2 = np.zeros((3, 6, sy), np.uint32)
    r2[1, 1, :length] = 1
    sides = [(1 + dz, 1 + dx, y) for y in range(0, length, 2) for dz, dx in ((-1, 0), (1, 0), (0, -1), (0, 1))][:count]
    order = np.random.default_rng(count).permutation(count)
    for k, i in enumerate(order):
        r2[sides[i]] = 2 + k
    for k in range(others):
        r2[1, 5, 2 * k] = 1
    mask = np.where(r2 != 0, 127, 0).astype(np.uint8)
    mask[r2 > 1] = 255
    mask[1, 5] = np.where(r2[1, 5] != 0, 255, 0)
    return mask, r2, [sides[i] for i in order]


@pytest.mark.parametrize("others", [0, 100])
@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 128, 129, 600, 1024, 1025, 2048, 2049, 2600])
def test_union_sizes(ctx, count, others):
    import torch
    import porousmediaanalysis_gb300 as pma
    mask, r2, sides = _corridor(count, others)
    d = torch.from_numpy(r2.view(np.int32)).cuda()
    labels, table = pma.assign_pore_and_throat_ids(ctx, torch.from_numpy(mask).cuda(), d, d, pma.D3Q7)
    labels = labels.cpu().numpy().view(np.uint32)
    pores, throats = table.rows()
    by_radius = sides[::-1]  # pores are numbered by decreasing radius
    assert len(pores) == count + others
    assert [(p[3], p[1], p[2]) for p in pores[:count]] == by_radius
    ids = [p[0] for p in pores]
    assert [labels[v] for v in by_radius] == ids[:count]
    corridor = labels[1, 1][r2[1, 1] == 1]
    if count == 1:
        assert throats == [] and (corridor == ids[0]).all() and pores[0][6] == 1 + corridor.size
        return
    assert len(throats) == 1 and (corridor == throats[0][0]).all() and throats[0][1] == corridor.size
    assert list(throats[0][2]) == [ids[1], ids[0]] + ids[2:count]
    assert all(p[6] == 1 for p in pores)
