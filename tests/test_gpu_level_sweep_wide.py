"""Seed-set unions of the level sweep over more edges than one block takes: 4096 and 16384 fill a block's
hash set while its other warps still read sets, 65536 edges are the most that a block looks at,
from 65537 on the union is spread over the GPU. `others` isolated voxels of the corridor's radius make its
level a launch of its own instead of one of a run. Compared with the rows that follow from the
construction."""
import numpy as np
import pytest

from test_gpu_level_sweep import _corridor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("others", [0, 100])
@pytest.mark.parametrize("count", [4096, 16384, 65536, 65537, 70000])
def test_wide_unions(pma_lib, count, others):
    import torch
    import porousmediaanalysis_gb300 as pma
    mask, r2, sides = _corridor(count, others)
    d = torch.from_numpy(r2.view(np.int32)).cuda()
    with pma.Context(0) as ctx:  # its own type numbering: the reference's takes a search a pore
        labels, table = pma.assign_pore_and_throat_ids(ctx, torch.from_numpy(mask).cuda(), d, d, pma.D3Q7)
    labels = labels.cpu().numpy().view(np.uint32)
    pores, throats = table.rows()
    by_radius = sides[::-1]  # pores are numbered by decreasing radius
    assert len(pores) == count + others
    assert [(p[3], p[1], p[2]) for p in pores[:count]] == by_radius
    ids = [p[0] for p in pores]
    assert [labels[v] for v in by_radius] == ids[:count]
    corridor = labels[1, 1][r2[1, 1] == 1]
    assert len(throats) == 1 and (corridor == throats[0][0]).all() and throats[0][1] == corridor.size
    assert list(throats[0][2]) == [ids[1], ids[0]] + ids[2:count]
    assert all(p[6] == 1 for p in pores)
