"""Plateau edges on extents around the tiles of the pair kernel (4 x 8 x 32 voxels): single rows, both ends of
a warp's row, short last tiles. Initial propagation bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 5), (1, 1, 33), (4, 8, 32), (5, 9, 33), (3, 7, 31), (8, 16, 64), (9, 17, 97), (13, 2, 128)]


@pytest.mark.parametrize("d3q7", [False, True])
@pytest.mark.parametrize("fraction", [0.01, 0.1, 0.5])
@pytest.mark.parametrize("shape", SHAPES)
def test_plateau_edges(ctx, oracle_mod, shape, fraction, d3q7):
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = (np.random.default_rng(5).random(shape) < fraction).astype(np.uint8)
    vol[0, 0, 0] = 1  # never all void
    o = oracle_mod.full(vol, d3q7=d3q7, geodesic_too=False)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()
    labels, table = pma.assign_pore_and_throat_ids(ctx, torch.from_numpy(o["mask"]).cuda(), up(o["edt2"]), up(o["crad2"]),
                                                   pma.D3Q7 if d3q7 else pma.D3Q27)
    assert table.rows() == (o["pores"].pores0, o["pores"].throats0)
    assert (labels.cpu().numpy().view(np.uint32) == o["pores"].labels_initial).all()
