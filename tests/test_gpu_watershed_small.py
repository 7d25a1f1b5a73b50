"""Watershed floods whose buckets and generations straddle the sizes at which it changes form: one
block (up to 64 nodes), the cluster (2048), the whole grid; buckets sorted by counting (128 entries),
by radix passes in shared memory (8192) and by the device-wide sort. Everything bit-exact against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _open(shape):
    """No solid at all: one pore, frontiers that grow and shrink over the whole box."""
    return np.zeros(shape, np.uint8)


def _specks(shape, fraction, seed):
    """Single solid voxels: many pores, few radii (large buckets), many shared voxels."""
    return (np.random.default_rng(seed).random(shape) < fraction).astype(np.uint8)


VOLUMES = {
    "line": lambda: _open((1, 5, 300)),
    "plane": lambda: _open((1, 70, 90)),
    "box": lambda: _open((31, 33, 37)),
    "specks_sparse": lambda: _specks((40, 44, 48), 0.002, 3),
    "specks": lambda: _specks((48, 52, 64), 0.02, 5),
    "specks_dense": lambda: _specks((36, 30, 41), 0.15, 7),
}


@pytest.mark.parametrize("d3q7", [False, True])
@pytest.mark.parametrize("name", list(VOLUMES))
def test_watershed_forms(ctx, oracle_mod, name, d3q7):
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = VOLUMES[name]()
    o = oracle_mod.full(vol, d3q7, geodesic_too=False)
    stencil = pma.D3Q7 if d3q7 else pma.D3Q27
    solid = torch.from_numpy(vol).cuda()
    edt2, mx, _ = pma.compute_euclidean_distances(ctx, solid)
    crad2, _, _, _, mask, _ = pma.set_containing_balls(ctx, edt2, mx)
    labels, table = pma.assign_pore_and_throat_ids(ctx, mask, edt2, crad2, stencil)
    pma.remove_empty_pores(ctx, table, labels)
    ws, ws_table = pma.assign_watershed_ids(ctx, table, crad2, mx, stencil)
    assert (ws.cpu().numpy().view(np.uint32) == o["pores"].labels_ws).all()
    assert ws_table.rows() == (o["pores"].pores_ws, o["pores"].throats_ws)
