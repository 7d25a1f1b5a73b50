"""Geodesics on extents around the bricks of the sweep (32 x 8 x 8 voxels, one-voxel halo): one brick,
remainders on every axis, single rows and slices, many restarts; bit-exact against the oracle."""
import numpy as np
import pytest

from cases import many_pockets

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 1, 70), (1, 70, 1), (70, 1, 1), (1, 17, 65), (8, 8, 32), (9, 9, 33), (7, 16, 31), (17, 8, 64), (25, 23, 97)]


@pytest.mark.parametrize("d3q7", [False, True])
@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("shape", SHAPES + ["pockets"])
def test_geodesic_bricks(ctx, oracle_mod, shape, fp64, d3q7):
    import torch
    import porousmediaanalysis_gb300 as pma
    volumes = [many_pockets(shape=(40, 44, 70), count=150)] if shape == "pockets" else \
        [(np.random.default_rng(5).random(shape) < f).astype(np.uint8) for f in (0.0, 0.3, 0.6)]
    for vol in volumes:
        d, c, rows = oracle_mod.geodesic(vol, d3q7, fp64)
        dist, cav, got = pma.compute_shortest_path_distances(ctx, torch.from_numpy(vol).cuda(), pma.D3Q7 if d3q7 else pma.D3Q27, fp64=fp64)
        bits = np.uint64 if fp64 else np.uint32
        assert (dist.cpu().numpy().view(bits) == d.view(bits)).all()
        assert (cav.cpu().numpy().view(np.uint32) == c).all()
        assert [r[:4] + r[5:] for r in got] == [r[:4] + r[5:] for r in rows]
