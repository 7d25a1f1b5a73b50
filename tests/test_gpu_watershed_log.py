"""Watershed floods through every state of the extension log and of the lists of claims that
ws_small keeps: launches that start with the log just below the half at which it is emptied (their
own blocks' reservations cross it), floods that stop for a full log, logs that overflow inside a
launch, and generations with more claims of shallower voxels than a block's list holds, in one
block and in the cluster. The counters of the timing report show that each state was met.
Everything bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sheets():
    """24 sheets of 9600 voxels, each a depth of its own, flooded one after the other from two seeds:
    each sheet's bucket is too large for ws_small, which is launched anew behind it and reserves
    8192 log entries before it looks at the log, of which 2^15 + n / 16 = 47168 are the half."""
    crad = np.empty((64, 150, 24), np.uint32)
    crad[...] = 100 - np.arange(24, dtype=np.uint32)
    return crad, [(3, 0, 5), (140, 0, 60)], {"ws.small_launches": 24, "ws.log_entries": 4}


def _blocks(shape, radii):
    """A seed in every 3 x 3 x 3 voxels, at the deepest depth; radii 1 to `radii` between them."""
    crad = np.random.default_rng(radii).integers(1, radii + 1, shape).astype(np.uint32)
    seeds = [(x, y, z) for z in range(1, shape[0], 3) for x in range(1, shape[1], 3) for y in range(1, shape[2], 3)]
    for x, y, z in seeds:
        crad[z, x, y] = 50
    return crad, seeds


def _one_block():
    crad, seeds = _blocks((12, 12, 12), 7)
    assert len(seeds) == 64  # one generation of one block, 26 claims a node: 1664, the list holds 1024
    return crad, seeds, {}


def _cluster():
    crad, seeds = _blocks((36, 36, 39), 40)
    assert 64 < len(seeds) <= 2048  # 117 nodes a block, 1200 entries a depth: ten to a voxel go to the log
    return crad, seeds, {"ws.log_stops": 1}


def _grid():
    crad, seeds = _blocks((60, 66, 72), 9)
    assert len(seeds) > 8192  # the device-wide sort, then generations of the whole grid that overflow the log
    return crad, seeds, {"ws.log_overflow": 1}


VOLUMES = {"sheets": _sheets, "one_block": _one_block, "cluster": _cluster, "grid": _grid}


@pytest.mark.parametrize("d3q7", [False, True])
@pytest.mark.parametrize("name", list(VOLUMES))
def test_watershed_log(ctx, oracle_mod, name, d3q7):
    import torch
    import porousmediaanalysis_gb300 as pma
    crad, seeds, met = VOLUMES[name]()
    pores = [(127 + i, x, y, z, int(crad[z, x, y]), 0, 1) for i, (x, y, z) in enumerate(seeds)]
    most = int(crad.max())
    want, want_pores, want_throats = oracle_mod.watershed(pores, crad, most, d3q7)
    ctx.timing_report()
    ctx.set_timing(True)
    try:
        ws, table = pma.assign_watershed_ids(ctx, pma.Table.from_rows(pores), torch.from_numpy(crad.view(np.int32)).cuda(), most,
                                             pma.D3Q7 if d3q7 else pma.D3Q27)
        report = ctx.timing_report()
    finally:
        ctx.set_timing(False)
    assert (ws.cpu().numpy().view(np.uint32) == want).all()
    assert table.rows() == (want_pores, want_throats)
    for counter, times in met.items():  # [sum, increments]
        assert d3q7 or report["count." + counter][1] >= times
