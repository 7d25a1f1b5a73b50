"""EDT on the extents at which its passes change form: groups of 8 outputs, rows of 32 and 256, tiles of
16, bit words of 32, four columns a thread or one (row length, alignment), the tile's two pitches, and
extents whose squares leave 32 bits in a sum (general kernels). Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [  # (SZ, SX, SY)
    (1, 1, 1), (1, 1, 9), (2, 33, 8), (9, 31, 7), (8, 32, 16), (17, 64, 255), (16, 65, 256), (31, 20, 257),
    (33, 96, 260), (255, 9, 33), (257, 10, 20), (3113, 5, 3), (3200, 4, 20), (2, 5, 3000), (3, 2600, 12),
    (2, 43700, 3), (2, 30000, 4),
]


@pytest.mark.parametrize("fraction", [0.0, 0.0005, 0.02, 0.3])
@pytest.mark.parametrize("shape", SHAPES)
def test_edt_forms(ctx, oracle_mod, shape, fraction):
    import torch
    import porousmediaanalysis_gb300 as pma
    if shape[1] > 43690 and fraction == 0.0:
        pytest.skip("the distance to the virtual walls has no square in 32 bits: there is no right answer")
    vol = (np.random.default_rng(sum(shape)).random(shape) < fraction).astype(np.uint8) * 200
    e, most, hist = oracle_mod.edt(vol)
    flat = torch.zeros(vol.size + 1, dtype=torch.uint8, device="cuda")
    for offset in (0, 1):  # aligned and misaligned input
        solid = flat[offset:offset + vol.size].view(shape)
        solid.copy_(torch.from_numpy(vol))
        edt2, mx, h = pma.compute_euclidean_distances(ctx, solid, hist_cap=6000)
        assert mx == most and (edt2.cpu().numpy().view(np.uint32) == e).all()
        want = np.zeros(len(h), np.int64)
        k = min(len(h), len(hist))
        want[:k] = hist[:k]
        assert (np.array(h) == want).all()
