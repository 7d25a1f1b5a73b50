"""Pass Y in blocks of eight rows and stretches of 32: row counts and lengths around both, and rows so long
that a block holds four, two and one of them. Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 31), (1, 7, 32), (3, 3, 33), (2, 8, 257), (9, 1, 1025), (1, 3, 5000), (2, 5, 8001),
                                   (1, 2, 17000), (1, 3, 33000)])
@pytest.mark.parametrize("fraction", [0.002, 0.2])
def test_edt_rows(ctx, oracle_mod, shape, fraction):
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = (np.random.default_rng(9).random(shape) < fraction).astype(np.uint8)
    vol[:, :, ::997] = 1
    want, most, hist = oracle_mod.edt(vol)
    got, got_most, got_hist = pma.compute_euclidean_distances(ctx, torch.from_numpy(vol).cuda(), hist_cap=most + 1)
    assert (got.cpu().numpy().view(np.uint32) == want).all() and got_most == most
    assert list(got_hist) == [int(v) for v in hist[: most + 1]]
