"""EDT of volumes whose slices straddle the block sizes of pass Z (128 threads up to 128 slices, 64 slices a round)
and whose smallest extent decides how many bins its shared histogram has. Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fraction", [0.0, 0.002, 0.2])
@pytest.mark.parametrize("shape", [(sz, 21, 37) for sz in (1, 2, 3, 7, 8, 9, 63, 64, 65, 127, 128, 129, 300)] +
                         [(70, 92, 16), (92, 93, 95), (95, 91, 94), (128, 3, 200)])
def test_edt_slices(ctx, oracle_mod, shape, fraction):
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = (np.random.default_rng(7).random(shape) < fraction).astype(np.uint8)
    want, most, hist = oracle_mod.edt(vol)
    edt2, got_most, got_hist = pma.compute_euclidean_distances(ctx, torch.from_numpy(vol).cuda(), hist_cap=most + 1)
    assert (edt2.cpu().numpy().view(np.uint32) == want).all() and got_most == most
    assert (np.array(got_hist, np.uint64) == hist).all()
