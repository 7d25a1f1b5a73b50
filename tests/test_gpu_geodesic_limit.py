"""The bucket limit of the geodesic flood is looked at after every 32 buckets: a flood of 42 buckets is
past a limit of 31 then, and not past one of 32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit,refused", [(1, True), (31, True), (32, False), (33, False)])
@pytest.mark.parametrize("fp64", [False, True])
def test_bucket_limit(pma_lib, oracle_mod, limit, refused, fp64):
    import torch
    import porousmediaanalysis_gb300 as pma
    vol = np.zeros((48, 48, 48), np.uint8)  # distances up to 24 sqrt(3) = 41.6
    want, cavity, _ = oracle_mod.geodesic(vol, False, fp64)
    assert 32 < want.max() < 63
    with pma.Context(0) as ctx:
        ctx.set_limits(geodesic_buckets=limit)
        call = lambda: pma.compute_shortest_path_distances(ctx, torch.from_numpy(vol).cuda(), fp64=fp64)
        if refused:
            with pytest.raises(pma.PmaError) as e:
                call()
            assert e.value.status == 5 and "bucket sweep" in str(e.value)
        else:
            dist, cav, _ = call()
            assert (dist.cpu().numpy() == want).all()
            assert (cav.cpu().numpy().view(np.uint32) == cavity).all()
