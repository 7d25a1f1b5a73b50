"""Empty-pore removal of tables made for it (EmptyPoresRemover.cpp:126-244): lists that lose all, all but one or
some pores, lists that become equal, in any order of ids and list elements, on one thread and (from 2^15
types on) several. Against the rules written out in Python."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _remove(pores, throats, labels):
    empty = {p[0] for p in pores if p[6] == 0}
    to, groups = {}, {}
    for tid, vol, ids in sorted(throats):
        ids = tuple(sorted(i for i in ids if i not in empty))
        if len(ids) < 2:
            if ids:
                to[tid] = ids[0]
            continue
        groups.setdefault(ids, []).append((tid, vol))
    out = []
    for ids, types in groups.items():
        out.append((types[-1][0], types[-1][1], ids))
        to.update({tid: types[-1][0] for tid, _ in types[:-1]})
    return [p for p in pores if p[6]], sorted(out), np.array([to.get(v, v) for v in labels.ravel().tolist()]).reshape(labels.shape)


@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("types", [0, 1, 15, 16, 300, 33000])
def test_removal(ctx, types, ordered):
    import torch
    import porousmediaanalysis_gb300 as pma
    rng = np.random.default_rng(types)
    ids = [i for i in range(127, 127 + 60) if i % 255]
    pores = [(i, 0, 0, 0, 1, 0, int(rng.integers(0, 3))) for i in ids]
    top = 2 ** 32 - 2
    tids = [top - k for k in range(types)][::-1]
    if not ordered:
        tids = [int(v) for v in rng.permutation(tids)]
    throats = [(tid, int(rng.integers(1, 9)), tuple(int(v) for v in rng.choice(ids, rng.integers(2, 6), replace=False)))
               for tid in tids]
    labels = rng.choice(np.array(ids + tids, np.int64), (3, 20, 50))
    dev = torch.from_numpy(labels.astype(np.uint32).view(np.int32)).cuda()
    table = pma.Table.from_rows(pores, throats)
    pma.remove_empty_pores(ctx, table, dev)
    want_pores, want_throats, want_labels = _remove(pores, throats, labels)
    assert table.rows() == (want_pores, want_throats)
    assert (dev.cpu().numpy().view(np.uint32) == want_labels).all()
