"""The order of the maximum balls is std::sort's exact permutation: isolated voxels, all of one
containing radius and each its own pore, so that the table's seeds are the sorted balls. Sizes around what
one leaf, one block and one chunk of a partition hold; keys with many ties, in order, and in the order
in which std::sort goes to its depth limit (McIlroy's adversary, "A killer adversary for quicksort", 1999)."""
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <vector>
// stdin: keys; stdout: the indices as std::sort leaves them, by descending key. With an
// argument n: n adversary keys instead.
int main(int argc, char** argv) {
    if (argc > 1) {
        const size_t n = std::atoi(argv[1]);
        std::vector<uint32_t> key(n, 0), idx(n);  // 0: not decided yet, and lower than all that are
        std::iota(idx.begin(), idx.end(), 0u);
        uint32_t next = n + 1, candidate = 0;
        std::sort(idx.begin(), idx.end(), [&](uint32_t x, uint32_t y) {
            if (!key[x] && !key[y]) key[x == candidate ? x : y] = next--;
            if (!key[x]) candidate = x;
            else if (!key[y]) candidate = y;
            return key[x] > key[y];
        });
        for (auto& k : key) k = k ? k : 1;
        std::fwrite(key.data(), 4, n, stdout);
        return 0;
    }
    std::vector<uint64_t> v;
    for (uint32_t k; std::fread(&k, 4, 1, stdin) == 1;) v.push_back(uint64_t(k) << 32 | v.size());
    std::sort(v.begin(), v.end(), [](uint64_t a, uint64_t b) { return a >> 32 > b >> 32; });
    for (uint64_t x : v) {
        const uint32_t i = static_cast<uint32_t>(x);
        std::fwrite(&i, 4, 1, stdout);
    }
}
"""


@pytest.fixture(scope="module")
def std_sort(tmp_path_factory):
    d = tmp_path_factory.mktemp("std_sort")
    (d / "s.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", str(d / "s.cpp"), "-o", str(d / "s")], check=True)

    def run(keys=None, adversary=None):
        args = [str(d / "s")] + ([str(adversary)] if adversary else [])
        out = subprocess.run(args, input=None if keys is None else keys.tobytes(), capture_output=True, check=True)
        return np.frombuffer(out.stdout, np.uint32)
    return run


@pytest.mark.parametrize("kind", ["equal", "ties", "distinct", "rising", "falling", "adversary"])
@pytest.mark.parametrize("n", [1, 2, 16, 17, 35, 2049, 8192, 8193, 20000, 150001])
def test_ball_order(ctx, std_sort, n, kind):
    import torch
    import porousmediaanalysis_gb300 as pma
    rng = np.random.default_rng(n)
    if kind == "adversary":
        if n not in (35, 2049, 20000):
            pytest.skip("three sizes are enough: one warp, one block, the grid")
        keys = std_sort(adversary=n)
    else:
        distinct = {"equal": 1, "ties": 5}.get(kind, 1 << 20)
        keys = rng.integers(1, distinct + 1, n).astype(np.uint32)
        if kind in ("rising", "falling"):
            keys = np.sort(keys)[::1 if kind == "rising" else -1].copy()
    r2 = np.zeros((1, 1, 2 * n), np.uint32)
    r2[0, 0, ::2] = keys
    outer = torch.from_numpy((r2 != 0)).cuda()
    table = pma.assign_pore_and_throat_ids(ctx, outer.to(torch.uint8) * 255, torch.from_numpy(r2.view(np.int32)).cuda(),
                                           outer.to(torch.int32), pma.D3Q27)[1]
    pores, throats = table.rows()
    order = std_sort(keys)
    assert throats == [] and len(pores) == n
    assert np.array_equal([p[2] for p in pores], 2 * order.astype(np.int64))
    assert np.array_equal([p[4] for p in pores], keys[order])
