"""Candidate lists gathered by a warp per sub-block and by a block of four
warps: a whole structure (many sub-blocks), slices of its bricks down to one
(few), and a spacing whose lists fill several rounds of the lanes, run twice
so that the second run takes the first one's list sizes.  Ids, orders and
blockers equal the oracle's, so no tolerance applies."""
import numpy as np
import pytest

import oracle as O
from helpers import arrangement_from_oracle, lattice_from_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spacing,brick", [(1500, 0.25, 10), (1500, 0.8, 10), (700, 1.3, 16), (5, 0.2, 8)])
def test_lists_equal_oracle(n, spacing, brick):
    from sesmesh_b200 import native, workloads
    spheres, probe = workloads.globule(3, n), 1.4
    eng = O.Engine(spheres, probe, spacing, brick)
    arr = arrangement_from_oracle(eng)
    arr["probe"] = probe
    dev = native.Device(0)
    res = native.Resident(dev, arr, lattice_from_oracle(eng, spacing, brick))
    res.classify()
    bricks = res.bricks()
    nb = len(bricks)
    want = {}
    for first, count in ((0, nb), (0, nb), (nb // 3, 1), (nb // 2, max(1, min(40, nb // 4)))):
        batch = native.Batch(res)
        batch.run(first, count)
        rec, ids = batch.records(), batch.ids()
        sampled = np.nonzero(rec[:, 0] == 0)[0]
        assert np.all(rec[sampled, 11] == 0)
        for j in sampled[::max(1, len(sampled) // 60)]:
            key = (first + int(j) // 8, int(j) % 8)
            if key not in want:
                want[key] = eng.gather(bricks[key[0]], key[1])
            got = batch.lists(rec[j], ids)
            assert got["n_inside"] == want[key]["n_inside"], key
            for name in ("near", "s", "s_off", "s_blk", "c", "c_off", "c_blk", "v"):
                assert np.array_equal(got[name], want[key][name]), (key, name)
