"""Fitting-mode Myers with a lane per pair (batches of at least 16,384 pairs) against the
oracle: block counts 1..9 (the last takes the group kernel), targets that run on or not,
abandoned searches, and the smaller batch that keeps the group kernel."""
import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P

pytestmark = pytest.mark.gpu


def fit_pairs(n, seed):
    rng = np.random.default_rng(seed)
    base = rng.choice(np.frombuffer(b"ACGT", np.uint8), 4_000_000)
    pairs = []
    for i in range(n):
        m = int(rng.choice([1, 20, 63, 64, 65, 100, 127, 128, 129, 150, 200, 256, 300, 449, 512, 513]))
        if m > 256 and i % 7:
            m = 150
        s = int(rng.integers(0, base.size - 3 * m - 64))
        q = base[s:s + m].copy()
        for p in rng.integers(0, m, int(rng.integers(0, m // 12 + 1))):
            q[p] = b"ACGT"[int(rng.integers(4))]
        if i % 5 == 1 and m > 10:
            q = np.delete(q, slice(m // 2, m // 2 + int(rng.integers(1, 6))))
        if i % 13 == 2:                       # unrelated window: the search is abandoned
            s = int(rng.integers(0, base.size - 3 * m - 64))
        more = [0, m // 3, m // 2 + 10, m // 2 + 11, m][i % 5]
        pairs.append((q.tobytes(), base[s:s + m + more].tobytes()))
    return pairs


@pytest.mark.parametrize("n", [16383, 16384, 16401])
def test_fit_lanes(n):
    packed = O.PackedPairs(fit_pairs(n, n))
    with P.Engine(0) as eng:
        eng.set_timing(True)
        ga, gc = eng.extend_packed(A.ENGINE_MYERS_FIT, packed)
        assert ("myers_lane" in eng.kernel_times()) == (n >= 16384)
    oa, oc = O.extend_packed(A.ENGINE_MYERS_FIT, packed, (2, 4, 1))
    for field in ("status", "edit_distance", "query_start", "query_end", "target_start", "target_end", "cigar_len"):
        bad = np.flatnonzero(ga[field] != oa[field])
        assert bad.size == 0, (field, bad[:5], ga[bad[:1]], oa[bad[:1]])
    assert bytes(gc) == bytes(oc[: len(gc)])
