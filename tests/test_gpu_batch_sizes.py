"""Batch sizes around the edges of the one-CTA batch preparation and tail (32 pairs packed by
it, 1,024 pairs prepared by it) and of the early tail (65,536 pairs), with byte pairs,
empty sequences and invalid seeds among them, against the oracle."""
import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P

pytestmark = pytest.mark.gpu


def mixed_pairs(n, seed):
    rng = np.random.default_rng(seed)
    pairs = []
    for i in range(n):
        m = int(rng.integers(1, 90))
        q = bytes(rng.choice(list(b"ACGT"), m).tolist())
        t = bytearray(q)
        for _ in range(int(rng.integers(0, 4))):
            t[int(rng.integers(0, len(t)))] = int(rng.choice(list(b"ACGT")))
        t += bytes(rng.choice(list(b"ACGT"), int(rng.integers(0, 60))).tolist())
        if i % 11 == 3:
            t[0] = ord("N")
        if i % 17 == 5:
            q = b""
        if i % 19 == 7:
            t = b""
        seed_pos = len(q) + 1 if i % 23 == 9 else min(i % 3, len(q), len(t))
        pairs.append((q, bytes(t), seed_pos, min(i % 3, len(t))))
    return pairs


@pytest.mark.parametrize("engine", [A.ENGINE_WFA_LINEAR, A.ENGINE_WFA_AFFINE, A.ENGINE_MYERS_FIT, A.ENGINE_MYERS_GLOBAL])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1024, 1025])
def test_batch_sizes(n, engine):
    pairs = mixed_pairs(n, 50 + n)
    with P.Engine(0) as eng:
        got = eng.extend(engine, pairs)
        assert got == O.extend(engine, pairs)
        assert eng.extend(engine, pairs[: n // 2]) == got[: n // 2]   # the same context, another size


@pytest.mark.parametrize("n", [65536, 65537])
def test_redo_after_the_early_tail(n):
    """Pairs that leave their first band (Myers) are redone after the text was laid out."""
    pairs = mixed_pairs(64, 7) * (n // 64) + mixed_pairs(n % 64, 8)
    far = (b"ACGT" * 300, b"TTGA" * 300)
    pairs[5] = pairs[n - 3] = far
    with P.Engine(0) as eng:
        eng.set_tune("myers_band_base", 0)
        ga, gc = eng.extend_packed(A.ENGINE_MYERS_GLOBAL, O.PackedPairs(pairs))
    oa, oc = O.extend_packed(A.ENGINE_MYERS_GLOBAL, O.PackedPairs(pairs), (2, 4, 1))
    for field in ("status", "edit_distance", "cigar_len", "cigar_off", "query_end", "target_end"):
        assert np.array_equal(ga[field], oa[field]), field
    assert bytes(gc) == bytes(oc[: len(gc)])
