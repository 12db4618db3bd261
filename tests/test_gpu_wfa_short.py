"""Short gap-affine and linear pairs, wavefronts in one warp's registers, against the oracle where the
path can go wrong: bands that end at, cross and leave 32, 64 and 128 diagonals, both end
rules, gaps at either sequence's end, matches longer than a word, lengths around words."""
import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P

pytestmark = pytest.mark.gpu

BASES = b"ACGT"


def rand(rng, n):
    return bytes(rng.choice(list(BASES), n).tolist())


def mutate(rng, s, rate):
    out = bytearray()
    for c in s:
        x = rng.random()
        if x < rate * 0.6:
            out.append(BASES[int(rng.integers(4))])
        elif x < rate * 0.8:
            out += rand(rng, int(rng.integers(1, 4))) + bytes([c])
        elif x >= rate:
            out.append(c)
    return bytes(out) or b"A"


def pairs_of(rng):
    pairs = []
    for n in (1, 2, 15, 16, 17, 31, 32, 33, 48, 100, 255, 256, 257, 480):
        q = rand(rng, n)
        pairs += [(q, q), (q, q[: n // 2] or q), (q, q + rand(rng, 3)), (rand(rng, 2) + q, q), (q, rand(rng, n)),
                  (q, mutate(rng, q, 0.05) + rand(rng, n // 2 + 11)), (q, rand(rng, n // 2 + 11) + mutate(rng, q, 0.05))]
        pairs += [(q, mutate(rng, q, r)) for r in (0.01, 0.05, 0.1, 0.2, 0.4)]
    for gap in (1, 14, 15, 16, 17, 30, 31, 32, 33, 62, 63, 64, 65, 127, 128, 129):  # the path follows the band's rim
        core = rand(rng, 60)
        pairs += [(core + rand(rng, gap) + core, core + core), (core + core, core + rand(rng, gap) + core),
                  (b"A" * (gap + 3), b"C" * (gap + 3)), (b"A" * gap, core)]
    return pairs


ENGINES = [(A.ENGINE_WFA_AFFINE, c) for c in ((2, 4, 1), (4, 6, 2), (6, 12, 3), (4, 8, 2), (1, 3, 1))]


@pytest.mark.parametrize("engine,costs", ENGINES + [(A.ENGINE_WFA_LINEAR, (2, 4, 1))])
@pytest.mark.parametrize("copies", [1, 40, 540])
def test_short(engine, costs, copies):
    """Batches of a few hundred pairs, of more than the small-batch limit, and of enough for
    the kernel for short pairs alone, which leaves the wide ones to the general one."""
    rng = np.random.default_rng(71)
    packed = O.PackedPairs(pairs_of(rng) * copies)
    oa, oc = O.extend_packed(engine, O.PackedPairs(pairs_of(np.random.default_rng(71))), costs)
    want = P.unpack(oa, oc) * copies
    with P.Engine(0) as eng:
        ga, gc = eng.extend_packed(engine, packed, P.AffineCosts(*costs))
    got = P.unpack(ga, gc)
    bad = [i for i in range(packed.n) if got[i] != want[i]]
    assert not bad, (len(bad), got[bad[0]], want[bad[0]])
    if engine == A.ENGINE_WFA_AFFINE:
        assert np.array_equal(ga["affine_score"], np.tile(oa["affine_score"], copies))
