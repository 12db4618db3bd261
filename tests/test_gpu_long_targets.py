"""Queries of a few hundred to a few thousand symbols against targets of millions, where the
bounds of the register tiles' value words lie (wfa_tile.cu, wfa_affine_tile.cu): the search
ends near the target's start, so the result is that of the target cut to three queries."""
import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P

pytestmark = pytest.mark.gpu

DNA, AA = b"ACGT", b"ACDEFGHIKLMNPQRSTVWY"
TARGETS = [(1 << 21) - 64, (1 << 21) + 64, 3_000_000, (1 << 22) + 5]


def queries(t):
    """Queries off the target's start with gaps of a few target symbols in their path, one of
    them by both kinds of gap and mismatches."""
    q = [t[:1500] + t[1503:3000], t[:40] + t[41:900] + t[908:2500], t[:1400] + t[1402:1700] + t[1704:1800]]
    mixed = bytearray(t[:700] + t[705:1300] + t[1290:2400])
    for i in (90, 800, 1900):
        mixed[i] = t[0] if mixed[i] != t[0] else t[1] if t[1] != t[0] else mixed[i] ^ 6
    return q + [bytes(mixed)]


@pytest.mark.parametrize("engine,costs", [(A.ENGINE_WFA_AFFINE, (2, 4, 1)), (A.ENGINE_WFA_AFFINE, (4, 6, 2)),
                                          (A.ENGINE_WFA_LINEAR, (2, 4, 1))], ids=["2-4-1", "4-6-2", "linear"])
@pytest.mark.parametrize("alphabet", [DNA, AA], ids=["2bit", "bytes"])
@pytest.mark.parametrize("big_min", [4096, 1 << 30], ids=["cta", "warp"])
def test_long_targets(engine, costs, alphabet, big_min):
    rng = np.random.default_rng(91)
    base = rng.choice(np.frombuffer(alphabet, np.uint8), max(TARGETS)).tobytes()
    whole = [(q, base[:n]) for n in TARGETS for q in queries(base)]
    cut = [(q, base[: 3 * len(q)]) for q in queries(base)] * len(TARGETS)
    with P.Engine(0) as eng:
        eng.set_tune("wfa_big_min", big_min)
        got = [P.unpack(a, c) + [list(a["affine_score"])]
               for a, c in (eng.extend_packed(engine, O.PackedPairs(p), P.AffineCosts(*costs)) for p in (whole, cut))]
    assert got[0] == got[1]
    # (the oracle keeps full-width wavefronts: the pair of the fewest score steps)
    oa, oc = O.extend_packed(engine, O.PackedPairs([whole[len(cut) // 2]]), costs)
    assert [got[0][len(cut) // 2]] == P.unpack(oa, oc)


@pytest.mark.parametrize("n", [(1 << 22) - 1, 1 << 22, (1 << 22) + 333])
@pytest.mark.parametrize("company", [0, 1500], ids=["alone", "among_short"])
def test_long_linear_queries(n, company):
    """Near-identical linear pairs on both sides of the register tiles' longest query, both end
    rules and symbol modes, alone and in a batch of short pairs, in a small workspace."""
    rng = np.random.default_rng(92)
    base = rng.choice(np.frombuffer(DNA, np.uint8), 2 * n).tobytes()
    q = base[:n]
    near = q[:70_000] + q[70_002:2_000_000] + (b"C" if q[2_000_000:2_000_001] != b"C" else b"G") + q[2_000_001:] + b"ACG"
    window = near + base[n: n + n // 2 + 20]
    pairs = [(q, near), (q, window), (q[:100_000] + b"N" + q[100_001:], near)]
    for _ in range(company):
        s = int(rng.integers(0, n - 300))
        pairs.append((base[s:s + 150], base[s:s + 70] + base[s + 72:s + 160]))
    packed = O.PackedPairs(pairs)
    with P.Engine(0, workspace_bytes=256 << 20) as eng:
        eng.set_timing(True)
        ga, gc = eng.extend_packed(A.ENGINE_WFA_LINEAR, packed)
        ran = eng.kernel_times()
    assert ("wfa_linear_long" in ran) == (n >= 1 << 22)
    oa, oc = O.extend_packed(A.ENGINE_WFA_LINEAR, packed, (2, 4, 1))
    assert P.unpack(ga, gc) == P.unpack(oa, oc)
