"""WFA in register tiles (wfa_tile.cu linear, wfa_affine_tile.cu gap-affine with both
specialised cost ratios) against the oracle where it can go wrong: bands that end at, cross and leave tile edges, both end rules, both symbol modes, paths
along the band's rim, sequences and frames that do not fit shared memory, and a scratch
pool that runs out."""
import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P

pytestmark = pytest.mark.gpu

DNA, AA = b"ACGT", b"ACDEFGHIKLMNPQRSTVWY"
ENGINES = [(A.ENGINE_WFA_LINEAR, (2, 4, 1)), (A.ENGINE_WFA_AFFINE, (2, 4, 1)), (A.ENGINE_WFA_AFFINE, (4, 6, 2)),
           (A.ENGINE_WFA_AFFINE, (6, 12, 3))]
engines = pytest.mark.parametrize("engine,costs", ENGINES, ids=["linear", "2-4-1", "4-6-2", "6-12-3"])


def check(eng, engine, costs, pairs):
    packed = O.PackedPairs(pairs)
    ga, gc = eng.extend_packed(engine, packed, P.AffineCosts(*costs))
    oa, oc = O.extend_packed(engine, packed, costs)
    got, want = P.unpack(ga, gc), P.unpack(oa, oc)
    bad = [i for i in range(packed.n) if got[i] != want[i]]
    assert not bad, (len(bad), bad[:5], got[bad[0]], want[bad[0]], pairs[bad[0]])
    if engine == A.ENGINE_WFA_AFFINE:
        assert np.array_equal(ga["affine_score"], oa["affine_score"])


def rand(rng, n, alphabet=DNA):
    return bytes(rng.choice(list(alphabet), n).tolist())


def mutate(rng, s, rate, alphabet=DNA):
    out = bytearray()
    for c in s:
        x = rng.random()
        if x < rate * 0.6:
            out.append(alphabet[int(rng.integers(len(alphabet)))])
        elif x < rate * 0.8:
            out += rand(rng, int(rng.integers(1, 4)), alphabet) + bytes([c])
        elif x < rate:
            pass
        else:
            out.append(c)
    return bytes(out)


def edge_pairs(rng, alphabet):
    """Similar, unrelated and rim pairs with lengths and scores around the tile sizes
    (8 scores, 240 kept diagonals of 256)."""
    pairs = []
    for n in (31, 64, 119, 120, 121, 127, 128, 239, 240, 241, 256, 257, 500):
        q = rand(rng, n, alphabet)
        pairs += [(q, q), (q, mutate(rng, q, 0.08, alphabet) or q), (q, rand(rng, n, alphabet)),
                  (q, q[: n // 2] or q), (q, rand(rng, 7, alphabet) + q),
                  (q, mutate(rng, q, 0.05, alphabet) + rand(rng, n, alphabet)),     # fitting: the target runs on
                  (q, rand(rng, 2 * n + 20, alphabet)), (q[:17], rand(rng, n, alphabet))]
    a, c = alphabet[:1], alphabet[1:2]
    for n in (7, 8, 9, 112, 120, 128, 240, 250):   # one gap of n: the path follows the band's rim
        core = rand(rng, 60, alphabet)
        pairs += [(core + a * n + core, core + core), (core + core, core + c * n + core), (a * (n + 30), c * (n + 30))]
    return pairs


@engines
@pytest.mark.parametrize("alphabet", [DNA, AA], ids=["2bit", "bytes"])
@pytest.mark.parametrize("tune", [{"wfa_big_min": 32, "wfa_big_smem": 16 << 10}, {"wfa_big_min": 32},
                                  {"wfa_big_min": 1 << 20, "wfa_long_min": 32}], ids=["cta16k", "cta", "warp"])
def test_tile_edges(alphabet, tune, engine, costs):
    """Every pair on one CTA (with and without room for its frames), or one warp."""
    rng = np.random.default_rng(41)
    pairs = edge_pairs(rng, alphabet)
    with P.Engine(0) as eng:
        for key, value in tune.items():
            eng.set_tune(key, value)
        check(eng, engine, costs, pairs)


@engines
@pytest.mark.parametrize("alphabet", [DNA, AA], ids=["2bit", "bytes"])
@pytest.mark.parametrize("big_min", [4096, 1 << 20], ids=["cta", "warp"])
def test_bands_beyond_shared_memory(alphabet, big_min, engine, costs):
    """Unrelated pairs: wavefronts of thousands of diagonals, frames in global memory."""
    rng = np.random.default_rng(42)
    pairs = [(rand(rng, n, alphabet), rand(rng, m, alphabet)) for n, m in ((3000, 3100), (2500, 2900), (2100, 2000))]
    q = rand(rng, 9000, alphabet)
    pairs += [(q, mutate(rng, q, 0.1, alphabet)), (q[:5000], mutate(rng, q, 0.03, alphabet))]
    with P.Engine(0) as eng:
        eng.set_tune("wfa_big_smem", 24 << 10)
        eng.set_tune("wfa_big_min", big_min)
        check(eng, engine, costs, pairs)


@engines
@pytest.mark.parametrize("budget", [1 << 20, 4 << 20])
def test_pool_runs_out(budget, engine, costs):
    """More records than the workspace holds at once: pairs are redone with their own
    scratch and give the same results."""
    rng = np.random.default_rng(43)
    q = [rand(rng, n) for n in (4000, 4100, 5000, 2300, 2050, 3000)]
    pairs = [(s, mutate(rng, s, 0.04)) for s in q] + [(rand(rng, 1500), rand(rng, 2600)) for _ in range(4)]
    if engine == A.ENGINE_WFA_AFFINE:   # 28 bytes a diagonal and 8 steps: the same pairs need more
        budget *= 32
    with P.Engine(0, workspace_bytes=budget) as eng:
        check(eng, engine, costs, pairs)
        assert eng.counter("scratch_oom_pairs") == 0
