"""Long WFA pairs that the CTA kernels leave to clusters of CTAs once most SMs have run out of
pairs (wfa_tile.cuh): when that happens, and that the results stay the oracle's."""
import time

import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P
from phraya_b200 import casegen as G

pytestmark = pytest.mark.gpu

DNA, AA = b"ACGT", b"ACDEFGHIKLMNPQRSTVWY"
ENGINES = [(A.ENGINE_WFA_LINEAR, (2, 4, 1)), (A.ENGINE_WFA_AFFINE, (2, 4, 1)), (A.ENGINE_WFA_AFFINE, (4, 6, 2))]
engines = pytest.mark.parametrize("engine,costs", ENGINES, ids=["linear", "2-4-1", "4-6-2"])
RESUME = {A.ENGINE_WFA_LINEAR: "wfa_linear_resume", A.ENGINE_WFA_AFFINE: "wfa_affine_resume"}


def divergent(rng, n, length, alphabet=DNA, rate=0.15):
    """Pairs of about `length` symbols whose score passes the step at which a pair is left."""
    pairs = []
    for i in range(n):
        q = rng.choice(np.frombuffer(alphabet, np.uint8), length + 17 * i)
        t = q.copy()
        hit = rng.random(t.size) < rate
        t[hit] = rng.choice(np.frombuffer(alphabet, np.uint8), int(hit.sum()))
        t = np.delete(t, np.flatnonzero(rng.random(t.size) < rate / 4))
        pairs.append((q.tobytes(), t.tobytes()))
    return pairs


def run(eng, engine, costs, pairs):
    """The pairs' results, the oracle's, and how often each kernel ran."""
    packed = O.PackedPairs(pairs)
    eng._lib.phr_ctx_reset_timing(eng.handle)
    eng.set_timing(True)
    ga, gc = eng.extend_packed(engine, packed, P.AffineCosts(*costs))
    ran = {k: v[0] for k, v in eng.kernel_times().items()}
    eng.set_timing(False)
    oa, oc = O.extend_packed(engine, packed, costs)
    if engine == A.ENGINE_WFA_AFFINE:
        assert np.array_equal(ga["affine_score"], oa["affine_score"])
    return P.unpack(ga, gc), P.unpack(oa, oc), ran


@engines
def test_resident_blocks_do_not_decide(engine, costs):
    """"max_blocks_per_sm" is about resident blocks only; "wfa_cluster_max" 1 keeps every pair on
    its CTA."""
    pairs = divergent(np.random.default_rng(61), 3, 3000)
    with P.Engine(0) as eng:
        for blocks in (4, 3, 2, 1):
            eng.set_tune("max_blocks_per_sm", blocks)
            got, want, ran = run(eng, engine, costs, pairs)
            assert got == want and ran.get(RESUME[engine], 0) == 1, (blocks, ran)
        eng.set_tune("wfa_cluster_max", 1)
        got, want, ran = run(eng, engine, costs, pairs)
        assert got == want and RESUME[engine] not in ran


@pytest.mark.parametrize("streams,short_lane,blocks", [(1, -1, 4), (2, -1, 4), (2, 1, 4), (2, 1, 2)])
@pytest.mark.parametrize("clusters", [16, 1])
def test_server_workers(streams, short_lane, blocks, clusters, tmp_path, monkeypatch):
    """A server's workers follow its context's setting, whatever the lanes and blocks per SM."""
    trace = tmp_path / "trace.txt"
    monkeypatch.setenv("PHRAYA_SERVER_TRACE", str(trace))
    ref = G.repeat_reference(2_000_000, 20, seed=62)
    packed, _, _ = G.long_reads(ref, 60, seed=63, error=0.12)
    reads = [bytes(packed.seq[o:o + n]) for o, n in zip(packed.off.tolist(), packed.len.tolist())]
    with P.Engine(0) as eng:
        eng.set_tune("wfa_cluster_max", clusters)
        idx = eng.index(ref)
        batched, _ = eng.align_reads(idx, reads, A.BALANCED)
        srv = eng.server(idx, strategy=A.BALANCED, max_batch_reads=64, max_wait_us=20000, n_streams=streams,
                         short_lane=short_lane, long_blocks_per_sm=blocks)
        ids = srv.submit_many(reads)
        got, until = {}, time.time() + 120
        while len(got) < len(reads) and time.time() < until:
            for rid, res, _ in srv.poll(4096, wait_us=20000):
                got[rid] = res
        srv.close()
    assert [got[i] for i in ids] == batched
    assert ("wfa_linear_resume" in trace.read_text()) == (clusters > 1)


@engines
@pytest.mark.parametrize("alphabet", [DNA, AA], ids=["2bit", "bytes"])
@pytest.mark.parametrize("clusters,n", [(16, 4), (16, 14), (16, 30), (8, 4), (4, 4)])
def test_cluster_sizes(engine, costs, alphabet, clusters, n):
    """16, 8 and 4 CTAs a pair: by the number of pairs left (148 SMs) and by the setting, which a
    device without room for the larger ones has too."""
    pairs = divergent(np.random.default_rng(64), n, 2200, alphabet)
    with P.Engine(0) as eng:
        eng.set_tune("wfa_cluster_max", clusters)
        got, want, ran = run(eng, engine, costs, pairs)
    assert got == want and ran.get(RESUME[engine], 0) == 1, ran


@engines
@pytest.mark.parametrize("clusters", [16, 4, 1])
def test_records_run_out(engine, costs, clusters):
    """A workspace that the pair's records outgrow: on its cluster, after the hand-over, or on its
    one CTA. Either way a redo pass follows and fits."""
    pairs = divergent(np.random.default_rng(65), 1, 3000)
    # (record chunks double from 64 KiB: a CTA's first three end at 448, its first seven at 8,128)
    budget = 8000 if engine == A.ENGINE_WFA_AFFINE else 550 if clusters > 1 else 430
    with P.Engine(0, workspace_bytes=budget << 10) as eng:
        eng.set_tune("wfa_cluster_max", clusters)
        got, want, ran = run(eng, engine, costs, pairs)
        assert eng.counter("scratch_oom_pairs") == 0
    # (one pair: were it redone before the hand-over, no cluster would have run)
    assert got == want and ran.get(RESUME[engine], 0) == (1 if clusters > 1 else 0) and ran["redo_tasks"] >= 1, ran


@engines
def test_one_warp_records_run_out(engine, costs):
    """Six unrelated pairs, a warp each, in a workspace for the records of about one."""
    rng = np.random.default_rng(66)
    pairs = [(rng.choice(np.frombuffer(DNA, np.uint8), 900).tobytes(), rng.choice(np.frombuffer(DNA, np.uint8), 950).tobytes())
             for _ in range(6)]
    with P.Engine(0, workspace_bytes=10 << 20 if engine == A.ENGINE_WFA_AFFINE else 512 << 10) as eng:
        got, want, ran = run(eng, engine, costs, pairs)
        assert eng.counter("scratch_oom_pairs") == 0
    assert got == want and ran["redo_tasks"] >= 1, ran
