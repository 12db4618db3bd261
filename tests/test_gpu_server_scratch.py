"""A server's workers hold the scratch they took at creation: batches of long reads do not make
it grow (allocating while serving stalls every worker on the device)."""
import time

import pytest
import torch

from phraya_b200 import _abi as A
from phraya_b200 import api as P
from phraya_b200 import casegen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", [A.FAST, A.BALANCED])
def test_scratch_does_not_grow(strategy):
    ref = G.repeat_reference(2_000_000, 20, seed=71)
    packed, _, _ = G.long_reads(ref, 1000, seed=72)
    reads = [bytes(packed.seq[o:o + n]) for o, n in zip(packed.off.tolist(), packed.len.tolist())]
    used = lambda: torch.cuda.mem_get_info()[1] - torch.cuda.mem_get_info()[0]  # noqa: E731
    with P.Engine(0) as eng:
        idx = eng.index(ref)
        srv = eng.server(idx, strategy=strategy, max_batch_reads=1024, max_wait_us=50_000, n_streams=2)
        before = used()
        ids = srv.submit_many(reads)
        got, until = {}, time.time() + 120
        while len(got) < len(reads) and time.time() < until:
            for rid, res, _ in srv.poll(4096, wait_us=20000):
                got[rid] = res
        grown = used() - before
        srv.close()
        batched, _ = eng.align_reads(idx, reads, strategy)
    assert [got[i] for i in ids] == batched
    assert grown < 1 << 30   # (every other buffer was sized for a full batch at creation)
