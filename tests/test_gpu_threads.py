"""Contexts of different settings used from several threads at once."""
import threading

import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine,costs", [(A.ENGINE_WFA_LINEAR, (2, 4, 1)), (A.ENGINE_WFA_AFFINE, (2, 4, 1)),
                                          (A.ENGINE_WFA_AFFINE, (1, 2, 3))], ids=["linear", "2-4-1", "1-2-3"])
def test_shared_memory_sizes_side_by_side(engine, costs):
    """A kernel's limit of shared memory belongs to the process: one context's launch must not
    depend on another's "wfa_big_smem"."""
    rng = np.random.default_rng(51)
    q = rng.choice(np.frombuffer(b"ACGT", np.uint8), 2100)
    t = q.copy()
    t[rng.integers(0, q.size, 5)] = ord("C")
    packed = O.PackedPairs([(q.tobytes(), t.tobytes()), (q[:150].tobytes(), t[:160].tobytes())])
    want = P.unpack(*O.extend_packed(engine, packed, costs))
    errors = []

    def work(smem, block):
        try:
            with P.Engine(0) as eng:
                eng.set_tune("wfa_big_smem", smem)
                eng.set_tune("block_threads", block)
                for _ in range(1500):
                    if P.unpack(*eng.extend_packed(engine, packed, P.AffineCosts(*costs))) != want:
                        raise AssertionError("another result with %d bytes" % smem)
        except Exception as e:   # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(kib << 10, block))
               for kib, block in ((16, 32), (60, 128), (120, 64), (200, 256))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
