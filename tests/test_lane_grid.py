"""The lane-per-pair Myers kernel takes one scratch slot per warp: its launch has no more warps
than the pass has slots, for every block size the other kernels may be set to."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include <cstdio>
#include "kernels.cuh"
int main() {
    for (unsigned long long blocks = 1; blocks <= 592; ++blocks)
        for (int threads = 32; threads <= 256; threads += 32)
            for (int per_sm = 2; per_sm <= 3; ++per_sm) {
                const unsigned long long slots = blocks * (threads / 32);
                const phr::LaneGrid g = phr::lane_grid(slots, 148, per_sm);
                const bool ok = g.blocks >= 1 && g.threads >= 32 && g.threads <= phr::kLaneThreads && g.blocks <= 148 * per_sm &&
                                1ull * g.blocks * (g.threads / 32) <= slots &&
                                // and no slot idles that a whole block or the one block could take
                                (slots - 1ull * g.blocks * (g.threads / 32) < 8 || g.blocks == 148 * per_sm);
                if (!ok) { std::printf("%llu %d %d: %d x %d\\n", blocks, threads, per_sm, g.blocks, g.threads); return 1; }
            }
    return 0;
}
"""


def test_no_more_warps_than_slots(tmp_path):
    from phraya_b200 import build as B
    if not shutil.which(B.nvcc()):
        pytest.skip("nvcc not available")
    (tmp_path / "grid.cu").write_text(SRC)
    subprocess.run([B.nvcc(), *B.NVCC_FLAGS, "-I", os.path.join(ROOT, "phraya_b200", "csrc"), str(tmp_path / "grid.cu"),
                    "-o", str(tmp_path / "grid")], check=True)
    r = subprocess.run([str(tmp_path / "grid")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 96, 224, 256])
def test_few_tasks_of_large_slots(threads):
    """Two tasks of 32 long pairs: with one-warp blocks the pass has two slots of 9 MB."""
    import oracle as O
    from phraya_b200 import _abi as A
    from phraya_b200 import api as P
    rng = np.random.default_rng(81)
    pairs = []
    for _ in range(64):
        q = rng.choice(np.frombuffer(b"ACGT", np.uint8), 3000)
        t = q.copy()
        t[rng.integers(0, 3000, 40)] = ord("A")
        pairs.append((q.tobytes(), np.delete(t, rng.integers(0, 3000, 5)).tobytes()))
    packed = O.PackedPairs(pairs)
    oa, oc = O.extend_packed(A.ENGINE_MYERS_GLOBAL, packed, (2, 4, 1))
    for ckpt in (0, 1):
        with P.Engine(0) as eng:
            eng.set_tune("block_threads", threads)
            eng.set_tune("myers_lane_ckpt", ckpt)
            eng.set_timing(True)
            ga, gc = eng.extend_packed(A.ENGINE_MYERS_GLOBAL, packed)
            assert "myers_lane" in eng.kernel_times()
            assert P.unpack(ga, gc) == P.unpack(oa, oc)
