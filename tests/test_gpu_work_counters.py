"""Work counters say what was computed."""
import numpy as np
import pytest

import oracle as O
from phraya_b200 import _abi as A
from phraya_b200 import api as P

pytestmark = pytest.mark.gpu


def test_fitting_lanes_count_the_columns_they_advance():
    """Windows ten queries long: a distance is at least the columns past the query's 64 rows, so
    a search is over (8 above the best, 0) by column 72 and its warp by the next multiple of 8."""
    n, m = 16384, 64
    rng = np.random.default_rng(31)
    t = rng.choice(np.frombuffer(b"ACGT", np.uint8), (n, 10 * m))
    packed = O.PackedPairs([(w[:m].tobytes(), w.tobytes()) for w in t])
    with P.Engine(0) as eng:
        aln, _ = eng.extend_packed(A.ENGINE_MYERS_FIT, packed)
        columns = eng.counter("myers_lane_block_columns")
    assert (aln["edit_distance"] == 0).all() and (aln["target_end"] == m).all()
    assert m * n <= columns <= 80 * n
