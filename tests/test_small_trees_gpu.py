"""Trees of a few points, either side of the size from which the presorted
lists build them, against the oracle."""
import numpy as np
import pytest

import fkdtree_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("values", [0, 3, 1])  # distinct coordinates, three values, one
@pytest.mark.parametrize("n", [1, 2, 3, 31, 64, 127, 128, 129, 200])
@pytest.mark.parametrize("dim", [3, 4])
def test_small_trees(cuda, dim, n, values):
    rng = np.random.default_rng(10 * n + values)
    x = rng.random((dim, n), dtype=np.float32)
    if values:
        x = np.floor(x * values).astype(np.float32)
    ids = rng.permutation(n).astype(np.uint32)
    for knob in (0, 1, 2):
        t = F.FKDTree(x, ids).set_param("subtree", knob).build()
        tab, tid = t.tables()
        want = O.build(x, ids)
        assert np.array_equal(tab.view(np.uint32), want[0].view(np.uint32)) and np.array_equal(tid, want[1])
        t.close()
