"""States that are not in order are refused, wherever they lie: also above the last one, outside the bucket table that its
highest bit lays out."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("states", [[5, 3, 4], [1 << 60, 1, 2, 3], [0, 1 << 63, 1 << 40, 7], [3, 3], [(1 << 64) + 1, 1 << 64, 9]])
def test_unsorted_states_are_refused(states):
    lohi = np.array([[s & (2**64 - 1), s >> 64] for s in states], dtype=np.uint64)
    with pytest.raises(q.QsiError) as e:
        q.ZBasis(lohi)
    assert e.value.status == 1  # QSI_INVALID_ARG
    assert len(q.ZBasis(np.unique(lohi[::-1], axis=0)[:1])) == 1


def test_a_long_unsorted_basis_is_refused():
    lohi = np.zeros((100_000, 2), dtype=np.uint64)
    lohi[:, 0] = np.random.default_rng(1).integers(0, 1 << 62, 100_000, dtype=np.uint64)
    lohi[-1] = [1 << 20, 0]
    with pytest.raises(q.QsiError):
        q.ZBasis(lohi)
