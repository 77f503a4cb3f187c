"""eigval0 at the ends of what max_iterations takes."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q
from qsi_subspace_ed_gb300 import workloads

pytestmark = pytest.mark.gpu


def operator():
    lat = workloads.lattice("pyro_1x2x1")
    g, B = workloads.ring_zeeman_params(5)
    return q.LazyOpSum(q.ZBasis(q.enumerate_basis(lat, sector=(4, 4, 4, 4))), q.build_ring_zeeman(lat, g, B))


@pytest.mark.parametrize("most", [0, -1])
@pytest.mark.parametrize("vector", [False, True])
def test_no_iterations(most, vector):
    """No step is taken: no iterations are reported and the accumulated vector is zero."""
    op = operator()
    _, vec, its = q.eigval0(op, max_iterations=most, calc_eigenvector=vector)
    assert its == 0
    assert vec is None if not vector else not vec.any()
    assert np.isfinite(q.eigval0(op, max_iterations=30, calc_eigenvector=vector)[0])


def test_an_open_number_of_iterations():
    """As many iterations as there may be on a basis where the recurrence ends by itself: device memory for the
    coefficients of a batch, not for all that were allowed."""
    torch = pytest.importorskip("torch")
    H = q.SymbolicOpSum()
    for k in range(3):
        H.add_term(1.0 + k, q.SymbolicPMROperator(f"{k}x"))
    op = q.LazyOpSum(q.ZBasis(np.stack([np.arange(8, dtype=np.uint64), np.zeros(8, dtype=np.uint64)], axis=1)), H)
    want = q.eigval0(op, max_iterations=40)
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(max(0, free - (8 << 30)), dtype=torch.uint8, device="cuda")
    try:
        got = q.eigval0(op, max_iterations=2**31 - 1)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert got[0] == want[0] and got[2] == want[2] <= 8 and np.array_equal(got[1], want[1])


def test_a_stop_behind_the_last_iteration(tmp_path):
    """After a resumption, stops and checkpoints so far off that the iteration to come to is no 32-bit number."""
    op = operator()
    path = str(tmp_path / "ck.h5")
    want = q.eigval0(op, max_iterations=90)
    with pytest.raises(q.QsiError):
        q.eigval0(op, max_iterations=90, checkpoint=path, stop_after=37)
    got = q.eigval0(op, max_iterations=90, checkpoint=path, stop_after=2**31 - 1, checkpoint_every=2**31 - 1)
    assert got[0] == want[0] and got[2] == want[2] and np.array_equal(got[1], want[1])
