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
