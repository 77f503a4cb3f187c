"""The lookup caches that solves build for themselves are memory to spare: a call that fits without them fits."""
import threading
import time

import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q
from qsi_subspace_ed_gb300 import workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MB = 1 << 20


@pytest.fixture(scope="module")
def basis():
    return q.ZBasis(q.enumerate_basis_gpu(workloads.lattice("pyro_1x2x2")))  # 2,891,562 states, caches of 207 MB


def operator(basis, seed):
    g, B = workloads.ring_zeeman_params(seed)
    return q.LazyOpSum(basis, q.build_ring_zeeman(workloads.lattice("pyro_1x2x2"), g, B))


def free():
    return torch.cuda.mem_get_info()[0]


def run(f, *args, **kw):
    """f in a thread of its own: the thread, what it returned or raised, and the least memory free meanwhile."""
    out = {"least": free()}

    def body():
        try:
            out["result"] = f(*args, **kw)
        except q.QsiError as e:
            out["error"] = e

    t = threading.Thread(target=body)
    t.start()
    return t, out


def finish(t, out):
    while t.is_alive():
        out["least"] = min(out["least"], free())
        time.sleep(0.0005)
    t.join()
    return out


def test_another_solve_takes_the_memory(basis):
    """A long recurrence holds a cache; a second one needs more than is left beside it, but no more than without it."""
    a, b = operator(basis, 1), operator(basis, 2)
    small = dict(nev=1, ncv=60, tol=1e-8, want_vectors=False)
    want, _, _ = q.diagonalise(b, seed=3, **small)
    torch.cuda.synchronize()
    before = free()
    b.materialise(True)
    cache = before - free()
    one = finish(*run(q.diagonalise, b, seed=3, **small))  # materialised already: no cache of its own
    need = before - cache - one["least"]
    b.materialise(False)
    assert np.array_equal(one["result"][0], want) and cache > 150 * MB
    long = dict(seed=1, max_iterations=9000, calc_eigenvector=False)
    level = q.eigval0(a, **long)[0]
    held, out = run(q.eigval0, a, **long)
    time.sleep(0.4)  # hundreds of applies: the cache is there
    fill = torch.empty(max(0, free() - need + 60 * MB), dtype=torch.uint8, device="cuda")
    try:
        assert held.is_alive()
        got, _, _ = q.diagonalise(b, seed=3, **small)
        assert held.is_alive()
    finally:
        held.join()
        del fill
        torch.cuda.empty_cache()
    assert np.array_equal(got, want)
    assert out["result"][0] == level  # bit for bit, with the cache for a part of the iterations


@pytest.mark.parametrize("most,cached", [(-1, True), (0, False), (100 * MB, False), (1 << 40, True)])
def test_the_limit_of_a_solves_own_cache(basis, most, cached):
    """The cache is built where the limit allows all of it; the results are the same."""
    op = operator(basis, 4)
    kw = dict(seed=2, max_iterations=2500, calc_eigenvector=False)
    op.set_solve_cache(0)
    want = q.eigval0(op, **kw)[0]
    least = finish(*run(q.eigval0, op, **kw))["least"]
    op.set_solve_cache(most)
    out = finish(*run(q.eigval0, op, **kw))
    assert out["result"][0] == want
    assert (least - out["least"] > 150 * MB) == cached
