"""Admission of the lookup caches that plain solves build for themselves, on the CPU: what a solve may take is counted
while it runs, and leaves room for every solve that would have been admitted beside it."""
import threading

import numpy as np
import pytest

from qsi_subspace_ed_gb300 import serve


class Recorder(serve.RequestLoop):
    """Plain solves that meet at a barrier and note what they were allowed and what was counted meanwhile."""

    def __init__(self, dims, meet, **kw):
        self.allowed, self.counted = [], []
        self.gate = threading.Barrier(meet)
        secs = {k: serve.Sector(k, None, np.zeros((d, 2), np.uint64)) for k, d in dims.items()}
        super().__init__(secs, batching=False, make_basis=lambda lohi: len(lohi), **kw)

    def _solve_default(self, req, basis, sec, cache_bytes=-1):
        self.allowed.append(cache_bytes)
        self.gate.wait(20)
        self.counted.append(self._in_use)
        self.gate.wait(20)
        return np.zeros(1)


@pytest.mark.parametrize("solves,extra", [(1, 0.0), (2, 0.0), (2, 0.4), (3, 0.9)])
def test_caches_leave_room_for_the_other_solves(solves, extra):
    """A budget for `solves` solves and a part of another one, which is all that their caches may share."""
    dims = {"a": 100_000, "b": 60_000}
    one = serve.solve_footprint(100_000, 5, 20)
    budget = int((solves + extra) * one) + sum(serve.basis_footprint(d) for d in dims.values())
    loop = Recorder(dims, solves, slots=4, hbm_budget=budget)
    try:
        reqs = [loop.submit(serve.Request(rid=k, sector="a", g=[1] * 4, B=[0] * 3)) for k in range(2 * solves)]
        loop.drain(timeout=60)
    finally:
        loop.close()
    assert all(r.error is None for r in reqs)  # `solves` at a time met, so none was kept out by a cache
    assert max(loop.counted) <= budget
    assert all(0 <= c <= extra * one for c in loop.allowed)
    assert (max(loop.allowed) > 0) == (extra > 0)
