"""Expectation values of many long vectors where device memory holds them once but not their images too."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu


# 2^20 states and 200 vectors, 1.6 GiB: images of some of them at a time; the last operator has a diagonal part
@pytest.mark.parametrize("room", [3.1, 2.2])
def test_images_of_some_vectors_at_a_time(room):
    torch = pytest.importorskip("torch")
    n, nvec = 1 << 20, 200
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n, dtype=np.uint64)
    basis = q.ZBasis(lohi)
    ops = []
    for specs in (["0x"], ["7x"], ["3x", "3z"]):
        H = q.SymbolicOpSum()
        for s in specs:
            H.add_term(1.0, q.SymbolicPMROperator(s))
        ops.append(H)
    psi = np.random.default_rng(1).standard_normal((nvec, n))
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(max(0, free - int(room * (1 << 30))), dtype=torch.uint8, device="cuda")
    try:
        got, _ = q.expectations(basis, ops, psi.T, cross=False)
    finally:
        del fill
        torch.cuda.empty_cache()
    i = np.arange(n)
    spin3 = np.where((i >> 3) & 1, 1.0, -1.0)
    for a in (0, 1, 127, 128, 129, 199):
        for l, image in enumerate([psi[a][i ^ 1], psi[a][i ^ 128], psi[a][i ^ 8] + spin3 * psi[a]]):
            # up to 2^16 sums in a row, then the parts', of products that add up to 2n/3 in magnitude
            np.testing.assert_allclose(got[l, a], psi @ image, rtol=0, atol=2**16 * 1.1e-16 * n)
