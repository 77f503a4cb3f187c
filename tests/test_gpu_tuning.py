"""Launch settings as they are asked for, reported and tuned."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q
from qsi_subspace_ed_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cached", [False, True])
def test_a_setting_that_comes_to_the_same_kernel_is_not_timed(cached):
    """Built-in choices are reported as such until a setting is made, which is kept; the tuner times no two settings that
    come to one kernel: eight vectors per lane are built in for 64 with the look-ups, and four (lists of up to 256) for a
    materialised operator, which takes eight as four."""
    lat = workloads.lattice("pyro_1x2x1")
    g, B = workloads.ring_zeeman_params(5)
    op = q.LazyOpSum(q.ZBasis(q.enumerate_basis(lat)), q.build_ring_zeeman(lat, g, B))
    assert op.tuning(1)["list_cap"] == op.tuning(1)["vec_width"] == 0
    X = np.random.default_rng(1).standard_normal((op.rows(), 64)).astype(np.float32)
    ref, Y = np.zeros_like(X), np.zeros_like(X)
    op.apply_batched(X, ref)
    op.materialise(cached)

    def timed():
        return [line.split()[0] for line in op.autotune(R=64, dtype="f32", reps=1).splitlines()
                if line.startswith(("vec_width", "list_cap"))]

    log = timed()
    widths = [v for v in log if v.startswith("vec_width")]
    assert widths == (["vec_width=16"] if cached else ["vec_width=4", "vec_width=16"])
    op.set_tuning(0, 0, which=1, vec_width=4)
    for cap in (256, 128):
        op.set_kernel(1, 1, list_cap=cap)
        assert op.tuning(1)["list_cap"] == cap
        op.apply_batched(X, Y)
        assert np.array_equal(Y, ref)
    if cached:
        op.set_tuning(0, 0, which=1, vec_width=8)
        lists = [v for v in timed() if v.startswith("list_cap")]
        if op.tuning(1)["vec_width"] != 16:
            assert lists == ["list_cap=192", "list_cap=256"]
    op.apply_batched(X, Y)
    assert np.array_equal(Y, ref)
