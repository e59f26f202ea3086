"""The group walk where it has fewer groups than the GPU holds warps, and each SM takes an even share of them: a
system on its own, for every number of warps per block, gets the bits that it gets beside a system of so many groups
that every resident warp takes part."""
import numpy as np
import pytest

from next_b200 import ic
from next_b200.native import Simulation

pytestmark = pytest.mark.gpu

COLS = ("ax", "ay", "az")


@pytest.mark.parametrize("precision", ["mixed", "fp64group"])
@pytest.mark.parametrize("n,group", [(1, 8), (9, 8), (300, 8), (1000, 8), (1100, 2), (2400, 4), (2500, 4), (5000, 8), (5000, 3),
                                     (5000, 32), (5000, 2)])
def test_few_groups_equal_many(precision, n, group):
    b, rest = ic.plummer(n, seed=n + group), ic.uniform_sphere(40000, seed=3)
    knobs = dict(eps=0.01, leaf_cap=2, group_cap=group)
    both = Simulation("accurate", precision, **knobs)
    both.upload({c: np.concatenate([b[c], rest[c]]) for c in b}, np.array([0, n, n + 40000]))
    want = both.accel()
    assert both.stats()["n_groups"] > 20 * 148 or group == 32
    both.close()
    for warps in (1, 2, 3, 4):
        one = Simulation("accurate", precision, walk_warps=warps, **knobs)
        one.upload(b)
        got = one.accel()
        assert one.stats()["device_error"] == 0
        for c in COLS:
            np.testing.assert_array_equal(got[c], want[c][:n])
        one.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64group"])
@pytest.mark.parametrize("n", [33, 1000, 5000, 30000])
def test_few_full_groups_equal_many(precision, n):
    """The same with the default leaf and group sizes, beside so many bodies that every resident warp takes part."""
    b, rest = ic.plummer(n, seed=n), ic.uniform_sphere(200000, seed=3)
    both, one = Simulation("accurate", precision, eps=0.01), Simulation("accurate", precision, eps=0.01)
    both.upload({c: np.concatenate([b[c], rest[c]]) for c in b}, np.array([0, n, n + 200000]))
    one.upload(b)
    want, got = both.accel(), one.accel()
    assert both.stats()["n_groups"] > 20 * 148 > one.stats()["n_groups"]
    assert one.stats()["device_error"] == 0
    for c in COLS:
        np.testing.assert_array_equal(got[c], want[c][:n])
    both.close()
    one.close()
