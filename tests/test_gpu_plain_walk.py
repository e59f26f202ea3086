"""The plain FP64 walks at the edges of their warps, lists and stacks.

The accurate walk takes seven bodies of one system per warp and sums a body's
terms in another order than the oracle: at most a few thousand terms, each
rounded a few times, so forces and potentials agree to 1e-12 of the largest one
(2^-53 times the term count leaves a factor of two); the opening decisions are
the same FP64 comparisons, so the interaction counts are equal.
"""
import numpy as np
import pytest

from next_b200 import ic
from next_b200.native import Simulation

pytestmark = pytest.mark.gpu

TOL = 1e-12


def close(a, b, names):
    scale = max(np.max(np.abs(b[c])) for c in names)
    for c in names:
        np.testing.assert_allclose(a[c], b[c], rtol=0, atol=TOL * scale)


@pytest.mark.parametrize("n,leaf_cap,theta,eps,quad", [
    (1, 1, 0.5, 0.01, 1), (2, 1, 0.5, 0.0, 1), (3, 1, 0.5, 0.01, 1), (4, 2, 0.5, 0.01, 1), (5, 1, 0.5, 0.01, 1),
    (31, 1, 0.5, 0.01, 1), (33, 3, 0.3, 0.01, 0), (129, 64, 0.5, 0.01, 1), (1003, 1, 0.2, 0.0, 1),
    (1001, 17, 1.0, 0.01, 1), (4097, 1, 0.7, 0.005, 0), (4099, 64, 0.5, 0.01, 1),
])
def test_accurate_walk_sizes(oracle, n, leaf_cap, theta, eps, quad):
    b = ic.plummer(n, seed=n)
    sim = Simulation("accurate", "fp64", theta=theta, eps=eps, leaf_cap=leaf_cap, quadrupole=quad)
    sim.upload(b)
    sim.reset_timers()
    a = sim.accel(potential=True)
    r = oracle.accel(b, mode="accurate", theta=theta, eps=eps, leaf_cap=leaf_cap, quad=bool(quad), potential=True)
    st = sim.stats()
    assert (st["pp_interactions"], st["pc_interactions"], st["device_error"]) == (r["pp"], r["pc"], 0)
    if n > 1:
        close(a, r, ("ax", "ay", "az"))
        close(a, r, ("pot",))
    f = Simulation("accurate", "fp64", theta=theta, eps=eps, leaf_cap=leaf_cap, quadrupole=quad)
    f.upload(b)
    g = f.accel()                                   # the walk without the potential: the same forces
    for c in ("ax", "ay", "az"):
        np.testing.assert_array_equal(g[c], a[c])
    sim.close()
    f.close()


def test_accurate_walk_buckets_and_massless(oracle):
    """Coincident bodies (leaves of more bodies than the leaf size) and zero masses."""
    b = ic.plummer(700, seed=5)
    for k in ("x", "y", "z"):
        b[k][100:200] = b[k][100]
        b[k][300:303] = b[k][300]
    b["m"][::7] = 0.0
    sim = Simulation("accurate", "fp64", theta=0.5, eps=0.02, leaf_cap=1)
    sim.upload(b)
    a = sim.accel(potential=True)
    r = oracle.accel(b, mode="accurate", theta=0.5, eps=0.02, leaf_cap=1, potential=True)
    close(a, r, ("ax", "ay", "az"))
    close(a, r, ("pot",))
    sim.close()


def test_accurate_walk_full_stack(oracle):
    """An opening angle so small that nearly every cell opens: the stack fills and the rounds are cut short."""
    b = ic.plummer(3000, seed=9)
    sim = Simulation("accurate", "fp64", theta=0.02, eps=0.01, leaf_cap=1)
    sim.upload(b)
    a = sim.accel()
    r = oracle.accel(b, mode="accurate", theta=0.02, eps=0.01, leaf_cap=1)
    close(a, r, ("ax", "ay", "az"))
    assert sim.stats()["device_error"] == 0
    sim.close()


def test_accurate_walk_ensemble_of_odd_sizes():
    """Systems whose sizes are no multiples of a warp's bodies, some empty: bit-equal to each system alone."""
    sizes = [5, 0, 1, 130, 3, 0, 2, 517, 64, 7]
    parts = [ic.plummer(k, seed=i) for i, k in enumerate(sizes) if k]
    b = {c: np.concatenate([p[c] for p in parts]) for c in parts[0]}
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    sim = Simulation("accurate", "fp64")
    sim.upload(b, offsets)
    a = sim.accel()
    for i, k in enumerate(sizes):
        if k == 0:
            continue
        one = Simulation("accurate", "fp64")
        one.upload(ic.plummer(k, seed=i))
        r = one.accel()
        for c in ("ax", "ay", "az"):
            np.testing.assert_array_equal(a[c][offsets[i]:offsets[i + 1]], r[c])
        one.close()
    sim.close()


def reference_bodies(n, seed):
    b = ic.plummer(n, seed=seed)
    rng = np.random.default_rng(seed)
    b["type"][:] = rng.integers(0, 3, n)
    return b


@pytest.mark.parametrize("n,theta,masses", [
    (1, 0.5, "equal"), (2, 0.5, "equal"), (9, 0.5, "equal"), (127, 0.5, "mixed"), (129, 0.3, "equal"),
    (1001, 0.5, "mixed"), (4097, 0.5, "equal"), (4097, 0.05, "mixed"), (3000, 1.5, "equal"),
])
def test_reference_walk_sizes(oracle, n, theta, masses):
    """Dark bodies of one mass (its softening stored per node) and of several (some computed per interaction),
    lists and warps that end early: the oracle's forces up to the last bit of cbrt and pow (another opening decision
    would move them by 1e-3 and more)."""
    b = reference_bodies(n, n)
    if masses == "mixed":
        b["m"] *= np.random.default_rng(1).uniform(0.1, 3.0, n)
        b["m"][::11] = 0.0
    sim = Simulation("reference", "fp64", theta=theta)
    sim.upload(b)
    a = sim.accel()
    r = oracle.accel(b, mode="ref", theta=theta)
    assert sim.stats()["device_error"] == 0
    if n > 1:
        close(a, r, ("ax", "ay", "az"))
    sim.close()


def test_reference_walk_ties_and_buckets(oracle):
    """A lattice, whose distances tie with the opening test's limit exactly, with coincident bodies among it."""
    g = np.arange(12, dtype=np.float64) / 8.0
    x, y, z = (v.ravel() for v in np.meshgrid(g, g, g, indexing="ij"))
    b = reference_bodies(x.size, 3)
    b["x"], b["y"], b["z"] = x.copy(), y.copy(), z.copy()
    for k in ("x", "y", "z"):
        b[k][500:520] = b[k][500]
    for theta in (0.25, 0.5, 1.0):
        sim = Simulation("reference", "fp64", theta=theta)
        sim.upload(b)
        a = sim.accel()
        r = oracle.accel(b, mode="ref", theta=theta)
        assert sim.stats()["device_error"] == 0
        close(a, r, ("ax", "ay", "az"))
        sim.close()


def test_reference_walk_after_other_dark_masses(oracle):
    """The stored softening follows the uploaded bodies: another upload with other masses, then one without dark bodies."""
    sim = Simulation("reference", "fp64")
    for seed, scale, kind in ((1, 1.0, 1), (2, 4.0, 1), (3, 0.5, 0)):
        b = ic.plummer(600, seed=seed)
        b["m"] *= scale
        b["type"][::3] = kind
        sim.upload(b)
        a = sim.accel()
        close(a, oracle.accel(b, mode="ref"), ("ax", "ay", "az"))
    sim.close()


@pytest.mark.parametrize("n", [1, 2, 3, 7, 9, 33, 1000, 2960, 2961, 5920, 5921, 11841, 16000, 20001])
def test_reference_walk_small_equals_large(n):
    """A small system, walked by 32, 16 or 8 lanes per body, gets the bits it gets beside a system so large that one
    thread walks for each body: with dark matter of two masses, coincident bodies (buckets) and massless ones."""
    b, rest = reference_bodies(n, n), reference_bodies(50000, 2)
    if n > 700:
        for k in ("x", "y", "z"):
            b[k][100:140] = b[k][100]
            b[k][300:303] = b[k][300]
        b["m"][200:600:9] = 0.0
        b["m"][5:400:7] *= 3.0
    one, both = Simulation("reference", "fp64"), Simulation("reference", "fp64")
    one.upload(b)
    both.upload({c: np.concatenate([b[c], rest[c]]) for c in b}, np.array([0, n, n + 50000]))
    got, want = one.accel(), both.accel()
    assert one.stats()["device_error"] == 0 and both.stats()["device_error"] == 0
    for c in ("ax", "ay", "az"):
        np.testing.assert_array_equal(got[c], want[c][:n])
    one.close()
    both.close()


@pytest.mark.parametrize("length", [2.0 ** -400, 2.0 ** 400])
def test_accurate_walk_far_from_unit_lengths(length):
    """Lengths scaled by a power of two round nothing: forces and potentials scale exactly, where the distances'
    own fifth powers would leave the range."""
    b = ic.plummer(999, seed=4)
    c = dict(b, **{k: b[k] * length for k in ("x", "y", "z")})
    out = []
    for bodies, eps in ((b, 0.01), (c, 0.01 * length)):
        sim = Simulation("accurate", "fp64", theta=0.5, eps=eps)
        sim.upload(bodies)
        out.append(sim.accel(potential=True))
        assert sim.stats()["device_error"] == 0
        sim.close()
    for k in ("ax", "ay", "az"):
        np.testing.assert_array_equal(out[1][k] * length * length, out[0][k])
    np.testing.assert_array_equal(out[1]["pot"] * length, out[0]["pot"])


@pytest.mark.parametrize("n,theta", [(300, 0.6), (2000, 0.4), (5000, 0.25), (5000, 0.5), (9000, 0.39), (20001, 0.3), (20001, 0.5)])
def test_reference_walk_buckets_of_every_size(n, theta):
    """Coincident bodies in buckets below, at and above the numbers of lanes, with two masses, massless ones and dark
    matter among them: the walks of several lanes per body, of lists and of small opening angles give the same bits."""
    b, rest = reference_bodies(n, n + 1), reference_bodies(50000, 2)
    at = 0
    for size in (2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 65):
        for k in ("x", "y", "z"):
            b[k][at:at + size] = b[k][at]
        at += size
    b["m"][0:at:3] *= 2.0
    b["m"][1:at:7] = 0.0
    one, both = Simulation("reference", "fp64", theta=theta), Simulation("reference", "fp64", theta=theta)
    one.upload(b)
    both.upload({c: np.concatenate([b[c], rest[c]]) for c in b}, np.array([0, n, n + 50000]))
    one.reset_timers()
    got, want = one.accel(), both.accel()
    assert one.stats()["device_error"] == 0 and both.stats()["device_error"] == 0
    for c in ("ax", "ay", "az"):
        np.testing.assert_array_equal(got[c], want[c][:n])
    one.close()
    both.close()


def test_reference_walk_buckets_against_the_oracle(oracle):
    """The same buckets in a walk of one thread per body, at an opening angle on either side of the lists' limit."""
    b = reference_bodies(50001, 7)
    for at, size in ((0, 70), (100, 33), (200, 2)):
        for k in ("x", "y", "z"):
            b[k][at:at + size] = b[k][at]
    b["m"][0:70:3] *= 2.0
    for theta in (0.39, 0.4):
        sim = Simulation("reference", "fp64", theta=theta)
        sim.upload(b)
        a, r = sim.accel(), oracle.accel(b, mode="ref", theta=theta)
        assert sim.stats()["device_error"] == 0
        close(a, r, ("ax", "ay", "az"))
        sim.close()


@pytest.mark.parametrize("n,leaf_cap,theta,eps,quad,shape", [
    (6, 1, 0.5, 0.01, 1, "sphere"), (8, 1, 0.5, 0.0, 1, "sphere"), (50, 1, 1.0, 0.01, 0, "sphere"),
    (79, 1, 0.5, 0.01, 1, "sphere"), (80, 1, 0.5, 0.01, 1, "sphere"), (81, 5, 0.5, 0.01, 1, "sphere"),
    (79, 64, 0.5, 0.01, 1, "sphere"), (79, 1, 0.02, 0.01, 1, "sphere"), (77, 3, 0.02, 0.01, 1, "chain"),
    (60, 1, 0.5, 0.01, 1, "chain"), (79, 1, 0.5, 0.02, 1, "bucket"), (30, 2, 0.7, 0.02, 1, "bucket"),
])
def test_accurate_walk_of_small_systems(oracle, n, leaf_cap, theta, eps, quad, shape):
    """Eight lanes for seven bodies: around the size where whole warps take over, full stacks, cells down to the deepest
    level, leaves of many bodies, massless ones."""
    b = ic.plummer(n, seed=n)
    if shape == "chain":
        r = 2.0 ** -np.linspace(0, 19, n)
        for k, s in zip("xyz", (1.0, -0.7, 0.4)):
            b[k] = s * r
    if shape == "bucket":
        for k in "xyz":
            b[k][: n // 2] = b[k][0]
        b["m"][::5] = 0.0
    sim = Simulation("accurate", "fp64", theta=theta, eps=eps, leaf_cap=leaf_cap, quadrupole=quad)
    sim.upload(b)
    sim.reset_timers()
    a = sim.accel(potential=True)
    r = oracle.accel(b, mode="accurate", theta=theta, eps=eps, leaf_cap=leaf_cap, quad=bool(quad), potential=True)
    st = sim.stats()
    assert (st["pp_interactions"], st["pc_interactions"], st["device_error"]) == (r["pp"], r["pc"], 0)
    close(a, r, ("ax", "ay", "az"))
    close(a, r, ("pot",))
    sim.close()


def test_accurate_walk_batch_of_small_systems():
    """Systems of 0 to 90 bodies, walked by groups of lanes and by whole warps, and one large one: every system's
    forces and potentials are bit-equal to its own."""
    rng = np.random.default_rng(4)
    sizes = [*rng.integers(0, 91, 400), 700, 79, 80, 1, 0]
    parts = [ic.plummer(int(k), seed=i) for i, k in enumerate(sizes) if k]
    b = {c: np.concatenate([p[c] for p in parts]) for c in parts[0]}
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    sim = Simulation("accurate", "fp64")
    sim.upload(b, offsets)
    a = sim.accel(potential=True)
    assert sim.stats()["device_error"] == 0
    for i in [*range(0, 400, 23), 400, 401, 402, 403]:
        if sizes[i] == 0:
            continue
        one = Simulation("accurate", "fp64")
        one.upload(ic.plummer(int(sizes[i]), seed=i))
        r = one.accel(potential=True)
        for c in ("ax", "ay", "az", "pot"):
            np.testing.assert_array_equal(a[c][offsets[i]:offsets[i + 1]], r[c])
        one.close()
    sim.close()
