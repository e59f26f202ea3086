"""The one-pass cell and child scans at the edges of their tiles (1,024 positions, 256 cells), for every way a leaf
size meets the four positions a thread owns: the exported tree equals the oracle's node for node (levels, bodies,
half-widths and masses of single bodies exactly; masses of cells to the rounding of a sum, 1e-14)."""
import numpy as np
import pytest

from next_b200 import ic, native
from next_b200.native import Simulation

pytestmark = pytest.mark.gpu

LEVEL, MASS, HALF, LEAF, COUNT = 0, 1, 5, 12, 15


@pytest.mark.parametrize("n,leaf_cap", [(1, 1), (2, 1), (5, 3), (255, 4), (257, 5), (1023, 1), (1024, 2), (1025, 3), (1027, 4),
                                        (2047, 16), (2049, 64), (4097, 5), (33000, 1), (70001, 16)])
def test_tree_at_tile_edges(oracle, n, leaf_cap):
    b = ic.plummer(n, seed=n) if n % 2 else ic.uniform_sphere(n, seed=n)
    sim = Simulation("accurate", "fp64", leaf_cap=leaf_cap)
    sim.upload(b)
    t, r = sim.debug_tree(), oracle.tree(b, mode="accurate", leaf_cap=leaf_cap)
    assert t.shape == r.shape
    for c in (LEVEL, HALF, LEAF):
        np.testing.assert_array_equal(t[:, c], r[:, c])
    leaves = r[:, LEAF] == 1                        # the device exports the body counts of leaves
    np.testing.assert_array_equal(t[leaves, COUNT], r[leaves, COUNT])
    np.testing.assert_allclose(t[:, MASS], r[:, MASS], rtol=1e-14, atol=0)
    assert sim.stats()["device_error"] == 0
    sim.close()


def test_build_of_coincident_bodies_and_many_systems(oracle):
    """Long chains of cells at one position, and systems that start and end inside a tile: every system's forces
    equal its own."""
    sizes = [700, 1, 0, 1500, 3, 900]
    parts = [ic.plummer(k, seed=i + 20) for i, k in enumerate(sizes) if k]
    for k in ("x", "y", "z"):
        parts[0][k][10:60] = parts[0][k][10]
    b = {c: np.concatenate([p[c] for p in parts]) for c in parts[0]}
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    sim = Simulation("accurate", "fp64", leaf_cap=2)
    sim.upload(b, offsets)
    a, j = sim.accel(), 0
    for i, k in enumerate(sizes):
        if k == 0:
            continue
        one = Simulation("accurate", "fp64", leaf_cap=2)
        one.upload(parts[j])
        r = one.accel()
        for c in ("ax", "ay", "az"):
            np.testing.assert_array_equal(a[c][offsets[i]:offsets[i + 1]], r[c])
        one.close()
        j += 1
    sim.close()


@pytest.mark.parametrize("leaf_cap", [1, 3, 16])
def test_cells_of_every_length_and_alignment(oracle, leaf_cap):
    """Clumps of 1 to 150 bodies, deep cells that start at every offset from a 16-byte boundary and end before, at and
    behind the reach of the forward scan for a cell's end: the oracle's tree, node for node."""
    rng = np.random.default_rng(6)
    sizes = list(range(1, 40)) + [61, 62, 63, 64, 65, 95, 96, 97, 111, 112, 113, 126, 127, 128, 129, 130, 143, 144, 145, 150]
    parts = [rng.uniform(-1.0, 1.0, 3) + rng.uniform(-1e-3, 1e-3, (k, 3)) for k in rng.permutation(sizes)]
    p = np.concatenate(parts)
    b = {k: np.ascontiguousarray(p[:, a]) for a, k in enumerate("xyz")}
    for k in ("vx", "vy", "vz"):
        b[k] = np.zeros(len(p))
    b["m"] = np.full(len(p), 1.0 / len(p))
    sim = Simulation("accurate", "fp64", leaf_cap=leaf_cap)
    sim.upload(b)
    t, r = sim.debug_tree(), oracle.tree(b, mode="accurate", leaf_cap=leaf_cap)
    assert t.shape == r.shape
    for c in (LEVEL, HALF, LEAF):
        np.testing.assert_array_equal(t[:, c], r[:, c])
    np.testing.assert_allclose(t[:, MASS], r[:, MASS], rtol=1e-14, atol=0)
    assert sim.stats()["device_error"] == 0
    sim.close()


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 148 * 1024, 148 * 1024 + 1, 148 * 2048, 148 * 2048 + 1, 148 * 4096,
                               148 * 4096 + 1, 148 * 7680, 148 * 7680 + 1])
def test_sort_at_the_layouts_edges(n):
    """Pairs at the sizes where the tile layout changes, most keys equal in most digits: stable order, bit for bit."""
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 62, n, dtype=np.uint64)
    keys[rng.random(n) < 0.5] &= np.uint64(0xff00ff)
    vals = np.arange(n, dtype=np.uint32)
    sim = Simulation("accurate", "mixed")
    for bits in (17, 63):
        ko, vo = sim.sort_pairs(keys, vals, bits)
        order = np.argsort(keys & np.uint64((1 << bits) - 1), kind="stable")
        np.testing.assert_array_equal(vo, vals[order])
        np.testing.assert_array_equal(ko, keys[order])
    sim.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097, 8192,
                               8193, 16383, 16384, 16385])
@pytest.mark.parametrize("bits", [1, 8, 13, 24, 63, 64])
def test_sort_in_one_launch(n, bits):
    """Small sorts at the edges of their blocks and clusters and with partial last digits, among them keys of all ones (as the padding
    behind the pairs): stable order by the low bits, bit for bit, by both entry points."""
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 2 ** 64, n, dtype=np.uint64, endpoint=False)
    keys[rng.random(n) < 0.3] = np.uint64(2 ** 64 - 1)
    vals = rng.integers(0, 2 ** 32, n, dtype=np.uint32)
    order = np.argsort(keys & np.uint64(2 ** bits - 1), kind="stable")
    sim = Simulation("accurate", "mixed")
    k, v = sim.sort_pairs(keys, vals, bits)
    np.testing.assert_array_equal(k, keys[order])
    np.testing.assert_array_equal(v, vals[order])
    sim.close()
    torch = pytest.importorskip("torch")
    src = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals.view(np.int32)).cuda()
    out = torch.empty_like(src[0]), torch.empty_like(src[1])
    rc = native.load().next_sort_pairs_noalloc(src[0].data_ptr(), src[1].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), n,
                                               bits, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    np.testing.assert_array_equal(out[0].cpu().numpy().view(np.uint64), keys[order])
    np.testing.assert_array_equal(out[1].cpu().numpy().view(np.uint32), vals[order])


@pytest.mark.parametrize("systems,top", [(3, 400), (40, 60), (5000, 6)])
def test_steps_of_many_systems(systems, top):
    """Root cubes boxed by the kick-drift (several systems in a warp's bodies, more systems than the last block
    takes): two steps of the batch equal two steps of a system alone."""
    rng = np.random.default_rng(systems)
    sizes = rng.integers(1, top, systems)
    b = ic.plummer(int(sizes.sum()), seed=systems)
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    sim = Simulation("accurate", "fp64", eps=0.05)
    sim.upload(b, offsets)
    sim.steps(1e-3, 2)
    s = sim.download()
    for i in (0, 1, systems // 2, systems - 1):
        at = slice(offsets[i], offsets[i + 1])
        one = Simulation("accurate", "fp64", eps=0.05)
        one.upload({k: v[at] for k, v in b.items()})
        one.steps(1e-3, 2)
        o = one.download()
        for k in s:
            np.testing.assert_array_equal(s[k][at], o[k])
        one.close()
    sim.close()


@pytest.mark.parametrize("kind", ["random", "lattice", "offset", "narrow", "plane", "huge"])
def test_keys_by_cell_number_equal_the_descent(oracle, kind):
    """Keys from cell numbers, with the level-by-level descent where a body is too near a cell boundary: on
    boundaries (lattice), far from the origin, with extents near the coordinates' rounding, in a plane, at 1e200."""
    rng = np.random.default_rng(11)
    n = 20011
    p = rng.uniform(-1.0, 1.0, (3, n))
    if kind == "lattice":
        p = np.round(p * 64.0) / 64.0
    elif kind == "offset":
        p = p * 1e-3 + np.array([[1e6], [-3e5], [7.0]])
    elif kind == "narrow":
        p = 1.0 + p * 1e-14
    elif kind == "plane":
        p[2] = 0.25
    elif kind == "huge":
        p = p * 1e200
    b = {"x": p[0].copy(), "y": p[1].copy(), "z": p[2].copy(), "m": np.full(n, 1.0 / n)}
    for k in ("vx", "vy", "vz"):
        b[k] = np.zeros(n)
    sim = Simulation("reference", "fp64")
    sim.upload(b)
    keys, cube = sim.debug_keys()
    np.testing.assert_array_equal(cube, oracle.root_cube(b))
    np.testing.assert_array_equal(keys, oracle.keys(b))
    sim.close()


def test_moments_of_buckets_of_every_remainder(oracle):
    """Leaves of the deepest level with more bodies than any leaf size, at every alignment and remainder of the loop
    over them: masses and centres of the oracle's tree (both sides round some thousand terms; one body left out of a
    bucket would move its centre by 1e-10)."""
    rng = np.random.default_rng(8)
    sizes = rng.permutation([*range(60, 84), 127, 128, 129, 1001, 1006, 1, 2, 3, 5])
    p = np.concatenate([rng.uniform(-1.0, 1.0, 3) + rng.uniform(-1e-7, 1e-7, (k, 3)) for k in sizes])
    b = {k: np.ascontiguousarray(p[:, a]) for a, k in enumerate("xyz")}
    for k in ("vx", "vy", "vz"):
        b[k] = np.zeros(len(p))
    b["m"] = rng.uniform(0.5, 1.5, len(p)) / len(p)
    sim = Simulation("accurate", "fp64", leaf_cap=4)
    sim.upload(b)
    t, r = sim.debug_tree(), oracle.tree(b, mode="accurate", leaf_cap=4)
    assert t.shape == r.shape
    leaves = r[:, LEAF] == 1
    np.testing.assert_array_equal(t[leaves, COUNT], r[leaves, COUNT])
    assert np.max(t[leaves, COUNT]) > 900 and np.sum(t[leaves, COUNT] > 64) > 15
    np.testing.assert_allclose(t[:, MASS], r[:, MASS], rtol=1e-12, atol=0)
    np.testing.assert_allclose(t[:, MASS + 1:MASS + 4], r[:, MASS + 1:MASS + 4], rtol=0, atol=1e-12)
    assert sim.stats()["device_error"] == 0
    sim.close()
