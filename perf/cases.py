"""The work a user of this package has it do, as cases that can be timed and compared.

Every case goes through the package's public entry points: `Simulation` (create, upload, steps, step, step_host,
adaptive_dt, download, diagnostics) or the C ABI's device-buffer sort.  The sizes, opening angles, softenings and
time steps are those of the five workloads of `bench.py`, of the GPU tests, and odd sizes between them; leaf and
group sizes are what the autotuner picks for them (fixed here, so that two runs walk the same tree).

Bodies are drawn on the GPU from the case's seed.  They all move: a simulation spends its steps in motion, so the
collapsing sphere is taken part of the way into its collapse rather than at rest.
"""
import math

import numpy as np
import torch

from next_b200 import native

GPU = "cuda"
LANES = ("x", "y", "z", "vx", "vy", "vz")
# body-body and body-cell interactions per body that the walks need at 1 M bodies: the warp-group walk of the
# accurate physics (theta 0.5), one body per leaf of the same physics, and the reference's wider opening test
GROUP_PAIRS = (1100.0, 1200.0)
PLAIN_PAIRS = (150.0, 900.0)
REFERENCE_PAIRS = (40.0, 220.0)


def _sim(name, ic, n, steps, physics="accurate", precision="mixed", theta=0.5, eps=0.01, dt=1e-3, systems=1, leaf=0,
         group=0, warps=0, stack=0, path="steps"):
    return {"name": name, "path": path, "ic": ic, "n": n, "steps": steps, "physics": physics, "precision": precision,
            "theta": theta, "eps": eps, "dt": dt, "systems": systems, "leaf": leaf, "group": group, "warps": warps,
            "stack": stack}     # n: bodies (ensemble: of the largest system); leaf, group, warps, stack 0: defaults


def listed():
    return [
        # the smallest system of the batched ensemble on its own, untuned: launches and latency
        _sim("plummer_1k_mixed", "plummer", 1024, 1),
        # the plain FP64 method at its configured size
        _sim("plummer_16k_fp64", "plummer", 16384, 2, precision="fp64"),
        # the same bodies with FP32 interactions and the autotuned small-system groups
        _sim("plummer_16k_mixed", "plummer", 16384, 4, leaf=8, group=8, warps=4, stack=640),
        # the flagship workload: a million-body collapse, a short run and a snapshot
        _sim("collapse_1m_mixed", "infall", 1048576, 2, eps=0.005, dt=5e-4, leaf=16, group=32, warps=2, stack=896),
        # its plain FP64 form, the comparator of the flagship workload
        _sim("collapse_1m_fp64", "infall", 1048576, 1, precision="fp64", eps=0.005, dt=5e-4),
        # FP64 interactions in the group walk, an odd size, with the energy check that follows a run
        _sim("collapse_262k_fp64group", "infall", 262143, 1, precision="fp64group", eps=0.005, dt=5e-4, leaf=16,
             group=32, warps=4, stack=1024, path="energy"),
        # two disk galaxies: strongly clustered, two centres, a deep tree
        _sim("galaxies_4m_mixed", "galaxies", 4194304, 1, theta=0.6, leaf=16, group=32, warps=2, stack=1088),
        # 256 independent spheres of uneven size in one batch
        _sim("ensemble_256_mixed", "ensemble", 65536, 1, systems=256, leaf=16, group=32, warps=2, stack=1280),
        # the largest single system
        _sim("halo_16m_mixed", "halo", 16777216, 2, theta=0.7, eps=0.002, dt=2.5e-4, leaf=24, group=32, warps=4,
             stack=768),
        # the drop-in Step() on the caller's own arrays: reference physics, a fifth of the bodies dark matter
        _sim("reference_64k_host", "plummer", 65536, 1, physics="reference", precision="fp64", path="host"),
        # the reference's main loop, adaptive time step and Step(), with the bodies kept on the device
        _sim("reference_1m_loop", "infall", 1048576, 1, physics="reference", precision="fp64", dt=5e-4, path="loop"),
        # the key sort alone, between the caller's device buffers: full-depth octant keys
        {"name": "sort_1m_pairs", "path": "sort", "n": 1048576, "bits": 63},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("mixed", "mixed", "mixed", "ensemble", "fp64", "fp64group", "reference", "reference", "sort"))
    if kind == "sort":
        return {"path": "sort", "n": _log_uniform(rng, 1000, 1048576), "bits": rng.randint(24, 64)}
    if kind == "reference":
        c = _sim("", rng.choice(("plummer", "infall")), _log_uniform(rng, 1000, 1100000), 1, physics="reference",
                 precision="fp64", dt=5e-4, path=rng.choice(("host", "loop")))
    elif kind == "fp64":
        c = _sim("", rng.choice(("plummer", "infall")), _log_uniform(rng, 1000, 300000), 1, precision="fp64",
                 theta=rng.choice((0.5, 0.6, 0.7)), eps=0.005, dt=5e-4)
    elif kind == "fp64group":
        c = _sim("", rng.choice(("plummer", "infall", "halo")), _log_uniform(rng, 1000, 1100000), 1,
                 precision="fp64group", theta=rng.choice((0.5, 0.6, 0.7)), eps=0.005, dt=5e-4,
                 path=rng.choice(("steps", "energy")))
    elif kind == "ensemble":
        c = _sim("", "ensemble", _log_uniform(rng, 2048, 65536), 1, systems=_log_uniform(rng, 8, 256), leaf=16,
                 group=32, warps=2, stack=1280)
    else:
        n = _log_uniform(rng, 1000, 4200000)
        c = _sim("", rng.choice(("plummer", "infall", "halo", "galaxies")), n, rng.randint(1, 2),
                 theta=rng.choice((0.5, 0.6, 0.7)), eps=rng.choice((0.005, 0.01)), dt=5e-4)
        if n <= 65536 and rng.random() < 0.7:
            c.update(leaf=8, group=8, warps=4, stack=640)
        elif rng.random() < 0.7:
            c.update(leaf=rng.choice((16, 24)), group=32, warps=rng.choice((2, 4)), stack=1088)
    del c["name"]
    return c


# ---- bodies ---------------------------------------------------------------------------------------------------------

def _uniform(g, n):
    return torch.rand(n, generator=g, device=GPU, dtype=torch.float64).clamp_(1e-12, 1.0 - 1e-12)


def _isotropic(g, r):
    c = 2.0 * _uniform(g, r.numel()) - 1.0
    s = torch.sqrt(1.0 - c * c)
    phi = 2.0 * math.pi * _uniform(g, r.numel())
    return r * s * torch.cos(phi), r * s * torch.sin(phi), r * c


def _speed_fraction(g, n):
    """v / v_escape with density q^2 (1 - q^2)^3.5, as of an isotropic sphere in equilibrium: sqrt of a beta variate."""
    # q^2 ~ Beta(3/2, 9/2), from gamma variates of shape 3/2 and 9/2 (halves of chi-squares with 3 and 9 degrees)
    z = torch.randn((12, n), generator=g, device=GPU, dtype=torch.float64).square_()
    a = z[:3].sum(0)
    return torch.sqrt(a / (a + z[3:].sum(0)))


def _plummer(g, n, a=1.0, mass=1.0):
    top = (1.0 + 1.0 / 400.0) ** -1.5                      # mass fraction inside 20 scale radii
    r = a / torch.sqrt((top * _uniform(g, n)) ** (-2.0 / 3.0) - 1.0)
    v = _speed_fraction(g, n) * math.sqrt(2.0 * mass / a) * (1.0 + (r / a) ** 2) ** -0.25
    return [*_isotropic(g, r), *_isotropic(g, v), torch.full_like(r, mass / n)]


def _halo(g, n, a=1.0, mass=1.0):
    """Hernquist profile inside 50 scale radii, isotropic speeds below the escape speed."""
    s = torch.sqrt((50.0 / 51.0) ** 2 * _uniform(g, n))
    r = a * s / (1.0 - s)
    v = _speed_fraction(g, n) * torch.sqrt(2.0 * mass / (r + a))
    return [*_isotropic(g, r), *_isotropic(g, v), torch.full_like(r, mass / n)]


def _infall(g, n):
    """The cold sphere when it has fallen to 0.8 of its first radius: uniform density, speed along the radius and a
    slow turn about a tilted axis."""
    x, y, z = _isotropic(g, 0.8 * _uniform(g, n) ** (1.0 / 3.0))
    h, (a, b, c) = -math.sqrt(2.0 * (1.0 / 0.8 - 1.0)) / 0.8, (0.1, 0.15, 0.2)
    return [x, y, z, h * x + b * z - c * y, h * y + c * x - a * z, h * z + a * y - b * x, torch.full_like(x, 1.0 / n)]


def _galaxy(g, n):
    """Exponential disk (60%, thickness 0.1), Plummer bulge (10%, a = 0.2), Hernquist halo (30%, a = 5)."""
    nd, nb = int(0.6 * n), int(0.1 * n)
    nh = n - nd - nb
    md, mb, mh = nd / n, nb / n, nh / n
    R = -torch.log(_uniform(g, nd) * _uniform(g, nd))
    phi = 2.0 * math.pi * _uniform(g, nd)
    z = 0.1 * torch.atanh(1.999 * _uniform(g, nd) - 0.9995)
    rs = torch.sqrt(R * R + z * z)
    inside = md * (1.0 - (1.0 + R) * torch.exp(-R)) + mb * rs ** 3 / (rs * rs + 0.04) ** 1.5 + mh * rs * rs / (rs + 5.0) ** 2
    vc = torch.sqrt(inside / rs)
    disk = [R * torch.cos(phi), R * torch.sin(phi), z, -vc * torch.sin(phi), vc * torch.cos(phi), torch.zeros_like(R),
            torch.full_like(R, md / max(nd, 1))]
    parts = (disk, _plummer(g, nb, 0.2, mb), _halo(g, nh, 5.0, mh))
    return [torch.cat([p[k] for p in parts]) for k in range(7)]


def _galaxies(g, n):
    """Two such galaxies 30 apart on a parabolic orbit, the second one's disk tilted by 60 degrees."""
    a, b = _galaxy(g, n // 2), _galaxy(g, n - n // 2)
    c, s = math.cos(math.pi / 3.0), math.sin(math.pi / 3.0)
    for p, q in ((1, 2), (4, 5)):
        b[p], b[q] = c * b[p] - s * b[q], s * b[p] + c * b[q]
    vt = math.sqrt(20.0) / 30.0
    vr = -math.sqrt(4.0 / 30.0 - vt * vt)
    for lanes, side in ((a, -0.5), (b, 0.5)):
        lanes[0] = lanes[0] + 30.0 * side
        lanes[3] = lanes[3] + vr * side
        lanes[4] = lanes[4] + vt * side
    return [torch.cat([p, q]) for p, q in zip(a, b)]


def _bodies(case, seed):
    """Seven FP64 lanes x y z vx vy vz m on the GPU, int32 types, and the systems' offsets (None for one system)."""
    g = torch.Generator(device=GPU).manual_seed(seed)
    n, offsets = case["n"], None
    if case["ic"] == "ensemble":
        # sizes log-uniform over up to a factor of 64 below the largest one, the same for every seed
        u = np.random.default_rng(3).uniform(0.0, 1.0, case["systems"])
        lo = max(256, n // 64)
        sizes = np.exp(math.log(lo) + u * math.log(n / lo)).astype(np.int64)
        offsets = np.concatenate([[0], np.cumsum(sizes)])
        lanes = _plummer(g, int(offsets[-1]))
        lanes[6] = torch.from_numpy(np.repeat(1.0 / sizes, sizes)).to(GPU)
    else:
        lanes = {"plummer": _plummer, "halo": _halo, "infall": _infall, "galaxies": _galaxies}[case["ic"]](g, n)
    types = torch.zeros(lanes[0].numel(), dtype=torch.int32, device=GPU)
    if case["physics"] == "reference":
        types[::5] = 1
    return lanes, types, offsets


# ---- the cases ------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    if case["path"] == "sort":
        g = torch.Generator(device=GPU).manual_seed(seed)
        n = case["n"]
        keys = torch.randint(0, 1 << 62, (n,), generator=g, device=GPU) * 2 + torch.randint(0, 2, (n,), generator=g, device=GPU)
        vals = torch.arange(n, dtype=torch.int32, device=GPU)
        return {"case": case, "lib": native.load(), "in": (keys, vals), "out": (torch.empty_like(keys), torch.empty_like(vals))}
    lanes, types, offsets = _bodies(case, seed)
    lanes = [v.cpu().numpy() for v in lanes]
    types = types.cpu().numpy()
    knobs = {"leaf_cap": case["leaf"], "group_cap": case["group"], "walk_warps": case["warps"], "walk_stack": case["stack"]}
    knobs = {k: v for k, v in knobs.items() if v}
    if case["physics"] == "accurate":
        knobs["eps"] = case["eps"]
    sim = native.Simulation(case["physics"], case["precision"], theta=case["theta"], **knobs)
    state = {"case": case, "sim": sim}
    if case["path"] == "host":
        state.update(lanes=lanes, types=types)
        return state
    sim.upload(dict(zip(LANES + ("m",), lanes), type=types), offsets)
    state["out"] = {k: torch.empty(types.shape[0], dtype=torch.float64, pin_memory=True).numpy() for k in LANES}
    return state


def run(state):
    case = state["case"]
    if case["path"] == "sort":
        (keys, vals), (ko, vo) = state["in"], state["out"]
        rc = state["lib"].next_sort_pairs_noalloc(keys.data_ptr(), vals.data_ptr(), ko.data_ptr(), vo.data_ptr(), case["n"],
                                                  case["bits"], torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(f"sort failed ({rc})")
        return ko, vo
    sim, dt = state["sim"], case["dt"]
    if case["path"] == "host":
        for _ in range(case["steps"]):
            sim.step_host(state["lanes"], dt, state["types"])
        return state["lanes"][:6]
    if case["path"] == "loop":
        for _ in range(case["steps"]):
            dt = sim.adaptive_dt(case["dt"])
            sim.step(dt)
        return {**sim.download(state["out"]), "dt": dt}
    sim.steps(dt, case["steps"])
    out = dict(sim.download(state["out"]))
    if case["path"] == "energy":
        out.update(sim.diagnostics())
    return out


def _count(case):
    if case["ic"] == "ensemble":
        lo = max(256, case["n"] // 64)
        span = math.log(case["n"] / lo)
        return case["systems"] * (case["n"] - lo) / span if span > 0 else case["systems"] * case["n"]
    return case["n"]


def work(case):
    if case["path"] == "sort":
        return {"bytes": 24.0 * case["n"], "flops": 0.0}
    n = _count(case)
    if case["physics"] == "reference":
        pairs = REFERENCE_PAIRS
    else:
        pairs = PLAIN_PAIRS if case["precision"] == "fp64" else GROUP_PAIRS
    # interactions per body grow with the logarithm of the body count and fall with the opening angle
    scale = math.log(max(n / case["systems"], 64.0)) / math.log(1048576.0) * (0.5 / case["theta"]) ** 2
    forces = case["steps"]                                   # one force evaluation a step: the one before is known
    if case["path"] == "energy":
        forces += 1                                          # the potential
    flops = n * scale * forces * (20.0 * pairs[0] + 56.0 * pairs[1])
    # a step reads and writes positions and velocities and reads masses; the state leaves once
    return {"bytes": n * (case["steps"] * 104.0 + 48.0), "flops": flops}


# ---- values in 64 bits ----------------------------------------------------------------------------------------------

def _direct(lanes, mass, offsets, eps):
    """Softened direct summation, system by system: accelerations and potential."""
    acc = [torch.zeros_like(mass) for _ in range(4)]
    for s, e in zip(offsets[:-1], offsets[1:]):
        p = [v[s:e] for v in lanes]
        m = mass[s:e]
        rows = max(1, (1 << 26) // int(e - s))
        for i in range(0, int(e - s), rows):
            d = [v[None, :] - v[i:i + rows, None] for v in p]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps * eps
            w = m / torch.sqrt(r2)
            acc[3][s + i:s + i + rows] = m[i:i + rows] / eps - w.sum(1)
            w = w / r2
            for k in range(3):
                acc[k][s + i:s + i + rows] = (w * d[k]).sum(1)
    return acc


def _octree(p, m):
    """The one-body-per-leaf octree over the root cube, with the reference's moments: per node mass, centre of mass,
    half-width, quadrupole, children range and body (-1 for a cell)."""
    n = m.numel()
    lo, hi = [v.min() for v in p], [v.max() for v in p]
    c = [((a + b) * 0.5).expand(n).clone() for a, b in zip(lo, hi)]
    h0 = float(max((b - a) for a, b in zip(lo, hi)) * 0.5)
    h, key = h0, torch.zeros(n, dtype=torch.int64, device=m.device)
    for _ in range(21):
        bits = [v > w for v, w in zip(p, c)]
        key = key * 8 + bits[0].long() + 2 * bits[1].long() + 4 * bits[2].long()
        h *= 0.5
        c = [w + torch.where(b, h, -h) for w, b in zip(c, bits)]
    order = torch.argsort(key, stable=True)
    key = key[order]
    start, count = torch.zeros(1, dtype=torch.int64, device=m.device), torch.full((1,), n, dtype=torch.int64, device=m.device)
    levels = []                                              # (start, count, index of the parent in the level above)
    parent = torch.full((1,), -1, dtype=torch.int64, device=m.device)
    for level in range(22):
        levels.append((start, count, parent))
        split = (count > 1).nonzero().squeeze(1) if level < 21 else start[:0]
        if split.numel() == 0:
            break
        pre = key >> (3 * (20 - level))
        first = torch.ones(n, dtype=torch.bool, device=m.device)
        first[1:] = pre[1:] != pre[:-1]
        begin = first.nonzero().squeeze(1)
        end = torch.cat([begin[1:], torch.full((1,), n, device=m.device)])
        owner = torch.searchsorted(start, begin, right=True) - 1
        inside = (owner >= 0) & (begin < (start + count)[owner]) & (count[owner] > 1)
        start, count, parent = begin[inside], (end - begin)[inside], owner[inside]
    base = np.concatenate([[0], np.cumsum([s.numel() for s, _, _ in levels])])
    total = int(base[-1])
    body = torch.full((total,), -1, dtype=torch.int64, device=m.device)
    child = torch.zeros((total, 2), dtype=torch.int64, device=m.device)
    mom = torch.zeros((total, 4), dtype=torch.float64, device=m.device)
    quad = torch.zeros((total, 6), dtype=torch.float64, device=m.device)
    half = torch.cat([torch.full((s.numel(),), h0 * 0.5 ** l, dtype=torch.float64, device=m.device)
                      for l, (s, _, _) in enumerate(levels)])
    state = torch.stack([m, *p], 1)[order]
    for l in range(len(levels) - 1, -1, -1):
        s, cnt, _ = levels[l]
        at = slice(int(base[l]), int(base[l + 1]))
        one = cnt == 1
        body[at] = torch.where(one, order[s], body[at])
        mine = torch.where(one[:, None], state[s], torch.zeros_like(state[s]))
        q = quad[at].clone()
        if l + 1 < len(levels):
            par, below = levels[l + 1][2], slice(int(base[l + 1]), int(base[l + 2]))
            num = torch.bincount(par, minlength=s.numel())
            child[at] = torch.stack([int(base[l + 1]) + torch.cumsum(num, 0) - num, num], 1)
            k = mom[below]
            tot = torch.zeros_like(mine).index_add_(0, par, torch.cat([k[:, :1], k[:, :1] * k[:, 1:]], 1))
            com = tot[:, 1:] / torch.where(tot[:, :1] > 0, tot[:, :1], torch.ones_like(tot[:, :1]))
            mine = torch.where(one[:, None], mine, torch.cat([tot[:, :1], com], 1))
            r = k[:, 1:] - com[par]
            r2 = (r * r).sum(1) + half[at][par] ** 2 * 0.01
            term = torch.stack([3 * r[:, 0] ** 2 - r2, 3 * r[:, 1] ** 2 - r2, 3 * r[:, 2] ** 2 - r2, 3 * r[:, 0] * r[:, 1],
                                3 * r[:, 0] * r[:, 2], 3 * r[:, 1] * r[:, 2]], 1) * k[:, :1]
            q.index_add_(0, par, term)
        mom[at], quad[at] = mine, q
    return mom, quad, half, child, body


def _reference_forces(p, m, types, theta):
    """The reference's own Barnes-Hut force: half-width opening test, softening by cell size, mass and distance."""
    mom, quad, half, child, body = _octree(p, m)
    n = m.numel()
    acc = torch.zeros((n, 3), dtype=torch.float64, device=m.device)
    pos = torch.stack(p, 1)
    for i0 in range(0, n, 32768):
        who = torch.arange(i0, min(n, i0 + 32768), device=m.device)
        node = torch.zeros_like(who)
        while who.numel():
            d = mom[node, 1:] - pos[who]
            r2 = (d * d).sum(1)
            dist = torch.sqrt(r2 + 1e-20)
            leaf = child[node, 1] == 0
            near = leaf | (half[node] / dist < theta)
            use = near & ~(leaf & (body[node] == who)) & (mom[node, 0] != 0)
            w, k, e, s2, ds = who[use], node[use], d[use], r2[use], dist[use]
            mass, size, q = mom[k, 0], half[k], quad[k]
            eps = torch.clamp((size * 0.015 + mass ** (1.0 / 3.0) * 0.002) / (1.0 + 10.0 * ds), min=1e-4)
            dark = 2.0 * size / (mass / m[w]) ** 0.333333333
            eps = torch.where(types[w] == 1, torch.maximum(eps, dark), eps)
            inv2 = 1.0 / (s2 + eps * eps)
            inv3 = inv2 * torch.sqrt(inv2)
            inv5 = inv3 * inv2
            x, y, z = e[:, 0], e[:, 1], e[:, 2]
            qr = 2.0 * torch.stack([q[:, 0] * x + q[:, 3] * y + q[:, 4] * z, q[:, 3] * x + q[:, 1] * y + q[:, 5] * z,
                                    q[:, 4] * x + q[:, 5] * y + q[:, 2] * z], 1)
            qs = 0.5 * (qr * e).sum(1)
            f = (mass * inv3)[:, None] * e + 0.5 * (qr * inv5[:, None] - (5.0 * qs * inv5 * inv2)[:, None] * e)
            acc.index_add_(0, w, f)
            more = ~near & (mom[node, 0] != 0)
            who, node = who[more], node[more]
            num = child[node, 1]
            off = torch.arange(int(num.sum()), device=m.device) - torch.repeat_interleave(torch.cumsum(num, 0) - num, num)
            who, node = torch.repeat_interleave(who, num), torch.repeat_interleave(child[node, 0], num) + off
    return [acc[:, k].contiguous() for k in range(3)]


def exact(case, seed):
    """Leapfrog steps in 64 bits: by direct summation for the accurate physics (what its tree approximates), by a
    plain tree walk for the reference's physics (whose softening depends on the tree)."""
    if case["path"] == "sort":
        return None
    if case["physics"] == "accurate":
        per = _count(case) / case["systems"]
        spread = 3.0 if case["systems"] > 1 else 1.0         # mean square over squared mean of the uneven sizes
        if spread * per * per * case["systems"] * (case["steps"] + 1) > 2.5e11:
            return None
    lanes, types, offsets = _bodies(case, seed)
    p, v, m = lanes[:3], lanes[3:6], lanes[6]
    if offsets is None:
        offsets = np.array([0, m.numel()])

    def forces():
        if case["physics"] == "reference":
            return _reference_forces(p, m, types, case["theta"])
        return _direct(p, m, offsets, case["eps"])

    dt, acc = case["dt"], forces()
    for _ in range(case["steps"]):
        if case["path"] == "loop":
            top = min(math.sqrt(float((v[0] ** 2 + v[1] ** 2 + v[2] ** 2).max())), 1e4)
            dt = case["dt"] if top < 1e-8 else min(max(case["dt"] / (1.0 + top), case["dt"] * 0.01), case["dt"])
        v = [a + b * (0.5 * dt) for a, b in zip(v, acc)]
        p = [a + b * dt for a, b in zip(p, v)]
        acc = forces()
        v = [a + b * (0.5 * dt) for a, b in zip(v, acc)]
    if case["path"] == "host":
        return [*p, *v]
    out = dict(zip(LANES, [*p, *v]))
    if case["path"] == "loop":
        out["dt"] = dt
    if case["path"] == "energy":
        out["kinetic"] = float(0.5 * (m * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)).sum())
        out["potential"] = float(0.5 * (m * acc[3]).sum())
        out["momentum"] = torch.stack([(m * a).sum() for a in v])
        spin = [(p[a] * v[b] - p[b] * v[a]) * m for a, b in ((1, 2), (2, 0), (0, 1))]
        out["angular_momentum"] = torch.stack([a.sum() for a in spin])
    return out
