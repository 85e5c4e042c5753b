"""The calls that planners make on this backend, as cases to be timed.

A case names a kind of call and its sizes.  The kinds are the directions of
the backend: collision queries one call at a time and in batches (sphere arms
and point agents, device tensors and host arrays), nearest-neighbour and
radius queries on a node store, distance matrices, the penetration cost of
paths with its gradient, and the serving step of many planner instances.
Scenes are the package's synthetic ones (fixed per case); the inputs come from
the seed.
"""
import importlib
import math

import numpy as np
import torch

PKG = "multirobot-pathplanning-benchmark_gb300"
scenes = importlib.import_module(PKG + ".scenes")
env_mod = importlib.import_module(PKG + ".env")
knn_mod = importlib.import_module(PKG + ".knn")
cfg_mod = importlib.import_module(PKG + ".configuration")
pen_mod = importlib.import_module(PKG + ".penetration")
serving_mod = importlib.import_module(PKG + ".serving")

ARM_DIM, ARM_AGENTS, ARM_LINKS, ARM_SPHERES = 28, 4, 28, 168
ARM_PAIRS = 6 * 42 * 42
# box counts of arm scenes in which no box covers a fixed part of an arm
FEW_BOXES = (3, 4, 5, 6, 8, 10, 11, 13, 17, 20)
MANY_BOXES = (22, 26, 28, 30, 32, 34, 36, 38, 40, 46, 50, 52, 56, 58)


def listed():
    return [
        # RRT extension: the planner checks one sampled configuration and one
        # edge at a time, on numpy vectors; launches and waits count
        {"name": "single calls", "kind": "calls", "n": 32, "boxes": 5},
        # the abstract two-disc problems: a roadmap batch of edges from numpy
        {"name": "disc edges", "kind": "disc", "n": 1000, "boxes": 10},
        # rejection sampling of roadmap vertices: a large configuration batch
        {"name": "arm configurations", "kind": "configs", "n": 200_003, "boxes": 50, "f64": False},
        # candidate edges of a roadmap in a cluttered scene: most collide at
        # their first checked position; one in 32 is a short local edge
        {"name": "dense edges", "kind": "edges", "n": 100_000, "boxes": 50, "f64": False},
        # edges between free configurations: most are free, so every
        # interpolated position is checked; FP64 endpoints as planners hold them
        {"name": "sparse edges", "kind": "sparse", "n": 60_013, "boxes": 5, "f64": True},
        # roadmap construction: k neighbours of a batch of new vertices
        {"name": "knn euclidean", "kind": "knn", "q": 4096, "m": 200_000, "modes": 16, "k": 10,
         "metric": "euclidean"},
        # RRT*: nearest and radius query of one new sample, from numpy
        {"name": "one nearest and near", "kind": "rrt", "q": 1, "m": 200_000, "modes": 16, "k": 1,
         "metric": "euclidean"},
        # rewiring / connection sets: radius neighbours of a ragged batch
        {"name": "near max over agents", "kind": "near", "q": 2001, "m": 150_000, "modes": 16, "k": 16,
         "metric": "max_euclidean"},
        # cost-to-go tables: distances of all pairs, two 2-D agents
        {"name": "distance matrix", "kind": "dist", "q": 1000, "m": 10_000, "agents": 2, "per": 2,
         "metric": "euclidean"},
        # gradient repair of one shortcut candidate set: few short paths
        {"name": "small path gradient", "kind": "path", "p": 12, "t": 45, "boxes": 20},
        # path optimisation of a large batch
        {"name": "large path gradient", "kind": "path", "p": 512, "t": 256, "boxes": 50},
        # one step of 64 planner instances on the eight mobile manipulators
        {"name": "serving step", "kind": "serving", "instances": 64, "boxes": 60, "configs": 20_000, "edges": 5000,
         "steps": 800},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calls", "disc", "configs", "edges", "sparse", "knn", "rrt", "near", "dist", "path", "serving"])
    if kind == "calls":
        return {"kind": kind, "n": rng.randint(1, 48), "boxes": rng.choice(FEW_BOXES)}
    if kind == "disc":
        return {"kind": kind, "n": _log(rng, 10, 20_000), "boxes": rng.randint(3, 24)}
    if kind == "configs":
        return {"kind": kind, "n": _log(rng, 1000, 400_000),
                "boxes": rng.choice(FEW_BOXES + MANY_BOXES), "f64": rng.random() < 0.5}
    if kind == "edges":
        return {"kind": kind, "n": _log(rng, 1000, 120_000),
                "boxes": rng.choice(MANY_BOXES), "f64": rng.random() < 0.5}
    if kind == "sparse":
        return {"kind": kind, "n": _log(rng, 100, 90_000), "boxes": rng.choice(FEW_BOXES), "f64": rng.random() < 0.5}
    if kind in ("knn", "near"):
        return {"kind": kind, "q": _log(rng, 40, 4096), "m": _log(rng, 2000, 200_000), "modes": rng.randint(1, 24),
                "k": rng.randint(1, 16), "metric": rng.choice(["euclidean", "max_euclidean"])}
    if kind == "rrt":
        return {"kind": kind, "q": rng.randint(1, 8), "m": _log(rng, 500, 200_000), "modes": rng.randint(1, 24),
                "k": rng.randint(1, 8), "metric": rng.choice(["euclidean", "max_euclidean"])}
    if kind == "dist":
        return {"kind": kind, "q": _log(rng, 1, 1500), "m": _log(rng, 100, 15_000), "agents": rng.randint(1, 4),
                "per": rng.randint(2, 7),
                "metric": rng.choice(["euclidean", "sum_euclidean", "max_euclidean", "max"])}
    if kind == "path":
        return {"kind": kind, "p": _log(rng, 2, 512), "t": rng.randint(20, 256),
                "boxes": rng.choice(FEW_BOXES + MANY_BOXES)}
    return {"kind": kind, "instances": rng.randint(2, 48), "boxes": rng.randint(8, 70),
            "configs": _log(rng, 500, 20_000), "edges": _log(rng, 50, 5000), "steps": rng.randint(40, 800)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, lo=-math.pi, hi=math.pi, dtype=torch.float64):
    return (torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo).to(dtype)


def _arm_env(case, resolution):
    scene = scenes.make_arm_scene(1 if case["boxes"] in FEW_BOXES else 0, n_boxes=case["boxes"])
    return env_mod.Gb300ArmEnvironment(scene, collision_resolution=resolution)


def _free_configs(env, g, n, dtype):
    """n collision-free configurations, by rejection."""
    got, have = [], 0
    for _ in range(400):
        if have >= n:
            break
        q = _uniform(g, (max(4 * n, 4096), ARM_DIM), dtype=dtype)
        q = q[env.batch_is_collision_free(q)]
        got.append(q)
        have += len(q)
    if have < n:
        raise RuntimeError("could not draw enough collision-free configurations")
    return torch.cat(got)[:n].contiguous()


def _blocks(agents, per):
    return [[i * per, (i + 1) * per] for i in range(agents)]


def _store_inputs(case, seed):
    """Nodes in clusters, grouped by mode with Zipf sizes, and queries."""
    g = _gen(seed)
    m, modes, q = case["m"], case["modes"], case["q"]
    p = 1.0 / np.arange(1, modes + 1) ** 1.1
    p /= p.sum()
    sizes = np.floor(p * m).astype(np.int64)
    sizes[0] += m - sizes.sum()
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    centres = _uniform(g, (64, ARM_DIM))
    which = torch.randint(0, 64, (m,), generator=g, device="cuda")
    nodes = centres[which] + 0.3 * torch.randn((m, ARM_DIM), generator=g, device="cuda", dtype=torch.float64)
    queries = _uniform(g, (q, ARM_DIM))
    modes_q = np.random.default_rng(seed).choice(modes, q, p=p).astype(np.int32)
    return nodes, offsets, queries, modes_q


def _metric64(q, x, metric, slices):
    """Distances of rows q [Q, D] to rows x [M, D], 64 bits, in torch."""
    if metric == "max":
        return torch.cdist(q, x, p=float("inf"))
    if metric == "euclidean":
        return torch.cdist(q, x, compute_mode="donot_use_mm_for_euclid_dist")
    per = [torch.cdist(q[:, s:e].contiguous(), x[:, s:e].contiguous(), compute_mode="donot_use_mm_for_euclid_dist")
           for s, e in slices]
    d = torch.stack(per)
    return d.sum(0) if metric == "sum_euclidean" else d.max(0).values


def _by_query(nodes, offsets, queries, modes_q, metric, f):
    """f(distances to the query's mode) for blocks of queries of one mode;
    returns a list of per-query results in query order."""
    out = [None] * len(modes_q)
    for mode in np.unique(modes_q):
        x = nodes[int(offsets[mode]):int(offsets[mode + 1])]
        rows = np.nonzero(modes_q == mode)[0]
        for a in range(0, len(rows), 256):
            r = rows[a:a + 256]
            d = _metric64(queries[torch.from_numpy(r).cuda()], x, metric, _blocks(ARM_AGENTS, ARM_DIM // ARM_AGENTS))
            for i, v in zip(r, f(d, r)):
                out[i] = v
    return out


def _radii(nodes, offsets, queries, modes_q, metric, k):
    """Per query a radius that holds k nodes: halfway between the k-th and
    the next distance, so no node lies on it."""
    def between(d, _):
        n = d.shape[1]
        t = torch.topk(d, min(k + 1, n), dim=1, largest=False, sorted=True).values
        return (0.5 * (t[:, -1] + t[:, -2]) if t.shape[1] > 1 else 1.5 * t[:, 0]).cpu().tolist()
    return np.array(_by_query(nodes, offsets, queries, modes_q, metric, between))


def _paths(case, seed):
    """Straight lines between random configurations with a noise on the
    interior waypoints, as a shortcutter proposes them."""
    g = _gen(seed)
    p, t = case["p"], case["t"]
    e = _uniform(g, (2, p, 1, ARM_DIM))
    s = torch.linspace(0, 1, t, device="cuda", dtype=torch.float64)[None, :, None]
    w = e[0] + s * (e[1] - e[0])
    w[:, 1:-1] += 0.05 * torch.randn((p, t - 2, ARM_DIM), generator=g, device="cuda", dtype=torch.float64)
    return w.float().contiguous()


def _requests(case, seed, limits):
    """One step's requests of many planner instances, in host memory: uneven
    numbers of configurations and edges (a property of the case), edges with
    explicit step counts."""
    size, g = np.random.default_rng(case["instances"]), _gen(seed)
    lo = torch.as_tensor(limits[0], device="cuda")
    span = torch.as_tensor(limits[1], device="cuda") - lo

    def rows(n):
        u = torch.rand((n, len(lo)), generator=g, device="cuda", dtype=torch.float64)
        return (u * span + lo).float().cpu().numpy()

    out = []
    for _ in range(case["instances"]):
        nc, ne = int(size.integers(100, case["configs"] + 1)), int(size.integers(10, case["edges"] + 1))
        steps = torch.randint(5, case["steps"] + 1, (ne,), generator=g, device="cuda").cpu().numpy()
        out.append({"configs": rows(nc), "q1": rows(ne), "q2": rows(ne), "N": steps})
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "calls":
        env = _arm_env(case, 0.05)
        g = _gen(seed)
        a = _free_configs(env, g, case["n"], torch.float64)
        b = a + _uniform(g, a.shape, -0.6, 0.6)
        s |= {"env": env, "a": list(a.cpu().numpy()), "b": list(b.cpu().numpy())}
    elif kind == "disc":
        env = env_mod.Gb300AbstractEnvironment(scenes.make_disc_scene(0, case["boxes"]))
        r = np.random.default_rng(seed)
        s |= {"env": env, "a": r.uniform(-1, 1, (case["n"], 4)), "b": r.uniform(-1, 1, (case["n"], 4))}
    elif kind == "configs":
        dt = torch.float64 if case["f64"] else torch.float32
        s |= {"env": _arm_env(case, 0.05), "q": _uniform(_gen(seed), (case["n"], ARM_DIM), dtype=dt)}
    elif kind == "edges":
        dt = torch.float64 if case["f64"] else torch.float32
        g = _gen(seed)
        n = case["n"]
        steps = torch.exp(math.log(40.0) + 0.6 * torch.randn((n, 1), generator=g, device="cuda", dtype=torch.float64))
        a = _uniform(g, (n, ARM_DIM))
        b = a + _uniform(g, (n, ARM_DIM), -1.0, 1.0) * 0.05 * torch.clamp(torch.round(steps), 5, 500)
        env = _arm_env(case, 0.05)
        local = torch.arange(0, n, 32, device="cuda")
        a[local] = _free_configs(env, g, len(local), torch.float64)
        b[local] = a[local] + _uniform(g, (len(local), ARM_DIM), -0.15, 0.15)
        s |= {"env": env, "a": a.to(dt).contiguous(), "b": b.to(dt).contiguous()}
    elif kind == "sparse":
        dt = torch.float64 if case["f64"] else torch.float32
        env = _arm_env(case, 0.02)
        g = _gen(seed)
        a = _free_configs(env, g, case["n"], dt)
        b = (a.double() + _uniform(g, a.shape, -0.3, 0.3)).to(dt).contiguous()
        s |= {"env": env, "a": a, "b": b}
    elif kind in ("knn", "rrt", "near"):
        nodes, off, q, mq = _store_inputs(case, seed)
        store = knn_mod.NodeStore(nodes, off, _blocks(ARM_AGENTS, ARM_DIM // ARM_AGENTS), case["metric"])
        s |= {"store": store, "q": q, "mq": mq}
        if kind != "knn":
            s["radius"] = _radii(nodes, off, q, mq, case["metric"], 16 if kind == "rrt" else case["k"])
        if kind == "rrt":
            s["q"] = q.cpu().numpy()
    elif kind == "dist":
        g = _gen(seed)
        d = case["agents"] * case["per"]
        s |= {"q": _uniform(g, (case["q"], d), -1, 1), "x": _uniform(g, (case["m"], d), -1, 1),
              "sl": _blocks(case["agents"], case["per"])}
    elif kind == "path":
        s |= {"env": _arm_env(case, 0.05), "w": _paths(case, seed)}
    elif kind == "serving":
        sc = scenes.make_mobile_scene(0, n_boxes=case["boxes"])
        env = env_mod.Gb300ArmEnvironment(sc)
        req = _requests(case, seed, sc.limits)
        batcher = serving_mod.ServingBatcher(env._gb300)
        # the batcher captures its graph of this capacity once and keeps it
        batcher.step([{"configs": np.zeros_like(r["configs"]), "q1": np.zeros_like(r["q1"]),
                       "q2": np.zeros_like(r["q2"]), "N": np.full_like(r["N"], 2)} for r in req])
        s |= {"env": env, "batcher": batcher, "req": req}
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "calls":
        env, a, b = s["env"], s["a"], s["b"]
        free = np.zeros((2, len(a)), dtype=np.uint8)
        for i in range(len(a)):
            free[0, i] = env.is_collision_free(b[i], None)
            free[1, i] = env.is_edge_collision_free(a[i], b[i], None)
        return free
    if kind == "disc":
        return [s["env"].batch_is_collision_free(s["a"]), s["env"].batch_is_edge_collision_free(s["a"], s["b"])]
    if kind == "configs":
        return s["env"].batch_is_collision_free(s["q"])
    if kind in ("edges", "sparse"):
        return s["env"].batch_is_edge_collision_free(s["a"], s["b"])
    if kind == "knn":
        return s["store"].knn(s["q"], s["mq"], case["k"])
    if kind == "near":
        return s["store"].near(s["q"], s["mq"], s["radius"])
    if kind == "rrt":
        return [s["store"].knn(s["q"], s["mq"], case["k"]), s["store"].near(s["q"], s["mq"], s["radius"])]
    if kind == "dist":
        return cfg_mod.config_dist_matrix(s["q"], s["x"], s["sl"], case["metric"])
    if kind == "path":
        w = s["w"].detach().requires_grad_(True)
        cost = pen_mod.penetration_cost(w, s["env"]._gb300)
        (grad,) = torch.autograd.grad(cost.sum(), w)
        return [cost.detach(), grad]
    r = s["batcher"].step(s["req"])
    return [np.concatenate(r.config_free), np.concatenate(r.edge_free)]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    # one configuration of the four arms: forward kinematics, and one sphere
    # test where it collides or every test where it is free
    fk = 63 * ARM_LINKS + 18 * ARM_SPHERES
    hit = fk + 9
    full = fk + 9 * ARM_SPHERES * case.get("boxes", 0) + 9 * ARM_PAIRS
    wide = 8 if case.get("f64", True) else 4
    if kind == "calls":
        n = case["n"]
        return {"bytes": n * (2 * ARM_DIM * 8 + 2), "flops": n * 8 * full}
    if kind == "disc":
        n = case["n"]
        per = 2 * case["boxes"] * 8 + 8
        return {"bytes": n * (2 * 4 * 8 + 2), "flops": n * (1 + 50) * per}
    if kind == "configs":
        return {"bytes": case["n"] * (ARM_DIM * wide + 1), "flops": case["n"] * hit}
    if kind == "edges":
        return {"bytes": case["n"] * (2 * ARM_DIM * wide + 1), "flops": case["n"] * hit}
    if kind == "sparse":
        return {"bytes": case["n"] * (2 * ARM_DIM * wide + 1), "flops": case["n"] * 11 * full}
    if kind in ("knn", "near", "rrt"):
        q, m, modes = case["q"], case["m"], case["modes"]
        p = 1.0 / np.arange(1, modes + 1) ** 1.1
        p /= p.sum()
        pairs = float(q * m * (p * p).sum())
        out = 16 * q * case["k"]
        nodes = min(m, pairs) * ARM_DIM * 8
        return {"bytes": nodes + q * ARM_DIM * 8 + out, "flops": 3 * ARM_DIM * pairs * (2 if kind == "rrt" else 1)}
    if kind == "dist":
        d = case["agents"] * case["per"]
        q, m = case["q"], case["m"]
        return {"bytes": 8 * (q * m + (q + m) * d), "flops": 3.0 * d * q * m}
    if kind == "path":
        n = case["p"] * case["t"]
        pairs = ARM_SPHERES * case["boxes"] + ARM_PAIRS
        return {"bytes": n * ARM_DIM * 8 + 4 * case["p"], "flops": n * (3 * fk + 30 * pairs)}
    # serving: half the largest request per instance on average; mobile
    # manipulators of 72 coordinates, 48 links and 304 spheres
    nc, ne = case["instances"] * case["configs"] / 2, case["instances"] * case["edges"] / 2
    fk = 63 * 48 + 18 * 304
    return {"bytes": nc * (72 * 4 + 1) + ne * (2 * 72 * 4 + 9), "flops": (nc + ne) * (fk + 9)}


# ---------------------------------------------------------------------------
# 64-bit values of the floating outputs, in plain torch
# ---------------------------------------------------------------------------
def _centres64(a, q):
    """Sphere centres [W, S, 3] of fixed-base arms for q [W, D]: standard DH,
    frame k = frame k-1 * Rz(theta) Tz(d) Tx(a) Rx(alpha)."""
    t = {k: torch.as_tensor(np.asarray(v), device=q.device) for k, v in a.items() if v is not None}
    n = q.shape[0]
    out = torch.zeros((n, len(t["sphere_radius"]), 3), dtype=torch.float64, device=q.device)
    for r in range(len(t["q_offset"])):
        rot = t["base_pose"][r, :9].double().reshape(1, 3, 3).expand(n, 3, 3)
        pos = t["base_pose"][r, 9:].double().reshape(1, 3).expand(n, 3)
        for k in range(int(t["n_links"][r])):
            la, ld, ca, sa = (float(v) for v in t["dh"][r, k])
            th = q[:, int(t["q_offset"][r]) + k]
            x = rot[..., 0] * torch.cos(th)[:, None] + rot[..., 1] * torch.sin(th)[:, None]
            y = rot[..., 1] * torch.cos(th)[:, None] - rot[..., 0] * torch.sin(th)[:, None]
            z = rot[..., 2]
            pos = pos + ld * z + la * x
            rot = torch.stack([x, ca * y + sa * z, ca * z - sa * y], dim=-1)
            at = torch.nonzero((t["sphere_robot"] == r) & (t["sphere_link"] == k + 1)).reshape(-1)
            loc = t["sphere_local"][at].double()
            out = out.index_copy(1, at, pos[:, None, :] + torch.einsum("nij,sj->nsi", rot, loc))
    return out


def _path_exact(case, seed):
    a = scenes.make_arm_scene(1 if case["boxes"] in FEW_BOXES else 0, n_boxes=case["boxes"]).arrays()
    w = _paths(case, seed).double()
    rad = torch.as_tensor(np.asarray(a["sphere_radius"]), device="cuda").double()
    lo, hi = (torch.as_tensor(np.asarray(a[k]), device="cuda").double() for k in ("box_lo", "box_hi"))
    robot = torch.as_tensor(np.asarray(a["sphere_robot"]), device="cuda")
    i, j = torch.triu_indices(len(rad), len(rad), 1, device="cuda")
    keep = robot[i] != robot[j]
    i, j = i[keep], j[keep]
    margin, scale, weight = 0.02, 0.02, 0.1
    p, t, d = w.shape
    flat = w.reshape(-1, d)
    terms, grads = [], []
    for c in range(0, len(flat), 2048):
        q = flat[c:c + 2048].clone().requires_grad_(True)
        x = _centres64(a, q)
        off = torch.abs(x[:, :, None, :] - 0.5 * (lo + hi)) - 0.5 * (hi - lo)
        near = off.max(-1).values
        far = torch.sqrt(torch.clamp((torch.clamp(off, min=0) ** 2).sum(-1), min=1e-300))
        one = torch.nn.functional.softplus(margin - (torch.where(near > 0, far, near) - rad[:, None]), threshold=700)
        gap = torch.sqrt(((x[:, i] - x[:, j]) ** 2).sum(-1)) - rad[i] - rad[j]
        two = torch.nn.functional.softplus(margin - gap, threshold=700)
        e = (one.sum((1, 2)) + two.sum(1)) / scale
        (g,) = torch.autograd.grad(e.sum(), q)
        terms.append(e.detach())
        grads.append(g)
    cost = torch.cat(terms).reshape(p, t).sum(1)
    grad = torch.cat(grads).reshape(p, t, d)
    step = w[:, 1:] - w[:, :-1]
    cost = cost + weight * (step ** 2).sum((1, 2))
    grad[:, 1:] += 2 * weight * step
    grad[:, :-1] -= 2 * weight * step
    return [cost, grad]


def _store_exact(case, seed):
    nodes, off, q, mq = _store_inputs(case, seed)
    metric, k = case["metric"], case["k"]

    def nearest(d, _):
        t = torch.topk(d, min(k, d.shape[1]), dim=1, largest=False, sorted=True).values
        pad = torch.full((d.shape[0], k - t.shape[1]), math.inf, dtype=torch.float64, device="cuda")
        return list(torch.cat([t, pad], dim=1))

    knn = near = None
    if case["kind"] != "near":
        knn = [None, torch.stack(_by_query(nodes, off, q, mq, metric, nearest))]
    if case["kind"] != "knn":
        r = _radii(nodes, off, q, mq, metric, 16 if case["kind"] == "rrt" else k)

        def inside(d, rows):
            return [v[v <= r[i]] for v, i in zip(d, rows)]

        near = [None, None, torch.cat(_by_query(nodes, off, q, mq, metric, inside))]
    return [knn, near] if case["kind"] == "rrt" else near if case["kind"] == "near" else knn


def exact(case, seed):
    kind = case["kind"]
    if kind == "path":
        return _path_exact(case, seed)
    if kind in ("knn", "near", "rrt"):
        return _store_exact(case, seed)
    if kind == "dist":
        g = _gen(seed)
        d = case["agents"] * case["per"]
        q, x = _uniform(g, (case["q"], d), -1, 1), _uniform(g, (case["m"], d), -1, 1)
        return _metric64(q, x, case["metric"], _blocks(case["agents"], case["per"]))
    return None  # verdicts: no floating outputs
