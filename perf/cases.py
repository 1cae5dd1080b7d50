"""The work that users have this package do, as cases that can be timed: planners that check one
motion or a few hundred at a time from host memory, batch callers that check tens of thousands of
motions or a million configurations on the GPU, perception loops that filter a cloud and build its
tree, and the learned block order's training and use.

A case is a dict of plain values; `prepare` makes what the caller's program holds before the call,
`run` makes the call through the package's public entry points, `work` says what it cannot do
without, and `exact` gives float64 values where outputs are computed numbers (the verdicts,
block counts and kept points of the other cases are whole numbers or copies of inputs).
"""
from __future__ import annotations

import math

import numpy as np

ROBOTS = ("panda", "ur5", "fetch", "baxter")
POINTS = 50_000  # points of a scene's cloud
WIDTH = 256  # width of the learned order's hidden layers

# Per robot: joints, sphere slots, coarse link spheres, self-checked link pairs, states per radian
# (resolution) and the mean joint-space distance of two uniform configurations.
SHAPE = {
    "panda": (7, 70, 11, 21, 32, 5.3),
    "ur5": (6, 57, 17, 55, 32, 6.1),
    "fetch": (8, 126, 15, 48, 32, 5.2),
    "baxter": (14, 108, 33, 349, 64, 7.0),
}


def listed() -> list[dict]:
    return [
        # A planner's extension steps: 32 motions one after the other, host arrays, each answer
        # needed before the next.
        {"name": "steps_32", "kind": "steps", "robot": "panda", "n": 32, "length": 1.0, "points": 0},
        # FCIT*'s lazy edge checks: a node's 256 nearest neighbours in one call, host arrays.
        {"name": "neighbours_256", "kind": "host_edges", "robot": "panda", "n": 256, "length": 1.2, "points": 0},
        # The whole roadmap's motions at once: uneven lengths, 60 primitives, verdicts and block
        # counts (the benchmark's headline workload).
        {"name": "motions_65536", "kind": "edges", "robot": "panda", "n": 65536, "points": 0, "lanes": 8, "counts": True},
        # Fetch at a ragged batch size among primitives and a scanned cloud.
        {"name": "motions_fetch_cloud", "kind": "edges", "robot": "fetch", "n": 12345, "points": POINTS, "lanes": 8,
         "counts": False},
        # Callers that give start, vector and length, with the Arm build's semantics (4 lanes,
        # exact square root).
        {"name": "vectors_arm_lanes", "kind": "vectors", "robot": "ur5", "n": 9973, "points": 0, "lanes": 4},
        # A carried object over terrain: attachment, heightfield and primitives in one scene.
        {"name": "motions_carrying", "kind": "carry", "robot": "panda", "n": 8191, "lanes": 8},
        # Sampling in a scanned scene: a million configurations against a 50,000-point cloud.
        {"name": "states_cloud_1m", "kind": "states", "robot": "panda", "n": 1048576, "points": POINTS},
        # Four robots' batches replayed as one graph, primitives and a cloud each.
        {"name": "four_robots", "kind": "mixed", "n": 16384},
        # A depth camera's frame: filter a million points, build the tree, check configurations.
        {"name": "camera_frame", "kind": "sense", "robot": "panda", "n": 1048576, "cull": True, "states": 4096},
        # A PRM* roadmap from 16,384 samples: neighbours, candidate motions, verdicts.
        {"name": "roadmap_16384", "kind": "roadmap", "robot": "panda", "n": 16384},
        # The headline motions in the learned block order, 8 probes a motion.
        {"name": "learned_order", "kind": "learned", "robot": "panda", "n": 65536, "probes": 8},
        # Fitting the learned order's network to a scene's labels: one epoch of 1,024-row batches.
        {"name": "train_order", "kind": "train", "robot": "panda", "n": 65536, "batch": 1024},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(("steps", "host_edges", "edges", "edges", "vectors", "carry", "states", "states", "mixed", "sense",
                       "roadmap", "learned", "train"))
    robot = rng.choice(ROBOTS)
    points = rng.choice((0, POINTS))
    top = 16384 if robot == "baxter" else 65536
    if kind == "steps":
        return {"kind": kind, "robot": robot, "n": 32, "length": round(rng.uniform(0.05, 4.0), 3), "points": points}
    if kind == "host_edges":
        return {"kind": kind, "robot": robot, "n": _log(rng, 2, 2048), "length": round(rng.uniform(0.2, 3.0), 3),
                "points": points}
    if kind == "edges":
        return {"kind": kind, "robot": robot, "n": _log(rng, 100, top), "points": points, "lanes": rng.choice((8, 8, 4)),
                "counts": rng.random() < 0.5}
    if kind == "vectors":
        return {"kind": kind, "robot": robot, "n": _log(rng, 100, top), "points": points, "lanes": rng.choice((8, 4))}
    if kind == "carry":
        return {"kind": kind, "robot": robot, "n": _log(rng, 100, top // 8), "lanes": rng.choice((8, 8, 4))}
    if kind == "states":
        return {"kind": kind, "robot": robot, "n": _log(rng, 1024, 1048576 if robot != "baxter" else 262144), "points": points}
    if kind == "mixed":
        return {"kind": kind, "n": _log(rng, 256, 16384)}
    if kind == "sense":
        return {"kind": kind, "robot": "panda", "n": _log(rng, 20000, 1048576), "cull": rng.random() < 0.7,
                "states": _log(rng, 64, 65536)}
    if kind == "roadmap":
        return {"kind": kind, "robot": rng.choice(("panda", "ur5", "fetch")), "n": _log(rng, 1000, 16384)}
    if kind == "learned":
        return {"kind": kind, "robot": rng.choice(("panda", "ur5", "fetch")), "n": _log(rng, 4096, 65536),
                "probes": rng.choice((4, 8, 16))}
    batch = rng.choice((512, 1024, 2048))
    return {"kind": "train", "robot": robot, "n": batch * _log(rng, 4, 65536 // batch), "batch": batch}


# ------------------------------------------------------------------------------------- inputs

def _device(x):
    import torch

    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _environment(robot, seed: int, points: int, lanes: int = 8, primitives: bool = True, extra=None):
    """24 spheres, 24 cuboids and 12 capsules around the robot, a cloud whose tree is built on the
    GPU, and what `extra(env, seed)` adds.  Scenes that leave the robot no room (fewer than one
    uniform configuration in ten valid) are drawn again."""
    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    mode = vg.SQRT_X86 if lanes == 8 else vg.SQRT_EXACT
    probe = scenes.configurations(robot.s_m, robot.s_a, 1024, seed)
    for k in range(64):
        s = seed + 104729 * k
        env = vg.Environment.from_scene(scenes.scene_config1(s) if primitives else {}, lanes, mode)
        if points:
            lo, hi = robot.min_max_radii()
            env.add_pointcloud_device(_device(scenes.surface_pointcloud(s, points)), lo, hi, scenes.POINT_RADIUS)
        if extra:
            extra(env, s)
        if robot.validate_batch(probe, env).mean() >= 0.1:
            return env
    raise RuntimeError(f"no scene leaves the {robot.name} room to move")


def _short_edges(robot, n: int, length: float, seed: int):
    """Starts uniform in the joint limits, goals about `length` radians away, inside the limits."""
    from vamp_gb300 import scenes

    rng = np.random.default_rng(seed)
    a = scenes.configurations(robot.s_m, robot.s_a, n, seed)
    v = rng.normal(size=a.shape)
    v *= length * rng.uniform(0.5, 1.5, size=(n, 1)) / np.linalg.norm(v, axis=1, keepdims=True)
    margin = 1e-3 * robot.s_m
    b = np.clip(a + v, robot.s_a + margin, robot.s_a + robot.s_m - margin).astype(np.float32)
    return a, b


def _train_inputs(robot, n: int, seed: int):
    """Configurations, labels of a fixed random two-layer function of them (about half of them
    valid), and He-uniform weights in the package's order: W1, b1, W2, b2, w3, b3."""
    from vamp_gb300 import scenes

    dim = robot.dimension()
    rng = np.random.default_rng(seed + 17)
    q = scenes.configurations(robot.s_m, robot.s_a, n, seed)
    f = np.stack([np.sin(q), np.cos(q)], axis=2).reshape(n, 2 * dim)
    t = np.tanh(f @ (rng.normal(size=(2 * dim, 32)) * 1.5)) @ rng.normal(size=32)
    valid = (t > np.median(t)).astype(np.uint8)
    kin = (2 * dim + 15) // 16 * 16
    w1 = np.zeros((WIDTH, kin))
    w1[:, :2 * dim] = rng.uniform(-1, 1, size=(WIDTH, 2 * dim)) * math.sqrt(3.0 / dim)
    w2 = rng.uniform(-1, 1, size=(WIDTH, WIDTH)) * math.sqrt(6.0 / WIDTH)
    w3 = rng.uniform(-1, 1, size=WIDTH) * math.sqrt(6.0 / WIDTH)
    zero = np.zeros(WIDTH)
    params = np.concatenate([w1.ravel(), zero, w2.ravel(), zero, w3, np.zeros(1)]).astype(np.float32)
    return q, valid, params


def prepare(case: dict, seed: int) -> dict:
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    kind = case["kind"]
    state = {"case": case}
    if kind == "mixed":
        state["batch"] = vg.Batch()
        state["outs"] = []
        for k, name in enumerate(ROBOTS):
            robot = getattr(vg, name)
            env = _environment(robot, seed, POINTS)
            a, b = scenes.edges(robot.s_m, robot.s_a, case["n"], seed + 31 * k)
            out = torch.empty(case["n"], dtype=torch.uint8, device="cuda")
            state["batch"].add(robot, env, _device(a), _device(b), out)
            state["outs"].append(out)
        return state
    robot = getattr(vg, case["robot"])
    state["robot"] = robot
    if kind in ("steps", "host_edges"):
        state["env"] = _environment(robot, seed, case["points"])
        n = case["n"]
        # a planner asks about motions from valid configurations: starts that are in collision are
        # replaced while some are left
        a, b = _short_edges(robot, 4 * n + 64, case["length"], seed)
        order = np.argsort(1 - robot.validate_batch(a, state["env"]).astype(np.int64), kind="stable")[:n]
        state["a"], state["b"] = np.ascontiguousarray(a[order]), np.ascontiguousarray(b[order])
    elif kind == "edges":
        state["env"] = _environment(robot, seed, case["points"], case["lanes"])
        a, b = scenes.edges(robot.s_m, robot.s_a, case["n"], seed)
        state["a"], state["b"] = _device(a), _device(b)
        state["blocks"] = torch.empty(case["n"], dtype=torch.int32, device="cuda") if case["counts"] else None
    elif kind == "vectors":
        state["env"] = _environment(robot, seed, case["points"], case["lanes"])
        a, b = scenes.edges(robot.s_m, robot.s_a, case["n"], seed)
        v = b - a
        # planners extend by at most their range along the vector
        d = np.linalg.norm(v, axis=1, keepdims=True)
        v = (v * np.minimum(1.0, 2.0 / d)).astype(np.float32)
        state["a"], state["v"] = _device(a), _device(v)
        state["d"] = _device(np.linalg.norm(v, axis=1).astype(np.float32))
    elif kind == "carry":
        def extra(env, s):
            # terrain up to 0.17 m below the base, and a rod of four spheres in the hand
            hf = scenes.heightfield(s, centre=(0.2, 0.0, -0.5))
            env.add_heightfield(vg.HeightField(hf["centre"], hf["scale"], (hf["xd"], hf["yd"]), hf["data"]))
            tf = np.eye(4, dtype=np.float32)
            tf[2, 3] = 0.12
            held = vg.Attachment(tf)
            held.add_spheres([[0.0, 0.0, 0.03 * k, 0.04] for k in range(4)])
            env.attach(held)

        env = _environment(robot, seed, 0, case["lanes"], extra=extra)
        a, b = scenes.edges(robot.s_m, robot.s_a, case["n"], seed)
        state.update(env=env, a=_device(a), b=_device(b))
    elif kind == "states":
        state["env"] = _environment(robot, seed, case["points"], primitives=not case["points"])
        state["q"] = _device(scenes.configurations(robot.s_m, robot.s_a, case["n"], seed))
    elif kind == "sense":
        state["points"] = _device(scenes.surface_pointcloud(seed, case["n"]))
        state["cloud"] = torch.empty((case["n"], 3), dtype=torch.float32, device="cuda")
        state["q"] = _device(scenes.configurations(robot.s_m, robot.s_a, case["states"], seed))
    elif kind == "roadmap":
        n = case["n"]
        state["nodes"] = torch.empty((n, robot.dimension()), dtype=torch.float32, device="cuda")
        state["edges"] = torch.empty((40 * n, 2), dtype=torch.int64, device="cuda")
        state["lengths"] = torch.empty(40 * n, dtype=torch.float32, device="cuda")
        state["env"] = _environment(robot, seed, 0)
        state["q"] = _device(scenes.configurations(robot.s_m, robot.s_a, case["n"], seed))
    elif kind == "learned":
        state["env"] = _environment(robot, seed, 0)
        state["predictor"] = vg.CollisionPredictor(robot, seed % 1000)
        state["predictor"].train_on_environment(state["env"], n=1 << 15, epochs=1, seed=seed)
        a, b = scenes.edges(robot.s_m, robot.s_a, case["n"], seed)
        state["a"], state["b"] = _device(a), _device(b)
    else:
        q, valid, state["params"] = _train_inputs(robot, case["n"], seed)
        state["q"], state["valid"] = _device(q), _device(valid)
    return state


def _into(buffer, rows):
    """The rows at the head of the caller's fixed-size buffer, zeros behind them."""
    buffer.zero_()
    buffer[:len(rows)] = rows
    return buffer


def run(state: dict):
    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    case = state["case"]
    kind = case["kind"]
    if kind == "mixed":
        state["batch"].launch()
        return state["outs"]
    robot = state["robot"]
    if kind == "steps":
        res = robot.resolution()
        return [int(robot.validate_motion(a, b, state["env"], resolution=res)) for a, b in zip(state["a"], state["b"])]
    if kind == "host_edges":
        return robot.validate_motion_batch(state["a"], state["b"], state["env"])
    if kind == "edges":
        ok = robot.validate_motion_batch(state["a"], state["b"], state["env"], blocks=state["blocks"])
        return (ok, state["blocks"]) if case["counts"] else ok
    if kind == "vectors":
        return robot.validate_vector_batch(state["a"], state["v"], state["d"], state["env"])
    if kind == "carry":
        return robot.validate_motion_batch(state["a"], state["b"], state["env"])
    if kind == "states":
        return robot.validate_batch(state["q"], state["env"])
    if kind == "sense":
        # the benchmark's settings: origin at the first joint, 1.19 m reach, 1 cm spacing
        o = np.array([0.0, 0.0, 0.333], np.float32)
        kept = vg.filter_pointcloud_device(state["points"], 0.01, 1.19, o, o - 1.19, o + 1.19, case["cull"])
        env = vg.Environment()
        env.add_pointcloud_device(kept, *robot.min_max_radii(), scenes.POINT_RADIUS)
        return len(kept), _into(state["cloud"], kept), robot.validate_batch(state["q"], env)
    if kind == "roadmap":
        from vamp_gb300 import roadmap

        r = roadmap.build_roadmap(robot, state["env"], state["q"])
        return (r["valid_samples"], r["candidates"], r["valid_edges"], _into(state["nodes"], r["nodes"]),
                _into(state["edges"], r["edges"]), _into(state["lengths"], r["lengths"]))
    if kind == "learned":
        return state["predictor"].validate_motion_batch(state["a"], state["b"], state["env"], probes=case["probes"])
    predictor = vg.CollisionPredictor(robot)
    predictor.load_parameters(state["params"])
    losses = predictor.train(state["q"], state["valid"], epochs=1, batch=case["batch"])
    return losses, predictor.parameters()


# --------------------------------------------------------------------------------- accounting

def work(case: dict) -> dict:
    """Inputs read once, outputs written once; per state checked, the kinematics (18 operations a
    sphere slot), a query per coarse link sphere (8, and one test of 20 per primitive in reach,
    about one in five of 60) and the coarse self pairs (11).  Half of an edge's states are taken
    as checked (colliding motions stop early)."""
    kind = case["kind"]
    if kind == "mixed":
        parts = [work({"kind": "edges", "robot": r, "n": case["n"], "points": POINTS, "lanes": 8, "counts": False})
                 for r in ROBOTS]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    dim, slots, coarse, pairs, res, mean = SHAPE[case["robot"]]
    per_state = 18 * slots + coarse * (8 + 12 * 20) + 11 * pairs
    cloud = 12 * case.get("points", 0)
    kin = (2 * dim + 15) // 16 * 16
    mlp = 2 * (kin * WIDTH + WIDTH * WIDTH + WIDTH)
    n = case["n"]

    def edges(count, length):
        return count * max(8.0, 0.5 * length * res) * per_state

    if kind in ("steps", "host_edges"):
        return {"bytes": n * (8 * dim + 1) + cloud, "flops": edges(n, case["length"])}
    if kind == "edges":
        return {"bytes": n * (8 * dim + 1 + (4 if case["counts"] else 0)) + cloud, "flops": edges(n, mean)}
    if kind == "vectors":
        return {"bytes": n * (8 * dim + 5) + cloud, "flops": edges(n, 2.0)}
    if kind == "carry":
        return {"bytes": n * (8 * dim + 1) + 4 * 96 * 80, "flops": edges(n, mean)}
    if kind == "states":
        return {"bytes": n * (4 * dim + 1) + cloud, "flops": n * per_state}
    if kind == "sense":
        kept = 0.006 * n if case["cull"] else 0.07 * n
        return {"bytes": 12 * n + 12 * kept + case["states"] * (4 * dim + 1),
                "flops": n * 60.0 + case["states"] * per_state}
    if kind == "roadmap":
        pairs_kept = 24 * n
        return {"bytes": n * 4 * dim + pairs_kept * 20, "flops": n * per_state + 1.5 * dim * n * n + edges(pairs_kept, 0.8)}
    if kind == "learned":
        return {"bytes": n * (8 * dim + 1) + 2 * (kin * WIDTH + WIDTH * WIDTH),
                "flops": edges(n, mean) + n * case["probes"] * mlp}
    params = WIDTH * kin + WIDTH + WIDTH * WIDTH + 2 * WIDTH + 1
    return {"bytes": n * (4 * dim + 1) + 8 * params, "flops": 3.0 * n * mlp}


def exact(case: dict, seed: int):
    """The trained network's epoch loss and weights in float64 (Adam at 1e-3 on the mean binary
    cross-entropy of the collision logit); the other cases' outputs have no such value."""
    if case["kind"] != "train":
        return None
    import torch

    import vamp_gb300 as vg

    robot = getattr(vg, case["robot"])
    q, valid, params = _train_inputs(robot, case["n"], seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dim, batch = q.shape[1], case["batch"]
    kin = (2 * dim + 15) // 16 * 16
    q = torch.from_numpy(q).to(dev, torch.float64)
    x = torch.zeros((len(q), kin), dtype=torch.float64, device=dev)
    x[:, 0:2 * dim:2] = torch.sin(q)
    x[:, 1:2 * dim:2] = torch.cos(q)
    y = 1.0 - torch.from_numpy(valid).to(dev, torch.float64)
    w = torch.from_numpy(params).to(dev, torch.float64)
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    cuts = np.cumsum([WIDTH * kin, WIDTH, WIDTH * WIDTH, WIDTH, WIDTH]).tolist()
    steps = case["n"] // batch
    total = 0.0
    for step in range(1, steps + 1):
        w1, b1, w2, b2, w3, b3 = torch.tensor_split(w, cuts)
        w1, w2 = w1.view(WIDTH, kin), w2.view(WIDTH, WIDTH)
        xb, yb = x[(step - 1) * batch:step * batch], y[(step - 1) * batch:step * batch]
        h1 = torch.relu(xb @ w1.T + b1)
        h2 = torch.relu(h1 @ w2.T + b2)
        z = h2 @ w3 + b3
        total += float(torch.mean(torch.relu(z) - z * yb + torch.log1p(torch.exp(-z.abs()))))
        dz = (torch.sigmoid(z) - yb) / batch
        d2 = torch.where(h2 > 0, dz[:, None] * w3[None, :], 0.0)
        d1 = torch.where(h1 > 0, d2 @ w2, 0.0)
        g = torch.cat([(d1.T @ xb).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ dz, dz.sum().view(1)])
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return np.array([total / steps]), w.cpu().numpy()
