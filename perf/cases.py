"""Performance cases: the calls a program built on this package spends its time in.

Each case is one call, or one short chain of calls, of the public Python API on inputs
with the shapes and distributions of the package's own workloads (delta_b200.scenarios):

- pair lists through ``pairs_device``: every method, FP64 and FP32, from a few hundred
  pairs (one body pair's triangles) to millions;
- the learned hybrid through ``learned_pairs``, without and with the network;
- one training step of the warm-start network;
- the particle-pair drivers through ``delta_detect`` over a broadphase's candidate pairs, into
  a contact buffer that the program keeps;
- the time step through ``Simulation.step``, graph-replayed and stepped, restarted from a
  checkpoint of the body state before each run of steps (as a parameter study does).
"""
import ctypes
import math

import numpy as np
import torch

from delta_b200 import detection, lib
from delta_b200.engine import DeviceScene, Simulation, StepParams, broadphase
from delta_b200.learned import WarmStartMLP, labelled, learned_pairs
from delta_b200.narrowphase import Context, pairs_device
from delta_b200.scenarios import hopper_obstacles, lattice_scene, narrowphase_pairs, particle_cloud_scene

# drivers by name: those of delta_detect, and the subset the time step runs
DRIVERS = {"bf": detection.DRV_BF, "penalty": detection.DRV_PENALTY, "hybrid_batch": detection.DRV_HYBRID_BATCH,
           "hybrid_triangle": detection.DRV_HYBRID_TRIANGLE, "gjk": detection.DRV_GJK,
           "bf_cert": detection.DRV_BF_CERT, "bf_culled": detection.DRV_BF_CULLED, "learned": detection.DRV_LEARNED}
# arithmetic operations of one triangle pair in each pair method (multiply, add, divide,
# square root counted as one each); GJK's count varies with the pair, about this many
PAIR_FLOPS = {"bf": 1214, "bf_cert": 1214, "penalty": 905, "penalty_iter": 905, "hybrid": 905, "gjk": 900}
MLP_FLOPS = 2 * (18 * 128 + 128 * 128 + 128 * 128 + 128 * 4)
PAIR_BYTES = 18 * 8 + 7 * 8 + 1
BODY_STATE = ("pos", "vel", "ang", "ref_ang", "rot")
CONTACT_FIELDS = ("x", "normal", "P", "Q", "depth", "eps_total", "master", "slave", "tri_a", "tri_b")
MAX_CONTACTS = 1 << 15
BASE_PAIRS = 1 << 15


def listed():
    return [
        # the triangles two small particles bring to one call: latency
        {"name": "bf_few_pairs", "kind": "pairs", "method": "bf", "precision": "f64", "pairs": 1000},
        # the exact solver over a large candidate list, the yardstick of the other methods
        {"name": "bf_many_pairs", "kind": "pairs", "method": "bf", "precision": "f64", "pairs": 1 << 22},
        # the certified solver over the candidates of one time step of a mid-sized scene
        {"name": "cert_ragged", "kind": "pairs", "method": "bf_cert", "precision": "f64", "pairs": 777_777},
        # the reference's recommended method: penalty iterations with the exact fallback
        {"name": "hybrid_pairs", "kind": "pairs", "method": "hybrid", "precision": "f64", "pairs": 1 << 20},
        # single precision where a rough distance is enough
        {"name": "gjk_f32", "kind": "pairs", "method": "gjk", "precision": "f32", "pairs": 262_143},
        # the microbenchmark workload at its full size, in the tuned setting
        {"name": "learned_16m", "kind": "learned", "network": False, "sweeps": 2, "features": 3, "pairs": 1 << 24},
        # the learned hybrid with its network
        {"name": "learned_network", "kind": "learned", "network": True, "sweeps": 1, "features": 3,
         "pairs": 1_000_003},
        # one optimiser step at the training recipe's batch
        {"name": "train_step", "kind": "train", "batch": 65536},
        # the reference's bf() driver over the candidate body pairs of the small lattice
        {"name": "detect_bf_lattice", "kind": "detect", "driver": "bf", "nx": 8, "ny": 4, "nz": 8},
        # time steps: small (launch latency), uneven hopper, box with the learned driver
        {"name": "steps_lattice", "kind": "steps", "scene": "lattice", "bodies": 256, "driver": "bf_cert",
         "graph": True, "steps": 100},
        {"name": "steps_hopper", "kind": "steps", "scene": "hopper", "bodies": 10000, "driver": "bf_cert",
         "graph": True, "steps": 100},
        {"name": "steps_box_learned", "kind": "steps", "scene": "box", "bodies": 16000, "driver": "learned",
         "graph": True, "steps": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pairs", "pairs", "pairs", "learned", "learned", "train", "detect", "steps", "steps"])
    if kind == "pairs":
        method = rng.choice(["bf", "bf_cert", "penalty", "penalty_iter", "hybrid", "gjk"])
        precision = "f64" if method == "bf_cert" else rng.choice(["f64", "f64", "f32"])
        return {"kind": kind, "method": method, "precision": precision, "pairs": _log_int(rng, 200, 1 << 22)}
    if kind == "learned":
        network = rng.random() < 0.4
        return {"kind": kind, "network": network, "sweeps": rng.choice([1, 2]), "features": rng.choice([3, 7, 15]),
                "pairs": _log_int(rng, 1000, 1 << (21 if network else 23))}
    if kind == "train":
        return {"kind": kind, "batch": _log_int(rng, 2048, 65536)}
    if kind == "detect":
        return {"kind": kind, "driver": rng.choice(sorted(DRIVERS)), "nx": rng.randint(2, 8), "ny": rng.randint(1, 4),
                "nz": rng.randint(2, 8)}
    scene = rng.choice(["lattice", "hopper", "box"])
    graph = rng.random() < 0.75
    driver = rng.choice(["bf_cert", "bf_culled", "learned"]) if graph else rng.choice(["bf", "bf_cert"])
    most = {"lattice": 256, "hopper": 10000, "box": 12000}[scene] if graph else 256
    return {"kind": kind, "scene": scene, "bodies": _log_int(rng, 16, most), "driver": driver, "graph": graph,
            "steps": rng.randint(20, 100) if graph else rng.randint(2, 10)}


# ---- inputs -------------------------------------------------------------------------------
def _pairs(n, seed):
    """n pairs of the microbenchmark distribution on the GPU: up to BASE_PAIRS drawn on the
    host, then that set again and again, each pair under a random rigid motion of its own
    (which keeps the separations, angles and classes) and a random vertex order."""
    m = min(n, BASE_PAIRS)
    a0, b0, _, _ = narrowphase_pairs(m, seed=seed)
    base = torch.from_numpy(np.stack([a0, b0])).cuda().view(2, 3, 3, m)  # triangle, vertex, coordinate, pair
    out = torch.empty((2, 9, n), dtype=torch.float64, device="cuda")
    out[:, :, :m] = base.reshape(2, 9, m)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    for lo in range(m, n, 32 * m):
        k = min(32 * m, n - lo)
        copies = -(-k // m)
        t = base.repeat(1, 1, 1, copies)[..., :k]
        w, x, y, z = torch.nn.functional.normalize(
            torch.randn((4, k), dtype=torch.float64, device="cuda", generator=gen), dim=0)
        rot = ((1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)),
               (2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)),
               (2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)))
        u = t - 0.5
        moved = torch.stack([r[0] * u[:, :, 0] + r[1] * u[:, :, 1] + r[2] * u[:, :, 2] for r in rot], 2) + 0.5
        moved += 0.1 * torch.rand((3, k), dtype=torch.float64, device="cuda", generator=gen) - 0.05
        order = torch.rand((2, 3, k), device="cuda", generator=gen).argsort(1)
        moved = torch.gather(moved, 1, order[:, :, None, :].expand(2, 3, 3, k))
        out[:, :, lo:lo + k] = moved.reshape(2, 9, k)
    return out[0], out[1]


def _training_rows(ctx, n, seed):
    a, b = _pairs(n, seed)
    return labelled(ctx, a, b)


def _moments(n, seed):
    """Adam moments of a training under way: gradients of about 1e-3."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    m = 1e-3 * torch.randn(n, device="cuda", generator=gen)
    v = 1e-6 * (0.5 + torch.rand(n, device="cuda", generator=gen))
    return m, v


def _outputs(n):
    f8 = dict(dtype=torch.float64, device="cuda")
    return (torch.empty((3, n), **f8), torch.empty((3, n), **f8), torch.empty(n, **f8),
            torch.empty(n, dtype=torch.uint8, device="cuda"))


def _lattice_dims(bodies):
    nx = max(1, round((2 * bodies) ** (1 / 3)))
    ny = max(1, nx // 2)
    return nx, ny, max(1, -(-bodies // (nx * ny)))


def _walls(box):
    """The six faces of a box, two triangles each, standing on y = 0."""
    hx, hy, hz = box[0] / 2, box[1], box[2] / 2
    corner = np.array([[x, y, z] for y in (0, hy) for x, z in ((-hx, -hz), (hx, -hz), (hx, hz), (-hx, hz))], float)
    quads = ((0, 1, 2, 3), (4, 7, 6, 5), (0, 4, 5, 1), (1, 5, 6, 2), (2, 6, 7, 3), (3, 7, 4, 0))
    return [(corner[list(q)], np.array([[0, 1, 2], [0, 2, 3]])) for q in quads]


def _scene(case, seed):
    """The package's lattice, hopper and box workloads; the mesh sizes are drawn the same for
    every seed, so that a case has the same number of triangles on any inputs."""
    n = case["bodies"]
    if case["scene"] == "lattice":
        nx, ny, nz = _lattice_dims(n)
        return lattice_scene(seed=seed, nx=nx, ny=ny, nz=nz)
    hopper = case["scene"] == "hopper"
    sizes, radius = ((40, 80, 160, 320), (0.005, 0.015)) if hopper else ((80, 160, 320, 500), (0.004, 0.012))
    n_tri = np.random.default_rng(n).choice(np.asarray(sizes), n)
    rng = np.random.default_rng(seed)
    spacing = 2.0 * radius[1] * 1.2 * (1.05 if hopper else 1.02)
    side = int(math.ceil(math.sqrt(n / 30))) if hopper else int(0.6 / spacing) - 1
    k = np.arange(n)
    grid = np.stack([k // side % side, k // (side * side), k % side], 1)  # layer by layer from the bottom
    origin = np.array([-(side - 1) * spacing / 2, 0.3 if hopper else spacing, -(side - 1) * spacing / 2])
    jitter = (0.1 if hopper else 0.05) * spacing
    centres = origin + grid * spacing + rng.uniform(-jitter, jitter, (n, 3))
    return particle_cloud_scene(centres, rng.uniform(radius[0], radius[1], n), n_tri,
                                hopper_obstacles() if hopper else _walls((0.6, 1.2, 0.6)), seed=seed + 1, eps=1e-4)


def prepare(case, seed):
    ctx = Context(0)
    s = {"case": case, "ctx": ctx}
    if case["kind"] in ("pairs", "learned"):
        s["a"], s["b"] = _pairs(case["pairs"], seed)
        s["out"] = _outputs(case["pairs"])
        s["model"] = WarmStartMLP.load(ctx) if case.get("network") else None
    elif case["kind"] == "train":
        s["X"], s["T"], s["valid"] = _training_rows(ctx, case["batch"], seed)
        s["n_valid"] = int(s["valid"].sum().item())
        model = s["model"] = WarmStartMLP.load(ctx)
        m, v = _moments(model.L["total"], seed)
        model.m.copy_(m)
        model.v.copy_(v)
        model.steps = 1000
    elif case["kind"] == "detect":
        scene = lattice_scene(seed=seed, nx=case["nx"], ny=case["ny"], nz=case["nz"])
        dev = DeviceScene(scene)
        pa, pb = broadphase(ctx, dev)
        s["pa"], s["pb"] = torch.from_numpy(pa).cuda(), torch.from_numpy(pb).cuda()
        s["meshes"] = detection.Meshes(scene["tri_offset"], scene["x"], scene["y"], scene["z"], scene["eps"],
                                       scene["friction"])
        contacts = s["contacts"] = detection.Contacts(MAX_CONTACTS)
        for k in CONTACT_FIELDS:
            getattr(contacts, k).zero_()
    else:
        sim = s["sim"] = Simulation(ctx, _scene(case, seed), DRIVERS[case["driver"]])
        s["start"] = {k: sim.dev.t[k].clone() for k in BODY_STATE}
        dt = {"lattice": 1e-5, "hopper": 5e-6, "box": 2e-6}[case["scene"]]
        s["params"] = StepParams.make(dt=dt)
    return s


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["kind"] == "pairs":
        p, q, d, flags = pairs_device(ctx, case["method"], state["a"], state["b"], out=state["out"],
                                      precision=0 if case["precision"] == "f64" else 1, max_error=1e-3)
        return {"p": p, "q": q, "dist": d, "flags": flags}
    if case["kind"] == "learned":
        p, q, d, flags = learned_pairs(ctx, state["model"], state["a"], state["b"], case["sweeps"], out=state["out"],
                                       features=case["features"])
        return {"p": p, "q": q, "dist": d, "flags": flags}
    if case["kind"] == "train":
        model = state["model"]
        model.train_step(state["X"], state["T"], state["valid"], state["n_valid"])
        return {"loss": model.loss, "grads": model.grads, "params": model.params}
    if case["kind"] == "detect":
        count, contacts, meshes = ctypes.c_int64(0), state["contacts"], state["meshes"]
        status = lib().delta_detect(ctx.handle, DRIVERS[case["driver"]], 0, ctypes.byref(meshes.struct()),
                                    state["pa"].data_ptr(), state["pb"].data_ptr(), state["pa"].numel(),
                                    ctypes.byref(contacts.struct()), ctypes.byref(count), None)
        if status:
            raise RuntimeError(f"delta_detect: status {status}")
        return {"count": count.value, **{k: getattr(contacts, k) for k in CONTACT_FIELDS}}
    sim = state["sim"]
    for k, v in state["start"].items():
        sim.dev.t[k].copy_(v)
    per_step = sim.step(case["steps"], state["params"], graph=case["graph"])
    return {"contacts": per_step, **{k: sim.dev.t[k] for k in BODY_STATE + ("x", "y", "z")}}


# ---- what a pass cannot do without ----------------------------------------------------------
def work(case):
    if case["kind"] == "pairs":
        n = case["pairs"]
        return {"bytes": n * PAIR_BYTES, "flops": n * PAIR_FLOPS[case["method"]]}
    if case["kind"] == "learned":
        # two projections a sweep, the features tried and the separating plane's tests
        n = case["pairs"]
        flops = 120 * case["sweeps"] + 60 * case["features"] + 100 + (MLP_FLOPS if case["network"] else 0)
        return {"bytes": n * PAIR_BYTES, "flops": n * flops}
    if case["kind"] == "train":
        # rows, targets and validity read; parameters, gradients and moments read and written
        params = 37768
        return {"bytes": case["batch"] * (64 + 16 + 1) + params * (7 * 4 + 2), "flops": 3 * case["batch"] * MLP_FLOPS}
    if case["kind"] == "detect":
        # nearest neighbours on the lattice and the floor under the lowest layer, 80 triangles a body
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        close = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
        exhaustive = case["driver"] in ("bf", "penalty", "hybrid_batch", "hybrid_triangle", "gjk")
        flops = PAIR_FLOPS["bf" if case["driver"] == "bf" else "penalty"] * (close * 6400 + nx * nz * 160)
        return {"bytes": n * 80 * 72, "flops": flops if exhaustive else n * 80 * 100}
    # per step every moving body's state is read and written (21 doubles) and its mass, inertia
    # and reference read (25); the vertices once a pass
    n = case["bodies"]
    tri = {"lattice": 80, "hopper": 150, "box": 265}[case["scene"]]
    return {"bytes": n * ((2 * 21 + 25) * 8 * case["steps"] + tri * 9 * 16), "flops": n * 500 * case["steps"]}


# ---- the same in plain torch, 64 bits ---------------------------------------------------------
def _seg_seg(p1, q1, p2, q2):
    """Distance of segments (n, 3): the lines' closest points where both lie inside, else the
    nearest of the four end points against the other segment."""
    u, v, w = q1 - p1, q2 - p2, p1 - p2
    dot = lambda x, y: (x * y).sum(-1)  # noqa: E731
    a, b, c, d, e = dot(u, u), dot(u, v), dot(v, v), dot(u, w), dot(v, w)
    det = a * c - b * b
    s, t = (b * e - c * d) / det, (a * e - b * d) / det
    inside = (det > 0) & (s >= 0) & (s <= 1) & (t >= 0) & (t <= 1)
    line = (w + s[:, None] * u - t[:, None] * v).norm(dim=-1)
    best = torch.where(inside, line, torch.full_like(line, math.inf))
    for x, o, r in ((p1, p2, v), (q1, p2, v), (p2, p1, u), (q2, p1, u)):
        k = (dot(x - o, r) / dot(r, r)).clamp(0, 1)
        best = torch.minimum(best, (x - o - k[:, None] * r).norm(dim=-1))
    return best


def _point_face(t0, t1, t2, x):
    """Distance of points to the inside of triangles (inf where the foot lies outside)."""
    u, v, w = t1 - t0, t2 - t0, x - t0
    dot = lambda x, y: (x * y).sum(-1)  # noqa: E731
    uu, uv, vv, wu, wv = dot(u, u), dot(u, v), dot(v, v), dot(w, u), dot(w, v)
    det = uu * vv - uv * uv
    s, t = (vv * wu - uv * wv) / det, (uu * wv - uv * wu) / det
    d = (w - s[:, None] * u - t[:, None] * v).norm(dim=-1)
    return torch.where((det > 0) & (s >= 0) & (t >= 0) & (s + t <= 1), d, torch.full_like(d, math.inf))


def _triangle_distance(a, b):
    """The least of the 9 edge-edge and 6 vertex-face distances of triangles (n, 3, 3)."""
    best = torch.full((a.shape[0],), math.inf, dtype=torch.float64, device=a.device)
    for i in range(3):
        for j in range(3):
            best = torch.minimum(best, _seg_seg(a[:, i], a[:, (i + 1) % 3], b[:, j], b[:, (j + 1) % 3]))
        best = torch.minimum(best, _point_face(a[:, 0], a[:, 1], a[:, 2], b[:, i]))
        best = torch.minimum(best, _point_face(b[:, 0], b[:, 1], b[:, 2], a[:, i]))
    return best


def _exact_train(case, seed):
    ctx = Context(0)
    X, T, valid = _training_rows(ctx, case["batch"], seed)
    model = WarmStartMLP.load(ctx)
    m, v = _moments(model.L["total"], seed)
    L, f8 = model.L, torch.float64
    p = model.params.to(f8)
    low = model.params.bfloat16().to(f8)  # the layers multiply by 16-bit weights
    shapes = ((128, 32), (128, 128), (128, 128), (4, 128))
    weight = [low[L[f"W{k}"]:L[f"W{k}"] + r * c].view(r, c).clone().requires_grad_() for k, (r, c) in
              enumerate(shapes, 1)]
    bias = [p[L[f"b{k}"]:L[f"b{k}"] + r].clone().requires_grad_() for k, (r, _) in enumerate(shapes, 1)]
    h = X.to(f8)
    for k in range(4):
        h = h @ weight[k].T + bias[k]
        if k < 3:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    n_valid = max(int(valid.sum().item()), 1)
    loss = (((h - T.to(f8)) ** 2).sum(1) * valid.to(f8)).sum() / n_valid
    loss.backward()
    g = torch.zeros_like(p)
    for k in range(4):
        g[L[f"W{k + 1}"]:L[f"W{k + 1}"] + weight[k].numel()] = weight[k].grad.reshape(-1)
        g[L[f"b{k + 1}"]:L[f"b{k + 1}"] + bias[k].numel()] = bias[k].grad
    step, b1, b2 = 1001, 0.9, 0.999
    m, v = b1 * m.to(f8) + (1 - b1) * g, b2 * v.to(f8) + (1 - b2) * g * g
    p = p - 1e-3 * (m / (1 - b1 ** step)) / ((v / (1 - b2 ** step)).sqrt() + 1e-8)
    return {"loss": loss.detach().reshape(1), "grads": g, "params": p}


def _exact_depths(case, seed):
    """The contact depths of the lattice in (body pair, triangle, triangle) order."""
    s = prepare(case, seed)
    m, off = s["meshes"], s["meshes"].tri_offset.cpu()
    tri = torch.stack([m.x, m.y, m.z], 1).view(-1, 3, 3)
    depth = torch.zeros(MAX_CONTACTS, dtype=torch.float64, device="cuda")
    found = 0
    for i, j in zip(s["pa"].tolist(), s["pb"].tolist()):
        a, b = tri[off[i]:off[i + 1]], tri[off[j]:off[j + 1]]
        near = ((a.amax((0, 1)) + 1e-3 > b.amin((0, 1))) & (b.amax((0, 1)) + 1e-3 > a.amin((0, 1)))).all()
        if not near:
            continue
        d = _triangle_distance(a.repeat_interleave(b.shape[0], 0), b.repeat(a.shape[0], 1, 1))
        eps = float(m.eps[i] + m.eps[j])
        d = eps - d[d <= eps]
        depth[found:found + d.numel()] = d
        found += d.numel()
    return {"count": None, **{k: None for k in CONTACT_FIELDS}, "depth": depth}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "learned" or (case["kind"] == "pairs" and case["method"] in ("bf", "bf_cert")):
        a, b = _pairs(case["pairs"], seed)
        n, dist = case["pairs"], []
        for lo in range(0, n, 1 << 18):
            t = [x[:, lo:lo + (1 << 18)].T.reshape(-1, 3, 3) for x in (a, b)]
            dist.append(_triangle_distance(*t))
        # the points are not unique where triangles are parallel
        return {"p": None, "q": None, "dist": torch.cat(dist), "flags": None}
    if case["kind"] == "detect" and case["driver"] in ("bf", "bf_cert", "bf_culled"):
        return _exact_depths(case, seed)
    # an unfinished iteration, or a run of time steps
    return None
