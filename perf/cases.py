"""The work whose speed this framework is judged by, through its public entry points.

`listed()` names the cases, `draw()` gives more of the same ranges,
`prepare()` makes what a program holds before the call, `run()` is one pass,
`work()` is what a pass cannot do without and `exact()` is the 64-bit result
where one exists without following the float code's branches.

The paths:

  narrowphase   one step's algorithm batches on device arrays (rp3dg_narrowphase_device),
                optionally with the temporal cache and the manifold step
                (rp3dg_reduce_contacts_device), which is what an engine that keeps its
                pairs on the GPU calls every step
  input_host    the same batches from pinned host arrays in one call
                (rp3dg_narrowphase_input_host), which is what a CPU engine calls
  broadphase    fat-AABB update and overlapping-pair search of one world
  dynamics      one dynamics stage (velocities, contact solver, positions) of many worlds
  world         PhysicsWorld::update of one world and its body states read back
  group         the same for many worlds stepped together
  raycast       a batch of rays against a world
  axis_mlp      forward and backward of the separating-axis model on one minibatch
"""
import ctypes
import math
import os

import numpy as np
import torch

from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import broadphase as BP
from reactphysics3d_b200 import dynamics as D
from reactphysics3d_b200 import engine, scenes

CAPTURES = os.path.join(scenes.REPO_ROOT, "tests", "golden", "np_dynamics.npz")
SINGLE = scenes.BATCH_NAMES + ("hull_hull",)


def listed():
    return [
        # a few dozen bodies in a game: every algorithm has a handful of pairs and launches are all there is
        {"name": "np_small_step", "path": "narrowphase", "batch": "all", "pairs": 294, "coherent": True, "manifolds": True},
        # the benchmark workload: 1,048,576 pairs in seven batches, no temporal records
        {"name": "np_step_1m", "path": "narrowphase", "batch": "all", "pairs": 1048576, "coherent": False, "manifolds": False},
        # resting boxes: temporal records answer most pairs, then the manifolds are reduced
        {"name": "np_boxes_coherent", "path": "narrowphase", "batch": "box_box", "pairs": 100003, "coherent": True, "manifolds": True},
        # debris of convex hulls: mesh against mesh, the costliest pair
        {"name": "np_hulls", "path": "narrowphase", "batch": "hull_hull", "pairs": 20011, "coherent": False, "manifolds": False},
        # a CPU engine handing over a step's pairs and reading the contacts back
        {"name": "np_host_step", "path": "input_host", "pairs": 300007},
        # the large world's broad phase
        {"name": "broadphase_100k", "path": "broadphase", "colliders": 100003},
        # a training farm's dynamics stage
        {"name": "dynamics_4096_worlds", "path": "dynamics", "worlds": 4096},
        # the plain box pile, one island
        {"name": "world_pile", "path": "world", "scene": "pile", "side": 10, "steps": 200},
        # a game level: bodies resting on a height field
        {"name": "world_terrain", "path": "world", "scene": "terrain", "bodies": 3000, "steps": 120},
        # many small worlds with ragdolls
        {"name": "group_256", "path": "group", "worlds": 256, "steps": 60},
        # visibility and ground queries over a large terrain
        {"name": "raycast_terrain", "path": "raycast", "scene": "terrain", "bodies": 20000, "rays": 300007, "mode": A.RAYCAST_CLOSEST, "hits": 1, "steps": 21},
        # one minibatch of the learned separating axis
        {"name": "axis_mlp_grads", "path": "axis_mlp", "samples": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["narrowphase", "narrowphase", "narrowphase", "input_host", "broadphase", "dynamics", "world",
                       "world", "group", "raycast", "raycast", "axis_mlp"])
    if path == "narrowphase":
        batch = rng.choice(("all",) + SINGLE)
        top = {"all": 1000000, "hull_box": 140000, "hull_hull": 30000}.get(batch, 400000)
        coherent = rng.random() < 0.5
        return {"path": path, "batch": batch, "pairs": _log(rng, 35, top), "coherent": coherent,
                "manifolds": coherent or rng.random() < 0.3}
    if path == "input_host":
        return {"path": path, "pairs": _log(rng, 700, 500000)}
    if path == "broadphase":
        return {"path": path, "colliders": _log(rng, 100, 200000)}
    if path == "dynamics":
        return {"path": path, "worlds": _log(rng, 1, 4096)}
    if path == "world":
        scene = rng.choice(["pile", "mixed", "hulls", "terrain"])
        if scene == "terrain":
            return {"path": path, "scene": scene, "bodies": _log(rng, 100, 3000), "steps": 120}
        return {"path": path, "scene": scene, "side": rng.randint(2, 10 if scene == "pile" else 7), "steps": rng.randint(60, 200)}
    if path == "group":
        return {"path": path, "worlds": _log(rng, 4, 256), "steps": rng.randint(40, 90)}
    if path == "raycast":
        scene = rng.choice(["terrain", "hulls"])
        mode = rng.choice([A.RAYCAST_CLOSEST, A.RAYCAST_CLOSEST, A.RAYCAST_ANY, A.RAYCAST_ALL])
        size = {"bodies": _log(rng, 500, 20000), "steps": 21} if scene == "terrain" else {"side": rng.randint(2, 8), "steps": 30}
        return dict({"path": path, "scene": scene, "rays": _log(rng, 32, 300000), "mode": mode,
                     "hits": 4 if mode == A.RAYCAST_ALL else 1}, **size)
    return {"path": "axis_mlp", "samples": _log(rng, 256, 65536)}


# ---- inputs -----------------------------------------------------------------

def _hull_hull_scene(n, seed):
    """Pairs of the workload's hull with the same hull at scale 0.7, placed as the other batches are."""
    rng = np.random.default_rng(seed)
    verts, faces = scenes.load_hull()
    radius = float(np.max(np.linalg.norm(verts.astype(np.float64), axis=1)))
    shapes = np.zeros(2, A.SHAPE_DTYPE)
    shapes["kind"] = A.SHAPE_CONVEX_MESH
    shapes["mesh"] = (0, 1)
    pos1, pos2 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    centre = rng.uniform(-10.0, 10.0, (n, 3))
    pos1[:, :3] = centre
    pos2[:, :3] = centre + scenes.random_unit_vectors(rng, n) * (rng.uniform(0.5, 1.5, n) * 1.7 * radius)[:, None]
    pairs = A.HostPairs(np.zeros(n), np.ones(n), pos1, scenes.random_quaternions(rng, n), pos2,
                        scenes.random_quaternions(rng, n))
    return scenes.NarrowphaseScene(shapes, {"hull_hull": (A.ALGO_CONVEX_POLYHEDRON_VS_CONVEX_POLYHEDRON, pairs)},
                                   verts, faces, seed)


def _narrowphase_scene(case, seed):
    batch, n = case.get("batch", "all"), case["pairs"]
    if batch == "hull_hull":
        return _hull_hull_scene(n, seed)
    if batch == "all":
        return scenes.narrowphase_scene(total_pairs=n, seed=seed)
    return scenes.narrowphase_scene(total_pairs=7 * n, seed=seed, names=(batch,))


def _narrowphase_context(sc):
    ctx = engine.Context(0)
    mesh = ctx.create_convex_mesh(sc.hull_vertices, sc.hull_faces)
    ctx.create_convex_mesh_shape(mesh)
    ctx.create_convex_mesh_shape(mesh, (0.7, 0.7, 0.7))
    ctx.set_shapes(sc.shapes)
    return ctx


def _prepare_narrowphase(case, seed):
    sc = _narrowphase_scene(case, seed)
    calls = []
    for name, (algo, pairs) in sc.batches.items():
        if case["coherent"]:
            pairs.cache = A.fresh_cache(pairs.n)
        calls.append((name, algo, engine.DevicePairs(pairs), engine.DeviceContacts(pairs.n)))
    return {"ctx": _narrowphase_context(sc), "calls": calls}


def _run_narrowphase(case, s):
    ctx, out = s["ctx"], {}
    for name, algo, pairs, contacts in s["calls"]:
        ctx.narrowphase_device(algo, pairs, contacts)
        if case["manifolds"]:
            ctx.reduce_contacts_device(pairs, contacts)
        out[name] = {"colliding": contacts.is_colliding, "count": contacts.nb_contacts,
                     "normal_depth": contacts.normal_depth, "local1": contacts.local1, "local2": contacts.local2}
        if pairs.cache is not None:
            out[name]["cache"] = pairs.cache
    return out


def _pinned(a):
    """A page-locked copy of a numpy array (as a numpy array over the pinned tensor)."""
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    v = t.numpy().view(a.dtype).reshape(a.shape)
    v[...] = a
    return v, t


def _prepare_input_host(case, seed):
    sc = _narrowphase_scene(case, seed)
    keep, batches = [], []
    for algo, pairs in sc.batches.values():
        out = A.HostContacts(pairs.n)
        for obj, fields in ((pairs, ("shape1", "shape2", "pos1", "rot1", "pos2", "rot2")),
                            (out, ("is_colliding", "nb_contacts", "normal_depth", "local1", "local2"))):
            for f in fields:
                v, t = _pinned(getattr(obj, f))
                setattr(obj, f, v)
                keep.append(t)
        batches.append((algo, pairs, out))
    ctx = _narrowphase_context(sc)
    return {"ctx": ctx, "names": list(sc.batches), "call": ctx.narrowphase_input_call(batches), "keep": keep}


def _run_input_host(case, s):
    return {name: {"colliding": o.is_colliding, "count": o.nb_contacts, "normal_depth": o.normal_depth,
                   "local1": o.local1, "local2": o.local2} for name, o in zip(s["names"], s["call"]())}


def _prepare_broadphase(case, seed):
    rng = np.random.default_rng(seed)
    n = case["colliders"]
    side = int(math.ceil(n ** (1.0 / 3.0)))
    cell = rng.permutation(side ** 3)[:n]
    grid = np.stack([cell % side, cell // side % side, cell // (side * side)], 1)
    kind = rng.choice([A.SHAPE_BOX, A.SHAPE_SPHERE, A.SHAPE_CAPSULE], size=n, p=[0.4, 0.3, 0.3]).astype(np.int32)
    table = np.zeros(n, A.SHAPE_DTYPE)
    table["kind"] = kind
    table["params"][:, 0] = np.where(kind == A.SHAPE_SPHERE, rng.uniform(0.2, 0.5, n),
                                     np.where(kind == A.SHAPE_CAPSULE, 0.2, rng.uniform(0.2, 0.6, n)))
    table["params"][:, 1] = np.where(kind == A.SHAPE_CAPSULE, 0.3, rng.uniform(0.2, 0.6, n))
    table["params"][:, 2] = rng.uniform(0.2, 0.6, n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = grid * 1.5 + rng.uniform(-0.1, 0.1, (n, 3))
    moved_pos = pos.copy()
    moved_pos[:, :3] += rng.normal(scale=0.02, size=(n, 3))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ctx = engine.Context(0)
    ctx.set_shapes(table)
    t = {"shape": dev(np.arange(n, dtype=np.int32)), "body": dev(np.arange(n, dtype=np.int32)),
         "pos": dev(moved_pos), "rot": dev(scenes.random_quaternions(rng, n)),
         "fat_min": torch.zeros((n, 4), device="cuda"), "fat_max": torch.zeros((n, 4), device="cuda"),
         "moved": torch.zeros(n, dtype=torch.uint8, device="cuda")}
    start_pos, force = dev(pos), torch.ones(n, dtype=torch.uint8, device="cuda")
    fat = {"shape": t["shape"], "body": t["body"], "world_orientation": t["rot"], "fat_min": t["fat_min"],
           "fat_max": t["fat_max"], "moved": t["moved"]}
    # the fat AABBs of the step before
    ctx.broadphase_update(BP.make(n, n, 0, world_position=start_pos, force_reinsert=force, **fat))
    # room for four pairs a collider, kept between steps
    t["pairs"] = torch.zeros((4 * n, 2), dtype=torch.int32, device="cuda")
    t["count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    return {"ctx": ctx, "bp": BP.make(n, n, 0, world_position=t["pos"], **fat), "arrays": t}


def _run_broadphase(case, s):
    ctx, t = s["ctx"], s["arrays"]
    ctx.broadphase_update(s["bp"])
    ctx.order_in()
    ctx._check(ctx.lib.rp3dg_broadphase_pairs_device(ctx.h, ctypes.byref(s["bp"]), -1, t["pairs"].data_ptr(),
                                                     4 * case["colliders"], t["count"].data_ptr()))
    ctx.order_out()
    return {k: t[k] for k in ("fat_min", "fat_max", "moved", "count", "pairs")}


def _captured():
    with np.load(CAPTURES) as z:
        names = sorted({k.split("/")[0] for k in z.files})
        return [{k.split("/", 1)[1]: z[k] for k in z.files if k.startswith(n + "/")} for n in names]


def _prepare_dynamics(case, seed):
    rng = np.random.default_rng(seed)
    caps = _captured()
    base = [D.world_from_capture(c) for c in caps]
    order = [base[i] for i in rng.permutation(np.arange(case["worlds"]) % len(base))]
    batch, _ = D.batch_worlds(order)
    n = batch.nb_enabled
    batch.a["linear_velocity"][:n, :3] += rng.normal(scale=0.02, size=(n, 3)).astype(np.float32)
    return {"ctx": engine.Context(0), "params": D.params_from_capture(caps[0]),
            "world": D.DynWorld(batch.a, batch.nb_enabled, batch.nc_enabled, device="cuda")}


def _run_dynamics(case, s):
    w = s["ctx"].dynamics_step(s["params"], s["world"])
    return {k: w[k] for k in D.OUTPUTS}


def _scene(case, seed):
    if case["scene"] == "terrain":
        n = case["bodies"]
        cols = max(12, int(math.ceil(1.2 * math.sqrt(n))))
        sc = scenes.heightfield_world(n_bodies=n, cols=cols, rows=cols, seed=seed)
    else:
        k = case["side"]
        make = {"pile": scenes.box_pile, "mixed": scenes.mixed_world, "hulls": scenes.hull_world}[case["scene"]]
        sc = make(nx=k, ny=k, nz=k, seed=seed)
    # every body stays awake, so that a pass costs the same however many went before it
    sc.settings["sleeping_enabled"] = 0
    return sc


def _prepare_world(case, seed):
    ctx = engine.Context(0)
    world = engine.World(ctx, _scene(case, seed))
    world.update(1.0 / 60.0, case["steps"])
    return {"ctx": ctx, "world": world}


def _run_world(case, s):
    s["world"].update(1.0 / 60.0)
    return dict(zip(("position", "orientation", "linear_velocity", "angular_velocity", "sleeping"), s["world"].bodies()))


def _prepare_group(case, seed):
    # the same worlds for every seed, thrown with other velocities
    shapes, scs = scenes.many_worlds(case["worlds"], seed=case["worlds"])
    rng = np.random.default_rng(seed)
    for sc in scs:
        sc.bodies["linear_velocity"][1:] = rng.normal(scale=0.3, size=(len(sc.bodies) - 1, 3))
    scs[0].settings["sleeping_enabled"] = 0
    ctx = engine.Context(0)
    world = engine.WorldGroup(ctx, scs, shapes)
    world.update(1.0 / 120.0, case["steps"])
    return {"ctx": ctx, "world": world}


def _run_group(case, s):
    s["world"].update(1.0 / 120.0)
    return dict(zip(("position", "orientation", "linear_velocity", "angular_velocity", "sleeping"), s["world"].bodies()))


def _prepare_raycast(case, seed):
    sc = _scene(case, seed)
    ctx = engine.Context(0)
    world = engine.World(ctx, sc)
    world.update(1.0 / 60.0, case["steps"])
    if case["scene"] == "terrain":
        rays = scenes.terrain_rays(sc, case["rays"], seed=seed + 1)
    else:
        p = sc.bodies["position"][1:]
        rays = scenes.world_rays(case["rays"], p.min(0) - 1.0, p.max(0) + 1.0, seed=seed + 1)
    n = case["rays"]
    return {"ctx": ctx, "world": world, "rays": torch.from_numpy(rays.view(np.uint8)).cuda(),
            "hits": torch.zeros((n, case["hits"] * A.RAYCAST_HIT_DTYPE.itemsize), dtype=torch.uint8, device="cuda"),
            "counts": torch.zeros(n, dtype=torch.int32, device="cuda")}


def _run_raycast(case, s):
    s["world"].raycast_device(s["rays"].data_ptr(), case["rays"], s["hits"].data_ptr(), s["counts"].data_ptr(),
                              mode=case["mode"], max_hits=case["hits"])
    return {"hits": s["hits"], "counts": s["counts"]}


MLP_SIZES = ((engine.MLP_FEATURES, 64), (64, 64), (64, engine.MLP_CLASSES))


def _mlp_inputs(case, seed):
    """He-uniform weights (w1, b1, w2, b2, w3, b3 in one vector), features of the range of box pairs' and labels."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, o in MLP_SIZES:
        lim = math.sqrt(6.0 / i)
        parts += [rng.uniform(-lim, lim, i * o), rng.uniform(-0.1, 0.1, o)]
    x = rng.uniform(-1.0, 1.0, (case["samples"], engine.MLP_FEATURES))
    x[:, 12:18] = rng.uniform(0.2, 1.0, (case["samples"], 6))
    y = rng.integers(0, engine.MLP_CLASSES, case["samples"])
    return np.concatenate(parts).astype(np.float32), x.astype(np.float32), y.astype(np.uint8)


def _prepare_axis_mlp(case, seed):
    params, x, y = _mlp_inputs(case, seed)
    ctx = engine.Context(0)
    mlp = engine.AxisMLP(ctx, seed=0)
    mlp.set_params(params)
    return {"ctx": ctx, "mlp": mlp, "x": torch.from_numpy(x).cuda(), "y": torch.from_numpy(y).cuda()}


def _run_axis_mlp(case, s):
    grads, loss = s["mlp"].grads(s["x"], s["y"])
    return {"grads": grads, "loss": torch.tensor(loss, dtype=torch.float32)}


PREPARE = {"narrowphase": _prepare_narrowphase, "input_host": _prepare_input_host, "broadphase": _prepare_broadphase,
           "dynamics": _prepare_dynamics, "world": _prepare_world, "group": _prepare_group,
           "raycast": _prepare_raycast, "axis_mlp": _prepare_axis_mlp}
RUN = {"narrowphase": _run_narrowphase, "input_host": _run_input_host, "broadphase": _run_broadphase,
       "dynamics": _run_dynamics, "world": _run_world, "group": _run_group, "raycast": _run_raycast,
       "axis_mlp": _run_axis_mlp}


def prepare(case, seed):
    s = PREPARE[case["path"]](case, seed)
    s["case"] = case
    return s


def run(state):
    return RUN[state["case"]["path"]](state["case"], state)


# ---- what a pass cannot do without --------------------------------------------

# float operations per pair, orders of magnitude of the cheapest exact test
PAIR_FLOPS = {"sphere_sphere": 100, "sphere_capsule": 200, "capsule_capsule": 300, "sphere_box": 1000,
              "capsule_box": 2000, "box_box": 2500, "hull_box": 12000, "hull_hull": 60000}


def _pairs_of(case):
    batch = case.get("batch", "all")
    if batch != "all":
        return {batch: case["pairs"]}
    return dict(zip(scenes.BATCH_NAMES, scenes.batch_sizes(case["pairs"])))


def work(case):
    path = case["path"]
    if path in ("narrowphase", "input_host"):
        per = _pairs_of(case)
        n = sum(per.values())
        # shape ids, two shape records, two transforms, flag and count, ~0.4 contacts a pair; the 16-byte record twice
        bytes_ = n * (8 + 64 + 64 + 2 + 19 + (32 if case.get("coherent") else 0))
        return {"bytes": bytes_, "flops": sum(PAIR_FLOPS[b] * k for b, k in per.items())}
    if path == "broadphase":
        n = case["colliders"]
        # shape id, body, shape record, transform, fat AABB read and written, moved flag; ~1 pair a collider
        return {"bytes": n * (8 + 32 + 32 + 64 + 1 + 8), "flops": n * 600}
    if path == "dynamics":
        # per captured world on average 88 bodies, 92 manifolds, 210 points
        w = case["worlds"]
        return {"bytes": w * (88 * 380 + 92 * 100 + 210 * 60), "flops": w * (88 * 300 + 210 * 7 * 250)}
    if path in ("world", "group"):
        if path == "group":
            bodies = case["worlds"] * 147
        else:
            bodies = case["bodies"] if case["scene"] == "terrain" else case["side"] ** 3
        return {"bytes": bodies * 1500, "flops": bodies * 20000}
    if path == "raycast":
        n = case["rays"]
        return {"bytes": n * (32 + 4 + 40 * case["hits"]), "flops": n * 2000}
    n = case["samples"]
    macs = sum(i * o for i, o in MLP_SIZES)
    return {"bytes": n * (4 * engine.MLP_FEATURES + 1) + 2 * 4 * engine.MLP_NPARAMS, "flops": 6 * macs * n}


# ---- 64-bit results -------------------------------------------------------------

def _sphere_sphere_exact(shapes, pairs):
    """Contacts of a sphere-sphere batch in 64 bits (slot 0 holds the contact)."""
    n = pairs.n
    r1, r2 = (shapes["params"][i, 0].astype(np.float64) for i in (pairs.shape1, pairs.shape2))
    p1, p2 = pairs.pos1[:, :3].astype(np.float64), pairs.pos2[:, :3].astype(np.float64)
    d = p2 - p1
    dist = np.linalg.norm(d, axis=1)
    normal = d / dist[:, None]

    def unrotate(q, v):
        q = q.astype(np.float64)
        u, w = -q[:, :3], q[:, 3:]
        return v + 2.0 * np.cross(u, np.cross(u, v) + w * v)
    out = {k: np.zeros((A.MAX_CONTACTS, n, 4)) for k in ("normal_depth", "local1", "local2")}
    hit = dist < r1 + r2
    out["normal_depth"][0, :, :3] = np.where(hit[:, None], normal, 0.0)
    out["normal_depth"][0, :, 3] = np.where(hit, r1 + r2 - dist, 0.0)
    out["local1"][0, :, :3] = np.where(hit[:, None], unrotate(pairs.rot1, normal) * r1[:, None], 0.0)
    out["local2"][0, :, :3] = np.where(hit[:, None], unrotate(pairs.rot2, -normal) * r2[:, None], 0.0)
    return out


def _bf16(a):
    return torch.from_numpy(a).to(torch.bfloat16).double().numpy()


def _mlp_exact(case, seed):
    """Mean cross-entropy and its gradients in 64 bits; the model's weight matrices are bfloat16, its biases float."""
    params, x, y = _mlp_inputs(case, seed)
    ws, bs, at = [], [], 0
    for i, o in MLP_SIZES:
        ws.append(_bf16(params[at:at + i * o]).reshape(i, o))
        bs.append(params[at + i * o:at + i * o + o].astype(np.float64))
        at += i * o + o
    n = len(x)
    h0 = x.astype(np.float64)
    h1 = np.maximum(h0 @ ws[0] + bs[0], 0.0)
    h2 = np.maximum(h1 @ ws[1] + bs[1], 0.0)
    z = h2 @ ws[2] + bs[2]
    e = np.exp(z - z.max(axis=1, keepdims=True))
    p = e / e.sum(axis=1, keepdims=True)
    loss = float(np.mean(-np.log(p[np.arange(n), y])))
    dz = p
    dz[np.arange(n), y] -= 1.0
    dz /= n
    dh2 = (dz @ ws[2].T) * (h2 > 0)
    dh1 = (dh2 @ ws[1].T) * (h1 > 0)
    grads = [h0.T @ dh1, dh1.sum(0), h1.T @ dh2, dh2.sum(0), h2.T @ dz, dz.sum(0)]
    return {"grads": np.concatenate([g.ravel() for g in grads]), "loss": torch.tensor(loss, dtype=torch.float64)}


def exact(case, seed):
    path = case["path"]
    if path == "axis_mlp":
        return _mlp_exact(case, seed)
    if path in ("narrowphase", "input_host"):
        sc = _narrowphase_scene(case, seed)
        if "sphere_sphere" not in sc.batches:
            return None
        # the other batches walk GJK and SAT branches that 64 bits would take differently
        out = {name: None for name in sc.batches}
        out["sphere_sphere"] = _sphere_sphere_exact(sc.shapes, sc.batches["sphere_sphere"][1])
        return out
    return None
