"""The collision work that a program using this library has it do, as cases to
be timed: loading meshes into OBB trees, colliding batches of entity pairs
with contacts and uncollide rays, the mid phase alone, whole collision frames,
ray shooting, the broad phase, deforming meshes and the differentiable
penetration energy. Every case goes through the public calls (capi.Context,
energy.penetration_energy) from host or device inputs as that call takes them.

Inputs are seeded and synthetic: the meshes and poses of
inmyroom_vulkan_gb300.scenes, in the sizes of this repository's benchmark and
tests. Results that a call returns in no fixed order (colliding pairs, frame
records, broad pairs) are put into order by the ids they carry. Results go into
buffers of a fixed capacity that the program keeps, with their counts beside
them, as a program that runs every frame does.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from inmyroom_vulkan_gb300 import capi, energy, scenes

RECORD_BYTES, TRI_BYTES, QUERY_BYTES, RAY_BYTES, PAIR_BYTES = 64, 48, 72, 32, 36
SAT_FLOPS, TRI_TEST_FLOPS = 714, 147  # a box-pair test with its transform; a triangle-pair test


# ------------------------------------------------------------------- the cases

def listed() -> list:
    return [
        # One entity pair through the drop-in call (mid and narrow phase, contacts, rays): a game
        # with two objects, or an engine that calls per pair. Latency and launches.
        dict(name="pair_single", kind="pairs", queries=1, tris_a=2048, tris_b=2048, check="none"),
        # The rigid-pair workload: two 2,048-triangle bodies at 1,000 sampled poses in one batch
        # (a planner or a sampler), the FP64 recheck deciding.
        dict(name="pair_poses_1000", kind="pairs", queries=1000, tris_a=2048, tris_b=2048, check="robust"),
        # The scene of the benchmark: 256 rigid entities of 500..20,000 triangles, all overlapping
        # pairs in one step, queries from the host and results into pinned host buffers.
        dict(name="scene_256", kind="scene", entities=256, models=256, tri_lo=500, tri_hi=20000, check="recheck"),
        # The mid phase alone, candidate leaf pairs in the reference's order: what the engine's
        # OBBtreesCollision call returns when only it is replaced.
        dict(name="midphase_128", kind="mid", entities=128, models=64, tri_lo=500, tri_hi=20000),
        # 10,000 uneven mesh pairs in one captured launch, queries resident on the device.
        dict(name="sweep_10000", kind="sweep", queries=10000, models=48, tri_lo=256, tri_hi=65536),
        # One model loaded: its tree built from vertex and index buffers and read back (tree cache).
        dict(name="build_one", kind="build", models=1, tri_lo=5003, tri_hi=5003, read_back=True),
        # A level loaded: 256 models' trees built in one call, then the level's first collide step.
        dict(name="build_level", kind="build", models=256, tri_lo=500, tri_hi=20000, read_back=False),
        # A frame of skinned, morphed meshes: 64 tubes of 12,000 triangles deformed, their trees
        # refitted, collided with a 198,450-triangle heightfield, contacts and rays read.
        dict(name="deform_64", kind="deform", meshes=64, rings=100, around=60, targets=8, grid=316),
        # Forward and backward of the penetration energy for the same meshes (pose optimisation).
        dict(name="energy_64", kind="energy", meshes=64, rings=100, around=60, targets=8, grid=316),
        # The uncollide rays of a scene's step shot at its trees.
        dict(name="shoot_256", kind="shoot", entities=256, models=64, tri_lo=500, tri_hi=20000),
        # A whole collision frame of the engine: broad phase, collide, shooting, delta split.
        dict(name="frame_256", kind="frame", entities=256, models=64, tri_lo=500, tri_hi=20000),
        # The broad phase of a crowded level.
        dict(name="broad_4096", kind="broad", entities=4096),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["pairs", "scene", "mid", "sweep", "build", "deform", "energy", "shoot", "frame", "broad"])
    if kind == "pairs":
        return dict(kind=kind, queries=_log_int(rng, 1, 1000), tris_a=_log_int(rng, 500, 4000),
                    tris_b=_log_int(rng, 500, 4000), check=rng.choice(["none", "recheck", "robust"]))
    if kind == "sweep":
        return dict(kind=kind, queries=_log_int(rng, 300, 9000), models=rng.randint(8, 40), tri_lo=256, tri_hi=32768)
    if kind == "build":
        one = rng.random() < 0.5
        if one:
            t = _log_int(rng, 100, 20000)
            return dict(kind=kind, models=1, tri_lo=t, tri_hi=t, read_back=True)
        return dict(kind=kind, models=_log_int(rng, 8, 200), tri_lo=500, tri_hi=_log_int(rng, 2000, 20000),
                    read_back=False)
    if kind in ("deform", "energy"):
        return dict(kind=kind, meshes=_log_int(rng, 2, 60), rings=rng.randint(20, 100), around=rng.randint(12, 60),
                    targets=rng.randint(1, 8), grid=rng.randint(64, 300))
    if kind == "broad":
        return dict(kind=kind, entities=_log_int(rng, 32, 4000))
    case = dict(kind=kind, entities=_log_int(rng, 12, 120 if kind == "mid" else 250), models=rng.randint(8, 60),
                tri_lo=500, tri_hi=_log_int(rng, 4000, 20000))
    if kind == "scene":
        case["check"] = rng.choice(["none", "recheck", "robust"])
    return case


# -------------------------------------------------------------------- inputs

CHECK_FLAGS = {"none": 0, "recheck": capi.CG_RECHECK, "robust": capi.CG_ROBUST}


def _rng(case, seed: int) -> np.random.Generator:
    return np.random.Generator(np.random.PCG64([int(seed), len(case["kind"])]))


def _model(k: int, tris: int, radius: float, rng) -> scenes.Mesh:
    return scenes.uv_sphere(tris, radius, 0.01 * radius, rng) if k % 2 == 0 else scenes.hull_blob(tris, radius, rng)


def _models(case, rng, radius=None) -> list:
    out = []
    for k in range(case["models"]):
        t = int(round(math.exp(rng.uniform(math.log(case["tri_lo"]), math.log(case["tri_hi"])))))
        out.append(_model(k, t, rng.uniform(0.5, 2.0) if radius is None else radius, rng))
    return out


def _level(case, rng, n: int):
    """(models, the model of each entity, world matrices): n entities at the benchmark scene's
    density (256 in a 20 m cube)."""
    models = _models(case, rng)
    which = np.arange(n) % len(models)
    cube = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    mats = np.stack([scenes.pose(scenes.random_rotation(rng), rng.uniform(0.0, cube, size=3)) for _ in range(n)])
    return models, which, mats


def _relative(first, second) -> np.ndarray:
    return np.stack([capi.relative_matrix(a, b) for a, b in zip(first, second)])


def _level_queries(models, which, mats, ids) -> tuple:
    pairs = scenes.aabb_pairs([models[w] for w in which], mats)
    if len(pairs) == 0:
        pairs = np.array([[0, 1]], np.uint32)
    tree = np.asarray(ids)[which]
    return pairs, capi.make_queries(tree[pairs[:, 0]], tree[pairs[:, 1]],
                                    _relative(mats[pairs[:, 0]], mats[pairs[:, 1]]))


def _deforming(case, seed: int) -> scenes.DeformingScene:
    return scenes.deforming(n_meshes=case["meshes"], seed=int(seed), rings=case["rings"], around=case["around"],
                            n_targets=case["targets"], grid=case["grid"])


def _buffer(n: int, dtype, pinned: bool = False) -> np.ndarray:
    return torch.zeros(n * dtype.itemsize, dtype=torch.uint8, pin_memory=pinned).numpy().view(dtype)


def _result_buffers(queries: int, rays: int, pinned: bool = False) -> dict:
    """The program's own buffers for a step's results, kept from frame to frame."""
    return dict(rays=_buffer(rays, capi.RAY_DTYPE, pinned), averages=_buffer(queries, capi.RAY_AVERAGE_DTYPE, pinned),
                contacts=_buffer(rays, capi.CONTACT_DTYPE, pinned))


def _level_buffers(entities: int, pinned: bool = False) -> dict:
    return _result_buffers(8 * entities + 64, 512 * entities + 4096, pinned)


def prepare(case, seed: int) -> dict:
    kind = case["kind"]
    rng = _rng(case, seed)
    s = dict(kind=kind, case=case)
    if kind == "pairs":
        ctx = capi.Context()
        ids = ctx.build_trees([_model(0, case["tris_a"], 1.0, rng), _model(1, case["tris_b"], 1.0, rng)])
        n = case["queries"]
        a = np.stack([scenes.pose(scenes.random_rotation(rng), np.zeros(3)) for _ in range(n)])
        # a single pair is a pair that the broad phase let through: its bodies touch
        reach = 1.5 if n > 1 else 1.2
        b = np.stack([scenes.pose(scenes.random_rotation(rng), scenes.ball_point(rng, reach)) for _ in range(n)])
        s.update(ctx=ctx, flags=capi.CG_CONTACTS | CHECK_FLAGS[case["check"]],
                 queries=capi.make_queries(np.full(n, ids[0]), np.full(n, ids[1]), _relative(a, b)),
                 out=_result_buffers(n, 512 * n + 1024))
    elif kind in ("scene", "mid", "shoot"):
        ctx = capi.Context()
        models, which, mats = _level(case, rng, case["entities"])
        pairs, q = _level_queries(models, which, mats, ctx.build_trees(models))
        s.update(ctx=ctx, queries=q)
        if kind == "scene":
            s["flags"] = capi.CG_CONTACTS | CHECK_FLAGS[case["check"]]
            s["out"] = _level_buffers(case["entities"], pinned=True)
            s["pairs"] = _buffer(4096 * case["entities"], capi.TRI_PAIR_DTYPE, pinned=True)
            ctx.set_host_outputs(s["pairs"], s["out"]["rays"], s["out"]["averages"])
        if kind == "mid":
            s["out"] = _buffer(6144 * case["entities"] + 65536, capi.LEAF_PAIR_DTYPE)
        if kind == "shoot":
            ctx.collide(q, capi.CG_CONTACTS)
            rays, avg = ctx.rays(), ctx.ray_averages()
            # the rays of a step are grouped by query, then side: the order shooting takes them in
            sq = np.zeros(len(q), capi.SHOOT_QUERY_DTYPE)
            sq["tree_a"], sq["tree_b"] = q["tree_a"], q["tree_b"]
            sq["first_global"], sq["second_global"] = mats[pairs[:, 0]], mats[pairs[:, 1]]
            sq["n_first"], sq["n_second"] = avg["rays_first"], avg["rays_second"]
            s["shots"] = sq
            s["rays"] = np.ascontiguousarray(np.concatenate([rays["origin"], rays["direction"]], 1))
            s["deltas"] = np.zeros((8 * case["entities"] + 64, 3), np.float32)
    elif kind == "sweep":
        n = case["queries"]
        ctx = capi.Context(max_queries=16384, max_tri_pairs=1 << 23, max_leaf_pairs=1 << 24)
        ids = ctx.build_trees(_models(case, rng, radius=1.0))
        qa, qb = rng.integers(0, len(ids), n), rng.integers(0, len(ids), n)
        a = np.stack([scenes.pose(scenes.random_rotation(rng), np.zeros(3)) for _ in range(n)])
        b = np.stack([scenes.pose(scenes.random_rotation(rng), scenes.ball_point(rng, 2.52)) for _ in range(n)])
        q = capi.make_queries(ids[qa], ids[qb], _relative(a, b))
        d_q = torch.from_numpy(q.view(np.uint8).copy()).cuda()
        torch.cuda.synchronize()
        ctx.graph_capture(d_q.data_ptr(), n, 0)
        s.update(ctx=ctx, d_queries=d_q, pairs=torch.zeros(512 * n + 65536, 9, dtype=torch.int32, device="cuda"))
    elif kind == "build":
        ctx = capi.Context()
        s.update(ctx=ctx, meshes=_models(case, rng))
        if case["read_back"]:
            # a split leaves two or more triangles' worth of leaves: fewer nodes than triangles
            t = case["tri_hi"] + 64
            s["out"] = dict(node_obbs=np.zeros((t, 2, 12), np.float32), node_ref=np.zeros((t, 2), np.uint32),
                            node_cnt=np.zeros((t, 2), np.uint32), tri_pos=np.zeros((t, 9), np.float32),
                            tri_nrm=np.zeros((t, 9), np.float32), tri_idx=np.zeros((t, 3), np.uint32))
        else:
            n = case["models"]
            s["out"] = _level_buffers(n)
            cube = 20.0 * (n / 256.0) ** (1.0 / 3.0)
            mats = np.stack([scenes.pose(scenes.random_rotation(rng), rng.uniform(0.0, cube, size=3)) for _ in range(n)])
            _, q = _level_queries(s["meshes"], np.arange(n), mats, np.arange(n))
            s["queries"] = q  # by model; the trees' ids are put in once they are built
    elif kind in ("deform", "energy"):
        sc = _deforming(case, seed)
        ctx = capi.Context()
        rest = ctx.export_tree(int(ctx.build_trees([sc.mesh])[0]))
        field = int(ctx.build_trees([sc.field])[0])
        n = case["meshes"]
        relative = _relative(sc.models, np.tile(scenes.pose(np.eye(3), np.zeros(3)), (n, 1)))
        if kind == "energy":
            parent, offsets = scenes.chain_skeleton(sc)
            s["collider"] = energy.DeformingCollider(ctx, rest, capi.Skeleton(parent, offsets), sc.vertices, sc.joints,
                                                     sc.weights, sc.inverse_bind, field, relative)
            s["axis_angles"] = torch.tensor(sc.axis_angles, dtype=torch.float32, device="cuda", requires_grad=True)
            s["morph_weights"] = torch.tensor(sc.morph_weights, device="cuda", requires_grad=True)
        else:
            dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda()
                   for k, v in (("vertices", sc.vertices), ("morph", sc.morph_weights),
                                ("joints", sc.joints.view(np.int16)), ("weights", sc.weights),
                                ("matrices", sc.joint_matrices), ("bind", sc.inverse_bind))}
            V = sc.vertices.shape[1]
            s["positions"] = torch.zeros(n, V, 4, device="cuda")
            s["trees"] = [ctx.upload_flat(rest) for _ in range(n)]
            s["views"] = [capi.cg_deform_view(V, case["targets"], 1, sc.axis_angles.shape[1],
                                              dev["vertices"][m].data_ptr(), dev["morph"][m].data_ptr(),
                                              dev["joints"].data_ptr(), dev["weights"].data_ptr(),
                                              dev["matrices"][m].data_ptr(), dev["bind"].data_ptr()) for m in range(n)]
            s["places"] = [s["positions"][m].data_ptr() for m in range(n)]
            q = capi.make_queries(s["trees"], [field] * n, relative)
            s.update(dev=dev, n_vertices=V, d_queries=torch.from_numpy(q.view(np.uint8).copy()).cuda(),
                     out=_result_buffers(n, 4096 * n + 4096))
        s["ctx"] = ctx
    elif kind == "frame":
        ctx = capi.Context()
        models, which, mats = _level(case, rng, case["entities"])
        ids = np.asarray(ctx.build_trees(models))[which]
        previous, callback = scenes.frame_motion(scenes.Scene([models[w] for w in which], mats, np.zeros((0, 2))),
                                                 seed=int(seed))
        s.update(ctx=ctx, ids=ids, mats=mats, previous=previous, callback=callback,
                 out=np.zeros(8 * case["entities"] + 64, capi.FRAME_RESULT_DTYPE))
    elif kind == "broad":
        ctx = capi.Context(max_contacts=0)
        n = case["entities"]
        ids = np.asarray(ctx.build_trees([_model(k, 96, 0.3 + 0.1 * k, rng) for k in range(8)]))
        cube = 20.0 * (n / 256.0) ** (1.0 / 3.0)
        mats = np.stack([scenes.pose(scenes.random_rotation(rng), rng.uniform(0.0, cube, size=3)) for _ in range(n)])
        s.update(ctx=ctx, ids=ids[rng.integers(0, len(ids), n)], mats=mats,
                 callback=(rng.random(n) < 0.7).astype(np.uint8), cap=64 * n, out=np.zeros((64 * n, 2), np.uint32))
    else:
        raise ValueError(kind)
    return s


# -------------------------------------------------------------------- one pass

class _DeviceInts:
    """n rows of 32-bit words at a device address, for torch."""

    def __init__(self, ptr: int, n: int, words: int):
        self.__cuda_array_interface__ = dict(shape=(n, words), typestr="<i4", data=(ptr, False), version=3, strides=None)


def _rays(rays) -> dict:
    return dict(query=rays["query"], side=rays["side"], origin=rays["origin"], direction=rays["direction"])


def _averages(avg) -> dict:
    return dict(first=avg["first"], second=avg["second"], rays_first=avg["rays_first"],
                rays_second=avg["rays_second"])


def _contacts(c) -> dict:
    return dict(query=c["query"], side=c["side"], tri=c["tri"], mask=c["mask"], average=c["weighted_avg"],
                weight=c["weight"])


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _step_results(ctx, out, st, contacts: bool) -> dict:
    """The step's results read into the program's buffers."""
    ctx.rays(out["rays"], st["rays"])
    ctx.ray_averages(out["averages"], st.get("queries"))
    res = dict(rays=_rays(out["rays"]), averages=_averages(out["averages"]), n_rays=st["rays"],
               tri_pairs=st["tri_pairs"], tri_tests=st["tri_tests"], leaf_pairs=st["leaf_pairs"])
    if contacts:
        ctx.contacts(out["contacts"], st["contacts"])
        res["contacts"] = _contacts(out["contacts"])
    return res


def _run_pairs(s):
    ctx, q = s["ctx"], s["queries"]
    st = ctx.collide(q, s["flags"])
    st["queries"] = len(q)
    res = _step_results(ctx, s["out"], st, contacts=True)
    res.update(rechecked=st["rechecked"], disagreements=st["disagreements"])
    return res


def _run_scene(s):
    st = s["ctx"].collide(s["queries"], s["flags"])
    return dict(rays=_rays(s["out"]["rays"]), averages=_averages(s["out"]["averages"]), n_rays=st["rays"],
                tri_pairs=st["tri_pairs"], tri_tests=st["tri_tests"], leaf_pairs=st["leaf_pairs"],
                rechecked=st["rechecked"], disagreements=st["disagreements"])


def _run_mid(s):
    ctx, out = s["ctx"], s["out"]
    ctx.collide(s["queries"], capi.CG_KEEP_LEAF_PAIRS | capi.CG_DFS_ORDER | capi.CG_MID_ONLY)
    n = ctypes.c_uint64()
    rc = ctx.lib.cg_read_leaf_pairs(ctx.h, out.ctypes.data, len(out), ctypes.byref(n))
    if rc != capi.CG_OK:
        raise capi.CgError(rc, ctx.last_error())
    return dict(count=n.value, **{k: out[k] for k in ("query", "offset_a", "offset_b", "count_a", "count_b")})


def _run_sweep(s):
    ctx = s["ctx"]
    ctx.graph_launch(energy.current_stream())
    st = ctx.sync_stats()
    n = st["tri_pairs"]
    words = torch.as_tensor(_DeviceInts(ctx.device_results()[0], n, 9), device="cuda")
    key = (words[:, 0].long() << 40) | (words[:, 1].long() << 20) | words[:, 2].long()
    torch.index_select(words, 0, torch.argsort(key), out=s["pairs"][:n])
    return dict(pairs=s["pairs"][:, :3], segments=s["pairs"].view(torch.float32)[:, 3:], n_pairs=n,
                tri_tests=st["tri_tests"], leaf_pairs=st["leaf_pairs"])


def _run_build(s):
    ctx, out = s["ctx"], s["out"]
    ids = ctx.build_trees(s["meshes"])
    if s["case"]["read_back"]:
        tree = ctx.export_tree(int(ids[0])).arrays()
        res = dict(root=tree.pop("root"), nodes=len(tree["node_ref"]))
        for k, v in tree.items():
            out[k][:len(v)] = v
        res.update(out)
    else:
        q = s["queries"].copy()
        q["tree_a"], q["tree_b"] = ids[q["tree_a"]], ids[q["tree_b"]]
        st = ctx.collide(q, capi.CG_CONTACTS)
        st["queries"] = len(q)
        res = _step_results(ctx, out, st, contacts=True)
        res["node_pairs"] = st["node_pairs"]
    for i in ids:
        ctx.free_tree(int(i))
    return res


def _run_deform(s):
    ctx, stream, n = s["ctx"], energy.current_stream(), len(s["trees"])
    ctx.deform_batch(s["views"], s["places"], stream)
    ctx.tree_refit_batch(s["trees"], s["places"], [s["n_vertices"]] * n, stream)
    ctx.collide_async(s["d_queries"].data_ptr(), n, capi.CG_CONTACTS, stream)
    st = ctx.sync_stats()
    ctx.rays(s["out"]["rays"], st["rays"])
    ctx.ray_averages(s["out"]["averages"], n)
    return dict(positions=s["positions"], rays=_rays(s["out"]["rays"]), averages=_averages(s["out"]["averages"]),
                n_rays=st["rays"], tri_pairs=st["tri_pairs"])


def _run_energy(s):
    e = energy.penetration_energy(s["axis_angles"], s["morph_weights"], s["collider"])
    g = torch.autograd.grad(e, (s["axis_angles"], s["morph_weights"]))
    return dict(energy=e.detach(), grad_axis_angles=g[0], grad_morph_weights=g[1])


def _run_shoot(s):
    s["ctx"].shoot_packed(s["shots"], s["rays"], out=s["deltas"])
    return s["deltas"]


def _run_frame(s):
    res = s["ctx"].collision_frame(s["ids"], s["mats"], s["previous"], s["callback"])
    out = s["out"]
    out[:len(res)] = res[np.lexsort((res["second"], res["first"]))]
    return dict(count=len(res), **{k: out[k] for k in ("first", "second", "first_delta", "second_delta")})


def _run_broad(s):
    p = s["ctx"].broad_phase(s["ids"], s["mats"], s["callback"], cap=s["cap"])
    s["out"][:len(p)] = p[np.lexsort((p[:, 1], p[:, 0]))]
    return dict(count=len(p), pairs=s["out"])


# ---------------------------------------------------- what a pass cannot do without

def _mean_tris(case) -> float:
    lo, hi = case["tri_lo"], case["tri_hi"]
    return float(lo) if hi == lo else (hi - lo) / math.log(hi / lo)


def _collide_work(queries: float, tris: float, touched: float = 0.12) -> tuple:
    """(bytes, flops) of `queries` overlapping pairs of trees of `tris` triangles each: the boxes
    and triangles near the contact read once (`touched` of the tree), the rays written once; a
    box test and three triangle tests per touched triangle."""
    near = 2.0 * touched * tris
    return (queries * (QUERY_BYTES + near * (TRI_BYTES + RECORD_BYTES) + 0.05 * near * RAY_BYTES),
            queries * near * (SAT_FLOPS + 3 * TRI_TEST_FLOPS))


def _build_work(tris: float) -> tuple:
    """Corners read and records, triangles and links written once; per level of the tree (about
    log2 of the leaves) the sums, products and projections of every corner."""
    levels = max(1.0, math.log2(max(tris, 8.0) / 2.0))
    return tris * (36 + TRI_BYTES + 2 * RECORD_BYTES), tris * 3 * levels * 33


def work(case) -> dict:
    kind = case["kind"]
    if kind == "pairs":
        b, f = _collide_work(case["queries"], 0.5 * (case["tris_a"] + case["tris_b"]))
        b = min(b, case["queries"] * (QUERY_BYTES + 2000) + (case["tris_a"] + case["tris_b"]) * (TRI_BYTES + RECORD_BYTES))
    elif kind in ("scene", "mid"):
        b, f = _collide_work(2.0 * case["entities"], _mean_tris(case), 0.06)
        b = min(b, case["models"] * _mean_tris(case) * (TRI_BYTES + RECORD_BYTES) + 2.0 * case["entities"] * 4000)
    elif kind == "sweep":
        b, f = _collide_work(0.5 * case["queries"], _mean_tris(case), 0.06)
        b = case["models"] * _mean_tris(case) * (TRI_BYTES + RECORD_BYTES) + case["queries"] * (QUERY_BYTES + 120 * PAIR_BYTES)
    elif kind == "build":
        b, f = (case["models"] * x for x in _build_work(_mean_tris(case)))
    elif kind in ("deform", "energy"):
        V = (case["rings"] + 1) * case["around"] * case["meshes"]
        T = 2 * case["rings"] * case["around"] * case["meshes"]
        b = V * (16 * (1 + case["targets"]) + 24 + 16) + T * (TRI_BYTES + RECORD_BYTES) * 2.0
        f = V * (6 * case["targets"] + 4 * 32) + T * (100 + 0.3 * SAT_FLOPS)
        if kind == "energy":
            b, f = b + V * 16 * (1 + case["targets"]), 1.5 * f
    elif kind == "shoot":
        rays = 110.0 * case["entities"]
        b, f = rays * 24 + case["models"] * _mean_tris(case) * 0.2 * (TRI_BYTES + RECORD_BYTES), rays * 2 * 60 * 60
    elif kind == "frame":
        b, f = _collide_work(case["entities"], _mean_tris(case), 0.06)
        b = min(b, case["models"] * _mean_tris(case) * (TRI_BYTES + RECORD_BYTES) + case["entities"] * 8000)
        f += 110.0 * case["entities"] * 2 * 60 * 60
    else:
        n = case["entities"]
        b, f = n * (69 + 24) + 12.0 * n * 8, n * n / 2.0 * 6
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------ the values in 64 bits

def exact(case, seed: int):
    """The deformed positions, and the penetration energy with its gradients, in FP64. The other
    cases' outputs are verdicts of FP32 predicates and values selected by them, whose definition
    is the FP32 procedure itself."""
    if case["kind"] == "deform":
        sc = _deforming(case, seed)
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device="cuda")  # noqa: E731
        skin = torch.matmul(t(sc.joint_matrices).view(case["meshes"], -1, 4, 4).mT,
                            t(sc.inverse_bind).view(-1, 4, 4).mT)
        return dict(positions=_deformed(sc, t(sc.morph_weights), skin))
    if case["kind"] == "energy":
        return _exact_energy(case, seed)
    return None


def _deformed(sc, morph_weights, skin) -> torch.Tensor:
    """Morph targets, then linear-blend skinning, (n, V, 4); skin (n, bones, 4, 4)."""
    t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device="cuda")  # noqa: E731
    verts = t(sc.vertices)
    v = verts[:, :, 0] + torch.einsum("nvtc,nt->nvc", verts[:, :, 1:], morph_weights)
    joints, weights = torch.as_tensor(sc.joints[:, 0].astype(np.int64), device="cuda"), t(sc.weights[:, 0])
    out = torch.zeros_like(v)
    for k in range(joints.shape[1]):
        out = out + weights[None, :, k, None] * torch.einsum("nvij,nvj->nvi", skin[:, joints[:, k]], v)
    return out


def _rotation(a: torch.Tensor) -> torch.Tensor:
    """(..., 3) axis-angle -> (..., 3, 3)."""
    th = torch.sqrt((a * a).sum(-1) + 1e-300)[..., None, None]
    z = torch.zeros_like(a[..., 0])
    K = torch.stack([z, -a[..., 2], a[..., 1], a[..., 2], z, -a[..., 0], -a[..., 1], a[..., 0], z], -1)
    K = K.view(a.shape[:-1] + (3, 3))
    eye = torch.eye(3, dtype=a.dtype, device=a.device)
    return eye + torch.sin(th) / th * K + (1 - torch.cos(th)) / (th * th) * (K @ K)


def _distances(p: torch.Tensor, q: torch.Tensor) -> tuple:
    """(normal of the triangles p, distances of q's corners to p's plane): not normalised, those
    below 1e-6 are zero, as the engine's triangle test takes them."""
    n = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    d = ((q - p[:, :1]) * n[:, None]).sum(-1)
    return n, torch.where(d.abs() < 1e-6, 0.0, d)


def _interval(x: torch.Tensor, d: torch.Tensor) -> tuple:
    """(whether there is one, its ends): the interval that a triangle with corners at x along the
    planes' common line, d from the other plane, covers of that line."""
    d0, d1, d2 = d.unbind(-1)
    alone = torch.where(d0 * d1 > 0, 2, torch.where(d0 * d2 > 0, 1, torch.where(
        (d1 * d2 > 0) | (d0 != 0), 0, torch.where(d1 != 0, 1, 2))))[:, None]
    xa, da = x.gather(1, alone), d.gather(1, alone)
    others = torch.cat([(alone + 1) % 3, (alone + 2) % 3], 1)
    ends = xa + (x.gather(1, others) - xa) * da / (da - d.gather(1, others))
    return (d != 0).any(-1), ends.amin(1), ends.amax(1)


def _crossing(p: torch.Tensor, q: torch.Tensor) -> torch.Tensor:
    """Whether triangles p and q (n, 3, 3) intersect and are not coplanar (Moller 1997)."""
    n1, dq = _distances(p, q)
    n2, dp = _distances(q, p)
    apart = ((dq > 0).all(-1) | (dq < 0).all(-1)) | ((dp > 0).all(-1) | (dp < 0).all(-1))
    line = torch.linalg.cross(n1, n2)
    line = line / line.norm(dim=-1, keepdim=True)
    ok1, lo1, hi1 = _interval((p * line[:, None]).sum(-1), dp)
    ok2, lo2, hi2 = _interval((q * line[:, None]).sum(-1), dq)
    return ~apart & ok1 & ok2 & (hi1 >= lo2) & (hi2 >= lo1)


def _depths(points: torch.Tensor, plane: torch.Tensor) -> torch.Tensor:
    """Summed squared depth of the vertices (n, 3, 3) below the planes of the triangles (n, 3, 3)."""
    normal = torch.linalg.cross(plane[:, 1] - plane[:, 0], plane[:, 2] - plane[:, 0])
    normal = normal / normal.norm(dim=-1, keepdim=True)
    s = ((points - plane[:, :1]) * normal[:, None]).sum(-1)
    return torch.clamp(s, max=0.0).square().sum()


def _exact_energy(case, seed: int) -> dict:
    sc = _deforming(case, seed)
    t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device="cuda")  # noqa: E731
    n, bones = sc.axis_angles.shape[:2]
    aa = t(sc.axis_angles.astype(np.float32)).requires_grad_()
    mw = t(sc.morph_weights).requires_grad_()
    parent, offsets = scenes.chain_skeleton(sc)
    local = torch.zeros(n, bones, 4, 4, dtype=torch.float64, device="cuda")
    local[..., 3, 3] = 1.0
    local = torch.cat([torch.cat([_rotation(aa), t(offsets)[None, :, :, None].expand(n, -1, -1, -1)], -1),
                       local[..., 3:, :]], -2)
    world = []
    for j in range(bones):
        world.append(local[:, j] if parent[j] < 0 else world[parent[j]] @ local[:, j])
    skin = torch.stack(world, 1) @ t(sc.inverse_bind).view(-1, 4, 4).mT
    place = t(sc.models).view(n, 4, 4).mT
    pos = torch.einsum("nij,nvj->nvi", place, _deformed(sc, mw, skin))[..., :3]
    tri = pos[:, torch.as_tensor(sc.mesh.indices.reshape(-1, 3).astype(np.int64), device="cuda")].reshape(-1, 3, 3)
    field = t(sc.field.points)[torch.as_tensor(sc.field.indices.reshape(-1, 3).astype(np.int64), device="cuda")]
    # the heightfield's cells under each triangle
    g = case["grid"]
    with torch.no_grad():
        cell = tri.detach()[..., [0, 2]] * ((g - 1) / 20.0)
        lo = (cell.amin(1) - 1e-3).floor().long()
        hi = (cell.amax(1) + 1e-3).floor().long()
        ok = ((hi >= 0) & (lo <= g - 2)).all(1)
        lo, hi = lo.clamp(0, g - 2), hi.clamp(0, g - 2)
        size = torch.where(ok[:, None], hi - lo + 1, 0)
        count = size[:, 0] * size[:, 1]
        owner, other = [], []
        for part in torch.arange(len(tri), device="cuda").split(1 << 16):
            o = torch.repeat_interleave(part, count[part])
            k = torch.arange(len(o), device="cuda") - torch.repeat_interleave(count[part].cumsum(0) - count[part], count[part])
            w = size[o, 1]
            c = (lo[o, 0] + k // w) * (g - 1) + lo[o, 1] + k % w
            o, c = o.repeat_interleave(2), torch.stack([2 * c, 2 * c + 1], 1).reshape(-1)
            near = (tri[o, :, 1].amin(1) <= field[c, :, 1].amax(1)) & (tri[o, :, 1].amax(1) >= field[c, :, 1].amin(1))
            o, c = o[near], c[near]
            cut = _crossing(tri[o], field[c])
            owner.append(o[cut])
            other.append(c[cut])
    a, b = tri[torch.cat(owner)], field[torch.cat(other)]
    e = _depths(a, b) + _depths(b, a)
    ga, gm = torch.autograd.grad(e, (aa, mw))
    return dict(energy=e.detach(), grad_axis_angles=ga, grad_morph_weights=gm)
