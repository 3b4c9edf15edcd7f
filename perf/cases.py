"""Performance cases of the visibility path, through its public entry points.

Each case is one pass as a host program issues it: buffers, contexts and scenes stay from
pass to pass, the per-frame calls (prepare, execute, cameras) are made every time. The
kinds:

  frame      one view: Hi-Z build, then object select, meshlet cull and draw emission, by
             the two drop-in passes (HiZBuildPass, VirtualGeometryPass); optionally a range
             of moved instances is patched first
  hiz        a Hi-Z pyramid alone (a depth-only consumer, any window size)
  instances  per-draw frustum and occlusion culling (IndirectDispatchPass and
             OcclusionCullPass, separate as in the frame graph, or fused)
  shadow     per-face shadow culling of the movable draws (ShadowCullPass)
  edit       the scene's object set changed: rebuild on the device (VgBuilder), upload, and
             the cull that follows (one view, or a small batch)
  batch      many views of one scene (BatchedCull), with the cameras set and the draws
             packed for the read-back every pass; `rebind` binds new views every pass, as a
             serving slot does for each request
"""
from __future__ import annotations

import math

import numpy as np
import torch

from helio_b200 import native as N
from helio_b200 import passes as P
from helio_b200 import scene as S

PACK_CAPACITY = 2_000_000  # packed draws of a batch
PUBLISHED = 262_144        # default publication limit of a view


def listed() -> list:
    return [
        # A small indoor level in a 1024x1024 window: the call where latency counts most.
        {"name": "frame_small", "kind": "frame", "instances": 4096, "meshlets": 64, "width": 1024, "height": 1024,
         "clustered": False, "moved": 0, "lod_quality": 1, "alias": False},
        # A game level at 1080p whose characters and props move: 5% of the instances are patched.
        {"name": "frame_moving", "kind": "frame", "instances": 10000, "meshlets": 100, "width": 1920, "height": 1080,
         "clustered": False, "moved": 500, "lod_quality": 1, "alias": False},
        # A large open world at 4K: 10M meshlets.
        {"name": "frame_large", "kind": "frame", "instances": 100000, "meshlets": 100, "width": 3840, "height": 2160,
         "clustered": True, "moved": 0, "lod_quality": 1, "alias": False},
        # A free-size editor window: odd width and height, rows that no wide load fits.
        {"name": "hiz_odd", "kind": "hiz", "width": 1367, "height": 769, "alias": False},
        # The ordinary draws of a small scene, the two passes of the frame graph one after the other.
        {"name": "instances_small", "kind": "instances", "draws": 4099, "fused": False, "static_grid": 0,
         "width": 1280, "height": 720},
        # A large scene's draws in one fused pass, with a baked static Hi-Z grid.
        {"name": "instances_large", "kind": "instances", "draws": 1000000, "fused": True, "static_grid": 32,
         "width": 3840, "height": 2160},
        # One point light and the cascades moved in a small scene.
        {"name": "shadow_small", "kind": "shadow", "draws": 2000, "spots": 0, "points": 1, "dirty": 10},
        # Every light of a busy scene is dirty.
        {"name": "shadow_large", "kind": "shadow", "draws": 100000, "spots": 16, "points": 4, "dirty": 44},
        # An editor adds and removes objects: rebuild, upload, the frame that follows.
        {"name": "edit_frame", "kind": "edit", "slots": 10000, "meshes": 256, "meshlets": 100, "free": 0.05,
         "views": 0, "width": 1920, "height": 1080},
        # A streamed world region: a large rebuild for the batched path, and its first small batch.
        {"name": "edit_large", "kind": "edit", "slots": 500000, "meshes": 256, "meshlets": 100, "free": 0.05,
         "views": 4, "width": 1920, "height": 1080},
        # One serving request: a few views, bound anew every time.
        {"name": "batch_request", "kind": "batch", "instances": 30000, "meshlets": 100, "clustered": False,
         "library": 256, "main": 1, "cascades": 4, "spots": 2, "probes": 2, "scale": 0.5, "alias": True,
         "rebind": True},
        # Every view of a frame: main camera, cascades, spot lights and probes against 10M meshlets.
        {"name": "batch_85", "kind": "batch", "instances": 200000, "meshlets": 50, "clustered": True, "library": 0,
         "main": 1, "cascades": 4, "spots": 16, "probes": 64, "scale": 1.0, "alias": True, "rebind": False},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["frame", "frame", "hiz", "instances", "shadow", "edit", "batch", "batch"])
    if kind == "frame":
        n, m = _log_int(rng, 1000, 100000), rng.randint(8, 100)
        return {"kind": kind, "instances": n, "meshlets": m, "width": rng.randint(320, 3840),
                "height": rng.randint(200, 2160), "clustered": rng.random() < 0.4,
                "moved": rng.choice([0, 0, n // 20, n // 3]), "lod_quality": rng.randint(0, 3),
                "alias": rng.random() < 0.3}
    if kind == "hiz":
        return {"kind": kind, "width": _log_int(rng, 64, 7680), "height": _log_int(rng, 64, 4320),
                "alias": rng.random() < 0.3}
    if kind == "instances":
        return {"kind": kind, "draws": _log_int(rng, 100, 1000000), "fused": rng.random() < 0.5,
                "static_grid": rng.choice([0, 0, 16, 32]), "width": rng.randint(320, 3840),
                "height": rng.randint(200, 2160)}
    if kind == "shadow":
        spots, points = rng.randint(0, 16), rng.randint(0, 8)
        return {"kind": kind, "draws": _log_int(rng, 100, 100000), "spots": spots, "points": points,
                "dirty": rng.randint(1, 4 + spots + 6 * points)}
    if kind == "edit":
        return {"kind": kind, "slots": _log_int(rng, 1000, 500000), "meshes": _log_int(rng, 8, 20000),
                "meshlets": rng.randint(8, 100), "free": rng.uniform(0.0, 0.3), "views": rng.choice([0, 0, 2, 4]),
                "width": rng.randint(320, 3840), "height": rng.randint(200, 2160)}
    clustered = rng.random() < 0.5  # (a view sees far more of a scene that is not)
    return {"kind": kind, "instances": _log_int(rng, 2000, 200000 if clustered else 40000),
            "meshlets": rng.randint(8, 50), "clustered": clustered, "library": rng.choice([0, 256, 4096]),
            "main": rng.randint(0, 1), "cascades": rng.randint(0, 4), "spots": rng.randint(1, 16),
            "probes": rng.randint(0, 64), "scale": rng.uniform(0.2, 1.0), "alias": rng.random() < 0.7,
            "rebind": rng.random() < 0.5}


# ── Inputs ────────────────────────────────────────────────────────────────────────

def _bytes(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()


def _seed(seed: int) -> int:
    return S.SEED_BASE + 1000 + int(seed)


def _scene(case: dict, seed: int, instances: int, library: int = 0) -> S.Scene:
    if case.get("clustered"):
        return S.make_scene(_seed(seed), instances, case["meshlets"], 4, 1, 1000.0, 64, 20.0, mesh_library=library)
    return S.make_scene(_seed(seed), instances, case["meshlets"], 4, 0, 100.0, mesh_library=library)


def _rects(width: int, height: int) -> int:
    return max(1, int(round(20000 * (width * height) / (3840 * 2160))))


def _main(case: dict, seed: int):
    v = S.main_view(_seed(seed), case["width"], case["height"], _rects(case["width"], case["height"]))
    return v, torch.from_numpy(v.depth).cuda()


def _views(case: dict, seed: int) -> list:
    """The batch's views: a part of the 85-view mix (dicts as BatchedCull.prepare takes them)."""
    mix = S.multiview_set(_seed(seed), depth=False, scale=case["scale"])
    pick = ([("main", i) for i in range(case["main"])] + [("cascade", i) for i in range(case["cascades"])]
            + [("spot", i) for i in range(case["spots"])] + [("probe", i) for i in range(case["probes"])])
    by = {k: [v for v in mix if v.kind == k] for k in ("main", "cascade", "spot", "probe")}
    out = []
    for j, (kind, i) in enumerate(pick):
        v = by[kind][i]
        cam = v.camera
        d = S.make_depth(_seed(seed) + 2000 + j, v.width, v.height, _rects(v.width, v.height), cam.position_near[3],
                         cam.forward_far[3], kind == "cascade")
        out.append({"camera": cam, "depth": torch.from_numpy(d).cuda(), "alias_mip0": case["alias"]})
    return out


def _zero(*tensors) -> None:
    # Published buffers are defined up to the draw count only; the rest starts as zeros.
    for t in tensors:
        t.zero_()


def _packed(views: int) -> dict:
    dev = {"dtype": torch.int32, "device": "cuda"}
    return {"indirect": torch.zeros((PACK_CAPACITY, 5), **dev), "draws": torch.zeros((PACK_CAPACITY, 4), **dev),
            "offsets": torch.zeros(views + 1, **dev)}


def _owned(tensor: torch.Tensor, *owners) -> torch.Tensor:
    # A view of library memory keeps what it looks into alive.
    tensor.owners = owners
    return tensor


def _levels(hz: P.HiZBuildPass, depth: torch.Tensor) -> list:
    return [_owned(hz.level(l), hz, depth) for l in range(hz.publish().mip_count)]


def _vg_outputs(vg: P.VirtualGeometryPass) -> dict:
    o = vg.outputs()
    o.pop("capacity")
    _zero(o["indirect"], o["draws"], o["counters"], o["visibility"])
    return {k: _owned(v, vg) for k, v in o.items()}


def _prepare_frame(case: dict, seed: int) -> dict:
    sc = _scene(case, seed, case["instances"])
    view, depth = _main(case, seed)
    hz = P.HiZBuildPass(view.width, view.height, alias_mip0=case["alias"])
    hz.prepare(depth)
    vg = P.VirtualGeometryPass(view.width, view.height, lod_quality=case["lod_quality"])
    arrays = {"meshlets": _bytes(sc.meshlets), "objects": _bytes(sc.objects), "instances": _bytes(sc.instances),
              "work_items": _bytes(sc.work_items)}
    first = case["instances"] // 3
    frame = S.frame_data(sc, dirty=(first, case["moved"]), device=arrays)
    vg.prepare(frame)
    torch.cuda.synchronize()  # the pass has its copies
    keep = arrays["instances"] if case["moved"] else None
    return {"hz": hz, "vg": vg, "depth": depth, "camera": _bytes(P.camera_bytes(view.camera)), "frame": frame,
            "keep": keep, "moved": case["moved"], "pyramid": hz.publish(), "out": _vg_outputs(vg),
            "levels": _levels(hz, depth)}


def _prepare_hiz(case: dict, seed: int) -> dict:
    _, depth = _main(case, seed)
    hz = P.HiZBuildPass(case["width"], case["height"], alias_mip0=case["alias"])
    hz.prepare(depth)
    return {"hz": hz, "depth": depth, "levels": _levels(hz, depth)}


def _prepare_instances(case: dict, seed: int) -> dict:
    n = case["draws"]
    sc = S.make_scene(_seed(seed), n, 4, 1, 1, 1000.0, 64, 20.0, mesh_library=16)
    view, depth = _main(case, seed)
    hz = P.HiZBuildPass(view.width, view.height)
    hz.prepare(depth)
    hz.execute()  # the pyramid of the frame before
    stats = torch.zeros(8, dtype=torch.int32, device="cuda")
    frustum, occlusion = P.IndirectDispatchPass(stats), P.OcclusionCullPass(view.width, view.height, stats)
    g = case["static_grid"]
    if g:
        texels = np.random.default_rng(seed).uniform(5.0, 1500.0, (6 * g, g, g)).astype(np.float32)
        occlusion.set_static_hiz(torch.from_numpy(texels).cuda(), (g, g, g), (-1000.0,) * 3, (1000.0,) * 3)
    cam, inst, calls, aabbs = (_bytes(P.camera_bytes(view.camera)), _bytes(sc.instances), _bytes(sc.draw_calls),
                               _bytes(sc.aabbs))
    indirect = torch.zeros((n, 5), dtype=torch.int32, device="cuda")
    sb = P.scene_buffers(cam, inst, calls, aabbs, indirect)
    sb.instance_count = sb.draw_count = n
    return {"frustum": frustum, "occlusion": occlusion, "scene": sb, "camera": view.camera, "draws": n,
            "fused": case["fused"], "hz": hz, "pyramid": hz.publish(), "indirect": indirect, "stats": stats,
            "keep": (cam, inst, calls, aabbs, depth)}


def _prepare_shadow(case: dict, seed: int) -> dict:
    mats, faces = S.shadow_faces(_seed(seed), case["spots"], case["points"])
    inst, src = S.shadow_draws(_seed(seed), case["draws"], case["draws"])
    dirty = np.zeros(256, np.int32)
    dirty[np.random.default_rng(seed).permutation(faces)[:case["dirty"]]] = 1
    inputs = (torch.from_numpy(mats).cuda(), _bytes(inst), torch.from_numpy(src.view(np.int32)).cuda(),
              torch.from_numpy(dirty).cuda())
    sh = P.ShadowCullPass()
    out = {k: _owned(v, sh) for k, v in sh.outputs().items()}
    _zero(*out.values())
    return {"shadow": sh, "inputs": inputs, "faces": faces, "out": out}


def _prepare_edit(case: dict, seed: int) -> dict:
    objects = max(1, int(case["slots"] * (1.0 - case["free"])))
    sc = _scene(case, seed, objects, min(case["meshes"], objects))
    lib = S.library_from_scene(sc, case["slots"] / objects - 1.0, seed)
    st = {"builder": P.VgBuilder(), "library": tuple(_bytes(a) for a in (lib.pool, lib.meshes, lib.slot_mesh,
                                                                        lib.slot_instances))}
    view, depth = _main(case, seed)
    if case["views"]:
        st["scene"], st["batch"] = P.VgScene(), P.BatchedCull(max_views=case["views"])
        part = {"scale": 0.5, "main": 0, "cascades": 0, "spots": case["views"] - 1, "probes": 0, "alias": True}
        st["views"] = [{"camera": view.camera, "depth": depth, "alias_mip0": True}] + _views(part, seed)
        st["packed"] = _packed(case["views"])
        st["scene"].upload(st["builder"].run(*st["library"]))  # the region as it was before the edit
        st["batch"].prepare(st["scene"], st["views"])
        return st
    hz = P.HiZBuildPass(view.width, view.height)
    hz.prepare(depth)
    vg = P.VirtualGeometryPass(view.width, view.height)
    vg.prepare(st["builder"].run(*st["library"]))
    st.update({"hz": hz, "vg": vg, "depth": depth, "camera": _bytes(P.camera_bytes(view.camera)),
               "pyramid": hz.publish(), "out": _vg_outputs(vg)})
    return st


def _prepare_batch(case: dict, seed: int) -> dict:
    sc = _scene(case, seed, case["instances"], case["library"])
    scene = P.VgScene()
    scene.upload(S.frame_data(sc))
    views = _views(case, seed)
    batch = P.BatchedCull(max_views=len(views))
    batch.prepare(scene, views)
    st = {"scene": scene, "batch": batch, "views": views, "rebind": case["rebind"], "packed": _packed(len(views))}
    if not case["rebind"]:
        batch.autotune()  # a long-lived batch is tuned once
        st["cameras"] = _bytes(np.concatenate([P.camera_bytes(v["camera"]) for v in views]))
        st["counters"] = _batch_counters(batch, len(views))
        st["lod"] = [_owned(batch.view_outputs(v)["lod"], batch) for v in range(min(len(views), 24))]
    return st


def _batch_counters(batch: P.BatchedCull, views: int) -> torch.Tensor:
    # Every view's counters, 16 words apart, as a host reads them back in one copy.
    return _owned(P.device_view(batch.view_outputs(0)["counters"].data_ptr(), (views, 11), "<i4", (64, 4)), batch)


def prepare(case: dict, seed: int) -> dict:
    st = {"frame": _prepare_frame, "hiz": _prepare_hiz, "instances": _prepare_instances, "shadow": _prepare_shadow,
          "edit": _prepare_edit, "batch": _prepare_batch}[case["kind"]](case, seed)
    st["kind"] = case["kind"]
    return st


# ── One pass ──────────────────────────────────────────────────────────────────────

def _run_frame(st: dict):
    st["hz"].prepare(st["depth"])
    st["hz"].execute()
    if st["moved"]:
        st["frame"].instance_version += 1
    st["vg"].prepare(st["frame"])
    st["vg"].execute(st["camera"], st["pyramid"])
    return {**st["out"], "levels": st["levels"]}


def _run_hiz(st: dict):
    st["hz"].prepare(st["depth"])
    st["hz"].execute()
    return st["levels"]


def _run_instances(st: dict):
    st["stats"].zero_()
    st["frustum"].prepare(st["camera"], st["draws"])
    st["occlusion"].prepare(st["draws"])
    if st["fused"]:
        P.fused_instance_cull(st["frustum"], st["occlusion"], st["scene"], st["pyramid"], 1)
    else:
        st["frustum"].execute(st["scene"])
        st["occlusion"].execute(st["scene"], st["pyramid"], 1)
    return st["indirect"], st["stats"]


def _run_shadow(st: dict):
    st["shadow"].prepare(*st["inputs"], st["faces"])
    st["shadow"].execute()
    return st["out"]


def _built(builder: P.VgBuilder) -> dict:
    return {"built_" + k: _owned(v, builder) if isinstance(v, torch.Tensor) else v
            for k, v in builder.outputs().items()}


def _run_edit(st: dict):
    frame = st["builder"].run(*st["library"])
    if "batch" in st:
        st["scene"].upload(frame)
        st["batch"].prepare(st["scene"], st["views"])
        st["batch"].execute()
        p = st["packed"]
        st["batch"].pack_draws(p["indirect"], p["draws"], p["offsets"])
        info = st["scene"].info()
        return {**_built(st["builder"]), **p, "spans": info.max_spans, "lod0": info.lod0_meshlets}
    st["vg"].prepare(frame)
    st["hz"].prepare(st["depth"])
    st["hz"].execute()
    st["vg"].execute(st["camera"], st["pyramid"])
    return {**st["out"], **_built(st["builder"])}


def _run_batch(st: dict):
    batch, p = st["batch"], st["packed"]
    if st["rebind"]:
        batch.prepare(st["scene"], st["views"])
    else:
        batch.set_cameras_device(st["cameras"])
    batch.execute()
    batch.pack_draws(p["indirect"], p["draws"], p["offsets"])
    if st["rebind"]:
        return {**p, "counters": _batch_counters(batch, len(st["views"]))}
    return {**p, "counters": st["counters"], "lod": st["lod"]}


def run(st: dict):
    return {"frame": _run_frame, "hiz": _run_hiz, "instances": _run_instances, "shadow": _run_shadow,
            "edit": _run_edit, "batch": _run_batch}[st["kind"]](st)


# ── What a pass cannot do without ─────────────────────────────────────────────────

def _hiz_bytes(width: int, height: int, alias: bool) -> float:
    return 4.0 * width * height * ((1.0 if alias else 2.0) + 1.0 / 3.0)


# Share of a scene's LOD0 meshlets that a view tests (its selected LODs of the objects in its
# frustum): a main camera, and the average cascade, spot or probe view of a clustered scene,
# most of whose blobs lie out of their reach.
SEEN = 0.045
SEEN_SMALL_CLUSTERED = 0.0035


def _cull_bytes(objects: float, meshlets: int, main: float, other: float, clustered: bool) -> float:
    """Objects and instances once, one LOD byte per (view, object); the tested meshlets' 48
    bytes (a record is read once for all views), a third of the tests drawn (16 bytes read,
    36 written)."""
    seen = objects * meshlets * (main * SEEN + other * (SEEN_SMALL_CLUSTERED if clustered else SEEN))
    tested = min(seen, objects * meshlets)
    return objects * (128 + 64 + 16 + main + other) + 48.0 * tested + seen / 3.0 * 52.0


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "hiz":
        b = _hiz_bytes(case["width"], case["height"], case["alias"])
        return {"bytes": b, "flops": 0.75 * case["width"] * case["height"]}
    if kind == "instances":
        return {"bytes": case["draws"] * (20 + 20 + 32 + 20), "flops": case["draws"] * 120}
    if kind == "shadow":
        tests = case["draws"] * case["dirty"]
        return {"bytes": case["draws"] * (20 + 16) + tests / 10 * 20, "flops": tests * 6 * 8}
    if kind == "frame":
        b = _hiz_bytes(case["width"], case["height"], case["alias"])
        b += _cull_bytes(case["instances"], case["meshlets"], 1, 0, case["clustered"]) + 144 * 2 * case["moved"]
        return {"bytes": b, "flops": case["instances"] * (100 + 4.5 * case["meshlets"])}
    if kind == "edit":
        objects = case["slots"] * (1.0 - case["free"])
        items = objects * math.ceil(case["meshlets"] / 64)
        pool = min(case["meshes"], objects) * 1.9 * case["meshlets"]
        b = 4 * case["slots"] + objects * (144 + 144 + 128) + 8 * items + pool * 192  # rebuild
        b += objects * (2 * 144 + 2 * 128) + 128 * pool                               # upload
        b += _hiz_bytes(case["width"], case["height"], case["views"] > 0)
        b += _cull_bytes(objects, case["meshlets"], 1, max(0, case["views"] - 1), False)
        return {"bytes": b, "flops": objects * max(1, case["views"]) * 100}
    views = case["main"] + case["cascades"] + case["spots"] + case["probes"]
    px = (case["main"] * 3840 * 2160 + case["cascades"] * 2048 ** 2 + case["spots"] * 512 ** 2
          + case["probes"] * 128 ** 2) * case["scale"] ** 2
    b = _hiz_bytes(1, px, case["alias"])
    b += _cull_bytes(case["instances"], case["meshlets"], case["main"], views - case["main"], case["clustered"])
    return {"bytes": b, "flops": case["instances"] * views * (20 + 4.5 * case["meshlets"] / 4)}


# ── Exact values ──────────────────────────────────────────────────────────────────

def _exact_levels(depth: torch.Tensor) -> list:
    """The pyramid by 2x2 maxima in 64 bits; a source dimension of 1 stays, odd ones drop
    their last row or column."""
    lv = depth.double()
    mips = min(max(depth.shape).bit_length(), N.HELIO_HIZ_MAX_MIPS)
    out = [lv]
    for _ in range(mips - 1):
        h, w = lv.shape
        a = lv[0:2 * (h // 2):2].maximum(lv[1:2 * (h // 2):2]) if h > 1 else lv
        lv = a[:, 0:2 * (w // 2):2].maximum(a[:, 1:2 * (w // 2):2]) if w > 1 else a
        out.append(lv)
    return out


def exact(case: dict, seed: int):
    # Draws, counters, LODs and rebuilt records are whole numbers and bytes; the pyramids
    # are the computed values.
    if case["kind"] not in ("hiz", "frame"):
        return None
    _, depth = _main(case, seed)
    levels = _exact_levels(depth)
    if case["kind"] == "hiz":
        return levels
    return {"indirect": None, "draws": None, "counters": None, "visibility": None, "objects": None, "levels": levels}
