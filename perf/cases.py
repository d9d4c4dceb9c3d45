"""The measured workloads of the triangle ray-query library.

Every case is a pass that a program linked against the library has it do,
through its public entry points (the ctypes binding of the C ABI), over sizes
from this repository's configurations, tests and benchmark:

  probe_host          rtcIntersect1M on 1,000 rays in host memory: a tool or a game
                      loop that asks for a few rays at a time; latency decides
  camera_heightfield  1024 x 1024 primary rays on the 131k-triangle heightfield
  soup_closest        16M incoherent closest-hit rays on the 4M-triangle soup
  soup_shadow         16M shadow rays (half of them inactive) on the same soup
  robust_strided      a robust (watertight) scene, rays embedded in 96-byte records,
                      odd counts
  instances           one mesh instanced 125 times, primary rays: a two-level scene
  learned_ao          ambient-occlusion rays through the learned hit proposer
  rebuild_small       an 8k-triangle scene committed anew each frame, 4k rays
  rebuild_soup        a deforming 4M-triangle soup rebuilt each frame, 64k rays
  refit_soup          the same with RTC_BUILD_QUALITY_REFIT geometry
  batched_frame       128 independent scenes rebuilt and traced in one captured frame
  path_frame          one frame of the animated path tracer, image fetched

Queries overwrite their rays, so a pass begins by writing the rays anew (a copy
on the device, or in host memory), as the program that generates them does.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "embree-aarch64_gb300"))
from rtcgb import api  # noqa: E402

INVALID = -1  # RTC_INVALID_GEOMETRY_ID as int32

LISTED = [
    # smallest call: pageable host records, a small mesh
    {"name": "probe_host", "kind": "query", "scene": "heightfield", "tris": 8_192, "rays": "camera", "count": 1_000,
     "op": "closest", "robust": False, "stride": 80, "host": True},
    # the repository's first configuration
    {"name": "camera_heightfield", "kind": "query", "scene": "heightfield", "tris": 131_072, "rays": "camera",
     "count": 1_048_576, "op": "closest", "robust": False, "stride": 80, "host": False},
    # its second: incoherent closest hits, then shadow rays from them
    {"name": "soup_closest", "kind": "query", "scene": "soup", "tris": 4_000_000, "rays": "sphere",
     "count": 16_000_000, "op": "closest", "robust": False, "stride": 80, "host": False},
    {"name": "soup_shadow", "kind": "query", "scene": "soup", "tris": 4_000_000, "rays": "shadow",
     "count": 16_000_000, "op": "occluded", "robust": False, "stride": 48, "host": False},
    # robust scenes, records with a user's own fields behind the hit, odd sizes
    {"name": "robust_strided", "kind": "query", "scene": "heightfield", "tris": 499_998, "rays": "sphere",
     "count": 1_000_003, "op": "closest", "robust": True, "stride": 96, "host": False},
    {"name": "instances", "kind": "instances", "tris": 50_000, "copies": 125, "count": 1_048_576},
    {"name": "learned_ao", "kind": "learned", "tris": 1_000_000, "count": 2_000_000},
    {"name": "rebuild_small", "kind": "rebuild", "scene": "heightfield", "tris": 8_192, "count": 4_096,
     "refit": False},
    {"name": "rebuild_soup", "kind": "rebuild", "scene": "soup", "tris": 4_000_000, "count": 65_536, "refit": False},
    {"name": "refit_soup", "kind": "rebuild", "scene": "soup", "tris": 1_000_000, "count": 65_536, "refit": True},
    {"name": "batched_frame", "kind": "batched", "scenes": 128, "least": 1_000, "most": 60_000, "per_tri": 8},
    {"name": "path_frame", "kind": "path", "tris": 1_000_000, "width": 1280, "height": 720, "bounces": 4},
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: plain queries half of the time, the other kinds in turn."""
    kind = rng.choice(["query"] * 5 + ["instances", "learned", "rebuild", "rebuild", "batched", "path"])
    if kind == "query":
        host = rng.random() < 0.2
        op = rng.choice(["closest", "occluded"])
        rays = rng.choice(["camera", "sphere"]) if op == "closest" else rng.choice(["shadow", "sphere"])
        robust = rng.random() < 0.2
        stride = rng.choice([80, 80, 84, 96] if op == "closest" else [48, 48, 80])
        most = 1_000_000 if host else 8_000_000 if robust or stride % 16 else 16_000_000
        return {"kind": kind, "scene": rng.choice(["heightfield", "soup"]), "tris": _log_int(rng, 2_000, 4_000_000),
                "rays": rays, "count": _log_int(rng, 100, most), "op": op, "robust": robust, "stride": stride,
                "host": host}
    if kind == "instances":
        return {"kind": kind, "tris": _log_int(rng, 2_000, 50_000), "copies": _log_int(rng, 2, 125),
                "count": _log_int(rng, 10_000, 1_048_576)}
    if kind == "learned":
        return {"kind": kind, "tris": _log_int(rng, 100_000, 1_000_000), "count": _log_int(rng, 100_000, 2_000_000)}
    if kind == "rebuild":
        refit = rng.random() < 0.5
        return {"kind": kind, "scene": rng.choice(["heightfield", "soup"]),
                "tris": _log_int(rng, 2_000, 1_000_000 if refit else 4_000_000), "count": _log_int(rng, 1_000, 65_536),
                "refit": refit}
    if kind == "batched":
        return {"kind": kind, "scenes": _log_int(rng, 8, 128), "least": 1_000, "most": _log_int(rng, 4_000, 60_000),
                "per_tri": rng.randint(2, 8)}
    w = rng.randint(160, 1280)
    return {"kind": kind, "tris": _log_int(rng, 20_000, 1_000_000), "width": w, "height": w * 9 // 16,
            "bounces": rng.randint(1, 4)}


# ---------------------------------------------------------------------------
# inputs (made on the GPU from the seed alone)
# ---------------------------------------------------------------------------

_device = None


def _dev():
    global _device
    if _device is None:
        _device = api.Device(b"")
    return _device


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed & 0x7FFFFFFF)
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _unit(g, n):
    z = _uniform(g, n) * 2 - 1
    phi = _uniform(g, n) * (2 * math.pi)
    r = torch.sqrt(torch.clamp(1 - z * z, min=0))
    return torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], -1)


def _heightfield(g, tris):
    """Grid over [0,1]^2, two triangles per cell, z = 4 octaves of value noise in [0, 0.1]."""
    cells = max(2, int(round(math.sqrt(tris / 2))))
    n = cells + 1
    x = torch.arange(n, device="cuda", dtype=torch.float32) / cells
    z = torch.zeros(n, n, device="cuda")
    amp, total = 1.0, 0.0
    for octave in range(4):
        freq = 4 << octave
        lattice = _uniform(g, freq + 2, freq + 2)
        f = x * freq
        i = f.floor().long()
        t = f - i
        s = t * t * (3 - 2 * t)
        rows = lattice[i] * (1 - s)[:, None] + lattice[i + 1] * s[:, None]
        z += amp * (rows[:, i] * (1 - s)[None, :] + rows[:, i + 1] * s[None, :])
        total += amp
        amp *= 0.5
    z *= 0.1 / total
    yy, xx = torch.meshgrid(x, x, indexing="ij")
    verts = torch.stack([xx, yy, z], -1).reshape(-1, 3).contiguous()
    c = torch.arange(cells, device="cuda")
    p00 = (c[:, None] * n + c[None, :]).reshape(-1)
    p01, p10, p11 = p00 + 1, p00 + n, p00 + n + 1
    idx = torch.stack([torch.stack([p00, p01, p10], -1), torch.stack([p11, p10, p01], -1)], 1)
    return verts, idx.reshape(-1, 3).to(torch.int32).contiguous()


def _soup(g, tris):
    """Centroids from 64 Gaussians in the unit cube, vertices 1e-4 .. 1e-2 away from them."""
    means = _uniform(g, 64, 3)
    sigma = torch.exp(_uniform(g, 64) * math.log(10.0) + math.log(0.01))
    which = torch.randint(0, 64, (tris,), generator=g, device="cuda")
    cent = means[which] + torch.randn(tris, 3, generator=g, device="cuda") * sigma[which, None]
    verts = torch.empty(tris, 3, 3, device="cuda")
    for k in range(3):
        length = torch.exp(_uniform(g, tris) * math.log(100.0) + math.log(1e-4))
        verts[:, k] = cent + _unit(g, tris) * length[:, None]
    return verts.reshape(-1, 3).contiguous(), torch.arange(3 * tris, device="cuda", dtype=torch.int32).reshape(-1, 3)


def _mesh(g, scene, tris):
    return _heightfield(g, tris) if scene == "heightfield" else _soup(g, tris)


def _camera(g, count, eye=(0.5, -0.5, 0.6), look=(0.5, 0.5, 0.0), jitter=0.1):
    """About `count` pinhole rays (60 degrees, 1:1) through pixel centres, eye moved by the seed: exactly `count`."""
    w = max(1, math.isqrt(count))
    h = -(-count // w)
    eye = torch.tensor(eye, device="cuda", dtype=torch.float64) + (_uniform(g, 3).double() - 0.5) * jitter
    fwd = torch.tensor(look, device="cuda", dtype=torch.float64) - eye
    fwd = fwd / fwd.norm()
    right = torch.linalg.cross(fwd, torch.tensor([0.0, 0.0, 1.0], device="cuda", dtype=torch.float64))
    right = right / right.norm()
    up = torch.linalg.cross(right, fwd)
    th = math.tan(math.radians(30.0))
    px = ((torch.arange(w, device="cuda") + 0.5) / w * 2 - 1).double() * th
    py = (1 - (torch.arange(h, device="cuda") + 0.5) / h * 2).double() * th
    d = fwd + px[None, :, None] * right + py[:, None, None] * up
    d = d.reshape(-1, 3)[:count].float()
    return eye.float().expand_as(d), d


def _records(org, d, tnear, tfar, stride, hit):
    """RTCRayHit (80 B) or RTCRay (48 B) fields at the start of records of `stride` bytes, as float32 rows."""
    n = org.shape[0]
    r = torch.zeros(n, stride // 4, device="cuda")
    w = r.view(torch.int32)
    r[:, 0:3] = org
    r[:, 3] = tnear
    r[:, 4:7] = d
    r[:, 8] = tfar
    w[:, 9] = -1  # mask
    w[:, 10] = torch.arange(n, device="cuda", dtype=torch.int32)  # id
    if hit:
        w[:, 17:20] = INVALID
    return r


def _hit_points(records):
    """Rows whose ray hit something, with the point, the direction and the normal facing it."""
    hit = records.view(torch.int32)[:, 18] != INVALID
    p = records[:, 0:3].double() + records[:, 4:7].double() * torch.where(hit, records[:, 8], 0.0).double()[:, None]
    n = records[:, 12:15].double()
    n = n / torch.clamp(n.norm(dim=1, keepdim=True), min=1e-30)
    n = torch.where(((n * records[:, 4:7].double()).sum(1) > 0)[:, None], -n, n)
    return hit, p, n


class State:
    """What the program holds: device buffers, the committed scene, its handles."""

    def __init__(self):
        self.owned = []  # released in reverse order of their making

    def __del__(self):
        for o in reversed(self.owned):
            o.release()


def _add(st, sc, mesh, refit=False):
    verts, idx = mesh
    st.owned.append(_Kept(verts, idx))  # the scene reads the device buffers in place
    return sc.add_mesh_device(verts.data_ptr(), verts.shape[0], idx.data_ptr(), idx.shape[0],
                              quality=api.RTC_BUILD_QUALITY_REFIT if refit else None)


class _Kept:
    def __init__(self, *tensors):
        self.tensors = tensors

    def release(self):
        self.tensors = ()


def _scene(st, flags=0):
    sc = api.Scene(_dev(), flags)
    st.owned.append(sc)
    return sc


def _rays(case, g, sc):
    """The case's ray records; shadow rays start from a closest-hit pass over sphere rays."""
    n, kind, closest = case["count"], case["rays"], case["op"] == "closest"
    if kind == "camera":
        org, d = _camera(g, n)
    else:
        org, d = _uniform(g, n, 3), _unit(g, n)
        if case["scene"] == "heightfield":
            org[:, 2] *= 0.5
    if kind != "shadow":
        far = math.inf if closest else 0.5
        return _records(org, d, 0.0, far, case["stride"], closest)
    first = _records(org, d, 0.0, math.inf, 80, True)
    torch.cuda.synchronize()
    sc.intersect_ptr(first.data_ptr(), n)
    hit, p, _ = _hit_points(first)
    light = _uniform(g, 3).double()
    to = light - p
    dist = torch.clamp(to.norm(dim=1), min=1e-20)
    # misses become inactive rays, which a query leaves untouched
    tnear = torch.where(hit, 1e-4, math.inf).float()
    tfar = torch.where(hit, 0.999 * dist, 0.0).float()
    return _records(p.float(), (to / dist[:, None]).float(), tnear, tfar, case["stride"], False)


def _outputs(rows, closest):
    """The fields that a query writes, as views of the records."""
    if isinstance(rows, torch.Tensor):
        ints = rows.view(torch.int32)
    else:
        ints = rows.view(np.int32)
    if not closest:
        return {"tfar": rows[:, 8]}
    return {"tfar": rows[:, 8], "Ng": rows[:, 12:15], "u": rows[:, 15], "v": rows[:, 16], "ids": ints[:, 17:20]}


def _geometry(case, seed):
    """The triangles and rays of a query case, as prepare() makes them (rays None for shadow rays)."""
    g = _gen(seed)
    return _mesh(g, case["scene"], case["tris"]), g


def _prepare_query(case, seed, st):
    mesh, g = _geometry(case, seed)
    sc = st.scene = _scene(st, api.RTC_SCENE_FLAG_ROBUST if case["robust"] else 0)
    _add(st, sc, mesh)
    sc.commit()
    fresh = _rays(case, g, sc)
    if case["host"]:
        fresh = fresh.cpu().numpy()
        st.work = fresh.copy()
    else:
        st.work = fresh.clone()
    st.fresh = fresh
    st.closest = case["op"] == "closest"
    st.out = _outputs(st.work, st.closest)


def _run_query(st, case):
    n, stride = st.work.shape[0], st.work.shape[1] * 4
    if case["host"]:
        np.copyto(st.work, st.fresh)
        ptr = st.work.ctypes.data
    else:
        st.work.copy_(st.fresh)
        ptr = st.work.data_ptr()
    if st.closest:
        st.scene.intersect_ptr(ptr, n, stride)
    else:
        st.scene.occluded_ptr(ptr, n, stride)
    return st.out


def _prepare_instances(case, seed, st):
    g = _gen(seed)
    base = _scene(st)
    verts, idx = _soup(g, case["tris"])
    verts = (verts - 0.5) * 0.8
    _add(st, base, (verts.contiguous(), idx))
    base.commit()
    top = st.scene = _scene(st)
    k = math.ceil(case["copies"] ** (1 / 3) - 1e-9)
    rng = random.Random(seed)
    for i in range(case["copies"]):
        cell = (i % k, i // k % k, i // (k * k))
        a, s = rng.uniform(0, 2 * math.pi), rng.uniform(0.6, 1.0) / k
        c, sn = math.cos(a) * s, math.sin(a) * s
        pos = [(q + 0.5) / k for q in cell]
        top.add_instance(base, [c, sn, 0, -sn, c, 0, 0, 0, s] + pos)  # columns, then the translation
    top.commit()
    org, d = _camera(g, case["count"], eye=(0.5, -1.0, 0.8), look=(0.5, 0.5, 0.5))
    st.fresh = _records(org, d, 0.0, math.inf, 80, True)
    st.work = st.fresh.clone()
    st.closest = True
    st.out = _outputs(st.work, True)


def _prepare_learned(case, seed, st):
    """A heightfield under a soup; AO rays (length 0.2) about the camera's hits, 8 per hit, and a
    proposer trained on an earlier set of bounce rays."""
    g = _gen(seed)
    sc = st.scene = _scene(st)
    _add(st, sc, _heightfield(g, case["tris"] * 3 // 4))
    _add(st, sc, _soup(g, case["tris"] // 4))
    sc.commit()
    org, d = _camera(g, case["count"] // 4)
    view = _records(org, d, 0.0, math.inf, 80, True)
    torch.cuda.synchronize()
    sc.intersect_ptr(view.data_ptr(), view.shape[0])
    hit, p, n = _hit_points(view)
    p, n = p[hit], n[hit]

    def about_hits(count):
        which = torch.arange(count, device="cuda") // 8 % p.shape[0]
        d = _unit(g, count).double() * 0.999 + n[which]  # cosine-weighted
        return p[which].float(), (d / d.norm(dim=1, keepdim=True)).float()

    org, d = about_hits(min(case["count"], 500_000))
    log = _records(org, d, 1e-4, math.inf, 80, True)
    torch.cuda.synchronize()
    sc.intersect_ptr(log.data_ptr(), log.shape[0])
    st.prop = api.Proposer(sc, seed=7, max_treelets=1024)
    st.owned.append(st.prop)
    st.prop.train(log.data_ptr(), epochs=1, batch=16384, count=log.shape[0])
    org, d = about_hits(case["count"])
    st.fresh = _records(org, d, 1e-4, 0.2, 48, False)
    st.work = st.fresh.clone()
    st.out = _outputs(st.work, False)


def _run_learned(st, case):
    st.work.copy_(st.fresh)
    st.prop.occluded_ptr(st.work.data_ptr(), st.work.shape[0])
    return st.out


def _prepare_rebuild(case, seed, st):
    """A mesh whose vertices the program writes each frame; three frames have run."""
    mesh, g = _geometry(case, seed)
    rest, idx = mesh
    sc = st.scene = _scene(st)
    st.verts = rest.clone()
    st.gid = _add(st, sc, (st.verts, idx), case["refit"])
    st.pose = _pose(g, rest, case["scene"])
    org, d = _uniform(g, case["count"], 3), _unit(g, case["count"])
    if case["scene"] == "heightfield":
        org[:, 2] *= 0.5
    st.fresh = _records(org, d, 0.0, math.inf, 80, True)
    st.work = st.fresh.clone()
    st.closest = True
    st.out = _outputs(st.work, True)
    sc.commit()
    for _ in range(2):
        _run_rebuild(st, case)


def _pose(g, rest, scene):
    if scene == "heightfield":
        return (rest * torch.tensor([1.0, 1.0, 1.2], device="cuda")).contiguous()
    v = rest.reshape(-1, 3, 3)  # every triangle of a soup moves by itself
    return (v + (_unit(g, v.shape[0]) * 0.002)[:, None, :]).reshape(-1, 3).contiguous()


def _run_rebuild(st, case):
    st.verts.copy_(st.pose)
    L = st.scene.L
    L.rtcUpdateGeometryBuffer(L.rtcGetGeometry(st.scene.h, st.gid), api.RTC_BUFFER_TYPE_VERTEX, 0)
    st.scene.commit()
    st.work.copy_(st.fresh)
    st.scene.intersect_ptr(st.work.data_ptr(), st.work.shape[0])
    return st.out


def _batched_sizes(case):
    """Triangles of each scene: log-uniform, the same for every seed (the plan of the work)."""
    rng = random.Random(case["scenes"] * 1_000_003 + case["most"])
    return [_log_int(rng, case["least"], case["most"]) for _ in range(case["scenes"])]


def _prepare_batched(case, seed, st):
    g = _gen(seed)
    sc = st.scene = _scene(st)
    sc.set_batched(True)
    parts, start = [], [0]
    for i, tris in enumerate(_batched_sizes(case)):
        _add(st, sc, _heightfield(g, tris) if i % 2 else _soup(g, tris))
        n = tris * case["per_tri"]
        org, d = _camera(g, n // 2)
        parts.append(_records(org, d, 0.0, math.inf, 80, True))
        parts.append(_records(_uniform(g, n - n // 2, 3), _unit(g, n - n // 2), 0.0, math.inf, 80, True))
        start.append(start[-1] + n)
    sc.commit()
    st.fresh = torch.cat(parts)
    st.work = st.fresh.clone()
    st.out = _outputs(st.work, True)
    torch.cuda.synchronize()
    st.frame = api.BatchedFrame(sc, st.work.data_ptr(), start[-1], np.array(start, np.uint32),
                                pristine_ptr=st.fresh.data_ptr())
    st.owned.append(st.frame)


def _run_batched(st, case):
    st.frame.replay()
    return st.out


def _prepare_path(case, seed, st):
    g = _gen(seed)
    sc = st.scene = _scene(st)
    verts, idx = _soup(g, case["tris"])
    gid = _add(st, sc, (verts, idx), refit=True)
    torch.cuda.synchronize()
    sc.commit()
    st.pt = api.PathTracer(sc, case["width"], case["height"], bounces=case["bounces"])
    st.owned.append(st.pt)
    st.pt.animate_soup(gid, amplitude=0.002, seed=14)
    st.pt.render(0)  # captures the frame
    st.at = 1 + seed % 64


def _run_path(st, case):
    stats = st.pt.render(st.at)
    return {"image": st.pt.image(), "rays": stats["rays"]}


PREPARE = {"query": _prepare_query, "instances": _prepare_instances, "learned": _prepare_learned,
           "rebuild": _prepare_rebuild, "batched": _prepare_batched, "path": _prepare_path}
RUN = {"query": _run_query, "instances": lambda st, c: _run_query(st, {"host": False}), "learned": _run_learned,
       "rebuild": _run_rebuild, "batched": _run_batched, "path": _run_path}


def prepare(case, seed):
    st = State()
    st.case = case
    PREPARE[case["kind"]](case, seed, st)
    torch.cuda.synchronize()
    return st


def run(state):
    return RUN[state.case["kind"]](state, state.case)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

TRI_BYTES = 48        # three vertices and three indices
CLOSEST_BYTES = 84    # 48 B of ray in, tfar and 32 B of hit out
OCCLUDED_BYTES = 52   # 48 B of ray in, tfar out
TRI_FLOPS = 48        # one ray-triangle test


def work(case):
    kind = case["kind"]
    if kind == "query":
        tris, rays = case["tris"], case["count"]
        per = CLOSEST_BYTES if case["op"] == "closest" else OCCLUDED_BYTES
    elif kind == "batched":
        tris = sum(_batched_sizes(case))
        rays, per = tris * case["per_tri"], CLOSEST_BYTES
    elif kind == "path":  # camera rays, and the image written
        tris, rays, per = case["tris"], case["width"] * case["height"], 12
    elif kind == "learned":
        tris, rays, per = case["tris"], case["count"], OCCLUDED_BYTES
    else:
        tris, rays, per = case["tris"], case["count"], CLOSEST_BYTES
    flops = rays * TRI_FLOPS * (case["bounces"] if kind == "path" else 1)
    if kind == "learned":  # the 32-64-64-64-1024 network
        flops += rays * 2 * (32 * 64 + 64 * 64 + 64 * 64 + 64 * 1024)
    return {"bytes": tris * TRI_BYTES + rays * per, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit answers: every ray against every triangle
# ---------------------------------------------------------------------------

MOST_PAIRS = 7e10  # ray-triangle pairs that torch tests in under 20 seconds


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("query", "rebuild") or float(case["tris"]) * case["count"] > MOST_PAIRS:
        return None
    if kind == "query" and case["rays"] == "shadow":
        return None  # rays that start from the library's own hits
    (verts, idx), g = _geometry(case, seed)
    if kind == "query":
        rays, closest = _rays(case, g, None), case["op"] == "closest"
    else:
        verts = _pose(g, verts, case["scene"])
        org, d = _uniform(g, case["count"], 3), _unit(g, case["count"])
        if case["scene"] == "heightfield":
            org[:, 2] *= 0.5
        rays, closest = _records(org, d, 0.0, math.inf, 80, True), True
    tri = verts.double()[idx.long()]
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    ng = torch.linalg.cross(e1, e2)  # of the library's orientation: (v2 - v0) x (v0 - v1)
    n, m = rays.shape[0], tri.shape[0]
    best_t = rays[:, 8].double().clone()
    best = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    best_uv = torch.zeros(n, 2, dtype=torch.float64, device="cuda")
    chunk = max(1, 40_000_000 // m)
    step = min(m, 40_000_000)
    for a in range(0, n, chunk):
        o, d = rays[a:a + chunk, 0:3].double(), rays[a:a + chunk, 4:7].double()
        near = rays[a:a + chunk, 3].double()[:, None]
        for b in range(0, m, step):
            # scalar triple products as matrix products over (ray, triangle)
            den = d @ ng[b:b + step].T
            oxd = torch.linalg.cross(o, d)
            v0b, e1b, e2b, nb = v0[b:b + step], e1[b:b + step], e2[b:b + step], ng[b:b + step]
            # u den = d . (e2 x c), v den = -d . (e1 x c), t den = ng . c with c = v0 - o
            u = (d @ torch.linalg.cross(e2b, v0b).T - oxd @ e2b.T) / den
            v = -(d @ torch.linalg.cross(e1b, v0b).T - oxd @ e1b.T) / den
            t = ((v0b * nb).sum(1)[None, :] - o @ nb.T) / den
            ok = (den != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > near) & (t <= best_t[a:a + chunk, None])
            t = torch.where(ok, t, math.inf)
            tb, k = t.min(1)
            hit = torch.gather(ok, 1, k[:, None])[:, 0]
            rows = torch.nonzero(hit)[:, 0]
            best_t[a + rows] = tb[rows]
            best[a + rows] = k[rows] + b
            best_uv[a + rows, 0] = u[rows, k[rows]]
            best_uv[a + rows, 1] = v[rows, k[rows]]
    hit = best >= 0
    if not closest:
        return {"tfar": torch.where(hit, -math.inf, best_t)}
    normal = torch.where(hit[:, None], ng[best.clamp(min=0)], 0.0)
    return {"tfar": best_t, "Ng": normal, "u": best_uv[:, 0], "v": best_uv[:, 1], "ids": None}
