"""The work this framework is used for, as cases that can be timed.

Each case is one pass of a user's program through the public binding
(master-of-puppets_b200/mopcuda.py): a viewport's frames in the engine's modes (plain,
orbiting camera, dense geometry, shadows, transparency, wireframe, flat with fog), a batch
of viewports, a burst of served requests, and the work around frames (environment maps,
skinning).  Sizes and scenes are those of the repository's generators
(scenes.py), its benchmark and its tests.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the program's resident state: device, scene, buffers
  run(state)          one pass, with its outputs
  exact(case, seed)   the outputs that are computed numbers, in 64 bits
  work(case)          bytes and operations of a pass that no implementation can do without
"""
import ctypes as C
import dataclasses
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "master-of-puppets_b200"))
import mopcuda  # noqa: E402
import scenes  # noqa: E402

PICKS = 1000       # pick queries after an interactive frame
ORBIT_FRAMES = 4   # frames of one orbit pass
SKIN_BONES = 64
ENV_W, ENV_H = 512, 256


def listed():
    return [
        # an editor viewport showing one object: a frame, its image and a thousand picks (IDs
        # and depths); the smallest frame, where latency and launches count
        {"name": "viewport", "kind": "viewport", "width": 800, "height": 600, "ssaa": 1},
        # a full-HD anti-aliased view of a large lit scene while the camera orbits: frames
        # back to back, each image read while the next one renders
        {"name": "orbit", "kind": "orbit", "width": 1920, "height": 1080, "ssaa": 2,
         "instances": 256},
        # CAD-like geometry: two million pixel-sized triangles, clipping and coplanar ties
        {"name": "dense", "kind": "dense", "width": 1920, "height": 1080, "tris": 2000000},
        # a frame with the sun casting shadows, everything a caster; odd window size
        {"name": "shadowed", "kind": "shadowed", "width": 1365, "height": 767, "ssaa": 1,
         "instances": 128},
        # a third of the instances transparent, composited in order over the rest
        {"name": "blended", "kind": "blended", "width": 1280, "height": 720, "ssaa": 2,
         "instances": 96},
        # the wireframe mode on a modelling session's scene
        {"name": "wireframe", "kind": "wireframe", "width": 1280, "height": 720, "ssaa": 1,
         "tris": 40000},
        # flat shading with fog, tone mapping and vignette, at three samples per axis
        {"name": "fogged", "kind": "fogged", "width": 801, "height": 449, "ssaa": 3,
         "meshes": 60},
        # 64 viewports of every size over one resident scene in one launch; the largest call
        {"name": "batch", "kind": "batch", "views": 64, "max_px": 1920 * 1080,
         "instances": 256},
        # a render service's burst: renders and picks over four scenes, some instances moved
        {"name": "served", "kind": "served", "renders": 16, "picks": 4, "tris": 300000},
        # a new environment map: its irradiance, prefiltered and BRDF maps
        {"name": "environment", "kind": "environment", "width": ENV_W, "height": ENV_H},
        # a character crowd's vertices skinned for the next frame
        {"name": "skin", "kind": "skin", "vertices": 100000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice([c["kind"] for c in listed()])
    w = _log(rng, 320, 1920)
    h = max(200, int(w * rng.uniform(0.5, 0.75)))
    ssaa = rng.choice([1, 1, 2])
    if kind == "viewport":
        return {"kind": kind, "width": w, "height": h, "ssaa": ssaa}
    if kind in ("orbit", "shadowed", "blended"):
        return {"kind": kind, "width": w, "height": h, "ssaa": ssaa,
                "instances": _log(rng, 9, 128 if kind == "blended" else 256)}
    if kind == "dense":
        return {"kind": kind, "width": w, "height": h, "tris": _log(rng, 20000, 2000000)}
    if kind == "wireframe":
        return {"kind": kind, "width": w, "height": h, "ssaa": 1, "tris": _log(rng, 5000, 60000)}
    if kind == "fogged":
        return {"kind": kind, "width": _log(rng, 320, 1000), "height": rng.randint(200, 600),
                "ssaa": rng.choice([1, 2, 3]), "meshes": rng.randint(6, 80)}
    if kind == "batch":
        return {"kind": kind, "views": rng.randint(2, 64), "max_px": _log(rng, 20000, 900000),
                "instances": _log(rng, 16, 256)}
    if kind == "served":
        return {"kind": kind, "renders": rng.randint(2, 16), "picks": rng.randint(1, 4),
                "tris": _log(rng, 50000, 400000)}
    if kind == "environment":
        ew = _log(rng, 64, 1024)
        return {"kind": kind, "width": ew, "height": max(32, ew // 2)}
    return {"kind": kind, "vertices": _log(rng, 1000, 200000)}


# --------------------------------------------------------------------------
# scenes
# --------------------------------------------------------------------------

def _small_mesh_scene(seed, tris, width, height):
    """About `tris` triangles of icospheres and tori under the large scene's lights."""
    rng = np.random.default_rng(seed)
    sc = scenes.config2(seed=seed, width=width, height=height, ssaa=1, instances=0,
                        tex_size=256, n_textures=1)
    proto = [scenes.icosphere(3, 1.0, (1, 1, 1, 1)), scenes.torus(32, 24, 1.0, 0.35, (1, 1, 1, 1))]
    have = 0
    while have < tris:
        v, i = proto[int(rng.integers(0, 2))]
        v = v.copy()
        v[:, 6:10] = (*rng.uniform(0.2, 1.0, 3), 1.0)
        s = float(rng.uniform(0.8, 3.0))
        m = scenes.mat_trs(rng.uniform(-14, 14, 3), scenes.random_rotation(rng), (s, s, s))
        sc.meshes.append(scenes.Mesh(v, i, len(sc.meshes) + 1, m, float(rng.uniform(0, 1)),
                                     float(rng.uniform(0.05, 1)), texture=0))
        have += i.size // 3
    return sc


def _scene(case, seed):
    kind = case["kind"]
    if kind == "viewport":
        return scenes.config1(seed, case["width"], case["height"], case["ssaa"])
    if kind == "dense":
        return scenes.config3(seed, case["width"], case["height"], case["tris"])
    if kind == "wireframe":
        sc = _small_mesh_scene(seed, case["tris"], case["width"], case["height"])
        return dataclasses.replace(sc, wireframe=True)
    if kind == "fogged":
        sc = scenes.small_scene(seed, case["width"], case["height"], case["ssaa"],
                                case["meshes"])
        post = (scenes.POST_GAMMA | scenes.POST_TONEMAP | scenes.POST_VIGNETTE |
                scenes.POST_FOG | scenes.POST_FXAA)
        return dataclasses.replace(sc, smooth=False, post_effects=post,
                                   fog=((0.6, 0.7, 0.8, 1.0), 0.9, 1.0))
    sc = scenes.config2(seed, case.get("width", 1920), case.get("height", 1080),
                        case.get("ssaa", 1), case["instances"], tex_size=512, n_textures=2)
    if kind == "shadowed":
        sc.lights[0] = dataclasses.replace(sc.lights[0], cast_shadows=True)
    if kind == "blended":
        for k in range(0, len(sc.meshes), 3):
            sc.meshes[k] = dataclasses.replace(sc.meshes[k], opacity=0.35 + 0.1 * (k % 5),
                                               blend_mode=(1, 2, 3, 1)[k % 4])
    return sc


def _environment(case, seed):
    """An HDR panorama: a smooth sky with a bright sun and a little noise, RGBA float32."""
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    phi = ((np.arange(w) + 0.5) / w - 0.5) * 2.0 * math.pi
    th = ((np.arange(h) + 0.5) / h - 0.5) * math.pi
    d = np.stack([np.cos(th)[:, None] * np.cos(phi), np.repeat(np.sin(th)[:, None], w, 1),
                  np.cos(th)[:, None] * np.sin(phi)], -1)
    sun = rng.normal(size=3)
    sun[1] = abs(sun[1]) + 0.3
    sun /= np.linalg.norm(sun)
    glow = 20.0 * np.exp(80.0 * (d @ sun - 1.0))
    env = np.ones((h, w, 4), np.float32)
    env[..., :3] = (rng.uniform(0.2, 0.8, 3) * (1.2 + d[..., 1:2]) + glow[..., None] +
                    rng.uniform(0.0, 0.05, (h, w, 3)))
    return env


def _skin_input(case, seed):
    """Vertices (position, normal, 4 joints, 4 weights that sum to 1; 44 bytes) and bones."""
    rng = np.random.default_rng(seed)
    vc = case["vertices"]
    f = np.zeros((vc, 11), np.float32)
    f[:, 0:3] = rng.uniform(-1, 1, (vc, 3))
    n = rng.normal(size=(vc, 3))
    f[:, 3:6] = n / np.linalg.norm(n, axis=1, keepdims=True)
    f[:, 6] = rng.integers(0, SKIN_BONES, (vc, 4)).astype(np.uint8).view(np.float32)[:, 0]
    w = rng.uniform(0.05, 1.0, (vc, 4))
    f[:, 7:11] = w / w.sum(1, keepdims=True)
    bones = np.stack([scenes.mat_trs(rng.uniform(-1, 1, 3), scenes.random_rotation(rng),
                                     (1.0, 1.0, 1.0)) for _ in range(SKIN_BONES)])
    return f, bones.astype(np.float32)


# --------------------------------------------------------------------------
# the program's state
# --------------------------------------------------------------------------

class _State:
    """What a program holds for its device; everything is given back with it."""

    def __init__(self, case):
        self.case, self.kind = case, case["kind"]
        self.dev = mopcuda.Device(0)
        self.closers = []

    def keep(self, x):
        self.closers.append(x)
        return x

    def host(self, h, w):
        """A page-locked image; it lives as long as anyone holds it."""
        return torch.empty((h, w, 4), dtype=torch.uint8, pin_memory=True).numpy()

    def __del__(self):
        for x in reversed(self.closers):
            x.close()
        self.dev.close()


class _Buffers:
    def __init__(self, dev, handles):
        self.dev, self.handles = dev, handles

    def close(self):
        for b in self.handles:
            self.dev.L.mopcuda_buffer_destroy(self.dev.h, b)


def prepare(case, seed):
    st = _State(case)
    kind, dev = st.kind, st.dev
    if kind == "environment":
        st.env = _environment(case, seed)
        return st
    if kind == "skin":
        f, st.bones = _skin_input(case, seed)
        L = dev.L
        hs = [L.mopcuda_buffer_create(dev.h, f.ctypes.data, f.nbytes) for _ in range(2)]
        st.bind, st.dst = hs
        st.keep(_Buffers(dev, hs))
        st.layout = mopcuda.MopCudaDeformLayout(44, 0, 12, 24, 28)
        return st
    if kind == "served":
        rng = np.random.default_rng(seed)
        scs = [_small_mesh_scene(seed * 4 + k, int(case["tris"] * f), 1280, 720)
               for k, f in enumerate((0.2, 0.5, 0.8, 1.0))]
        ibl = scenes.procedural_ibl(scs[0].sun_dir)
        st.scenes = [st.keep(mopcuda.ResidentScene(dev, sc, ibl)) for sc in scs]
        st.server = st.keep(mopcuda.Server(dev, 100 << 30, max_views=32))
        ids = [st.server.add_scene(rs) for rs in st.scenes]
        sizes = [(256, 256), (1280, 720), (1920, 1080), (2560, 1440)]
        st.requests = []
        for k in range(case["renders"] + case["picks"]):
            n = int(rng.integers(0, 4))
            w, h = sizes[(k * k + k // 4) % 4 if k < case["renders"] else k % 4]
            v = scenes.batch_views(scs[n], 1, int(rng.integers(0, 1 << 30)))[0]
            v = dataclasses.replace(v, width=w, height=h, ssaa=1)
            if k < case["renders"]:
                st.requests.append((ids[n], v, st.host(h, w), None))
            else:
                xy = np.stack([rng.integers(0, w, 64), rng.integers(0, h, 64)], 1).astype(np.int32)
                st.requests.append((ids[n], v, None, xy))
        # the tick's moved instances: 1 % of each scene's
        st.moves = []
        for rs in st.scenes:
            for _ in range(max(1, len(rs.meshes) // 100)):
                k = int(rng.integers(0, len(rs.meshes)))
                m = np.array(rs.scene.meshes[k].transform, np.float32)
                m[12:15] += rng.uniform(-1, 1, 3)
                st.moves.append((rs, k, m))
        return st
    sc = _scene(case, seed)
    ibl = scenes.procedural_ibl(sc.sun_dir) if sc.env else None
    if kind == "batch":
        # the same windows for every seed, other cameras
        cams = scenes.batch_views(sc, case["views"], seed)
        st.views = [dataclasses.replace(v, eye=c.eye, target=c.target) for v, c in
                    zip(scenes.batch_views(sc, case["views"], 4, 128 * 128, case["max_px"]), cams)]
        st.batch = st.keep(mopcuda.BatchRenderer(dev, sc, st.views, ibl))
        st.outs = [st.host(v.height, v.width) for v in st.views]
        return st
    st.r = r = st.keep(mopcuda.SceneRenderer(dev, sc, ibl))
    if kind == "orbit":  # the poses' draw tables
        a0 = np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi)
        e = np.asarray(sc.eye)
        rad = math.hypot(e[0], e[2])
        st.poses = []
        for k in range(ORBIT_FRAMES):
            a = a0 + 0.02 * k
            r.scene = dataclasses.replace(sc, eye=(rad * math.cos(a), float(e[1]),
                                                   rad * math.sin(a)))
            r.update_camera()
            st.poses.append((r.draws, r.draw_array))
        st.outs = [st.host(sc.height, sc.width) for _ in range(ORBIT_FRAMES)]
        return st
    st.out = st.host(sc.height, sc.width)
    if kind == "viewport":
        st.xy = scenes.pick_points(sc, PICKS, seed)
    return st


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

def run(st):
    kind, dev = st.kind, st.dev
    if kind == "environment":
        dev.ibl_from_env(st.env)
        m = dev.ibl_maps()
        return {"irr": m["irr"], "pf": m["pf"], "brdf": m["brdf"]}
    if kind == "skin":
        L, vc = dev.L, st.case["vertices"]
        mopcuda._check(L.mopcuda_skin_apply(dev.h, st.dst, st.bind, vc, C.byref(st.layout),
                                            st.bones.ctypes.data, SKIN_BONES), "skin_apply")
        p = L.mopcuda_buffer_read(st.dst)
        shadow = (C.c_uint8 * (vc * 44)).from_address(p)
        shadow.owner = st  # the buffer lives as long as this view of it
        b = np.frombuffer(shadow, np.uint8).reshape(vc, 44)
        return {"position": b[:, 0:12].view(np.float32), "normal": b[:, 12:24].view(np.float32),
                "rest": b[:, 24:44]}
    if kind == "served":
        for rs, k, m in st.moves:
            rs.set_model(k, m)
        srv = st.server
        tickets = [srv.submit_render(s, v, out=out) if xy is None else srv.submit_pick(s, v, xy)
                   for s, v, out, xy in st.requests]
        for t in tickets:
            srv.wait(t)
        return [t.color if t.pick is None else t.pick for t in tickets]
    if kind == "batch":
        st.batch.submit()
        st.batch.wait()
        return st.batch.read_all(mopcuda.BATCH_PRESENTED, st.outs)
    r = st.r
    if kind == "orbit":
        for (draws, array), out in zip(st.poses, st.outs):
            r.draws, r.draw_array = draws, array
            r.submit()
            r.color_async(out)
        r.wait_readback()
        return st.outs
    r.submit()
    r.color(st.out)
    if kind == "viewport":
        ids, dep, hits = r.pick(st.xy)
        return {"color": st.out, "pick_ids": ids, "pick_depths": dep, "pick_hits": hits}
    return {"color": st.out}


# --------------------------------------------------------------------------
# 64-bit values of the computed outputs.  A frame's colours and IDs are bytes and whole
# numbers, and its depth is defined by the rasterizer's own sequence of single-precision
# additions, so frames have none.
# --------------------------------------------------------------------------

def _frames_of(w, h):
    """Texel directions and tangent frames of an equirectangular map: T, N, B [h*w, 3]."""
    phi = ((np.arange(w) + 0.5) / w - 0.5) * 2.0 * math.pi
    th = ((np.arange(h) + 0.5) / h - 0.5) * math.pi
    n = np.stack([np.cos(th)[:, None] * np.cos(phi), np.repeat(np.sin(th)[:, None], w, 1),
                  np.cos(th)[:, None] * np.sin(phi)], -1).reshape(-1, 3)
    up = np.where(np.abs(n[:, 1:2]) > 0.99, np.array([0.0, 0.0, 1.0]), np.array([0.0, 1.0, 0.0]))
    t = np.cross(up, n)
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    return t, n, np.cross(n, t)


def _hammersley(n):
    rev = np.array([int("{:032b}".format(s)[::-1], 2) for s in range(n)], np.float64)
    return np.arange(n) / n, rev * 2.0 ** -32


def _lookup(env, d):
    h, w = env.shape[:2]
    u = np.arctan2(d[..., 2], d[..., 0]) / (2.0 * math.pi) + 0.5
    v = np.arcsin(np.clip(d[..., 1], -1.0, 1.0)) / math.pi + 0.5
    fx, fy = (u - np.floor(u)) * (w - 1), (v - np.floor(v)) * (h - 1)
    x0, y0 = fx.astype(np.int64), fy.astype(np.int64)
    x1, y1 = (x0 + 1) % w, np.minimum(y0 + 1, h - 1)
    sx, sy = (fx - x0)[..., None], (fy - y0)[..., None]
    top = env[y0, x0] * (1 - sx) + env[y0, x1] * sx
    bot = env[y1, x0] * (1 - sx) + env[y1, x1] * sx
    return top * (1 - sy) + bot * sy


def _rgba(rgb):
    return np.concatenate([rgb, np.ones((rgb.shape[0], 1))], 1).reshape(-1)


def _exact_environment(case, seed):
    env = _environment(case, seed)[..., :3].astype(np.float64)
    # irradiance: 128 cosine-distributed samples per texel of a 64x32 map
    t, n, b = _frames_of(64, 32)
    x1, x2 = _hammersley(128)
    acc = np.zeros_like(n)
    for s in range(128):
        st, ct, ph = math.sqrt(1 - x1[s]), math.sqrt(x1[s]), 2 * math.pi * x2[s]
        acc += _lookup(env, t * (st * math.cos(ph)) + n * ct + b * (st * math.sin(ph)))
    irr = _rgba(acc / 128)
    # prefiltered: 64 GGX samples per texel of a 128x64 map and its four smaller levels
    x1, x2 = _hammersley(64)
    pf = []
    for lev in range(5):
        t, n, b = _frames_of(128 >> lev, 64 >> lev)
        a2 = max((lev / 4) ** 4, 1e-7)
        acc, tot = np.zeros_like(n), np.zeros((n.shape[0], 1))
        for s in range(64):
            ct = math.sqrt((1 - x1[s]) / (1 + (a2 - 1) * x1[s]))
            st, ph = math.sqrt(max(0.0, 1 - ct * ct)), 2 * math.pi * x2[s]
            hv = t * (st * math.cos(ph)) + n * ct + b * (st * math.sin(ph))
            lv = 2 * (n * hv).sum(1, keepdims=True) * hv - n
            ndl = np.maximum((n * lv).sum(1, keepdims=True), 0.0)
            acc += _lookup(env, lv) * ndl
            tot += ndl
        pf.append(_rgba(acc / tot))
    # BRDF table: 256x256 of (n.v, roughness)
    rough = ((np.arange(256) + 0.5) / 256)[:, None]
    nv = ((np.arange(256) + 0.5) / 256)[None, :]
    a2, k = np.maximum(rough ** 4, 1e-7), rough * rough * 0.5
    scale, bias = np.zeros((256, 256)), np.zeros((256, 256))
    for s in range(64):
        ct = np.sqrt((1 - x1[s]) / (1 + (a2 - 1) * x1[s]))
        hx = np.sqrt(1 - ct * ct) * math.cos(2 * math.pi * x2[s])
        vdh = np.sqrt(1 - nv * nv) * hx + nv * ct
        ndl = 2 * vdh * ct - nv
        ok = ndl > 0
        l = np.where(ok, ndl, 1.0)
        vc = np.maximum(vdh, 0.0)
        vis = np.where(ok, nv / (nv * (1 - k) + k) * l / (l * (1 - k) + k) * vc /
                       (ct * nv + 1e-6), 0.0)
        fc = (1 - vc) ** 5
        scale += vis * (1 - fc)
        bias += vis * fc
    lut = np.stack([scale / 64, bias / 64, np.zeros_like(scale), np.ones_like(scale)], -1)
    return {"irr": irr, "pf": np.concatenate(pf), "brdf": lut.reshape(-1)}


def exact(case, seed):
    if case["kind"] == "environment":
        return _exact_environment(case, seed)
    if case["kind"] == "skin":
        f, bones = _skin_input(case, seed)
        joints = np.ascontiguousarray(f[:, 6:7]).view(np.uint8)
        m = bones.astype(np.float64).reshape(-1, 4, 4).transpose(0, 2, 1)
        p, n, w = (f[:, s].astype(np.float64) for s in (slice(0, 3), slice(3, 6), slice(7, 11)))
        pos, nrm = np.zeros_like(p), np.zeros_like(n)
        for j in range(4):
            mj = m[joints[:, j]]
            pos += w[:, j:j + 1] * (np.einsum("vij,vj->vi", mj[:, :3, :3], p) + mj[:, :3, 3])
            nrm += w[:, j:j + 1] * np.einsum("vij,vj->vi", mj[:, :3, :3], n)
        nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
        return {"position": pos, "normal": nrm, "rest": None}
    return None


# --------------------------------------------------------------------------
# what a pass cannot do without: geometry read once, 12 bytes per sample and the image
# written once, the image or result over to the host; the lighting of half the samples
# --------------------------------------------------------------------------

def _geometry(instances):
    """Bytes of the large scene's vertices (48 B) and indices (4 B)."""
    kinds = ([(81920, 40962), (20480, 10242)] + [(16384, 8385)] * 6 +
             [(5120, 2562)] * max(0, instances - 8))[:instances]
    return sum(12 * t + 48 * v for t, v in kinds)


def work(case):
    kind = case["kind"]
    lit = 80 + 120 * 7 + 150  # float operations of a sample under seven lights and IBL
    if kind == "environment":
        texels = 64 * 32 * 128 + sum((128 >> l) * (64 >> l) for l in range(5)) * 64
        return {"bytes": 16 * (case["width"] * case["height"] + 64 * 32 + 10912 + 65536),
                "flops": 60 * texels + 65536 * 64 * 30}
    if kind == "skin":
        return {"bytes": 88 * case["vertices"], "flops": 4 * 45 * case["vertices"]}
    if kind == "served":
        px = case["renders"] * 1500000.0 + case["picks"] * 1500000.0
        return {"bytes": 16 * px + 4 * 2.5 * case["tris"] * 36, "flops": 0.3 * lit * px}
    if kind == "batch":
        lo, hi = 128 * 128, case["max_px"]
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo
        s = case["views"] * mean * 2.5
        return {"bytes": 12 * s + 4 * case["views"] * mean + _geometry(case["instances"]),
                "flops": 0.45 * lit * s}
    px = case["width"] * case["height"]
    s = px * case.get("ssaa", 1) ** 2
    if kind == "viewport":
        return {"bytes": 16 * s + 4 * px, "flops": 0.5 * 350 * s}
    if kind == "dense":
        return {"bytes": 156 * case["tris"] + 16 * s, "flops": 0.5 * 320 * s}
    if kind == "wireframe":
        return {"bytes": 36 * case["tris"] + 16 * s, "flops": 0}
    if kind == "fogged":
        return {"bytes": 12 * s + 4 * px, "flops": 60 * s}
    frames = ORBIT_FRAMES if kind == "orbit" else 1
    return {"bytes": frames * (_geometry(case["instances"]) + 12 * s + 4 * px),
            "flops": frames * 0.45 * lit * s}
