"""Cases for measuring the framework's speed: what its users have it do, through its public entry points.

A case names a kind of use (`_KINDS`) and its sizes; `listed` holds one case or two of each kind, `draw` gives more of the
same ranges.  Every session sees a seeded synthetic scene (spheres and boxes on a ground plane, axial noise, dropped
pixels) from the repository's generator: camera models, volumes, truncation and thresholds are those of the tests and of
the benchmark.  A state holds a few consecutive frames and goes through them back and forth, so that a session tracks and
fuses in every pass as a running scan does.  The weight cap is the storage's own (65535): with the usual 100 a state that
is passed through some hundred times would stop updating the voxels it sees.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vcl-volume-scanner_gb300"))

import vs_scanner as V  # noqa: E402

COS20 = math.cos(math.radians(20.0))
MAX_W = 65535.0
# the serving mix: (width, height, focal length, principal point) and voxels per axis over 1.5 m
MIX_SIZES = ((320, 240, 285.0, 160.0, 120.0), (512, 424, 365.0, 255.5, 211.5), (640, 480, 525.0, 319.5, 239.5))
MIX_VOLUMES = (128, 256, 384, 512)
STORAGE = {"int16": V.VS_TSDF_INT16, "fp16": V.VS_TSDF_FP16, "fp32": V.VS_TSDF_FP32}
REDUCE = {"fp32": V.VS_REDUCE_FP32, "two_sum": V.VS_REDUCE_KAHAN, "fp64": V.VS_REDUCE_FP64}


def listed():
    return [
        # the smallest scan: one 320x240 sensor, a 1 m cube, a host frame in and the pose out of each call
        dict(name="frame_qvga_256", kind="frame", w=320, h=240, f=285.0, dim=256, size=1.0, mu=0.03),
        # the usual desktop scan: 640x480 into 512^3 with the 20 degree normal test
        dict(name="frame_vga_512", kind="frame", w=640, h=480, f=525.0, dim=512, size=1.5, mu=0.02),
        # a colour scan at known poses that shows its model after each frame
        dict(name="colour_view_384", kind="colour", w=512, h=424, f=365.0, dim=384, size=1.5, mu=0.02),
        # a serving process with a few users: one frame of each submitted as it arrives, the results polled
        dict(name="serve_6", kind="serve", sessions=6, mix=11),
        # sixteen sessions of uneven size advanced together, frames from ordinary host memory
        dict(name="batch_16", kind="batch", sessions=16, mix=5, pinned=False),
        # the full batch of the serving mix, frames in pinned memory
        dict(name="batch_64", kind="batch", sessions=64, mix=5, pinned=True),
        # the tracker alone, with FP64 sums: a caller that fuses elsewhere or checks a pose
        dict(name="track_vga_fp64", kind="track", w=640, h=480, f=525.0, dim=256, size=1.5, mu=0.03, reduce="fp64"),
        # posed fusion (turntable, marker board): integrate at a known pose and ray-cast the model, half-precision volume
        dict(name="fuse_render_fp16", kind="fuse", w=512, h=424, f=365.0, dim=384, size=1.5, mu=0.02, tsdf="fp16"),
        # fusion into the caller's own buffer, odd image size
        dict(name="fuse_own_buffer", kind="own", w=431, h=333, f=380.0, dim=256, size=1.2, mu=0.025),
        # the viewer: a scan rendered at display size, with colour
        dict(name="view_960x540", kind="view", w=960, h=540, f=790.0, dim=512, size=1.5, mu=0.02, vertex=False),
        # one full-HD depth image smoothed for another program
        dict(name="filter_1080p", kind="filter", w=1920, h=1080),
        # a rig with a colour camera of its own: each depth frame seen from it
        dict(name="register_rig", kind="register", w=512, h=424, f=365.0, wr=1280, hr=960),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(_KINDS)
    if kind == "filter":
        return dict(kind=kind, w=int(_log(rng, 64, 1920)), h=int(_log(rng, 48, 1080)))
    if kind in ("serve", "batch"):
        c = dict(kind=kind, sessions=int(_log(rng, 2, 12 if kind == "serve" else 48)), mix=rng.randrange(1000))
        if kind == "batch":
            c["pinned"] = rng.random() < 0.5
        return c
    w = int(_log(rng, 200, 1100 if kind == "view" else 720))
    h = int(w * rng.uniform(0.55, 0.85))
    c = dict(kind=kind, w=w, h=h, f=w * rng.uniform(0.7, 0.9))
    if kind == "register":
        return dict(c, wr=int(w * rng.uniform(0.8, 2.5)), hr=int(h * rng.uniform(0.8, 2.5)))
    c["size"] = rng.uniform(1.0, 1.6)
    c["dim"] = 8 * int(_log(rng, 16, 64) + 0.5)
    c["mu"] = max(0.02, 5.0 * c["size"] / c["dim"])
    if kind in ("track", "frame"):
        c["reduce"] = rng.choice(sorted(REDUCE))
    if kind in ("fuse", "frame"):
        c["tsdf"] = rng.choice(sorted(STORAGE))
    if kind == "view":
        c["vertex"] = rng.random() < 0.5
    return c


# ---- inputs -------------------------------------------------------------------------------------------------------


def _frames(seed, w, h, f, cx, cy, n, colour=False, step=0.5):
    sc = V.synth_config(w, h, fx=f, fy=f, cx=cx, cy=cy, n_frames=n, seed=seed, dropout_blob=0.015, max_depth=2.5,
                        orbit_step_deg=step)
    if colour:
        return V.synth_generate_rgb(sc)
    depth, T, centre = V.synth_generate(sc)
    return depth, None, T, centre


def _centre_of(c):
    return 0.5 * c["w"] - 0.5, 0.5 * c["h"] - 0.5


def _config(w, h, f, cx, cy, centre, dim, size, mu, reduce="two_sum", tsdf="int16", colour=0):
    origin, vox = V.cube_around(centre, size, dim)
    return V.default_config(w, h, fx=f, fy=f, cx=cx, cy=cy, dim=(dim,) * 3, origin=origin, voxel_size=vox, mu=mu,
                            max_w=MAX_W, th_icp=0.1 ** 2, cos_normal=COS20, icp_iters=(10, 5, 4),
                            reduce_mode=REDUCE[reduce], tsdf_type=STORAGE[tsdf], color=colour)


class _Buffer:
    """a device buffer of a session, as torch takes it without a copy; the tensor holds this object, and with it the
    session whose memory it is"""

    def __init__(self, session, ptr, shape):
        self.session = session
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False), version=2, strides=None)


def _filtered(session):
    """the filtered depth of every level, in the session's own buffers"""
    return [torch.as_tensor(_Buffer(session, session.device_buffer(1 + k), (lv[1], lv[0])), device="cuda")
            for k, lv in enumerate(session.levels)]


def _poses(T_gc):
    """device copies of global-to-camera poses and their inverses, with the camera centres"""
    out = []
    for T in np.asarray(T_gc, np.float64):
        inv = np.linalg.inv(T)
        out.append((torch.from_numpy(T.astype(np.float32)).cuda(), torch.from_numpy(inv.astype(np.float32)).cuda(),
                    inv[:3, 3].astype(np.float32)))
    return out


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.int16, pin_memory=True)
    v = t.numpy().view(np.uint16)
    v[...] = a
    return t, v


class _Walk:
    """0, 1, .., n - 1, n - 2, .., 1, 0, 1, ..: consecutive frames, back and forth"""

    def __init__(self, n):
        self.order = list(range(n)) + list(range(n - 2, 0, -1))
        self.at = 0

    def next(self):
        k = self.order[self.at % len(self.order)]
        self.at += 1
        return k


def _mix(case, seed):
    """the sessions of a batch or a server: frame sizes in turn, volumes from the case's own draw"""
    r = random.Random(case["mix"])
    for i in range(case["sessions"]):
        w, h, f, cx, cy = MIX_SIZES[i % 3]
        dim = r.choice(MIX_VOLUMES)
        depth, _, _, centre = _frames(1000 * (seed % 1000003) + i, w, h, f, cx, cy, 5)
        yield depth, _config(w, h, f, cx, cy, centre, dim, 1.5, max(0.02, 5.0 * 1.5 / dim))


def _maps(w, h, vertex=True, colour=False):
    m = dict(depth=torch.zeros(h, w, device="cuda"), normal=torch.zeros(h, w, 3, device="cuda"),
             image=torch.zeros(h, w, dtype=torch.uint8, device="cuda"))
    if vertex:
        m["vertex"] = torch.zeros(h, w, 3, device="cuda")
    if colour:
        m["rgb"] = torch.zeros(3, h, w, dtype=torch.uint8, device="cuda")
    return m


LIGHT = (0.0, 0.0, -1.0)


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "filter":
        g = torch.Generator().manual_seed(seed)
        y, x = torch.meshgrid(torch.arange(c["h"]), torch.arange(c["w"]), indexing="ij")
        ph = torch.rand(4, generator=g) * 6.28
        d = (1.1 + 0.3 * torch.sin(x * 0.013 + ph[0]) * torch.cos(y * 0.017 + ph[1]) +
             0.25 * (torch.sin(x * 0.05 + ph[2]) * torch.sin(y * 0.04 + ph[3]) > 0.4))
        d = d + 0.002 * torch.randn(d.shape, generator=g)
        d[torch.rand(((c["h"] + 7) // 8, (c["w"] + 7) // 8), generator=g).repeat_interleave(8, 0).repeat_interleave(
            8, 1)[:c["h"], :c["w"]] < 0.015] = 0.0
        s = V.Session(V.default_config(c["w"], c["h"], dim=(64, 64, 64)))
        return dict(kind=kind, session=s, depth=d.float().numpy(), out=torch.zeros(c["h"], c["w"], device="cuda"))
    if kind == "serve":
        server, ids, frames = V.Server(), [], []
        for depth, cfg in _mix(c, seed):
            ids.append(server.open(cfg))
            frames.append(depth)
        st = dict(kind=kind, server=server, ids=ids, frames=frames, walk=_Walk(5))
        for _ in range(3):
            run(st)
        return st
    if kind == "batch":
        sessions, frames, keep = [], [], []
        for depth, cfg in _mix(c, seed):
            sessions.append(V.Session(cfg))
            if c["pinned"]:
                t, depth = _pinned(depth)
                keep.append(t)
            frames.append(depth)
        st = dict(kind=kind, sessions=sessions, frames=frames, keep=keep, batch=V.Batch(), walk=_Walk(5))
        for _ in range(3):
            run(st)
        return st
    cx, cy = _centre_of(c)
    colour = kind in ("colour", "view")
    posed = kind in ("fuse", "own", "view", "colour")
    depth, rgb, T, centre = _frames(seed, c["w"], c["h"], c["f"], cx, cy, 5, colour, 4.0 if posed else 0.5)
    if kind == "register":
        a = math.radians(2.0)
        K = np.array([c["f"], c["f"], cx, cy], np.float32)
        fr = c["f"] * c["wr"] / c["w"]
        Kr = np.array([fr, fr, 0.5 * c["wr"] - 0.5, 0.5 * c["hr"] - 0.5], np.float32)
        M = np.array([[math.cos(a), 0, math.sin(a), 0.025], [0, 1, 0, -0.002], [-math.sin(a), 0, math.cos(a), 0.004],
                      [0, 0, 0, 1]], np.float32)
        dev = torch.from_numpy(depth.view(np.int16)).cuda()
        return dict(kind=kind, case=c, depth=dev, K=K, Kr=Kr, M=M, walk=_Walk(5),
                    out=torch.zeros(c["hr"], c["wr"], dtype=torch.int16, device="cuda"))
    cfg = _config(c["w"], c["h"], c["f"], cx, cy, centre, c["dim"], c["size"], c["mu"],
                  c.get("reduce", "two_sum"), c.get("tsdf", "int16"), 1 if colour else 0)
    st = dict(kind=kind, walk=_Walk(5))
    if posed:
        st["depth"] = torch.from_numpy(depth.astype(np.float32) * np.float32(0.001)).cuda()
        st["poses"] = _poses(T)
    if kind == "own":
        st["volume"] = torch.full((c["dim"] ** 3,), 0x7FFF, dtype=torch.int32, device="cuda")
        st["args"] = (np.array(list(cfg.dim), np.int32), np.array(list(cfg.origin), np.float32),
                      np.array([cfg.fx, cfg.fy, cfg.cx, cfg.cy], np.float32))
        st["cfg"] = cfg
        for _ in range(5):
            run(st)
        return st
    s = st["session"] = V.Session(cfg)
    if kind in ("fuse", "colour"):
        st["maps"] = _maps(c["w"], c["h"], kind == "fuse", colour)
        st["rgb"] = torch.from_numpy(rgb).cuda() if colour else None
        torch.cuda.synchronize()
        for _ in range(5):
            run(st)
    elif kind == "view":
        st["maps"] = _maps(c["w"], c["h"], c["vertex"], True)
        dev = torch.from_numpy(rgb).cuda()
        for k in range(5):
            Tgc, Tcg, _ = st["poses"][k]
            s.cdtocc_convert_depth_to_tsdf_color(st["depth"][k].data_ptr(), dev[k].data_ptr(), Tgc.data_ptr(),
                                                 Tcg.data_ptr())
    elif kind == "track":
        for k in range(4):
            s.scan_frame_host(depth[k])
        st["depth"] = torch.from_numpy(depth[4].view(np.int16)).cuda()
        s.stage_filter(st["depth"].data_ptr())
    else:
        st["frames"], st["filtered"] = depth, _filtered(s)
        for _ in range(3):
            run(st)
    return st


def run(state):
    st = state
    kind = st["kind"]
    if kind == "filter":
        st["session"].bfd_bilateral_filter_depth(st["out"].data_ptr(), st["depth"])
        return st["out"]
    k = st["walk"].next() if "walk" in st else 0
    if kind == "serve":
        server, got = st["server"], {}
        for i, sid in enumerate(st["ids"]):
            server.submit(sid, st["frames"][i][k])
        while len(got) < len(st["ids"]):
            for r in server.poll(timeout_ms=1000):
                got[r["session"]] = r
        return dict(T_gc=np.stack([got[i]["T_gc"] for i in st["ids"]]),
                    tracked=np.array([got[i]["tracked"] for i in st["ids"]], np.int32))
    if kind == "batch":
        T, tracked = st["batch"].step_host(st["sessions"], [f[k] for f in st["frames"]])
        return dict(T_gc=T, tracked=tracked.astype(np.int32))
    if kind == "register":
        c = st["case"]
        V.warp_depth_to_color(st["depth"][k].data_ptr(), c["w"], c["h"], st["K"], st["M"], st["Kr"], c["wr"], c["hr"],
                              st["out"].data_ptr(), mm_scale=0.001)
        return st["out"]
    if kind == "own":
        cfg, (dim, origin, K) = st["cfg"], st["args"]
        Tgc, Tcg, _ = st["poses"][k]

        def p(a):
            return a.ctypes.data_as(ctypes.c_void_p)

        lib = V.load()
        rc = lib.vs_integrate_depth_noalloc(ctypes.c_void_p(st["volume"].data_ptr()), p(dim), p(origin), cfg.voxel_size,
                                            cfg.mu, cfg.max_w, ctypes.c_void_p(st["depth"][k].data_ptr()), cfg.width,
                                            cfg.height, p(K), ctypes.c_void_p(Tgc.data_ptr()),
                                            ctypes.c_void_p(Tcg.data_ptr()), None)
        if rc:
            raise V.VsError(rc, lib.vs_last_error().decode())
        return st["volume"]
    s = st["session"]
    if kind == "track":
        tracked = s.tp_track_pose()
        return dict(T_gc=s.pose()[0], tracked=tracked)
    if kind == "fuse":
        Tgc, Tcg, cen = st["poses"][k]
        m = st["maps"]
        s.cdtoc_convert_depth_to_tsdf(st["depth"][k].data_ptr(), Tgc.data_ptr(), Tcg.data_ptr())
        s.rmi_render_maps_for_icp(0, Tgc.data_ptr(), Tcg.data_ptr(), cen, LIGHT, m["depth"].data_ptr(),
                                  m["vertex"].data_ptr(), m["normal"].data_ptr(), m["image"].data_ptr())
        return m
    if kind == "view":
        Tgc, Tcg, cen = st["poses"][k]
        m = st["maps"]
        s.rmis_render_maps_for_scene(Tgc.data_ptr(), Tcg.data_ptr(), cen, LIGHT, m["depth"].data_ptr(),
                                     m["vertex"].data_ptr() if "vertex" in m else None, m["normal"].data_ptr(),
                                     m["image"].data_ptr(), m["rgb"].data_ptr())
        return m
    if kind == "colour":
        Tgc, Tcg, cen = st["poses"][k]
        m = st["maps"]
        s.cdtocc_convert_depth_to_tsdf_color(st["depth"][k].data_ptr(), st["rgb"][k].data_ptr(), Tgc.data_ptr(),
                                             Tcg.data_ptr())
        s.rmi_render_view(0, Tgc.data_ptr(), Tcg.data_ptr(), cen, LIGHT, m["depth"].data_ptr(), m["normal"].data_ptr(),
                          m["image"].data_ptr(), m["rgb"].data_ptr())
        return m
    T, tracked = s.scan_frame_host(st["frames"][k])
    return dict(T_gc=T, tracked=tracked, filtered=st["filtered"])


# ---- work and exact values ------------------------------------------------------------------------------------------


def _frame_work(w, h, f, dim, size, mu, word=4, colour=False):
    """one frame: {stage: (bytes, flops)}"""
    px = w * h
    pyr = px * 1.3125
    # filter: uint16 in; metres, filtered pyramid, vertex and normal maps out
    filt = px * (2 + 4 + 3 * colour) + pyr * (4 + 24), px * 25 * 8 + pyr * 60
    # tracking: depth (and normal) and the model's vertex and normal of each pixel, once per iteration
    per = sum(n * px / 4 ** level for level, n in enumerate((10, 5, 4)))
    track = per * (28 + 12), per * 150
    # the voxels of the 8^3 sub-cubes from 4 mu before to 1 mu behind the seen surface, which covers about 3/4 of a
    # cross-section of the cube, or what the camera sees of it from 1 m
    vox = size / dim
    area = min(0.75 * size * size, (w / f) * (h / f))
    voxels = area * (5 * mu + 8 * vox) / vox ** 3
    fuse = voxels * 2 * (word + 4 * colour) + px * 4, voxels * 60
    # ray-cast: the voxels around the surface once; depth, vertex, normal, shading (and colour) out
    cast = pyr * (29 + 3 * colour) + area / vox ** 2 * 4 * word, pyr * 400
    return dict(filter=filt, track=track, fuse=fuse, cast=cast)


def work(case):
    c = case
    kind = c["kind"]

    def total(parts):
        return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}

    if kind == "filter":
        return {"bytes": c["w"] * c["h"] * 8.0, "flops": c["w"] * c["h"] * 25 * 8.0}
    if kind == "register":
        return {"bytes": (c["w"] * c["h"] + c["wr"] * c["hr"]) * 2.0, "flops": c["w"] * c["h"] * 40.0}
    if kind in ("serve", "batch"):
        r = random.Random(c["mix"])
        parts = []
        for i in range(c["sessions"]):
            w, h, f = MIX_SIZES[i % 3][:3]
            dim = r.choice(MIX_VOLUMES)
            parts += _frame_work(w, h, f, dim, 1.5, max(0.02, 5.0 * 1.5 / dim)).values()
        return total(parts)
    p = _frame_work(c["w"], c["h"], c["f"], c["dim"], c["size"], c["mu"],
                    8 if c.get("tsdf") == "fp32" else 4, kind in ("colour", "view"))
    if kind == "track":
        return total([p["track"]])
    if kind == "own":
        return total([p["fuse"]])
    if kind == "view":
        return total([p["cast"]])
    if kind in ("fuse", "colour"):
        return total([p["fuse"], p["cast"]])
    return total(p.values())


def _bilateral64(d):
    """the filter's definition: taps are means of 2x2 pixels (borders repeat), 5x5 Gaussian of 4 pixels and 0.1 m;
    0 where a tap is not above 0"""
    h, w = d.shape
    y = np.clip(np.arange(-3, h + 2), 0, h - 1)
    x = np.clip(np.arange(-3, w + 2), 0, w - 1)
    t = d[np.ix_(y, x)]
    t = 0.25 * (t[:-1, :-1] + t[:-1, 1:] + t[1:, :-1] + t[1:, 1:])
    mid = t[2:2 + h, 2:2 + w]
    num, den, ok = np.zeros((h, w)), np.zeros((h, w)), np.ones((h, w), bool)
    for i in range(5):
        for j in range(5):
            tap = t[i:i + h, j:j + w]
            f = math.exp(-((i - 2) ** 2 + (j - 2) ** 2) / 32.0) * np.exp(-((mid - tap) ** 2) / 0.02)
            num += f * tap
            den += f
            ok &= tap > 0
    return np.where(ok, num / den, 0.0)


def _half64(d):
    """5x5 binomial smoothing (0 within two pixels of the border), every second pixel from 1 kept"""
    k = np.array([1.0, 4.0, 6.0, 4.0, 1.0]) / 16.0
    h, w = d.shape
    s = np.zeros((h, w))
    rows = sum(k[i] * d[i:h - 4 + i, :] for i in range(5))
    s[2:h - 2, 2:w - 2] = sum(k[i] * rows[:, i:w - 4 + i] for i in range(5))
    return s[1::2, 1::2][:h // 2, :w // 2]


def exact(case, seed):
    c = case
    if c["kind"] == "filter":
        return _bilateral64(prepare(c, seed)["depth"].astype(np.float64))
    if c["kind"] != "frame":
        return None
    cx, cy = _centre_of(c)
    depth = _frames(seed, c["w"], c["h"], c["f"], cx, cy, 5)[0]
    # prepare() passes three frames; the first pass after it sees the fourth
    levels = [_bilateral64(depth[3] * 0.001)]
    for _ in range(2):
        levels.append(_half64(levels[-1]))
    return dict(T_gc=None, tracked=None, filtered=levels)


_KINDS = ("frame", "colour", "serve", "batch", "track", "fuse", "own", "view", "filter", "register")
