"""What the framework's users have it do, as cases that can be timed and compared.

Every case goes through the public binding (``pyopenlpt_b200._ffi``) on seeded synthetic
recordings: particles in a box, seen by a ring of pinhole cameras or by cubic polynomial
cameras, rendered as Gaussian spots with noise into integer (or float) images.

Kinds of work
  detect        2D detection on the images of every camera, lists back on the host
  detect_device 2D detection of one image into the caller's device buffers
  stereo        detection and stereo matching of one frame, matched ids and positions
  shake         refinement of given 3D objects against the images (FP32 or FP64 arithmetic)
  ipr           a whole iterative particle reconstruction of one frame
  ipr_batch     independent frames at once, one context each
  stb           a whole short Shake-the-Box sequence, initial and convergence phase
  mlp_forward   the learned proposal's network on a batch of candidates
  mlp_grad      its loss and gradients on a training batch
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from pyopenlpt_b200 import _ffi, synth

DTYPES = {"u8": np.uint8, "u16": np.uint16, "f32": np.float32, "f64": np.float64}
OTF_POLY = (5, 5, 5)  # grid of the spatially varying OTF of the polynomial rigs


def listed():
    frame = dict(camera="pinhole", dtype="u8", focal=0.0, shake_px=0.25, loops=4)
    poly = dict(frame, camera="poly", dtype="u16")
    return [
        # the smallest call in use: the spots of one small 8-bit frame of a live preview
        dict(frame, name="detect_512_u8", kind="detect", n_cam=4, rows=512, cols=512,
             particles=2000),
        # a plug-in host with its own device buffers, one dense 4-megapixel 12-bit image
        dict(frame, name="detect_device_2048_u16", kind="detect_device", dtype="u16", n_cam=1,
             rows=2048, cols=2048, particles=400000),
        # matching of an ordinary 8-bit frame of four pinhole cameras
        dict(frame, name="stereo_1024_u8_4cam_10k", kind="stereo", n_cam=4, rows=1024, cols=1024,
             particles=10000, focal=5000.0),
        # matching at the highest density: six polynomial cameras, 0.1 particles per pixel
        dict(poly, name="stereo_2048_u16_6cam_419k", kind="stereo", n_cam=6, rows=2048, cols=2048,
             particles=419430),
        # predicted particles of a small recording refined in FP64 (the parity arithmetic)
        dict(frame, name="shake_512_u8_fp64", kind="shake", n_cam=4, rows=512, cols=512,
             particles=2500, objects=2000, precision=1),
        # predicted particles of a dense polynomial rig refined in FP32 (the production path)
        dict(poly, name="shake_2048_u16_6cam_120k", kind="shake", n_cam=6, rows=2048, cols=2048,
             particles=419430, objects=120000, precision=0),
        # one frame of the 10,000-particle benchmark, whole
        dict(frame, name="ipr_1024_u8_4cam_10k", kind="ipr", n_cam=4, rows=1024, cols=1024,
             particles=10000, focal=5000.0, shake_px=2.5, precision=0),
        # one frame of the densest recording, whole: 0.1 particles per pixel, six cameras
        dict(poly, name="ipr_2048_u16_6cam_419k", kind="ipr", n_cam=6, rows=2048, cols=2048,
             particles=419430, precision=0),
        # small frames of independent experiments, eight at once
        dict(frame, name="ipr_batch8_512_u8", kind="ipr_batch", frames=8, n_cam=4, rows=512,
             cols=512, particles=2000, precision=0),
        # a tracked sequence of 51,000 particles on 1280 x 800, from its first frame on
        dict(frame, name="stb_1280x800_u16_51k", kind="stb", dtype="u16", n_cam=4, rows=800,
             cols=1280, particles=51000, focal=5000.0, frames=6, precision=0),
        # the learned proposal on the candidates of a dense frame of six cameras
        dict(name="mlp_forward_6cam_100k", kind="mlp_forward", n_cam=6, rows=100000),
        # one training batch of the four-camera network
        dict(name="mlp_grad_4cam_8192", kind="mlp_grad", n_cam=4, rows=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["detect", "detect_device", "stereo", "stereo", "shake", "shake", "ipr",
                       "ipr_batch", "stb", "mlp_forward", "mlp_grad"])
    if kind.startswith("mlp"):
        hi = 100000 if kind == "mlp_forward" else 16384
        return dict(kind=kind, n_cam=rng.randint(2, 8), rows=_log_int(rng, 64, hi))
    poly = kind in ("stereo", "shake", "ipr") and rng.random() < 0.5
    side = _log_int(rng, 256, 2048 if kind in ("detect", "detect_device") else 1100)
    rows = side
    cols = side if poly else max(256, int(side * rng.uniform(0.7, 1.6)))
    case = dict(kind=kind, camera="poly" if poly else "pinhole",
                dtype="u16" if poly or rng.random() < 0.4 else "u8", focal=0.0, shake_px=0.25,
                loops=4, n_cam=rng.randint(3, 6), rows=rows, cols=cols)
    ppp = math.exp(rng.uniform(math.log(0.005), math.log(0.05)))
    case["particles"] = max(200, int(ppp * rows * cols))
    if kind in ("detect", "detect_device"):
        case["dtype"] = rng.choice(["u8", "u16", "f32", "f64"])
    if kind == "detect_device":
        case["n_cam"] = 1
    if kind in ("shake", "ipr", "ipr_batch", "stb"):
        case["precision"] = 1 if kind == "shake" and rng.random() < 0.3 else 0
    if kind == "shake":
        case["objects"] = max(100, int(case["particles"] * rng.uniform(0.3, 1.0)))
        case["shake_px"] = rng.choice([0.25, 1.0])
    if kind == "ipr":
        case["loops"] = rng.randint(2, 4)
    if kind == "ipr_batch":
        case.update(frames=rng.randint(2, 8), rows=min(rows, 640), cols=min(cols, 640))
        case["particles"] = max(200, int(ppp * case["rows"] * case["cols"]))
    if kind == "stb":
        case.update(frames=rng.randint(5, 7), rows=min(rows, 800), cols=min(cols, 1280))
        case["particles"] = max(200, int(ppp * case["rows"] * case["cols"]))
    return case


# ------------------------------------------------------------------ recordings
def _volume(case):
    if case["camera"] == "poly":  # the box grows with the images, so a pixel stays 0.04 mm
        h = 40.0 * case["rows"] / 2048.0
        return (-h, h, -h, h, -0.5 * h, 0.5 * h)
    if case["focal"] and case["kind"] == "stb":
        return (-30.0, 30.0, -20.0, 20.0, -15.0, 15.0)
    return (-20.0, 20.0, -20.0, 20.0, -10.0, 10.0)


class Recording:
    """Cameras, OTF, particle paths, images and the settings that fit the rig."""

    def __init__(self, case, seed, n_frames=1):
        rng = np.random.default_rng([seed, 77])
        self.volume = v = _volume(case)
        n_cam, rows, cols = case["n_cam"], case["rows"], case["cols"]
        dtype = DTYPES[case["dtype"]]
        bright = case["dtype"] != "u8"  # 12-bit levels
        if case["camera"] == "poly":
            self.cams = synth.poly_rig(n_cam, rows, v, seed=seed % 100003)
            self.otf_n = OTF_POLY
            self.otf = synth.otf_grid(n_cam, OTF_POLY, seed=seed % 100003 + 1)
        else:
            focal = case["focal"] or min(synth.focal_for_volume(max(n_cam, 2), min(rows, cols), v))
            self.cams = synth.ring_rig(n_cam, rows, cols, focal)
            self.otf_n = (2, 2, 2)
            self.otf = synth.otf_table_array(n_cam, (3000.0 if bright else 200.0, 0.5, 0.5))
        lo, hi = np.array(v[0::2]), np.array(v[1::2])
        c0 = 0.5 * (lo + hi)
        mm_px = 1.0 / max(synth.px_per_mm(cm, c0) for cm in self.cams)
        xyz = lo + (hi - lo) * rng.random((case["particles"], 3))
        self.frames = []
        self.truth = []
        for _ in range(n_frames):
            self.truth.append(xyz)
            noise = rng.standard_normal((n_cam, rows, cols), dtype=np.float32)
            noise *= 20.0 if bright else 2.0
            levels = 4095 if bright else 255
            im = synth.render_frame(self.cams, xyz, self.otf, self.otf_n, v, noise, levels,
                                    dtype if np.dtype(dtype).kind == "u" else np.uint16, "cuda")
            if np.dtype(dtype).kind == "f":  # the fractions that residual images have
                im = im.astype(dtype) + rng.random(im.shape, dtype=np.float32).astype(dtype)
            self.frames.append(np.ascontiguousarray(im))
            # unit-speed Taylor-Green cells, at most 3 px of motion a frame
            xyz = synth.rk4(lambda p: synth.taylor_green_velocity(p, 40.0), xyz, 3.0 * mm_px)
            out = np.any((xyz < lo) | (xyz > hi), axis=1)
            xyz[out] = lo + (hi - lo) * rng.random((int(out.sum()), 3))
        self.threshold = 300.0 if bright else 30.0
        self.mm_px = mm_px
        self.settings = synth.IPRSettings(
            min_obj_int=self.threshold, shake_width=case["shake_px"] * mm_px,
            tol_3d_mm=0.6 * mm_px, match_cam_count=n_cam, n_loop_ipr=case["loops"],
            n_obj2d_process_max=1_000_000)
        self.stb = synth.STBSettings(radius_search_obj=10.0 * mm_px,
                                     radius_search_track=10.0 * mm_px, pf_r=30.0 * mm_px)

    def start_objects(self, n, seed):
        """Predictions: particles displaced by 0.3 px, one in ten a ghost."""
        rng = np.random.default_rng([seed, 78])
        t = self.truth[0]
        x = t[rng.permutation(len(t))[:n]] + rng.normal(0.0, 0.3 * self.mm_px, (n, 3))
        lo, hi = np.array(self.volume[0::2]), np.array(self.volume[1::2])
        ghost = rng.random(n) < 0.1
        x[ghost] = lo + (hi - lo) * rng.random((int(ghost.sum()), 3))
        return x


class Bound:
    """A context with the rig loaded, and a recording's frames in device memory."""

    def __init__(self, rec):
        self.ctx = _ffi.Context(torch.cuda.current_device())
        self.ctx.upload_cameras([_ffi.camera_desc(c) for c in rec.cams])
        self.ctx.upload_otf(*rec.otf_n, rec.volume, rec.otf)
        self.dtype = _ffi._DTYPES[rec.frames[0].dtype]
        self.shape = rec.frames[0].shape[1:]
        as_int = {np.dtype(np.uint16): np.int16}.get(rec.frames[0].dtype, rec.frames[0].dtype)
        self.frames = [torch.from_numpy(f.view(as_int)).cuda() for f in rec.frames]

    def load(self, t=0):
        f = self.frames[t]
        self.ctx.upload_images_device([f[c].data_ptr() for c in range(len(f))], self.dtype,
                                      [self.shape[0]] * len(f), [self.shape[1]] * len(f))


def _weights(n_in, seed):
    """Flat f32 parameters W1, b1, W2, b2, W3, b3, W4, b4 at He scale."""
    rng = np.random.default_rng([seed, 79])
    parts = []
    for fan_out, fan_in, gain in ((256, n_in, 6.0), (256, 256, 6.0), (256, 256, 6.0),
                                  (4, 256, 1.0)):
        lim = math.sqrt(gain / fan_in)
        parts += [rng.uniform(-lim, lim, fan_out * fan_in), rng.uniform(-0.1, 0.1, fan_out)]
    return np.concatenate(parts).astype(np.float32)


def _batch(case, seed, device):
    """Candidates: normalised patches (mostly dark, one spot's worth of light), sub-pixel
    offsets, a constant 1; targets in units of the output scale and a ghost label."""
    n, c = case["rows"], case["n_cam"]
    g = torch.Generator(device="cpu").manual_seed(seed % (1 << 40) + 5)
    patch = torch.randn((n, 121 * c), generator=g).mul_(0.25).add_(0.1).clamp_(0.0, 1.5)
    off = torch.rand((n, 2 * c), generator=g) - 0.5
    x = torch.cat([patch, off, torch.ones((n, 1))], dim=1)
    t = torch.randn((n, 4), generator=g)
    t[:, 3] = (torch.rand(n, generator=g) < 0.3).float()
    return x.to(device), t.to(device)


class Lists:
    """The caller's result arrays: room for `cap` rows each, rows past the count are 0."""

    def __init__(self, cap, **columns):
        self.cap = cap
        self.n = 0
        self.columns = {k: np.zeros((cap, *shape), dtype) for k, (shape, dtype) in columns.items()}

    def fill(self, n, call, *names):
        """call(pointers) writes n rows; the count and the arrays."""
        if n > self.cap:
            raise RuntimeError(f"{n} rows, room for {self.cap}")
        check = call(*(self.columns[k].ctypes.data_as(ctypes.c_void_p) for k in names))
        if check:
            raise _ffi.OlptError(check, "reading results")
        if n < self.n:
            for v in self.columns.values():
                v[n:self.n] = 0
        self.n = n
        return (n, *self.columns.values())


# ------------------------------------------------------------------ preparation
def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("mlp"):
        ctx = _ffi.Context(torch.cuda.current_device())
        n_in = 121 * case["n_cam"] + 2 * case["n_cam"] + 1
        # the network's size follows the rig: any cameras of that count will do
        ctx.upload_cameras([_ffi.camera_desc(c) for c in
                            synth.ring_rig(case["n_cam"], 64, 64, 300.0)])
        ctx.mlp_set_params(_weights(n_in, seed))
        x, t = _batch(case, seed, "cuda")
        out = torch.empty((case["rows"], 4), device="cuda")
        torch.cuda.synchronize()
        return dict(case=case, ctx=ctx, x=x, t=t, out=out, n_params=ctx.mlp_dims()[1])
    if kind == "ipr_batch":
        recs = [Recording(case, seed + 1000 * i) for i in range(case["frames"])]
        bound = [Bound(r) for r in recs]
        torch.cuda.synchronize()
        r = recs[0]
        objects = [Lists(2 * case["particles"] + 1000, xyz=((3,), np.float64),
                         uv=((case["n_cam"], 2), np.float64)) for _ in bound]
        return dict(case=case, bound=bound, objects=objects,
                    params=_ffi.ipr_params(r.settings, r.volume, case["precision"]))
    rec = Recording(case, seed, case["frames"] if kind == "stb" else 1)
    state = dict(case=case, threshold=rec.threshold)
    if kind == "detect_device":
        im = rec.frames[0][0]
        esz = im.dtype.itemsize
        pitch = (im.shape[1] * esz + 15) // 16 * 16
        host = np.zeros((im.shape[0], pitch), np.uint8)
        host[:, :im.shape[1] * esz] = im.view(np.uint8).reshape(im.shape[0], -1)
        cap = (im.size + 1) // 2
        state.update(image=torch.from_numpy(host).cuda(), pitch=pitch, cap=cap,
                     dtype=_ffi._DTYPES[im.dtype], lib=_ffi.lib(),
                     x=torch.zeros(cap, dtype=torch.float64, device="cuda"),
                     y=torch.zeros(cap, dtype=torch.float64, device="cuda"),
                     rc=torch.zeros((cap, 2), dtype=torch.int32, device="cuda"),
                     count=torch.zeros(1, dtype=torch.int64, device="cuda"))
        torch.cuda.synchronize()
        return state
    state["bound"] = Bound(rec)
    s, v = rec.settings, rec.volume
    p, n_cam = case["particles"], case["n_cam"]
    if kind == "detect":
        state["spots"] = [Lists(p + p // 4 + 1000, xy=((2,), np.float64), rc=((2,), np.int32))
                          for _ in range(n_cam)]
    elif kind == "stereo":
        state["matches"] = Lists(p + p // 4 + 1000, ids=((n_cam,), np.int32),
                                 xyz=((3,), np.float64))
        state["params"] = _ffi.sm_params(s, v)
    elif kind == "shake":
        state["params"] = _ffi.shake_params(s, case["precision"])
        state["start"] = rec.start_objects(case["objects"], seed)
    elif kind == "ipr":
        state["objects"] = [Lists(2 * p + 1000, xyz=((3,), np.float64),
                                  uv=((n_cam, 2), np.float64))]
        state["params"] = _ffi.ipr_params(s, v, case["precision"])
    elif kind == "stb":
        state["tracks"] = [Lists((case["frames"] + 1) * p + 1000, track=((), np.int32),
                                 frame=((), np.int32), xyz=((3,), np.float64)) for _ in range(4)]
        state["params"] = _ffi.stb_params(s, rec.stb, v, 1, case["frames"], case["precision"])
    torch.cuda.synchronize()
    if kind in ("detect", "stereo", "shake"):
        state["bound"].load()  # these leave the images as they are
    return state


# ------------------------------------------------------------------ one pass
def _objects(ctx, n, into):
    return into.fill(n, lambda xyz, uv: ctx.L.olpt_ipr_result(ctx.h, xyz, uv), "xyz", "uv")


def _tracks(ctx, which, into):
    tracks, rows = ctypes.c_int64(), ctypes.c_int64()
    rc = ctx.L.olpt_stb_track_rows(ctx.h, which, ctypes.byref(tracks), ctypes.byref(rows))
    if rc:
        raise _ffi.OlptError(rc, "olpt_stb_track_rows")
    return into.fill(rows.value, lambda tid, frame, xyz: ctx.L.olpt_stb_get_tracks(
        ctx.h, which, tid, frame, xyz, ctypes.c_int64(into.cap)), "track", "frame", "xyz")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mlp_forward":
        state["ctx"].mlp_forward_device(state["x"].data_ptr(), case["rows"],
                                        state["out"].data_ptr())
        return state["out"]
    if kind == "mlp_grad":
        ctx = state["ctx"]
        loss = ctypes.c_double()
        grad = np.empty(state["n_params"], np.float32)
        rc = ctx.L.olpt_mlp_train_step(
            ctx.h, ctypes.c_int64(case["rows"]), ctypes.c_void_p(state["x"].data_ptr()),
            ctypes.c_void_p(state["t"].data_ptr()), 1, ctypes.c_double(1e-3),
            ctypes.c_double(1.0), 0, ctypes.byref(loss),
            grad.ctypes.data_as(ctypes.c_void_p))
        if rc:
            raise _ffi.OlptError(rc, "olpt_mlp_train_step")
        return loss.value, grad
    if kind == "detect_device":
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        rc = state["lib"].olpt_find_peaks_noalloc(
            ptr(state["image"]), state["dtype"], case["rows"], case["cols"],
            ctypes.c_int64(state["pitch"]), ctypes.c_double(state["threshold"]),
            ptr(state["x"]), ptr(state["y"]), ptr(state["rc"]), ctypes.c_int64(state["cap"]),
            ptr(state["count"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise _ffi.OlptError(rc, "olpt_find_peaks_noalloc")
        # entries past the count stay 0, as the caller left them
        return state["count"], state["x"], state["y"], state["rc"]
    if kind == "ipr_batch":
        for b in state["bound"]:
            b.load()
        n = _ffi.ipr_run_batch([b.ctx for b in state["bound"]], state["params"])
        return [_objects(b.ctx, int(k), o)
                for b, k, o in zip(state["bound"], n, state["objects"])]
    bound = state["bound"]
    ctx = bound.ctx
    if kind == "detect":
        n = ctx.find_peaks(state["threshold"])
        return [spots.fill(int(n[c]), lambda xy, rc: ctx.L.olpt_get_peaks(
            ctx.h, c, xy, rc, ctypes.c_int64(spots.cap)), "xy", "rc")
            for c, spots in enumerate(state["spots"])]
    if kind == "stereo":
        ctx.find_peaks(state["threshold"])
        n_cand, n = ctx.stereo_match(state["params"])
        return (n_cand, *state["matches"].fill(
            n, lambda ids, xyz: ctx.L.olpt_get_matches(ctx.h, ids, xyz), "ids", "xyz"))
    if kind == "shake":
        ctx.upload_objects(state["start"])
        ctx.shake(state["params"])
        o = ctx.objects()
        return o["xyz"], o["uv"], o["flags"], o["score"]
    if kind == "ipr":
        bound.load()
        return _objects(ctx, ctx.ipr_run(state["params"]), state["objects"][0])
    ctx.stb_configure(state["params"])
    for t in range(case["frames"]):
        bound.load(t)
        ctx.stb_process_frame(t + 1)
    return [_tracks(ctx, w, state["tracks"][w]) for w in range(4)]


# ------------------------------------------------------------------ the work itself
def work(case):
    kind, n_cam = case["kind"], case["n_cam"]
    if kind.startswith("mlp"):
        n, n_in = case["rows"], 123 * n_cam + 1
        params = 256 * (n_in + 1) + 2 * 256 * 257 + 4 * 257
        macs = n * (256 * n_in + 2 * 256 * 256 + 4 * 256)
        if kind == "mlp_forward":
            return {"bytes": 4.0 * (n * n_in + params + 4 * n), "flops": 2.0 * macs}
        # the gradient of the inputs is not needed
        return {"bytes": 4.0 * (n * n_in + 2 * params + 4 * n),
                "flops": 2.0 * (3 * macs - n * 256 * n_in)}
    px = case["rows"] * case["cols"]
    image = px * n_cam * np.dtype(DTYPES[case["dtype"]]).itemsize
    p = case["particles"]
    # a spot costs a local-maximum test per bright pixel and two three-point fits
    detect = {"bytes": image + 24.0 * p * n_cam, "flops": n_cam * (4.0 * px + 40.0 * p)}
    if kind in ("detect", "detect_device"):
        return detect
    # an object: 64 pixels a camera, about 11 residues of about 20 operations a pixel, per loop
    shake = 4.0 * n_cam * 64 * 11 * 20
    # a reference spot meets the spots within +- 1 px of its line on the next camera
    pairs = p * (p / px) * 2.0 * math.sqrt(px)
    match = pairs * 30.0 + p * n_cam * 200.0
    if kind == "stereo":
        return {"bytes": image + p * (4.0 * n_cam + 24.0), "flops": detect["flops"] + match}
    if kind == "shake":
        n = case["objects"]
        return {"bytes": image + n * (48.0 + 16.0 * n_cam + 9.0), "flops": n * shake}
    if kind in ("ipr", "ipr_batch"):
        k = case.get("frames", 1)
        return {"bytes": k * (image + p * (24.0 + 16.0 * n_cam)),
                "flops": k * (case["loops"] * (detect["flops"] + match) + p * shake)}
    f = case["frames"]
    return {"bytes": f * (image + 32.0 * p),
            "flops": f * (case["loops"] * (detect["flops"] + match) + p * shake)}


# ------------------------------------------------------------------ 64-bit values
def _peaks64(im, threshold):
    """Local maxima (strictly above right and below, not below left and above) of at least
    the threshold, raster order, with three-point log-parabola centres."""
    a = im.astype(np.float64)
    c = a[1:-1, 1:-1]
    left, right, up, down = a[1:-1, :-2], a[1:-1, 2:], a[:-2, 1:-1], a[2:, 1:-1]
    m = (c >= threshold) & (up <= c) & (left <= c) & (down < c) & (right < c)
    ln = lambda v: np.log(np.maximum(v[m], 1e-4))  # noqa: E731
    l0 = ln(c)
    r, q = np.nonzero(m)

    def centre(lo, hi, p):
        num = lo * (p * p - (p + 1) * (p + 1)) - l0 * ((p - 1) * (p - 1) - (p + 1) * (p + 1)) \
            + hi * ((p - 1) * (p - 1) - p * p)
        return -0.5 * num / (lo + hi - 2.0 * l0)

    xy = np.stack([centre(ln(left), ln(right), q + 1.0), centre(ln(up), ln(down), r + 1.0)], 1)
    return xy, np.stack([r + 1, q + 1], 1).astype(np.int32)


def _mlp64(case, seed, grad):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n_in = 123 * case["n_cam"] + 1
    flat = torch.from_numpy(_weights(n_in, seed)).to(dev, torch.float64).requires_grad_(grad)
    x, t = _batch(case, seed, dev)
    h, o = x.double(), 0
    for i, (fan_out, fan_in) in enumerate(((256, n_in), (256, 256), (256, 256), (4, 256))):
        w = flat[o:o + fan_out * fan_in].view(fan_out, fan_in)
        o += fan_out * fan_in
        h = h @ w.T + flat[o:o + fan_out]
        o += fan_out
        if i < 3:
            h = torch.nn.functional.gelu(h)
    if not grad:
        return h
    t = t.double()
    mse = ((h[:, :3] - t[:, :3]) ** 2).mean(1)
    bce = torch.nn.functional.binary_cross_entropy_with_logits(h[:, 3], t[:, 3], reduction="none")
    loss = ((1.0 - t[:, 3]) * mse + bce).mean()
    loss.backward()
    return float(loss), flat.grad.cpu().numpy()


def _padded(v, cap):
    return np.concatenate([v, np.zeros((cap - len(v), *v.shape[1:]), v.dtype)])


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp_forward":
        return _mlp64(case, seed, False)
    if kind == "mlp_grad":
        return _mlp64(case, seed, True)
    if kind == "detect":
        rec = Recording(case, seed)
        out = [_peaks64(im, rec.threshold) for im in rec.frames[0]]
        cap = case["particles"] + case["particles"] // 4 + 1000
        return [(len(xy), _padded(xy, cap), _padded(rc, cap)) for xy, rc in out]
    if kind == "detect_device":
        rec = Recording(case, seed)
        xy, rc = _peaks64(rec.frames[0][0], rec.threshold)
        cap = (case["rows"] * case["cols"] + 1) // 2
        return (np.array([len(xy)], np.int64), _padded(xy[:, 0], cap), _padded(xy[:, 1], cap),
                _padded(rc, cap))
    # what a search finds (matched sets, line-search positions, tracks) has no closed value
    return None
