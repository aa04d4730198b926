"""Workloads whose speed matters to a user of the detector, each through the public entry points.

A case is a dict of plain values; `kind` says which entry point it goes through:

  single   FaceDetector.Detect on one host frame, or FaceDetector.DetectDevice on one device frame
  batch    FaceDetector.DetectBatch on page-locked host frames, or ccnn_detect_device_batch on device frames
  serve    FaceServer: frames of the serving mix submitted together, every result waited for
  train    ccnn_gate_train: one pass of the gate's training over mini-batches of labelled frames

Frames are the seeded synthetic ones of the benchmark (rendered on the device). Detector settings not
in the case keep the library's defaults. The detection cascade decides by thresholds on fp32 values, so
its rectangles and scores have no 64-bit value to compare with; the gate's training does.
"""
import ctypes
import gc
import math
import os

import numpy as np
import torch

import compactcnncascade_b200 as ccnn
from compactcnncascade_b200 import _capi, autotune, gate

MODELS = os.path.join(os.path.dirname(os.path.abspath(ccnn.__file__)), "models")
LEGACY = [os.path.join(MODELS, "cnn4face%d_new.bin" % i) for i in (1, 2, 3)]
# the benchmark's serving mix: size and share of the frames
SERVE_MIX = (((640, 480), 0.3), ((1280, 720), 0.3), ((1920, 1080), 0.3), ((3840, 2160), 0.1))
CAPACITY = 1024  # faces a frame that the device-batch caller keeps room for
KEEP = 256  # faces a frame in the outputs


def _detect(kind, width, height, channels, frames, source, min_face, max_face, scale, **more):
    c = {"kind": kind, "width": width, "height": height, "channels": channels, "frames": frames, "source": source, "min_face": min_face,
         "max_face": max_face, "scale": scale, "gate": False, "facial": False, "legacy": False, "pad": 0, "slots": 0}
    c.update(more)
    return c


def listed():
    return [
        # one webcam frame from ordinary host memory, as an interactive program calls it: latency
        dict(_detect("single", 640, 480, 3, 1, "host", 40, 240, 1.15), name="vga_host_single"),
        # one full-HD frame that a decoder left in device memory: latency of the headline size
        dict(_detect("single", 1920, 1080, 3, 1, "device", 40, 240, 1.15), name="hd_device_single"),
        # full-HD frames from page-locked host memory, end to end
        dict(_detect("batch", 1920, 1080, 3, 16, "host", 40, 240, 1.15), name="hd_host_batch"),
        # the headline: full-HD frames in device memory, plain cascade, tuned schedule
        dict(_detect("batch", 1920, 1080, 3, 32, "device", 40, 240, 1.15), name="hd_device_batch"),
        # the same with the learned gate at its operating point
        dict(_detect("batch", 1920, 1080, 3, 32, "device", 40, 240, 1.15, gate=True), name="hd_gated_batch"),
        # a monochrome camera with the library's default parameters (smallest face 80: the frame is shrunk first)
        dict(_detect("batch", 1280, 720, 1, 16, "host", 80, 0, 1.1), name="camera_gray_default"),
        # BGRA frames of an odd size whose rows are not aligned, as a window capture leaves them
        dict(_detect("batch", 1277, 717, 4, 16, "device", 30, 0, 1.2), name="odd_bgra_batch"),
        # small faces in 4K frames over a fine pyramid (83 levels): the largest work a frame
        dict(_detect("batch", 3840, 2160, 3, 8, "device", 20, 0, 1.05, slots=4), name="uhd_deep_pyramid"),
        # gender, smile and glasses of every face in a 720p frame
        dict(_detect("single", 1280, 720, 3, 1, "host", 40, 240, 1.15, facial=True), name="facial_720p"),
        # the older model files (tanh networks) on VGA frames
        dict(_detect("batch", 640, 480, 3, 8, "host", 40, 240, 1.15, legacy=True), name="legacy_vga_batch"),
        # the serving loop: frames of four sizes in the benchmark's shares, all in flight at once
        {"kind": "serve", "frames": 20, "min_face": 40, "max_face": 240, "scale": 1.15, "gate": False, "name": "serve_mixed"},
        # training of the gate on labelled full-HD frames: forward, backward and Adam
        {"kind": "train", "w8": 240, "h8": 135, "frames": 256, "batch": 64, "lr": 3e-3, "pos_weight": 80.0, "name": "gate_train"},
    ]


def _log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choices(("single", "batch", "serve", "train"), weights=(4, 6, 1, 1))[0]
        if kind == "train":
            batch = _log_between(rng, 8, 96)
            c = {"kind": "train", "w8": _log_between(rng, 40, 240), "h8": _log_between(rng, 30, 135), "frames": batch * rng.randint(1, 4), "batch": batch,
                 "lr": rng.choice((1e-3, 3e-3)), "pos_weight": rng.choice((20.0, 40.0, 80.0))}
        elif kind == "serve":
            c = {"kind": "serve", "frames": rng.randint(10, 40), "min_face": rng.randint(30, 60), "max_face": 240, "scale": 1.15, "gate": rng.random() < 0.5}
        else:
            w = _log_between(rng, 320, 3840)
            h = max(200, min(2160, int(w * rng.choice((9 / 16, 3 / 4, 1.0, 10 / 16)) + rng.randint(-9, 9))))
            channels = rng.choice((1, 3, 3, 3, 4))
            min_face = rng.randint(20, 80)
            max_face = rng.choice((0, 240, 240, 480))
            c = _detect(kind, w, h, channels, 1 if kind == "single" else _log_between(rng, 2, 48), rng.choice(("host", "device")), min_face, max_face,
                        round(rng.uniform(1.05, 1.3), 3))
            option = rng.random()
            if option < 0.2 and channels > 1:
                c["gate"] = True
            elif option < 0.3 and kind == "single":
                c["facial"] = True
            elif option < 0.4 and w * h < 1000000:
                c["legacy"] = True
            if c["source"] == "device" and rng.random() < 0.3:
                c["pad"] = rng.choice((4, 12, 64))  # bytes after each row
            if w * h > 2500000:
                c["slots"] = 4
        if work(c)["flops"] <= 0.8 * most and (kind != "batch" or c["frames"] * c["width"] * c["height"] * c["channels"] < 4e8):
            return c


def _params(case, width, height):
    p = ccnn.default_params()
    p.max_image_width, p.max_image_height = width, height
    p.min_face_height, p.max_face_height, p.scale_factor = case["min_face"], case["max_face"], case["scale"]
    p.facial_analysis = 1 if case.get("facial") else 0
    return p


def _levels(case, width, height, channels):
    info, n = (_capi.LevelInfo * 512)(), ctypes.c_int()
    p = _params(case, width, height)
    _capi.check(_capi.lib().ccnn_plan_levels(ctypes.byref(p), width, height, channels, info, 512, ctypes.byref(n)), "ccnn_plan_levels")
    return [(v.width, v.height, v.resp_width, v.resp_height) for v in info[: n.value]]


def _scan_flops(case, width, height, channels):
    """The stage-1 network over every level, each multiply and add counted. The window networks of stages
    2 and 3 come on top; how many run depends on the frame, so they are not counted."""
    ops = 0
    for w, h, ow, oh in _levels(case, width, height, channels):
        p1 = ((w - 3) >> 1) * ((h - 3) >> 1)
        p2 = ((((w - 3) >> 1) - 2) >> 1) * ((((h - 3) >> 1) - 2) >> 1)
        ops += p1 * 582 + p2 * 718 + ow * oh * 2064
    return ops


def _serve_sizes(case):
    """The sizes of the frames, the mix's shares interleaved."""
    sizes, owed = [], [0.0] * len(SERVE_MIX)
    for _ in range(case["frames"]):
        owed = [o + share for o, (_, share) in zip(owed, SERVE_MIX)]
        k = max(range(len(owed)), key=lambda i: owed[i])
        owed[k] -= 1.0
        sizes.append(SERVE_MIX[k][0])
    return sizes


def work(case):
    if case["kind"] == "train":
        px, cells = case["w8"] * case["h8"], (case["w8"] // 2) * (case["h8"] // 2)
        n = case["frames"] // case["batch"] * case["batch"]
        # forward 8 x 9 and 8 x 8 x 9 taps a pixel; backward the input gradient of the second layer and both
        # layers' weight gradients; the head's products both ways a cell
        flops = n * (2 * px * (72 + 576 + 576 + 576 + 72) + 2 * cells * 4 * 8 * 3)
        return {"bytes": n * (2 * px + 4 * cells) + 2 * 4 * gate.N_PARAMS, "flops": flops}
    if case["kind"] == "serve":
        sizes = _serve_sizes(case)
        return {"bytes": sum(3 * w * h for w, h in sizes), "flops": sum(_scan_flops(case, w, h, 3) for w, h in sizes)}
    w, h, ch, n = case["width"], case["height"], case["channels"], case["frames"]
    return {"bytes": n * (w * h * ch + 32 * 8), "flops": n * _scan_flops(case, w, h, ch)}


def _render(width, height, channels, seed, min_face, step=None):
    """A seeded frame in device memory (rows of `step` bytes) and its face patches."""
    step = step or width * channels
    t = torch.empty(height * step, dtype=torch.uint8, device="cuda")
    n = max(5, min(60, width * height // 104000))
    lo = max(24, int(0.75 * min_face))
    hi = max(lo + 8, min(600 if width > 2000 else 300, int(0.4 * min(width, height))))
    faces = ccnn.synth_frame_device(t.data_ptr(), width, height, seed, n, lo, hi, channels=channels, step=step)
    return t, faces


def _host(frame, width, height, channels, pinned):
    shape = (height, width) if channels == 1 else (height, width, channels)
    a = ccnn.pinned_frame(shape) if pinned else np.empty(shape, np.uint8)
    a[...] = frame.cpu().numpy().reshape(shape)
    return a


def _detector(case):
    p = _params(case, case["width"], case["height"])
    det = ccnn.FaceDetector()
    schedule = autotune.lookup(p, gated=case["gate"]) or {}
    if case["slots"]:
        schedule = dict(schedule, frame_slots=case["slots"])
    if det.Init(p, models=LEGACY if case["legacy"] else None, schedule=schedule or None) != 0:
        raise RuntimeError(_capi.last_error())
    if case["gate"]:
        # the held-out operating point of the shipped weights
        det.setGate(gate.load(), threshold=0.4)
        det.setGateMargin(8)
    return det


def prepare(case, seed):
    gc.collect()
    first = (seed * 4096 + 17) & 0x7FFFFFFF
    if case["kind"] == "train":
        return _prepare_train(case, first)
    if case["kind"] == "serve":
        p = _params(case, 3840, 2160)
        server = ccnn.FaceServer(p, hbm_budget_bytes=16 << 30)
        if case["gate"]:
            server.set_gate(gate.load(), threshold=0.4, margin=8)
        frames = [_host(_render(w, h, 3, first + i, case["min_face"])[0], w, h, 3, True) for i, (w, h) in enumerate(_serve_sizes(case))]
        for f in {f.shape: f for f in frames}.values():
            server.wait(server.submit(f))  # a running server has met every size
        return {"case": case, "server": server, "frames": frames}
    w, h, ch = case["width"], case["height"], case["channels"]
    step = w * ch + case["pad"]
    rendered = [_render(w, h, ch, first + i, case["min_face"], step if case["source"] == "device" else None)[0] for i in range(case["frames"])]
    state = {"case": case, "det": _detector(case), "step": step}
    if case["source"] == "device":
        state["frames"] = rendered
        n = case["frames"]
        state["images"] = (_capi.Image * n)(*[_capi.Image(w, h, ch, t.data_ptr(), step) for t in rendered])
        state["faces"], state["count"] = (_capi.Face * (n * CAPACITY))(), (ctypes.c_int * n)()
    else:
        state["frames"] = [_host(t, w, h, ch, case["kind"] == "batch") for t in rendered]
    return state


def _prepare_train(case, first):
    w8, h8, n = case["w8"], case["h8"], case["frames"]
    L = _capi.lib()
    w, h = 8 * w8, 8 * h8
    pitch = (w + 15) // 16 * 16
    gray = torch.zeros((h, pitch), dtype=torch.float32, device="cuda")
    feat = torch.empty((n, h8, w8), dtype=torch.float16, device="cuda")
    labels = np.zeros((n, 4, h8 // 2, w8 // 2), np.uint8)
    step = (w + 63) // 64 * 64
    for i in range(n):
        t, faces = _render(w, h, 1, first + i, 40, step)
        _capi.check(L.ccnn_gray_u8_to_f32(t.data_ptr(), w, h, 1, step, gray.data_ptr(), pitch * 4, None), "ccnn_gray_u8_to_f32")
        _capi.check(L.ccnn_gate_features(gray.data_ptr(), w, h, pitch * 4, feat[i].data_ptr(), None), "ccnn_gate_features")
        for cx, cy, fw, fh, _angle, _contrast in faces:
            octave = min(3, max(0, int(math.log2(max(fh, 40) / 40))))
            labels[i, octave, min(h8 // 2 - 1, max(0, int(cy) // 16)), min(w8 // 2 - 1, max(0, int(cx) // 16))] = 1
    torch.cuda.synchronize()
    return {"case": case, "params": gate.init_params(first % 1000), "feat": feat, "labels": torch.from_numpy(labels).cuda()}


def _table(found):
    """Faces of several frames, each a list of tuples that start (x, y, width, height, score), as a table of
    KEEP rows a frame (zeros past a frame's count)."""
    rects = np.zeros((len(found), KEEP, 7), np.int32)
    scores = np.zeros((len(found), KEEP), np.float32)
    for i, faces in enumerate(found):
        for j, f in enumerate(faces[:KEEP]):
            rects[i, j, :4 + len(f) - 5] = f[:4] + f[5:]
            scores[i, j] = f[4]
    return {"count": np.array([len(faces) for faces in found], np.int32), "rects": rects, "scores": scores}


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        params = state["params"].copy()
        losses = np.zeros(1, np.float32)
        fp = ctypes.POINTER(ctypes.c_float)
        st = _capi.lib().ccnn_gate_train(params.ctypes.data_as(fp), state["feat"].data_ptr(), state["labels"].data_ptr(), case["frames"], case["w8"], case["h8"],
                                         case["batch"], 1, case["lr"], case["pos_weight"], losses.ctypes.data_as(fp))
        _capi.check(st, "ccnn_gate_train")
        return {"params": params, "losses": losses}
    if case["kind"] == "serve":
        tickets = [state["server"].submit(f) for f in state["frames"]]
        return _table([state["server"].wait(t)[0] for t in tickets])
    det, w, h, ch = state["det"], case["width"], case["height"], case["channels"]
    if case["kind"] == "single":
        if case["source"] == "device":
            return _table([det.DetectDevice(state["frames"][0].data_ptr(), w, h, ch, state["step"])])
        return _table([det.Detect(state["frames"][0], attributes=case["facial"])])
    if case["source"] == "host":
        return _table(det.DetectBatch(state["frames"]))
    n = case["frames"]
    st = _capi.lib().ccnn_detect_device_batch(det._h, state["images"], n, state["faces"], CAPACITY, state["count"], None)
    _capi.check(st, "ccnn_detect_device_batch")
    faces = state["faces"]
    return _table([[(f.x, f.y, f.width, f.height, f.score) for f in faces[i * CAPACITY: i * CAPACITY + min(state["count"][i], CAPACITY)]] for i in range(n)])


def exact(case, seed):
    if case["kind"] != "train":
        return None
    s = prepare(case, seed)
    F = torch.nn.functional
    p = torch.from_numpy(s["params"]).double().cuda()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    losses = []
    for k in range(case["frames"] // case["batch"]):
        part = slice(k * case["batch"], (k + 1) * case["batch"])
        x, y = s["feat"][part].double()[:, None], s["labels"][part].double()
        q = p.clone().requires_grad_(True)
        a = F.leaky_relu(F.conv2d(x, q[:72].reshape(8, 1, 3, 3), q[72:80], padding=1), 0.1)
        a = F.leaky_relu(F.conv2d(a, q[80:656].reshape(8, 8, 3, 3), q[656:664], padding=1), 0.1)
        z = F.conv2d(F.avg_pool2d(a, 2), q[664:696].reshape(4, 8, 1, 1), q[696:])
        loss = (case["pos_weight"] * y * F.softplus(-z) + (1 - y) * F.softplus(z)).mean()
        g, = torch.autograd.grad(loss, q)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - case["lr"] * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
        losses.append(loss.detach())
    return {"params": p.cpu().numpy(), "losses": torch.stack(losses).mean().reshape(1).cpu().numpy()}
