"""Workloads of the encoder-analysis library, as a program that uses it calls them.

`listed()` names the workloads, `draw(rng)` gives more of the same ranges,
`prepare` builds one workload's inputs on the GPU from a seed, `run` is one
pass through the public entry points and `work` the bytes and operations the
pass cannot do without. A picture's content follows the library's synthetic
sequences (vp8a.synth): a sum of gratings, cut into horizontal bands that move
by their own quarter-pel vectors, flat rectangles moving over it, fresh noise
on every frame. A program keeps one library context for its lifetime, so a
kind of workload shares one here.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oxideav-vp8_b200"))

import vp8a  # noqa: E402
from vp8a import abi, learned  # noqa: E402
from vp8a.stream import AltrefStreams  # noqa: E402

REF_IDS = (abi.REF_LAST, abi.REF_GOLDEN, abi.REF_ALTREF)


def listed():
    return [
        # The smallest call: one QCIF frame against LAST, as a low-resolution
        # call or a thumbnail stream makes it every frame.
        {"name": "analyse_176x144", "kind": "analyse", "w": 176, "h": 144, "refs": 1, "qi": 44},
        # The exhaustive analysis of one full-HD frame against all references.
        {"name": "analyse_1080p", "kind": "analyse", "w": 1920, "h": 1080, "refs": 3, "qi": 44},
        # The reduced (RD-effort) search of a live encoder at its middle effort.
        {"name": "rd_search_1080p", "kind": "rd", "w": 1920, "h": 1080, "refs": 3, "qi": 44, "effort": 2},
        # Batched block search of every MB from given centres; neither side a
        # multiple of 16.
        {"name": "descent_1366x766", "kind": "descent", "w": 1366, "h": 766, "qi": 44},
        # What follows the reconstruction in an encoder: the reference's
        # level / sharpness walk, then the filter pass over the picture.
        {"name": "loop_filter_720p", "kind": "loop_filter", "w": 1280, "h": 720, "qi": 72},
        # Every (level, sharpness) pair scored: the full 64 x 8 grid.
        {"name": "sweep_1080p", "kind": "sweep", "w": 1920, "h": 1080, "qi": 44},
        # One whole frame step on the device, the benchmark's: altref anchor,
        # analysis, reconstruction, loop-filter grid.
        {"name": "frame_1080p", "kind": "frame", "w": 1920, "h": 1080, "qi": 44, "lookahead": 7},
        # A frame coded from host pictures to a bitstream in one call.
        {"name": "encode_640x360", "kind": "encode", "w": 640, "h": 360, "qi": 56},
        # A transcoding node's step: streams of uneven sizes, each stage one
        # batched call, one reference each.
        {"name": "batch_streams", "kind": "batch", "qi": 44, "lookahead": 5,
         "mix": "3840x2160*1,1920x1080*2,1280x720*3,641x363*2,176x144*2"},
        # A lookahead group of lagged altref streams coded in lockstep with
        # the trellis on: the largest call.
        {"name": "altref_group", "kind": "group", "qi": 44, "frames": 5, "mix": "3840x2160*1,1280x720*2"},
        # The learned proposal search of one full-HD frame and reference.
        {"name": "proposals_1080p", "kind": "proposals", "w": 1920, "h": 1080},
        # The forward and backward pass that trains the proposal net.
        {"name": "train_2048", "kind": "train", "n": 2048},
    ]


def _size(rng, least, most, most_mbs):
    """A picture size, spread over the logarithm of its width; any parity."""
    while True:
        w = int(round(math.exp(rng.uniform(math.log(least), math.log(most)))))
        h = int(round(w * rng.uniform(0.45, 1.1)))
        if h >= 16 and _mbs(w, h) <= most_mbs:
            return w, h


def draw(rng):
    kind = rng.choice(["analyse", "rd", "descent", "loop_filter", "sweep", "frame", "encode", "batch", "group",
                       "proposals", "train"])
    c = {"kind": kind, "qi": rng.randint(8, 110)}
    if kind == "train":
        return {"kind": kind, "n": int(round(math.exp(rng.uniform(math.log(64), math.log(2048)))))}
    if kind in ("batch", "group"):
        left, mix = (50000, []) if kind == "batch" else (32000, [])
        for _ in range(rng.randint(2, 8 if kind == "batch" else 4)):
            w, h = _size(rng, 96, 2560, max(64, left // 2))
            n = rng.randint(1, 2)
            left -= n * _mbs(w, h)
            mix.append("%dx%d*%d" % (w, h, n))
        c["mix"] = ",".join(mix)
        c["frames" if kind == "group" else "lookahead"] = rng.randint(3, 5)
        return c
    c["w"], c["h"] = _size(rng, 64, 1000 if kind == "encode" else 1920, 3600 if kind == "encode" else 8160)
    if kind in ("analyse", "rd"):
        c["refs"] = rng.randint(1, 3)
    if kind == "rd":
        c["effort"] = rng.randint(0, 3)
    if kind == "frame":
        c["lookahead"] = rng.randint(3, 7)
    if kind == "proposals":
        del c["qi"]
    return c


# ------------------------------------------------------------------ pictures


def _mbs(w, h):
    return ((w + 15) // 16) * ((h + 15) // 16)


def _mix(text):
    """"WxH*N,..." -> one (width, height) per stream."""
    out = []
    for part in text.split(","):
        size, n = part.split("*")
        w, h = size.split("x")
        out += [(int(w), int(h))] * int(n)
    return out


def _plane(h, w, scale, waves, rows_dy, rows_dx, sigma, g):
    """One plane: gratings (theta, period, amplitude, phase) displaced per
    row, plus noise. `scale` 2 samples at half resolution."""
    y = torch.arange(h, device="cuda", dtype=torch.float32)[:, None] * scale + rows_dy
    x = torch.arange(w, device="cuda", dtype=torch.float32)[None, :] * scale + rows_dx
    acc = torch.full((h, w), 128.0, device="cuda")
    for theta, period, amp, phase in waves:
        f = 2.0 * math.pi / period
        acc += amp * torch.sin(x * (f * math.cos(theta)) + y * (f * math.sin(theta)) + phase)
    acc += sigma * torch.randn((h, w), device="cuda", generator=g)
    return acc


def _sequence(w, h, n, seed, bands=4, boxes=3):
    """n (y, u, v) uint8 device pictures of one moving scene. The noise of two
    frames differs by a sigma of 3 (luma) and 2 (chroma), vp8a.synth's."""
    rng = np.random.Generator(np.random.PCG64(seed))
    g = torch.Generator(device="cuda").manual_seed(seed)
    cw, ch = (w + 1) // 2, (h + 1) // 2

    def waves(k, lo, hi):
        return [(rng.uniform(0, math.pi), rng.uniform(8, 64), rng.uniform(lo, hi), rng.uniform(0, 2 * math.pi))
                for _ in range(k)]

    wy, wu, wv = waves(6, 20, 50), waves(2, 8, 16), waves(2, 8, 16)
    move = np.zeros((bands, 2))
    box = [[rng.uniform(0, w), rng.uniform(0, h), int(rng.integers(8, max(9, w // 4))),
            int(rng.integers(8, max(9, h // 4))), int(rng.integers(0, 256)), rng.uniform(-6, 6), rng.uniform(-6, 6)]
           for _ in range(boxes)]
    band_y = torch.arange(h, device="cuda") * bands // h
    band_c = torch.clamp(torch.arange(ch, device="cuda") * 2, max=h - 1) * bands // h
    frames = []
    for k in range(n):
        if k:
            move += rng.integers(-32, 33, (bands, 2)) / 4.0  # quarter pels, at most 8 px a frame
        m = torch.from_numpy(move.astype(np.float32)).cuda()
        dy, dx = m[band_y, 0][:, None], m[band_y, 1][:, None]
        cy, cx = m[band_c, 0][:, None], m[band_c, 1][:, None]
        y = _plane(h, w, 1, wy, dy, dx, 2.1, g)
        u = _plane(ch, cw, 2, wu, cy, cx, 1.4, g)
        v = _plane(ch, cw, 2, wv, cy, cx, 1.4, g)
        for b in box:
            x0, y0 = int(b[0]) % w, int(b[1]) % h
            y[y0:y0 + b[3], x0:x0 + b[2]] = float(b[4])
            u[y0 // 2:(y0 + b[3]) // 2, x0 // 2:(x0 + b[2]) // 2] = float(255 - b[4])
            b[0] += b[5]
            b[1] += b[6]
        frames.append(tuple(torch.clamp(torch.round(p), 0, 255).to(torch.uint8) for p in (y, u, v)))
    return frames


def _padded(frame):
    """Edge-replicated MB-padded planes of a picture: a reference's layout."""
    out = []
    h, w = frame[0].shape
    for k, p in enumerate(frame):
        s = 16 if k == 0 else 8
        ys = torch.arange((h + 15) // 16 * s, device="cuda").clamp(max=p.shape[0] - 1)
        xs = torch.arange((w + 15) // 16 * s, device="cuda").clamp(max=p.shape[1] - 1)
        out.append(p[ys][:, xs].contiguous())
    return out


def _zeros_padded(w, h):
    mr, mc = (h + 15) // 16, (w + 15) // 16
    return [torch.zeros((mr * s, mc * s), dtype=torch.uint8, device="cuda") for s in (16, 8, 8)]


def _bytes(n):
    return torch.zeros(n, dtype=torch.uint8, device="cuda")


_contexts = {}


def _context(kind):
    if kind not in _contexts:
        _contexts[kind] = vp8a.Context(0)
    return _contexts[kind]


def _ok(status, where):
    if status:
        raise vp8a.Vp8aError(status, where)


# ------------------------------------------------- one frame on the device


class Frame:
    """One stream's frame: its pictures, references and result buffers on the
    device and the C-ABI records that name them."""

    def __init__(self, ctx, w, h, seed, refs=3, qi=44, lookahead=0):
        self.ctx, self.lib, self.n = ctx, vp8a.load(), _mbs(w, h)
        self.n_refs, self.lam, self.quant = refs, vp8a.rd_lambda(qi), abi.quant_indices(qi)
        # Frame 3 is coded; LAST = 2, GOLDEN = 0, ALTREF = 5 (or the anchor
        # of the lookahead window 4 ..).
        seq = _sequence(w, h, 4 + max(2, lookahead), seed)
        self.src = seq[3]
        self.refs = [_padded(seq[2]), _padded(seq[0]), _padded(seq[5])][:refs]
        self.window = seq[4:4 + lookahead]
        self.dec = _bytes(self.n * abi.MB_DECISION_DTYPE.itemsize)
        self.lf = _bytes(self.n * abi.MB_LF_INFO_DTYPE.itemsize)
        self.recon = _zeros_padded(w, h)
        self.coeffs = torch.zeros((self.n, 400), dtype=torch.int16, device="cuda")
        self.flags = _bytes(self.n)
        self.table = torch.zeros(512, dtype=torch.int64, device="cuda")
        self.ids = np.array(REF_IDS[:refs], np.uint8)
        self.mvc = abi.default_mv_contexts()
        self.c_src, self.c_source = vp8a.i420(*self.src), vp8a.source(*self.src)
        self.c_refs = (abi.Planes * refs)(*[vp8a.planes(*r) for r in self.refs])
        self.p_refs = C.cast(self.c_refs, C.c_void_p)
        self.c_recon = vp8a.planes(*self.recon)
        self.base = abi.filter_config(0, 0)
        if lookahead:
            self.altref = _zeros_padded(w, h)
            self.c_altref = vp8a.planes(*self.altref)
            self.c_window = (abi.I420 * lookahead)(*[vp8a.i420(*f) for f in self.window])
            if refs == 3:
                self.refs[2] = self.altref
                self.c_refs[2] = self.c_altref

    def anchor(self):
        n = len(self.window)
        _ok(self.lib.vp8a_build_arnr_altref_planes(self.ctx.handle, C.cast(self.c_window, C.c_void_p), n, n // 2, 3,
                                                   C.byref(self.c_altref)), "vp8a_build_arnr_altref_planes")

    def analyse(self):
        _ok(self.lib.vp8a_analyse_inter_frame(self.ctx.handle, C.byref(self.c_src), self.p_refs, self.ids.ctypes.data,
                                              self.n_refs, C.byref(self.mvc), self.lam, self.dec.data_ptr(), None),
            "vp8a_analyse_inter_frame")

    def reconstruct(self):
        _ok(self.lib.vp8a_reconstruct_inter_frame(
            self.ctx.handle, C.byref(self.c_src), self.p_refs, self.ids.ctypes.data, self.n_refs, self.dec.data_ptr(),
            C.byref(self.quant), None, None, 0, 0, abi.FILTER_SIXTAP, C.byref(self.c_recon), self.coeffs.data_ptr(),
            self.flags.data_ptr(), self.lf.data_ptr()), "vp8a_reconstruct_inter_frame")

    def sweep(self):
        _ok(self.lib.vp8a_filter_sweep(self.ctx.handle, C.byref(self.c_recon), self.lf.data_ptr(), C.byref(self.base),
                                       C.byref(self.c_source), 0, self.table.data_ptr()), "vp8a_filter_sweep")

    # The same stages' records for the batched calls.
    def arnr_job(self):
        n = len(self.window)
        return abi.ArnrPlanesJob(C.cast(self.c_window, C.c_void_p), n, n // 2, 3, self.c_altref)

    def analysis_job(self):
        return abi.AnalysisJob(self.c_src, self.p_refs, self.ids.ctypes.data, self.n_refs,
                               C.cast(C.pointer(self.mvc), C.c_void_p), self.lam, self.dec.data_ptr(), None)

    def recon_job(self):
        return abi.ReconJob(self.c_src, self.p_refs, self.ids.ctypes.data, self.n_refs, 0, self.dec.data_ptr(),
                            self.quant, None, None, 0, abi.FILTER_SIXTAP, self.c_recon, self.coeffs.data_ptr(),
                            self.flags.data_ptr(), self.lf.data_ptr())

    def sweep_job(self):
        return abi.SweepJob(self.c_recon, self.lf.data_ptr(), self.base, self.c_source, 0, self.table.data_ptr())


# -------------------------------------------------------- the proposal net


def _net_weights(seed):
    """A net as training leaves it: a path that carries the matching cost
    from the input to the score, random features around it (BF16 values)."""
    g = torch.Generator().manual_seed(seed)
    out = []
    for k, (cin, cout) in enumerate(((2, 32), (32, 32), (32, 32), (32, 1))):
        w = torch.randn((cout, 9, cin), generator=g) * (0.3 * (2.0 / (9 * cin)) ** 0.5)
        w[0, :, 0] += 0.05
        w[0, 4, 0] += 1.0
        b = torch.randn(cout, generator=g) * 0.02
        out.append((w.to(torch.bfloat16).float().cuda(), b.cuda()))
    return out


def _net(ctx, seed):
    net = learned.ProposalNet(ctx, seed=seed % (1 << 30))
    with learned.on_ctx_stream(ctx):
        for layer, (w, b) in zip(net.layers, _net_weights(seed)):
            layer["w"].copy_(w.reshape(-1))
            layer["wh"].copy_(w.reshape(-1))
            layer["b"].copy_(b)
            layer["bh"].copy_(b)
    return net


def _train_inputs(n, seed):
    """Cost volumes around a known best cell ([n, 32, 32, 2] BF16: a bowl of
    matching cost over textured noise, the reference's texture) and that
    cell."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    label = torch.randint(0, 1024, (n,), device="cuda", generator=g, dtype=torch.int32)
    r, c = torch.meshgrid(torch.arange(32, device="cuda"), torch.arange(32, device="cuda"), indexing="ij")
    d2 = (r[None] - label[:, None, None] // 32) ** 2 + (c[None] - label[:, None, None] % 32) ** 2
    texture = torch.randn((n, 1, 8, 8), device="cuda", generator=g)
    texture = torch.nn.functional.interpolate(texture, (32, 32), mode="bilinear", align_corners=False)[:, 0]
    cost = 0.2 + 0.7 * torch.exp(-d2 / 18.0) + 0.15 * texture
    cost += 0.05 * torch.randn(cost.shape, device="cuda", generator=g)
    return torch.stack([cost, 0.6 * texture], dim=3).to(torch.bfloat16).contiguous(), label


def exact(case, seed):
    """The training pass in 64 bits: the scores, the summed cross-entropy and
    every layer's gradient. The other workloads' outputs are whole numbers
    (vectors, pixels, sums of squares, records compared byte by byte)."""
    if case["kind"] != "train":
        return None
    x, label = _train_inputs(case["n"], seed)
    params = []
    for w, b in _net_weights(seed):
        w = w.double().reshape(w.shape[0], 3, 3, w.shape[2]).permute(0, 3, 1, 2).contiguous()
        params.append((w.requires_grad_(), b.double().requires_grad_()))
    logits, loss = [], 0.0
    for k in range(0, case["n"], 256):
        h = x[k:k + 256].double().permute(0, 3, 1, 2)
        for i, (w, b) in enumerate(params):
            h = torch.nn.functional.conv2d(h, w, b, padding=1)
            h = torch.relu(h) if i < 3 else h
        z = h.reshape(h.shape[0], 1024)
        ce = torch.nn.functional.cross_entropy(z, label[k:k + 256].long(), reduction="sum")
        (ce / case["n"]).backward()
        logits.append(z.detach())
        loss += float(ce)
    return {"logits": torch.cat(logits), "loss": torch.tensor([loss], dtype=torch.float64),
            "gw": [w.grad.permute(0, 2, 3, 1).reshape(-1) for w, _ in params], "gb": [b.grad for _, b in params[:3]]}


# ------------------------------------------------------------------ passes


def prepare(case, seed):
    kind = case["kind"]
    ctx = _context(kind)
    s = {"kind": kind, "ctx": ctx}
    if kind in ("analyse", "sweep", "loop_filter", "frame", "rd", "descent"):
        f = s["frame"] = Frame(ctx, case["w"], case["h"], seed, case.get("refs", 3), case["qi"],
                               case.get("lookahead", 0))
        torch.cuda.synchronize()
        if kind in ("sweep", "loop_filter"):
            f.analyse()
            f.reconstruct()
            s["out"] = [torch.zeros_like(p) for p in f.recon]
            s["stream"] = torch.cuda.ExternalStream(ctx.stream)
        elif kind == "rd":
            f.analyse()
            ctx.synchronize()
            dec = f.dec.cpu().numpy().view(abi.MB_DECISION_DTYPE).reshape((case["h"] + 15) // 16, -1)
            near = vp8a.neighbours_from_decisions(dec)
            s["near"] = torch.from_numpy(near.view(np.uint8)).cuda()
            s["found"] = _bytes(f.n * abi.RD_INTER_DTYPE.itemsize)
            # y_ac_qi's AC step from lambda = step^2 / 32.
            s["y1_ac"], s["effort"] = int(round(math.sqrt(32 * f.lam))), case["effort"]
        elif kind == "descent":
            mc = (case["w"] + 15) // 16
            k = torch.arange(f.n, device="cuda")
            s["xy"] = torch.stack([k % mc, k // mc], 1).to(torch.int32).contiguous()
            y = _padded(f.src)[0]
            s["mbs"] = y.view(y.shape[0] // 16, 16, mc, 16).permute(0, 2, 1, 3).reshape(-1, 256).contiguous()
            g = torch.Generator(device="cuda").manual_seed(seed)
            s["mv"] = torch.randint(-32, 33, (f.n, 2), device="cuda", generator=g).to(torch.int16)
            s["found"] = [torch.zeros((f.n, 2), dtype=torch.int32, device="cuda") for _ in range(3)]
            s["ref"] = vp8a.luma_ref(f.refs[0][0])
    elif kind == "encode":
        host = [tuple(p.cpu().numpy() for p in f) for f in _sequence(case["w"], case["h"], 6, seed)]
        s["src"], s["qi"] = host[3], case["qi"]
        s["bits"] = np.zeros(1024 + 600 * _mbs(case["w"], case["h"]), np.uint8)
        s["refs"] = [vp8a.pad_to_mb(*host[k]) for k in (2, 0, 5)]
    elif kind == "batch":
        fs = s["frames"] = [Frame(ctx, w, h, seed * 64 + k, 1, case["qi"], case["lookahead"])
                            for k, (w, h) in enumerate(_mix(case["mix"]))]
        for name, record, make in (("arnr", abi.ArnrPlanesJob, Frame.arnr_job),
                                   ("analyse", abi.AnalysisJob, Frame.analysis_job),
                                   ("recon", abi.ReconJob, Frame.recon_job),
                                   ("sweep", abi.SweepJob, Frame.sweep_job)):
            s[name] = (record * len(fs))(*[make(f) for f in fs])
    elif kind == "group":
        sizes = _mix(case["mix"])
        n = case["frames"]
        seqs = [_sequence(w, h, n + 2, seed * 64 + k) for k, (w, h) in enumerate(sizes)]
        s["group"] = [q[2:] for q in seqs]
        s["streams"] = AltrefStreams(ctx, sizes, qi=case["qi"], write=False)
        torch.cuda.synchronize()
        s["streams"].encode_group([q[:2] for q in seqs])  # the streams' opening frames
    elif kind == "proposals":
        a, b = _sequence(case["w"], case["h"], 2, seed)
        s["src"], s["ref"] = b[0], _padded(a)[0]
        s["xy"] = learned.all_mbs((case["w"] + 15) // 16, (case["h"] + 15) // 16)
        s["net"] = _net(ctx, seed)
    elif kind == "train":
        s["x"], s["label"] = _train_inputs(case["n"], seed)
        s["net"] = _net(ctx, seed)
    torch.cuda.synchronize()
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    lib, f = vp8a.load(), s.get("frame")
    if kind == "analyse":
        f.analyse()
        return f.dec
    if kind == "rd":
        _ok(lib.vp8a_rd_inter_search(ctx.handle, C.byref(f.c_src), f.p_refs, f.ids.ctypes.data, f.n_refs,
                                     C.byref(f.mvc), f.lam, s["y1_ac"], s["effort"], s["near"].data_ptr(),
                                     s["found"].data_ptr()), "vp8a_rd_inter_search")
        return s["found"]
    if kind == "descent":
        w, h, q = s["found"]
        _ok(lib.vp8a_motion_descent(ctx.handle, C.byref(s["ref"]), s["mbs"].data_ptr(), s["xy"].data_ptr(),
                                    s["mv"].data_ptr(), 8, f.n, w.data_ptr(), h.data_ptr(), q.data_ptr()),
            "vp8a_motion_descent")
        return s["found"]
    if kind == "sweep":
        f.sweep()
        return f.table
    if kind == "loop_filter":
        level, sharp = C.c_uint8(), C.c_uint8()
        _ok(lib.vp8a_select_filter_params(ctx.handle, C.byref(f.c_recon), f.lf.data_ptr(), C.byref(f.base),
                                          C.byref(f.c_source), C.byref(level), C.byref(sharp)),
            "vp8a_select_filter_params")
        with torch.cuda.stream(s["stream"]):
            for d, p in zip(s["out"], f.recon):
                d.copy_(p)
        out, cfg = vp8a.planes(*s["out"]), abi.filter_config(level.value, sharp.value)
        _ok(lib.vp8a_filter_frame(ctx.handle, C.byref(out), f.lf.data_ptr(), C.byref(cfg)), "vp8a_filter_frame")
        return {"level": level.value, "sharpness": sharp.value, "planes": s["out"]}
    if kind == "frame":
        f.anchor()
        f.analyse()
        f.reconstruct()
        f.sweep()
        return {"altref": f.altref, "decisions": f.dec, "recon": f.recon, "coeffs": f.coeffs, "flags": f.flags,
                "lf": f.lf, "table": f.table}
    if kind == "encode":
        bits, out, d = vp8a.encode_p_frame(ctx, s["src"], s["refs"], list(REF_IDS), s["qi"])
        # In a buffer of the stream's own size: a frame's length depends on
        # its content.
        s["bits"][:len(bits)] = np.frombuffer(bits, np.uint8)
        s["bits"][len(bits):] = 0
        return {"bytes": s["bits"], "size": len(bits), "planes": list(out), "level": d["level"],
                "sharpness": d["sharpness"]}
    if kind == "batch":
        fs, n = s["frames"], len(s["frames"])
        for name, fn in (("arnr", "vp8a_build_arnr_altrefs_planes"), ("analyse", "vp8a_analyse_inter_frames"),
                         ("recon", "vp8a_reconstruct_inter_frames"), ("sweep", "vp8a_filter_sweeps")):
            _ok(getattr(lib, fn)(ctx.handle, C.cast(s[name], C.c_void_p), n), fn)
        return [[q.altref[0], q.dec, q.recon[0], q.table] for q in fs]
    if kind == "group":
        packets = s["streams"].encode_group(s["group"])
        return {"levels": [[[p["level"], p["sharpness"]] for p in q] for q in packets[:1]],
                "last": [s["streams"].references(k)[0] for k in range(len(packets))],
                "altref": [s["streams"].references(k)[2][0] for k in range(len(packets))]}
    if kind == "proposals":
        return list(learned.learned_search(ctx, s["net"], s["src"], s["ref"], s["xy"]))
    net = s["net"]
    net.zero_grad()
    logits = net.forward(s["x"], keep=True)
    loss, d, _ = net.loss_and_grad(logits, s["label"])
    net.backward(d)
    # The last layer's bias gradient is the sum of a softmax minus a one-hot:
    # zero but for rounding, so it is left out.
    return {"logits": logits, "loss": loss, "gw": [p["gw"] for p in net.layers],
            "gb": [p["gb"] for p in net.layers[:3]]}


def work(case):
    """Bytes: inputs once, outputs once. Operations: the integer work of the
    searches (about 92,000 per MB and reference), of the filters (9,000 per MB
    and distinct candidate: 436 of the full grid, about 30 of a walk) and of
    the anchor (33 x 256 per block and frame); multiply-adds of the net."""
    kind = case["kind"]
    if kind == "train":
        n = case["n"]
        return {"bytes": n * 1024 * 8.0, "flops": n * (3 * 39.5e6 - 2 * 9 * 64 * 1024)}
    if kind in ("batch", "group"):
        sizes = _mix(case["mix"])
        m = float(sum(_mbs(w, h) for w, h in sizes))
        px = float(sum(w * h for w, h in sizes))
        if kind == "batch":
            la = case["lookahead"]
            return {"bytes": 1.5 * px * (la + 1) + m * (616 + 2072 + 774),
                    "flops": m * (92e3 + 9e3 * 436 + 33 * 256 * (la - 1))}
        n = case["frames"]
        return {"bytes": 1.5 * px * (n + 1) + (n + 1) * m * (1128 + 2072 + 774 + 768),
                "flops": (n + 1) * m * (3 * 92e3 + 9e3 * 31) + m * 33 * 256 * (n - 1)}
    w, h, r = case["w"], case["h"], case.get("refs", 3)
    m = float(_mbs(w, h))
    if kind == "analyse":
        return {"bytes": m * (256 + 256 * r + 104), "flops": m * r * 92e3}
    if kind == "rd":
        return {"bytes": m * (256 + 256 * r + 216 + 56), "flops": m * r * 33 * 256.0}
    if kind == "descent":
        return {"bytes": m * (512 + 12 + 24), "flops": m * 49 * 256.0}
    if kind == "sweep":
        return {"bytes": m * 776 + 4096, "flops": m * 9e3 * 436}
    if kind == "loop_filter":
        return {"bytes": m * (776 + 768), "flops": m * 9e3 * 31}
    if kind == "frame":
        la = case["lookahead"]
        return {"bytes": 1.5 * w * h * (la + 1) + m * (1128 + 2072 + 776),
                "flops": m * (3 * 92e3 + 9e3 * 436 + 33 * 256 * (la - 1))}
    if kind == "encode":
        return {"bytes": m * (1128 + 2072 + 1544), "flops": m * (3 * 92e3 + 9e3 * 31)}
    return {"bytes": m * (512 + 9), "flops": m * 39.5e6}  # proposals
