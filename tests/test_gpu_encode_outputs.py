"""What vp8a_encode_inter_frame may write: the rows of its output planes, no byte
between them (planes are often rectangles of a larger surface), `filtered` only
when the level is not 0, and no byte of `out` past the frame."""
import ctypes as C

import numpy as np
import pytest

import vp8a
from vp8a import abi, synth

pytestmark = pytest.mark.gpu

FILL = 0xA5


def surfaces(ref, pad):
    """Sentinel-filled surfaces whose left parts are planes of `ref`'s sizes."""
    whole = [np.full((p.shape[0], p.shape[1] + pad), FILL, np.uint8) for p in ref]
    return whole, [s[:, :p.shape[1]] for s, p in zip(whole, ref)]


def encode(ctx, frame, refs, qi, level, auto_lf, recon, filtered, out, capacity):
    n = refs[0][0].size // 256
    dec, lf = np.zeros(n, abi.MB_DECISION_DTYPE), np.zeros(n, abi.MB_LF_INFO_DTYPE)
    cf, fl = np.zeros((n, 400), np.int16), np.zeros(n, np.uint8)
    pl = (abi.Planes * len(refs))(*[vp8a.planes(*r) for r in refs])
    ids = np.array([1, 2, 3][:len(refs)], np.uint8)
    hdr = abi.frame_header(frame[0].shape[1], frame[0].shape[0], abi.quant_indices(qi), loop_filter_level=level)
    lv, sh, size = C.c_uint8(), C.c_uint8(), C.c_uint64()
    st = ctx._lib.vp8a_encode_inter_frame(
        ctx.handle, C.byref(vp8a.i420(*frame)), C.cast(pl, C.c_void_p), ids.ctypes.data, len(refs),
        C.byref(abi.default_mv_contexts()), vp8a.rd_lambda(qi), None, C.byref(hdr), int(auto_lf), dec.ctypes.data,
        cf.ctypes.data, fl.ctypes.data, lf.ctypes.data, C.byref(vp8a.planes(*recon)), C.byref(vp8a.planes(*filtered)),
        C.byref(lv), C.byref(sh), out.ctypes.data, capacity, C.byref(size))
    return st, size.value, lv.value, (dec, cf, fl, lf)


def case(w, h, n_refs):
    frames, _ = synth.make_sequence(w, h, 4, seed=w + n_refs, pieces=3, occluders=2)
    return frames[3], [vp8a.pad_to_mb(*frames[k]) for k in (2, 0, 1)][:n_refs]


@pytest.mark.parametrize("pad", [16, 64, 4096])
@pytest.mark.parametrize("level,auto_lf", [(0, False), (30, False), (0, True)])
def test_only_the_outputs_change(ctx, pad, level, auto_lf):
    # 640 x 368 planes at a pitch of 704: six multiples of 4096 lie between rows.
    frame, refs = case(640, 360, 2)
    want_bits, want, d = vp8a.encode_p_frame(ctx, frame, refs, [1, 2], 50, loop_filter_level=level, auto_lf=auto_lf)
    big_r, recon = surfaces(refs[0], pad)
    big_f, filtered = surfaces(refs[0], pad)
    out = np.full(1024 + 600 * d["flags"].size + 9000, FILL, np.uint8)
    st, size, lv, _ = encode(ctx, frame, refs, 50, level, auto_lf, recon, filtered, out, out.size)
    assert st == abi.OK and lv == d["level"] and out[:size].tobytes() == want_bits
    assert (out[size:] == FILL).all()
    for s, p, q in zip(big_r, recon, d["recon"]):
        assert np.array_equal(p, q) and (s[:, q.shape[1]:] == FILL).all()
    for s, p, q in zip(big_f, filtered, want):
        assert (s[:, q.shape[1]:] == FILL).all()
        assert np.array_equal(p, q) if lv else (p == FILL).all()


@pytest.mark.parametrize("capacity", [0, 1, 5000])
def test_a_short_buffer_is_not_overrun(ctx, capacity):
    frame, refs = case(320, 240, 1)
    want_bits, want, d = vp8a.encode_p_frame(ctx, frame, refs, [1], 4)
    assert len(want_bits) > capacity
    _, recon = surfaces(refs[0], 0)
    _, filtered = surfaces(refs[0], 0)
    out = np.full(20000, FILL, np.uint8)
    st, size, lv, _ = encode(ctx, frame, refs, 4, 0, True, recon, filtered, out, capacity)
    assert st == abi.E_INVALID_ARGUMENT and size == len(want_bits) and (out[capacity:] == FILL).all()
    assert lv == d["level"] and all(np.array_equal(a, b) for a, b in zip(recon, d["recon"]))
