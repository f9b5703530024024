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


def encode(ctx, frame, refs, qi, level, auto_lf, recon, filtered, out, capacity, **header):
    n = refs[0][0].size // 256
    dec, lf = np.zeros(n, abi.MB_DECISION_DTYPE), np.zeros(n, abi.MB_LF_INFO_DTYPE)
    cf, fl = np.zeros((n, 400), np.int16), np.zeros(n, np.uint8)
    pl = (abi.Planes * len(refs))(*[vp8a.planes(*r) for r in refs])
    ids = np.array([1, 2, 3][:len(refs)], np.uint8)
    hdr = abi.frame_header(frame[0].shape[1], frame[0].shape[0], abi.quant_indices(qi), loop_filter_level=level, **header)
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


@pytest.mark.parametrize("level,auto_lf", [(30, False), (0, True)])
def test_the_headers_filter_deltas_are_applied(ctx, level, auto_lf):
    # What a decoder of the frame adds to its levels, the call's own filter adds.
    deltas = dict(lf_delta_enabled=1, lf_delta_update=1, lf_ref_delta_present=15, lf_mode_delta_present=15,
                  lf_ref_delta=[2, 9, -14, 6], lf_mode_delta=[4, -12, -2, 11])
    frame, refs = case(208, 144, 3)
    (_, recon), (_, filtered) = surfaces(refs[0], 0), surfaces(refs[0], 0)
    out = np.zeros(60000, np.uint8)
    st, size, lv, (dec, cf, fl, lf) = encode(ctx, frame, refs, 60, level, auto_lf, recon, filtered, out, out.size,
                                             **deltas)
    assert st == abi.OK
    r, m = deltas["lf_ref_delta"], deltas["lf_mode_delta"]
    cfg = lambda lv, sh: abi.filter_config(  # noqa: E731
        lv, sh, delta_enabled=1, ref_delta_current=r[0], ref_delta_last=r[1], ref_delta_golden=r[2],
        ref_delta_altref=r[3], bpred_mode_delta=m[0], zero_mv_mode_delta=m[1], other_mv_mode_delta=m[2],
        split_mv_mode_delta=m[3])
    sh = 0
    if auto_lf:
        level, sh = vp8a.select_filter_params(ctx, recon, lf, cfg(0, 0), frame)
    assert lv == level > 0
    for got, want in zip(filtered, vp8a.filter_frame(ctx, recon, lf, cfg(level, sh))):
        assert np.array_equal(got, want)
    hdr = abi.frame_header(208, 144, abi.quant_indices(60), loop_filter_level=level, sharpness_level=sh, **deltas)
    assert out[:size].tobytes() == vp8a.write_inter_frame(hdr, dec, cf)
