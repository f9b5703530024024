"""The whole-frame call of encode_p_frame gives what its stages give one by one:
bytes, planes, decisions, coefficients and levels, over sizes, row strides,
reference counts, partition counts and loop-filter settings."""
import numpy as np
import pytest

import vp8a
from vp8a import api, synth

pytestmark = pytest.mark.gpu


def wide(plane, pad):
    """The same pixels in rows `pad` bytes longer."""
    buf = np.full((plane.shape[0], plane.shape[1] + pad), 0x5a, np.uint8)
    buf[:, :plane.shape[1]] = plane
    return buf[:, :plane.shape[1]]


@pytest.mark.parametrize("w,h,n_refs,pad,kw", [
    (16, 16, 1, 0, {}),
    (49, 35, 2, 0, dict(n_partitions=2)),
    (176, 144, 3, 0, dict(n_partitions=8)),
    (97, 80, 3, 5, dict(sharpness_level=5)),
    (160, 48, 2, 16, dict(auto_lf=False, loop_filter_level=0)),
    (80, 64, 3, 3, dict(auto_lf=False, loop_filter_level=24, sharpness_level=3, simple=True)),
    (64, 64, 1, 0, dict(simple=True, refresh_last=False)),
])
@pytest.mark.parametrize("qi", [4, 60, 127])
def test_whole_frame_equals_its_stages(ctx, monkeypatch, w, h, n_refs, pad, kw, qi):
    frames, _ = synth.make_sequence(w, h, 5, seed=w + h, pieces=3, occluders=2)
    refs = [vp8a.pad_to_mb(*frames[k]) for k in (2, 0, 4)][:n_refs]
    if pad:
        frames[3] = tuple(wide(p, pad) for p in frames[3])
        refs = [tuple(wide(p, pad) for p in r) for r in refs]
    args = (frames[3], refs, [1, 2, 3][:n_refs], qi)
    assert api._host_frame(frames[3], refs, [1, 2, 3][:n_refs], qi, 0, 0, 1)
    before = [p.copy() for r in refs for p in r]
    bits, out, d = vp8a.encode_p_frame(ctx, *args, **kw)
    assert all(np.array_equal(a, b) for a, b in zip(before, (p for r in refs for p in r)))
    monkeypatch.setattr(api, "_host_frame", lambda *a: False)
    bits2, out2, d2 = vp8a.encode_p_frame(ctx, *args, **kw)
    assert bits == bits2 and (d["level"], d["sharpness"]) == (d2["level"], d2["sharpness"])
    assert all(np.array_equal(a, b) for a, b in zip((*out, *d["recon"]), (*out2, *d2["recon"])))
    for k in ("coeffs", "flags"):
        assert np.array_equal(d[k], d2[k]), k
    for k in ("decisions", "lf_info"):
        assert all(np.array_equal(d[k][f], d2[k][f]) for f in d[k].dtype.names if f != "reserved"), k


def test_whole_frame_refuses_as_its_stages_do(ctx):
    frames, _ = synth.make_sequence(64, 48, 2, seed=1)
    ref = vp8a.pad_to_mb(*frames[0])
    small = vp8a.pad_to_mb(*synth.make_sequence(32, 32, 1, seed=2)[0][0])
    with pytest.raises(vp8a.Vp8aError, match="ReferenceDimensionsMismatch"):
        vp8a.encode_p_frame(ctx, frames[1], [small], [1], 30)
    with pytest.raises(vp8a.Vp8aError, match="InvalidArgument"):
        vp8a.encode_p_frame(ctx, frames[1], [ref], [7], 30)
    with pytest.raises(vp8a.Vp8aError, match="LoopFilterLevelOutOfRange|InvalidArgument"):
        vp8a.encode_p_frame(ctx, frames[1], [ref], [1], 30, loop_filter_level=64, auto_lf=False)
