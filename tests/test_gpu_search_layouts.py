"""Parity of the motion searches where their load paths and search fields
split: planes and sources at any byte alignment and row stride, blocks next to
every edge of the plane, and walks of up to eight positions in any direction
(past the edge of the field of SADs around the predictor)."""
import numpy as np
import pytest
from util import extract_mbs, sr_tuples

import vp8a
from vp8a import synth

pytestmark = pytest.mark.gpu


def placed(plane, offset, pad):
    """A view of the same pixels `offset` bytes into a buffer whose rows are
    `pad` bytes longer than the plane's."""
    h, w = plane.shape
    buf = np.full(offset + h * (w + pad), 0xa5, np.uint8)
    view = np.lib.stride_tricks.as_strided(buf[offset:], (h, w), (w + pad, 1))
    view[:] = plane
    return view


def ramp(w, h, dx, dy, seed):
    """A smooth texture, `dx`, `dy` pixels on: SADs fall towards the true
    vector from far away, so walks are long."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w].astype(np.float64)
    x, y = x + dx, y + dy
    v = 128 + 60 * np.sin(x / 9.7 + 0.3 * np.cos(y / 17.0)) * np.cos(y / 8.3) + 20 * np.sin((x + y) / 31.0)
    return np.clip(v + rng.normal(0, 1.0, v.shape), 0, 255).astype(np.uint8)


@pytest.mark.parametrize("w,h", [(16, 16), (80, 16), (16, 80), (49, 65), (128, 96)])
@pytest.mark.parametrize("n_refs,offset,pad", [(1, 0, 0), (3, 1, 3), (2, 4, 4)])
def test_analysis_long_walks_any_layout(ctx, oracle, w, h, n_refs, offset, pad):
    shifts = [(6.25, -5.5), (-7.0, 0.0), (4.5, 7.75)][:n_refs]
    grey = lambda hh, ww: np.full((hh, ww), 128, np.uint8)  # noqa: E731
    uw, uh = (w + 1) // 2, (h + 1) // 2
    frame = [ramp(w, h, 0, 0, 1), grey(uh, uw), grey(uh, uw)]
    refs = [vp8a.pad_to_mb(ramp(w, h, dx, dy, 2 + i), grey(uh, uw), grey(uh, uw)) for i, (dx, dy) in enumerate(shifts)]
    ids = [1, 2, 3][:n_refs]
    lam = vp8a.rd_lambda(30)
    want, wtr = oracle.analyse_inter_frame(frame, refs, ids, lam, trace=True)
    got, gtr = vp8a.analyse_inter_frame(ctx, [placed(p, offset, pad) for p in frame],
                                        [[placed(p, offset, pad) for p in r] for r in refs], ids, lam, trace=True)
    assert np.array_equal(gtr, wtr)
    for f in ("ref_frame", "mode", "partition", "mv", "j", "total", "split_mvs", "submv_modes"):
        assert np.array_equal(got[f], want[f]), f


@pytest.mark.parametrize("w,h", [(16, 16), (33, 17), (64, 48)])
@pytest.mark.parametrize("offset,pad", [(0, 0), (3, 1), (4, 4)])
def test_searches_any_layout(ctx, oracle, w, h, offset, pad):
    ref = vp8a.pad_to_mb(*synth.make_sequence(w, h, 1, seed=w + h)[0][0])[0]
    plane = placed(ref, offset, pad)
    rows, cols = ref.shape[0] // 16, ref.shape[1] // 16
    rng = np.random.default_rng(w * 7 + offset)
    src = rng.integers(0, 256, ref.shape).astype(np.uint8)
    mbs, xy = extract_mbs((ref // 2 + src // 2).astype(np.uint8), rows, cols)
    n = len(mbs)
    for trial in range(4):
        # Vectors up to 24 px: blocks across and beyond each edge.
        mv = rng.integers(-96, 97, (n, 2)).astype(np.int16)
        even = (mv // 2 * 2).astype(np.int16)
        whole = (mv // 4 * 4).astype(np.int16)
        for name, arg in (("half_pixel_refine_luma", whole), ("quarter_pixel_refine_luma", even)):
            assert sr_tuples(getattr(vp8a, name)(ctx, plane, mbs, xy, arg)) == sr_tuples(
                getattr(oracle, name)(ref, mbs, xy, arg)), (name, trial)
        assert sr_tuples(vp8a.small_diamond_search_luma(ctx, plane, mbs, xy, mv, 8)) == sr_tuples(
            oracle.small_diamond_search_luma(ref, mbs, xy, mv, 8)), trial


@pytest.mark.parametrize("effort", [0, 2, 3])
@pytest.mark.parametrize("w,h,offset,pad", [(16, 16, 0, 0), (97, 80, 0, 0), (97, 80, 3, 1), (160, 48, 4, 4)])
def test_rd_search_long_descents_any_layout(ctx, oracle, effort, w, h, offset, pad):
    # Neighbours far from the true vector (up to 40 px) and descents of up to 32
    # rounds: more than the staged window covers, also across the plane's edges.
    uw, uh = (w + 1) // 2, (h + 1) // 2
    grey = np.full((uh, uw), 128, np.uint8)
    frame = [ramp(w, h, 0, 0, 1), grey, grey]
    refs = [vp8a.pad_to_mb(ramp(w, h, dx, dy, 2 + i), grey, grey) for i, (dx, dy) in enumerate([(13.5, -9.25), (0, 17)])]
    lam = vp8a.rd_lambda(12)
    nb = oracle.neighbours_from_decisions(oracle.analyse_inter_frame(frame, refs, [1, 2], lam))
    rng = np.random.default_rng(w + effort)
    for mv in (nb["mv"], nb["split_mvs"]) if "split_mvs" in nb.dtype.names else (nb["mv"],):
        for f in ("row", "col"):
            mv[f] = rng.integers(-160, 161, mv[f].shape)
    want = oracle.rd_inter_search(frame, refs, [1, 2], lam, 8, effort, nb)
    got = vp8a.rd_inter_search(ctx, [placed(p, offset, pad) for p in frame],
                               [[placed(p, offset, pad) for p in r] for r in refs], [1, 2], lam, 8, effort, nb)
    for f in ("ref_frame", "mode", "n_searched", "leader", "mv", "sad", "cost", "bits", "found"):
        assert np.array_equal(got[f], want[f]), f
