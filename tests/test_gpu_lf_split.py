"""The loop filter's passes split over the CTAs of a cluster, and the launches
that mix picture sizes: the filtered planes, the walk's choice and the tables
equal the oracle's at the edges of the bands (one row, a band and a row, more
rows than eight CTAs hold), with strides that allow only word or byte access,
and with pictures of fewer rows than the split has CTAs in one batch."""
import ctypes as C

import numpy as np
import pytest

import vp8a
from test_gpu_lf import lf_case
from vp8a import abi

pytestmark = pytest.mark.gpu

CONFIGS = {
    "normal": dict(level=33, sharpness=1),
    "key": dict(level=63, sharpness=0, key_frame=True),
    "simple": dict(level=45, sharpness=4, simple=True),
    "segments": dict(level=12, sharpness=3, segmentation_enabled=1, segment_abs=0, segment_lf_level=[-12, 20, 51, 0],
                     delta_enabled=1, ref_delta_golden=-7, split_mv_mode_delta=9),
}


@pytest.mark.parametrize("cfg", sorted(CONFIGS))
@pytest.mark.parametrize("size", [(16, 16), (48, 192), (40, 200), (21, 401), (333, 205), (64, 1552), (16, 8320)])
def test_filter_frame_bands(ctx, oracle, size, cfg):
    # 1, 12, 13, 26, 13, 97 and 520 MB rows.
    src, recon, m = lf_case(*size, seed=size[0] + size[1])
    c = abi.filter_config(**CONFIGS[cfg])
    for got, want in zip(vp8a.filter_frame(ctx, recon, m, c), oracle.filter_frame(recon, m, c)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("extra", [3, 4, 16])
def test_filter_frame_strides(ctx, oracle, extra):
    src, recon, m = lf_case(72, 220, seed=extra)
    wide = [np.pad(p, ((0, 0), (0, extra))) for p in recon]
    c = abi.filter_config(level=40, sharpness=2)
    planes = vp8a.planes(*[p[:, :q.shape[1]] for p, q in zip(wide, recon)])
    assert ctx._lib.vp8a_filter_frame(ctx.handle, C.byref(planes), m.ctypes.data, C.byref(c)) == abi.OK
    for got, want in zip(wide, oracle.filter_frame(recon, m, c)):
        assert np.array_equal(got[:, :want.shape[1]], want)
        assert not got[:, want.shape[1]:].any()


@pytest.mark.parametrize("size", [(16, 16), (33, 209), (210, 433), (500, 48)])
@pytest.mark.parametrize("sharp", [0, 5])
def test_walks(ctx, oracle, size, sharp):
    src, recon, m = lf_case(*size, seed=sharp + size[1])
    base = abi.filter_config(0, sharp)
    assert vp8a.select_filter_params(ctx, recon, m, base, src) == oracle.select_filter_params(recon, m, base, src,
                                                                                              threads=8)
    for every in (2, 5):
        got = vp8a.select_filter_params_sampled(ctx, recon, m, base, src, every, True)
        assert got == oracle.select_filter_params_sampled(recon, m, base, src, every, True, threads=8)


def test_batches_of_uneven_pictures(ctx, oracle):
    # One launch per shape; the split is common to the batch, so the one- and
    # two-row pictures leave most of their CTAs without rows.
    jobs = []
    for k, (size, simple) in enumerate([((320, 416), 0), ((96, 16), 0), ((17, 32), 1), ((208, 300), 1), ((1040, 72), 0),
                                        ((128, 700), 0)]):
        src, recon, m = lf_case(*size, seed=k)
        jobs.append((recon, m, abi.filter_config(0, k % 8, simple=bool(simple)), src))
    assert vp8a.select_filter_params_batch(ctx, jobs) == [
        oracle.select_filter_params(r, m, b, s, threads=8) for r, m, b, s in jobs]
    for got, (r, m, b, s) in zip(vp8a.filter_sweeps(ctx, [j + (0 if i % 2 else 3,) for i, j in enumerate(jobs)]), jobs):
        i = [j[0] is r for j in jobs].index(True)
        assert np.array_equal(got, oracle.filter_sweep(r, m, b, s, 0 if i % 2 else 3, threads=8))
