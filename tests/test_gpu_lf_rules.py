"""Which loop-filter launches are split over clusters, by the launch shape they
report: a grid of candidates over a tall, narrow picture is not (a split pass's CTAs
stay for all its steps, few of which have work for each), its frame filter is; wide
pictures as before. The results are the oracle's either way."""
import numpy as np
import pytest

import vp8a
from test_gpu_lf import lf_case
from vp8a import abi

pytestmark = pytest.mark.gpu


def split(ctx):
    return ctx.last_sweep_layout()[2] == 1  # a split pass fetches ahead, an unforced whole one does not


@pytest.mark.parametrize("w,h,of_grid,of_frame", [
    (32, 2048, False, True),
    (128, 4096, False, True),
    (80, 1200, False, True),
    (640, 368, False, True),
    (1280, 720, False, True),
    (176, 144, False, False),
    (2048, 32, False, False),
])
def test_rule(ctx, oracle, w, h, of_grid, of_frame):
    src, recon, m = lf_case(w, h, seed=w)
    base = abi.filter_config(0, 0)
    got = vp8a.filter_sweep(ctx, recon, m, base, src)
    assert split(ctx) == of_grid
    if w * h <= 100000:
        assert np.array_equal(got, oracle.filter_sweep(recon, m, base, src, 0, threads=8))
    cfg = abi.filter_config(30, 1)
    out = vp8a.filter_frame(ctx, recon, m, cfg)
    assert split(ctx) == of_frame
    assert all(np.array_equal(a, b) for a, b in zip(out, oracle.filter_frame(recon, m, cfg)))
