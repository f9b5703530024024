"""Analyses whose waits run out at the first poll or part of the way through, over
cluster sizes and uneven batches: each reports the timeout or finishes, its CTAs
leave only after their neighbours' messages, and the next analysis is exact."""
import numpy as np
import pytest

import vp8a
from vp8a import abi, synth

pytestmark = pytest.mark.gpu


def case(w, h, n_refs, seed):
    frames, _ = synth.make_sequence(w, h, 4, seed=seed, pieces=3, occluders=2)
    refs = [vp8a.pad_to_mb(*frames[k]) for k in (2, 0, 1)][:n_refs]
    return dict(frame=frames[3], refs=refs, ref_ids=[1, 2, 3][:n_refs], lam=vp8a.rd_lambda(44))


def same(got, want):
    return all(np.array_equal(got[f], want[f]) for f in got.dtype.names if f != "reserved")


def want_of(oracle, j):
    return oracle.analyse_inter_frame(j["frame"], j["refs"], j["ref_ids"], j["lam"], threads=8)


@pytest.mark.parametrize("n_refs", [1, 2, 3])
def test_single_frames(oracle, n_refs):
    job = case(336, 256, n_refs, seed=n_refs)
    want = want_of(oracle, job)
    with vp8a.Context(0) as c:
        for limit in (0, 0, 2, 40, 200, 1000):
            c.set_wait_limit(limit)
            try:
                assert same(vp8a.analyse_inter_frame(c, job["frame"], job["refs"], job["ref_ids"], job["lam"]), want)
            except vp8a.Vp8aError as e:
                assert e.status == abi.E_DEVICE_TIMEOUT
            else:
                assert limit
            c.set_wait_limit(1 << 24)
            assert same(vp8a.analyse_inter_frame(c, job["frame"], job["refs"], job["ref_ids"], job["lam"]), want)


def test_batches(oracle):
    jobs = [case(w, h, r, seed=w) for w, h, r in
            ((336, 256, 3), (16, 16, 3), (97, 50, 2), (640, 160, 2), (48, 300, 1), (176, 144, 1))]
    want = [want_of(oracle, j) for j in jobs]
    with vp8a.Context(0) as c:
        for limit in (0, 0, 5, 100):
            c.set_wait_limit(limit)
            try:
                vp8a.analyse_inter_frames(c, jobs)
            except vp8a.Vp8aError as e:
                assert e.status == abi.E_DEVICE_TIMEOUT
            else:
                assert limit
            c.set_wait_limit(1 << 24)
            assert all(same(g, w) for g, w in zip(vp8a.analyse_inter_frames(c, jobs), want))
