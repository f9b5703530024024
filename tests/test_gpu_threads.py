"""One context per host thread: launches of pictures of different sizes, prepared
at the same time, do not disturb one another."""
import ctypes as C
import threading

import numpy as np
import pytest

import vp8a
from test_gpu_lf import lf_case
from vp8a import abi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def device_sweep(c, w, h, seed):
    """The picture, and a call that scores one level of it, every buffer on the
    device: the call returns as soon as its launches are made."""
    src, recon, m = lf_case(w, h, seed=seed)
    base = abi.filter_config(0, 0)
    keep = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in (*recon, *src)]
    dm = torch.from_numpy(m.view(np.uint8).reshape(-1).copy()).cuda()
    table = torch.zeros(512, dtype=torch.int64, device="cuda")
    pl, so = vp8a.planes(*keep[:3]), vp8a.source(*keep[3:])
    torch.cuda.synchronize()
    call = lambda: c._lib.vp8a_filter_sweep_window(c.handle, C.byref(pl), dm.data_ptr(), C.byref(base),  # noqa: E731
                                                   C.byref(so), 10, 10, table.data_ptr())
    return call, table, (src, recon, m, base, keep)


def test_threads_with_pictures_of_two_sizes(oracle):
    # Rows of slots of 33 KB (no special limit needed) and of 50 KB (above the 48
    # KB a kernel may use without one), by the same kernel.
    sizes, calls = [(1280, 448), (1280, 688), (1280, 448)], 2000
    wrong = [[] for _ in sizes]
    ctxs = [vp8a.Context(0) for _ in sizes]
    try:
        jobs = [device_sweep(c, w, h, seed=k) for k, (c, (w, h)) in enumerate(zip(ctxs, sizes))]
        start = threading.Barrier(len(sizes))

        def work(k):
            start.wait()
            for _ in range(calls):
                st = jobs[k][0]()
                if st != abi.OK:
                    wrong[k].append((st, ctxs[k]._lib.vp8a_last_error().decode()))

        for c in ctxs:
            c.force_sweep_layout(1, 256, 0)
        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for c in ctxs:
            c.synchronize()
        assert not any(wrong), [(len(x), x[:1]) for x in wrong]
        for _, table, (src, recon, m, base, _) in jobs:
            want = oracle.filter_sweep(recon, m, base, src, 0, threads=8)
            assert np.array_equal(table.cpu().numpy().view(np.uint64).reshape(64, 8)[10], want[10])
    finally:
        for c in ctxs:
            c.close()
