"""The waits between the CTAs of a split loop-filter pass, made to run out.

With a poll budget of 0 the first poll that finds a neighbour's rows not yet there
gives up; a split picture meets that many times over. The pass runs to its end
without its neighbours, waits for the messages that are still on their way to it,
and the call (or, for device buffers, the next synchronize) returns
VP8A_E_DEVICE_TIMEOUT. The context must give exact results once the budget is
back."""
import ctypes as C

import numpy as np
import pytest

import vp8a
from test_gpu_lf import lf_case
from vp8a import abi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LIMIT = 1 << 24
SIZES = [(640, 368), (1280, 720), (96, 1040)]  # two, four and eight bands


@pytest.fixture()
def fresh():
    with vp8a.Context(0) as c:
        yield c


def runs_out(call):
    with pytest.raises(vp8a.Vp8aError, match="DeviceTimeout") as ei:
        call()
    assert ei.value.status == abi.E_DEVICE_TIMEOUT


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("simple", [False, True])
def test_filter_frame(fresh, oracle, size, simple):
    src, recon, m = lf_case(*size, seed=size[0])
    cfg = abi.filter_config(30, 2, simple=simple)
    for _ in range(3):
        fresh.set_wait_limit(0)
        runs_out(lambda: vp8a.filter_frame(fresh, recon, m, cfg))
        fresh.synchronize()  # the status was read and cleared
        fresh.set_wait_limit(LIMIT)
        for got, want in zip(vp8a.filter_frame(fresh, recon, m, cfg), oracle.filter_frame(recon, m, cfg)):
            assert np.array_equal(got, want)


def test_device_planes_report_at_synchronize(fresh, oracle):
    src, recon, m = lf_case(1280, 720, seed=4)
    cfg = abi.filter_config(40, 1)
    want = oracle.filter_frame(recon, m, cfg)
    dm = torch.from_numpy(m.view(np.uint8).reshape(-1).copy()).cuda()
    for limit, status in ((0, abi.E_DEVICE_TIMEOUT), (LIMIT, abi.OK)) * 2:
        d = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in recon]
        torch.cuda.synchronize()
        fresh.set_wait_limit(limit)
        pl = vp8a.planes(*d)
        assert fresh._lib.vp8a_filter_frame(fresh.handle, C.byref(pl), dm.data_ptr(), C.byref(cfg)) == abi.OK
        assert fresh._lib.vp8a_ctx_synchronize(fresh.handle) == status
    assert all(np.array_equal(p.cpu().numpy(), q) for p, q in zip(d, want))


@pytest.mark.parametrize("size", SIZES)
def test_walks(fresh, oracle, size):
    src, recon, m = lf_case(*size, seed=size[1])
    base = abi.filter_config(0, 3)
    for _ in range(2):
        fresh.set_wait_limit(0)
        runs_out(lambda: vp8a.select_filter_params(fresh, recon, m, base, src))
        fresh.set_wait_limit(LIMIT)
        assert vp8a.select_filter_params(fresh, recon, m, base, src) == oracle.select_filter_params(
            recon, m, base, src, threads=8)


def test_batched_walk(fresh, oracle):
    jobs = []
    for k, size in enumerate([(1280, 720), (320, 240), (33, 700)]):
        src, recon, m = lf_case(*size, seed=k)
        jobs.append((recon, m, abi.filter_config(0, k), src))
    want = [oracle.select_filter_params(r, m, b, s, threads=8) for r, m, b, s in jobs]
    for _ in range(2):
        fresh.set_wait_limit(0)
        runs_out(lambda: vp8a.select_filter_params_batch(fresh, jobs))
        fresh.set_wait_limit(LIMIT)
        assert vp8a.select_filter_params_batch(fresh, jobs) == want


def test_passes_that_are_not_split_do_not_wait(fresh, oracle):
    src, recon, m = lf_case(176, 144, seed=6)
    cfg = abi.filter_config(25, 0)
    fresh.set_wait_limit(0)
    for got, want in zip(vp8a.filter_frame(fresh, recon, m, cfg), oracle.filter_frame(recon, m, cfg)):
        assert np.array_equal(got, want)


def test_whole_frame_encode(fresh):
    # The analysis gives up first: the outputs keep what they held.
    from test_gpu_encode_outputs import FILL, case, encode, surfaces

    frame, refs = case(320, 240, 2)
    out = np.full(9000, FILL, np.uint8)
    (_, recon), (_, filtered) = surfaces(refs[0], 0), surfaces(refs[0], 0)
    fresh.set_wait_limit(0)
    assert encode(fresh, frame, refs, 40, 20, False, recon, filtered, out, out.size)[0] == abi.E_DEVICE_TIMEOUT
    assert all((p == FILL).all() for p in (*recon, *filtered, out))
    fresh.set_wait_limit(LIMIT)
    bits, want, d = vp8a.encode_p_frame(fresh, frame, refs, [1, 2], 40)
    assert encode(fresh, frame, refs, 40, 0, True, recon, filtered, out, out.size)[0] in (abi.OK, abi.E_INVALID_ARGUMENT)
    assert all(np.array_equal(p, q) for p, q in zip(recon, d["recon"]))
