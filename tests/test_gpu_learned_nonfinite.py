"""Infinities and NaN in the training layers: aligned tensors (the persistent
kernels) and tensors off the 16-byte boundary (the element-wise ones) give them in
the same places."""
import pytest

from test_gpu_learned_layers import SUM, shifted
from vp8a import abi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PLACES = {"corner": (0, 0), "right": (13, 31), "left": (16, 0), "bottom": (31, 9), "middle": (8, 20)}


def run(ctx, x, w, b, dy, cin, cout, offset):
    n, lib, last = x.shape[0], ctx._lib, cout == 1
    xs, dys = shifted(x, offset), shifted(dy, offset)
    y = shifted(torch.zeros((n, 32, 32, cout), dtype=torch.float32 if last else torch.bfloat16, device="cuda"), offset)
    gx = shifted(torch.zeros_like(x), offset)
    gw, gb = torch.zeros(cout * 9 * cin, device="cuda"), torch.zeros(cout, device="cuda")
    torch.cuda.synchronize()
    if cin != 32 or last:  # a 32 -> 32 forward takes aligned buffers only
        assert lib.vp8a_lp_conv_forward(ctx.handle, xs.data_ptr(), cin, w.data_ptr(), b.data_ptr(), cout, n, 0,
                                        None if last else y.data_ptr(), y.data_ptr() if last else None) == abi.OK
    assert lib.vp8a_lp_conv_backward(ctx.handle, xs.data_ptr(), cin, w.data_ptr(), cout, n, dys.data_ptr(), 1,
                                     gx.data_ptr(), gw.data_ptr(), gb.data_ptr()) == abi.OK
    ctx.synchronize()
    return {"y": y, "gx": gx, "gw": gw, "gb": gb}


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where", sorted(PLACES))
@pytest.mark.parametrize("tensor", ["x", "dy", "w"])
@pytest.mark.parametrize("cin,cout", [(2, 32), (32, 32), (32, 1)])
def test_both_routes_agree(ctx, cin, cout, tensor, where, value):
    n = 10  # two groups of half images
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    t = {"x": rnd(n, 32, 32, cin).bfloat16(), "w": (rnd(cout, 9, cin) * 0.2).bfloat16(),
         "dy": (rnd(n, 32, 32, cout) * 0.05).bfloat16()}
    b = rnd(cout)
    r, c = PLACES[where]
    if tensor == "w":
        t["w"][cout // 2, r % 9, cin // 2] = value
    else:
        t[tensor][n - 1, r, c, t[tensor].shape[3] // 2] = value
    got, want = (run(ctx, t["x"], t["w"], b, t["dy"], cin, cout, o) for o in (0, 2))
    for k in got:
        p, q = got[k].double().reshape(-1), want[k].double().reshape(-1)
        assert torch.equal(p.isnan(), q.isnan()), k
        assert torch.equal(p.isinf(), q.isinf()), k
        assert torch.equal(p[p.isinf()], q[q.isinf()]), k
        ok = p.isfinite()
        # Sums of at most 10 x 1024 products of magnitudes below 6 and 0.3 (dW, db),
        # a BF16 result within a place of the other.
        bound = 2 * SUM * (n * 1024 * 6 * 0.3) if k in ("gw", "gb") else 2.0 ** -7 * q[ok].abs() + 2 * SUM * 64
        assert bool(((p[ok] - q[ok]).abs() <= bound).all()), k
