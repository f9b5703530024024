"""The training layers against 64-bit convolutions, for aligned tensors (the
persistent tensor-core kernels) and for tensors off the 16-byte boundary (the
element-wise ones), over image counts below, at and beyond the number of SMs."""
import pytest

from vp8a import abi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def shifted(t, elements):
    """The same values `elements` elements into a new buffer."""
    buf = torch.zeros(t.numel() + elements + 8, dtype=t.dtype, device=t.device)
    out = buf[elements:elements + t.numel()].view(t.shape)
    out.copy_(t)
    return out


def conv64(x, w, b):
    """[n, 32, 32, cin], [cout, 9, cin] -> [n, 32, 32, cout], in 64 bits."""
    k = w.double().reshape(w.shape[0], 3, 3, w.shape[2]).permute(0, 3, 1, 2)
    y = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), k, None if b is None else b.double(), padding=1)
    return y.permute(0, 2, 3, 1)


def grads64(x, w, dy):
    x, w = x.double().requires_grad_(), w.double().requires_grad_()
    conv64(x, w, None).backward(dy.double())
    return x.grad, w.grad, dy.double().sum((0, 1, 2))


# FP32 sums of exact BF16 products, at most 1024 of them in a row: 1024 roundings
# of 2^-23 of the sum of magnitudes; a BF16 result adds half of its last place.
SUM = 2.0 ** -13
HALF = 2.0 ** -8


@pytest.mark.parametrize("n", [1, 5, 149, 301])
@pytest.mark.parametrize("cin,cout", [(2, 32), (32, 32), (32, 1)])
@pytest.mark.parametrize("offset", [0, 2])
def test_layers_match_64_bit_convolutions(ctx, n, cin, cout, offset):
    g = torch.Generator(device="cuda").manual_seed(n * 64 + cin + cout)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    x = rnd(n, 32, 32, cin)
    if cin == 32:
        x = x.relu()
    x, w = x.bfloat16(), (rnd(cout, 9, cin) * 0.2).bfloat16()
    b, dy = rnd(cout) * 0.1, (rnd(n, 32, 32, cout) * 0.05).bfloat16()
    xs, dys = shifted(x, offset), shifted(dy, offset)
    lib, last = ctx._lib, cout == 1
    tensor_core = cin == 32 and cout == 32
    y = torch.full((n, 32, 32, cout), float("nan"), dtype=torch.float32 if last else torch.bfloat16, device="cuda")
    yo = y if tensor_core else shifted(y, offset)
    gx = shifted(torch.full((n, 32, 32, cin), float("nan"), dtype=torch.bfloat16, device="cuda"), offset)
    gw, gb = torch.zeros(cout * 9 * cin, device="cuda"), torch.zeros(cout, device="cuda")
    torch.cuda.synchronize()
    fx = x if tensor_core else xs  # a 32 -> 32 forward takes aligned buffers only
    assert lib.vp8a_lp_conv_forward(ctx.handle, fx.data_ptr(), cin, w.data_ptr(), b.data_ptr(), cout, n, int(not last),
                                    None if last else yo.data_ptr(), yo.data_ptr() if last else None) == abi.OK
    for _ in range(2):  # gradients are added to what is there
        assert lib.vp8a_lp_conv_backward(ctx.handle, xs.data_ptr(), cin, w.data_ptr(), cout, n, dys.data_ptr(),
                                         int(cin == 32), gx.data_ptr(), gw.data_ptr(), gb.data_ptr()) == abi.OK
    ctx.synchronize()
    want, size = conv64(x, w, b), conv64(x.abs(), w.abs(), b.abs())
    got = yo.double()
    if not last:
        want = want.relu()
    assert bool(((got - want).abs() <= SUM * size + (0 if last else HALF) * want.abs()).all())
    dx, dw, db = grads64(x, w, dy)
    sx, sw, sb = grads64(x.abs(), w.abs(), dy.abs())
    if cin == 32:
        assert bool((gx[x == 0] == 0).all())
        dx = dx * (x > 0)
    assert bool(((gx.double() - dx).abs() <= SUM * sx + HALF * dx.abs()).all())
    assert bool(((gw.double().view(dw.shape) - 2 * dw).abs() <= 2 * SUM * sw).all())
    assert bool(((gb.double() - 2 * db).abs() <= 2 * SUM * sb).all())


@pytest.mark.parametrize("n", [1, 3, 8])
@pytest.mark.parametrize("cin,cout", [(2, 32), (32, 32), (32, 1)])
def test_both_routes_round_alike(ctx, n, cin, cout):
    # Up to 8 images are one FP32 chain: aligned and unaligned tensors then give
    # the same bits (but for dW and db of the last layer, whose chain runs over the
    # other tensor's pixels).
    g = torch.Generator(device="cuda").manual_seed(n + cin)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    x, w = rnd(n, 32, 32, cin).bfloat16(), (rnd(cout, 9, cin) * 0.2).bfloat16()
    b, dy, lib, last = rnd(cout), (rnd(n, 32, 32, cout) * 0.05).bfloat16(), ctx._lib, cout == 1
    got = []
    for offset in (0, 2):
        xs, dys = shifted(x, offset), shifted(dy, offset)
        y = shifted(torch.zeros((n, 32, 32, cout), dtype=torch.float32 if last else torch.bfloat16, device="cuda"), offset)
        gx, gw, gb = shifted(torch.zeros_like(x), offset), torch.zeros(cout * 9 * cin, device="cuda"), torch.zeros(
            cout, device="cuda")
        torch.cuda.synchronize()
        if cin != 32 or last:
            assert lib.vp8a_lp_conv_forward(ctx.handle, xs.data_ptr(), cin, w.data_ptr(), b.data_ptr(), cout, n, 1,
                                            None if last else y.data_ptr(), y.data_ptr() if last else None) == abi.OK
        assert lib.vp8a_lp_conv_backward(ctx.handle, xs.data_ptr(), cin, w.data_ptr(), cout, n, dys.data_ptr(), 1,
                                         gx.data_ptr(), gw.data_ptr(), gb.data_ptr()) == abi.OK
        ctx.synchronize()
        got.append((y, *(() if cin == 2 else (gx,)), *(() if last else (gw, gb))))
    assert all(torch.equal(p, q) for p, q in zip(*got))
