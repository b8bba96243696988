"""torch.nn modules over the engine (the caller layer, reference conv.py:305-340,446-481): constructor and
state_dict compatibility and argument checks on CPU; parity, the filter-transform cache, channels-last
zero-copy I/O and the fused epilogue on the GPU."""
import pytest
import torch

from oracle import winograd_oracle as wo
from pytorch_winoconv_b200 import conv as wconv


def test_constructor_and_state_dict_match_torch():
    ref = torch.nn.Conv2d(8, 12, 5, stride=1, padding=2, bias=True)
    m = wconv.Conv2d(8, 12, 5, stride=1, padding=2, bias=True)
    assert set(m.state_dict()) == set(ref.state_dict())
    m.load_state_dict(ref.state_dict())
    assert torch.equal(m.weight, ref.weight) and torch.equal(m.bias, ref.bias)
    m3 = wconv.Conv3d(4, 6, 3, padding=1, bias=False)
    assert m3.bias is None and tuple(m3.weight.shape) == (6, 4, 3, 3, 3)
    assert "compute_dtype" in repr(m)


def test_unsupported_arguments_raise():
    with pytest.raises(NotImplementedError):
        wconv.Conv2d(4, 4, 3, dilation=2)
    with pytest.raises(NotImplementedError):
        wconv.Conv2d(4, 4, 3, groups=2)
    with pytest.raises(NotImplementedError):
        wconv.Conv2d(4, 4, 3, padding=1, padding_mode="reflect")
    with pytest.raises(ValueError):
        wconv.Conv2d(4, 4, 3, activation="gelu")
    with pytest.raises(ValueError):
        wconv.Conv2d(4, 4, 3, pool=3)
    with pytest.raises(ValueError):
        wconv.Conv3d(4, 4, 3, pool=2)          # the epilogue pool is 2-D


def test_cpu_input_is_refused_loudly():
    m = wconv.Conv2d(4, 4, 3, padding=1).eval()
    with pytest.raises(RuntimeError, match="CUDA"):
        m(torch.zeros(1, 4, 8, 8))
    with pytest.raises(ValueError):
        m(torch.zeros(4, 8, 8))


@pytest.mark.gpu
@pytest.mark.parametrize("ks,stride,pad", [(3, 1, 1), (5, 1, 2), (7, 2, 3)])
def test_conv2d_module_parity(ks, stride, pad):
    torch.manual_seed(5)
    m = wconv.Conv2d(16, 24, ks, stride=stride, padding=pad, bias=True).cuda().eval()
    x = torch.randn(3, 16, 30, 28).half()
    y = m(x.cuda())
    o = wo.direct_conv_f64(x, m.weight.detach().cpu().half(), stride=stride, padding=pad) \
        + m.bias.detach().cpu().half().double().view(1, -1, 1, 1)
    assert y.dtype == torch.float16 and tuple(y.shape) == tuple(o.shape)
    assert wo.error_metrics(y.cpu().double(), o)["E_B"] < 2e-2          # the fp16 bound of the parity tests


@pytest.mark.gpu
def test_conv3d_module_parity_and_fp32():
    torch.manual_seed(6)
    m = wconv.Conv3d(8, 8, 3, padding=1, bias=False, compute_dtype=None).cuda().eval()
    x = torch.randn(1, 8, 6, 9, 10)
    y = m(x.cuda())                                                      # fp32 in -> fp32 path
    o = wo.direct_conv_f64(x, m.weight.detach().cpu(), padding=1)
    assert y.dtype == torch.float32
    assert wo.error_metrics(y.cpu().double(), o)["E_B"] < 1e-3


@pytest.mark.gpu
def test_channels_last_io_is_zero_copy_and_cache_follows_the_weight():
    torch.manual_seed(7)
    m = wconv.Conv2d(32, 32, 3, padding=1, bias=False, activation="relu", pool=2).cuda().half().eval()
    x = torch.randn(4, 32, 16, 16, device="cuda").half().contiguous(memory_format=torch.channels_last)
    y = m(x)
    assert y.is_contiguous(memory_format=torch.channels_last) and tuple(y.shape) == (4, 32, 8, 8)
    o = torch.nn.functional.max_pool2d(torch.relu(wo.direct_conv_f64(x.cpu(), m.weight.detach().cpu(), padding=1)), 2)
    assert wo.error_metrics(y.cpu().double(), o)["E_A"] < 5e-3
    assert list(m.planned_algorithms.values()) == ["row"]
    plan = next(iter(m._plans.values()))
    u_before = plan.u.clone()
    assert m(x).data_ptr() != 0 and next(iter(m._plans.values())) is plan      # second call: same plan, same U
    assert torch.equal(plan.u, u_before)
    with torch.no_grad():
        m.weight.mul_(2.0)                                                # in-place update bumps the version counter
    y2 = m(x)
    assert next(iter(m._plans.values())) is not plan                      # stale transforms were dropped
    assert wo.error_metrics(y2.cpu().double(), 2.0 * o)["E_A"] < 5e-3


def _grads_f64(x, w, b, gy, stride, pad, relu):
    """float64 torch.autograd.grad of F.conv2d / conv3d on the same rounded tensors."""
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    bd = None if b is None else b.double().requires_grad_(True)
    conv = torch.nn.functional.conv2d if w.dim() == 4 else torch.nn.functional.conv3d
    y = conv(xd, wd, bd, stride=stride, padding=pad)
    if relu:
        y = torch.relu(y)
    return torch.autograd.grad(y, [xd, wd] + ([bd] if bd is not None else []), gy.double())


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [
    # n, c, k, hw, kernel, stride, pad, relu
    (4, 32, 48, 20, 3, 1, 1, False),
    (2, 16, 24, 18, 5, 1, 2, True),
    (2, 8, 16, 23, 7, 2, 3, False),          # stride 2, and (23 + 6 - 7) % 2 == 0
    (2, 8, 16, 24, 3, 2, 1, False),          # stride 2 with an input row the forward never reads
])
def test_backward_matches_float64_autograd(shape):
    n, c, k, hw, ks, stride, pad, relu = shape
    torch.manual_seed(11)
    m = wconv.Conv2d(c, k, ks, stride=stride, padding=pad, bias=True, activation="relu" if relu else None).cuda()
    x = torch.randn(n, c, hw, hw).half()
    xg = x.cuda().requires_grad_(True)
    y = m(xg)
    gy = torch.randn(y.shape, generator=torch.Generator().manual_seed(12)).half()
    y.backward(gy.cuda())
    w16, b16 = m.weight.detach().cpu().half(), m.bias.detach().cpu().half()
    gx, gw, gb = _grads_f64(x, w16, b16, gy, stride, pad, relu)
    # the ReLU mask of the engine's fp16 output can differ from the float64 one where y is within rounding of zero
    tol = 2e-2 if not relu else 4e-2
    assert wo.error_metrics(xg.grad.cpu(), gx)["E_B"] < tol
    assert wo.error_metrics(m.weight.grad.cpu(), gw)["E_B"] < tol
    assert wo.error_metrics(m.bias.grad.cpu(), gb)["E_B"] < tol


@pytest.mark.gpu
def test_data_gradient_at_the_baseline_shapes():
    """grad_x of configs[1] (3x3, 256 -> 256 at 28 x 28) and configs[2]b (5x5, 128 -> 128 at 56 x 56) against float64."""
    for n, c, k, hw, ks, pad in [(32, 256, 256, 28, 3, 1), (8, 128, 128, 56, 5, 2)]:
        torch.manual_seed(13)
        m = wconv.Conv2d(c, k, ks, padding=pad, bias=False).cuda().eval()
        x = torch.randn(n, c, hw, hw).half()
        xg = x.cuda().requires_grad_(True)
        y = m(xg)
        gy = torch.randn(y.shape, generator=torch.Generator().manual_seed(14)).half()
        (gx,) = torch.autograd.grad(y, [xg], gy.cuda())
        ref = _grads_f64(x, m.weight.detach().cpu().half(), None, gy, 1, pad, False)[0]
        assert wo.error_metrics(gx.cpu(), ref)["E_B"] < 2e-2


@pytest.mark.gpu
def test_conv3d_backward_and_pool_refusal():
    torch.manual_seed(15)
    m = wconv.Conv3d(8, 8, 3, padding=1, bias=False).cuda()
    x = torch.randn(1, 8, 6, 9, 10).half()
    xg = x.cuda().requires_grad_(True)
    y = m(xg)
    gy = torch.randn(y.shape, generator=torch.Generator().manual_seed(16)).half()
    y.backward(gy.cuda())
    gx, gw = _grads_f64(x, m.weight.detach().cpu().half(), None, gy, 1, 1, False)
    assert wo.error_metrics(xg.grad.cpu(), gx)["E_B"] < 2e-2
    assert wo.error_metrics(m.weight.grad.cpu(), gw)["E_B"] < 2e-2
    mp = wconv.Conv2d(8, 8, 3, padding=1, pool=2).cuda()
    with pytest.raises(NotImplementedError):
        mp(torch.randn(1, 8, 8, 8, device="cuda"))                        # train mode: the fused pool has no gradient
    with torch.no_grad():
        assert tuple(mp(torch.randn(1, 8, 8, 8, device="cuda")).shape) == (1, 8, 4, 4)


def _by_torch(m, x, dtype=torch.float16):
    f = torch.nn.functional.conv2d if x.dim() == 4 else torch.nn.functional.conv3d
    b = None if m.bias is None else m.bias.detach().cpu().double()
    return f(x.cpu().to(dtype).double(), m.weight.detach().cpu().to(dtype).double(), b, m.stride, m.padding)


@pytest.mark.gpu
def test_inputs_and_gradients_that_do_not_start_on_16_bytes():
    from pytorch_winoconv_b200 import dwm
    torch.manual_seed(21)
    m = wconv.Conv2d(3, 16, 3, padding=1).cuda().eval()
    x = torch.randn(2 * 3 * 20 * 24 + 1, device="cuda").half()[1:].view(2, 3, 20, 24)      # few channels, read as they lie
    assert wo.error_metrics(m(x).detach().cpu().double(), _by_torch(m, x))["E_B"] < 2e-2
    w = torch.randn(8, 8, 3, 3, device="cuda") * 0.1
    xl = torch.randn(2 * 8 * 12 * 12 + 1, device="cuda")[1:].view(2, 12, 12, 8).permute(0, 3, 1, 2)
    ref = torch.nn.functional.conv2d(xl.cpu().double(), w.cpu().double(), None, 1, 1)
    assert wo.error_metrics(dwm.dwm2d(xl, w, padding=1).cpu(), ref)["E_B"] < 1e-3
    m = wconv.Conv2d(16, 16, 3, stride=2, padding=1).cuda().train()
    x = torch.randn(2, 16, 16, 16, device="cuda").half().to(memory_format=torch.channels_last).requires_grad_(True)
    gy = torch.randn(2 * 8 * 8 * 16 + 1, device="cuda").half()[1:].view(2, 8, 8, 16).permute(0, 3, 1, 2)
    m(x).backward(gy)
    got, got_w = x.grad.clone(), m.weight.grad.clone()
    x.grad = m.weight.grad = None
    m(x).backward(gy.clone(memory_format=torch.contiguous_format).contiguous(memory_format=torch.channels_last))
    assert torch.equal(got, x.grad) and torch.equal(got_w, m.weight.grad)


@pytest.mark.gpu
def test_a_weight_computed_anew_at_an_old_address_is_not_mistaken_for_it():
    torch.manual_seed(22)
    m = wconv.Conv2d(16, 16, 3, padding=1, bias=False).cuda().eval()
    x = torch.randn(1, 16, 10, 10, device="cuda").half()
    seen = set()
    for i in range(6):          # the allocator hands the freed weight's block to the next one
        w = torch.randn(16, 16, 3, 3, device="cuda") * 0.1
        m.weight = torch.nn.Parameter(w.clone())
        seen.add(m.weight.data_ptr())
        assert wo.error_metrics(m(x).detach().cpu().double(), _by_torch(m, x))["E_B"] < 2e-2
        del m.weight
        m.register_parameter("weight", None)
        del w
    assert len(seen) < 6


@pytest.mark.gpu
def test_inference_weights_and_wide_padding_are_refused_as_before():
    m = wconv.Conv2d(8, 8, 3, padding=1, bias=False).cuda().eval()
    with torch.inference_mode():
        m.weight = torch.nn.Parameter(torch.randn(8, 8, 3, 3, device="cuda"), requires_grad=False)
    with torch.no_grad(), pytest.raises(RuntimeError):
        m(torch.randn(1, 8, 6, 6, device="cuda").half())
    m = wconv.Conv2d(8, 8, 1, padding=1).cuda().train()
    y = m(torch.randn(1, 8, 6, 6, device="cuda").half().requires_grad_(True))
    with pytest.raises(NotImplementedError):
        y.sum().backward()


def test_a_tracer_sees_the_module_call():
    class Leaf(torch.fx.Tracer):
        def is_leaf_module(self, module, name):
            return isinstance(module, wconv.Conv2d)

    net = torch.nn.Sequential(wconv.Conv2d(8, 8, 3), torch.nn.ReLU())
    assert [n.op for n in Leaf().trace(net).nodes][1] == "call_module"


@pytest.mark.gpu
@pytest.mark.parametrize("k", [8, 72, 136])
def test_bias_gradient_is_an_fp32_sum(k):
    # chains of 8 in a tile, then of tiles and shares: a handful of roundings of 2**-24 on partial sums of the same size
    torch.manual_seed(23)
    m = wconv.Conv2d(16, k, 1).cuda().train()
    gy = torch.randn(16, k, 33, 35, device="cuda").half().to(memory_format=torch.channels_last)
    m(torch.randn(16, 16, 33, 35, device="cuda").half()).backward(gy)
    exact = gy.double().sum((0, 2, 3))
    assert float((m.bias.grad.double() - exact).norm() / exact.norm()) < 4e-7


_VIEWS = {      # what a network hands on: channels last in the order of the strides, but with gaps
    "crop": lambda b: b[:, :, 1:-1, 1:-1], "crop3d": lambda b: b[..., 2:, 1:-1], "channel slice": lambda b: b[:, 16:32],
    "chunk": lambda b: b.chunk(2, 1)[1], "space by two": lambda b: b[:, :, ::2, ::2], "batch by two": lambda b: b[::2],
}


def _gappy(nd, dtype, view, requires_grad=False):
    fmt = torch.channels_last if nd == 2 else torch.channels_last_3d
    base = torch.randn((4, 48, 13, 18) if nd == 2 else (4, 48, 6, 9, 12), device="cuda").to(dtype).to(memory_format=fmt)
    x = _VIEWS[view](base.requires_grad_(requires_grad))
    assert not x.is_contiguous() and not x.is_contiguous(memory_format=fmt)
    return base, x


def _rel(a, o):
    return float((a.detach().cpu().double() - o.detach()).norm() / o.detach().norm())


# one rounding of a result is half a unit of its last place, in the 2-norm too; fp32: sums of some hundred products
_ONE_ROUNDING = {torch.float16: 2.0 ** -11 * 1.02, torch.float32: 1e-5}


@pytest.mark.gpu
@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("view", _VIEWS)
def test_tensors_with_gaps_through_the_modules(nd, dtype, view):
    torch.manual_seed(31)
    base, x = _gappy(nd, dtype, view, requires_grad=True)
    layer = (wconv.Conv2d if nd == 2 else wconv.Conv3d)(x.shape[1], 24, 3, padding=1, bias=False, compute_dtype=None).cuda()
    with torch.no_grad():
        layer.weight.copy_(layer.weight.to(dtype))
        y = layer(x)
    f = torch.nn.functional.conv2d if nd == 2 else torch.nn.functional.conv3d
    bd = base.detach().cpu().double().requires_grad_(True)
    wd = layer.weight.detach().cpu().double().requires_grad_(True)
    o = f(_VIEWS[view](bd), wd, None, 1, 1)
    assert _rel(y, o) < _ONE_ROUNDING[dtype]
    gy = torch.randn_like(o).to(dtype)
    layer(x).backward(gy.cuda())
    o.backward(gy.double())
    assert _rel(base.grad, bd.grad) < _ONE_ROUNDING[dtype]
    # 16 bits: shares of the pixels, summed in fp32.  fp32: one chain of three products per 8 pixels, the accumulator cut off
    # after each, by 2**-23 of the running sum at most
    pixels = gy.numel() // gy.shape[1]
    assert _rel(layer.weight.grad, wd.grad) < (1e-5 if dtype == torch.float16 else 3 * (pixels / 8) * 2.0 ** -23)


@pytest.mark.gpu
@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("view", _VIEWS)
def test_gradients_with_gaps(nd, view):
    torch.manual_seed(32)
    _, gy = _gappy(nd, torch.float16, view)
    fmt = torch.channels_last if nd == 2 else torch.channels_last_3d
    x = torch.randn(gy.shape[0], 16, *gy.shape[2:], device="cuda").half().to(memory_format=fmt).requires_grad_(True)
    layer = (wconv.Conv2d if nd == 2 else wconv.Conv3d)(16, gy.shape[1], 3, padding=1).cuda()
    with torch.no_grad():
        layer.weight.copy_(layer.weight.half())
    layer(x).backward(gy)
    gx, gw, gb = _grads_f64(x.detach().cpu(), layer.weight.detach().cpu(), layer.bias.detach().cpu(), gy.cpu(), 1, 1, False)
    assert _rel(x.grad, gx) < _ONE_ROUNDING[torch.float16]
    assert _rel(layer.weight.grad, gw) < 1e-5 and _rel(layer.bias.grad, gb) < 1e-5


@pytest.mark.gpu
def test_gradients_behind_a_concatenation():
    torch.manual_seed(33)
    a, b = wconv.Conv2d(16, 8, 3, padding=1).cuda(), wconv.Conv2d(16, 24, 5, padding=2).cuda()
    x = torch.randn(2, 16, 11, 12, device="cuda").half().to(memory_format=torch.channels_last).requires_grad_(True)
    gy = torch.randn(2, 32, 11, 12, device="cuda").half().to(memory_format=torch.channels_last)
    torch.cat([a(x), b(x)], 1).backward(gy)
    xd = x.detach().cpu().double().requires_grad_(True)
    wd = [m.weight.detach().cpu().half().double().requires_grad_(True) for m in (a, b)]
    f = torch.nn.functional.conv2d
    torch.cat([f(xd, wd[0], None, 1, 1), f(xd, wd[1], None, 1, 2)], 1).backward(gy.cpu().double())
    # grad_x: two rounded results and their rounded sum
    assert _rel(x.grad, xd.grad) < 3 * _ONE_ROUNDING[torch.float16]
    assert _rel(a.weight.grad, wd[0].grad) < 1e-5 and _rel(b.weight.grad, wd[1].grad) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("view", _VIEWS)
def test_tensors_with_gaps_through_the_functional_operators(nd, view):
    from pytorch_winoconv_b200 import dwm, matrix_conv, matrix_conv3d
    torch.manual_seed(34)
    f = torch.nn.functional.conv2d if nd == 2 else torch.nn.functional.conv3d
    ops = matrix_conv if nd == 2 else matrix_conv3d
    for op, dtype in ((dwm.dwm2d if nd == 2 else dwm.dwm3d, torch.float32), (dwm.dwm2d if nd == 2 else dwm.dwm3d, torch.float16),
                      (ops.conv32, torch.float32), (ops.conv16, torch.float16)):
        _, x = _gappy(nd, dtype, view)
        w = (torch.randn(24, x.shape[1], *[3] * nd, device="cuda") * 0.1).to(dtype)
        y = op(x, w, padding=(1,) * nd)
        assert _rel(y, f(x.cpu().double(), w.cpu().double(), None, 1, 1)) < _ONE_ROUNDING[dtype], op


@pytest.mark.gpu
@pytest.mark.parametrize("new", [(8, 16, 3, 3), (72, 16, 3, 3), (24, 16, 5, 5), (24, 16, 1, 1), (40, 16, 2, 3)])
@pytest.mark.parametrize("bias", [False, True])
def test_a_weight_of_another_shape_gets_a_plan_of_its_own(new, bias):
    torch.manual_seed(35)
    m = wconv.Conv2d(16, 24, 3, padding=0, bias=bias).cuda()
    x = torch.randn(2, 16, 13, 14, device="cuda").half().to(memory_format=torch.channels_last)
    with torch.no_grad():
        m(x)
    m(x.clone().requires_grad_(True)).sum().backward()
    first = m.weight.detach().clone()
    for shape in (new, tuple(first.shape)):              # and back again
        m.weight = torch.nn.Parameter((torch.randn(shape, device="cuda") * 0.1).half().float())
        if bias:
            m.bias = torch.nn.Parameter(torch.randn(shape[0], device="cuda"))
        with torch.no_grad():
            y = m(x)
        o = _by_torch(m, x)
        assert y.shape == o.shape and _rel(y, o) < _ONE_ROUNDING[torch.float16]
        xg = x.clone().requires_grad_(True)
        gy = torch.randn(o.shape, device="cuda").half()
        m(xg).backward(gy)
        gx, gw, gb = (*_grads_f64(x.cpu(), m.weight.detach().cpu(), m.bias.detach().cpu() if bias else None, gy.cpu(), 1, 0, False), None)[:3]
        assert _rel(xg.grad, gx) < _ONE_ROUNDING[torch.float16] and _rel(m.weight.grad, gw) < 1e-5
        assert not bias or _rel(m.bias.grad, gb) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("length", [8, 48])
def test_a_bias_of_another_length_is_refused(length):
    m = wconv.Conv2d(16, 24, 3, padding=1).cuda().eval()
    x = torch.randn(1, 16, 8, 8, device="cuda").half()
    with torch.no_grad():
        m(x)
        m.bias = torch.nn.Parameter(torch.zeros(length, device="cuda"))
        with pytest.raises(ValueError, match="bias"):
            m(x)


@pytest.mark.gpu
@pytest.mark.parametrize("c,k", [(16, 24), (136, 136)])          # fp32: direct taps, and F(2,3) / F(4x4,3x3) with an output transform
def test_a_bias_that_starts_anywhere(c, k):
    from pytorch_winoconv_b200 import dwm, engine, matrix_conv
    torch.manual_seed(36)
    whole = torch.randn(3 * k + 3, device="cuda")                # the biases of three layers in one buffer
    f = torch.nn.functional
    w = torch.randn(k, c, 3, 3, device="cuda") * 0.1
    x = torch.randn(2, c, 12, 12, device="cuda")
    ref = f.conv2d(x.cpu().double(), w.cpu().double(), None, 1, 1)
    for start in (1, 2, 3):
        b = whole[start:start + k]
        o = ref + b.cpu().double().view(1, -1, 1, 1)
        for y in (dwm.dwm2d(x, w, b, padding=1), matrix_conv.conv32(x, w, b, padding=1), matrix_conv.conv32(x, w, b, padding=1, output_block=4)):
            assert _rel(y, o) < _ONE_ROUNDING[torch.float32]
        m = wconv.Conv2d(c, k, 3, padding=1, compute_dtype=None).cuda().eval()
        with torch.no_grad():
            m.weight.copy_(w)
            m.bias = torch.nn.Parameter(b)
            assert m.bias.data_ptr() == b.data_ptr()
            assert _rel(m(x), o) < _ONE_ROUNDING[torch.float32]
            m.compute_dtype = torch.float16                      # an fp32 bias read as it is
            assert _rel(m(x), f.conv2d(x.cpu().half().double(), w.cpu().half().double(), b.cpu().double(), 1, 1)) < _ONE_ROUNDING[torch.float16]
        x16, w16, b16 = x.half().permute(0, 2, 3, 1).contiguous(), w.half(), whole.half()[start:start + k]
        o16 = f.conv2d(x.cpu().half().double(), w16.cpu().double(), b16.cpu().double(), 1, 1)
        for tile_m in (0, 2, 4):
            y = engine.WinoConv(x16.shape, w16, padding=1, bias=b16, tile_m=tile_m)(x16)
            assert wo.error_metrics(y.permute(0, 3, 1, 2).cpu(), o16)["E_B"] < 2e-2


@pytest.mark.gpu
def test_threads_agree_on_what_the_gradients_cover():
    # every thread's first call of a layer whose data gradient is refused (padding beyond kernel - 1)
    import threading
    x = torch.randn(1, 8, 6, 6, device="cuda").half()
    names, n_threads = [], 8
    for _ in range(100):
        m = wconv.Conv2d(8, 8, 1, padding=1).cuda()
        start = threading.Barrier(n_threads)

        def call():
            start.wait()
            names.append(type(m(x).grad_fn).__name__)

        threads = [threading.Thread(target=call) for _ in range(n_threads)]
        [t.start() for t in threads]
        [t.join() for t in threads]
    assert len(names) == 100 * n_threads and set(names) == {"_WinoConvFnBackward"}, set(names)


def _layer_and_input(seed, c=32):
    torch.manual_seed(seed)
    m = wconv.Conv2d(c, c, 3, padding=1).cuda()
    with torch.no_grad():
        m.weight.copy_(m.weight.half())
    return m, torch.randn(2, c, 12, 12, device="cuda").half().to(memory_format=torch.channels_last)


def _warm():        # every kernel of _layer_and_input's calls loaded
    m, x = _layer_and_input(0)
    m(x.clone().requires_grad_(True)).backward(x)
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_a_second_stream_waits_for_the_transformed_filters():
    _warm()
    m, x = _layer_and_input(41)
    gy = torch.randn(x.shape, device="cuda").half().to(memory_format=torch.channels_last)
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    grads = {}
    with torch.cuda.stream(a):
        torch.cuda._sleep(40_000_000)                  # the transforms are queued behind tens of milliseconds
        xa = x.clone().requires_grad_(True)
        ya = m(xa)
        (grads["a"],) = torch.autograd.grad(ya, [xa], gy)
    with torch.cuda.stream(b):
        xb = x.clone().requires_grad_(True)
        yb = m(xb)
        (grads["b"],) = torch.autograd.grad(yb, [xb], gy)
    torch.cuda.synchronize()
    assert _rel(yb, _by_torch(m, x)) < _ONE_ROUNDING[torch.float16]
    assert torch.equal(ya, yb) and torch.equal(grads["a"], grads["b"])


@pytest.mark.gpu
def test_an_outgrown_filter_lives_until_other_streams_have_read_it():
    _warm()
    m, x = _layer_and_input(42)
    o = _by_torch(m, x)
    with torch.no_grad():
        m(x)
        torch.cuda.synchronize()
        old = next(iter(m._plans.values())).u
        address, size = old.data_ptr(), old.numel()
        del old
        m.__dict__["_views"].clear()
        b = torch.cuda.Stream()
        with torch.cuda.stream(b):
            torch.cuda._sleep(400_000_000)
            y = m(x)
        m.weight.zero_()
        m(x)                                           # a new filter takes the old one's place in the cache
        for _ in range(8):                             # whoever gets the old one's memory, gets it when b has read it
            t = torch.full((size,), 255, dtype=torch.uint8, device="cuda")
            assert t.data_ptr() != address or b.query()
        torch.cuda.synchronize()
    assert _rel(y, o) < _ONE_ROUNDING[torch.float16]


@pytest.mark.gpu
@pytest.mark.parametrize("warmed", ["not at all", "on another stream"])
def test_filters_and_graph_captures(warmed):
    _warm()
    m, x = _layer_and_input(43)
    with torch.no_grad():
        if warmed == "on another stream":
            m(x)
        g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(g, stream=s):
            y1, y2 = m(x), m(x)
        y = m(x)                                       # before the graph has run
        assert _rel(y, _by_torch(m, x)) < _ONE_ROUNDING[torch.float16]
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, y1) and torch.equal(y, y2)
        g2 = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g2, stream=s):
            y3 = m(x)
        g2.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, y3)


def test_a_patched_module_call_sees_calls_with_tensors(monkeypatch):
    seen = []
    monkeypatch.setattr(torch.nn.Module, "__call__", lambda self, *args: seen.append(self) or args[0])
    m = wconv.Conv2d(8, 8, 3)
    x = torch.zeros(1, 8, 4, 4)
    assert m(x) is x and seen == [m]
    monkeypatch.undo()
    with pytest.raises(RuntimeError, match="CUDA"):
        m(x)
    assert seen == [m]


@pytest.mark.gpu
def test_threads_that_have_made_no_cuda_call():
    import threading
    m, x = _layer_and_input(51)
    out = []
    with torch.no_grad():
        out.append(m(x))

        def call():
            with torch.no_grad():
                out.append(m(x))

        for _ in range(3):
            t = threading.Thread(target=call)
            t.start()
            t.join()
    assert len(out) == 4 and all(torch.equal(y, out[0]) for y in out)


@pytest.mark.gpu
def test_a_first_layer_trains_in_a_process_of_its_own():
    # no data gradient and nothing to convert: the weight gradient is the first thing autograd's thread does
    import subprocess
    import sys
    code = """
import torch
from pytorch_winoconv_b200 import conv
m = conv.Conv2d(16, 24, 3, padding=1).cuda()
x = torch.randn(2, 16, 19, 21, device="cuda").half().to(memory_format=torch.channels_last)
y = m(x)
gy = torch.randn(y.shape, device="cuda").half().to(memory_format=torch.channels_last)
y.backward(gy)
o = torch.nn.grad.conv2d_weight(x.cpu().double(), m.weight.shape, gy.cpu().double(), 1, 1)
assert float((m.weight.grad.cpu().double() - o).norm() / o.norm()) < 1e-5
"""
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.gpu
def test_a_captured_training_step_follows_its_weights():
    _warm()
    m, x = _layer_and_input(61)
    n = wconv.Conv2d(32, 32, 3, padding=1).cuda()
    n.load_state_dict(m.state_dict())
    graphed = torch.cuda.make_graphed_callables(n, (x.detach().clone().requires_grad_(True),))
    for _ in range(3):
        a, b = (x.detach().clone().requires_grad_(True) for _ in range(2))
        m.zero_grad()
        n.zero_grad()
        ya, yb = m(a), graphed(b)
        ya.backward(x)
        yb.backward(x)
        assert torch.equal(ya, yb) and torch.equal(a.grad, b.grad)
        for p, q in zip(m.parameters(), n.parameters()):
            assert torch.equal(p.grad, q.grad)
            with torch.no_grad():
                p.sub_(p.grad * 1e-3)
                q.sub_(q.grad * 1e-3)
    with torch.no_grad():
        assert torch.equal(m(x), n(x))


@pytest.mark.gpu
def test_a_graph_keeps_the_filters_it_was_captured_with():
    _warm()
    m, x = _layer_and_input(62)
    with torch.no_grad():
        m(x)
        torch.cuda.synchronize()
        size = next(iter(m._plans.values())).u.numel()
        m.__dict__["_views"].clear()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = m(x)
        g.replay()
        torch.cuda.synchronize()
        before = y.clone()
        m.weight.mul_(2.0)
        m.bias.add_(1.0)
        z = m(x)                                       # new filters: the old ones are the graph's alone
        spoil = [torch.full((size,), 255, dtype=torch.uint8, device="cuda") for _ in range(8)]
        g.replay()
        torch.cuda.synchronize()
        o = torch.nn.functional.conv2d(x.cpu().double(), m.weight.cpu().double() / 2, None, 1, 1)
        b = m.bias.cpu().double().view(1, -1, 1, 1) - 1        # an fp32 bias is read as it lies, in the graph too
        assert _rel(before, o + b) < _ONE_ROUNDING[torch.float16]
        assert _rel(y, o + b + 1) < _ONE_ROUNDING[torch.float16]
        assert _rel(z, _by_torch(m, x)) < _ONE_ROUNDING[torch.float16]
        del spoil
