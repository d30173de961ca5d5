"""The projection's weight gradient and the native layer, against float64 and `deconv_update`."""

import pytest
import torch

import deconver_b200 as dcb
from deconver_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tf32,tol", [(torch.float32, 1, 2e-3), (torch.float32, 0, 1e-5),
                                            (torch.bfloat16, 0, 6e-3)], ids=["tf32", "f32", "bf16"])
@pytest.mark.parametrize("batch,co,ci,n", [
    (1, 1, 1, 1), (2, 4, 1, 3), (1, 128, 64, 512), (2, 129, 65, 1023), (3, 64, 16, 514),
    (2, 200, 48, 4097), (1, 2048, 512, 256), (1, 16, 130, 40000),
])
def test_weight_gradient(dtype, tf32, tol, batch, co, ci, n):
    lib, dev = _lib.load(), torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(co + n)
    gy = torch.randn(batch, co, n, device=dev, generator=gen).to(dtype)
    x = torch.randn(batch, ci, n, device=dev, generator=gen).to(dtype)
    gw = torch.empty(co, ci, device=dev, dtype=dtype)
    nbytes = lib.ndc_proj_wgrad_workspace_bytes(batch, co, ci, n)
    ws = torch.empty(nbytes, device=dev, dtype=torch.uint8)
    args = (batch, co, ci, n, _lib.NDC_BF16 if dtype == torch.bfloat16 else _lib.NDC_F32, tf32, gy.data_ptr(),
            x.data_ptr(), gw.data_ptr(), ws.data_ptr())
    st = torch.cuda.current_stream().cuda_stream
    assert lib.ndc_proj_wgrad(*args, nbytes, st) == _lib.NDC_OK, lib.ndc_proj_last_error()
    ref = torch.einsum("bon,bcn->oc", gy.double(), x.double())
    err = ((gw.double() - ref).norm() / ref.norm()).item()
    assert err < tol, err
    assert lib.ndc_proj_wgrad(*args, nbytes - 4, st) == 3      # a short workspace is refused


@pytest.mark.parametrize("num_iters,num_grad_iters", [(1, 1), (3, 3), (3, 1), (2, 0)])
# among the sizes: rows that are padded inside the layer (one to three columns), on every kernel class
@pytest.mark.parametrize("channels,spatial,ks,groups", [(8, (5, 9, 7), (3, 3, 3), 8), (8, (12, 20), (5, 5), 8),
                                                        (8, (9, 10), (3, 3), 2), (192, (4, 8), (3, 3), 192),
                                                        (8, (4, 6, 5), (3, 3, 3), 8), (8, (30, 101), (3, 3), 8),
                                                        (6, (14, 45, 66), (3, 3, 3), 6), (4, (23, 17), (5, 5), 4)])
def test_layer_is_its_projection_followed_by_the_updates(num_iters, num_grad_iters, channels, spatial, ks, groups):
    """The native layer against `deconv_update` on a float64-accurate projection, every gradient."""
    dev = torch.device("cuda:0")
    torch.manual_seed(3)
    old = torch.backends.cudnn.allow_tf32
    torch.backends.cudnn.allow_tf32 = False
    try:
        mod = dcb.Deconv(channels, ks, ratio=2 if groups == 2 else 4, groups=groups, num_iters=num_iters,
                         num_grad_iters=num_grad_iters).to(dev)
        with torch.no_grad():
            mod.init.linear.linear.bias += 1.0
        x = torch.rand(2, channels, *spatial, device=dev)
        g = torch.randn(2, mod.groups * mod.source_channels, *spatial, device=dev)
        params = [mod.init.h0, mod.init.linear.linear.weight, mod.init.linear.linear.bias]
        xa = x.clone().requires_grad_(True)
        out = mod(xa)
        got = [out] + (list(torch.autograd.grad(out, [xa] + params, g, allow_unused=True)) if num_grad_iters else [])
        xb = x.clone().requires_grad_(True)
        h = torch.relu(mod.init.h0)
        s = (params[1][:, :, 0].double() @ xb.flatten(2).double()).float().view(2, -1, *spatial)
        bias = params[2]
        for it in range(1, num_iters + 1):
            with mod.context(it):
                s = dcb.deconv_update(xb, s, h, bias, groups=mod.groups, m=mod.filter_channels,
                                      sc=mod.source_channels, eps=mod.eps, relu_input=it == 1)
            bias = None
        ref = [s] + (list(torch.autograd.grad(s, [xb] + params, g, allow_unused=True)) if num_grad_iters else [])
    finally:
        torch.backends.cudnn.allow_tf32 = old
    assert out.requires_grad == bool(num_grad_iters)
    for a, b in zip(got, ref):
        assert (a is None) == (b is None)
        if a is not None:
            assert ((a - b).abs().max() / b.abs().max().clamp_min(1e-30)).item() < 1e-3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("rows,W,pitch", [(1, 5, 8), (7, 13, 16), (1000, 171, 176), (3, 8, 8)])
def test_row_padding(rows, W, pitch, dtype):
    lib, dev = _lib.load(), torch.device("cuda:0")
    x = torch.randn(rows, W, device=dev).to(dtype)
    p = torch.full((rows, pitch), 7.0, device=dev, dtype=dtype)
    y = torch.empty_like(x)
    st, code = torch.cuda.current_stream().cuda_stream, _lib.NDC_BF16 if dtype == torch.bfloat16 else _lib.NDC_F32
    assert lib.ndc_pad_rows(rows, W, pitch, code, x.data_ptr(), p.data_ptr(), st) == 0
    assert lib.ndc_unpad_rows(rows, W, pitch, code, p.data_ptr(), y.data_ptr(), st) == 0
    assert torch.equal(p[:, :W], x) and torch.equal(y, x) and not p[:, W:].any()
    assert lib.ndc_pad_rows(rows, W, W - 1, code, x.data_ptr(), p.data_ptr(), st) == 1


KERNEL, PRODUCT, SLICES, CONVOLUTION = range(4)      # WgradRoute


# f32: products of two-term operands, off by 2^-22 each at random, and sums rounded to nearest
@pytest.mark.parametrize("dtype,tf32,tol", [(torch.float32, True, 2e-3), (torch.float32, False, 1e-6), (torch.bfloat16, True, 6e-3)],
                         ids=["tf32", "f32", "bf16"])
@pytest.mark.parametrize("batch,co,ci,n,route", [
    (5, 96, 24, 34916, KERNEL),
    (4, 128, 32, 16384, KERNEL), (3, 40, 24, 1001, KERNEL), (2, 96, 24, 4095, KERNEL), (1, 192, 48, 4095, KERNEL),
    (8, 640, 160, 4096, PRODUCT), (16, 288, 72, 4096, PRODUCT), (1, 2048, 512, 512, PRODUCT), (16, 48, 192, 4096, PRODUCT),
    (1, 256, 64, 110592, SLICES), (1, 96, 384, 32768, SLICES), (3, 130, 70, 49992, SLICES),
    (1, 384, 96, 4095, CONVOLUTION), (2, 512, 512, 343, CONVOLUTION), (9, 640, 160, 101, CONVOLUTION),
])
def test_weight_gradient_of_every_route(dtype, tf32, tol, batch, co, ci, n, route):
    """Each side of each line of the dispatch, slices with a rest among them (49992 positions)."""
    dev = torch.device("cuda:0")
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    exact = dtype == torch.float32 and not tf32
    assert _lib.load_ext().weight_grad_route(batch, co, ci, n, dtype == torch.bfloat16, exact, sms) == (KERNEL if exact else route)
    gen = torch.Generator(device=dev).manual_seed(co + n)
    lin = dcb.Linear(ci, co).to(dev, dtype)
    x, g = torch.rand(batch, ci, n, device=dev, generator=gen).to(dtype), torch.randn(batch, co, n, device=dev, generator=gen).to(dtype)
    old = torch.backends.cudnn.allow_tf32
    torch.backends.cudnn.allow_tf32 = tf32
    try:
        (gw,) = torch.autograd.grad(lin(x), lin.linear.weight, g)
    finally:
        torch.backends.cudnn.allow_tf32 = old
    ref = torch.einsum("bon,bcn->oc", g.double(), x.double())
    assert gw.dtype == dtype and gw.shape == (co, ci, 1)
    assert ((gw[:, :, 0].double() - ref).norm() / ref.norm()).item() < tol
