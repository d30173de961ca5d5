"""The tensor-core forward (bfloat16 tensors, filter and bias) against the FMA kernels, which take the
same values as float32 parameters: edges of bands, chunks, blocks of eight columns and MMA tiles."""

import pytest
import torch

import deconver_b200 as dcb
from deconver_b200 import _lib
from deconver_b200 import functional as Fn

pytestmark = pytest.mark.gpu

CASES = [
    # channels, kernel, batch, spatial (large enough for the dispatch to take the tensor cores)
    (200, (3, 3, 3), 1, (7, 9, 64)),
    (13, (3, 3, 3), 2, (33, 31, 32)),
    (100, (3, 3, 3), 2, (9, 20, 24)),
    (32, (3, 3, 3), 1, (5, 40, 128)),
    (62, (3, 3, 3), 1, (3, 17, 256)),
    (2600, (3, 3, 3), 1, (1, 16, 20)),
    (150, (3, 3, 3), 1, (18, 17, 20)),
    (50, (5, 5), 4, (130, 128)),
    (45, (5, 5), 14, (77, 68)),
    (37, (5, 5), 1, (180, 512)),
    (280, (5, 5), 27, (16, 28)),
    (70, (3, 3), 3, (60, 252)),
    (420, (3, 3), 24, (9, 36)),
]


def _run(x, z, h, bias, relu, eps=1e-16):
    with torch.no_grad():
        return dcb.deconv_update(x, z, h, bias, groups=x.shape[1], m=1, sc=4, eps=eps, relu_input=relu)


@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "C%d_k%d_b%d_%s" % (c[0], c[1][0], c[2], "x".join(map(str, c[3]))))
def test_matches_the_fma_kernels(case, relu):
    C, ks, B, spatial = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(C + spatial[-1])
    x = torch.rand(B, C, *spatial, device=dev, generator=gen).bfloat16()
    z = (torch.randn(B, 4 * C, *spatial, device=dev, generator=gen) * 0.5 + 0.3).bfloat16()
    z = z if relu else z.abs()
    h = (torch.rand(C, 4, *ks, device=dev, generator=gen) / 27).bfloat16()
    bias = (torch.randn(4 * C, device=dev, generator=gen) * 0.1).bfloat16() if relu else None
    lib = _lib.load()
    before = lib.ndc_launch_count()
    got = _run(x, z, h, bias, relu)
    assert lib.ndc_launch_count() - before == 2
    ref = _run(x, z, h.float(), None if bias is None else bias.float(), relu)
    torch.cuda.synchronize()
    assert lib.ndc_wait_expired() == 0
    # the same exact products in another summation order: equal but for bfloat16 rounding of t1 and out
    diff = (got.float() - ref.float()).abs()
    assert (diff / ref.float().abs().clamp_min(1e-3)).max().item() < 0.02
    assert diff.norm().item() < 2e-3 * ref.float().norm().item()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C%d_k%d_b%d_%s" % (c[0], c[1][0], c[2], "x".join(map(str, c[3]))))
def test_gradients_match_the_fma_kernels(case):
    C, ks, B, spatial = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(C)
    x = torch.rand(B, C, *spatial, device=dev, generator=gen).bfloat16()
    z = (torch.randn(B, 4 * C, *spatial, device=dev, generator=gen) * 0.5 + 0.8).bfloat16()
    h = (torch.rand(C, 4, *ks, device=dev, generator=gen) / 27).bfloat16()
    bias = (torch.randn(4 * C, device=dev, generator=gen) * 0.1).bfloat16()
    g = torch.randn(B, 4 * C, *spatial, device=dev, generator=gen).bfloat16()
    res = []
    for dtype in (torch.bfloat16, torch.float32):      # of the parameters: the same values
        t = [v.clone().requires_grad_(True) for v in (x, z, h.to(dtype), bias.to(dtype))]
        out = dcb.deconv_update(*t, groups=C, m=1, sc=4, eps=1e-16, relu_input=True)
        out.backward(g)
        res.append([v.grad.float() for v in t])
    torch.cuda.synchronize()
    assert _lib.load().ndc_wait_expired() == 0
    for name, a, r in zip(("gx", "gz", "gh", "gb"), *res):
        assert ((a - r).norm() / r.norm()).item() < 5e-3, name


@pytest.mark.parametrize("channels,batch,spatial,ks", [(34, 2, (9, 31, 45), (3, 3, 3)), (150, 2, (5, 20, 27), (3, 3, 3)),
                                                       (8, 2, (33, 29, 62), (3, 3, 3)), (75, 6, (41, 171), (5, 5)),
                                                       (70, 6, (30, 253), (3, 3))])
def test_layer_with_padded_rows(channels, batch, spatial, ks):
    """Row lengths of every remainder modulo eight, two updates, against the generic kernels."""
    dev = torch.device("cuda:0")
    torch.manual_seed(1)
    mod = dcb.Deconv(channels, ks, ratio=4, num_iters=2).to(device=dev, dtype=torch.bfloat16)
    with torch.no_grad():
        mod.init.linear.linear.bias += 1.0
    x = torch.rand(batch, channels, *spatial, device=dev).bfloat16()
    g = torch.randn(batch, 4 * channels, *spatial, device=dev).bfloat16()
    res = []
    for generic in (False, True):
        xi = x.clone().requires_grad_(True)
        mod.zero_grad(set_to_none=True)
        with Fn.force_generic(generic):
            out = mod(xi)
            out.backward(g)
        res.append([out.detach(), xi.grad] + [p.grad for p in mod.parameters()])
    for a, r in zip(*res):
        assert ((a.float() - r.float()).norm() / r.float().norm()).item() < 1e-2
