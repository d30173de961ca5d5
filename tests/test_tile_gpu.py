"""The tile kernels (any grouping, 3x3x3 / 5x5 / 3x3 filters) against the generic ones, which the
fixtures pin: remainders of channel blocks, strips, row groups and planes, and rows wider than the
depthwise ratio-4 kernels take."""

import ctypes

import pytest
import torch

import deconver_b200 as dcb
from conftest import max_norm_error
from deconver_b200 import _lib
from deconver_b200 import functional as Fn
from oracle import c_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # groups, m, sc, kernel, batch, spatial
    (5, 1, 1, (3, 3, 3), 2, (5, 9, 33)),
    (2, 4, 16, (3, 3, 3), 1, (9, 17, 21)),
    (1, 16, 16, (3, 3, 3), 1, (3, 4, 6)),
    (3, 2, 5, (3, 3, 3), 2, (1, 1, 1)),
    (2, 4, 8, (3, 3, 3), 2, (8, 32, 32)),
    (3, 5, 2, (5, 5), 2, (37, 70)),
    (4, 2, 8, (5, 5), 3, (16, 16)),
    (8, 1, 2, (3, 3), 1, (130, 43)),
    (2, 3, 9, (3, 3), 2, (7, 129)),
    (2, 1, 4, (3, 3), 1, (9, 601)),
    (1, 1, 4, (3, 3, 3), 1, (2, 3, 300)),
]


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=["f32", "bf16"])
@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "g%d_m%d_sc%d_%s" % (c[0], c[1], c[2], "x".join(map(str, c[5]))))
def test_tile_kernels_match_the_generic_ones(case, relu, dtype, tol):
    G, m, sc, ks, B, spatial = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(G + sc + spatial[-1])
    x = torch.rand(B, G * m, *spatial, device=dev, generator=gen).to(dtype)
    z = (torch.randn(B, G * sc, *spatial, device=dev, generator=gen) * 0.5 + 0.3).to(dtype)
    z = z if relu else z.abs()
    h = torch.rand(G * m, sc, *ks, device=dev, generator=gen) / 27.0
    bias = torch.randn(G * sc, device=dev, generator=gen) * 0.1 if relu else None
    gout = torch.randn(B, G * sc, *spatial, device=dev, generator=gen).to(dtype)
    res = []
    for generic in (True, False):
        t = [None if v is None else v.clone().requires_grad_(True) for v in (x, z, h, bias)]
        with Fn.force_generic(generic):
            out = dcb.deconv_update(*t, groups=G, m=m, sc=sc, eps=1e-16, relu_input=relu)
            out.backward(gout)
        res.append([out.detach()] + [v.grad for v in t if v is not None])
    for name, a, r in zip(("out", "gx", "gz", "gh", "gb"), res[1], res[0]):
        assert max_norm_error(a.float().cpu().numpy(), r.float().cpu().numpy()) < tol, name


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=["f32", "bf16"])
@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "g%d_m%d_sc%d_%s" % (c[0], c[1], c[2], "x".join(map(str, c[5]))))
def test_tile_kernels_against_the_oracle(case, relu, dtype, tol):
    G, m, sc, ks, B, spatial = case
    family = ctypes.c_int32(-1)
    desc = _lib.make_desc(B, G, m, sc, spatial, ks, 1e-16, relu, _lib.NDC_BF16 if dtype == torch.bfloat16 else _lib.NDC_F32)
    assert _lib.load().ndc_kernel_family(desc, spatial[-1], ctypes.byref(family)) == _lib.NDC_OK and family.value == _lib.FAMILY_TILE
    gen = torch.Generator().manual_seed(G + sc + spatial[-1])
    x = torch.rand(B, G * m, *spatial, generator=gen).to(dtype)
    z = (torch.randn(B, G * sc, *spatial, generator=gen) * 0.5 + 0.3).to(dtype)
    z = z if relu else z.abs()
    h = torch.rand(G * m, sc, *ks, generator=gen) / 27.0
    bias = torch.randn(G * sc, generator=gen) * 0.1 if relu else None
    gout = torch.randn(B, G * sc, *spatial, generator=gen).to(dtype)
    t = [None if v is None else v.to("cuda:0").requires_grad_(True) for v in (x, z, h, bias)]
    cfg = dict(groups=G, m=m, sc=sc, eps=1e-16, relu_input=relu)
    out = dcb.deconv_update(*t, **cfg)
    out.backward(gout.to("cuda:0"))
    args = [None if v is None else v.double().numpy() for v in (x, z, h, bias)]
    ref = [c_oracle.forward(*args, **cfg)[0], *c_oracle.backward(*args, gout.double().numpy(), **cfg)]
    for name, a, r in zip(("out", "gx", "gz", "gh", "gb"), [out.detach()] + [v.grad for v in t if v is not None], ref):
        assert max_norm_error(a.float().cpu().numpy(), r) < tol, name


@pytest.mark.parametrize("mask", range(1, 16))
def test_partial_gradient_requests(mask):
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(1)
    v = [torch.rand(2, 6, 5, 6, 7, device=dev, generator=gen), torch.randn(2, 10, 5, 6, 7, device=dev, generator=gen),
         torch.rand(6, 5, 3, 3, 3, device=dev, generator=gen), torch.randn(10, device=dev, generator=gen)]
    g = torch.randn(2, 10, 5, 6, 7, device=dev, generator=gen)

    def run(bits):
        t = [a.clone().requires_grad_(bool(bits >> i & 1)) for i, a in enumerate(v)]
        dcb.deconv_update(*t, groups=2, m=3, sc=5, eps=1e-16, relu_input=True).backward(g)
        return [a.grad for a in t]

    full = run(15)
    for i, a in enumerate(run(mask)):
        assert (a is None) if not mask >> i & 1 else torch.equal(a, full[i])
