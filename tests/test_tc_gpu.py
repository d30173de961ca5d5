"""The tensor-core forward (bfloat16 tensors, filter and bias) against the FMA kernels, which take the
same values as float32 parameters: edges of bands, chunks, blocks of eight columns and MMA tiles."""

import pytest
import torch

import deconver_b200 as dcb
from deconver_b200 import _lib
from deconver_b200 import functional as Fn

pytestmark = pytest.mark.gpu

CASES = [
    # channels, kernel, batch, spatial
    (3, (3, 3, 3), 1, (7, 9, 64)),
    (2, (3, 3, 3), 2, (33, 31, 32)),
    (50, (3, 3, 3), 2, (9, 20, 24)),
    (2, (3, 3, 3), 1, (5, 40, 128)),
    (2, (3, 3, 3), 1, (3, 17, 256)),
    (4, (3, 3, 3), 1, (1, 16, 20)),
    (300, (3, 3, 3), 1, (18, 16, 16)),
    (6, (5, 5), 3, (130, 128)),
    (5, (5, 5), 5, (37, 68)),
    (3, (5, 5), 1, (40, 512)),
    (40, (5, 5), 9, (16, 28)),
    (3, (3, 3), 4, (45, 256)),
    (7, (3, 3), 20, (9, 36)),
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


@pytest.mark.parametrize("spatial,ks", [((9, 31, 45), (3, 3, 3)), ((5, 20, 27), (3, 3, 3)), ((33, 29, 62), (3, 3, 3)),
                                        ((41, 171), (5, 5)), ((30, 253), (3, 3))])
def test_layer_with_padded_rows(spatial, ks):
    """Row lengths of every remainder modulo eight, two updates, against the generic kernels."""
    dev = torch.device("cuda:0")
    torch.manual_seed(1)
    mod = dcb.Deconv(8, ks, ratio=4, num_iters=2).to(device=dev, dtype=torch.bfloat16)
    with torch.no_grad():
        mod.init.linear.linear.bias += 1.0
    x = torch.rand(2, 8, *spatial, device=dev).bfloat16()
    g = torch.randn(2, 32, *spatial, device=dev).bfloat16()
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
