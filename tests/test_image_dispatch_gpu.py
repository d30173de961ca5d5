"""Image updates on both sides of each line between the row-marching and the band kernels (short
marches with fewer CTAs than SMs; 5x5 rows of 129..192 columns), and images whose strips just fill or
just exceed the small band CTA, against the generic kernels."""

import pytest
import torch

import deconver_b200 as dcb
from conftest import max_norm_error
from deconver_b200 import functional as Fn

pytestmark = pytest.mark.gpu

CASES = [
    # batch, groups, kernel, height, width
    (2, 3, 5, 31, 64), (2, 3, 5, 32, 64), (2, 147, 3, 9, 66), (2, 148, 3, 9, 66),
    (1, 5, 5, 33, 128), (1, 5, 5, 33, 129), (1, 5, 5, 40, 192), (1, 5, 5, 40, 193), (2, 5, 3, 40, 171),
    (1, 9, 5, 16, 32), (1, 9, 5, 17, 32), (1, 9, 5, 20, 21), (1, 9, 3, 21, 24), (1, 9, 5, 31, 15), (1, 9, 5, 1, 3),
]


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=["f32", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_image_kernels_match_the_generic_ones(case, dtype, tol):
    B, G, k, H, W = case
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(H + W)
    x = torch.rand(B, G, H, W, device=dev, generator=gen).to(dtype)
    z = (torch.randn(B, G * 4, H, W, device=dev, generator=gen) * 0.5 + 0.3).to(dtype)
    h = torch.rand(G, 4, k, k, device=dev, generator=gen) / 27.0
    bias = torch.randn(G * 4, device=dev, generator=gen) * 0.1
    gout = torch.randn(B, G * 4, H, W, device=dev, generator=gen).to(dtype)
    res = []
    for generic in (True, False):
        t = [v.clone().requires_grad_(True) for v in (x, z, h, bias)]
        with Fn.force_generic(generic):
            out = dcb.deconv_update(*t, groups=G, m=1, sc=4, eps=1e-16, relu_input=True)
            out.backward(gout)
        res.append([out.detach()] + [v.grad for v in t])
    for name, a, r in zip(("out", "gx", "gz", "gh", "gb"), res[1], res[0]):
        assert max_norm_error(a.float().cpu().numpy(), r.float().cpu().numpy()) < tol, name


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=["f32", "bf16"])
@pytest.mark.parametrize("case", [(1, 5, 3, 20, 200), (2, 3, 3, 31, 129), (2, 3, 3, 31, 128), (1, 3, 3, 8, 96)], ids=lambda c: "x".join(map(str, c)))
def test_short_3x3_images_of_one_per_cta(case, dtype, tol):
    test_image_kernels_match_the_generic_ones(case, dtype, tol)


@pytest.mark.parametrize("k,spatial", [(5, (16, 16)), (5, (40, 128)), (3, (40, 171)), (3, (8, 8, 8)), (3, (9, 20, 33)), (7, (12, 12))])
def test_inference_rectifies_the_filter_as_training_does(k, spatial):
    torch.manual_seed(0)
    net = dcb.Deconv(6, kernel_size=(k,) * len(spatial), ratio=4, groups=-1, num_iters=2).to("cuda:0")
    with torch.no_grad():
        net.init.h0.copy_(torch.randn_like(net.init.h0) / k)     # a filter of both signs
    x = torch.rand(2, 6, *spatial, device="cuda:0")
    with torch.no_grad():
        y = net(x)
    assert torch.equal(y, net(x).detach())
