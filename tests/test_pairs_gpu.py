"""The tile kernels for rows of whole vectors against the oracle: each number of channels per thread, blocks that are
partly filled, an odd number of tiles (they go in pairs), one strip, and more strips than a tile has; and tensors
that are not on whole vectors, which other kernels take."""

import pytest
import torch

import deconver_b200 as dcb
from conftest import max_norm_error
from oracle import c_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # groups, m, sc, kernel, batch, spatial
    (3, 1, 1, (3, 3, 3), 1, (5, 9, 36)),
    (2, 2, 2, (3, 3, 3), 3, (3, 7, 4)),
    (2, 4, 8, (3, 3, 3), 1, (9, 19, 40)),
    (1, 16, 12, (3, 3, 3), 1, (2, 5, 8)),
    (2, 3, 7, (3, 3, 3), 1, (1, 1, 4)),
    (2, 1, 2, (5, 5), 1, (21, 68)),
    (1, 5, 16, (5, 5), 2, (35, 12)),
    (2, 8, 3, (3, 3), 1, (33, 132)),
    # warps that only stage, on the last grid that has them; the first without
    (8, 1, 1, (3, 3), 2, (41, 44)),
    (1, 1, 1, (3, 3, 3), 3, (9, 13, 20)),
    (4, 1, 2, (5, 5), 37, (16, 32)),
    (149, 1, 1, (3, 3), 1, (16, 32)),
    # more CTAs than multiprocessors: as much per thread as there is (half of it in the cases above)
    (300, 1, 1, (3, 3, 3), 1, (2, 9, 8)),
    (300, 2, 2, (3, 3, 3), 1, (3, 5, 8)),
    (300, 8, 4, (3, 3, 3), 1, (2, 5, 4)),
    (300, 1, 2, (5, 5), 1, (9, 12)),
    (300, 3, 8, (5, 5), 1, (7, 8)),
    (300, 1, 1, (5, 5), 1, (17, 8)),
    (300, 4, 8, (3, 3), 1, (10, 12)),
    (300, 1, 2, (3, 3), 1, (13, 4)),
]


def _data(case, dtype, shift=0):
    G, m, sc, ks, B, spatial = case
    gen = torch.Generator().manual_seed(G + sc + spatial[-1])

    def place(t):      # `shift` elements past an aligned address
        t = t.to(dtype)
        flat = torch.empty(t.numel() + shift, dtype=dtype, device="cuda:0")
        flat[shift:] = t.flatten().to("cuda:0")
        return flat[shift:].view(t.shape)

    x = torch.rand(B, G * m, *spatial, generator=gen)
    z = torch.randn(B, G * sc, *spatial, generator=gen) * 0.5 + 0.3
    gout = torch.randn(B, G * sc, *spatial, generator=gen)
    h = torch.rand(G * m, sc, *ks, generator=gen) / 27.0
    bias = torch.randn(G * sc, generator=gen) * 0.1
    x, z, gout = place(x), place(z), place(gout)
    return [v.requires_grad_(True) for v in (x, z, h.to("cuda:0"), bias.to("cuda:0"))], gout


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=["f32", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "g%d_m%d_sc%d_%s" % (c[0], c[1], c[2], "x".join(map(str, c[5]))))
def test_against_the_oracle(case, dtype, tol):
    t, gout = _data(case, dtype)
    cfg = dict(groups=case[0], m=case[1], sc=case[2], eps=1e-16, relu_input=True)
    out = dcb.deconv_update(*t, **cfg)
    out.backward(gout)
    args = [v.detach().cpu().double().numpy() for v in t]
    ref = [c_oracle.forward(*args, **cfg)[0], *c_oracle.backward(*args, gout.cpu().double().numpy(), **cfg)]
    for name, a, r in zip(("out", "gx", "gz", "gh", "gb"), [out.detach()] + [v.grad for v in t], ref):
        assert max_norm_error(a.float().cpu().numpy(), r) < tol, name


@pytest.mark.parametrize("case", [CASES[2], CASES[5]], ids=["volume", "image"])
def test_shifted_tensors_take_the_other_kernels(case):
    """The same values one element past an aligned address: summed in another order, so close and not equal."""
    cfg = dict(groups=case[0], m=case[1], sc=case[2], eps=1e-16, relu_input=True)
    res = []
    for shift in (0, 1):
        t, gout = _data(case, torch.float32, shift)
        out = dcb.deconv_update(*t, **cfg)
        out.backward(gout)
        res.append([out.detach()] + [v.grad for v in t])
    for name, a, r in zip(("out", "gx", "gz", "gh", "gb"), *res):
        assert max_norm_error(a.cpu().numpy(), r.cpu().numpy()) < 1e-4, name
    assert not all(torch.equal(a, r) for a, r in zip(*res))


@pytest.mark.parametrize("mask", range(1, 16))
def test_partial_gradient_requests(mask):
    """Either stream of K may be missing, and the direct term."""
    t, gout = _data((2, 3, 5, (3, 3, 3), 2, (5, 6, 8)), torch.float32)

    def run(bits):
        v = [a.detach().requires_grad_(bool(bits >> i & 1)) for i, a in enumerate(t)]
        dcb.deconv_update(*v, groups=2, m=3, sc=5, eps=1e-16, relu_input=True).backward(gout)
        return [a.grad for a in v]

    full = run(15)
    for i, a in enumerate(run(mask)):
        assert (a is None) if not mask >> i & 1 else torch.equal(a, full[i])


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=["f32", "bf16"])
@pytest.mark.parametrize("case", [CASES[2], CASES[5], CASES[7]], ids=["volume", "5x5", "3x3"])
def test_x_alone_off_a_vector_address(case, dtype, tol):
    """The tile kernels with whole vectors of everything else."""
    t, gout = _data(case, dtype)
    flat = torch.empty(t[0].numel() + 1, dtype=dtype, device="cuda:0")
    flat[1:] = t[0].detach().flatten()
    aligned, t[0] = t[0].detach(), flat[1:].view(t[0].shape).requires_grad_(True)
    cfg = dict(groups=case[0], m=case[1], sc=case[2], eps=1e-16, relu_input=True)
    out = dcb.deconv_update(*t, **cfg)
    out.backward(gout)
    args = [v.detach().cpu().double().numpy() for v in t]
    ref = [c_oracle.forward(*args, **cfg)[0], *c_oracle.backward(*args, gout.cpu().double().numpy(), **cfg)]
    for name, a, r in zip(("out", "gx", "gz", "gh", "gb"), [out.detach()] + [v.grad for v in t], ref):
        assert max_norm_error(a.float().cpu().numpy(), r) < tol, name
    if dtype == torch.float32:      # summed in another order
        assert not torch.equal(out.detach(), dcb.deconv_update(aligned, *t[1:], **cfg).detach())
