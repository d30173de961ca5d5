"""The tensor-core forward (bfloat16 tensors, filter and bias) against the FMA kernels, which take the
same values as float32 parameters: edges of bands, chunks, blocks of eight columns and MMA tiles."""

import ctypes
import subprocess
import sys

import numpy as np
import pytest
import torch

import deconver_b200 as dcb
from conftest import ROOT, max_norm_error
from deconver_b200 import _lib
from deconver_b200 import functional as Fn
from oracle import c_oracle
from oracle import ndc_oracle as O

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


def _family(C, ks, B, spatial, flags, relu=True):
    lib, family = _lib.load(), ctypes.c_int32(-1)
    desc = _lib.make_desc(B, C, 1, 4, spatial, ks, 1e-16, relu, _lib.NDC_BF16, flags)
    assert lib.ndc_kernel_family(desc, lib.ndc_row_pitch(desc), ctypes.byref(family)) == _lib.NDC_OK
    return family.value


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C%d_k%d_b%d_%s" % (c[0], c[1][0], c[2], "x".join(map(str, c[3]))))
def test_update_against_the_oracle(case):
    """Forward and every gradient on the tensor cores against the C oracle in 64 bits on the same bfloat16
    values.  `out`, of positive terms, element by element: t1 and out are each rounded once (2^-8).  The
    gradients have sums that cancel: largest error over the largest value, as for every bfloat16 update."""
    C, ks, B, spatial = case
    assert _family(C, ks, B, spatial, _lib.FLAG_BF16_PARAMS) == _lib.FAMILY_TENSOR
    assert _family(C, ks, B, spatial, 0) in (_lib.FAMILY_MARCH, _lib.FAMILY_MARCH_ROWS)
    gen = torch.Generator().manual_seed(C)
    x = torch.rand(B, C, *spatial, generator=gen).bfloat16()
    z = (torch.randn(B, 4 * C, *spatial, generator=gen) * 0.5 + 0.3).bfloat16()
    h = (torch.rand(C, 4, *ks, generator=gen) / 27).bfloat16()
    bias = (torch.randn(4 * C, generator=gen) * 0.1).bfloat16()
    g = torch.randn(B, 4 * C, *spatial, generator=gen).bfloat16()
    t = [v.to("cuda:0").requires_grad_(True) for v in (x, z, h, bias)]
    out = dcb.deconv_update(*t, groups=C, m=1, sc=4, eps=1e-16, relu_input=True)
    out.backward(g.to("cuda:0"))
    cfg = dict(groups=C, m=1, sc=4, eps=1e-16, relu_input=True)
    args = [v.double().numpy() for v in (x, z, h, bias)]
    ref, _ = c_oracle.forward(*args, **cfg)
    assert (np.abs(out.detach().double().cpu().numpy() - ref) <= (2.0 ** -7 + 2.0 ** -9) * ref).all()
    for name, a, r in zip(("gx", "gz", "gh", "gb"), (v.grad for v in t), c_oracle.backward(*args, g.double().numpy(), **cfg)):
        assert max_norm_error(a.float().cpu().numpy(), r) < 2e-2, name


# volumes and images, rows of whole blocks of eight columns and not, several bands and chunks of planes
CANCELLING = [(150, (3, 3, 3), 1, (18, 17, 20)), (200, (3, 3, 3), 1, (7, 9, 64)), (50, (5, 5), 4, (130, 128)),
              (45, (5, 5), 14, (77, 68)), (70, (3, 3), 3, (60, 252))]


@pytest.mark.parametrize("live", [0.0, 0.002, 0.05, 0.6])
@pytest.mark.parametrize("mixed", [False, True], ids=["even", "mixed"])
@pytest.mark.parametrize("case", CANCELLING, ids=lambda c: "C%d_k%d_b%d_%s" % (c[0], c[1][0], c[2], "x".join(map(str, c[3]))))
def test_rectified_sources_leave_no_rounding_behind(case, mixed, live):
    """A source that is rectified away all but for a share `live`, down to one unit of the bias's last
    place above it, against the oracle in 64 bits, element by element: zeros are zeros, and no value is
    further off than its roundings to bfloat16 (2^-8 each) and a float32 sum's share of one.  `mixed`: the
    channels' biases differ by factors of ten, so that what is left is small beside what cancelled."""
    C, ks, B, spatial = case
    assert _family(C, ks, B, spatial, _lib.FLAG_BF16_PARAMS) == _lib.FAMILY_TENSOR
    gen = torch.Generator().manual_seed(C)
    x = torch.rand(B, C, *spatial, generator=gen).bfloat16()
    bias = torch.rand(4 * C, generator=gen) * 0.2 + 0.9
    if mixed:
        bias = bias * 10.0 ** -(torch.arange(4 * C) % 4).float()
    bias = bias.bfloat16()
    b = bias.view(1, -1, *[1] * len(ks)).float()
    on = torch.rand(B, 4 * C, *spatial, generator=gen) < live
    share = torch.where(torch.rand(on.shape, generator=gen) < 0.5, 0.01, 1.0)
    z = torch.where(on, (torch.rand(on.shape, generator=gen) * share - 1.0) * b, -b - torch.rand(on.shape, generator=gen) * b).bfloat16()
    h = (torch.rand(C, 4, *ks, generator=gen) / 27).bfloat16()
    xd, zd, hd, bd = (t.to("cuda:0") for t in (x, z, h.float(), bias.float()))
    out, t1 = torch.empty_like(zd), torch.empty_like(xd)
    desc = _lib.make_desc(B, C, 1, 4, spatial, ks, 1e-16, True, _lib.NDC_BF16, _lib.FLAG_BF16_PARAMS)
    _lib.check(_lib.load().ndc_fwd(desc, xd.data_ptr(), zd.data_ptr(), hd.data_ptr(), bd.data_ptr(), out.data_ptr(), t1.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream))
    s = torch.relu(z.double() + b.double())
    ref_t1 = O.K(s, h.double(), C)
    got = t1.double().cpu()
    assert not got[ref_t1 == 0].any()
    assert ((got - ref_t1).abs() <= (2.0 ** -8 + 2.0 ** -10) * ref_t1).all()
    ref = s * (O.A(x.double(), h.double(), C) + 1e-16) / (O.A(ref_t1, h.double(), C) + 1e-16)
    assert ((out.double().cpu() - ref).abs() <= (2.0 ** -7 + 2.0 ** -9) * ref).all()


def test_a_wait_that_runs_out_is_reported():
    """By the next call, once, and from then on by ndc_wait_expired (hence a process of its own)."""
    program = """if True:
        import torch, deconver_b200 as dcb
        from deconver_b200 import _lib
        lib = _lib.load()
        mod, x = dcb.Deconv(4, (3, 3), ratio=4).cuda(), torch.rand(1, 4, 8, 8, device="cuda:0")
        want = mod(x)
        assert lib.ndc_probe_wait(2000, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        try:
            mod(x)
            raise SystemExit("not reported")
        except RuntimeError as e:
            assert "ran out" in str(e), e
        assert torch.equal(mod(x), want) and lib.ndc_wait_expired()
        """
    subprocess.run([sys.executable, "-c", program], check=True, timeout=300, cwd=ROOT)


@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("ks,B,spatial,pitch", [((3, 3, 3), 2, (9, 31, 45), 48), ((5, 5), 6, (41, 171), 172)])
def test_padding_of_the_source_is_not_read(ks, B, spatial, pitch, relu):
    """Only x has to be zero in the padding of the rows; z may hold anything there."""
    C, (*lead, W), lib, dev = 75, spatial, _lib.load(), "cuda:0"
    gen = torch.Generator(device=dev).manual_seed(3)
    x, z = (torch.zeros(B, n, *lead, pitch, device=dev, dtype=torch.bfloat16) for n in (C, 4 * C))
    x[..., :W] = torch.rand(B, C, *lead, W, device=dev, generator=gen)
    z[..., :W] = torch.rand(B, 4 * C, *lead, W, device=dev, generator=gen)
    assert _family(C, ks, B, spatial, _lib.FLAG_BF16_PARAMS, relu) == _lib.FAMILY_TENSOR
    h = (torch.rand(C, 4, *ks, device=dev, generator=gen) / 27).bfloat16().float()
    desc = _lib.make_desc(B, C, 1, 4, spatial, ks, 1e-16, relu, _lib.NDC_BF16, _lib.FLAG_BF16_PARAMS)
    res = []
    for garbage in (0.0, 1000.0):
        z[..., W:] = garbage
        out, t1 = torch.zeros_like(z), torch.empty_like(x)
        _lib.check(lib.ndc_fwd_rows(desc, pitch, pitch, x.data_ptr(), z.data_ptr(), h.data_ptr(), None, out.data_ptr(), t1.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream))
        res.append((out[..., :W].clone(), t1))
    assert all(torch.equal(a, b) for a, b in zip(*res)) and not t1[..., W:].any()


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
