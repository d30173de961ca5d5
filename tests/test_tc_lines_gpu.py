"""About the lines from which bfloat16 updates run on the tensor cores, which lie higher for the backward than for the forward:
which kernels each direction takes, and a forward on the tensor cores with a backward on the FMA kernels against the oracle."""

import ctypes

import numpy as np
import pytest
import torch

import deconver_b200 as dcb
from conftest import max_norm_error
from deconver_b200 import _lib
from oracle import c_oracle

FORWARD, BOTH, NEITHER = (True, False), (True, True), (False, False)
CASES = [
    # channels, kernel, batch, spatial, forward and backward on the tensor cores
    (64, (5, 5), 16, (28, 28), FORWARD),
    (88, (5, 5), 14, (30, 36), FORWARD),
    (172, (3, 3), 8, (28, 28), FORWARD),
    (24, (3, 3), 2, (256, 256), FORWARD),
    (92, (5, 5), 4, (49, 48), BOTH),
    (128, (5, 5), 2, (64, 64), BOTH),
    (256, (3, 3), 8, (28, 28), BOTH),
    (188, (3, 3), 8, (16, 32), NEITHER),
    (512, (5, 5), 4, (16, 16), NEITHER),
    (24, (3, 3, 3), 1, (28, 26, 36), BOTH),
    (128, (3, 3, 3), 1, (16, 16, 16), NEITHER),
]
ids = dict(ids=lambda c: "C%d_k%d_b%d_%s" % (c[0], c[1][0], c[2], "x".join(map(str, c[3]))))


@pytest.mark.parametrize("case", CASES, **ids)
def test_kernels_of_either_direction(case):
    C, ks, B, spatial, want = case
    lib, got = _lib.load(), []
    desc = _lib.make_desc(B, C, 1, 4, spatial, ks, 1e-16, True, _lib.NDC_BF16, _lib.FLAG_BF16_PARAMS)
    for query in (lib.ndc_kernel_family, lib.ndc_backward_family):
        family = ctypes.c_int32(-1)
        _lib.check(query(desc, lib.ndc_row_pitch(desc), ctypes.byref(family)))
        assert family.value in (_lib.FAMILY_MARCH, _lib.FAMILY_MARCH_ROWS, _lib.FAMILY_TENSOR)
        got.append(family.value == _lib.FAMILY_TENSOR)
    assert tuple(got) == want


@pytest.mark.gpu
@pytest.mark.parametrize("case", [c for c in CASES if c[4] == FORWARD][:3], **ids)
def test_mixed_against_the_oracle(case):
    C, ks, B, spatial, _ = case
    gen = torch.Generator().manual_seed(C)
    x = torch.rand(B, C, *spatial, generator=gen).bfloat16()
    z = (torch.randn(B, 4 * C, *spatial, generator=gen) * 0.5 + 0.3).bfloat16()
    h = (torch.rand(C, 4, *ks, generator=gen) / 27).bfloat16()
    bias = (torch.randn(4 * C, generator=gen) * 0.1).bfloat16()
    g = torch.randn(B, 4 * C, *spatial, generator=gen).bfloat16()
    t = [v.to("cuda:0").requires_grad_(True) for v in (x, z, h, bias)]
    cfg = dict(groups=C, m=1, sc=4, eps=1e-16, relu_input=True)
    out = dcb.deconv_update(*t, **cfg)
    out.backward(g.to("cuda:0"))
    args = [v.double().numpy() for v in (x, z, h, bias)]
    # `out`, of positive terms: t1 and out are each rounded once (2^-8); gradients cancel
    ref, _ = c_oracle.forward(*args, **cfg)
    assert (np.abs(out.detach().double().cpu().numpy() - ref) <= (2.0 ** -7 + 2.0 ** -9) * ref).all()
    for name, a, r in zip(("gx", "gz", "gh", "gb"), (v.grad for v in t), c_oracle.backward(*args, g.double().numpy(), **cfg)):
        assert max_norm_error(a.float().cpu().numpy(), r) < 2e-2, name
