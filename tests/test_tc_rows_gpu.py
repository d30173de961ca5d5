"""Sizes near the line from which bfloat16 updates run on the tensor cores, against the oracle: bands of image rows that
cross from one chunk into the next, a last band and a last chunk that are partly filled, one place of work per CTA and
several, with and without a change of channel between them."""

import numpy as np
import pytest
import torch

import deconver_b200 as dcb
from conftest import max_norm_error
from deconver_b200 import _lib
from oracle import c_oracle
from test_tc_gpu import _family

pytestmark = pytest.mark.gpu

CASES = [
    # channels, kernel, batch, spatial
    (40, (5, 5), 3, (128, 120)),      # one place per CTA
    (160, (5, 5), 24, (32, 32)),      # more places than CTAs; every one has another channel
    (9, (5, 5), 1, (300, 300)),       # one image: bands are chunks alone
    (5, (5, 5), 16, (260, 256)),      # several places per channel
    (128, (3, 3), 16, (24, 20)),
    (16, (3, 3), 1, (220, 240)),
    (32, (3, 3, 3), 1, (28, 28, 28)),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C%d_k%d_b%d_%s" % (c[0], c[1][0], c[2], "x".join(map(str, c[3]))))
def test_against_the_oracle(case):
    C, ks, B, spatial = case
    assert _family(C, ks, B, spatial, _lib.FLAG_BF16_PARAMS) == _lib.FAMILY_TENSOR
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
    torch.cuda.synchronize()
    assert _lib.load().ndc_wait_expired() == 0
    args = [v.double().numpy() for v in (x, z, h, bias)]
    # `out`, of positive terms: t1 and out are each rounded once (2^-8); gradients cancel
    ref, _ = c_oracle.forward(*args, **cfg)
    assert (np.abs(out.detach().double().cpu().numpy() - ref) <= (2.0 ** -7 + 2.0 ** -9) * ref).all()
    for name, a, r in zip(("gx", "gz", "gh", "gb"), (v.grad for v in t), c_oracle.backward(*args, g.double().numpy(), **cfg)):
        assert max_norm_error(a.float().cpu().numpy(), r) < 2e-2, name
