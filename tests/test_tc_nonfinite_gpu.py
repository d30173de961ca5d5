"""Infinities and NaN in bfloat16 updates on the tensor cores: they reach what the filter's taps reach, as with the FMA
kernels, and no other column, row, image or channel."""

import pytest
import torch

from deconver_b200 import _lib
from test_tc_gpu import _family

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")
CASES = [
    # channels, kernel, batch, spatial: rows whose last block of eight columns holds the filter's reach or not,
    # whole blocks, padded rows, chunks of one image, CTAs with one place of work and with several, volumes
    (160, (5, 5), 32, (28, 28)),
    (24, (5, 5), 16, (60, 60)),
    (60, (5, 5), 5, (101, 203)),
    (40, (5, 5), 3, (128, 128)),
    (36, (5, 5), 1, (300, 300)),
    (96, (3, 3), 9, (60, 60)),
    (32, (3, 3), 5, (203, 171)),
    (60, (3, 3, 3), 2, (30, 30, 30)),
    (48, (3, 3, 3), 1, (37, 32, 32)),
]


def _update(x, z, h, bias, gout, ks, flags, relu):
    """out, gx, gz, gh, gb of one update on rows of the pitch that the library asks for."""
    lib, (B, C, *lead, W) = _lib.load(), x.shape
    desc = _lib.make_desc(B, C, 1, 4, (*lead, W), ks, 1e-16, relu, _lib.NDC_BF16, flags)
    pitch, st = lib.ndc_row_pitch(desc), torch.cuda.current_stream().cuda_stream

    def rows(t):
        p = torch.zeros(*t.shape[:-1], pitch, dtype=t.dtype, device=t.device)
        p[..., :W] = t
        return p

    x, z, gout = rows(x), rows(z), rows(gout)
    out, t1, gx, gz = torch.zeros_like(z), torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(z)
    gh, gb = torch.zeros_like(h), torch.zeros_like(bias)
    _lib.check(lib.ndc_fwd_rows(desc, pitch, pitch, x.data_ptr(), z.data_ptr(), h.data_ptr(), bias.data_ptr(), out.data_ptr(),
                                t1.data_ptr(), st))
    need = lib.ndc_bwd_rows_workspace_bytes(desc, pitch)
    ws = torch.empty(need, dtype=torch.uint8, device=x.device)
    _lib.check(lib.ndc_bwd_rows(desc, pitch, pitch, x.data_ptr(), z.data_ptr(), t1.data_ptr(), h.data_ptr(), bias.data_ptr(),
                                gout.data_ptr(), gx.data_ptr(), gz.data_ptr(), gh.data_ptr(), gb.data_ptr(), ws.data_ptr(), need, st))
    assert not t1[..., W:].any() and not gx[..., W:].any() and not gz[..., W:].any()
    return [t[..., :W].float() for t in (out, t1, gx, gz)] + [gh, gb]


@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("value", [INF, -INF, NAN], ids=["inf", "minus_inf", "nan"])
@pytest.mark.parametrize("where", ["x", "z", "gout"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "C%d_k%d_b%d_%s" % (c[0], c[1][0], c[2], "x".join(map(str, c[3]))))
def test_reaches_what_the_taps_reach(case, where, value, relu):
    C, ks, B, spatial = case
    assert _family(C, ks, B, spatial, _lib.FLAG_BF16_PARAMS, relu) == _lib.FAMILY_TENSOR
    dev, gen = "cuda:0", torch.Generator(device="cuda:0").manual_seed(C)
    t = {"x": torch.rand(B, C, *spatial, device=dev, generator=gen).bfloat16(),
         "z": (torch.rand(B, 4 * C, *spatial, device=dev, generator=gen) + 0.1).bfloat16(),
         "gout": torch.randn(B, 4 * C, *spatial, device=dev, generator=gen).bfloat16()}
    h = (torch.rand(C, 4, *ks, device=dev, generator=gen) / 27 + 0.01).bfloat16().float()
    bias = (torch.rand(4 * C, device=dev, generator=gen) * 0.1).bfloat16().float()
    planted = t[where]
    # first and last columns of rows in the middle and at the ends, in one sample each of a few channels
    for n, (b, row, col) in enumerate([(B // 2, 0, 0), (B // 2, spatial[-2] // 2, 0), (B - 1, spatial[-2] - 1, 0), (0, 1, -1),
                                       (B // 2, 2, spatial[-1] // 2)]):
        c = (n * 7 + 3) % (planted.shape[1] - 4)
        v = planted[b, c] if len(ks) == 2 else planted[b, c, spatial[0] // 2]
        v[row, col] = value
    got = _update(t["x"], t["z"], h, bias, t["gout"], ks, _lib.FLAG_BF16_PARAMS, relu)
    ref = _update(t["x"], t["z"], h, bias, t["gout"], ks, 0, relu)       # the FMA kernels
    torch.cuda.synchronize()
    assert _lib.load().ndc_wait_expired() == 0
    for name, a, r in zip(("out", "t1", "gx", "gz", "gh", "gb"), got, ref):
        finite = r.isfinite()
        assert torch.equal(a.isfinite(), finite), (name, (a.isfinite() != finite).sum().item())
        assert (a[finite] - r[finite]).abs().max().item() <= 2e-2 * r[finite].abs().max().item(), name
