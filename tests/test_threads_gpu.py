"""Updates of several host threads, each on a stream of its own, whose kernels are instances of one template with different
amounts of shared memory: what one thread allows a kernel has to be enough for the others."""

import threading

import pytest
import torch

from deconver_b200 import _lib

pytestmark = pytest.mark.gpu

# two geometries each that run on the same instances, with more than 48 KB of shared memory: grouped, marching, tensor cores
PAIRS = {
    "grouped": (torch.float32, [(1, 16, 8, (3, 3, 3), 1, (8, 16, 32)), (1, 14, 8, (3, 3, 3), 1, (8, 16, 32))]),
    "grouped_ragged": (torch.float32, [(2, 2, 8, (3, 3, 3), 1, (9, 40, 33)), (2, 2, 8, (3, 3, 3), 1, (9, 40, 21))]),
    "marching": (torch.float32, [(4, 1, 4, (5, 5), 8, (40, 52)), (4, 1, 4, (5, 5), 8, (40, 36))]),
    "tensor": (torch.bfloat16, [(24, 1, 4, (3, 3, 3), 1, (32, 32, 32)), (24, 1, 4, (3, 3, 3), 1, (32, 40, 24))]),
}


def _problem(case, dtype):
    G, m, sc, ks, B, spatial = case
    desc = _lib.make_desc(B, G, m, sc, spatial, ks, 1e-16, True, _lib.NDC_BF16 if dtype == torch.bfloat16 else _lib.NDC_F32,
                          _lib.FLAG_BF16_PARAMS if dtype == torch.bfloat16 else 0)
    gen = torch.Generator(device="cuda").manual_seed(sum(spatial))
    x = torch.rand(B, G * m, *spatial, device="cuda", generator=gen).to(dtype)
    z = torch.rand(B, G * sc, *spatial, device="cuda", generator=gen).to(dtype)
    h = torch.rand(G * m, sc, *ks, device="cuda", generator=gen).bfloat16().float()
    bias = torch.zeros(G * sc, device="cuda")
    return desc, x, z, h, bias


def _step(problem, stream):
    """Forward and backward; the outputs and the statuses."""
    lib = _lib.load()
    desc, x, z, h, bias = problem
    with torch.cuda.stream(stream):
        out, t1, gx, gz, gh, gb = (torch.empty_like(v) for v in (z, x, x, z, h, bias))
        need = lib.ndc_bwd_workspace_bytes(desc)
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    st = stream.cuda_stream
    codes = [lib.ndc_fwd(desc, x.data_ptr(), z.data_ptr(), h.data_ptr(), bias.data_ptr(), out.data_ptr(), t1.data_ptr(), st),
             lib.ndc_bwd(desc, x.data_ptr(), z.data_ptr(), t1.data_ptr(), h.data_ptr(), bias.data_ptr(), z.data_ptr(),
                         gx.data_ptr(), gz.data_ptr(), gh.data_ptr(), gb.data_ptr(), ws.data_ptr(), need, st)]
    return codes, (out, gx, gz, gh, gb)


@pytest.mark.parametrize("kind", PAIRS)
def test_two_geometries_at_once(kind):
    dtype, cases = PAIRS[kind]
    problems = [_problem(c, dtype) for c in cases]
    alone = [_step(p, torch.cuda.current_stream()) for p in problems]
    torch.cuda.synchronize()
    assert all(c == _lib.NDC_OK for codes, _ in alone for c in codes)
    failed, last = [], [None] * 4

    def work(i):
        stream = torch.cuda.Stream()
        for _ in range(400):
            codes, last[i] = _step(problems[i % 2], stream)
            failed.extend(c for c in codes if c != _lib.NDC_OK)
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, (len(failed), _lib.load().ndc_status_string(failed[0]))
    for i, res in enumerate(last):
        assert all(torch.equal(a, b) for a, b in zip(res, alone[i % 2][1]))
