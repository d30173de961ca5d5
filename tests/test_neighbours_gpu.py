"""The native nodes around the layer (1x1 projection, bias + GELU, instance norm): every combination
of gradients asked for, parameters of another type, no positions, autocast, double backward."""

import itertools

import pytest
import torch
import torch.nn.functional as F
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.autograd import forward_ad

import deconver_b200 as dcb
from conftest import max_norm_error

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _norm(x, w, b):
    y = F.instance_norm(x.double())
    y = y if w is None else y * w.double().view(1, -1, 1)
    return y if b is None else y + b.double().view(1, -1, 1)


def _linear(x, w, b):
    return F.conv1d(x.double(), w.double(), None if b is None else b.double())


def _gelu(x, b):
    return F.gelu(x.double() if b is None else x.double() + b.double().view(1, -1, 1))


def _run_linear(x, w, b):
    m = dcb.Linear(w.shape[1], w.shape[0], bias=b is not None)
    del m.linear.weight, m.linear.bias
    m.linear.weight, m.linear.bias = w, b
    return m(x)


OPS = {"norm": (dcb.instance_norm, _norm, [(6,), (6,)]), "linear": (_run_linear, _linear, [(10, 6, 1), (10,)]),
       "gelu": (dcb.bias_gelu, _gelu, [(6,)])}


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-3), (torch.bfloat16, 2e-2)], ids=["f32", "bf16"])
@pytest.mark.parametrize("op", OPS)
def test_partial_gradients(op, dtype, tol):
    mine, ref, shapes = OPS[op]
    gen = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(2, 6, 37, device=DEV, generator=gen).to(dtype)
    ps = [torch.randn(s, device=DEV, generator=gen).to(dtype) for s in shapes]
    for mask in itertools.product([0, 1, 2], repeat=1 + len(ps)):   # 0 constant, 1 gradient, 2 absent
        if mask[0] == 2 or (op == "linear" and mask[1] == 2) or 1 not in mask:
            continue
        res = []
        for f in (mine, ref):
            t = [None if m == 2 else v.clone().requires_grad_(m == 1) for v, m in zip([x] + ps, mask)]
            y = f(*t)
            y.backward(torch.cos(torch.arange(y.numel(), device=DEV)).view(y.shape).to(y.dtype))
            res.append([y.detach()] + [v.grad for v in t if v is not None])
        for a, r in zip(*res):
            assert (a is None) == (r is None)
            if a is not None:
                assert a.dtype == dtype
                assert max_norm_error(a.double().cpu().numpy(), r.double().cpu().numpy()) < tol, mask


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("shape", [(0, 6, 5), (2, 6, 0)])
def test_no_positions(op, shape):
    mine, _, shapes = OPS[op]
    t = [torch.ones(s, device=DEV, requires_grad=True) for s in [shape] + shapes]
    y = mine(*t)
    y.sum().backward()
    assert y.shape[0] == shape[0] and y.shape[2:] == shape[2:]
    assert all(v.grad is not None and not v.grad.any() for v in t)


def test_parameters_of_another_type():
    x = torch.randn(2, 6, 9, device=DEV).bfloat16().requires_grad_(True)
    b = torch.randn(6, device=DEV, requires_grad=True)
    dcb.bias_gelu(x, b).sum().backward()
    dcb.instance_norm(x, b, b.detach()).sum().backward()
    assert b.grad.dtype == torch.float32 and x.grad.dtype == torch.bfloat16


@pytest.mark.parametrize("op", OPS)
def test_double_backward_is_refused(op):
    mine, _, shapes = OPS[op]
    t = [torch.randn(s, device=DEV, requires_grad=True) for s in [(2, 6, 8)] + shapes]
    g = torch.ones_like(mine(*t), requires_grad=True)
    (gx,) = torch.autograd.grad(mine(*t), t[0], g, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        gx.sum().backward()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_autocast(dtype):
    mlp = dcb.MLP(6).to(DEV)
    x = torch.randn(2, 6, 4, 8, device=DEV, dtype=dtype, requires_grad=True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = mlp(x)
    y.float().sum().backward()
    assert y.dtype == torch.bfloat16 and x.grad.dtype == dtype
    assert all(p.grad is not None and p.grad.dtype == torch.float32 for p in mlp.parameters())
    assert max_norm_error(y.detach().float().cpu().numpy(), mlp.cpu()(x.detach().float().cpu()).detach().numpy()) < 2e-2


MODULES = {"linear": lambda: dcb.Linear(6, 10), "mlp": lambda: dcb.MLP(6), "norm": lambda: dcb.InstanceNorm2d(6, affine=True),
           "deconv": lambda: dcb.Deconv(6, (3, 3), ratio=4, num_iters=2)}


@pytest.mark.parametrize("module", MODULES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_tensors_without_memory_are_refused(module, dtype):
    net, x = MODULES[module]().to(DEV, dtype), torch.rand(2, 6, 4, 8, device=DEV).to(dtype)
    with FakeTensorMode(allow_non_fake_inputs=True) as mode, pytest.raises(RuntimeError, match="memory|NULL"):
        net(mode.from_tensor(x))


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("module", MODULES)
def test_tangents_are_refused(module, grad):
    """Not dropped, whether or not anything asks for a gradient."""
    net, x = MODULES[module]().to(DEV), torch.rand(2, 6, 4, 8, device=DEV)
    net.requires_grad_(grad)
    with forward_ad.dual_level():
        with pytest.raises(RuntimeError, match="forward-mode|jvp"):
            net(forward_ad.make_dual(x, torch.ones_like(x)))
        p = next(net.parameters())
        with torch.no_grad(), pytest.raises(RuntimeError, match="forward-mode|jvp"):
            torch.func.functional_call(net, {next(iter(net.state_dict())): forward_ad.make_dual(p, torch.ones_like(p))}, x)


@pytest.mark.filterwarnings("ignore::DeprecationWarning", "ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("module", MODULES)
def test_traced_modules_compute_what_the_modules_do(module, grad):
    net, (x, y) = MODULES[module]().to(DEV), torch.rand(2, 2, 6, 4, 8, device=DEV)
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(net, (x,))
        assert torch.equal(traced(y), net(y))
    if grad:
        res = []
        for f in (traced, net):
            t = y.clone().requires_grad_(True)
            net.zero_grad(set_to_none=True)
            f(t).square().sum().backward()
            res.append([t.grad] + [p.grad for p in net.parameters()])
        assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("module", MODULES)
def test_tensor_subclasses_stay(module):
    class Tagged(torch.Tensor):
        pass

    net, x = MODULES[module]().to(DEV), torch.rand(2, 6, 4, 8, device=DEV, requires_grad=True)
    y = net(x.as_subclass(Tagged))
    assert type(y) is Tagged and torch.equal(y.as_subclass(torch.Tensor), net(x))
    y.sum().backward()
    assert x.grad is not None


def test_wrapped_submodules():
    """As sharding and checkpointing wrappers do: a module of another structure that passes attributes on."""
    class Wrapper(torch.nn.Module):
        def __init__(self, module):
            super().__init__()
            self.wrapped = module

        def __getattr__(self, name):
            try:
                return super().__getattr__(name)
            except AttributeError:
                return getattr(self.wrapped, name)

    net, x = MODULES["deconv"]().to(DEV), torch.rand(2, 6, 4, 8, device=DEV)
    want = net(x)
    net.init.linear = Wrapper(net.init.linear)
    assert torch.equal(net(x), want)
    net.init = Wrapper(net.init)
    assert torch.equal(net(x), want)
