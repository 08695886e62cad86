"""Which calls of lattice_filter reach torch as one call of its autograd function.  The kernels go through ctypes,
unseen by torch; here a stand-in does the same on the CPU (numpy on the tensors' memory), so no GPU is needed."""
import sys

import pytest
import torch

import permutohedral_lattice_b200 as plb

lf = sys.modules["permutohedral_lattice_b200.lattice_filter"]   # (the package re-exports a function of that name)


def _double_unseen(x):
    out = torch.empty_like(x.contiguous())
    out.detach().numpy()[...] = 2.0 * x.detach().numpy()
    return out


class _LatticeStandIn:
    def __init__(self, *args, **kw):
        pass

    def apply(self, x, reverse=False, mode="atomic", out=None):
        return _double_unseen(x)


@pytest.fixture(params=[False, True], ids=["rebuild", "reuse"])
def reuse(request, monkeypatch):
    monkeypatch.setattr(lf, "lattice_filter_raw", lambda x, *a, **kw: (_double_unseen(x), None, None))
    monkeypatch.setattr(lf, "Lattice", _LatticeStandIn)
    return request.param


def _x(seed=0):
    return torch.rand((1, 4, 5, 3), generator=torch.Generator().manual_seed(seed))


def test_traced_call_computes_the_filter(reuse):
    x, ref, other = _x(), _x(1), _x(2)
    traced = torch.jit.trace(lambda a, b: plb.lattice_filter(a, b, reuse_lattice=reuse), (x, ref), check_trace=False)
    assert torch.equal(traced(other, ref), 2.0 * other)


def test_forward_mode_is_refused(reuse):
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(_x(), torch.ones(1, 4, 5, 3))
        with pytest.raises(NotImplementedError):
            plb.lattice_filter(dual, _x(1), reuse_lattice=reuse)


@pytest.mark.parametrize("transform", ["jvp", "vmap"])
def test_functorch_transforms_are_refused(reuse, transform):
    ref = _x(1)

    def call(x):
        return plb.lattice_filter(x, ref, reuse_lattice=reuse)

    with pytest.raises(RuntimeError, match="autograd.Function"):
        if transform == "jvp":
            torch.func.jvp(call, (_x(),), (_x(),))
        else:
            torch.func.vmap(call)(torch.stack([_x(), _x(2)]))


@pytest.mark.parametrize("grad", [False, True])
def test_plain_calls(reuse, grad):
    x = _x().requires_grad_(grad)
    out = plb.lattice_filter(x, _x(1), reuse_lattice=reuse)
    assert torch.equal(out.detach(), 2.0 * x.detach())
    assert (out.grad_fn is not None) == grad
    if grad:
        out.sum().backward()
        assert torch.equal(x.grad, torch.full_like(x, 2.0))
