"""Which calls of lattice_filter take the short way through the host: only those whose reference a verified call of the kind
has just used, as lattice_filter_raw would find out by looking it up.  Every other one goes through lattice_filter_raw, and
both give the bits of a call sized for the worst case."""
import sys

import pytest

pytestmark = pytest.mark.gpu

ARGS = (True, 5.0, 0.1875, 1.0)      # floats: lattice_filter rounds the thetas, lattice_filter_raw does not


class Watched:
    """lattice_filter in the deterministic mode, compared with the worst case; `long`: calls of lattice_filter_raw so far."""

    def __init__(self, lf, plb, monkeypatch):
        self.raw, self.filter, self.long = lf.lattice_filter_raw, plb.lattice_filter, 0

        def raw(*args, **kw):
            self.long += 1
            return self.raw(*args, **kw)

        monkeypatch.setattr(lf, "lattice_filter_raw", raw)

    def way(self, x, ref, args=ARGS, reverse=False, mode="deterministic"):
        import torch
        before = self.long
        got = self.filter(x, ref, *args, reverse=reverse, mode=mode)
        way = "long" if self.long > before else "short"
        own = torch.empty(1 << 28, dtype=torch.uint8, device=x.device)      # (not the stream's workspace)
        want = self.raw(x, ref, *args, reverse=reverse, mode=mode, max_entries=0, workspace=own)[0]
        if mode == "deterministic":
            assert torch.equal(got, want)
        else:
            assert float((got - want).norm() / want.norm()) <= (1e-12 if x.dtype == torch.float64 else 1e-5)
        return way


@pytest.fixture()
def lf():
    """The module, without memory of earlier calls."""
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    import permutohedral_lattice_b200 as plb
    module = sys.modules["permutohedral_lattice_b200.lattice_filter"]   # (the package re-exports a function of that name)
    saved = dict(module._entries_per_item)
    module._entries_per_item.clear()
    plb.release_workspaces()
    yield module
    module._entries_per_item.clear()
    module._entries_per_item.update(saved)
    plb.release_workspaces()


@pytest.fixture()
def watched(lf, monkeypatch):
    import permutohedral_lattice_b200 as plb
    return Watched(lf, plb, monkeypatch)


def _data(c=4, batch=2, shape=(48, 44), seed=1, noise=False):
    import torch
    g = torch.Generator().manual_seed(seed)
    coarse = torch.rand((batch, -(-shape[0] // 8), -(-shape[1] // 8), 3), generator=g)
    ref = coarse.repeat_interleave(8, 1).repeat_interleave(8, 2)[:, :shape[0], :shape[1]].contiguous()
    if noise:
        ref = torch.rand(ref.shape, generator=g)
    return torch.randn((batch,) + shape + (c,), generator=g).cuda(), ref.cuda()


def test_the_same_reference(watched):
    x, ref = _data()
    assert watched.way(x, ref) == "long"
    assert watched.way(x, ref) == "short"
    assert watched.way(x + 1, ref, reverse=True) == "short"
    assert watched.way(x, ref, args=(True, 5.0, 0.25, 1.0)) == "long"
    assert watched.way(x, None, args=(False, 1.0, 1.0, 2.0)) == "long"
    assert watched.way(x, None, args=(False, 1.0, 1.0, 2.0)) == "short"
    assert watched.way(x[:1], None, args=(False, 1.0, 1.0, 2.0)) == "long"       # another batch


def test_a_reference_written_to_in_place(watched, lf):
    x, ref = _data()
    other = _data(seed=2, noise=True)[1]
    assert watched.way(x, ref) == "long" and watched.way(x, ref) == "short"
    ref.copy_(other)                     # needs several times the entries: unverified it would end in NaN
    assert watched.way(x, ref) == "long"
    assert watched.way(x, ref) == "short"


def test_another_tensor_in_the_memory_of_the_reference(watched):
    x, ref = _data()
    noise = _data(seed=2, noise=True)[1]
    flat = ref.new_empty(ref.shape)
    flat.data.copy_(ref)
    where, version = flat.data_ptr(), flat._version
    got = watched.filter(x, flat, *ARGS, mode="deterministic")
    del flat, got
    again = ref.new_empty(ref.shape)
    if again.data_ptr() != where or again._version != version:
        pytest.skip("the allocator gave other memory")
    again.data.copy_(noise)              # without the version counter, as a fresh upload would be
    assert watched.way(x, again) == "long"


def test_another_type_width_mode_or_workspace(watched, lf):
    import permutohedral_lattice_b200 as plb
    x, ref = _data()
    assert watched.way(x, ref) == "long" and watched.way(x, ref) == "short"
    assert watched.way(x.double(), ref.double(), mode="atomic") == "long"
    assert watched.way(x, ref) == "long"                       # (the kind's last reference was another one)
    wide = _data(c=40)[0]
    assert watched.way(wide, ref) == "long"                    # no plan, a larger workspace
    assert watched.way(wide, ref) == "short" and watched.way(x, ref) == "short"
    plb.release_workspaces()
    assert watched.way(x, ref) == "long"                       # a workspace for four channels
    assert watched.way(wide, ref) == "long"                    # too small for forty
    assert watched.way(wide, ref) == "short"
    plb.release_workspaces()
    assert watched.way(x, ref, mode="atomic") == "long"
    assert watched.way(x, ref) == "long"                       # the 64-bit sums have no room yet
    assert watched.way(x, ref) == "short"
    with pytest.raises(TypeError):
        watched.filter(x.double(), ref.double(), *ARGS, mode="deterministic")
    with pytest.raises(KeyError):
        watched.filter(x, ref, *ARGS, mode="no such mode")


def test_strides(watched):
    x, ref = _data()
    assert watched.way(x, ref) == "long" and watched.way(x, ref) == "short"
    assert watched.way(x.transpose(1, 2).contiguous().transpose(1, 2), ref) == "long"
    assert watched.way(x, ref.transpose(1, 2).contiguous().transpose(1, 2)) == "long"


def test_another_stream(watched):
    import torch
    x, ref = _data()
    assert watched.way(x, ref) == "long" and watched.way(x, ref) == "short"
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        assert watched.way(x, ref) == "long"                   # no workspace there yet
        assert watched.way(x, ref) == "short"
        torch.cuda.synchronize()
    assert watched.way(x, ref) == "short"


@pytest.mark.parametrize("expanded", [False, True])
def test_backward_is_the_second_call(watched, expanded):
    import torch
    x, ref = _data()
    x.requires_grad_(True)
    out = watched.filter(x, ref, *ARGS, mode="deterministic")
    assert watched.long == 1
    grad = torch.ones((), device="cuda").expand(out.shape) if expanded else torch.randn_like(out)
    (got,) = torch.autograd.grad(out, x, grad)
    assert watched.long == (2 if expanded else 1)
    want = watched.raw(grad, ref, *ARGS, reverse=True, mode="deterministic", max_entries=0)[0]
    assert torch.equal(got, want)
