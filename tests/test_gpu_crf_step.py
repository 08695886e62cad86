"""pl_crf_step_f32 against the two applies and pl_crf_update_f32 that it stands for: every row width, even and odd numbers of
labels, ragged images whose rows are not multiples of 16 bytes, lattices with the one-cluster blur and with wide passes,
and what it leaves to the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plb():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    import permutohedral_lattice_b200
    return permutohedral_lattice_b200


def _case(plb, shape, labels, channels=3, theta=(12.0, 0.1, 2.0), **kw):
    import torch
    g = torch.Generator().manual_seed(sum(shape) + labels)
    coarse = torch.rand(shape[:1] + tuple(-(-s // 8) for s in shape[1:]) + (channels,), generator=g)
    image = coarse
    for d in range(1, len(shape)):
        image = image.repeat_interleave(8, d).narrow(d, 0, shape[d])
    image = (image + 0.03 * torch.randn(image.shape, generator=g)).contiguous().cuda()
    crf = plb.DenseCRF(image, labels, *theta, bilateral_weight=1.5, spatial_weight=0.75, **kw)
    u = (3.0 * torch.randn(shape + (labels,), generator=g)).cuda()
    return crf, torch.softmax(-u, -1), u


def _apart(crf, q, u):
    """The same step as separate calls."""
    import torch
    m = 1.5 * crf.bilateral.apply(q).double() + 0.75 * crf.spatial.apply(q).double()
    compat = 1.0 - torch.eye(q.shape[-1], device="cuda", dtype=torch.float64)
    return torch.softmax(-u.double() - m @ compat, -1)


@pytest.mark.parametrize("labels", [4, 7, 8, 11, 12, 15, 16, 19, 20, 21, 22, 23, 27, 28, 31])
@pytest.mark.parametrize("shape", [(1, 37, 51), (2, 96, 128)])
def test_step_is_the_two_filters_and_the_update(plb, labels, shape):
    crf, q, u = _case(plb, shape, labels)
    got = crf._fused_step(q, u)
    want = _apart(crf, q, u)
    # float sums of some hundred products in another order, then an exponential of numbers up to about 15
    assert got is not None and float((got - want).abs().max()) <= 2e-5
    assert float((got.sum(-1) - 1).abs().max()) <= 1e-5


@pytest.mark.parametrize("theta", [(60.0, 0.3, 30.0), (12.0, 0.1, 2.0), (1.5, 0.02, 0.4)])
def test_step_through_lattices_of_any_size(plb, theta):
    """One-cluster blurs, wide ones, tiles with more entries than the staged rows."""
    for shape in ((1, 40, 44), (3, 130, 90)):
        crf, q, u = _case(plb, shape, 21, theta=theta)
        want = _apart(crf, q, u)
        assert float((crf.step(q, u) - want).abs().max()) <= 2e-5


@pytest.mark.parametrize("shape,labels", [((1, 500, 500), 21), ((1, 700, 700), 21), ((2, 700, 700), 8)])
def test_step_with_passes_together_and_one_after_the_other(plb, shape, labels):
    """Noisy images: bounds of the worst case, 14, 26 and 26 million pieces of 16 bytes in both lattices."""
    crf, q, u = _case(plb, shape, labels, theta=(1.5, 0.02, 0.4))
    got = crf._fused_step(q, u)
    assert float((got - _apart(crf, q, u)).abs().max()) <= 2e-5


def test_steps_that_are_left_to_the_separate_calls(plb):
    import torch
    for shape, labels, channels in (((1, 30, 30), 3, 3), ((1, 30, 30), 32, 3), ((1, 30, 30), 5, 1), ((1, 9, 12, 14), 5, 1)):
        crf, q, u = _case(plb, shape, labels, channels)
        assert crf._fused_step(q, u) is None
        assert float((crf.step(q, u) - _apart(crf, q, u)).abs().max()) <= 2e-5
    crf, q, u = _case(plb, (1, 30, 30), 5, compatibility=torch.rand((5, 5)))
    assert torch.isfinite(crf.step(q, u)).all()


def test_step_through_a_failed_lattice_is_nan_and_bad_shapes_are_refused(plb):
    import torch
    from permutohedral_lattice_b200 import capi
    crf, q, u = _case(plb, (1, 64, 64), 6)
    with pytest.raises(ValueError):
        crf.step(q[:, :32], u[:, :32])
    with pytest.raises(TypeError):
        crf.step(q.double(), u)
    crf.spatial.workspace[8:12] = torch.tensor([1 << capi.PL_CAPACITY_EXCEEDED, 0, 0, 0], dtype=torch.uint8, device="cuda")
    assert torch.isnan(crf.step(q, u)).all()


@pytest.mark.parametrize("n_points,labels", [(1, 1), (255, 2), (257, 21), (1000, 32), (130, 33), (129, 128), (40, 129)])
def test_inference_starts_from_the_softmax_of_the_unaries(plb, n_points, labels):
    import torch
    g = torch.Generator().manual_seed(labels)
    u = (5.0 * torch.randn((1, n_points, labels), generator=g)).cuda()
    want = torch.softmax(-u.double(), -1)
    for x in (u, u.transpose(0, 1).contiguous().transpose(0, 1)):
        q = plb.DenseCRF._start(x)
        assert q.shape == u.shape and float((q - want).abs().max()) <= 1e-6      # an exponential and a quotient
    assert torch.equal(plb.DenseCRF._start(u.cpu()), torch.softmax(-u.cpu(), -1))
    assert plb.DenseCRF._start(u.double()).dtype == torch.float64
    assert plb.DenseCRF._start(u[:, :0]).numel() == 0


def test_inference_starts_from_torchs_softmax_where_torch_follows_the_unaries(plb):
    """Forward mode, vmap, jvp and tracers used to go through torch.softmax: none of them sees a kernel launched by ctypes."""
    import torch
    from torch.autograd import forward_ad
    g = torch.Generator().manual_seed(7)
    u, v, t = (torch.randn((1, 6, 7, 5), generator=g).cuda() for _ in range(3))
    start = plb.DenseCRF._start

    def softmax(x):
        return torch.softmax(-x, -1)

    with forward_ad.dual_level():
        q = forward_ad.unpack_dual(start(forward_ad.make_dual(u, t)))
        want = forward_ad.unpack_dual(softmax(forward_ad.make_dual(u, t)))
        assert torch.equal(q.primal, want.primal) and torch.equal(q.tangent, want.tangent)
    assert torch.equal(torch.func.vmap(start)(torch.stack([u, v])), softmax(torch.stack([u, v])))
    got, want = torch.func.jvp(start, (u,), (t,)), torch.func.jvp(softmax, (u,), (t,))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    traced = torch.jit.trace(start, (u,), check_trace=False)
    assert torch.equal(traced(v), softmax(v))
    crf, _, unaries = _case(plb, (1, 30, 30), 5)
    assert torch.equal(torch.func.vmap(lambda x: crf.infer(x, 0))(unaries[None]), softmax(unaries)[None])
