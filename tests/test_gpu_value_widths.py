"""Splat and slice over value rows of every width class, against the oracle.

Lanes of a splat window (2, 4, 8, 16, 32; in double 1 too) and the slice's row width change at the vd below and beside each of
them; a channel count that is a multiple of four leaves the homogeneous channel a quad of its own.  The bounds are
those of every comparison with the oracle (gpu_helpers): float sums of a few hundred terms in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    import gpu_helpers
    return gpu_helpers


CHANNELS = [1, 2, 3, 4, 5, 7, 8, 11, 12, 15, 16, 19, 20, 21, 23, 24, 27, 28, 31, 32, 33, 47, 63, 64, 127, 130]


@pytest.mark.parametrize("shape,r", [((35, 32), 3), ((18, 33), 3), ((19, 21), 1), ((301,), 2), ((5, 9, 11), 3)])
def test_every_width_class(shape, r, gpu, oracle):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(41)
    ref = rng.random((2,) + shape + (r,), dtype=np.float32)
    wide = rng.standard_normal((2,) + shape + (CHANNELS[-1],)).astype(np.float32)
    wants = [oracle.lattice_filter(wide, ref, True, 4.0, 0.2, 1.0, reverse) for reverse in (False, True)]
    rt = torch.from_numpy(ref).cuda()
    lattice = plb.Lattice(rt, None, True, 4.0, 0.2, max_channels=CHANNELS[-1])
    for c in CHANNELS:
        x = torch.from_numpy(np.ascontiguousarray(wide[..., :c])).cuda()
        for reverse in (False, True):
            got = plb.lattice_filter(x, rt, True, 4.0, 0.2, reverse=reverse).cpu().numpy()
            gpu.assert_outputs_close(got, wants[reverse][..., :c], "%d channels" % c)
            got = lattice.apply(x, reverse).cpu().numpy()
            gpu.assert_outputs_close(got, wants[reverse][..., :c], "%d channels, lattice kept" % c)


@pytest.mark.parametrize("pd,n", [(16, 301), (8, 515), (7, 300), (1, 700)])
def test_widths_on_the_positions_path(pd, n, gpu, oracle):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(43)
    pos = (rng.standard_normal((2, n, pd)) * 1.2).astype(np.float32)
    wide = rng.standard_normal((2, n, 70)).astype(np.float32)
    want = np.stack([oracle.filter(wide[i], pos[i], structure=False).out for i in range(2)])
    for c in (3, 4, 6, 8, 10, 13, 17, 22, 26, 30, 40, 70):
        x = torch.from_numpy(np.ascontiguousarray(wide[..., :c])).cuda()
        got = plb.filter_positions(x, torch.from_numpy(pos).cuda())[0].cpu().numpy()
        gpu.assert_outputs_close(got, want[..., :c], "pd %d, %d channels" % (pd, c))


def test_rows_that_do_not_start_on_sixteen_bytes(gpu, oracle):
    """An input that begins four bytes into its allocation is staged by 4-byte copies at every width."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(47)
    shape = (1, 20, 32)
    ref = rng.random(shape + (3,), dtype=np.float32)
    rt = torch.from_numpy(ref).cuda()
    for c in (3, 4, 10, 21, 31):
        inp = rng.standard_normal(shape + (c,)).astype(np.float32)
        flat = torch.empty(inp.size + 1, device="cuda")
        x = flat[1:].view(inp.shape)
        x.copy_(torch.from_numpy(inp))
        out, _, _ = plb.lattice_filter_raw(x, rt, True, 4.0, 0.2, out=torch.empty(inp.size + 1, device="cuda")[1:].view(inp.shape))
        gpu.assert_outputs_close(out.cpu().numpy(), oracle.lattice_filter(inp, ref, True, 4.0, 0.2), "%d channels" % c)


@pytest.mark.parametrize("shape,r", [((35, 32), 3), ((18, 33), 3), ((301,), 2)])
def test_every_width_class_in_double(shape, r, gpu, oracle):
    """Rows of 1 to 32 pairs and beyond; blocks of 32 doubles, the last of them with the homogeneous channel alone."""
    import torch
    import permutohedral_lattice_b200 as plb
    from conftest import rel_l2
    rng = np.random.default_rng(67)
    ref = rng.random((2,) + shape + (r,))
    wide = rng.standard_normal((2,) + shape + (130,))
    rt = torch.from_numpy(ref).cuda()
    for reverse in (False, True):
        want = oracle.lattice_filter(wide, ref, True, 4.0, float(np.float32(0.2)), 1.0, reverse, dtype=np.float64)
        for c in (1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 21, 31, 32, 33, 40, 62, 63, 64, 65, 96, 130):
            x = torch.from_numpy(np.ascontiguousarray(wide[..., :c])).cuda()
            got = plb.lattice_filter(x, rt, True, 4.0, 0.2, reverse=reverse).cpu().numpy()
            # double sums in another order: the bound of every comparison in double with the oracle
            assert rel_l2(got, want[..., :c]) <= 1e-12, "%d channels" % c


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3, 1e30])
@pytest.mark.parametrize("shape,r", [((35, 32), 3), ((18, 33), 3), ((5, 9, 11), 1)])
def test_fixed_point_sums_at_every_width(shape, r, scale, gpu, oracle):
    """The deterministic mode at every lane count: identical bits from run to run and through a kept lattice."""
    import torch
    import permutohedral_lattice_b200 as plb
    from conftest import bits
    rng = np.random.default_rng(71)
    ref = rng.random((2,) + shape + (r,), dtype=np.float32)
    wide = (scale * rng.standard_normal((2,) + shape + (70,))).astype(np.float32)
    rt = torch.from_numpy(ref).cuda()
    for c in (1, 3, 4, 6, 8, 13, 21, 30, 40, 70):
        inp = np.ascontiguousarray(wide[..., :c])
        x = torch.from_numpy(inp).cuda()
        got = plb.lattice_filter(x, rt, True, 4.0, 0.2, mode="deterministic").cpu().numpy()
        again = plb.lattice_filter(x, rt, True, 4.0, 0.2, mode="deterministic").cpu().numpy()
        kept = plb.Lattice(rt, None, True, 4.0, 0.2, max_channels=c, mode="deterministic").apply(
            x, mode="deterministic").cpu().numpy()
        assert np.array_equal(bits(got), bits(again)) and np.array_equal(bits(got), bits(kept))
        if scale <= 1e3:
            # the grid, 2^-36 of at most 8e3, is 1e-7 of the weights and finer than that of the values
            gpu.assert_outputs_close(got / scale, oracle.lattice_filter(inp, ref, True, 4.0, 0.2) / scale, "%d channels" % c)


def test_grid_follows_the_largest_value_wherever_it_lies(gpu):
    """The largest magnitude among the floats before the first 16-byte boundary, in the vector loads or after the last
    one: a grid too fine for it would overflow the sums, one too coarse lose the constant 1 around it."""
    import torch
    import permutohedral_lattice_b200 as plb
    ref = torch.zeros((1, 16, 19, 1), device="cuda")
    for offset in (0, 1, 2, 3):
        for where in (0, 1, 3, 4, 150, 299, 300, 301, 302, 303):
            flat = torch.ones(16 * 19 + offset, device="cuda")
            x = flat[offset:].view(1, 16, 19, 1)
            x.view(-1)[where] = -1e30
            out, ws, _ = plb.lattice_filter_raw(x, ref, True, 4.0, 0.2, mode="deterministic")
            bits = int(ws[16:20].view(torch.int32).item())      # the header's word for the largest magnitude
            assert bits == int(np.float32(1e30).view(np.int32)), (offset, where)


@pytest.mark.parametrize("pd,atomic,deterministic", [(4, 176, 185), (5, 172, 182), (8, 160, 173), (16, 328, 349)])
def test_widest_rows_taken_and_first_refused(pd, atomic, deterministic, gpu, oracle):
    """The splat stage's limits on the value dimension, which have not moved since its first kernels."""
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    rng = np.random.default_rng(103)
    pos = rng.standard_normal((1, 300, pd)).astype(np.float32)
    pt = torch.from_numpy(pos).cuda()
    for mode, widest in (("atomic", atomic), ("deterministic", deterministic)):
        val = rng.random((1, 300, widest - 1), dtype=np.float32)
        got = plb.filter_positions(torch.from_numpy(val).cuda(), pt, mode=mode)[0].cpu().numpy()
        gpu.assert_outputs_close(got[0], oracle.filter(val[0], pos[0], structure=False).out, "%s, vd %d" % (mode, widest))
        with pytest.raises(plb.PlError) as err:
            plb.filter_positions(torch.rand((1, 300, widest), device="cuda"), pt, mode=mode)
        assert err.value.status == capi.PL_UNSUPPORTED_DIMS
