"""The index of small lattices in shared memory and their blur in clusters, around the sizes where the wide kernels take over:
by the bound on the entries (10240; pd 4 and 5 9216 where that is the worst case) for the index; for the blur 1, 2 and 4 vertices a thread of a cluster (bounds of 8192,
16384, 32768; where the bound is the worst case 1 and 2) and the number of clusters, one for 16 bytes of a row (64, which
only rows of doubles reach; beyond 8192 entries 16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOST = 10240


@pytest.fixture(scope="module")
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    import gpu_helpers
    return gpu_helpers


@pytest.mark.parametrize("pd", [1, 2, 3, 4, 5, 6, 7, 8, 16])
@pytest.mark.parametrize("spread", [0.4, 60.0])      # many equal keys; none
@pytest.mark.parametrize("bound,batch", [(MOST, 1), (MOST + 1, 1), (1021, 2)])
def test_index_around_its_largest_bound(pd, spread, bound, batch, gpu, oracle):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(79)
    n = min(bound, MOST) // (pd + 1) // batch        # as many entries as the bound allows, if all keys are distinct
    pos = (rng.standard_normal((batch, n, pd)) * spread).astype(np.float32)
    val = rng.random((batch, n, 2), dtype=np.float32)
    pt, xt = torch.from_numpy(pos).cuda(), torch.from_numpy(val).cuda()
    items = [oracle.filter(val[i], pos[i]) for i in range(batch)]
    info = {}
    out, ws = plb.filter_positions(xt, pt, max_entries=bound, info=info)
    st = plb.lattice_stats(ws)
    vk, vi, pv, pw = plb.export_lattice(ws, st, batch, n, pd, 3, positions=pt)
    gpu.assert_structure_equal(vk, vi, pv, pw, items, "pd %d" % pd)
    gpu.assert_outputs_close(out.cpu().numpy(), np.stack([o.out for o in items]), "pd %d" % pd)


@pytest.mark.parametrize("pd", [2, 4, 5, 8])
@pytest.mark.parametrize("bound,twice", [(9216, False), (9217, False), (MOST, True)])
def test_index_with_its_table_at_its_fullest(pd, bound, twice, gpu, oracle):
    """All keys distinct: as many entries as the bound has room for, of the worst case or (every point twice) of half of it."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(81)
    n = bound // (pd + 1)
    pos = (rng.standard_normal((1, n, pd)) * 60).astype(np.float32)
    if twice:
        pos = np.repeat(pos, 2, 1)
    val = rng.random((1, pos.shape[1], 2), dtype=np.float32)
    pt, xt = torch.from_numpy(pos).cuda(), torch.from_numpy(val).cuda()
    item = oracle.filter(val[0], pos[0])
    out, ws = plb.filter_positions(xt, pt, max_entries=bound)
    st = plb.lattice_stats(ws)
    vk, vi, pv, pw = plb.export_lattice(ws, st, 1, pos.shape[1], pd, 3, positions=pt)
    gpu.assert_structure_equal(vk, vi, pv, pw, [item], "pd %d" % pd)
    gpu.assert_outputs_close(out.cpu().numpy(), item.out[None], "pd %d" % pd)


@pytest.mark.parametrize("bound,channels", [(2048, 127), (2048, 130), (8192, 3), (8192, 16), (8193, 63), (8193, 64), (16384, 7),
                                            (16385, 3), (32768, 12), (32769, 12)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_blur_around_its_limits(bound, channels, dtype, gpu, oracle):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(83)
    for pd, reverse in ((2, True), (5, False)):       # an odd and an even number of passes
        n = bound // (pd + 1)                         # distinct keys: nearly as many vertices as the bound
        pos = (rng.standard_normal((1, n, pd)) * 60).astype(dtype)
        val = rng.random((1, n, channels)).astype(dtype)
        out, _ = plb.filter_positions(torch.from_numpy(val).cuda(), torch.from_numpy(pos).cuda(), reverse=reverse,
                                      max_entries=bound)
        want = oracle.filter(val[0], pos[0], reverse=reverse, dtype=np.dtype(dtype).type).out
        # 32-bit sums of some tens of products in another order, as elsewhere; in 64 bits the same, 2^29 times finer
        rel = np.linalg.norm(out[0].cpu().numpy() - want) / np.linalg.norm(want)
        assert rel <= (1e-5 if dtype == "float32" else 1e-12), (pd, rel)


@pytest.mark.parametrize("bound,channels", [(8193, 3), (8193, 63), (16384, 7), (16385, 3), (32768, 12), (32769, 12)])
@pytest.mark.parametrize("pd", [2, 5, 16])
def test_blur_of_bounds_below_the_worst_case(bound, channels, pd, gpu):
    """Every point twice: a bound of half the worst case, all of it vertices.  The bits of a lattice with room for the worst."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(97)
    n = bound // (pd + 1)
    pos = torch.from_numpy(np.repeat((rng.standard_normal((1, n, pd)) * 60).astype(np.float32), 2, 1)).cuda()
    x = torch.from_numpy(rng.random((1, 2 * n, channels), dtype=np.float32)).cuda()
    for reverse in (False, True):
        got = plb.filter_positions(x, pos, reverse, "deterministic", max_entries=bound)[0].clone()
        want = plb.filter_positions(x, pos, reverse, "deterministic", max_entries=2 * n * (pd + 1))[0]
        assert torch.equal(got, want)


@pytest.mark.parametrize("n", [1500, 2000, 3600])
def test_slice_of_few_tiles_behind_wide_passes(n, gpu, oracle):
    """Fewer tiles than SMs, worst-case bounds beyond the small blur: the slice of wide rows is launched plainly."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(101)
    pos = (rng.standard_normal((1, n, 5)) * 6).astype(np.float32)
    for channels in (5, 21, 33):
        val = rng.random((1, n, channels), dtype=np.float32)
        out, _ = plb.filter_positions(torch.from_numpy(val).cuda(), torch.from_numpy(pos).cuda(), max_entries=0)
        gpu.assert_outputs_close(out.cpu().numpy(), oracle.filter(val[0], pos[0]).out[None], "%d channels" % channels)
        # in double: sums of some tens of products in another order
        out, _ = plb.filter_positions(torch.from_numpy(val).double().cuda(), torch.from_numpy(pos).double().cuda(), max_entries=0)
        want = oracle.filter(val[0].astype(np.float64), pos[0].astype(np.float64), dtype=np.float64).out
        assert np.linalg.norm(out[0].cpu().numpy() - want) / np.linalg.norm(want) <= 1e-12


def test_blur_keeps_infinite_rows_infinite(gpu):
    """An infinite row stays infinite, and other channels stay what they are."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(89)
    for n in (64, 40000):                             # one cluster, wide passes
        pos = torch.from_numpy((rng.standard_normal((1, n, 3)) * 2).astype(np.float32)).cuda()
        x = torch.rand((1, n, 2), device="cuda")
        x[0, 0, 0] = float("inf")
        out, _ = plb.filter_positions(x, pos)
        plain, _ = plb.filter_positions(torch.rand((1, n, 2), device="cuda").copy_(x).nan_to_num_(posinf=0.5), pos)
        assert torch.isposinf(out[0, 0, 0]) and not torch.isnan(out[..., 0]).any()
        assert torch.isfinite(out[..., 1]).all() and torch.allclose(out[..., 1], plain[..., 1], rtol=1e-4, atol=1e-5)
