"""Spatial-only filters (bilateral=False, src/LatticeFilterKernel.cpp:137-142): the CUDA path locates
vertices by direct indexing instead of hashing.  Same bar as every other case: vertex count, key set,
per-point simplex keys and weights bit-exact against the CPU oracle, outputs within rel-L2 1e-5 /
max-abs 1e-4; and the hashed path (developer switch) must build the identical lattice."""
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


@pytest.fixture
def hashed_path():
    """Turns direct indexing off for one test and restores the previous setting afterwards."""
    from permutohedral_lattice_b200 import capi
    was = capi.lib().pl_debug_direct_index(0)
    yield
    capi.lib().pl_debug_direct_index(was)


# (spatial shape, channels, theta_gamma, direct indexing expected).  The last three are so small or so
# sparse that the dense index (whose bounds carry a fixed margin) outgrows the table region of the
# workspace: the call then hashes, and must give the same results.
CASES = [
    ((64, 48), 4, 3.0, True),        # 2-D image, the CRF smoothness kernel
    ((33, 17), 21, 1.0, True),       # theta_gamma 1: nearly one vertex per point, wide rows
    ((40, 56), 2, 8.0, True),        # coarse lattice
    ((24, 20, 22), 2, 2.0, True),    # volume, pd 3
    ((300,), 1, 5.0, True),          # 1-D signal, pd 1
    ((1, 1), 3, 3.0, True),          # a single point
    ((9, 10, 11), 2, 2.0, False),    # tiny volume
    ((3, 4, 5, 6), 2, 1.5, False),   # four spatial dimensions, a few points each
    ((50, 70), 3, 0.37, False),      # theta_gamma below one: vertices far sparser than the index
]


@pytest.mark.parametrize("shape,c,tg,direct", CASES)
def test_spatial_only_matches_oracle(shape, c, tg, direct, gpu, oracle):
    rng = np.random.default_rng(5)
    inp = rng.standard_normal((2,) + shape + (c,)).astype(np.float32)
    for reverse in (False, True):
        want, items = oracle.lattice_filter(inp, None, False, 1.0, 1.0, tg, reverse, structure=True)
        out, ws, call, x, r = gpu.run_op(inp, None, False, 1.0, 1.0, tg, reverse)
        st, (vk, vi, pv, pw) = gpu.export_op(ws, call, r)
        assert st.direct_index == int(direct)
        gpu.assert_structure_equal(vk, vi, pv, pw, items, str(shape))
        gpu.assert_outputs_close(out.cpu().numpy(), want, str(shape))


def test_bilateral_calls_keep_the_hash_table(gpu):
    rng = np.random.default_rng(6)
    inp = rng.standard_normal((1, 20, 20, 2)).astype(np.float32)
    ref = rng.random((1, 20, 20, 3), dtype=np.float32)
    out, ws, call, x, r = gpu.run_op(inp, ref, True, 4.0, 0.25, 1.0, False)
    st, _ = gpu.export_op(ws, call, r)
    assert st.direct_index == 0


def test_hashed_and_direct_paths_build_the_same_lattice(gpu, hashed_path):
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    from conftest import bits, sorted_rows
    rng = np.random.default_rng(7)
    inp = rng.standard_normal((3, 45, 52, 5)).astype(np.float32)
    res = {}
    for name, enable in (("hashed", 0), ("direct", 1)):
        capi.lib().pl_debug_direct_index(enable)
        out, ws, call, x, r = gpu.run_op(inp, None, False, 1.0, 1.0, 2.5, False, mode="deterministic")
        st, (vk, vi, pv, pw) = gpu.export_op(ws, call, r)
        assert st.direct_index == enable
        vk, vi, pv, pw = (t.cpu().numpy() for t in (vk, vi, pv, pw))
        res[name] = (st.num_vertices, sorted_rows(np.concatenate([vi[:, None].astype(np.int16), vk], 1)),
                     vk[pv.reshape(-1)], bits(pw), bits(out.cpu().numpy()))
    assert res["hashed"][0] == res["direct"][0]
    for a, b in zip(res["hashed"][1:], res["direct"][1:]):
        assert np.array_equal(a, b)   # deterministic mode: outputs bit for bit as well


def test_small_table_falls_back_to_hashing(gpu, oracle):
    """max_entries shrinks the workspace's table region; when the dense index no longer fits, the call
    hashes, with the same results."""
    rng = np.random.default_rng(8)
    inp = rng.standard_normal((8, 16, 16, 2)).astype(np.float32)
    want = oracle.lattice_filter(inp, None, False, 1.0, 1.0, 16.0, False)
    for max_entries, direct in ((0, 1), (200, 0)):
        out, ws, call, x, r = gpu.run_op(inp, None, False, 1.0, 1.0, 16.0, False, max_entries=max_entries)
        st, _ = gpu.export_op(ws, call, r, max_entries=max_entries)
        assert st.direct_index == direct
        gpu.assert_outputs_close(out.cpu().numpy(), want, "max_entries %d" % max_entries)


def test_spatial_only_lattice_reuse(gpu, oracle):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(9)
    inp = rng.standard_normal((2, 30, 41, 4)).astype(np.float32)
    lat = plb.Lattice(None, spatial_shape=(2, 30, 41), bilateral=False, theta_gamma=3.0, max_channels=4)
    assert lat.stats().direct_index == 1
    for reverse in (False, True):
        want = oracle.lattice_filter(inp, None, False, 1.0, 1.0, 3.0, reverse)
        got = lat.apply(torch.from_numpy(inp).cuda(), reverse=reverse)
        gpu.assert_outputs_close(got.cpu().numpy(), want, "reuse")


@pytest.mark.parametrize("shape,theta,bound", [((512, 512), 3.0, 40000), ((1500, 1500), 1.0, 2200000)])
def test_a_call_that_outgrew_its_bound_reports_no_index(gpu, shape, theta, bound):
    """The index, cleared with the header (1 MB) or by a launch of its own (29 MB), is not built by a call that failed before."""
    import torch
    import permutohedral_lattice_b200 as plb
    x = torch.rand((1,) + shape + (1,), device="cuda")
    for dtype in (torch.float32, torch.float64):
        out, ws, _ = plb.lattice_filter_raw(x.to(dtype), None, False, 1.0, 1.0, theta, max_entries=bound, check=False)
        st = plb.lattice_stats(ws)
        assert st.device_status == plb.capi.PL_CAPACITY_EXCEEDED and torch.isnan(out).all()
        assert st.direct_index == 0 and st.table_slots == 1
        out, ws, _ = plb.lattice_filter_raw(x.to(dtype), None, False, 1.0, 1.0, theta, max_entries=2 * bound)
        assert plb.lattice_stats(ws).direct_index == 1 and torch.isfinite(out).all()


@pytest.mark.parametrize("shape,c,theta,batch", [
    ((1, 1), 2, 3.0, 2),             # a single point
    ((33, 47), 3, 3.0, 5),           # the index and the blur of small lattices
    ((130, 150), 1, 1.5, 3),         # narrow rows, passes in pairs
    ((200, 260), 21, 2.0, 4),        # wide rows, a pass a launch
    ((20, 24, 31), 2, 2.0, 3),       # volumes
    ((70, 50), 6, 0.37, 3),          # hashed: the index would not fit
    ((4000,), 1, 5.0, 16),           # one dimension
    ((40, 50), 70, 2.0, 2),          # rows beyond the staged ones
])
def test_one_lattice_for_all_items(shape, c, theta, batch, gpu):
    """The items of a spatial-only call share a lattice: every one of them as if filtered alone, bit for bit, the counters
    and the exported vertices as of a lattice of them all, and the bound that of the whole call."""
    import torch
    import permutohedral_lattice_b200 as plb
    x = torch.randn((batch,) + shape + (c,), generator=torch.Generator("cuda").manual_seed(3), device="cuda")
    x[:, ..., 0].view(batch, -1)[:, 0] = 6.0    # one grid of the fixed-point sums for all
    x.clamp_(-6.0, 6.0)
    for reverse in (False, True):
        out, ws, call = plb.lattice_filter_raw(x, None, False, 1.0, 1.0, theta, reverse, mode="deterministic", max_entries=0)
        st = plb.lattice_stats(ws)
        vk, vi, pv, _ = (t.cpu().numpy() for t in gpu.export_op(ws, call, None, max_entries=0)[1])
        for b in range(batch):
            alone, ws1, call1 = plb.lattice_filter_raw(x[b:b + 1], None, False, 1.0, 1.0, theta, reverse, mode="deterministic",
                                                       max_entries=0, workspace_owner="alone")
            assert torch.equal(out[b:b + 1], alone)
        st1 = plb.lattice_stats(ws1)
        vk1, _, pv1, _ = (t.cpu().numpy() for t in gpu.export_op(ws1, call1, None, max_entries=0)[1])
        assert (st.num_entries, st.num_vertices) == (batch * st1.num_entries, batch * st1.num_vertices)
        for b in range(batch):
            assert (vi[pv[b]] == b).all() and np.array_equal(vk[pv[b]], vk1[pv1[0]])
    for bound, code in ((st.num_entries, 0), (st.num_entries - 1, plb.capi.PL_CAPACITY_EXCEEDED)):
        out, ws, _ = plb.lattice_filter_raw(x, None, False, 1.0, 1.0, theta, max_entries=bound, check=False)
        st = plb.lattice_stats(ws)
        assert st.device_status == code and st.max_entries == bound
        assert torch.isfinite(out).all() if code == 0 else torch.isnan(out).all()
