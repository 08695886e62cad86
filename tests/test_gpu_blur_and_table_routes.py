"""Bounds at which a call takes another route and must give the same bits (deterministic sums): two blur passes a launch or
one, rows made doubles by moves of bits or (more than 5,000,000 float4 of them) by conversions, the table cleared with the header or by a launch of its own, for hash tables and for the direct index."""
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


def _positions(n, pd, seed):
    import torch
    rng = np.random.default_rng(seed)
    return torch.from_numpy(np.repeat(rng.standard_normal((1, -(-n // 6), pd)) * 4, 6, 1)[:, :n].astype(np.float32)).cuda()


@pytest.mark.parametrize("pd", [1, 2, 3, 4, 5, 6, 8, 16])
def test_pairs_of_passes_give_the_bits_of_single_ones(plb, pd):
    """Worst cases beyond 300,000 items go pass by pass, other bounds up to 1,000,000 items in pairs."""
    import torch
    n = 310000 // (pd + 1) + 1
    pos, worst = _positions(n, pd, pd), n * (pd + 1)
    for c in (1, 3, 7, 11):                            # rows of 1 to 3 float4
        x = torch.randn((1, n, c), generator=torch.Generator().manual_seed(c)).cuda()
        for reverse in (False, True):
            single = plb.filter_positions(x, pos, reverse, "deterministic", max_entries=worst)[0].clone()
            pairs = plb.filter_positions(x, pos, reverse, "deterministic", max_entries=worst - 1)[0].clone()
            assert torch.equal(single, pairs), (c, reverse)
    x64, p64 = x[..., :2].double(), pos.double()
    single = plb.filter_positions(x64, p64, max_entries=worst)[0].clone()
    pairs = plb.filter_positions(x64, p64, max_entries=worst - 1)[0].clone()
    assert float((single - pairs).norm() / single.norm()) <= 1e-12      # double sums in varying order


def test_rows_mixed_by_moves_give_the_bits_of_conversions(plb):
    """The same first channels beside 68 others: 330,000 rows of 18 float4, or of one.  Both signs, thirty binades."""
    import torch
    g = torch.Generator().manual_seed(3)
    pos = (60 * torch.randn((1, 60000, 5), generator=g)).cuda()
    x = torch.rand((1, 60000, 71), generator=g).cuda()          # below 1: the same fixed-point grid for both
    x *= torch.exp2(-30 * torch.rand((1, 60000, 71), generator=g)).cuda() * (torch.randint(0, 2, (1, 60000, 71), generator=g) * 2 - 1).cuda()
    for reverse in (False, True):
        wide, ws = plb.filter_positions(x, pos, reverse, "deterministic", max_entries=0)
        assert plb.lattice_stats(ws).num_vertices * 18 > 5000000
        narrow, _ = plb.filter_positions(x[..., :3].contiguous(), pos, reverse, "deterministic", max_entries=0)
        assert torch.equal(wide[..., :3], narrow)


@pytest.mark.parametrize("pd", [1, 3, 5, 7, 16])
def test_tables_cleared_with_the_header_or_by_themselves(plb, pd):
    """Bounds below 2^18 entries have no sketch: their whole table is cleared with the header.  A second call on the same
    workspace finds the first one's rows where its table goes."""
    import torch
    n = (1 << 18) // (pd + 1) + 40
    pos = _positions(n, pd, pd + 20)
    x = torch.rand((1, n, 2), device="cuda")
    want = plb.filter_positions(x, pos, mode="deterministic", max_entries=0)[0].clone()
    ws = torch.empty(4 << 30, dtype=torch.uint8, device="cuda")
    for bound in ((1 << 18) - 1, 1 << 18, (1 << 18) - 1, 1 << 17):
        for _ in range(2):
            got, _ = plb.filter_positions(x, pos, mode="deterministic", max_entries=bound, workspace=ws)
            assert torch.equal(got, want), bound
        st = plb.lattice_stats(ws)
        assert st.device_status == 0 and st.num_vertices * 2 <= st.table_slots


@pytest.mark.parametrize("batch", [1, 8, 16])          # 1, 7.5 and 15 MB of index
def test_direct_index_cleared_with_the_header_or_by_itself(plb, batch):
    import torch
    from permutohedral_lattice_b200 import capi
    shape = (batch, 20, 24, 28)
    x = torch.rand(shape + (2,), device="cuda")
    got = []
    for enable in (1, 0, 1):
        was = capi.lib().pl_debug_direct_index(enable)
        try:
            out, ws, _ = plb.lattice_filter_raw(x, None, False, 1.0, 1.0, 1.0, mode="deterministic", max_entries=2000000)
            assert plb.lattice_stats(ws).direct_index == enable
            got.append(out.clone())
        finally:
            capi.lib().pl_debug_direct_index(was)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("pd", [3, 5, 6])
@pytest.mark.parametrize("noise", [0.0, 0.3])
@pytest.mark.parametrize("more", [False, True])
def test_slots_claimed_unseen_or_not(pd, noise, more):
    """Entries that are mostly vertices (a noisy guide) and entries that are not, in tables cleared with the header (up to
    2^19 entries) and sized by the sketch of the lattice: every key one vertex, each item as if filtered alone."""
    import torch
    import permutohedral_lattice_b200 as plb
    n = (1 << 19) // (2 * (pd + 1))                 # two items of n points have just no more than 2^19 entries
    h, w = 128, n // 128 + (2 if more else 0)
    gen = torch.Generator("cuda").manual_seed(pd)
    ref = torch.linspace(0, 1, w, device="cuda").expand(2, h, w).unsqueeze(-1).repeat(1, 1, 1, pd - 2)
    ref = (ref + noise * torch.randn(ref.shape, generator=gen, device="cuda")).contiguous()
    x = torch.randn((2, h, w, 3), generator=gen, device="cuda").clamp_(-4, 4)
    x[:, 0, 0, 0] = 4.0                             # one grid of the fixed-point sums for all
    out, ws, call = plb.lattice_filter_raw(x, ref, True, 8.0, 0.1, 1.0, mode="deterministic", max_entries=0)
    st = plb.lattice_stats(ws)
    assert st.device_status == 0 and st.table_slots >= 2 * st.num_vertices
    keys, item, _, _ = plb.export_lattice(ws, st, call.batch, call.n, call.pd, call.vd, reference=ref, sdims=call.sdims,
                                          spatial_std=call.spatial_std, feature_std=call.feature_std, max_entries=0)
    both = torch.cat([item.view(-1, 1).to(torch.int16), keys], 1)
    assert len(torch.unique(both, dim=0)) == st.num_vertices
    total = 0
    for b in range(2):
        alone, ws1, _ = plb.lattice_filter_raw(x[b:b + 1], ref[b:b + 1], True, 8.0, 0.1, 1.0, mode="deterministic",
                                               max_entries=0, workspace_owner="alone")
        assert torch.equal(out[b:b + 1], alone)
        total += plb.lattice_stats(ws1).num_vertices
    assert total == st.num_vertices
