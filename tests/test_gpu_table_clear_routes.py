"""Who clears the index of a call: the launch that clears the header, or one of its own when the index is larger than 16 MB (8 MB
with 16 feature dimensions).  On both sides of that line, in turn, on a workspace that holds whatever the call before left."""
import pytest

pytestmark = pytest.mark.gpu


def _launches(call):
    """What call() returns, and the kernels it launched."""
    from permutohedral_lattice_b200 import capi
    before = capi.lib().pl_launch_count()
    got = call()
    return got, capi.lib().pl_launch_count() - before


@pytest.mark.parametrize("pd", [1, 3, 5, 6, 8, 16])
def test_hash_tables(pd):
    """Slots of 16 bytes up to pd 5, else of 8; the smallest power of two that gives every entry of the bound two."""
    import torch
    import permutohedral_lattice_b200 as plb
    last = 1 << (20 if 5 < pd < 16 else 19)              # the largest bound whose table is cleared with the header
    n = last // (pd + 1) + 50                            # so that the worst case is beyond it
    gen = torch.Generator(device="cuda").manual_seed(pd)
    pos = 4 * torch.randn((1, -(-n // 8), pd), generator=gen, device="cuda")
    pos = pos.repeat_interleave(8, 1)[:, :n].contiguous()   # an eighth of the worst case in entries, at least
    x = torch.rand((1, n, 2), generator=gen, device="cuda")
    assert n * (pd + 1) > last
    want = plb.filter_positions(x, pos, mode="deterministic", max_entries=0)[0].clone()
    most = torch.randint(0, 256, (3 << 30,), dtype=torch.uint8, device="cuda")
    counts = {}
    for bound in (last, last + 1, last, last + 1, last - 1):
        (got, ws), launches = _launches(lambda: plb.filter_positions(x, pos, mode="deterministic", max_entries=bound, workspace=most))
        assert torch.equal(got, want), bound
        st = plb.lattice_stats(ws)
        assert st.device_status == 0 and st.table_slots >= 2 * st.num_vertices
        counts.setdefault(bound <= last, set()).add(launches)
    assert counts[False] == {min(counts[True]) + 1} and len(counts[True]) == 1      # the launch that clears the table
    x64, p64 = x.double(), pos.double()
    want = plb.filter_positions(x64, p64, max_entries=0)[0].clone()
    counts = {}
    for bound in (last, last + 1, last, last + 1):
        (got, _), launches = _launches(lambda: plb.filter_positions(x64, p64, max_entries=bound, workspace=most))
        assert float((got - want).norm() / want.norm()) <= 1e-12, bound             # double sums in varying order
        counts.setdefault(bound <= last, set()).add(launches)
    assert counts[False] == {min(counts[True]) + 1} and len(counts[True]) == 1


# slots of the index of an item, 4 bytes each, from the grid and theta: 1000 x 1000 13 MB, 1500 x 1500 27 MB, 20 x 24 x 28 1 MB
@pytest.mark.parametrize("shape,theta,own,table_own", [
    ((1, 1000, 1000), 1.0, False, True),
    ((1, 1500, 1500), 1.0, True, True),
    ((2, 1500, 1500), 1.0, True, True),
    ((16, 20, 24, 28), 1.0, False, False),
])
def test_direct_indexes(shape, theta, own, table_own):
    """Against the hash table, bit for bit.  Of a batch both are of one item.  own: the index has a launch of its own to clear it;
    table_own: so has the table."""
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    x = torch.rand(shape + (1,), device="cuda")
    need = plb.lattice_filter_raw(x, None, False, 1.0, 1.0, theta, mode="deterministic", max_entries=0)[2].workspace_bytes(
        0, mode="deterministic")
    most = torch.randint(0, 256, (need,), dtype=torch.uint8, device="cuda")
    got, launches = [], {}
    for enable in (1, 0, 1):
        was = capi.lib().pl_debug_direct_index(enable)
        try:
            (out, ws, _), count = _launches(lambda: plb.lattice_filter_raw(x, None, False, 1.0, 1.0, theta, mode="deterministic",
                                                                           max_entries=0, workspace=most))
        finally:
            capi.lib().pl_debug_direct_index(was)
        assert plb.lattice_stats(ws).direct_index == enable
        got.append(out.clone())
        launches[enable] = count
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert launches[1] - launches[0] == int(own) - int(table_own)


@pytest.mark.parametrize("shape,theta", [((1, 1500, 1500), 1.0), ((40, 20, 24, 28), 1.0)])
def test_direct_indexes_in_double(shape, theta):
    """A lattice of all items, whose index is as many times as large: 27 and 37 MB, by a launch of its own."""
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    x = torch.rand(shape + (1,), dtype=torch.float64, device="cuda")
    got = []
    for enable in (1, 0, 1):
        was = capi.lib().pl_debug_direct_index(enable)
        try:
            out, ws, _ = plb.lattice_filter_raw(x, None, False, 1.0, 1.0, theta, max_entries=0)
        finally:
            capi.lib().pl_debug_direct_index(was)
        st = plb.lattice_stats(ws)
        assert st.direct_index == enable and (not enable or 4 * st.table_slots > 16 << 20)
        got.append(out.clone())
        ws.fill_(0x5a)
    for other in got[1:]:
        assert float((other - got[0]).norm() / got[0].norm()) <= 1e-12
