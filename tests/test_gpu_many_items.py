"""Batches without a guide, of many small grids above all: one lattice serves every item, and what is done for each of them (its
value rows, its copy of the list of entries, its share of the blur) is spread over the whole GPU, not walked item by item."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,shape,c,theta,hashed", [
    (65535, (4, 4), 1, 3.0, False),      # as many items as a call may have, fewer entries than threads of a block
    (65535, (1,), 2, 3.0, False),        # a point each
    (3001, (5, 3), 21, 2.0, False),
    (1500, (9, 11), 5, 0.4, True),       # the one-launch index
    (700, (65, 33), 2, 0.5, True),       # the table of keys, blur passes in pairs or one by one
    (700, (300,), 1, 5.0, False),        # one dimension
    (260, (4, 5, 6), 3, 1.0, True),      # volumes
    (2, (16, 16), 7, 2.0, False),
    (40, (16, 16), 35, 2.0, False),      # rows of nine float4, 360 of them a vertex
    (40, (90, 100), 3, 30.0, False),     # an item's rows together, by the bound: fewer entries than threads
    (3, (420, 500), 2, 0.4, False),      # more
    (2, (420, 500), 1, 0.4, True),
    (4, (512, 512), 21, 0.7, False),     # beyond 256 MB of rows
])
def test_every_item_as_if_alone(batch, shape, c, theta, hashed):
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    gen = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn((batch,) + shape + (c,), generator=gen, device="cuda").clamp_(-6.0, 6.0)
    x.view(batch, -1)[:, 0] = 6.0                  # one grid of the fixed-point sums for all
    was = capi.lib().pl_debug_direct_index(0 if hashed else 1)
    try:
        for reverse in (False, True):
            out, ws, call = plb.lattice_filter_raw(x, None, False, 1.0, 1.0, theta, reverse, mode="deterministic", max_entries=0)
            st = plb.lattice_stats(ws)
            assert st.device_status == 0 and not (hashed and st.direct_index)
            _, item, pv, pw = plb.export_lattice(ws, st, call.batch, call.n, call.pd, call.vd, sdims=call.sdims,
                                                 spatial_std=call.spatial_std, feature_std=call.feature_std, max_entries=0)
            pv = pv.view(batch, -1).long()
            assert torch.equal(item[pv].long(), torch.arange(batch, device="cuda").view(-1, 1).expand_as(pv))
            assert torch.equal(pw.view(batch, -1), pw.view(batch, -1)[:1].expand(batch, -1))
            plain = plb.lattice_filter(x, None, False, 1.0, 1.0, theta, reverse=reverse)
            # a float sum of at most 2^11 terms in any order, on either side of the fixed-point one
            assert float((plain - out).norm() / out.norm()) <= 1e-5
            for b in sorted({0, 1, batch // 2, batch - 1}):
                alone, ws1, _ = plb.lattice_filter_raw(x[b:b + 1], None, False, 1.0, 1.0, theta, reverse, mode="deterministic",
                                                       max_entries=0, workspace_owner="alone")
                assert torch.equal(out[b:b + 1], alone), b
            st1 = plb.lattice_stats(ws1)
            assert (st.num_entries, st.num_vertices) == (batch * st1.num_entries, batch * st1.num_vertices)
    finally:
        capi.lib().pl_debug_direct_index(was)


@pytest.mark.parametrize("batch,shape", [(4096, (4, 4)), (16384, (8, 8)), (2048, (300,))])
def test_many_items_take_no_longer_than_a_lattice_each(batch, shape):
    """Against a flat guide, with which every item builds its own lattice of one dimension more: that takes longer.  Item by item,
    the lattice that serves all took five to thirty times as long; the limit is twice."""
    import torch
    import permutohedral_lattice_b200 as plb
    x = torch.rand((batch,) + shape + (1,), device="cuda")
    guide = torch.zeros((batch,) + shape + (1,), device="cuda")

    def ms(*args):
        best = float("inf")
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(10):
                plb.lattice_filter(x, *args)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) / 10)
        return best

    assert ms(None, False, 1.0, 1.0, 3.0) <= 2.0 * ms(guide, True, 3.0, 1.0)
