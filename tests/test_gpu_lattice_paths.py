"""Lattice construction where its paths part: a hash table sized by a sketch of the vertices or by the entries, tiles
whose keys are all distinct (several rounds of de-duplication) or all equal, verified calls from several threads.
The structure is compared exactly."""
import threading

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


@pytest.mark.parametrize("guide,theta", [("flat", (30.0, 0.2)), ("cells", (8.0, 0.1)), ("noise", (0.3, 0.01))])
@pytest.mark.parametrize("size", [(128, 160), (256, 192)])
def test_table_has_room_for_the_lattice(guide, theta, size, gpu, oracle):
    """2 x 128 x 160 points x 6 lie below the size at which a sketch is kept, 2 x 256 x 192 x 6 above."""
    rng = np.random.default_rng(53)
    shape = (2,) + size
    if guide == "flat":
        ref = np.full(shape + (3,), 0.5, np.float32)
    elif guide == "cells":
        ref = np.kron(rng.random((2, size[0] // 16, size[1] // 16, 3)), np.ones((1, 16, 16, 1))).astype(np.float32)
    else:
        ref = rng.random(shape + (3,), dtype=np.float32)
    inp = rng.random(shape + (1,), dtype=np.float32)
    want, items = oracle.lattice_filter(inp, ref, True, *theta, 1.0, False, structure=True)
    out, ws, call, _, rt = gpu.run_op(inp, ref, True, *theta, 1.0, False, max_entries=0)
    st, (vk, vi, pv, pw) = gpu.export_op(ws, call, rt)
    gpu.assert_structure_equal(vk, vi, pv, pw, items, guide)
    gpu.assert_outputs_close(out.cpu().numpy(), want, guide)
    assert st.table_slots >= 2 * st.num_vertices
    # by vertices: four slots each, rounded up to a power of two (the sketch is 4 % off at most), or the smallest
    # table that the sketch chooses; by entries: at least two slots an entry
    assert st.table_slots <= max(4 * st.num_entries, 1024)
    if size == (256, 192):
        assert st.table_slots <= max(16 * st.num_vertices, 1 << 16)


@pytest.mark.parametrize("pd", [1, 2, 3, 4, 5, 6, 7, 8, 16])
@pytest.mark.parametrize("spread", [0.0, 1.0, 40.0])
def test_tiles_of_equal_and_of_distinct_keys(pd, spread, gpu, oracle):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(59)
    n = 611
    pos = (rng.standard_normal((2, n, pd)) * spread).astype(np.float32)
    val = rng.random((2, n, 2), dtype=np.float32)
    pt = torch.from_numpy(pos).cuda()
    out, ws = plb.filter_positions(torch.from_numpy(val).cuda(), pt, max_entries=0)
    st = plb.lattice_stats(ws)
    vk, vi, pv, pw = plb.export_lattice(ws, st, 2, n, pd, 3, positions=pt)
    items = [oracle.filter(val[i], pos[i]) for i in range(2)]
    gpu.assert_structure_equal(vk, vi, pv, pw, items, "pd %d spread %g" % (pd, spread))
    gpu.assert_outputs_close(out.cpu().numpy(), np.stack([o.out for o in items]), "pd %d spread %g" % (pd, spread))
    # the rounds find every repeated key of a tile: as many entries as the tiles have distinct keys
    tile = 128 if pd > 8 else 256
    distinct = sum(len(set(map(bytes, items[i].pixel_keys()[a:a + tile].reshape(-1, pd))))
                   for i in range(2) for a in range(0, n, tile))
    assert st.num_entries == distinct


def test_verified_calls_from_several_threads(gpu):
    """Every thread's calls on new reference images wait for their own counters, on the thread's own stream."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(61)
    refs = [torch.from_numpy(rng.random((1, 40 + 8 * i, 48, 3), dtype=np.float32)).cuda() for i in range(6)]
    xs = [torch.rand(r.shape[:-1] + (2,), device="cuda") for r in refs]
    want = [plb.lattice_filter_raw(x, r, True, 2.0, 0.05, mode="deterministic", max_entries=0)[0].clone()
            for x, r in zip(xs, refs)]
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(24):
                    j = (i + k) % len(refs)
                    got = plb.lattice_filter(xs[j], refs[j].clone(), True, 2.0, 0.05, mode="deterministic")
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(got, want[j]):
                        wrong.append((k, j))
        except Exception as e:   # noqa: BLE001 - reported below
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_calls_of_several_widths_from_several_threads(dtype, gpu):
    """Threads whose calls need more shared memory of the same kernels than one another's, all at once."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(67)
    pos = torch.from_numpy(rng.standard_normal((1, 700, 7))).to(getattr(torch, dtype)).cuda()
    xs = [torch.from_numpy(rng.random((1, 700, c))).to(pos.dtype).cuda() for c in (30, 5, 60, 9, 100, 16)]
    got, wrong, together = [None] * len(xs), [], threading.Barrier(len(xs))
    torch.cuda.synchronize()

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                together.wait(30)
                got[k] = plb.filter_positions(xs[k], pos, max_entries=0)[0]
                torch.cuda.current_stream().synchronize()
        except Exception as e:   # noqa: BLE001 - reported below
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for x, g in zip(xs, got):
        want = plb.filter_positions(x, pos, max_entries=0)[0]
        # sums in varying order
        assert float((g - want).norm() / want.norm()) <= (1e-12 if dtype == "float64" else 1e-5)


@pytest.mark.parametrize("pd,n", [(1, 8200), (2, 5470), (3, 4100), (5, 2735), (8, 1825), (16, 970)])
def test_small_lattices_give_the_bits_of_wide_ones(pd, n, gpu, oracle):
    """A bound of 6144 entries takes the index and the blur of small lattices, the worst case the wide index and, beyond its
    limits, the passes one by one.  Deterministic sums make small and wide comparable."""
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(79)
    pos = np.repeat(rng.standard_normal((1, (n + 4) // 5, pd)), 5, 1)[:, :n].astype(np.float32)
    pt = torch.from_numpy(pos).cuda()
    assert n * (pd + 1) > 16384   # the worst case: wide launches
    for c in (1, 3, 4, 7, 8):
        val = rng.standard_normal((1, n, c)).astype(np.float32)
        x = torch.from_numpy(val).cuda()
        for reverse in (False, True):
            small = plb.filter_positions(x, pt, reverse=reverse, mode="deterministic", max_entries=6144)[0].clone()
            wide = plb.filter_positions(x, pt, reverse=reverse, mode="deterministic", max_entries=0)[0].clone()
            assert torch.equal(small, wide), "pd %d, %d channels" % (pd, c)
        x64, p64 = x.double(), pt.double()
        small = plb.filter_positions(x64, p64, max_entries=6144)[0].clone()
        wide = plb.filter_positions(x64, p64, max_entries=0)[0].clone()
        # double sums in varying order
        assert float((small - wide).norm() / wide.norm()) <= 1e-12, "pd %d, %d channels in double" % (pd, c)
    got = plb.filter_positions(x, pt, max_entries=6144)[0].cpu().numpy()[0]
    gpu.assert_outputs_close(got, oracle.filter(val[0], pos[0], structure=False).out, "pd %d" % pd)


def _large_table(gpu, oracle, width, guide):
    """Word 8 of the header: the filter's bits, as a logarithm (0: none)."""
    import torch
    rng = np.random.default_rng(73)
    ref = np.repeat(rng.random((1, 1024, width // 2, guide), dtype=np.float32), 2, 2)
    inp = rng.random((1, 1024, width, 1), dtype=np.float32)
    theta = 0.05 if guide == 3 else 0.1
    want, items = oracle.lattice_filter(inp, ref, True, 3.0, theta, 1.0, False, structure=True)
    out, ws, call, _, rt = gpu.run_op(inp, ref, True, 3.0, theta, 1.0, False, max_entries=0)
    st, (vk, vi, pv, pw) = gpu.export_op(ws, call, rt)
    assert st.table_slots == 1 << 23
    gpu.assert_structure_equal(vk, vi, pv, pw, items, "large table")
    gpu.assert_outputs_close(out.cpu().numpy(), want, "large table")
    return int(ws[:64].view(torch.int32)[8])


def test_filter_in_front_of_a_large_table(gpu, oracle):
    """pd 6: 2.8 M vertices in a table of 2^23 slots, half of what the workspace has room for: the lookups pass the filter."""
    assert _large_table(gpu, oracle, 600, 4) == 26


def test_large_table_of_keys(gpu, oracle):
    """pd 5: 2.9 M vertices in a table of 2^23 slots that hold the key, which has no filter."""
    assert _large_table(gpu, oracle, 720, 3) == 0


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_features_without_a_simplex_stay_in_their_own_points(dtype, gpu, oracle):
    """pd = 16: item 0 has NaN, infinite and huge features, in full tiles and in a last tile of one point; item 1 has
    none and is filtered as ever."""
    import torch
    import permutohedral_lattice_b200 as plb
    from conftest import rel_l2
    from test_host_simplex import features_without_a_simplex
    n = 4 * 128 + 1
    pos = np.stack([np.resize(features_without_a_simplex(dtype)[::-1], (n, 16)),
                    np.random.default_rng(83).standard_normal((n, 16)).astype(dtype)])
    val = np.random.default_rng(89).random((2, n, 3)).astype(dtype)
    pt = torch.from_numpy(pos).cuda()
    for _ in range(3):   # the shared memory of a call holds what the one before left
        out, ws = plb.filter_positions(torch.from_numpy(val).cuda(), pt, max_entries=0)
        st = plb.lattice_stats(ws)
        assert st.device_status == 0 and st.num_entries <= 2 * n * 17
        _, vitem, pv, _ = plb.export_lattice(ws, st, 2, n, 16, 4, positions=pt)
        assert int(pv.min()) >= 0 and int(pv.max()) < st.num_vertices
        assert bool((vitem[pv[0].long()] == 0).all()) and bool((vitem[pv[1].long()] == 1).all())
        want = oracle.filter(val[1], pos[1], structure=False, dtype=dtype).out
        assert rel_l2(out[1].cpu().numpy(), want) <= (1e-12 if dtype == np.float64 else 1e-5)


@pytest.mark.parametrize("pd", [1, 2, 3, 5, 8])
def test_keys_beyond_their_range_stay_in_their_own_tiles(pd, gpu, oracle):
    """Item 0 has features so large that splats of different remainders get one key; item 1 is filtered as ever, and
    every splat of either item still points to a vertex of its own item."""
    import torch
    import permutohedral_lattice_b200 as plb
    from test_host_simplex import far_features
    n = 3 * 256 + 1
    pos = np.stack([far_features(pd, n), np.random.default_rng(97).standard_normal((n, pd)).astype(np.float32)])
    val = np.random.default_rng(101).random((2, n, 3), dtype=np.float32)
    pt = torch.from_numpy(pos).cuda()
    for _ in range(3):
        out, ws = plb.filter_positions(torch.from_numpy(val).cuda(), pt, max_entries=0)
        st = plb.lattice_stats(ws)
        assert st.device_status == 0 and st.num_entries <= 2 * n * (pd + 1)
        _, vitem, pv, _ = plb.export_lattice(ws, st, 2, n, pd, 4, positions=pt)
        assert int(pv.min()) >= 0 and int(pv.max()) < st.num_vertices
        assert bool((vitem[pv[0].long()] == 0).all()) and bool((vitem[pv[1].long()] == 1).all())
        want = oracle.filter(val[1], pos[1], structure=False).out
        gpu.assert_outputs_close(out[1].cpu().numpy(), want, "pd %d" % pd)
