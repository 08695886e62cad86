"""How much workspace a call gets by default (sized from what its lattice needs instead of the bound that can
never overflow), and what happens when a lattice outgrows it: a call on a new reference image is verified and
repeated on the spot; a call on the reference a verified call just used runs with that call's bound; calls made
with verify="deferred" (HostPipeline) that do not fit fill their output with NaN, are reported by
check_pending() and repeated by the pipeline.  Nothing here faults the GPU: a bound that is too small only sets
a status bit on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(bilateral=True, theta_alpha=5.0, theta_beta=0.2, theta_gamma=1.0)


def _data(seed, batch=2, shape=(48, 44), c=4, blocky=True):
    import torch
    rng = np.random.default_rng(seed)
    if blocky:   # few lattice entries per point, so a bound well below the worst case suffices
        blocks = rng.random((batch, (shape[0] + 7) // 8, (shape[1] + 7) // 8, 3), dtype=np.float32)
        ref_n = np.repeat(np.repeat(blocks, 8, 1), 8, 2)[:, :shape[0], :shape[1]]
    else:        # white noise: nearly every splat its own entry
        ref_n = rng.random((batch,) + shape + (3,), dtype=np.float32)
    ref = torch.from_numpy(np.ascontiguousarray(ref_n)).cuda()
    x = torch.from_numpy(rng.standard_normal((batch,) + shape + (c,)).astype(np.float32)).cuda()
    return x, ref


@pytest.fixture()
def policy():
    """A clean slate for the module's memory of earlier calls."""
    import permutohedral_lattice_b200 as plb
    import sys
    lf = sys.modules["permutohedral_lattice_b200.lattice_filter"]   # (the package re-exports a function of that name)
    saved = (dict(lf._entries_per_item), lf.FIRST_GUESS_DIVISOR)
    lf._entries_per_item.clear()
    lf._pending.clear()
    lf._verified.clear()
    plb.release_workspaces()
    yield lf
    lf._entries_per_item.clear()
    lf._entries_per_item.update(saved[0])
    lf.FIRST_GUESS_DIVISOR = saved[1]
    lf._pending.clear()
    lf._verified.clear()


def test_default_workspace_is_smaller_than_the_worst_case_and_results_agree(policy):
    import permutohedral_lattice_b200 as plb
    from conftest import bits
    x, ref = _data(1)
    want, ws0, call0 = plb.lattice_filter_raw(x, ref, mode="deterministic", max_entries=0, **KW)
    worst_bytes = call0.workspace_bytes(0, mode="deterministic")
    plb.release_workspaces()
    got, ws, call = plb.lattice_filter_raw(x, ref, mode="deterministic", **KW)     # first of its kind: verified
    assert 0 < call.max_entries < call.batch * call.n * (call.pd + 1)
    assert ws.numel() < worst_bytes
    assert np.array_equal(bits(got.cpu().numpy()), bits(want.cpu().numpy()))
    got2, ws2, call2 = plb.lattice_filter_raw(x, ref, mode="deterministic", **KW)  # same reference: same bound
    st = plb.lattice_stats(ws2)
    assert st.device_status == 0 and st.num_entries <= call2.max_entries == st.max_entries
    assert call2.max_entries == call.max_entries
    assert np.array_equal(bits(got2.cpu().numpy()), bits(want.cpu().numpy()))


def test_first_call_of_a_kind_is_repeated_until_the_lattice_fits(policy):
    import permutohedral_lattice_b200 as plb
    from conftest import bits
    x, ref = _data(2)
    want, _, _ = plb.lattice_filter_raw(x, ref, mode="deterministic", max_entries=0, **KW)
    policy.FIRST_GUESS_DIVISOR = 64          # a first guess far too small: several repeats
    policy._entries_per_item.clear()
    policy._verified.clear()
    got, ws, call = plb.lattice_filter_raw(x, ref, mode="deterministic", **KW)
    st = plb.lattice_stats(ws)
    assert st.device_status == 0 and st.num_entries <= st.max_entries
    assert np.array_equal(bits(got.cpu().numpy()), bits(want.cpu().numpy()))


def test_new_reference_is_verified_even_when_earlier_data_needed_far_less(policy):
    import torch
    import permutohedral_lattice_b200 as plb
    from conftest import bits
    x, ref = _data(3, blocky=False)
    want, _, call = plb.lattice_filter_raw(x, ref, mode="deterministic", max_entries=0, **KW)
    kind = policy._kind(x.device, call)
    policy._entries_per_item[kind] = 10.0     # as if earlier data of this kind had needed almost nothing
    out, ws, call = plb.lattice_filter_raw(x, ref, mode="deterministic", **KW)
    assert np.array_equal(bits(out.cpu().numpy()), bits(want.cpu().numpy()))
    assert policy._entries_per_item[kind] > 10.0
    # the same reference again (a backward call): the verified bound is reused as it is
    out2, ws2, call2 = plb.lattice_filter_raw(x, ref, mode="deterministic", reverse=True, **KW)
    assert call2.max_entries == call.max_entries
    assert plb.lattice_stats(ws2).device_status == 0
    # written to in place: no longer "the same lattice", verified again
    ref.mul_(0.5)
    policy._entries_per_item[kind] = 10.0
    want3 = plb.lattice_filter_raw(x, ref, mode="deterministic", max_entries=0, **KW)[0]
    out3 = plb.lattice_filter_raw(x, ref, mode="deterministic", **KW)[0]
    assert np.array_equal(bits(out3.cpu().numpy()), bits(want3.cpu().numpy()))


def test_new_tensor_in_the_memory_of_an_old_one_is_verified(policy):
    """A reference image that got the memory, shape and version counter of one that is gone is another image."""
    import torch
    import permutohedral_lattice_b200 as plb
    from conftest import bits
    x, ref = _data(3, blocky=False)
    want, _, _ = plb.lattice_filter_raw(x, ref, mode="deterministic", max_entries=0, **KW)
    flat = ref.new_empty(ref.shape)
    flat.data.fill_(0.5)
    where, version = flat.data_ptr(), flat._version
    plb.lattice_filter_raw(x, flat, mode="deterministic", **KW)
    del flat
    again = ref.new_empty(ref.shape)
    assert again.data_ptr() == where and again._version == version, "the allocator gave other memory: nothing tested"
    again.data.copy_(ref)      # without the version counter, as a fresh upload would be
    policy._entries_per_item.clear()
    kind_before = dict(policy._verified)
    out, _, _ = plb.lattice_filter_raw(x, again, mode="deterministic", **KW)
    assert policy._verified != kind_before
    assert np.array_equal(bits(out.cpu().numpy()), bits(want.cpu().numpy()))


def test_deferred_call_that_does_not_fit_is_reported_and_succeeds_when_repeated(policy):
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    from conftest import bits
    x, ref = _data(3, blocky=False)
    want, _, call = plb.lattice_filter_raw(x, ref, mode="deterministic", max_entries=0, **KW)
    kind = policy._kind(x.device, call)
    policy._entries_per_item[kind] = 10.0
    out, ws, _ = plb.lattice_filter_raw(x, ref, mode="deterministic", verify="deferred", **KW)
    torch.cuda.synchronize()
    assert torch.isnan(out).all()             # a call that did not fit never leaves plausible values
    with pytest.raises(plb.PlError) as err:
        plb.check_pending()
    assert err.value.status == capi.PL_CAPACITY_EXCEEDED
    for _ in range(24):                       # every report raises the bound; the repeat ends up fitting
        out, ws, _ = plb.lattice_filter_raw(x, ref, mode="deterministic", verify="deferred", **KW)
        try:
            plb.check_pending()
            break
        except plb.PlError as e:
            assert e.status == capi.PL_CAPACITY_EXCEEDED
    assert np.array_equal(bits(out.cpu().numpy()), bits(want.cpu().numpy()))


def test_host_pipeline_repeats_chunks_that_did_not_fit(policy):
    import torch
    import permutohedral_lattice_b200 as plb
    x, ref = _data(4, batch=5, blocky=False)
    hx, href = x.cpu().pin_memory(), ref.cpu().pin_memory()
    want = plb.lattice_filter(x, ref, **KW).cpu().numpy()
    pipe = plb.HostPipeline(torch.device("cuda", 0), n_streams=2, chunk_items=2, edge_chunks=1)
    pipe.filter(hx, href, **KW)               # teaches the policy what a chunk of this kind needs
    from permutohedral_lattice_b200.lattice_filter import FilterCall
    for batch in (1, 2):
        call = FilterCall((batch,) + tuple(x.shape[1:]), (batch,) + tuple(ref.shape[1:]), True, 5.0, 0.2, 1.0)
        policy._entries_per_item[policy._kind(x.device, call)] = 10.0
    out = pipe.filter(hx, href, **KW)         # chunks overflow, synchronize() finds out and repeats them
    got = out.numpy()
    assert np.isfinite(got).all()
    assert np.abs(got - want).max() <= 1e-4


def test_host_pipeline_gives_back_its_workspaces_when_closed(policy):
    import torch
    import permutohedral_lattice_b200 as plb
    x, ref = _data(6, batch=3)
    pipe = plb.HostPipeline(torch.device("cuda", 0), n_streams=2)
    pipe.filter(x.cpu().pin_memory(), ref.cpu().pin_memory(), **KW)
    mine = [k for k in policy._workspaces if isinstance(k[1], tuple) and k[1][:2] == ("HostPipeline", id(pipe))]
    assert mine                                   # one workspace per stream slot that was used
    pipe.close()
    assert not [k for k in policy._workspaces if isinstance(k[1], tuple) and k[1][:2] == ("HostPipeline", id(pipe))]


def _watched(lib):
    """What awaiting the watched call of this thread returns: (return code, entries)."""
    import ctypes
    import torch
    entries, status = ctypes.c_int64(-1), ctypes.c_int(-1)
    torch.cuda.synchronize()
    rc = lib.pl_await_watched_call(ctypes.byref(entries), ctypes.byref(status), torch.cuda.current_stream().cuda_stream)
    return rc, entries.value


@pytest.mark.parametrize("failure", ["workspace", "argument", "memory", "empty"])
def test_watch_of_a_call_that_failed_is_not_taken_by_the_next_one(policy, failure, monkeypatch):
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    x, ref = _data(8)
    _, ws, call = plb.lattice_filter_raw(x, ref, max_entries=0, **KW)
    lib, stream = capi.lib(), torch.cuda.current_stream().cuda_stream
    if failure == "memory":
        policy._verified.clear()

        def no_memory(*args):
            raise torch.cuda.OutOfMemoryError("no memory for the workspace")

        with monkeypatch.context() as m:
            m.setattr(policy, "_workspace", no_memory)
            with pytest.raises(torch.cuda.OutOfMemoryError):
                plb.lattice_filter_raw(x, ref, **KW)
    else:
        assert lib.pl_watch_next_call(stream) == capi.PL_OK
        batch, nbytes, out, want = call.batch, ws.numel(), x.data_ptr(), capi.PL_OK
        if failure == "workspace":
            nbytes, want = 16, capi.PL_WORKSPACE_TOO_SMALL
        elif failure == "argument":
            out, want = 0, capi.PL_INVALID_ARGUMENT
        else:
            batch = 0
        assert lib.pl_lattice_filter_f32(out, x.data_ptr(), ref.data_ptr(), batch, len(call.sdims), call.c_sdims,
                                         call.c, call.r, 1, *call.theta, 0, ws.data_ptr(), nbytes, 0, 0, stream) == want
    plb.lattice_filter_raw(x, ref, max_entries=0, **KW)      # nobody watches this one
    assert _watched(lib)[0] == capi.PL_INVALID_ARGUMENT


def test_call_that_is_being_captured_is_not_watched(policy):
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    x, ref = _data(9)
    out, ws, _ = plb.lattice_filter_raw(x, ref, max_entries=0, **KW)
    want, lib = out.clone(), capi.lib()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    assert lib.pl_watch_next_call(torch.cuda.current_stream().cuda_stream) == capi.PL_OK
    with torch.cuda.graph(graph):
        plb.lattice_filter_raw(x, ref, out=out, workspace=ws, **KW)
    graph.replay()
    assert _watched(lib)[0] == capi.PL_INVALID_ARGUMENT
    assert torch.allclose(out, want, atol=1e-5)


@pytest.mark.parametrize("dtype,c", [("float32", 21), ("float32", 40), ("float64", 8)])
@pytest.mark.parametrize("told_by", ["next call", "check_pending"])
def test_failure_after_the_report_is_raised_later(policy, dtype, c, told_by):
    """A verified call returns when its lattice is complete.  Here a copy on another stream then sets the status bit
    that a splat which gives up its bounded wait would set (the rest of the call takes hundreds of microseconds more;
    every kernel looks at the status when it starts, whatever it is)."""
    import torch
    import permutohedral_lattice_b200 as plb
    from permutohedral_lattice_b200 import capi
    gen = torch.Generator(device="cuda").manual_seed(7)
    ref = torch.rand((8, 64, 64, 3), device="cuda", generator=gen).repeat_interleave(8, 1).repeat_interleave(8, 2)
    ref = ref.to(getattr(torch, dtype)).contiguous()
    x = torch.rand((8, 512, 512, c), device="cuda", generator=gen).to(ref.dtype)
    kw = dict(bilateral=True, theta_alpha=8.0, theta_beta=0.1)
    plb.lattice_filter_raw(x, ref, **kw)                      # the workspace has its size from here on
    bit = torch.tensor([1 << capi.PL_INTERNAL_ERROR], dtype=torch.int32).pin_memory()
    ws = policy._workspaces[(x.device.index, torch.cuda.current_stream().cuda_stream)]
    status, side = ws[8:12].view(torch.int32), torch.cuda.Stream()
    for _ in range(20):
        torch.cuda.synchronize()
        policy._verified.clear()
        out, used, _ = plb.lattice_filter_raw(x, ref, **kw)
        with torch.cuda.stream(side):
            status.copy_(bit, non_blocking=True)
        assert used.data_ptr() == ws.data_ptr()
        torch.cuda.synchronize()
        if torch.isnan(out).all():
            break
        try:                                                  # too late for some of the slice: again
            plb.check_pending()
        except plb.PlError:
            pass
    else:
        pytest.fail("the copy never came before the slice")
    policy._verified.clear()
    with pytest.raises(plb.PlError) as err:
        plb.check_pending() if told_by == "check_pending" else plb.lattice_filter_raw(x, ref, **kw)
    assert err.value.status == capi.PL_INTERNAL_ERROR
    plb.check_pending()                                       # told once
    out, _, _ = plb.lattice_filter_raw(x, ref, **kw)
    assert torch.isfinite(out).all()


def test_waiting_for_a_report_leaves_the_core_to_others(policy):
    """A verified call behind a long queue: the thread sleeps most of the wait."""
    import time
    import torch
    import permutohedral_lattice_b200 as plb
    x, ref = _data(10)
    plb.lattice_filter_raw(x, ref, **KW)
    big = torch.zeros(1 << 28, device="cuda")
    torch.cuda.synchronize()
    policy._verified.clear()
    for _ in range(600):                     # some 0.3 ms each
        big.add_(1.0)
    wall, busy = time.perf_counter(), time.thread_time()
    plb.lattice_filter_raw(x, ref, **KW)
    wall, busy = time.perf_counter() - wall, time.thread_time() - busy
    assert wall > 0.05, "the queue was empty before the call: nothing tested"
    assert busy < 0.5 * wall
