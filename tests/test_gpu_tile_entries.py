"""Tile construction at its edges: coordinates on ties between two lattice cells and far from the origin (the float floor
of the GPU is not the host's), tiles of more entries than threads, grids of one to four dimensions.  Exact structure."""
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


@pytest.mark.parametrize("pd", [1, 2, 3, 4, 5, 6, 7, 8, 16])
@pytest.mark.parametrize("batch", [1, 2])
def test_ties_and_far_points(pd, batch, gpu, oracle):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(71)
    n = 700
    pos = np.rint(rng.standard_normal((batch, n, pd)) * 3).astype(np.float32) / 2      # many coordinates alike, many halves
    pos[:, 200:400] += rng.integers(-400, 400, (batch, 200, 1)).astype(np.float32)     # keys near the ends of 16 bits (pd 16)
    pos[:, 400:500] = 0.0                                                              # every residual a tie
    val = rng.random((batch, n, 1), dtype=np.float32)
    pt = torch.from_numpy(pos).cuda()
    out, ws = plb.filter_positions(torch.from_numpy(val).cuda(), pt, max_entries=0)
    st = plb.lattice_stats(ws)
    vk, vi, pv, pw = plb.export_lattice(ws, st, batch, n, pd, 2, positions=pt)
    items = [oracle.filter(val[i], pos[i]) for i in range(batch)]
    gpu.assert_structure_equal(vk, vi, pv, pw, items, "pd %d" % pd)
    gpu.assert_outputs_close(out.cpu().numpy(), np.stack([o.out for o in items]), "pd %d" % pd)


@pytest.mark.parametrize("sizes", [(517,), (19, 35), (5, 17, 18), (3, 2, 9, 21)])
@pytest.mark.parametrize("noise", [0.0, 30.0])
def test_grids_of_one_to_four_dimensions(sizes, noise, gpu, oracle):
    """noise 30: all keys of a tile are distinct, several times as many entries as threads."""
    rng = np.random.default_rng(73)
    shape = (2,) + sizes
    ref = (rng.random(shape + (1,)) * noise).astype(np.float32)
    inp = rng.random(shape + (2,), dtype=np.float32)
    args = (True, 3.0, 0.1, 1.0, False)
    want, items = oracle.lattice_filter(inp, ref, *args, structure=True)
    out, ws, call, _, rt = gpu.run_op(inp, ref, *args, max_entries=0)
    _, (vk, vi, pv, pw) = gpu.export_op(ws, call, rt)
    gpu.assert_structure_equal(vk, vi, pv, pw, items, str(sizes))
    gpu.assert_outputs_close(out.cpu().numpy(), want, str(sizes))
