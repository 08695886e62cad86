"""The splat that walks columns of points instead of sorting a tile's splats: partial tiles, narrow images, every lane
count, both sides of the rule that chooses it (theta 1 has few splats an entry, theta 6 many), against the oracle with the
bounds of every comparison with it (gpu_helpers: float sums in another order)."""
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


def _check(gpu, oracle, shape, channels, r, theta, seed, noise=0.0):
    import torch
    import permutohedral_lattice_b200 as plb
    from conftest import bits
    rng = np.random.default_rng(seed)
    # a guide that is constant over blocks, so that points share vertices
    ref = None
    if r:
        ref = np.zeros((2,) + shape + (r,), np.float32)
        ref[..., :] = (np.arange(shape[-1]) // 9 % 3 * np.float32(0.4))[..., None]
        ref += np.float32(noise) * rng.standard_normal(ref.shape).astype(np.float32)
    wide = rng.standard_normal((2,) + shape + (max(channels),)).astype(np.float32)
    rt = None if ref is None else torch.from_numpy(ref).cuda()
    args = (bool(r), theta, 0.3, theta)
    want = oracle.lattice_filter(wide, ref, *args)
    for c in channels:
        flat = torch.empty(wide[..., :c].size + 1, device="cuda")
        for x in (flat[:-1], flat[1:]):   # on a 16-byte boundary and off it
            x = x.view((2,) + shape + (c,))
            x.copy_(torch.from_numpy(np.ascontiguousarray(wide[..., :c])))
            what = "%s, %d channels, theta %g" % (shape, c, theta)
            got, _, _ = plb.lattice_filter_raw(x, rt, *args)
            gpu.assert_outputs_close(got.cpu().numpy(), want[..., :c], what)
            lattice = plb.Lattice(rt, (2,) + shape, *args, max_channels=c, mode="deterministic")
            gpu.assert_outputs_close(lattice.apply(x).cpu().numpy(), want[..., :c], what + ", lattice kept")
            fixed, _, _ = plb.lattice_filter_raw(x, rt, *args, mode="deterministic")
            kept = lattice.apply(x, mode="deterministic")
            assert np.array_equal(bits(fixed.cpu().numpy()), bits(kept.cpu().numpy())), what
            gpu.assert_outputs_close(kept.cpu().numpy(), want[..., :c], what + ", fixed-point sums")


@pytest.mark.parametrize("theta", [1.0, 6.0])
@pytest.mark.parametrize("shape", [(1, 1), (7, 16), (9, 17), (33, 45), (70, 1), (40, 3), (17, 7), (16, 100)])
def test_images_without_guide(shape, theta, gpu, oracle):
    _check(gpu, oracle, shape, [1, 2, 3, 4, 5, 8, 10, 15, 16, 20, 21, 33, 62, 63, 64, 70], 0, theta, 5)


@pytest.mark.parametrize("theta", [1.0, 6.0])
@pytest.mark.parametrize("shape,r", [((33, 45), 1), ((70, 1), 1), ((3, 9, 20), 0), ((3, 17, 33), 1), ((2, 40, 5), 1)])
def test_guides_and_volumes(shape, r, theta, gpu, oracle):
    _check(gpu, oracle, shape, [1, 2, 3, 4, 7, 12, 21, 64], r, theta, 6)


@pytest.mark.parametrize("noise", [0.1, 0.4])
@pytest.mark.parametrize("shape,r", [((33, 45), 1), ((40, 3), 1), ((3, 17, 33), 1), ((20, 37), 2)])
def test_noisy_guides(shape, r, noise, gpu, oracle):
    """Few entries (theta 40), between which the noise sends neighbouring points: both sides of the rule on changes of entry
    from row to row."""
    _check(gpu, oracle, shape, [1, 2, 3, 5, 21, 64], r, 40.0, 7, noise)


@pytest.mark.parametrize("shape,r,theta", [((100, 120), 0, 40.0), ((97, 33), 0, 12.0), ((30, 17, 33), 0, 6.0), ((30, 17, 33), 0, 40.0),
                                           ((40, 35, 20), 1, 20.0), ((100, 70), 1, 60.0)])
def test_vertices_that_many_tiles_share(shape, r, theta, gpu, oracle):
    """Narrow rows in pieces of eight points, where a vertex has more than 4 (pd 2), 10 (pd 3) or 16 (pd 4) entries."""
    _check(gpu, oracle, shape, [1, 2, 3], r, theta, 8)
