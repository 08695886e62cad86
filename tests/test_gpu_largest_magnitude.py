"""The deterministic mode's grid follows the largest magnitude of the call's input, which the lattice construction finds on its
way (spatial-only batches, whose lattice is one item's, and kept lattices by a pass of its own): wherever it stands, to the bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ABSMAX_BYTE = 16   # of the workspace's header


def _absmax(ws):
    return ws[ABSMAX_BYTE:ABSMAX_BYTE + 4].cpu().numpy().view(np.float32)[0]


# edges of tiles, rows of every width of tile, one dimension, volumes; channels that leave warps a remainder
@pytest.mark.parametrize("shape,c,guide", [((1, 1), 1, 3), ((17, 16), 21, 3), ((16, 33), 3, 3), ((45, 3), 7, 3), ((300, 1), 2, 3),
                                           ((1000,), 5, 2), ((5, 18, 19), 2, 1), ((40, 50), 40, 1), ((33, 65), 64, 0)])
@pytest.mark.parametrize("batch", [1, 3])
def test_found_wherever_it_stands(shape, c, guide, batch):
    import torch
    import permutohedral_lattice_b200 as plb
    rng = np.random.default_rng(2)
    ref = torch.rand((batch,) + shape + (guide,), device="cuda") if guide else None
    n = batch * int(np.prod(shape))
    for at in {0, n * c - 1, *rng.integers(0, n * c, 12).tolist()}:
        x = torch.empty((batch,) + shape + (c,), device="cuda").uniform_(-3.0, 3.0)
        x.view(-1)[at] = float(rng.choice([-1, 1]) * 5.75)
        _, ws, _ = plb.lattice_filter_raw(x, ref, guide > 0, 8.0, 0.2, 3.0, mode="deterministic", max_entries=0)
        assert _absmax(ws) == 5.75, at


@pytest.mark.parametrize("pd,n", [(1, 257), (6, 700), (16, 130)])
def test_of_positions(pd, n):
    import torch
    import permutohedral_lattice_b200 as plb
    pos = torch.randn((2, n, pd), device="cuda")
    for at in (0, 127, 128, n - 1, n, 2 * n - 1):
        x = torch.rand((2, n, 3), device="cuda")
        x.view(-1, 3)[at, 1] = -7.5
        _, ws = plb.filter_positions(x, pos, mode="deterministic")[:2]
        assert _absmax(ws) == 7.5, at
