"""The blur passes of float rows, bit for bit: three products and two sums in double, rounded once to float.

Points on a line (pd 1), one in every second cell, so that every vertex has the product of one weight and one value in
its row and no sum depends on an order: what follows is fixed to the last bit, in the kernels as in the oracle.  The
values spread over sixty binades with both signs, and in some channels lie where a quarter of them is subnormal: sums
of three that fit no float, ties among them.  Every form the passes come in: small lattices (1, 2 and 4 vertices a
thread), two passes a launch, one, and more rows than stay in L2."""
import numpy as np
import pytest

STEP = np.float32(np.sqrt(3.0) / 2.0)        # a cell of the line


def _points(batch, n, channels, seed, twice=False):
    """twice: the last point stands there twice, the second time with zeros, so that the bound need not be the worst case."""
    rng = np.random.default_rng(seed)
    cell = 2 * np.arange(n) - n + rng.uniform(0.3, 0.7, (batch, n))
    pos = (cell * STEP).astype(np.float32)[..., None]
    x = rng.standard_normal((batch, n, channels)) * np.exp2(rng.uniform(-40, 20, (batch, n, channels)))
    x[..., ::3] = rng.choice([-1, 1], x[..., ::3].shape) * np.exp2(rng.uniform(-124, -120, x[..., ::3].shape))
    if twice:
        pos, x = np.concatenate([pos, pos[:, -1:]], 1), np.concatenate([x, 0 * x[:, -1:]], 1)
    return pos, x.astype(np.float32)


def _mix(a, b, c):
    a, b, c = (t.astype(np.float64) for t in (a, b, c))
    return ((0.25 * a + 0.5 * b) + 0.25 * c).astype(np.float32)


def _by_hand(x, weight, key, reverse):
    """x [n, c]; weight [n, 2] and key [n, 2] (first coordinate) of each point's two vertices -> output [n, c]."""
    n, c = x.shape
    first = key.min() - 1
    rows = np.zeros((key.max() - first + 2, c + 1), np.float32)
    there = np.zeros(len(rows), bool)
    twice = n - 1 if (key[-1] == key[-2]).all() else n
    for r in range(2):
        at = key[:, r] - first
        assert len(np.unique(at)) == twice and not there[at].any()     # one point a vertex
        there[at] = True
        rows[at[:twice], :c] = (weight[:, r, None] * x)[:twice]
        np.add.at(rows[:, c], at, weight[:, r])
    for axis in ((1, 0) if reverse else (0, 1)):
        step = -1 if axis == 0 else 1                              # the "+" neighbour: one up in all but `axis`, pd down there
        plus, minus = np.roll(rows, -step, 0), np.roll(rows, step, 0)
        rows = np.where(there[:, None], _mix(plus, rows, minus), np.float32(0))
    acc = weight[:, :1] * rows[key[:, 0] - first] + weight[:, 1:] * rows[key[:, 1] - first]
    return acc[:, :c] * (1.0 / acc[:, c:].astype(np.float64)).astype(np.float32)


@pytest.mark.parametrize("reverse", [False, True])
def test_by_hand_is_the_oracle(oracle, reverse):
    pos, x = _points(1, 3000, 6, 5)
    want = oracle.filter(x[0], pos[0], reverse=reverse)
    got = _by_hand(x[0], want.pix_weight, want.pixel_keys()[..., 0].astype(np.int64), reverse)
    assert np.array_equal(got.view(np.uint32), want.out.view(np.uint32))


ROUTES = [
    (1, 2000, 3, 0), (1, 4096, 14, 8192), (1, 6000, 7, 0), (1, 15000, 3, -1),        # small lattices
    (1, 15000, 3, 0), (2, 15000, 5, 0), (4, 15000, 11, 150000),                      # pairs of passes
    (12, 15000, 3, 0), (6, 15000, 21, 0),                                            # one a launch
    (12, 15000, 71, 0),                                                              # 6.5 M float4
]


@pytest.mark.gpu
@pytest.mark.parametrize("extremes", [False, True], ids=["finite", "extremes"])
@pytest.mark.parametrize("batch,n,channels,bound", ROUTES)
def test_blur_has_the_bits_of_sums_in_double(batch, n, channels, bound, extremes):
    """bound -1: one less than the worst case.  extremes: infinities, NaN and the largest floats among the values, so that a pass meets every mixture of them."""
    import torch
    import permutohedral_lattice_b200 as plb
    pos, x = _points(batch, n, channels, n + channels, bound < 0)
    if bound < 0:
        n += 1
        bound += 2 * batch * n
    if extremes:
        rng = np.random.default_rng(7)
        odd = np.array([np.inf, -np.inf, np.nan, 3.4028235e38, -3.4028235e38, 0.0, -0.0], np.float32)
        x = np.where((rng.random(x.shape) < 0.1) & (x != 0), rng.choice(odd, x.shape), x)
    pt, xt = torch.from_numpy(pos).cuda(), torch.from_numpy(x).cuda()
    for reverse in (False, True):
        out, ws = plb.filter_positions(xt, pt, reverse, max_entries=bound)
        st = plb.lattice_stats(ws)
        assert st.num_vertices == len(np.unique(pos)) * 2 if batch == 1 else 2 * batch * n
        keys, _, vertex, weight = plb.export_lattice(ws, st, batch, n, 1, channels + 1, positions=pt)
        key = keys.cpu().numpy()[:, 0].astype(np.int64)[vertex.cpu().numpy()]
        for b in range(batch):
            with np.errstate(all="ignore"):
                want = _by_hand(x[b], weight[b].cpu().numpy(), key[b], reverse)
            got = out[b].cpu().numpy()
            differ = (got != want) & ~(np.isnan(got) & np.isnan(want))
            assert not differ.any(), "%d of %d differ" % (differ.sum(), differ.size)
