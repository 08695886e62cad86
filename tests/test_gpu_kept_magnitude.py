"""Deterministic calls through a kept lattice right behind the kernel that writes their input: its largest magnitude, which is
looked for before the launch it overlaps has ended, is that of the values written, every time."""
import pytest

pytestmark = pytest.mark.gpu

ABSMAX_BYTE = 16   # of the workspace's header


@pytest.mark.parametrize("shape,guide,c", [((2, 300, 280), 3, 21), ((1, 64, 70), 3, 3), ((3, 200, 200), 0, 5)])
def test_of_what_the_kernel_before_wrote(shape, guide, c):
    import torch
    import permutohedral_lattice_b200 as plb
    gen = torch.Generator(device="cuda").manual_seed(4)
    ref = torch.rand(shape + (guide,), generator=gen, device="cuda") if guide else None
    lat = plb.Lattice(ref, spatial_shape=shape, bilateral=guide > 0, theta_alpha=8.0, theta_beta=0.2, theta_gamma=3.0,
                      max_channels=c, mode="deterministic")
    values = torch.rand(shape + (c,), generator=gen, device="cuda")
    values.view(-1)[-1] = 1.0
    x = torch.empty_like(values)
    words, wants, outs = [], [], []
    for k in range(40):
        scale = 2.0 ** ((7 * k) % 23 - 5)                # up and down
        torch.mul(values, scale, out=x)                  # the kernel right before the call
        outs.append(lat.apply(x, mode="deterministic"))
        words.append(lat.workspace[ABSMAX_BYTE:ABSMAX_BYTE + 4].clone())
        wants.append(scale)
    assert [float(w.view(torch.float32)) for w in words] == wants
    for out, scale in zip(outs, wants):                  # the same to the bit when nothing is under way
        torch.mul(values, scale, out=x)
        torch.cuda.synchronize()
        assert torch.equal(out, lat.apply(x, mode="deterministic"))
    # and a chain: every call's input is the output of the call before it
    y, stored = values, []
    for _ in range(6):
        y = lat.apply(y, mode="deterministic")
        stored.append((lat.workspace[ABSMAX_BYTE:ABSMAX_BYTE + 4].clone(), y))
    before = [values] + [o for _, o in stored[:-1]]
    assert [float(w.view(torch.float32)) for w, _ in stored] == [float(b.abs().max()) for b in before]
