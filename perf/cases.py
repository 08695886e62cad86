"""The work that a user of this package has it do, as timed cases.

`listed()` names twelve calls through the public entry points: `lattice_filter` forward and with its gradient,
in single and double precision, in the deterministic mode, with one lattice for both directions and with a purely
spatial kernel; `filter_positions`; `DenseCRF`; `HostPipeline`.  `draw(rng)` gives further cases of the same ranges.
Inputs are synthetic, made on the GPU from a seed with the distributions of `permutohedral_lattice_b200/workloads.py`:
piecewise constant images with shading and noise, ellipsoid phantoms, label distributions, patch features.
"""
import math

import torch

from permutohedral_lattice_b200.crf import DenseCRF
from permutohedral_lattice_b200.host_pipeline import HostPipeline
from permutohedral_lattice_b200.lattice_filter import filter_positions, lattice_filter

# The largest listed call: 16 images of 512 x 512 with 21 labels.  No drawn case has more points or values.
MOST_POINTS = 16 * 512 * 512
MOST_VALUES = MOST_POINTS * 21


def _case(what, shape, batch=1, channels=3, guide=3, bilateral=True, train=False, reuse=False, mode="atomic",
          dtype="float32", theta_alpha=8.0, theta_beta=0.125, theta_gamma=3.0, pd=0, iterations=0, name=None):
    """what: "filter", "positions", "crf" or "host".  shape: the spatial sizes, as text.  guide: channels of the
    reference image.  train: the gradient is computed too.  pd: feature dimensions of a positions call."""
    case = {"what": what, "shape": shape, "batch": batch, "channels": channels, "guide": guide,
            "bilateral": bilateral, "train": train, "reuse": reuse, "mode": mode, "dtype": dtype,
            "theta_alpha": theta_alpha, "theta_beta": theta_beta, "theta_gamma": theta_gamma, "pd": pd,
            "iterations": iterations}
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # a thumbnail or a crop, filtered on its own: latency of one call (odd sides)
        _case("filter", "33x45", name="thumbnail"),
        # one photograph of the demo's size, smoothed by itself
        _case("filter", "800x1200", name="photo"),
        # a noisy grey image guided by the clean colour image, as a layer in training
        _case("filter", "1024x1024", channels=1, train=True, theta_alpha=16.0, theta_beta=0.1, name="grey_by_rgb"),
        # message passing of a dense CRF over a training batch with 21 labels: the benchmark's workload, the largest
        _case("filter", "512x512", batch=16, channels=21, train=True, theta_alpha=80.0, theta_beta=0.0625,
              name="crf_messages"),
        # the same CRF's inference on one photograph of ragged size: two lattices, five iterations
        _case("crf", "375x500", channels=21, theta_alpha=80.0, theta_beta=0.0625, iterations=5, name="crf_inference"),
        # a small training batch of ragged images with another number of classes, one lattice for both directions
        _case("filter", "321x481", batch=4, channels=10, train=True, reuse=True, theta_alpha=40.0, theta_beta=0.1,
              name="ragged_batch_reuse"),
        # two volumes of a scan (odd depth), two channels guided by one, in training
        _case("filter", "111x128x120", batch=2, channels=2, guide=1, train=True, theta_alpha=5.0, theta_beta=0.1,
              name="volumes"),
        # non-local-means style filtering: 16-dimensional patch features given as positions
        _case("positions", "1024x1024", pd=16, name="patch_features"),
        # the CRF's smoothness kernel: no reference image
        _case("filter", "512x512", batch=8, channels=21, guide=0, bilateral=False, train=True, name="spatial_only"),
        # a layer in double precision
        _case("filter", "512x512", train=True, dtype="float64", name="double"),
        # bitwise reproducible training
        _case("filter", "512x512", batch=2, channels=21, train=True, mode="deterministic", theta_alpha=80.0,
              theta_beta=0.0625, name="deterministic"),
        # images that live in host memory, through the copying pipeline
        _case("host", "512x512", batch=6, channels=21, theta_alpha=80.0, theta_beta=0.0625, name="host_batch"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["filter"] * 6 + ["spatial", "volume", "volume", "positions", "crf", "host"])
    alpha = round(math.exp(rng.uniform(math.log(4.0), math.log(100.0))), 2)
    beta = round(rng.uniform(0.05, 0.2), 3)
    train = rng.random() < 0.5
    h, w = _log_int(rng, 24, 1200), _log_int(rng, 24, 1200)
    batch = _log_int(rng, 1, 16)
    channels = rng.choice([1, 2, 3, 21, _log_int(rng, 1, 40)])
    if what == "positions":
        pd = rng.choice([3, 5, 8, 16])
        h, w = _log_int(rng, 32, 1000), _log_int(rng, 32, 1000)
        batch = max(1, min(batch, 1048576 // (h * w)))
        return _case("positions", "%dx%d" % (h, w), batch=batch, channels=rng.choice([1, 3, 4]), pd=pd)
    if what == "volume":
        d, h, w = (_log_int(rng, 12, 140) for _ in range(3))
        batch = max(1, min(batch, MOST_POINTS // (d * h * w)))
        return _case("filter", "%dx%dx%d" % (d, h, w), batch=batch, channels=rng.choice([1, 2]), guide=1, train=train,
                     theta_alpha=round(rng.uniform(3.0, 10.0), 2), theta_beta=beta)
    if what == "crf":
        h, w, channels = _log_int(rng, 64, 640), _log_int(rng, 64, 640), rng.choice([2, 21, 21, _log_int(rng, 3, 30)])
        batch = max(1, min(batch, 4, MOST_VALUES // (10 * h * w * channels)))
        return _case("crf", "%dx%d" % (h, w), batch=batch, channels=channels, theta_alpha=max(20.0, alpha),
                     theta_beta=beta, iterations=rng.choice([3, 5]))
    most = MOST_VALUES
    mode, dtype, reuse = "atomic", "float32", False
    if what == "host":
        most, train = MOST_VALUES // 4, False
    elif what == "filter":
        option = rng.random()
        if option < 0.15:
            dtype, most = "float64", MOST_VALUES // 32
        elif option < 0.3:
            mode, most = "deterministic", MOST_VALUES // 8
        else:
            reuse = train and rng.random() < 0.3
    batch = max(1, min(batch, MOST_POINTS // (h * w), most // (h * w * channels)))
    channels = max(1, min(channels, most // (h * w * batch)))
    if what == "spatial":
        return _case("filter", "%dx%d" % (h, w), batch=batch, channels=channels, guide=0, bilateral=False, train=train,
                     theta_gamma=round(rng.uniform(1.0, 8.0), 2))
    return _case(what, "%dx%d" % (h, w), batch=batch, channels=channels, train=train, reuse=reuse, mode=mode,
                 dtype=dtype, theta_alpha=alpha, theta_beta=beta)


def _sizes(case):
    return tuple(int(s) for s in case["shape"].split("x"))


def _images(gen, batch, h, w, cells=64):
    """Voronoi colour maps with slow shading and noise (sigma 0.05), in 0..1: [batch, h, w, 3]."""
    dev = gen.device
    sites = torch.rand((batch, cells, 2), generator=gen, device=dev) * torch.tensor([h, w], device=dev)
    colours = torch.rand((batch, cells, 3), generator=gen, device=dev)
    y = torch.arange(h, device=dev, dtype=torch.float32).view(1, h, 1)
    x = torch.arange(w, device=dev, dtype=torch.float32).view(1, 1, w)
    best = torch.full((batch, h, w), math.inf, device=dev)
    label = torch.zeros((batch, h, w), dtype=torch.int64, device=dev)
    for k in range(cells):
        dist = (y - sites[:, k, 0].view(-1, 1, 1)) ** 2 + (x - sites[:, k, 1].view(-1, 1, 1)) ** 2
        nearer = dist < best
        best = torch.where(nearer, dist, best)
        label = torch.where(nearer, k, label)
    img = torch.gather(colours, 1, label.view(batch, h * w, 1).expand(-1, -1, 3)).view(batch, h, w, 3)
    freq = 1.0 + 2.0 * torch.rand((batch, 2, 1, 1), generator=gen, device=dev)
    phase = 2 * math.pi * torch.rand((batch, 1, 1, 3), generator=gen, device=dev)
    shade = torch.sin(2 * math.pi * (freq[:, 0] * y / h + freq[:, 1] * x / w))
    img = img + 0.1 * shade[..., None] * torch.cos(phase)
    img = img + 0.05 * torch.randn(img.shape, generator=gen, device=dev)
    return img.clamp_(0.0, 1.0)


def _phantoms(gen, batch, d, h, w, count=12):
    """Overlapping ellipsoids of constant intensity: [batch, d, h, w, 1]."""
    dev = gen.device
    axes = [torch.arange(s, device=dev, dtype=torch.float32).view([-1 if i == k else 1 for i in range(3)])
            for k, s in enumerate((d, h, w))]
    size = torch.tensor([d, h, w], dtype=torch.float32)
    vol = torch.zeros((batch, d, h, w, 1), device=dev)
    for b in range(batch):
        par = torch.rand((count, 7), generator=gen, device=dev).cpu()
        for k in range(count):
            centre, radius = (0.2 + 0.6 * par[k, :3]) * size, (0.08 + 0.22 * par[k, 3:6]) * size
            inside = sum(((axes[i] - float(centre[i])) / float(radius[i])) ** 2 for i in range(3)) <= 1.0
            vol[b, ..., 0][inside] = float(par[k, 6])
    return vol


def _labels(gen, shape, channels):
    """Label distributions: softmax of normal logits."""
    return torch.softmax(3.0 * torch.randn(shape + (channels,), generator=gen, device=gen.device), -1)


def _patch_features(gen, rgb, pd):
    """The 5 x 5 colour patches around every pixel on pd orthonormal directions: [batch, h * w, pd]."""
    batch, h, w, _ = rgb.shape
    pad = torch.nn.functional.pad(rgb.permute(0, 3, 1, 2), (2, 2, 2, 2), mode="replicate").permute(0, 2, 3, 1)
    directions = torch.linalg.qr(torch.randn((75, pd), generator=gen, device=gen.device).cpu().double())[0]
    out = torch.zeros((batch, h, w, pd), device=gen.device, dtype=torch.float64)
    for k in range(25):
        part = pad[:, k // 5:k // 5 + h, k % 5:k % 5 + w].double()
        for c in range(3):
            out += part[..., c:c + 1] * directions[3 * k + c].to(gen.device)
    return (out / 0.2).float().reshape(batch, h * w, pd)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    sizes, batch, channels = _sizes(case), case["batch"], case["channels"]
    shape = (batch,) + sizes
    state = {"case": case}
    if case["what"] == "positions":
        rgb = _images(gen, batch, *sizes)
        state["positions"] = _patch_features(gen, rgb, case["pd"])
        extra = torch.rand((batch, sizes[0] * sizes[1], max(0, channels - 3)), generator=gen, device="cuda")
        state["input"] = torch.cat([rgb.view(batch, -1, 3)[..., :channels], extra], -1).contiguous()
        return state
    if len(sizes) == 3:
        ref = _phantoms(gen, batch, *sizes)
        x = ref + 0.2 * torch.randn(shape + (channels,), generator=gen, device="cuda")
    else:
        ref = _images(gen, batch, *sizes) if case["bilateral"] else None
        if channels == 1:
            grey = ref.mean(-1, keepdim=True) if ref is not None else torch.rand(shape + (1,), generator=gen, device="cuda")
            x = grey + 0.1 * torch.randn(grey.shape, generator=gen, device="cuda")
        elif channels == 3 and ref is not None:
            x = ref.clone()
        else:
            x = _labels(gen, shape, channels)
    if case["what"] == "crf":
        # a user's program has the network's unaries and the image; building the CRF is part of the call
        state["unaries"], state["image"] = -torch.log(x + 1e-6), ref
        return state
    if case["what"] == "host":
        # the pipeline and the pinned buffers are what a program keeps
        state["input"], state["reference"] = x.cpu().pin_memory(), ref.cpu().pin_memory()
        state["output"] = torch.empty_like(state["input"]).pin_memory()
        state["pipeline"] = HostPipeline()
        return state
    dtype = getattr(torch, case["dtype"])
    state["input"] = x.to(dtype).contiguous()
    state["reference"] = None if ref is None else ref.to(dtype).contiguous()
    if case["train"]:
        state["input"].requires_grad_()
        state["grad"] = torch.randn(x.shape, generator=gen, device="cuda").to(dtype)
    return state


def run(state):
    case = state["case"]
    thetas = (case["theta_alpha"], case["theta_beta"], case["theta_gamma"])
    if case["what"] == "positions":
        return filter_positions(state["input"], state["positions"])[0]
    if case["what"] == "crf":
        crf = DenseCRF(state["image"], case["channels"], *thetas)
        return crf.infer(state["unaries"], case["iterations"])
    if case["what"] == "host":
        return state["pipeline"].filter(state["input"], state["reference"], True, *thetas, out_host=state["output"])
    out = lattice_filter(state["input"], state["reference"], case["bilateral"], *thetas, mode=case["mode"],
                         reuse_lattice=case["reuse"])
    if not case["train"]:
        return out
    return [out.detach(), torch.autograd.grad(out, state["input"], state["grad"])[0]]


def work(case):
    """Every input read once and every output written once; the multiply-adds of the simplex search (about
    3 (pd + 1)^2 operations a point) and of splatting and slicing (2 (pd + 1)(channels + 1) each a point and pass)."""
    sizes = _sizes(case)
    n = case["batch"] * math.prod(sizes)
    c = case["channels"]
    real = 8 if case["dtype"] == "float64" else 4
    if case["what"] == "positions":
        pd = case["pd"]
        values, features = 2 * c, pd
    else:
        features = case["guide"] if case["bilateral"] else 0
        pd = len(sizes) + features
        values = 2 * c if not case["train"] else 4 * c
    per_apply = 4 * (pd + 1) * (c + 1)
    applies = 2 * case["iterations"] if case["what"] == "crf" else 2 if case["train"] else 1
    return {"bytes": real * n * (values + features), "flops": n * (3 * (pd + 1) ** 2 + applies * per_apply)}


def tolerance(case):
    """Sums of 32-bit (64-bit) values in any order, through splat, blur and slice."""
    return {"rel": 1e-12} if case["dtype"] == "float64" else {"rel": 1e-5}
