"""What this framework is asked to do, as cases that can be timed.

Every case is one pass through the public operators (`pyapr.aprnet.cuda`, `pyapr.tree`) or through the U-Net that is
assembled from them (`apr_unet.APRUNet`), on an APR built from a seeded blob volume.  Kinds:

  train   forward + cross-entropy + backward of the U-Net (base 32, depth 3, two stencils): a training step
  infer   forward of the same U-Net without gradients over a batch of APRs of different sizes
  stack   forward of conv3x3x3 1->32, MaxPool, conv3x3x3 32->64, UpSampleConst, conv1x1x1 64->2 (biases, one stencil)
  layer   one APRConv (3x3x3 or 1x1x1), forward and all gradients
  tree    pyapr.tree.fill_tree_mean and fill_tree_max of the same particle features
  image   SampleParticles (image -> particles) followed by Reconstruct (particles -> image), forward and backward
"""
import os
import sys
from types import SimpleNamespace

import torch

_PACKAGE = os.path.join(os.getcwd(), "apr-cnn_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import pyapr  # noqa: E402
from apr_unet import APRUNet  # noqa: E402
from pyapr import synthetic  # noqa: E402
from pyapr.aprnet import cuda as ops  # noqa: E402
from _pyaprwrapper.aprnet.cuda import set_conv_precision  # noqa: E402

BASE, DEPTH, CLASSES = 32, 3, 2

# Blobs per voxel: the large volumes of the benchmark (5000 blobs in 512x1024x1024), and ten times as many (the
# crowded 128^3 / 200-blob volume), where a quarter of the voxels becomes a particle.
SPARSE, DENSE = 9.3e-6, 9.5e-5


def listed():
    return [
        # the smallest calls: a narrow first layer on a thumbnail of a volume, where launches and host work are the time
        dict(name="layer_f32_tiny", kind="layer", z=32, x=32, y=32, blobs=4, precision="fp32", cin=1, cout=16, k=3, dl=0, stencils=1),
        # training on small patches: 26 convolutions with a few tens of thousands of particles each
        dict(name="train_bf16_patch", kind="train", z=64, x=128, y=128, blobs=10, precision="bf16"),
        # training on one ordinary volume
        dict(name="train_bf16_volume", kind="train", z=256, x=512, y=512, blobs=625, precision="bf16"),
        # training on the largest volume that the benchmark states (28 M particles)
        dict(name="train_bf16_largest", kind="train", z=512, x=1024, y=1024, blobs=5000, precision="bf16"),
        # training in the default arithmetic (exact fp32), crowded volume
        dict(name="train_f32_dense", kind="train", z=128, x=128, y=128, blobs=200, precision="fp32"),
        # inference over a mixed batch: images of one size, 50 to 400 blobs, so the items' particle counts differ
        dict(name="infer_bf16_batch", kind="infer", z=256, x=256, y=256, blobs=50, blobs_to=400, batch=4, precision="bf16"),
        # forward-only block stack in fp32 with biases
        dict(name="stack_f32", kind="stack", z=256, x=512, y=512, blobs=625, precision="fp32"),
        # one fp32 layer of a user's own network, forward and backward
        dict(name="layer_f32_16", kind="layer", z=256, x=512, y=512, blobs=625, precision="fp32", cin=16, cout=16, k=3, dl=0, stencils=2),
        # odd everything: odd extents, odd channel counts, three stencils, one level pooled away, tensor-core arithmetic
        dict(name="layer_bf16_odd", kind="layer", z=195, x=305, y=441, blobs=500, precision="bf16", cin=33, cout=33, k=3, dl=1, stencils=3),
        # per-level channel mix of a decoder (1x1x1)
        dict(name="layer_bf16_1x1", kind="layer", z=256, x=512, y=512, blobs=625, precision="bf16", cin=64, cout=128, k=1, dl=0, stencils=2),
        # tree statistics of particle features
        dict(name="tree_f32", kind="tree", z=256, x=512, y=512, blobs=625, channels=8),
        # image in, piecewise-constant image out
        dict(name="image_f32", kind="image", z=256, x=320, y=384, blobs=300, channels=2),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    """A case of the same ranges: extents (odd ones too), blob density, channels, level, arithmetic."""
    kind = rng.choice(["train", "train", "train", "infer", "stack", "layer", "layer", "layer", "tree", "image"])
    precision = rng.choice(["bf16", "bf16", "fp32"]) if kind in ("train", "layer") else "fp32" if kind == "stack" else "bf16"
    most = {"train": 4e8 if precision == "bf16" else 8e6, "infer": 1.7e7, "stack": 7e7, "layer": 7e7, "tree": 1.3e8, "image": 4e7}[kind]
    voxels = _log(rng, 3.3e4, most)
    side = voxels ** (1 / 3)
    z = int(min(1024, max(16, side * _log(rng, 0.45, 1.0))))
    x = int(min(1024, max(16, (voxels / z) ** 0.5 * _log(rng, 0.75, 1.3))))
    y = int(min(1024, max(32, voxels / (z * x))))
    volume = z * x * y
    blobs = max(4, int(volume * _log(rng, SPARSE, max(SPARSE, min(DENSE, 4000 / volume)))))
    case = dict(kind=kind, z=z, x=x, y=y, blobs=blobs)
    if kind in ("train", "infer", "stack", "layer"):
        case["precision"] = precision
    if kind == "infer":
        case["batch"] = rng.choice([1, 2, 3, 4])
        case["blobs_to"] = min(4 * blobs, int(blobs + DENSE * volume))
    elif kind == "layer":
        case["k"] = rng.choice([3, 3, 1])
        case["dl"] = rng.choice([0, 0, 1, 2])
        widths = [1, 3, 8, 16, 24, 32, 33, 48, 64, 96, 128] if precision == "bf16" else [1, 2, 8, 16, 24, 33]
        case["cin"], case["cout"] = rng.choice(widths), rng.choice(widths[2:])
        case["stencils"] = rng.choice([1, 2, 3])
    elif kind in ("tree", "image"):
        case["channels"] = rng.choice([1, 2, 3, 4, 8] if kind == "tree" else [1, 2, 3])
    return case


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _volume(case, blobs, item=0):
    """The volume of a case: its blobs, and so the APR, belong to the case.  What is measured on the APR - intensities,
    features, gradients, weights - comes from the seed, like another channel or another frame of the same sample."""
    return synthetic.blob_image((case["z"], case["x"], case["y"]), blobs, 2000 + item, device="cuda")


def _apr(image, level_deltas):
    """The access structure on the GPU with the tables of the levels that the program uses, as a user keeps it."""
    arrays = synthetic.apr_from_image(image)
    apr = pyapr.apr_from_arrays(arrays)
    apr.init_cuda()
    for dl in level_deltas:
        apr.plan(dl)
    return arrays, apr


def _intensities(image, arrays):
    """Cell means of the volume under another exposure, with shot noise of their own."""
    parts = torch.from_numpy(synthetic.sample_particles_from_image(image, arrays)).cuda()
    return torch.poisson(parts * (0.9 + 0.2 * torch.rand(1, device="cuda")))


def _normalised(parts):
    return (parts - 100.0) / 500.0


def prepare(case, seed):
    kind = case["kind"]
    if "precision" in case:
        set_conv_precision(case["precision"])
    torch.manual_seed(seed)
    s = SimpleNamespace(kind=kind)
    if kind == "infer":
        items = []
        for b in range(case["batch"]):
            step = (case["blobs_to"] - case["blobs"]) / max(1, case["batch"] - 1)
            image = _volume(case, int(case["blobs"] + step * b), b)
            arrays, apr = _apr(image, range(DEPTH + 1))
            items.append((apr, _normalised(_intensities(image, arrays))))
        s.aprs = [apr for apr, _ in items]
        s.x = torch.zeros(len(items), 1, max(x.numel() for _, x in items), device="cuda")
        for b, (_, x) in enumerate(items):
            s.x[b, 0, :x.numel()] = x
        s.model = APRUNet(ops, 1, CLASSES, depth=DEPTH, n_filters_base=BASE).cuda().eval()
        return s

    image = _volume(case, case["blobs"])
    if kind == "image":
        _, apr = _apr(image, ())
        s.aprs = [apr]
        gain = torch.rand(1, case["channels"], 1, 1, 1, device="cuda") + 0.5
        s.image = (_normalised(torch.poisson(image))[None, None] * gain).requires_grad_(True)
        s.grad = torch.randn_like(s.image)
        s.sample, s.reconstruct = ops.SampleParticles(), ops.Reconstruct()
        return s
    if kind == "tree":
        arrays, s.apr = _apr(image, ())
        s.parts = _intensities(image, arrays)[None] * (torch.rand(case["channels"], 1, device="cuda") + 0.5)
        return s

    dls = {"train": range(DEPTH + 1), "stack": (0, 1), "layer": (case.get("dl"),)}[kind]
    arrays, apr = _apr(image, dls)
    s.aprs = [apr]
    if kind == "layer":
        n = int(pyapr.aprnet.utils.number_particles(apr, case["dl"]))
        s.level_deltas = torch.full((1,), case["dl"], dtype=torch.int32)
        s.conv = ops.APRConv(case["cin"], case["cout"], nstencils=case["stencils"], kernel_size=(case["k"],) * 3, precision=case["precision"]).cuda()
        s.x = torch.randn(1, case["cin"], n, device="cuda").relu_().requires_grad_(True)
        s.grad = torch.randn(1, case["cout"], n, device="cuda")
        return s
    parts = _intensities(image, arrays)
    s.x = _normalised(parts)[None, None]
    if kind == "train":
        s.labels = (parts > 300.0).long()[None]
        s.model = APRUNet(ops, 1, CLASSES, depth=DEPTH, n_filters_base=BASE).cuda()
    else:
        s.modules = torch.nn.ModuleList([ops.APRConv(1, 32), ops.MaxPool(), ops.APRConv(32, 64), ops.UpSampleConst(),
                                         ops.APRConv(64, CLASSES, kernel_size=(1, 1, 1))]).cuda()
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(s):
    if s.kind == "train":
        s.model.zero_grad(set_to_none=True)
        logits = s.model(s.x, s.aprs)
        loss = torch.nn.functional.cross_entropy(logits, s.labels)
        loss.backward()
        return [loss.detach(), logits.detach()] + [p.grad for p in s.model.parameters()]
    if s.kind == "infer":
        with torch.no_grad():
            return s.model(s.x, s.aprs)
    if s.kind == "stack":
        with torch.no_grad():
            level_deltas = torch.zeros(1, dtype=torch.int32)
            y = s.x
            for m in s.modules:
                y = m(y, s.aprs, level_deltas)
            return y
    if s.kind == "layer":
        s.conv.zero_grad(set_to_none=True)
        s.x.grad = None
        out = s.conv(s.x, s.aprs, s.level_deltas)
        out.backward(s.grad)
        return [out.detach(), s.x.grad, s.conv.weight.grad, s.conv.bias.grad]
    if s.kind == "tree":
        return [pyapr.tree.fill_tree_mean(s.apr, s.parts), pyapr.tree.fill_tree_max(s.apr, s.parts)]
    s.image.grad = None
    parts = s.sample(s.image, s.aprs)
    out = s.reconstruct(parts, s.aprs)
    out.backward(s.grad)
    return [parts.detach(), out.detach(), s.image.grad]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _particles(case, blobs):
    """Particles of a blob volume, from its blob density (fitted to the generator, within about 15 %)."""
    volume = case["z"] * case["x"] * case["y"]
    return volume * min(0.6, 0.235 * (blobs / volume / DENSE) ** 0.65)


#: feature locations at level deltas 0 to 3, and tree nodes, per particle
_AT_LEVEL = (1.0, 0.5, 0.15, 0.033)
_TREE = 1 / 7


def _unet_flops(n):
    """Multiply-adds x 2 of one forward pass of the U-Net over n particles."""
    w = [BASE << i for i in range(DEPTH + 1)]
    total = 54.0 * (w[0] + w[0] * w[0])
    for i in range(DEPTH):
        total += 54.0 * (w[i] * w[i + 1] + w[i + 1] * w[i + 1]) * _AT_LEVEL[i + 1]
        total += 2.0 * w[i + 1] * w[i] * _AT_LEVEL[i + 1] + 54.0 * (w[i + 1] * w[i] + w[i] * w[i]) * _AT_LEVEL[i]
    return n * (total + 2.0 * w[0] * CLASSES)


def _unet_bytes(n, train):
    """fp32 activations of the U-Net: GroupNorm needs a whole layer before its first value, so every convolution's
    output is written once and read once, and a training pass also reads each of them once more and does the same with its gradient."""
    w = [BASE << i for i in range(DEPTH + 1)]
    values = 2.0 * w[0]
    for i in range(DEPTH):
        values += 2.0 * w[i + 1] * _AT_LEVEL[i + 1] + w[i] * _AT_LEVEL[i + 1] + 2.0 * w[i] * _AT_LEVEL[i]
    return n * (4.0 * values * (5 if train else 2) + 4 + 4 * CLASSES + (8 if train else 0))


def work(case):
    """Bytes and operations of one pass, from the expected number of particles."""
    kind = case["kind"]
    n = _particles(case, case["blobs"])
    if kind == "train":
        return {"bytes": _unet_bytes(n, True), "flops": 3 * _unet_flops(n)}
    if kind == "infer":
        step = (case["blobs_to"] - case["blobs"]) / max(1, case["batch"] - 1)
        n = sum(_particles(case, int(case["blobs"] + step * b)) for b in range(case["batch"]))
        return {"bytes": _unet_bytes(n, False), "flops": _unet_flops(n)}
    if kind == "stack":
        return {"bytes": n * (4.0 + 4 * CLASSES), "flops": n * (54.0 * 32 + 54.0 * 32 * 64 * _AT_LEVEL[1] + 2.0 * 64 * CLASSES)}
    if kind == "layer":
        n *= _AT_LEVEL[case["dl"]]
        per = (54.0 if case["k"] == 3 else 2.0) * case["cin"] * case["cout"]
        # features and upstream gradient in, output and input gradient out
        return {"bytes": n * 8.0 * (case["cin"] + case["cout"]), "flops": 3 * per * n}
    if kind == "tree":
        return {"bytes": 4.0 * case["channels"] * n * (1 + 2 * _TREE), "flops": 2.0 * case["channels"] * n * (1 + _TREE)}
    volume = case["z"] * case["x"] * case["y"]
    # image and upstream gradient in, image and image gradient out, particles out
    return {"bytes": 4.0 * case["channels"] * (4 * volume + n), "flops": 2.0 * case["channels"] * volume}


def tolerance(case):
    if case["kind"] == "tree":
        return {"rel": 1e-6, "max": 1e-5}
    if case.get("precision") == "bf16":
        return {"rel": 1e-2}        # operands of the contractions are bf16
    if case["kind"] == "train":
        return {"rel": 1e-4}        # fp32 sums through some forty layers, each way, with ReLU gates between them
    return {"rel": 1e-5}
