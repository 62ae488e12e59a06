"""The work that programs built on this library give it, as cases that can be timed.

A case names one kind of call with its sizes and options:
  pair     one stereo pair on device buffers (elas_b200_process_device): the call of a perception pipeline whose
           images are on the GPU already
  frames   a pass over a ring of device frame buffers through one handle: video, where capture fills one set of
           buffers while the other is matched
  host     one pair from host arrays to host arrays (Elas.process): the drop-in call of a program that has its
           images in ordinary memory
  learned  one pair on device buffers with the learned support-point proposal
  batch    independent pairs of mixed sizes and disparity ranges in one call (elas_b200_process_batch_device)
  train    one optimisation step of the proposal network (forward, loss, backward, Adam)

Inputs are the library's seeded synthetic scenes (slanted textured planes with textureless patches and noise); the
training step gets seeded features of the range that pooled descriptors have.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cuda-stereo-matching_b200"))

import elas_b200 as eb  # noqa: E402
import proposal  # noqa: E402

CH, TAPS, LAYERS, NBINS = 32, 9, 4, 64      # the proposal network: channels, 3x3 taps, layers, disparity bins
LAYER_PARAMS = TAPS * CH * CH + CH
SCALE = 0.125                               # score = SCALE * <left feature, right feature>


def _pair(name, width, height, disp_max, scene, kind="pair", params="post", subsampling=False, **more):
    return dict(name=name, kind=kind, width=width, height=height, disp_max=disp_max, scene=scene, params=params,
                subsampling=subsampling, **more)


def listed():
    return [
        # the smallest calls: a thumbnail, where launches and latency are all there is
        _pair("pair_160x120", 160, 120, 47, 3),
        # an indoor still of the size of the classic stereo sets
        _pair("pair_450x375", 450, 375, 63, 0),
        # the driving-camera size that the benchmark quotes
        _pair("pair_1242x375", 1242, 375, 255, 1),
        # the same camera with the parameters that a default-constructed matcher has (corner points, wide gaps
        # interpolated, median)
        _pair("pair_1242x375_defaults", 1242, 375, 255, 1, params="defaults"),
        # matching and left/right check alone, at a size that no tile divides: the reference's own process()
        _pair("pair_741x497_plain", 741, 497, 127, 3, params="plain"),
        # full HD, half-resolution output maps
        _pair("pair_1920x1080_subsampled", 1920, 1080, 255, 3, subsampling=True),
        # the largest single pair: high-resolution survey images
        _pair("pair_2880x1988", 2880, 1988, 511, 2),
        # a VGA video stream, double-buffered
        _pair("frames_640x480", 640, 480, 128, 3, kind="frames", buffers=2),
        # host arrays in, host arrays out
        _pair("host_1242x375", 1242, 375, 255, 1, kind="host"),
        # the learned proposal at the size it was trained for
        _pair("learned_1242x375", 1242, 375, 255, 1, kind="learned"),
        # offline processing of a mixed collection: widths 320-1920, heights 240-1080, ranges 64-256
        dict(name="batch_16", kind="batch", pairs=16, shapes_seed=7),
        # training step: 16 pairs of 1242x375 (93 x 310 cells), the trainer's default batch
        dict(name="train_16", kind="train", pairs=16, hd=93, wd=310, disp_max=255),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair"] * 8 + ["frames"] * 2 + ["host"] * 2 + ["learned", "batch", "train"])
    if kind == "batch":
        return dict(kind=kind, pairs=rng.randint(2, 16), shapes_seed=rng.randrange(1 << 20))
    if kind == "train":
        w, h = _log(rng, 320, 1242), _log(rng, 240, 375)
        return dict(kind=kind, pairs=rng.randint(2, 16), hd=h // 4, wd=w // 4, disp_max=rng.choice([63, 127, 255]))
    width = _log(rng, 120, 2880)
    height = max(80, min(1988, int(width * rng.uniform(0.3, 0.75))))
    case = dict(kind=kind, width=width, height=height, disp_max=_log(rng, 24, max(32, min(511, width // 4))),
                scene=3, params=rng.choice(["post", "post", "defaults", "plain"]),
                subsampling=rng.random() < 0.15 and kind == "pair")
    if kind == "learned":
        case["params"] = "post"
    if kind == "frames":
        case["buffers"] = rng.randint(2, 4)
        case["width"] = min(case["width"], 1242)
        case["height"] = min(case["height"], 931)
    return case


def _shapes(case):
    """(width, height, disp_max) of a batch's pairs: the ranges of the benchmark's mixed batch."""
    rng = random.Random(case["shapes_seed"])
    return [(16 * rng.randint(20, 120), 16 * rng.randint(15, 67), rng.choice([64, 128, 256]))
            for _ in range(case["pairs"])]


def _params(case):
    if case["params"] == "defaults":
        p = eb.params_default()
        p.disp_max = case["disp_max"]
    else:
        p = eb.params_config(case["disp_max"], post=case["params"] == "post")
    p.subsampling = case["subsampling"]
    return p


def _device_pair(scene, seed, width, height, disp_max, out_shape):
    left, right, _, _ = eb.synth_pair(scene, seed, width=width, height=height, disp_max=disp_max, gt=False)
    return [torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(),
            torch.empty(out_shape, dtype=torch.float32, device="cuda"),
            torch.empty(out_shape, dtype=torch.float32, device="cuda")]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(case, seed)
    if kind == "batch":
        shapes = _shapes(case)
        bufs = [_device_pair(3, 1000 * seed + i, w, h, d, (h, w)) for i, (w, h, d) in enumerate(shapes)]
        torch.cuda.synchronize()        # the call without a stream of its own runs on one of the handle's
        return dict(kind=kind, handle=eb.Elas(eb.params_config(64)), bufs=bufs,
                    ptrs=[[b[k].data_ptr() for b in bufs] for k in range(4)],
                    dims=[(w, h) for w, h, _ in shapes], disp_max=[d for _, _, d in shapes])
    width, height = case["width"], case["height"]
    p = _params(case)
    handle = eb.Elas(p)
    if kind == "host":
        left, right, _, _ = eb.synth_pair(case["scene"], seed, width=width, height=height, disp_max=case["disp_max"],
                                          gt=False)
        return dict(kind=kind, handle=handle, left=left, right=right)
    if kind == "learned":
        handle.set_proposal(eb.load_proposal())
    n = case.get("buffers", 1)
    bufs = [_device_pair(case["scene"], 10 * seed + i, width, height, case["disp_max"], handle.out_shape(width, height))
            for i in range(n)]
    return dict(kind=kind, handle=handle, bufs=bufs, width=width, height=height)


def run(state):
    kind, stream = state["kind"], torch.cuda.current_stream().cuda_stream
    if kind == "train":
        return _run_train(state)
    handle = state["handle"]
    if kind == "host":
        return handle.process(state["left"], state["right"])
    if kind == "batch":
        handle.process_batch_device(*state["ptrs"], state["dims"], state["disp_max"], stream=stream)
    else:
        for left, right, d1, d2 in state["bufs"]:
            handle.process_device(left.data_ptr(), right.data_ptr(), d1.data_ptr(), d2.data_ptr(), state["width"],
                                  state["height"], stream=stream)
    return [m for b in state["bufs"] for m in b[2:]]


def work(case):
    """Bytes: both images read, both maps written (a training step: features and labels read, the parameters and
    their optimiser state read and written).  Operations: of the candidate sweep (four 16-byte descriptors at every
    disparity, for the lattice candidates of one view) and of the network's convolutions."""
    if case["kind"] == "train":
        cells = 2 * case["pairs"] * case["hd"] * case["wd"]
        params = LAYERS * LAYER_PARAMS
        return {"bytes": 4 * CH * cells + 16 * _labels(case) + 4 * 7 * params,
                "flops": 2 * TAPS * CH * CH * cells * (3 * LAYERS - 1)}
    if case["kind"] == "batch":
        shapes = [(w, h, d, 1) for w, h, d in _shapes(case)]
    else:
        shapes = [(case["width"], case["height"], case["disp_max"], case.get("buffers", 1))]
    out = 0.25 if case.get("subsampling") else 1.0
    step = 5
    conv = 2 * TAPS * CH * CH * LAYERS * 2 / 16 if case["kind"] == "learned" else 0
    return {"bytes": sum(n * w * h * (2 + 8 * out) for w, h, _, n in shapes),
            "flops": sum(n * ((w // step) * (h // step) * (d + 1) * 2 * 64 + conv * w * h) for w, h, d, n in shapes)}


# ---- the training step ----

def _labels(case):
    return case["pairs"] * max(1, int(0.07 * case["hd"] * case["wd"]))      # support points: 7 % of the cells


def _shift(b, disp_max):
    w = (disp_max + NBINS) // NBINS
    return (b * w + w // 2) // 4


def _train_inputs(case, seed):
    """Features of the range of pooled descriptors (means in [-2, 2), deviations in [0, 2)), He-initialised
    parameters with Adam's state some steps into a run, and a label per support point, its bin inside the image."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    n, hd, wd = 2 * case["pairs"], case["hd"], case["wd"]
    x = torch.randn((n, hd, wd, CH), generator=g, device="cuda") * 0.25
    x[..., CH // 2:] = x[..., CH // 2:].abs()
    x = x.bfloat16().float()
    theta = []
    for _ in range(LAYERS):
        theta.append(rng.normal(0.0, math.sqrt(2.0 / (TAPS * CH)), TAPS * CH * CH))
        theta.append(rng.normal(0.0, 0.01, CH))
    theta = torch.from_numpy(np.concatenate(theta).astype(np.float32)).cuda()
    m = torch.randn(theta.numel(), generator=g, device="cuda") * 1e-3
    v = torch.rand(theta.numel(), generator=g, device="cuda") * 1e-4 + 1e-5
    nl = _labels(case)
    lab = np.empty((nl, 4), np.int32)
    lab[:, 0] = np.sort(rng.integers(0, case["pairs"], nl))
    lab[:, 1] = rng.integers(0, wd, nl)
    lab[:, 2] = rng.integers(0, hd, nl)
    shifts = np.array([_shift(b, case["disp_max"]) for b in range(NBINS)])
    lab[:, 3] = (rng.random(nl) * (shifts[None, :] <= lab[:, 1:2]).sum(1)).astype(np.int32)
    return x, theta, m, v, torch.from_numpy(lab).cuda()


def _prepare_train(case, seed):
    x, theta, m, v, labels = _train_inputs(case, seed)
    return dict(kind="train", net=proposal.Net(torch, case["hd"], case["wd"], case["pairs"]), x=x, theta=theta, m=m,
                v=v, labels=labels, grad=torch.empty_like(theta), pairs=case["pairs"], disp_max=case["disp_max"],
                step=100)


def _run_train(state):
    """One step as proposal.train() makes it.  The count of best-scoring bins that equal the label is left out: it
    turns on near-tied scores."""
    theta, grad = state["theta"], state["grad"]
    grad.zero_()
    loss, _ = state["net"].forward_backward(theta, grad, state["x"], state["labels"], state["pairs"],
                                            state["disp_max"])
    state["step"] += 1
    eb.pn_adam(theta.data_ptr(), grad.data_ptr(), state["m"].data_ptr(), state["v"].data_ptr(), theta.numel(), 1e-4,
               0.9, 0.999, 1e-8, state["step"])
    return {"loss": loss, "grad": grad, "theta": theta, "m": state["m"], "v": state["v"]}


def _exact_train(case, seed):
    x, theta, m, v, lab = _train_inputs(case, seed)
    F = torch.nn.functional
    p = theta.double().requires_grad_(True)
    a = x.double().permute(0, 3, 1, 2)
    for i in range(LAYERS):
        q = p[i * LAYER_PARAMS:(i + 1) * LAYER_PARAMS]
        w = q[:TAPS * CH * CH].view(3, 3, CH, CH).permute(3, 2, 0, 1)       # [co][ci][dy][dx]
        a = F.conv2d(a, w, q[TAPS * CH * CH:], padding=1)
        if i < LAYERS - 1:
            a = F.relu(a)
    f = a.permute(0, 2, 3, 1)
    lab = lab.long()
    pair, cx, cy, tb = lab[:, 0], lab[:, 1], lab[:, 2], lab[:, 3]
    left = f[2 * pair, cy, cx]
    scores = []
    for b in range(NBINS):
        xr = cx - _shift(b, case["disp_max"])
        s = SCALE * (left * f[2 * pair + 1, cy, xr.clamp(min=0)]).sum(1)
        scores.append(torch.where(xr >= 0, s, torch.full_like(s, -math.inf)))
    loss = F.cross_entropy(torch.stack(scores, 1), tb, reduction="sum")
    g, = torch.autograd.grad(loss / lab.shape[0], p)
    m = 0.9 * m.double() + 0.1 * g
    v = 0.999 * v.double() + 0.001 * g * g
    p = p.detach() - 1e-4 * (m / (1 - 0.9 ** 101)) / ((v / (1 - 0.999 ** 101)).sqrt() + 1e-8)
    return {"loss": float(loss), "grad": g, "theta": p, "m": m, "v": v}


def exact(case, seed):
    """The training step in 64 bits.  The matcher's maps have no closed form outside the library: they are chosen
    disparities, compared value by value with the ones the same inputs gave before."""
    return _exact_train(case, seed) if case["kind"] == "train" else None
