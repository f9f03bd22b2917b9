"""The measured cases: what programs built on ettention_b200 have it do, over the sizes they
have it do it at.

Every case goes through the operator layer that a user's program calls (the single-view
projection operators, the block-iterative reconstruction, the batch, the weighted back
projection, the learned warm start).  Test objects are sums of ellipsoids whose line
integrals are known in closed form, seen with Poisson noise and put through -log, as the
tilt series of a microscope are.  `exact` restates each computation in 64 bits with plain
torch: intersection lengths of the rays with the voxel grid, bilinear sampling with weights
in steps of 1/256, the relaxed update, the network and its gradient.
"""
import math
import os

import numpy as np
import torch

from ettention_b200 import _abi
from ettention_b200.learned import DEFAULT_WEIGHTS, WarmStartNet, load_weights
from ettention_b200.operators import (AlgebraicParameterSet, BackProjectionOperator, BatchReconstructionOperator,
                                      BlockIterativeReconstructionOperator, Context, ForwardProjectionOperator,
                                      GPUMappedVolume, ScannerGeometry, WBPOperator)

VOXELS = {"float32": _abi.VOXEL_FLOAT32, "f16_master": _abi.VOXEL_F16_MASTER, "bf16_master": _abi.VOXEL_BF16_MASTER}
ORDERS = {"identity": _abi.ORDER_IDENTITY, "maxangle": _abi.ORDER_MAXANGLE, "random": _abi.ORDER_RANDOM}
EPS = 1e-4   # ray lengths below it are skipped (EPSILON of the reference's Math.hl)
LEARNING_RATE = 1e-3


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # One view of a small volume through the forward operator: an interactive preview or a
        # residual check, where the launch and the call itself count.
        {"name": "forward_view_96", "kind": "forward", "x": 96, "y": 96, "z": 96, "tilt": 33.0},
        # One view back projected into a cropped volume of sizes that are no multiple of a vector.
        {"name": "back_view_ragged", "kind": "back", "x": 501, "y": 363, "z": 179, "tilt": -27.5, "samples": 1},
        # Plain SART on a small volume, the whole five-iteration run of a quick reconstruction.
        {"name": "sart_128", "kind": "recon", "x": 128, "y": 128, "z": 64, "views": 61, "tilt": 60.0, "block": 1,
         "iterations": 5, "lam": 0.3, "voxel": "float32", "order": "identity"},
        # SART at the size of a binned tomogram: one sweep over the views.
        {"name": "sart_1024", "kind": "recon", "x": 1024, "y": 1024, "z": 256, "views": 61, "tilt": 60.0, "block": 1,
         "iterations": 1, "lam": 0.3, "voxel": "float32", "order": "identity"},
        # SIRT of the same tomogram: every view in one block.
        {"name": "sirt_1024", "kind": "recon", "x": 1024, "y": 1024, "z": 256, "views": 61, "tilt": 60.0, "block": 0,
         "iterations": 1, "lam": 0.3, "voxel": "float32", "order": "identity"},
        # A careful reconstruction of a cropped region: blocks of ten, several samples per pixel
        # and voxel, long-object compensation, the volume in four slabs, alternating angles.
        {"name": "block10_oversampled", "kind": "recon", "x": 250, "y": 231, "z": 90, "views": 61, "tilt": 60.0,
         "block": 10, "iterations": 2, "lam": 0.3, "voxel": "float32", "order": "maxangle", "fp_samples": 2,
         "bp_samples": 4, "loc": True, "slabs": 4},
        # A cone-beam scan of a large sample: blocks of eight, the projector reading a BF16 copy.
        {"name": "perspective_2048", "kind": "recon", "x": 2048, "y": 2048, "z": 512, "views": 31, "tilt": 60.0,
         "block": 8, "iterations": 1, "lam": 0.2, "voxel": "bf16_master", "order": "random", "perspective": True},
        # Cone-beam SART of a small volume in FP32.
        {"name": "perspective_sart_256", "kind": "recon", "x": 256, "y": 256, "z": 128, "views": 61, "tilt": 60.0,
         "block": 1, "iterations": 1, "lam": 0.2, "voxel": "float32", "order": "identity", "perspective": True},
        # Many small tilt series of uneven sizes (sub-tomograms of one session) in one batch.
        {"name": "batch_16", "kind": "batch", "series": 16, "mix": 4000, "iterations": 1, "lam": 0.3,
         "voxel": "f16_master"},
        # Weighted back projection, the first look at a tilt series, from host projections.
        {"name": "wbp_512", "kind": "wbp", "x": 512, "y": 512, "z": 128, "views": 61, "tilt": 60.0},
        # The learned warm start at the size its weights were trained for: one inference ...
        {"name": "warmstart_infer_256", "kind": "infer", "x": 256, "y": 256, "z": 128},
        # ... and one training step on one pair, the updated weights read back.
        {"name": "warmstart_train_256", "kind": "train", "x": 256, "y": 256, "z": 128},
    ]


def _size(rng, lo, hi, step=1):
    """lo .. hi, even over the logarithm, a multiple of step."""
    return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    kind = rng.choice(["forward", "back", "recon", "recon", "recon", "perspective", "batch", "wbp", "infer", "train"])
    if kind in ("forward", "back"):
        c = {"kind": kind, "x": _size(rng, 64, 1024), "y": _size(rng, 64, 1024), "z": _size(rng, 32, 256),
             "tilt": round(rng.uniform(-70.0, 70.0), 2)}
        if kind == "back":
            c["samples"] = rng.choice([1, 1, 4])
        return c
    if kind == "recon":
        step = rng.choice([1, 2, 16, 16])
        block = rng.choice([1, 1, 0, rng.randrange(2, 13)])
        c = {"kind": kind, "x": _size(rng, 64, 640, step), "y": _size(rng, 64, 640, step),
             "z": _size(rng, 32, 192, step), "views": rng.randrange(20, 41) * 2 + 1,
             "tilt": round(rng.uniform(50.0, 70.0), 1), "block": block, "iterations": rng.choice([1, 2]), "lam": 0.3,
             "voxel": rng.choice(["float32", "float32", "f16_master", "bf16_master"]),
             "order": rng.choice(["identity", "maxangle"])}
        if rng.random() < 0.25:
            c["loc"] = True
        if rng.random() < 0.25:
            c["slabs"] = rng.randrange(2, 5)
        if rng.random() < 0.25:
            c["fp_samples"], c["bp_samples"], c["iterations"] = 2, 4, 1
        return c
    if kind == "perspective":
        step = rng.choice([1, 2, 16])
        return {"kind": "recon", "x": _size(rng, 64, 512, step), "y": _size(rng, 64, 512, step),
                "z": _size(rng, 32, 160, step), "views": rng.randrange(10, 31) * 2 + 1,
                "tilt": round(rng.uniform(40.0, 60.0), 1), "block": rng.choice([1, 8, rng.randrange(2, 13), 0]),
                "iterations": 1, "lam": 0.2, "voxel": rng.choice(["float32", "f16_master", "bf16_master"]),
                "order": rng.choice(["identity", "maxangle"]), "perspective": True}
    if kind == "batch":
        return {"kind": "batch", "series": rng.randrange(2, 25), "mix": rng.randrange(1, 10 ** 6), "iterations": 1,
                "lam": 0.3, "voxel": rng.choice(["float32", "f16_master", "bf16_master"])}
    if kind == "wbp":
        return {"kind": "wbp", "x": _size(rng, 64, 512), "y": _size(rng, 64, 512), "z": _size(rng, 32, 128),
                "views": rng.randrange(20, 41) * 2 + 1, "tilt": round(rng.uniform(50.0, 70.0), 1)}
    return {"kind": kind, "x": _size(rng, 32, 320, 4), "y": _size(rng, 32, 256, 4), "z": _size(rng, 16, 128, 4)}


# ------------------------------------------------------------------ geometry
def _views(case):
    """The tilt angles of a series, evenly spaced."""
    if "views" not in case:
        return [case["tilt"]]
    return [float(a) for a in np.linspace(-case["tilt"], case["tilt"], case["views"])]


def _geometry(case, angle):
    """(source, detector, horizontal pitch, vertical pitch) as float32 values: a detector of the
    volume's x and y turned by -angle about y.  Parallel: unit pitch, the source plane at the
    corner of the volume's footprint.  Perspective: the source ten volume widths in front of the
    volume's centre, the detector one width behind it with a pitch that spans the volume."""
    W, H = case["x"], case["y"]
    if case.get("perspective"):
        D, p = 10.0 * W, 1.1
        base = ([0.0, 0.0, D], [-0.5 * W * p, -0.5 * H * p, -float(W)], [p, 0.0, 0.0], [0.0, p, 0.0])
    else:
        base = ([-0.5 * W, -0.5 * H, float(W)], [-0.5 * W, -0.5 * H, -float(W)], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0])
    t = -math.radians(angle)
    c, s = math.cos(t), math.sin(t)
    return [np.array([v[0] * c - v[2] * s, v[1], v[0] * s + v[2] * c], np.float32) for v in base]


def _scanner(case, angle):
    return ScannerGeometry(*[[float(v) for v in p] for p in _geometry(case, angle)], case["x"], case["y"],
                           bool(case.get("perspective")))


# ------------------------------------------------------------------ test objects and their tilt series
def _ellipsoids(case, seed, count=24):
    """(M, centre, density): |sqrt(M) (p - c)| <= 1 inside; the densities keep the line integrals
    of a large volume between about 0 and 4."""
    rng = np.random.Generator(np.random.PCG64(seed))
    size = np.array([case["x"], case["y"], case["z"]], np.float64)
    M, centre, density = [], [], []
    # a cone-beam sample lies inside the volume, a tomogram is cut out of a larger specimen
    size_max, spread = (0.2 * size.min(), 0.25) if case.get("perspective") else (0.25 * size[:2].min(), 0.4)
    for _ in range(count):
        R, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        a = rng.uniform(0.12, 1.0, 3) * size_max
        M.append(R.T @ np.diag(1.0 / a ** 2) @ R)
        centre.append(rng.uniform(-spread, spread, 3) * size)
        density.append(rng.uniform(0.05, 1.0) * 2.0 / size[0])
    return (torch.tensor(np.array(v), dtype=torch.float32, device="cuda") for v in (M, centre, density))


def _phantom(case, seed):
    """The object on the voxel grid, (z, y, x) float32."""
    M, centre, density = _ellipsoids(case, seed)
    X, Y, Z = case["x"], case["y"], case["z"]
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) + (0.5 - 0.5 * n) for n in (X, Y, Z)]
    vol = torch.zeros((Z, Y, X), device="cuda")
    for m, c, d in zip(M, centre, density):
        dx, dy, dz = ax[0] - c[0], ax[1] - c[1], ax[2] - c[2]
        xy = m[0, 0] * dx[None, :] ** 2 + m[1, 1] * dy[:, None] ** 2 + 2 * m[0, 1] * dy[:, None] * dx[None, :]
        lin = 2 * (m[0, 2] * dx[None, :] + m[1, 2] * dy[:, None])
        for z0 in range(0, Z, 32):
            z = dz[z0:z0 + 32, None, None]
            vol[z0:z0 + 32] += d * (xy + z * lin + m[2, 2] * z * z <= 1.0)
    return vol


def _projections(case, seed, counts=100.0):
    """The noisy tilt series, (views, y, x) float32: closed-form line integrals of the object,
    Poisson counts, -log.  Cone-beam series come as a scanner writes them, at a higher dose and
    with the air around the object set to zero (noise there would be divided by the ray lengths
    of rays that only graze the volume, and one sweep would amplify the last bit of those
    lengths to a tenth of the result)."""
    if case.get("perspective"):
        counts = 2e4
    M, centre, density = _ellipsoids(case, seed)
    angles = _views(case)
    W, H = case["x"], case["y"]
    out = torch.empty((len(angles), H, W), device="cuda")
    gx = torch.arange(W, device="cuda", dtype=torch.float32) + 0.5
    gy = torch.arange(H, device="cuda", dtype=torch.float32) + 0.5
    for i, a in enumerate(angles):
        src, det, hp, vp = (torch.tensor(v, device="cuda") for v in _geometry(case, a))
        if case.get("perspective"):
            d = (det - src)[None, None] + gx[None, :, None] * hp + gy[:, None, None] * vp
            d = d / d.norm(dim=-1, keepdim=True)
            o = src.expand(1, 1, 3)
        else:
            d = ((det - src) / (det - src).norm()).expand(1, 1, 3)
            o = src[None, None] + gx[None, :, None] * hp + gy[:, None, None] * vp
        acc = torch.zeros((H, W), device="cuda")
        for m, c, rho in zip(M, centre, density):
            dm = d @ m
            od = o - c
            # the chord depends on the offset of the ray from the centre only: taking it at the
            # closest point keeps float32 accurate for a far source
            od = od - (od * d).sum(-1, keepdim=True) * d
            A, B, C = (dm * d).sum(-1), (dm * od).sum(-1), ((od @ m) * od).sum(-1) - 1.0
            acc += rho * 2.0 * (B * B - A * C).clamp_min_(0.0).sqrt_() / A
        out[i] = acc
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    for i in range(out.shape[0]):
        n = torch.poisson(counts * torch.exp(-out[i]), generator=gen)
        out[i] = -torch.log(n.clamp_min(1.0) / counts)
    if case.get("perspective"):
        out[out < 0.03] = 0.0
    return out


class _DeviceArray:
    """A volume's device memory as an array other libraries can wrap without a copy."""

    def __init__(self, volume):
        X, Y, Z = volume.resolution
        self.volume = volume
        self.__cuda_array_interface__ = {"shape": (Z, Y, X), "typestr": "<f4", "data": (volume.device_ptr(), False),
                                         "version": 3}


def _volume(ctx, case, voxel="float32"):
    v = GPUMappedVolume(ctx, (case["x"], case["y"], case["z"]), voxel_type=VOXELS[voxel],
                        subvolume_count=case.get("slabs", 1))
    return v, torch.as_tensor(_DeviceArray(v), device="cuda")


def _parameters(case):
    block = case.get("block", 1)
    return AlgebraicParameterSet(
        algorithm={1: "sart", 0: "sirt"}.get(block, "blockIterative"), block_size=block or _abi.BLOCK_ALL,
        iterations=case["iterations"], lam=case["lam"], use_long_object_compensation=case.get("loc", False),
        fp_samples=case.get("fp_samples", 1), bp_samples=case.get("bp_samples", 1), voxel_type=VOXELS[case["voxel"]],
        order=ORDERS[case.get("order", "identity")])


def _batch_members(case):
    """The members of a batch: 96^3 to 256 x 256 x 128 voxels, 41 to 81 views over +-50 to +-70."""
    rng = np.random.Generator(np.random.PCG64(case["mix"]))
    return [{"x": int(rng.integers(6, 17)) * 16, "y": int(rng.integers(6, 17)) * 16, "z": int(rng.integers(6, 9)) * 16,
             "views": int(rng.integers(20, 41)) * 2 + 1, "tilt": float(rng.uniform(50.0, 70.0)), "block": 1,
             "iterations": case["iterations"], "lam": case["lam"], "voxel": case["voxel"], "order": "identity"}
            for _ in range(case["series"])]


def _pair(case, seed):
    """(input, target) of the warm start: a blurred, noisy and a nearly converged state."""
    v = _phantom(case, seed)[None, None]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    pool = torch.nn.functional.avg_pool3d
    rms = float(v.square().mean().sqrt()) + 1e-12
    a = pool(v, 5, 1, 2) + 0.2 * rms * torch.randn(v.shape, device="cuda", generator=gen)
    b = pool(v, 3, 1, 1) + 0.05 * rms * torch.randn(v.shape, device="cuda", generator=gen)
    k = load_weights()[1] / rms   # the network expects the magnitude it was trained on
    return (k * a[0]).contiguous(), (k * b[0]).contiguous()


# ------------------------------------------------------------------ what a program has in hand, and one pass
def prepare(case, seed):
    ctx = Context(0)
    s = {"case": case, "ctx": ctx}
    kind = case["kind"]
    if kind in ("infer", "train"):
        params, scale, _ = load_weights()
        s["in"], s["target"] = _pair(case, seed)
        s["out"] = torch.empty_like(s["in"])
        s["net"] = WarmStartNet(ctx, (case["x"], case["y"], case["z"]), 1, params, scale)
    elif kind == "forward":
        s["volume"], s["view"] = _volume(ctx, case)
        s["volume"].upload_device(_phantom(case, seed))
        s["op"] = ForwardProjectionOperator(s["volume"], 1)
        s["op"].setScannerGeometry(_scanner(case, case["tilt"]))
        s["p"] = torch.zeros((case["y"], case["x"]), device="cuda")
        s["l"] = torch.zeros_like(s["p"])
        s["op"].SetOutput(s["p"], s["l"])
    elif kind == "back":
        s["volume"], s["view"] = _volume(ctx, case)
        s["volume"].upload_device(_phantom(case, seed))
        s["r"], s["l"] = _residual(case, seed)
        s["op"] = BackProjectionOperator(s["volume"], 0.3, case["samples"])
        s["op"].setScannerGeometry(_scanner(case, case["tilt"]))
        s["op"].setInput(s["r"], s["l"], 1)
    elif kind == "batch":
        s["init"], series, s["views"] = [], [], []
        for j, m in enumerate(_batch_members(case)):
            v, view = _volume(ctx, m, m["voxel"])
            s["views"].append(view)
            s["init"].append((v, torch.zeros_like(view)))
            series.append((v, [_scanner(m, a) for a in _views(m)], _projections(m, seed + 7919 * j).cpu().numpy()))
        s["op"] = BatchReconstructionOperator(series, _parameters(case))
    else:
        s["volume"], s["view"] = _volume(ctx, case, case.get("voxel", "float32"))
        s["init"] = torch.zeros_like(s["view"])
        geometries = [_scanner(case, a) for a in _views(case)]
        s["b"] = _projections(case, seed)
        if kind == "wbp":
            s["op"] = WBPOperator(s["volume"], geometries, s["b"].cpu().numpy(),
                                  AlgebraicParameterSet(algorithm="wbp", lam=1.0))
        else:
            s["op"] = BlockIterativeReconstructionOperator(s["volume"], geometries, s["b"], _parameters(case))
    ctx.synchronize()
    return s


def _residual(case, seed):
    """A residual image and the ray lengths of one view, as a comparison leaves them."""
    r = _projections(case, seed)[0]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 1)
    r = 0.1 * r + 0.05 * torch.randn(r.shape, device="cuda", generator=gen)
    cos = max(abs(math.cos(math.radians(case["tilt"]))), 1e-3)
    u = (torch.arange(case["x"], device="cuda", dtype=torch.float32) + (0.5 - 0.5 * case["x"])).abs()
    sin = abs(math.sin(math.radians(case["tilt"])))
    full = min(case["z"] / cos, case["x"] / max(sin, 1e-3))
    edge = (0.5 * (case["x"] * cos + case["z"] * sin) - u) / max(sin * cos, 1e-3)
    l = edge.clamp(0.0, full).expand(case["y"], case["x"]).contiguous()
    return r.contiguous(), l


def run(s):
    kind = s["case"]["kind"]
    if kind == "infer":
        s["net"].infer(s["in"], s["out"], 1)
        return s["out"]
    if kind == "train":
        loss = s["net"].train_step(s["in"], s["target"], 1, LEARNING_RATE)
        return {"loss": loss, "params": s["net"].get_params()}
    if kind == "forward":
        s["p"].zero_()
        s["l"].zero_()
        s["op"].Execute(0)
        return {"projection": s["p"], "length": s["l"]}
    if kind == "back":
        s["op"].execute()
        return s["view"]
    if kind == "batch":
        for v, z in s["init"]:
            v.upload_device(z)
        s["op"].run()
        return {"volumes": s["views"], "residual_sq": np.array(s["op"].last_residual_sq())}
    s["volume"].upload_device(s["init"])
    s["op"].run()
    if kind == "wbp":
        return s["view"]
    return {"volume": s["view"], "residual_sq": s["op"].last_residual_sq()}


# ------------------------------------------------------------------ work and tolerances
def _conv_flops(case):
    level = [case["x"] * case["y"] * case["z"] // 8 ** k for k in range(3)]
    return sum(2.0 * 27 * cin * co * level[l] for cin, co, l in _LAYERS)


def _series_work(c):
    """Bytes: the series and the start in, the volume out.  Operations: two per ray and voxel
    crossed, about fourteen per voxel and view (two coordinates, the blend of residual and
    length, the update)."""
    V, P, n = c["x"] * c["y"] * c["z"], c["x"] * c["y"], len(_views(c))
    it = c.get("iterations", 1)
    crossed = np.mean([min(c["z"] / max(abs(math.cos(math.radians(a))), 1e-3),
                           c["x"] / max(abs(math.sin(math.radians(a))), 1e-3)) for a in _views(c)]) * 1.3
    fs, bs = c.get("fp_samples", 1) ** 2, c.get("bp_samples", c.get("samples", 1))
    fp, bp = 2.0 * n * P * crossed * fs, 14.0 * n * V * bs
    if c["kind"] == "forward":
        return {"bytes": 4.0 * V + 8.0 * P, "flops": fp}
    if c["kind"] == "back":
        return {"bytes": 8.0 * V + 8.0 * P, "flops": bp}
    if c["kind"] == "wbp":
        return {"bytes": 4.0 * n * P + 8.0 * V, "flops": bp + 130.0 * n * P}
    return {"bytes": 4.0 * n * P + 8.0 * V, "flops": it * (fp + bp)}


def work(case):
    kind = case["kind"]
    if kind in ("infer", "train"):
        V = case["x"] * case["y"] * case["z"]
        n = sum(27 * cin * co + co for cin, co, _ in _LAYERS)
        if kind == "infer":
            return {"bytes": 8.0 * V + 2.0 * n, "flops": _conv_flops(case)}
        # the gradient with respect to weights and, but for the first layer, to inputs
        return {"bytes": 8.0 * V + 24.0 * n, "flops": 3.0 * _conv_flops(case) - 2.0 * 27 * 16 * V}
    if kind == "batch":
        w = [_series_work(dict(m, kind="recon")) for m in _batch_members(case)]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    return _series_work(case)


def tolerance(case):
    """About four times what was seen between two kernels of the same call (unfused against fused,
    per-tap against z-streamed convolutions), between this and `exact`, or after moving the
    geometry by its last bits, whichever another correct implementation would show.  A last-bit
    change of a coordinate moves some sampling weights by their step of 1/256, and SART divides
    by the lengths of rays that only graze the volume: that, and not the sums, is the scale of
    the reconstructions' figures."""
    kind = case["kind"]
    if kind == "forward":
        return {"rel": 3e-6, "max": 6e-5}
    if kind == "back":
        return {"rel": 6e-5, "max": 0.02}
    if kind == "wbp":
        return {"rel": 1.5e-3, "max": 0.25}
    if kind == "infer":   # bf16 activations: 2e-3 between the two convolution kernels
        return {"rel": 1e-2, "max": 0.12}
    if kind == "train":   # the first step moves each weight by the rate, towards its gradient's sign
        return {"rel": 3.5e-3, "max": 0.08}
    if kind == "recon" and case["block"] != 1 and not case.get("perspective"):
        return {"rel": 2.5e-4, "max": 0.03}
    return {"rel": 1e-3, "max": 0.1}


# ------------------------------------------------------------------ the same in 64 bits
def _f64(v):
    return torch.as_tensor(np.asarray(v, np.float64), device="cuda")


def _walk(o, d, case):
    """Rays o + t d (K, 3) through the volume: voxel indices (x, y, z) and lengths, (K, n) each.
    As in the reference's walk, a ray's voxel is found from the volume's corner where it enters,
    and from there changes at whole world coordinates (DDARaytracer.hl): along an axis of odd
    size the grid that a ray sees lies half a voxel off the volume's."""
    res = [case["x"], case["y"], case["z"]]
    enter = []
    for i in range(3):
        di = d[:, i:i + 1]
        t = [torch.where(di == 0, torch.full_like(di, math.nan), (f * res[i] - o[:, i:i + 1]) / di) for f in (-0.5, 0.5)]
        enter.append([torch.minimum(*t).nan_to_num(-1e200), torch.maximum(*t).nan_to_num(1e200)])
    lo = torch.maximum(torch.maximum(enter[0][0], enter[1][0]), enter[2][0])
    hit = lo < torch.minimum(torch.minimum(enter[0][1], enter[1][1]), enter[2][1])
    ts, shift, hi = [lo], [], torch.full_like(lo, 1e200)
    for i in range(3):
        di, half = d[:, i:i + 1], 0.5 * res[i]
        e = (o[:, i:i + 1] + lo * di).clamp(-half, half)
        e = torch.where(enter[i][0] == lo, -half * torch.sign(di), e)
        k = torch.floor(e + half).clamp(0, res[i] - 1) - torch.where(di < 0, torch.ceil(e) - 1.0, torch.floor(e))
        shift.append(k)
        if bool((di == 0).all()):
            continue
        planes = torch.arange(res[i] + 1, device="cuda", dtype=torch.float64)
        t = ((planes[None] - k - o[:, i:i + 1]) / torch.where(di == 0, torch.full_like(di, 1e-300), di)).clamp(-1e200, 1e200)
        hi = torch.where(di == 0, hi, torch.minimum(hi, torch.maximum(t[:, :1], t[:, -1:])))
        ts.append(t)
    t = torch.cat(ts, 1)
    t = torch.minimum(torch.maximum(t, lo), torch.maximum(lo, hi)).sort(1).values
    length = (t[:, 1:] - t[:, :-1]) * hit
    mid = 0.5 * (t[:, 1:] + t[:, :-1])
    del t, ts
    idx = [torch.floor(o[:, i:i + 1] + mid * d[:, i:i + 1] + shift[i]).clamp_(0, res[i] - 1).long() for i in range(3)]
    return idx, length


def _project(vol, case, angle):
    """(line integrals, lengths) of one view, (y, x) float64; vol (z, y, x)."""
    W, H = case["x"], case["y"]
    src, det, hp, vp = (_f64(v) for v in _geometry(case, angle))
    n = case.get("fp_samples", 1)
    P, L = torch.zeros((H, W), device="cuda", dtype=torch.float64), torch.zeros((H, W), device="cuda", dtype=torch.float64)
    gx = torch.arange(W, device="cuda", dtype=torch.float64)
    gy = torch.arange(H, device="cuda", dtype=torch.float64)
    for k in range(n * n):
        fx, fy = (k % n + 0.5) / n, (k // n + 0.5) / n
        if not case.get("perspective"):
            # tilted about y: the rays of a detector column cross the same (z, x) cells, each in
            # the volume row its detector row lies in
            d = (det - src) / (det - src).norm()
            o = src + (gx + fx)[:, None] * hp
            (ix, _, iz), length = _walk(torch.stack([o[:, 0], 0 * o[:, 1], o[:, 2]], 1), d.expand(W, 3), case)
            rows = torch.floor(src[1] + (gy + fy) * vp[1] + 0.5 * case["y"]).long()
            ok = (rows >= 0) & (rows < case["y"])
            at = torch.stack([torch.arange(W, device="cuda")[:, None].expand_as(ix), iz * case["x"] + ix]).reshape(2, -1)
            cells = torch.sparse_coo_tensor(at, length.reshape(-1), (W, case["z"] * case["x"]), check_invariants=False)
            keep = ok.double()[:, None]
            rows = rows.clamp(0, case["y"] - 1)
            v = torch.sparse.mm(cells, vol.permute(0, 2, 1).reshape(-1, case["y"]))
            P += v.T[rows] * keep
            L += length.sum(1)[None] * keep
        else:
            for y0 in range(0, H, 64):
                p = det + (gx + fx)[None, :, None] * hp + (gy[y0:y0 + 64] + fy)[:, None, None] * vp
                d = (p - src).reshape(-1, 3)
                d = d / d.norm(dim=1, keepdim=True)
                (ix, iy, iz), length = _walk(src.expand_as(d), d, case)
                v = vol.reshape(-1)[(iz * case["y"] + iy) * case["x"] + ix]
                P[y0:y0 + 64] += (v * length).sum(1).reshape(-1, W)
                L[y0:y0 + 64] += length.sum(1).reshape(-1, W)
    return P / (n * n), L / (n * n)


def _taps(c, n):
    """Texel index and weight of the second tap, in steps of 1/256 (half up)."""
    q = torch.floor(256.0 * c - 127.5).clamp(-1000.0, 256.0 * n + 1000.0).long()
    return q >> 8, (q & 255).double() / 256.0


def _padded(img):
    return torch.nn.functional.pad(img, (8, 8, 8, 8))


def _pattern(case, angle):
    """Offsets (x, y, z) and chords of the per-voxel samples of a parallel view (unit voxels)."""
    src, det, hp, vp = (np.asarray(v, np.float64) for v in _geometry(case, angle))
    ray = (det - src) / np.linalg.norm(det - src)
    h, v = hp / np.linalg.norm(hp), vp / np.linalg.norm(vp)
    n = int(round(math.sqrt(case.get("bp_samples", case.get("samples", 1)))))
    out = []
    for k in range(n * n):
        p = ((k % n + 0.5) / n - 0.5) * h + ((k // n + 0.5) / n - 0.5) * v
        with np.errstate(divide="ignore", invalid="ignore"):
            a, b = (-0.5 - p) / ray, (0.5 - p) / ray
        use = ray != 0
        out.append((p, np.maximum(a, b)[use].min() - np.minimum(a, b)[use].max()))
    return out


def _back(vol, case, angle, r, L, lam):
    """vol += the relaxed, length-normalised back projection of r, in place."""
    X, Y, Z = case["x"], case["y"], case["z"]
    src, det, hp, vp = (np.asarray(v, np.float64) for v in _geometry(case, angle))
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) + (0.5 - 0.5 * n) for n in (X, Y, Z)]
    rp, lp = _padded(r), _padded(L)
    if not case.get("perspective"):
        ray = (det - src) / np.linalg.norm(det - src)
        m = np.linalg.inv(np.stack([hp, vp, ray], 1)).astype(np.float32).astype(np.float64)
        pattern = _pattern(case, angle)
        step = max(1, int(6e7 // (Z * X)))
        for y0 in range(0, Y, step):
            y = ax[1][y0:y0 + step]
            total = torch.zeros((Z, y.numel(), X), device="cuda", dtype=torch.float64)
            used = torch.zeros_like(total)
            for p, chord in pattern:
                u = m[0, 0] * (ax[0] + p[0])[None, :] + m[0, 2] * (ax[2] + p[2])[:, None] + 0.5 * X + 0.5
                v = m[1, 1] * (y + p[1]) + 0.5 * Y + 0.5
                (iu, a), (iv, b) = _taps(u, X), _taps(v, Y)
                iu, iv = (iu + 8).clamp(0, X + 14), (iv + 8).clamp(0, Y + 14)
                val = []
                for img in (rp, lp):
                    rows = (1 - b)[:, None] * img[iv] + b[:, None] * img[iv + 1]
                    val.append(((1 - a) * rows[:, iu] + a * rows[:, iu + 1]).permute(1, 0, 2))
                ok = val[1] > EPS
                total += torch.where(ok, val[0] * lam * chord / torch.where(ok, val[1], 1.0), 0.0)
                used += ok
            vol[:, y0:y0 + step] += total / used.clamp_min(1.0)
        return
    # world to detector pixels (times the depth), as the view's 4 x 4 float matrix holds it
    centre = det + 0.5 * (X * hp + Y * vp)
    m = np.linalg.inv(np.stack([hp, vp, centre - src], 1))
    m = np.stack([m[0] + 0.5 * X * m[2], m[1] + 0.5 * Y * m[2], m[2]])
    m = np.concatenate([m, -(m @ src)[:, None]], 1).astype(np.float32).astype(np.float64)
    step = max(1, int(2e7 // (X * Y)))
    for z0 in range(0, Z, step):
        z = ax[2][z0:z0 + step]
        d = [ax[0][None, None] - src[0], ax[1][None, :, None] - src[1], z[:, None, None] - src[2]]
        a, b, c = (m[i, 0] * ax[0][None, None] + m[i, 1] * ax[1][None, :, None] + m[i, 2] * z[:, None, None] + m[i, 3]
                   for i in range(3))
        (iu, fu), (iv, fv) = _taps(a / c, X), _taps(b / c, Y)
        iu, iv = (iu + 8).clamp(0, X + 14), (iv + 8).clamp(0, Y + 14)
        val = []
        for img in (rp, lp):
            f, w, at = img.reshape(-1), img.shape[1], iv * img.shape[1] + iu
            val.append((1 - fv) * ((1 - fu) * f[at] + fu * f[at + 1]) + fv * ((1 - fu) * f[at + w] + fu * f[at + w + 1]))
        size = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt()
        big = torch.maximum(torch.maximum(d[0].abs(), d[1].abs()), d[2].abs())
        ok = val[1] >= EPS
        vol[z0:z0 + z.numel()] += torch.where(ok, lam * val[0] * (size / big) / torch.where(ok, val[1], 1.0), 0.0)


def _order(case, n):
    if case.get("order", "identity") == "identity":
        return list(range(n))
    j, k, out = n // 2, 0, []
    for i in range(n):
        out.append(j if i % 2 == 0 else k)
        j, k = j + (i % 2 == 0), k + (i % 2 == 1)
    return out


def _reconstruct(case, b):
    angles = _views(case)
    vol = torch.zeros((case["z"], case["y"], case["x"]), device="cuda", dtype=torch.float64)
    order = _order(case, len(angles))
    size = case["block"] or len(order)
    stored = {"float32": None, "f16_master": torch.float16, "bf16_master": torch.bfloat16}[case["voxel"]]
    for _ in range(case["iterations"]):
        total = 0.0
        for k in range(0, len(order), size):
            block = order[k:k + size]
            seen = vol if stored is None else vol.float().to(stored).double()
            images = []
            for i in block:
                p, l = _project(seen, case, angles[i])
                if case.get("loc"):
                    src, det, _, _ = (np.asarray(v, np.float64) for v in _geometry(case, angles[i]))
                    c = case["z"] / abs((det - src)[2] / np.linalg.norm(det - src))
                    p, l = torch.where(l > EPS, p * c / l.clamp_min(EPS), 0.0), torch.full_like(l, c)
                images.append((b[i].double() - p, l))
                total += float(images[-1][0].square().sum())
            for i, (r, l) in zip(block, images):
                _back(vol, case, angles[i], r, l, case["lam"] / len(block))
    return {"volume": vol, "residual_sq": total}


def _ramlak(b):
    """The 128-tap RamLak filtering of every row on the power-of-two grid the reference's
    Fourier-space convolution works on: mirrored padding, the kernel's row one off the centre."""
    H, W = b.shape[-2:]
    taps = torch.arange(128, device="cuda", dtype=torch.float64) - 64
    ker = torch.where(taps % 2 != 0, -1.0 / ((taps ** 2) * math.pi ** 2).clamp_min(1e-9), 0.0)
    ker[64] = 0.25
    Wu, Hu = 1 << (max(W, 128) - 1).bit_length(), 1 << (max(H, 1) - 1).bit_length()

    def mirror(n, nu):
        i = np.arange(nu)
        lo, hi = (nu - n) // 2, (nu + n) // 2
        return torch.as_tensor(np.where((i >= lo) & (i < hi), i - lo, np.where(i < hi, lo - i, n + hi - 1 - i)), device="cuda")

    padded = torch.zeros((Hu, Wu), device="cuda", dtype=torch.float64)
    padded[(Hu - 1) // 2, (Wu - 128) // 2:(Wu - 128) // 2 + 128] = ker
    padded = padded.roll((-(Hu // 2), -(Wu // 2)), (0, 1))
    out = torch.empty_like(b, dtype=torch.float64)
    x0, y0 = Wu // 2 - W // 2, Hu // 2 - H // 2
    spectrum = torch.fft.fft2(padded)
    for i in range(b.shape[0]):
        src = b[i].double()[mirror(H, Hu)][:, mirror(W, Wu)]
        out[i] = torch.fft.ifft2(torch.fft.fft2(src) * spectrum).real[y0:y0 + H, x0:x0 + W]
    return out


# layers of the network: input channels, output channels, level
_LAYERS = [(1, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (96, 32, 1), (32, 32, 1),
           (48, 16, 0), (16, 16, 0), (16, 1, 0)]


def _shifted(p, t, shape):
    z, y, x = shape
    return p[:, t // 9:t // 9 + z, (t // 3) % 3:(t // 3) % 3 + y, t % 3:t % 3 + x].reshape(p.shape[0], -1)


class _Conv(torch.autograd.Function):
    """3 x 3 x 3 convolution of (channels, z, y, x) as 27 matrix products."""

    @staticmethod
    def forward(ctx, x, w, b):
        ctx.save_for_backward(x, w)
        p = torch.nn.functional.pad(x, (1,) * 6)
        out = b[:, None].expand(-1, x[0].numel()).clone()
        for t in range(27):
            out.addmm_(w[t], _shifted(p, t, x.shape[1:]))
        return out.reshape((-1,) + x.shape[1:])

    @staticmethod
    def backward(ctx, g):
        x, w = ctx.saved_tensors
        p, q = torch.nn.functional.pad(x, (1,) * 6), torch.nn.functional.pad(g, (1,) * 6)
        flat = g.reshape(g.shape[0], -1)
        gx, gw = torch.zeros((x.shape[0], x[0].numel()), device="cuda", dtype=x.dtype), torch.empty_like(w)
        for t in range(27):
            gx.addmm_(w[t].T, _shifted(q, 26 - t, x.shape[1:]))
            gw[t] = flat @ _shifted(p, t, x.shape[1:]).T
        return gx.reshape(x.shape), gw, flat.sum(1)


def _network(params, v, scale):
    parts, at = [], 0
    for cin, co, _ in _LAYERS:
        parts.append((params[at:at + 27 * co * cin].reshape(27, co, cin), params[at + 27 * co * cin:at + 27 * co * cin + co]))
        at += 27 * co * cin + co
    layer = lambda k, x: _Conv.apply(x, *parts[k])  # noqa: E731
    relu = torch.relu
    pool = lambda x: torch.nn.functional.avg_pool3d(x, 2)  # noqa: E731
    up = lambda x: x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)  # noqa: E731
    e1 = relu(layer(1, relu(layer(0, v[None] / scale))))
    e2 = relu(layer(3, relu(layer(2, pool(e1)))))
    e3 = relu(layer(5, relu(layer(4, pool(e2)))))
    d2 = relu(layer(7, relu(layer(6, torch.cat([up(e3), e2])))))
    d1 = relu(layer(9, relu(layer(8, torch.cat([up(d2), e1])))))
    return v + scale * layer(10, d1)[0]


def exact(case, seed):
    kind = case["kind"]
    V = case.get("x", 0) * case.get("y", 0) * case.get("z", 0)
    if kind in ("infer", "train"):
        with np.load(os.path.join(os.path.dirname(DEFAULT_WEIGHTS), "warmstart_256x256x128.npz")) as f:
            weights, scale = f["params"], float(f["scale"])
        v, target = _pair(case, seed)
        params = _f64(weights)
        if kind == "infer":
            with torch.no_grad():
                return _network(params, v[0].double(), scale)[None]
        params.requires_grad_(True)
        loss = ((_network(params, v[0].double(), scale) - target[0].double()) / scale).square().mean()
        loss.backward()
        g = params.grad
        return {"loss": float(loss.detach()), "params": (params.detach() - LEARNING_RATE * g / (g.abs() + 1e-8)).cpu().numpy()}
    if kind == "forward":
        p, l = _project(_phantom(case, seed).double(), case, case["tilt"])
        return {"projection": p, "length": l}
    if kind == "back":
        vol = _phantom(case, seed).double()
        r, l = _residual(case, seed)
        _back(vol, case, case["tilt"], r.double(), l.double(), 0.3)
        return vol
    if kind == "wbp":
        b = _ramlak(_projections(case, seed))
        vol = torch.zeros((case["z"], case["y"], case["x"]), device="cuda", dtype=torch.float64)
        empty = torch.zeros((case["z"], case["y"], case["x"]), device="cuda", dtype=torch.float64)
        for i, a in enumerate(_views(case)):
            _back(vol, case, a, b[i], _project(empty, case, a)[1], 1.0 / b.shape[0])
        return vol
    if kind == "batch":
        found = [_reconstruct(m, _projections(m, seed + 7919 * j)) for j, m in enumerate(_batch_members(case))]
        return {"volumes": [f["volume"] for f in found], "residual_sq": np.array([f["residual_sq"] for f in found])}
    if case.get("slabs", 1) > 1 and case["z"] % 2:
        return None   # every slab's own half-voxel grid is not restated here
    if case.get("perspective"):
        rays = case["x"] * case["y"] * case["views"] * case["iterations"]
        if case["order"] == "random" or rays * float(case["x"] + case["y"] + case["z"]) > 1e10:
            return None
    return _reconstruct(case, _projections(case, seed))
