"""The kernels that a call's shape selects against the general ones they stand in for, at the
edges of their tiles and of the rules that select them.

* bp_persp_row_kernel (perspective views tilted about y, columns along y) against
  bp_perspective_kernel (a context created with ETCU_BP_COLUMN=0) and the oracle.  The same
  operations per voxel: the updates are equal but for columns whose u lies within a last bit of the
  edge of a 1/256 step.  That is a share of about 256 ulp(u) = 256 * 2^-18 = 1e-3 of the columns (u
  below 128), each off by at most 1/256 of the two texels' difference, of the size of the values
  themselves: STEP_TOL = sqrt(1e-3) / 256 = 1.2e-4 relative.
* bp_block_kernel for one view (rows that the column kernel does not take, from the size
  at which they fill the chip) against bp_sart_row_kernel: the detector rows are blended first, a few
  ulps per update: SAME_TOL.  Each one's own error is held to a 64-bit restatement.
* the forward projector's counted walk (shallow volumes) against its walk in rounds.
* several views of one launch side by side against each view in a launch of its own.
* the persistent fused SART step's narrow rows (several groups of threads on a chunk's
  slices) against the unfused kernels: bit-identical, widths around whole warps and the 256 voxels
  from which the wide form takes over.
* input gradients on the z-streamed convolution against the per-tap kernel (ETCU_CONV_ZFOLD=0):
  two orders of FP32 sums whose BF16 roundings flip here and there, within the bar that both keep to
  the oracle."""
import os

import numpy as np
import pytest

from tests.helpers import launched_back_projectors, require_records

pytestmark = pytest.mark.gpu

BP_TOL = 1e-4
SAME_TOL = 1e-6
STEP_TOL = 1.2e-4


def _context(**env):
    from ettention_b200.operators import Context
    os.environ.update(env)
    try:
        return Context(0)
    finally:
        for k in env:
            del os.environ[k]


@pytest.fixture(scope="module")
def ctxs():
    import torch
    assert torch.cuda.is_available()
    general, rows = _context(ETCU_BP_COLUMN="0"), _context()
    yield general, rows
    rows.close()
    general.close()


PERSP = [
    # (X, Y, Z), views, detector (W, H) or None, sign of the row pitch, source distance / X, clamp, sub-volumes, storage,
    # whether the row kernel takes it
    ((32, 16, 4), 3, None, 1, 10.0, None, 1, "float32", True),
    ((33, 15, 5), 4, None, 1, 10.0, None, 1, "float32", True),
    ((70, 31, 9), 5, None, -1, 10.0, None, 2, "float32", True),
    ((100, 48, 37), 7, (60, 20), 1, 3.0, None, 1, "float32", True),   # most voxels project off the detector
    ((64, 32, 20), 1, None, 1, 10.0, (0.1, 0.9), 1, "float32", True),
    ((96, 30, 24), 8, None, 1, 10.0, None, 3, "bf16_master", True),
    ((96, 30, 24), 3, None, 1, 10.0, None, 1, "f16_master", True),
    ((96, 30, 24), 3, None, 1, 10.0, None, 1, "half", True),
    ((32, 17, 8), 2, None, 1, 10.0, None, 1, "float32", True),        # mostly padding, but resident
    ((256, 129, 56), 1, None, 1, 10.0, None, 1, "float32", False),    # one view, the second round of blocks half empty
    ((256, 129, 56), 2, None, 1, 10.0, None, 1, "float32", True),
    ((256, 64, 64), 1, None, 1, 10.0, None, 1, "bf16_master", False),  # one view, more than half of the residency
    ((256, 129, 56), 2, None, 1, 10.0, None, 1, "bf16_master", False),
    ((256, 17, 224), 2, None, 1, 10.0, None, 1, "float32", False),    # a third more padding than along z
    ((256, 129, 56), 4, None, 1, 10.0, None, 1, "half", True),
]


@pytest.mark.parametrize("shape,nviews,det,sign,dist,clamp,subs,storage,rows", PERSP)
def test_perspective_rows_match_general(ctxs, shape, nviews, det, sign, dist, clamp, subs, storage, rows):
    from oracle import oracle as O
    from ettention_b200 import _abi
    from ettention_b200.operators import (AlgebraicParameterSet, BlockIterativeReconstructionOperator,
                                          GPUMappedVolume, ScannerGeometry)
    X, Y, Z = shape
    W, H = det or (X, Y)
    p = 1.1
    base = ScannerGeometry([0.0, 0.0, dist * X], [-0.5 * W * p, -0.5 * sign * H * p, -float(X)], [p, 0.0, 0.0],
                           [0.0, sign * p, 0.0], W, H, True)
    geoms = [base.rotated(float(a)) for a in np.linspace(-58.0, 61.0, nviews)]
    rng = np.random.Generator(np.random.PCG64(X * 100 + Y))
    projs = rng.uniform(0.0, 4.0, size=(nviews, H, W)).astype(np.float32)
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    kind = {"float32": _abi.VOXEL_FLOAT32, "f16_master": _abi.VOXEL_F16_MASTER, "bf16_master": _abi.VOXEL_BF16_MASTER,
            "half": _abi.VOXEL_HALF16}[storage]
    params = AlgebraicParameterSet(algorithm="sirt", block_size=_abi.BLOCK_ALL, iterations=1, lam=0.2,
                                   order=_abi.ORDER_IDENTITY)
    outs, names = [], []
    for ctx in ctxs:
        vol = GPUMappedVolume(ctx, shape, voxel_type=kind, subvolume_count=subs)
        if clamp:
            vol.set_intensity_clamp(clamp[0], clamp[1])
        rec = BlockIterativeReconstructionOperator(vol, geoms, projs, params, use_graph=False)

        def run():
            vol.upload(init)
            rec.runNiterations(1)
        names.append(launched_back_projectors(run, subs))
        outs.append(rec.getReconstructedVolume())
        rec.close()
        vol.close()
    assert np.abs(outs[0] - init).max() > 0
    update, general = outs[1] - init, outs[0] - init
    if storage == "half":  # re-rounded after every view: a last-bit difference can move a voxel by one half ulp
        assert O.rel_l2(outs[1], outs[0]) <= 1e-3
    else:
        assert O.rel_l2(update, general) <= STEP_TOL
        assert (np.abs(update - general).max(axis=1) > 1e-6 * np.abs(general).max()).mean() <= 1e-2  # columns along y
    require_records(*names)
    assert not any("bp_persp_row_kernel" in n for n in names[0])
    assert any("bp_persp_row_kernel" in n for n in names[1]) == rows


@pytest.mark.parametrize("shape,det,sign,dist,subs", [((32, 16, 4), None, 1, 10.0, 1), ((33, 15, 5), None, 1, 10.0, 1),
                                                      ((70, 31, 9), None, -1, 10.0, 2),
                                                      ((100, 48, 37), (60, 20), 1, 3.0, 1),
                                                      ((96, 96, 40), (110, 90), 1, 10.0, 1)])
def test_perspective_rows_match_oracle(ctxs, shape, det, sign, dist, subs):
    """The back projection alone against the oracle's, within BP_TOL whatever the general kernel's distance is.  The
    images of residuals and ray lengths are smooth (a tenth of a value from texel to texel), so that a
    coordinate on the other side of a 1/256 step moves a contribution by 0.1 / 256: with u and v some ulps
    (2^-18 .. 2^-17) off that is 256 * 2^-16 = 4e-3 of the voxels, sqrt(4e-3) * 0.1 / 256 = 2.5e-5 in the
    2-norm."""
    import torch
    from oracle import oracle as O
    from ettention_b200.operators import BackProjectionOperator, GPUMappedVolume, ScannerGeometry
    from tests.helpers import oracle_geometry
    X, Y, Z = shape
    W, H = det or (X, Y)
    p = 1.1
    base = ScannerGeometry([0.0, 0.0, dist * X], [-0.5 * W * p, -0.5 * sign * H * p, -float(X)], [p, 0.0, 0.0],
                           [0.0, sign * p, 0.0], W, H, True)
    rng = np.random.Generator(np.random.PCG64(X * 10 + Y))
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    for tilt in (-58.0, 0.0, 33.0):
        g = base.rotated(tilt)
        px, py = np.meshgrid(np.arange(W), np.arange(H))
        res = (1.5 + np.sin(0.15 * px + tilt) * np.cos(0.11 * py)).astype(np.float32)
        length = (Z * (1.2 + 0.4 * np.cos(0.13 * px) * np.sin(0.1 * py + tilt))).astype(np.float32)
        vol = GPUMappedVolume(ctxs[1], shape, subvolume_count=subs)
        bp = BackProjectionOperator(vol, 0.3, 1)
        bp.setScannerGeometry(g)
        bp.setInput(torch.tensor(res, device="cuda"), torch.tensor(length, device="cuda"), 1)

        def run():
            vol.upload(init)
            bp.execute()
        names = launched_back_projectors(run, subs)
        out = vol.download()
        vol.close()
        vo = init.copy()
        O.back_project(vo, O.VolumeGeometry.centered(shape, subvolumes=subs), oracle_geometry(g), res, length, 0.3, 1, 32,
                       O.WEIGHTS_Q8)
        assert np.abs(vo - init).max() > 0
        assert O.rel_l2(out - init, vo - init) <= BP_TOL
        require_records(names)
        assert all("bp_persp_row_kernel" in n for n in names)


@pytest.mark.parametrize("shape,tilt,storage,block", [((1001, 61, 64), -27.5, "float32", True),
                                                       ((1999, 33, 57), 63.0, "float32", True),
                                                       ((255, 240, 61), 41.0, "bf16_master", True),
                                                       ((256, 240, 61), 41.0, "half", False),
                                                       ((129, 601, 68), 41.0, "float32", False)])  # half of it padding
def test_one_view_block_matches_row_kernel(ctxs, shape, tilt, storage, block):
    import torch
    from oracle import oracle as O
    from ettention_b200 import _abi
    from ettention_b200.operators import BackProjectionOperator, GPUMappedVolume, mrc_base_geometry
    X, Y, Z = shape
    kind = {"float32": _abi.VOXEL_FLOAT32, "bf16_master": _abi.VOXEL_BF16_MASTER, "half": _abi.VOXEL_HALF16}[storage]
    rng = np.random.Generator(np.random.PCG64(X))
    g = mrc_base_geometry(X, Y).rotated(tilt)
    res = torch.tensor(rng.normal(size=(Y, X)).astype(np.float32), device="cuda")
    length = torch.tensor(rng.uniform(0.5, 2.0 * Z, size=(Y, X)).astype(np.float32), device="cuda")
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    outs, names = [], []
    for ctx in ctxs:
        vol = GPUMappedVolume(ctx, shape, voxel_type=kind)
        bp = BackProjectionOperator(vol, 0.3, 1)
        bp.setScannerGeometry(g)
        bp.setInput(res, length, 1)

        def run():
            vol.upload(init)
            bp.execute()
        names.append(launched_back_projectors(run, 1))
        outs.append(vol.download())
        vol.close()
    assert np.abs(outs[0] - init).max() > 0
    if block:
        assert O.rel_l2(outs[1] - init, outs[0] - init) <= SAME_TOL
    else:
        assert np.array_equal(outs[1], outs[0])
    require_records(*names)
    assert any("bp_sart_row_kernel" in n for n in names[0])
    assert any("bp_block_kernel" in n for n in names[1]) == block


def _exact_update(shape, g, res, length, lam, samples):
    """One view's update in 64 bits, at the kernels' coordinates and 1/256 weights: u and v step by
    step in FP32 as both kernels form them, then the bilinear sums, the quotient and the samples' mean."""
    f = np.float32
    m = g.projection_matrix()
    assert m[1] == 0 and m[9] == 0  # one detector row coordinate per y
    centre = [f(-0.5 * n) + (np.arange(n, dtype=f) + f(0.5)) for n in shape]

    def split(c, n):
        t = c - f(0.5)
        base = np.floor(t)
        frac = np.floor((t - base) * f(256) + f(0.5)).astype(np.float64) / 256
        return np.clip(base.astype(np.int64), -2, n) + 2, frac  # + 2: the padded images' offset
    pad = [np.pad(a.astype(np.float64), 2) for a in (res, length)]
    total, used = np.zeros(shape[::-1]), np.zeros(shape[::-1])
    for s in g.sample_pattern([1, 1, 1], samples):
        px, py, pz = (c + s[i] for i, c in enumerate(centre))
        v0, b = split((m[1] * px[0] + m[5] * py) + m[13], res.shape[0])
        rows = [a[v0] * (1 - b)[:, None] + a[v0 + 1] * b[:, None] for a in pad]
        for z in range(shape[2]):
            u = ((m[0] * px)[None, :] + (m[4] * py)[:, None] + m[8] * pz[z]) + m[12]
            u0, a = split(u, res.shape[1])
            R, L = (np.take_along_axis(r, u0, 1) * (1 - a) + np.take_along_axis(r, u0 + 1, 1) * a for r in rows)
            total[z] += np.where(L > 1e-4, R * (float(f(lam)) * float(s[3])) / np.maximum(L, 1e-4), 0.0)
            used[z] += L > 1e-4
    return total / np.maximum(used, 1)


@pytest.mark.parametrize("shape,tilt,smooth,samples", [((1001, 61, 64), -27.5, False, 1), ((999, 64, 63), 48.0, False, 1),
                                                       ((501, 91, 91), 0.0, False, 1), ((501, 91, 91), 69.0, False, 1),
                                                       ((1001, 61, 64), -27.5, True, 1), ((501, 91, 91), 61.5, True, 1),
                                                       ((130, 64, 65), -35.0, False, 4), ((130, 64, 65), 20.0, True, 9)])
def test_staged_update_is_as_close_to_64_bits_as_the_general_kernels(ctxs, shape, tilt, smooth, samples):
    """bp_block_kernel's FP32 error per update is no larger than that of bp_sart_row_kernel (one sample) and
    bp_parallel_kernel (several), in the 2-norm and in the largest error, for noise residuals and ray
    lengths (taps that differ by their own size) and for smooth ones."""
    import torch
    from ettention_b200.operators import BackProjectionOperator, GPUMappedVolume, mrc_base_geometry
    X, Y, Z = shape
    rng = np.random.Generator(np.random.PCG64(X + Y))
    g = mrc_base_geometry(X, Y).rotated(tilt)
    if smooth:
        x, y = np.meshgrid(np.arange(X) / 17.0, np.arange(Y) / 13.0)
        res, length = np.sin(x) * np.cos(y) + 0.3, Z * (1.2 + 0.2 * np.sin(0.3 * x))
    else:
        res, length = rng.normal(size=(Y, X)), rng.uniform(0.5, 2.0 * Z, size=(Y, X))
    res, length = res.astype(np.float32), length.astype(np.float32)
    exact = _exact_update(shape, g, res, length, 0.3, samples)
    errors = []
    for ctx in ctxs:
        vol = GPUMappedVolume(ctx, shape)
        vol.upload(np.zeros((Z, Y, X), np.float32))
        bp = BackProjectionOperator(vol, 0.3, samples)
        bp.setScannerGeometry(g)
        bp.setInput(torch.tensor(res, device="cuda"), torch.tensor(length, device="cuda"), 1)
        bp.execute()
        d = vol.download().astype(np.float64) - exact
        errors.append((np.linalg.norm(d) / np.linalg.norm(exact), np.abs(d).max() / np.sqrt((exact ** 2).mean())))
        vol.close()
    assert errors[0][0] < 2e-7  # the 64-bit restatement takes the kernels' taps
    assert errors[1][0] <= errors[0][0]
    assert errors[1][1] <= 1.1 * errors[0][1]  # the extreme of some 10^5 .. 10^6 updates


@pytest.mark.parametrize("shape", [(4, 5, 3), (60, 9, 70), (64, 6, 64), (68, 12, 130), (256, 7, 9), (260, 5, 33),
                                   (508, 4, 40), (512, 6, 16), (516, 4, 20), (1024, 3, 24)])
@pytest.mark.parametrize("storage", ["float32", "bf16_master"])
def test_narrow_fused_rows_are_bit_identical_to_unfused(shape, storage):
    from ettention_b200 import _abi
    from ettention_b200.operators import (AlgebraicParameterSet, BlockIterativeReconstructionOperator,
                                          GPUMappedVolume, mrc_base_geometry)
    X, Y, Z = shape
    rng = np.random.Generator(np.random.PCG64(X + Z))
    geoms = [mrc_base_geometry(X, Y).rotated(float(a)) for a in (-62.0, -20.5, 0.0, 33.0, 90.0, 120.0, 180.0)]
    projs = rng.uniform(0.0, 4.0, size=(len(geoms), Y, X)).astype(np.float32)
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    kind = {"float32": _abi.VOXEL_FLOAT32, "bf16_master": _abi.VOXEL_BF16_MASTER}[storage]
    p = AlgebraicParameterSet(algorithm="sart", block_size=1, iterations=2, lam=0.3, order=_abi.ORDER_IDENTITY)
    outs = []
    for env in ({"ETCU_FUSED": "0"}, {}):
        ctx = _context(**env)
        vol = GPUMappedVolume(ctx, shape, voxel_type=kind)
        vol.upload(init)
        rec = BlockIterativeReconstructionOperator(vol, geoms, projs, p)
        assert rec.launches_per_iteration == (3 if not env else 2 * len(geoms))
        rec.runNiterations(2)
        outs.append((rec.getReconstructedVolume(), rec.last_residual_sq()))
        rec.close()
        vol.close()
        ctx.close()
    assert np.abs(outs[0][0] - init).max() > 0
    assert np.array_equal(outs[1][0], outs[0][0])
    assert outs[1][1] == pytest.approx(outs[0][1], rel=1e-12)


@pytest.mark.parametrize("shape", [(4, 5, 3), (64, 6, 100), (70, 5, 33), (130, 3, 97), (900, 2, 112), (37, 4, 101),
                                   (64, 3, 260)])
@pytest.mark.parametrize("storage", ["float32", "bf16_master", "half"])
def test_forward_walks_are_bit_identical(ctxs, shape, storage):
    """Volumes up to 100 slices deep, or an eighth of their width, take the counted walk; a mask of ones
    sends them to the walk in rounds with the same weights.  The last two shapes take the rounds both ways,
    with and without mask (depths around the line)."""
    import torch
    from ettention_b200 import _abi
    from ettention_b200.operators import ForwardProjectionOperator, GPUMappedVolume, mrc_base_geometry
    X, Y, Z = shape
    kind = {"float32": _abi.VOXEL_FLOAT32, "bf16_master": _abi.VOXEL_BF16_MASTER, "half": _abi.VOXEL_HALF16}[storage]
    rng = np.random.Generator(np.random.PCG64(X + Z))
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    for samples in (1, 2):
        images = []
        for mask in (None, np.full((Z, Y, X), 255, np.uint8)):
            vol = GPUMappedVolume(ctxs[1], shape, voxel_type=kind)
            vol.upload(init)
            if mask is not None:
                vol.set_mask(mask)
            op = ForwardProjectionOperator(vol, samples)
            for tilt in (-89.5, -61.0, -30.3, 0.0, 12.5, 45.0, 70.0, 90.0, 135.0, 180.0, 233.0):
                v, length = (torch.zeros((Y, X), device="cuda") for _ in range(2))
                op.setScannerGeometry(mrc_base_geometry(X, Y).rotated(tilt))
                op.SetOutput(v, length)
                op.Execute(0)
                images.append(torch.stack([v, length]).cpu().numpy())
            vol.close()
        n = len(images) // 2
        assert all(i.max() > 0 for i in images)
        assert all(np.array_equal(a, b) for a, b in zip(images[:n], images[n:]))


@pytest.mark.parametrize("perspective", [False, True])
def test_views_side_by_side_write_their_own_images(ctxs, perspective):
    """A volume of 92 MB, whose views share a launch's detector rows: the sum of the squared residuals
    over 3 views equals the sum over a launch per view (the same FP32 values, sums in FP64)."""
    from ettention_b200 import _abi
    from ettention_b200.operators import (AlgebraicParameterSet, BlockIterativeReconstructionOperator,
                                          GPUMappedVolume, ScannerGeometry)
    X, Y, Z, W, H = 300, 300, 256, 291, 77
    if perspective:
        base = ScannerGeometry([0.0, 0.0, 10.0 * X], [-0.55 * X, -0.55 * Y, -float(X)], [1.1 * X / W, 0.0, 0.0],
                               [0.0, 1.1 * Y / H, 0.0], W, H, True)
    else:
        base = ScannerGeometry([-0.5 * X, -0.5 * Y, float(X)], [-0.5 * X, -0.5 * Y, -float(X)], [X / W, 0.0, 0.0],
                               [0.0, Y / H, 0.0], W, H, False)
    geoms = [base.rotated(a) for a in (-50.0, 3.0, 41.0)]
    rng = np.random.Generator(np.random.PCG64(3))
    projs = (rng.uniform(0.0, 4.0, size=(3, H, W)) * np.array([1.0, 8.0, 64.0])[:, None, None]).astype(np.float32)
    vol = GPUMappedVolume(ctxs[1], (X, Y, Z))
    vol.upload(rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32))

    def residual(views):
        p = AlgebraicParameterSet(algorithm="sirt", block_size=_abi.BLOCK_ALL, iterations=1, lam=0.3,
                                  order=_abi.ORDER_IDENTITY)
        rec = BlockIterativeReconstructionOperator(vol, [geoms[v] for v in views], projs[views], p, use_graph=False)
        r = rec.data_residual_sq()
        rec.close()
        return r
    together, apart = residual([0, 1, 2]), [residual([v]) for v in range(3)]
    vol.close()
    assert all(a > 0 for a in apart)
    assert together == pytest.approx(sum(apart), rel=1e-12)


@pytest.mark.parametrize("res,batch", [((4, 4, 4), 2), ((124, 12, 36), 1), ((264, 4, 68), 2)])
def test_zstreamed_input_gradients_match_per_tap(monkeypatch, res, batch):
    import torch
    from oracle import warmstart_oracle as W
    from ettention_b200.learned import WarmStartNet
    from tests.test_gpu_learned import GRAD_TOL, _params, _rel, _volumes
    p = _params(21)
    v, t = _volumes(res, batch, 22)
    ctx, grads = _context(), []
    try:
        for mode in ("0", "1"):
            monkeypatch.setenv("ETCU_CONV_ZFOLD", mode)
            with WarmStartNet(ctx, res, max_batch=batch, params=p, scale=0.7) as net:
                grads.append(net.gradients(torch.as_tensor(v).cuda(), torch.as_tensor(t).cuda(), batch))
    finally:
        ctx.close()
    assert abs(grads[0][0] - grads[1][0]) <= 1e-3 * grads[0][0]
    for i, (wo, bo) in enumerate(W.layer_offsets()):
        end = bo + W.LAYERS[i][2]
        assert _rel(grads[1][1][wo:end], grads[0][1][wo:end]) <= GRAD_TOL, f"layer {i}"
