"""The kernels that a call's shape selects against the general ones they stand in for, at the
edges of their tiles and of the rules that select them.

* bp_persp_row_kernel (perspective views tilted about y, columns along y) against
  bp_perspective_kernel (a context created with ETCU_BP_COLUMN=0) and the oracle.  The same
  operations per voxel: the updates are equal but for columns whose u lies within a last bit of the
  edge of a 1/256 step.  That is a share of about 256 ulp(u) = 256 * 2^-18 = 1e-3 of the columns (u
  below 128), each off by at most 1/256 of the two texels' difference, of the size of the values
  themselves: STEP_TOL = sqrt(1e-3) / 256 = 1.2e-4 relative.
* bp_block_kernel for one view (rows that the column kernel does not take, from the size
  at which they fill the chip) against bp_sart_row_kernel: the detector rows are blended first
  and the ray length's reciprocal estimated, a few ulps per update: SAME_TOL.
* the persistent fused SART step's narrow rows (several groups of threads on a chunk's
  slices) against the unfused kernels: bit-identical, widths around whole warps and the half
  block at which the wide form takes over.
* input gradients on the z-streamed convolution against the per-tap kernel (ETCU_CONV_ZFOLD=0):
  two orders of FP32 sums whose BF16 roundings flip here and there, within the bar that both keep to
  the oracle."""
import os

import numpy as np
import pytest

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


def _kernels(run):
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    return {e.name for e in prof.events()}


PERSP = [
    # (X, Y, Z), views, detector (W, H) or None, sign of the row pitch, source distance / X, clamp, sub-volumes, storage
    ((32, 16, 4), 3, None, 1, 10.0, None, 1, "float32"),
    ((33, 15, 5), 4, None, 1, 10.0, None, 1, "float32"),
    ((70, 31, 9), 5, None, -1, 10.0, None, 2, "float32"),
    ((100, 48, 37), 7, (60, 20), 1, 3.0, None, 1, "float32"),   # most voxels project off the detector
    ((64, 32, 20), 1, None, 1, 10.0, (0.1, 0.9), 1, "float32"),
    ((96, 30, 24), 8, None, 1, 10.0, None, 3, "bf16_master"),
    ((96, 30, 24), 3, None, 1, 10.0, None, 1, "f16_master"),
    ((96, 30, 24), 3, None, 1, 10.0, None, 1, "half"),
    ((32, 17, 8), 2, None, 1, 10.0, None, 1, "float32"),        # too many idle rows: the general kernel
]


@pytest.mark.parametrize("shape,nviews,det,sign,dist,clamp,subs,storage", PERSP)
def test_perspective_rows_match_general_and_oracle(ctxs, shape, nviews, det, sign, dist, clamp, subs, storage):
    from oracle import oracle as O
    from ettention_b200 import _abi
    from ettention_b200.operators import (AlgebraicParameterSet, BlockIterativeReconstructionOperator,
                                          GPUMappedVolume, ScannerGeometry)
    from tests.helpers import oracle_geometry
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
        vol.upload(init)
        rec = BlockIterativeReconstructionOperator(vol, geoms, projs, params, use_graph=False)
        names.append(_kernels(lambda: rec.runNiterations(1)))
        outs.append(rec.getReconstructedVolume())
        rec.close()
        vol.close()
    assert not any("bp_persp_row_kernel" in n for n in names[0])
    assert any("bp_persp_row_kernel" in n for n in names[1]) == (shape != (32, 17, 8))
    assert np.abs(outs[0] - init).max() > 0
    if storage == "half":  # re-rounded after every view: a last-bit difference can move a voxel by one half ulp
        assert O.rel_l2(outs[1], outs[0]) <= 1e-3
        return
    update, general = outs[1] - init, outs[0] - init
    assert O.rel_l2(update, general) <= STEP_TOL
    assert (np.abs(update - general).max(axis=1) > 1e-6 * np.abs(general).max()).mean() <= 1e-2  # columns along y
    if storage == "float32" and clamp is None:
        setup = O.ReconstructionSetup(O.VolumeGeometry.centered(shape, subvolumes=subs),
                                      [oracle_geometry(g) for g in geoms], projs, 0.2, nviews)
        vo = init.copy()
        O.block_iterative(setup, vo, 1, 32)
        # the forward projection of random values along grazing rays takes part too, so the bar is the
        # general kernel's own distance (BP_TOL for the back projection alone, test_gpu_parity.py)
        assert O.rel_l2(update, vo - init) <= max(BP_TOL, O.rel_l2(general, vo - init) + STEP_TOL)


@pytest.mark.parametrize("shape,tilt,half", [((1001, 61, 64), -27.5, False), ((1999, 33, 57), 63.0, False),
                                             ((256, 240, 61), 41.0, True)])
def test_one_view_block_matches_row_kernel(ctxs, shape, tilt, half):
    import torch
    from oracle import oracle as O
    from ettention_b200 import _abi
    from ettention_b200.operators import BackProjectionOperator, GPUMappedVolume, mrc_base_geometry
    X, Y, Z = shape
    rng = np.random.Generator(np.random.PCG64(X))
    g = mrc_base_geometry(X, Y).rotated(tilt)
    res = torch.tensor(rng.normal(size=(Y, X)).astype(np.float32), device="cuda")
    length = torch.tensor(rng.uniform(0.5, 2.0 * Z, size=(Y, X)).astype(np.float32), device="cuda")
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    outs, names = [], []
    for ctx in ctxs:
        vol = GPUMappedVolume(ctx, shape, voxel_type=_abi.VOXEL_HALF16 if half else _abi.VOXEL_FLOAT32)
        vol.upload(init)
        bp = BackProjectionOperator(vol, 0.3, 1)
        bp.setScannerGeometry(g)
        bp.setInput(res, length, 1)
        names.append(_kernels(bp.execute))
        outs.append(vol.download())
        vol.close()
    assert any("bp_sart_row_kernel" in n for n in names[0])
    assert any("bp_block_kernel" in n for n in names[1])
    assert np.abs(outs[0] - init).max() > 0
    if half:
        assert O.rel_l2(outs[1], outs[0]) <= 1e-3
    else:
        assert O.rel_l2(outs[1] - init, outs[0] - init) <= SAME_TOL


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
