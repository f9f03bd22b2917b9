"""The window-staged back projection of a block of views tilted about y (bp_block_kernel)
against the general kernel (a context created with ETCU_BP_COLUMN=0 never uses it) and the
oracle: reconstructions of one block from a random start, so that the update of every voxel
is the sum over the block's views.

The two kernels form the same coordinates and 1/256 weights; the staged one blends the two
detector rows first, a few ulps per view's contribution, so the updates agree to 1e-6 relative (SAME_TOL), and both with the
FP32 oracle to the back-projection bar of 1e-4.  Shapes: rows of less than, exactly and one
more than the 64 / 128 / 256 voxels of a block, odd sizes, slices that leave a block's last
ones empty, detector rows between volume rows, a detector narrower than the volume's
shadow, several sub-volumes, several samples per voxel, every storage."""
import os

import numpy as np
import pytest

from tests.helpers import launched_back_projectors, require_records

pytestmark = pytest.mark.gpu

BP_TOL = 1e-4
SAME_TOL = 1e-6


@pytest.fixture(scope="module")
def ctxs():
    import torch
    from ettention_b200.operators import Context
    assert torch.cuda.is_available()
    os.environ["ETCU_BP_COLUMN"] = "0"
    try:
        general = Context(0)
    finally:
        del os.environ["ETCU_BP_COLUMN"]
    staged = Context(0)
    yield general, staged
    staged.close()
    general.close()


CASES = [
    # (X, Y, Z), views, detector row pitch, detector width, sub-volumes, samples per voxel, storage
    ((1, 3, 5), 3, 1.0, None, 1, 1, "float32"),
    ((64, 6, 8), 4, 1.0, None, 1, 1, "float32"),
    ((65, 7, 9), 5, 1.0, None, 1, 1, "float32"),
    ((129, 5, 33), 7, 0.75, None, 2, 1, "float32"),
    ((250, 4, 70), 9, 1.0, 130, 1, 1, "float32"),
    ((257, 3, 31), 6, 1.0, None, 3, 4, "float32"),
    ((130, 9, 17), 3, 1.25, None, 1, 9, "float32"),
    ((96, 8, 40), 5, 1.0, None, 1, 1, "f16_master"),
    ((96, 8, 40), 5, 1.0, None, 1, 4, "bf16_master"),
    ((96, 8, 40), 5, 1.0, None, 1, 1, "half"),
]


@pytest.mark.parametrize("shape,nviews,vpitch,width,subs,samples,storage", CASES)
def test_staged_block_matches_general_and_oracle(ctxs, shape, nviews, vpitch, width, subs, samples, storage):
    from oracle import oracle as O
    from ettention_b200 import _abi
    from ettention_b200.operators import (AlgebraicParameterSet, BlockIterativeReconstructionOperator,
                                          GPUMappedVolume, ScannerGeometry)
    from tests.helpers import oracle_geometry
    X, Y, Z = shape
    W = X if width is None else width
    H = max(1, int(round(Y / vpitch)))
    base = ScannerGeometry([-0.5 * W, -0.5 * H * vpitch, float(X + Z)], [-0.5 * W, -0.5 * H * vpitch, -float(X + Z)],
                           [1.0, 0.0, 0.0], [0.0, vpitch, 0.0], W, H, False)
    angles = np.linspace(-63.0, 58.0, nviews)
    geoms = [base.rotated(float(a)) for a in angles]
    rng = np.random.Generator(np.random.PCG64(X * 100 + Z + samples))
    projs = rng.uniform(0.0, 4.0, size=(nviews, H, W)).astype(np.float32)
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    kind = {"float32": _abi.VOXEL_FLOAT32, "f16_master": _abi.VOXEL_F16_MASTER, "bf16_master": _abi.VOXEL_BF16_MASTER,
            "half": _abi.VOXEL_HALF16}[storage]
    p = AlgebraicParameterSet(algorithm="sirt", block_size=_abi.BLOCK_ALL, iterations=1, lam=0.3, bp_samples=samples,
                              order=_abi.ORDER_IDENTITY)
    outs, names = [], []
    for ctx in ctxs:
        vol = GPUMappedVolume(ctx, shape, voxel_type=kind, subvolume_count=subs)
        rec = BlockIterativeReconstructionOperator(vol, geoms, projs, p, use_graph=False)

        def run():
            vol.upload(init)
            rec.runNiterations(1)
        names.append(launched_back_projectors(run, subs))
        outs.append(rec.getReconstructedVolume())
        rec.close()
        vol.close()
    assert np.abs(outs[0] - init).max() > 0
    if storage == "half":  # re-rounded after every view: a last-bit difference can move a voxel by one half ulp
        assert O.rel_l2(outs[1], outs[0]) <= 1e-3
    else:
        # a pixel whose true ray length is near the 1e-4 threshold would be kept by one kernel and skipped by the
        # other: random projections leave none here
        assert O.rel_l2(outs[1] - init, outs[0] - init) <= SAME_TOL
    if storage == "float32":
        setup = O.ReconstructionSetup(O.VolumeGeometry.centered(shape, subvolumes=subs),
                                      [oracle_geometry(g) for g in geoms], projs, 0.3, nviews, 1, samples)
        vo = init.copy()
        O.block_iterative(setup, vo, 1, 32)
        assert O.rel_l2(outs[1] - init, vo - init) <= BP_TOL
    require_records(*names)
    assert all("bp_parallel_kernel" in n for n in names[0])
    assert all("bp_block_kernel" in n for n in names[1])


@pytest.mark.parametrize("order", ["identity", "maxangle"])
def test_views_over_several_launches(ctxs, order):
    """90 views of 9 samples: their constants exceed a launch's 32 KB (56 views), so a second one goes on with
    the views that remain, on the volume that the first one left."""
    from oracle import oracle as O
    from ettention_b200 import _abi
    from ettention_b200.operators import (AlgebraicParameterSet, BlockIterativeReconstructionOperator,
                                          GPUMappedVolume, mrc_base_geometry)
    from tests.helpers import oracle_geometry
    X, Y, Z, N = 65, 4, 9, 90
    geoms = [mrc_base_geometry(X, Y).rotated(float(a)) for a in np.linspace(-63.0, 58.0, N)]
    rng = np.random.Generator(np.random.PCG64(N))
    projs = rng.uniform(0.0, 4.0, size=(N, Y, X)).astype(np.float32)
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    p = AlgebraicParameterSet(algorithm="sirt", block_size=_abi.BLOCK_ALL, iterations=1, lam=0.3, bp_samples=9,
                              order={"identity": _abi.ORDER_IDENTITY, "maxangle": _abi.ORDER_MAXANGLE}[order])
    outs, names = [], []
    for ctx, launches in zip(ctxs, (1, 2)):
        vol = GPUMappedVolume(ctx, (X, Y, Z))
        rec = BlockIterativeReconstructionOperator(vol, geoms, projs, p, use_graph=False)
        assert (rec.view_order() == list(range(N))) == (order == "identity")

        def run():
            vol.upload(init)
            rec.runNiterations(1)
        names.append(launched_back_projectors(run, launches))
        outs.append(rec.getReconstructedVolume())
        rec.close()
        vol.close()
    assert O.rel_l2(outs[1] - init, outs[0] - init) <= SAME_TOL
    if order == "identity":
        setup = O.ReconstructionSetup(O.VolumeGeometry.centered((X, Y, Z)), [oracle_geometry(g) for g in geoms], projs,
                                      0.3, N, 1, 9)
        vo = init.copy()
        O.block_iterative(setup, vo, 1, 32)
        assert O.rel_l2(outs[1] - init, vo - init) <= BP_TOL
    require_records(*names)
    assert all("bp_parallel_kernel" in n for n in names[0]) and all("bp_block_kernel" in n for n in names[1])


@pytest.mark.parametrize("samples", [1, 4])
def test_boxes_far_along_the_rays_keep_the_general_kernels(ctxs, samples):
    """A box four million pixels from the origin along the view's rays: its columns are the detector's, but the two
    terms of u that cancel there are a quarter of a pixel apart in FP32, and a window bounded in
    advance need not hold every tap.  Neither the column kernel (one sample) nor the staged one (several)
    takes it, and the results are the general kernels'."""
    import torch
    from ettention_b200.operators import BackProjectionOperator, GPUMappedVolume, mrc_base_geometry
    X, Y, Z, far = 64, 8, 16, 3.0e6
    g = mrc_base_geometry(X, Y).rotated(45.0)
    m = g.projection_matrix()
    cz = float(np.round(-far * float(m[0]) / float(m[8])))
    assert abs(float(m[0]) * far + float(m[8]) * cz) < 4.0  # u of the centre: that of a box at the origin
    rng = np.random.Generator(np.random.PCG64(5))
    res = torch.tensor(rng.normal(size=(Y, X)).astype(np.float32), device="cuda")
    length = torch.tensor(rng.uniform(0.5, 30.0, size=(Y, X)).astype(np.float32), device="cuda")
    init = rng.uniform(0.0, 1.0, size=(Z, Y, X)).astype(np.float32)
    outs, names = [], []
    for ctx in ctxs:
        vol = GPUMappedVolume(ctx, (X, Y, Z), [far - 32.0, -4.0, cz - 8.0], [far + 32.0, 4.0, cz + 8.0])
        bp = BackProjectionOperator(vol, 0.3, samples)
        bp.setScannerGeometry(g)
        bp.setInput(res, length, 1)

        def run():
            vol.upload(init)
            bp.execute()
        names.append(launched_back_projectors(run, 1))
        outs.append(vol.download())
        vol.close()
    assert np.abs(outs[0] - init).max() > 0
    assert np.array_equal(outs[1], outs[0])
    require_records(*names)
    assert names[0] == names[1]

