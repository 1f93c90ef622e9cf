"""Level2 normals by runs of voxels where they can go wrong: grids with enough voxels for runs of several,
sub-grids whose outputs are not 16-byte (or 4-byte) aligned, several triangles on one cell in a batch, and
batches whose runs are cut where the mesh changes.  Sums run in list order, so every value equals the
oracle's; bytes are the encoding of the floats."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _check(ctx, res, tris, spec, mode, gpv):
    ref = orc.Run(tris, spec, fill=orc.FILL_CAND)
    l1, _, bi, l2 = ctx.fetch(res)
    np.testing.assert_array_equal(bi, ref.boundary_index())
    n1, n2 = ctx.fetch_normals(res)
    w1, w2 = ref.level1_normals(), ref.level2_normals() if spec.ndiv2[0] else None
    if mode == gpv.NORMALS_BYTES:
        w1, w2 = orc.normal_bytes(w1), None if w2 is None else orc.normal_bytes(w2)
    np.testing.assert_array_equal(n1, w1)
    if w2 is not None:
        np.testing.assert_array_equal(l2, ref.level2_bytes())
        np.testing.assert_array_equal(n2, w2)
    return len(bi)


@pytest.mark.parametrize("n2", [(2, 2, 2), (3, 3, 3), (5, 1, 7), (8, 8, 8), (1, 1, 1)])
@pytest.mark.parametrize("mode", ["float", "bytes"])
def test_many_voxels(ctx, built, n2, mode):
    gpv = built
    mode = gpv.NORMALS_FLOAT if mode == "float" else gpv.NORMALS_BYTES
    tris = gpv.gen_torus(5, 300, 150, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004)
    mn, mx = gpv.mesh_bounds(tris)
    spec = gpv.grid_padded(mn, mx, (110, 100, 70), n2)
    ctx.set_normals(mode)
    try:
        res = ctx.voxelize_host(tris, spec)
        assert _check(ctx, res, tris, spec, mode, gpv) > 20000
        ctx.release(res)
    finally:
        ctx.set_normals(gpv.NORMALS_OFF)


@pytest.mark.parametrize("mode", ["float", "bytes"])
def test_runs_end_with_their_mesh(ctx, built, mode):
    import torch

    gpv = built
    mode = gpv.NORMALS_FLOAT if mode == "float" else gpv.NORMALS_BYTES
    meshes = []
    for k in range(9):
        tris = gpv.gen_torus(k, 160 + k, 90, (0.5, 0.5, 0.5), 0.35, 0.12, 0.004)
        mn, mx = gpv.mesh_bounds(tris)
        n2 = [(3, 3, 3), (2, 3, 1), (4, 4, 4), (0, 0, 0), (5, 5, 5)][k % 5]
        meshes.append((tris, gpv.grid_padded(mn, mx, (61 + k, 60, 40) if k != 6 else (3, 3, 3), n2)))
    dev = [torch.from_numpy(t).cuda() for t, _ in meshes]
    ctx.set_normals(mode)
    try:
        rs = ctx.voxelize_batch([d.data_ptr() for d in dev], [d.numel() // 9 for d in dev], [s for _, s in meshes])
        assert sum(_check(ctx, r, t, s, mode, gpv) for (t, s), r in zip(meshes, rs)) > 20000
        for r in rs:
            ctx.release(r)
    finally:
        ctx.set_normals(gpv.NORMALS_OFF)
