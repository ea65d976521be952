"""The SDF construct's two ways to its per-triangle jobs -- an array made beside the words' initialisation,
and each warp making its own (small meshes, and the build that allocates nothing) -- and its skipping of
cells a triangle cannot lower, bit for bit against the oracle: triangle counts on both sides of the rule
between the two, counts that are no multiple of the order's spread, boxes too large to be counted in
floats, degenerate triangles, and words that start within a few ulps of the result."""
import ctypes as C

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _grid(lo, cell, dims):
    from tressfx_gb300 import _capi as A
    g = A.SdfGrid()
    for k in range(3):
        g.origin[k] = float(lo[k])
    g.cell_size = float(cell)
    g.num_cells_x, g.num_cells_y, g.num_cells_z = (int(d) for d in dims)
    return g


def _mix(rng, n):
    """Small triangles, exact duplicates, slivers, points and segments."""
    a = rng.uniform(-0.1, 0.1, (n, 3))
    tri = a[:, None, :] + rng.normal(0, 0.004, (n, 3, 3))
    q = n // 8
    tri[q:2 * q] = tri[:q]
    t = rng.uniform(0, 1, (q, 1))
    tri[2 * q:3 * q, 2] = tri[2 * q:3 * q, 0] * (1 - t) + tri[2 * q:3 * q, 1] * t + rng.normal(0, 1e-7, (q, 3))
    tri[3 * q:3 * q + 5, 1:] = tri[3 * q:3 * q + 5, :1]
    tri[3 * q + 5:3 * q + 10, 2] = 0.5 * (tri[3 * q + 5:3 * q + 10, 0] + tri[3 * q + 5:3 * q + 10, 1])
    return tri


def _verts(tri):
    v = np.zeros((3 * len(tri), 8), np.float32)
    v[:, :3] = tri.astype(np.float32).reshape(-1, 3)
    return v, np.arange(3 * len(tri), dtype=np.uint32)


def _around(v, cells):
    p = v[:, :3]
    lo = p.min(0) - 0.015
    cell = np.float32((p.max(0) - p.min(0)).max() / cells)
    return _grid(lo, cell, np.ceil((p.max(0) + 0.015 - lo) / cell) + 1)


def _flip(f):
    u = f.view(np.uint32)
    return ((u << np.uint32(1)) | (u >> np.uint32(31))).astype(np.uint32)


def _build(ctx, v, idx, g, start=None, static=False):
    torch = pytest.importorskip("torch")
    from tressfx_gb300 import _capi as A
    from tressfx_gb300.api import SDFCollision
    cells = g.num_cells
    dv, di = torch.from_numpy(v.reshape(-1)).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    torch.cuda.synchronize()
    if static:
        out = torch.empty(cells, device="cuda")
        torch.cuda.synchronize()
        A.check(A.lib().tfx_sdf_build_static(ctx.handle, C.byref(g), dv.data_ptr(), len(v), di.data_ptr(), len(idx) // 3,
                                             out.data_ptr()), "tfx_sdf_build_static")
        ctx.synchronize()
        return out.cpu().numpy().view(np.uint32)
    sdf = SDFCollision(ctx, cells)
    try:
        sdf.set_mesh_device(dv.data_ptr(), len(v), di.data_ptr(), len(idx) // 3)
        if start is None:
            sdf.update(g)
        else:
            sdf.write(start)
            sdf.dispatch(A.K_SDF_CONSTRUCT, g)
        return sdf.read(cells)
    finally:
        sdf.close()


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("count", [1, 31, 3647, 3648, 3661, 9001])
def test_build_around_the_rule(ctx, count, static):
    rng = np.random.default_rng(count)
    v, idx = _verts(_mix(rng, count) if count > 100 else rng.uniform(-0.05, 0.05, (count, 3, 3)))
    g = _around(v, 44)
    got = _build(ctx, v, idx, g, static=static)
    want = oracle.sdf_build(g, v, idx)
    assert np.array_equal(got, want), f"{int((got != want).sum())} of {len(want)} cells differ"


def test_boxes_beyond_the_float_count(ctx):
    """Boxes of 2^20 cells and more, and cells whose offsets in a grid plane pass 2^23, are walked with
    integers and evaluated whole; small triangles share the grid with them."""
    rng = np.random.default_rng(5)
    tri = np.concatenate([_mix(rng, 4001), rng.uniform(-0.13, 0.13, (3, 3, 3))])
    v, idx = _verts(tri)
    g = _grid((-0.14, -0.14, -0.14), 0.28 / 112, (112, 112, 112))
    got, want = _build(ctx, v, idx, g), oracle.sdf_build(g, v, idx)
    assert np.array_equal(got, want), f"{int((got != want).sum())} cells differ"
    flat = _grid((-0.14, -0.14, -0.004), 0.28 / 2100, (2100, 2100, 3))   # few cells deep, 4.4M to a plane
    got, want = _build(ctx, v[:12000], idx[:12000], flat), oracle.sdf_build(flat, v[:12000], idx[:12000])
    assert np.array_equal(got, want), f"{int((got != want).sum())} cells differ"


@pytest.mark.parametrize("offset", [0.0, 40.0])
def test_job_array_from_words_near_its_result(ctx, offset):
    """Construct alone, on the job array, from words within a few ulps of the result with either sign."""
    rng = np.random.default_rng(int(offset) + 3)
    tri = _mix(rng, 5003) + np.array([offset, -0.5 * offset, 0.25 * offset])
    v, idx = _verts(tri)
    g = _around(v, 40)
    result = _flip(np.full(g.num_cells, 1e10, np.float32))
    oracle.sdf_construct(g, result, v, idx)
    mag = ((result >> np.uint32(1)) | (result << np.uint32(31))) & np.uint32(0x7FFFFFFF)
    mag = np.clip(mag.astype(np.int64) + rng.integers(-3, 4, len(mag)), 0, 0x7F7FFFFF).astype(np.uint32)
    start = _flip((mag | (rng.integers(0, 2, len(mag)).astype(np.uint32) << np.uint32(31))).view(np.float32))
    want = start.copy()
    oracle.sdf_construct(g, want, v, idx)
    assert int((want != start).sum()) > 0
    got = _build(ctx, v, idx, g, start=start)
    assert np.array_equal(got, want), f"{int((got != want).sum())} of {len(want)} cells differ"


def test_larger_mesh_after_a_smaller_one(ctx):
    """Binding a larger mesh to the same SDF takes a larger job array; the earlier one stays valid."""
    torch = pytest.importorskip("torch")
    from tressfx_gb300.api import SDFCollision
    rng = np.random.default_rng(9)
    meshes = [_verts(_mix(rng, n)) for n in (4000, 13001, 4000)]
    g = _around(meshes[1][0], 40)
    sdf = SDFCollision(ctx, g.num_cells)
    keep = []
    try:
        for v, idx in meshes:
            dv, di = torch.from_numpy(v.reshape(-1)).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
            keep += [dv, di]
            torch.cuda.synchronize()
            sdf.set_mesh_device(dv.data_ptr(), len(v), di.data_ptr(), len(idx) // 3)
            sdf.update(g)
            assert np.array_equal(sdf.read(g.num_cells), oracle.sdf_build(g, v, idx))
    finally:
        sdf.close()
