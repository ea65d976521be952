"""The SDF construct of meshes with few, large triangles: launches too small to fill the device evaluate every cell of
a triangle's box, larger ones without a job array test them.  Boxes with their faces along the grid's axes, so that
whole planes of cells have numerators of exactly zero (on the grid's points and between them), a box that is not
narrow (2^20 cells or more of a triangle), and heads on both sides of the line of 24 triangles an SM -- through the
plain build, the allocation-free build and a batch, against the oracle bit for bit."""
import ctypes as C

import numpy as np
import pytest

import oracle
from tressfx_gb300 import _capi as A
from tressfx_gb300.api import Batch, CollisionMesh, HairObject, SDFCollision
from tressfx_gb300.synthetic import head_mesh, scene_small

pytestmark = pytest.mark.gpu


def box(n, half=0.1):
    """The surface of a cube around the origin, n x n squares of two triangles a face."""
    v, t = [], []
    for axis in range(3):
        for side in (-half, half):
            first = len(v)
            for i in range(n + 1):
                for j in range(n + 1):
                    p = [0.0, 0.0, 0.0]
                    p[axis], p[(axis + 1) % 3], p[(axis + 2) % 3] = side, 2 * half * i / n - half, 2 * half * j / n - half
                    v.append(p)
            for i in range(n):
                for j in range(n):
                    k = first + i * (n + 1) + j
                    t += [k, k + 1, k + n + 1, k + 1, k + n + 2, k + n + 1]
    verts = np.zeros((len(v), 8), np.float32)
    verts[:, :3] = v
    verts[:, 5] = 1.0
    skin = np.zeros((len(v), 8), np.float32)
    skin[:, 4] = 1.0
    return verts, np.array(t, np.uint32), skin


def diagonal(half=0.1):
    """Two triangles across the cube: their boxes are the whole grid's."""
    verts = np.zeros((4, 8), np.float32)
    verts[:, :3] = np.array([[-1, -1, -1], [1, 1, -1], [1, -1, 1], [-1, 1, 1]], np.float32) * half
    verts[:, 5] = 1.0
    skin = np.zeros((4, 8), np.float32)
    skin[:, 4] = 1.0
    return verts, np.array([0, 1, 2, 0, 2, 3], np.uint32), skin


def grid(lo, hi, dim, margin=2.5):
    g = A.SdfGrid()
    g.cell_size = float(np.float32((hi - lo).max() / (dim - 2 * margin)))
    for k in range(3):
        g.origin[k] = float(np.float32(lo[k]) - np.float32(margin) * np.float32(g.cell_size))
    g.num_cells_x = g.num_cells_y = g.num_cells_z = dim
    return g


def cases():
    for n, dim, margin in ((1, 16, 2.0), (1, 33, 2.5), (1, 132, 2.0), (2, 40, 4.0), (5, 64, 2.0), (18, 64, 5.0)):
        yield f"box {12 * n * n} in {dim}", box(n), dim, margin
    for dim in (96, 110):   # boxes of fewer than 2^20 cells, and of more
        yield f"diagonal in {dim}", diagonal(), dim, 2.0
    for tris in (300, 3300, 4500):
        m = head_mesh(tris)
        yield f"head {len(m.indices) // 3} in 48", (m.vertices, m.indices, m.skinning), 48, 2.5


@pytest.mark.parametrize("name,mesh,dim,margin", list(cases()), ids=[c[0] for c in cases()])
def test_build_equals_oracle(ctx, name, mesh, dim, margin):
    verts, indices, skin = mesh
    p = verts[:, :3]
    g = grid(p.min(0), p.max(0), dim, margin)
    cells = dim ** 3
    one = np.tile(np.eye(4, dtype=np.float32).reshape(1, 16), (8, 1))
    m = CollisionMesh(ctx, verts, indices, skin)
    m.skin(one)
    want = oracle.sdf_build(g, m.read_skinned().reshape(-1, 8), indices)
    assert (want.view(np.float32) < 1e10).sum() > 200
    sdf = SDFCollision(ctx, cells)
    sdf.bind_mesh(m)
    sdf.update(g)
    got = sdf.read(cells).view(np.uint32)
    assert np.array_equal(got, want), f"plain: {int((got != want).sum())} of {cells} cells differ"

    out = SDFCollision(ctx, cells)
    ptr = C.c_void_p()
    assert A.lib().tfx_sdf_get_buffer(out.handle, C.byref(ptr), None) == 0
    if cells <= 2097152:
        st = A.lib().tfx_sdf_build_static(ctx.handle, C.byref(g), C.c_void_p(m.skinned_ptr), m.num_vertices,
                                          C.c_void_p(m.index_ptr), m.num_triangles, ptr)
        assert st == 0, A.lib().tfx_last_error()
        got = out.read(cells).view(np.uint32)
        assert np.array_equal(got, want), f"static: {int((got != want).sum())} of {cells} cells differ"

    sc = scene_small(num_guides=64, n=8)
    hair = HairObject(ctx, sc.objects[0].asset)
    b = Batch(ctx)
    b.add_sdf(sdf, m, (dim, dim, dim))
    b.add_hair(hair, 0)
    b.build()
    from tressfx_gb300.headless import FrameInputs
    fin = FrameInputs(sc, 0)
    hair.update_simulation_parameters(fin.settings[0], sc.dt)
    hair.update_bone_matrices(fin.hair_bones[0])
    b.set_hair_constants(0, hair.current_params(), hair.num_bones, hair.cpu_local_iterations)
    b.set_sdf_frame(0, g, 0.0)
    b.set_mesh_bones(0, one)
    for block in (64, 128, 256):
        b.set_option(b.SDF_BLOCK, block)
        sdf.write(np.zeros(cells, np.uint32))
        b.run()
        b.synchronize()
        got = sdf.read(cells).view(np.uint32)
        assert np.array_equal(got, want), f"batch, blocks of {block}: {int((got != want).sum())} of {cells} cells differ"
    for x in (b, hair, sdf, out, m):
        x.close()
