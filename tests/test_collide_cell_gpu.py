"""The collision from one cell's corners (the gradient's probes share them, divide in the short exact form and
hand what does not fit to the shader's own form), bit for bit against the oracle: grids with unset cells,
plateaus and signed zeros, vertices on cell faces, at zero coordinates, on the grid's last cells and
outside, cells near the coordinates' rounding, cell sizes outside the short form's range, and margins that
take in unset cells."""
from types import SimpleNamespace

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
G, N, F = 256, 16, 1
DIMS = (13, 11, 17)


def _grid(lo, cell):
    from tressfx_gb300 import _capi as A
    g = A.SdfGrid()
    for k in range(3):
        g.origin[k] = float(np.float32(lo[k]))
    g.cell_size = float(np.float32(cell))
    g.num_cells_x, g.num_cells_y, g.num_cells_z = DIMS
    return g


def _values(rng, kind, cell):
    z, y, x = np.meshgrid(*(np.arange(d) for d in DIMS[::-1]), indexing="ij")
    r = np.sqrt((x - 6.1) ** 2 + (y - 5.2) ** 2 + (z - 8.3) ** 2)
    d = ((r - 4.0) * cell).astype(np.float32)
    if kind == "unset":
        d[rng.random(d.shape) < 0.04] = np.float32(1e10)
    if kind == "flat":      # equal neighbours, zeros of both signs
        d = (np.round(d / np.float32(2 * cell)) * np.float32(2 * cell)).astype(np.float32)
        d[(d == 0) & (rng.random(d.shape) < 0.5)] = np.float32(-0.0)
    return d


CASES = {
    # name: origin, cell, margin in cells, grid values, vertices on cell faces
    "ordinary": ((-0.31, 0.07, 1.9), 0.037, 1.5, "smooth", False),
    "unset": ((-0.31, 0.07, 1.9), 0.037, 1.5, "unset", False),
    "faces": ((-0.25, -0.25, -0.25), 0.0625, 2.0, "smooth", True),
    "flat": ((-0.25, -0.25, -0.25), 0.0625, 2.0, "flat", True),
    "rounding": ((1000.0, -4000.0, 250.0), 1e-3, 2.0, "smooth", False),
    "tiny": ((0.0, 0.0, 0.0), 2.0 ** -38, 2.0, "smooth", False),
    "huge": ((0.0, 0.0, 0.0), 2.0 ** 41, 2.0, "smooth", False),
    "open": ((-0.31, 0.07, 1.9), 0.037, np.inf, "unset", False),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_collision_equals_oracle(ctx, case):
    from tressfx_gb300 import _capi as A
    from tressfx_gb300.api import HairObject, SDFCollision
    lo, cell, margin, kind, faces = CASES[case]
    rng = np.random.default_rng(sum(map(ord, case)))
    g = _grid(lo, cell)
    words = _values(rng, kind, cell).reshape(-1).view(np.uint32).copy()
    s, v = G * (F + 1), G * (F + 1) * N
    t = rng.uniform(-0.6, np.array(DIMS) + 0.6, (v, 3))
    t[::7, 0] = DIMS[0] - 2 - rng.uniform(0, 0.12, len(t[::7]))     # probes that leave the grid
    t[1::7, 2] = DIMS[2] - 2 - rng.uniform(0, 0.12, len(t[1::7]))
    if faces:
        t[::2] = np.round(t[::2])
        t[::3, 1] = np.round(t[::3, 1])
    pos = np.zeros((v, 4), np.float32)
    pos[:, :3] = (np.asarray(lo, np.float64) + t * cell).astype(np.float32)
    if faces:
        zero = rng.random((v, 3)) < 0.1
        pos[:, :3][zero] = np.where(rng.random(int(zero.sum())) < 0.5, np.float32(0.0), np.float32(-0.0))
    pos[:, 3] = rng.uniform(0, 2, v)
    prev = rng.normal(0, 1, (v, 4)).astype(np.float32)
    asset = SimpleNamespace(num_guide_strands=G, verts_per_strand=N, follow_per_guide=F, positions=pos, tangents=prev,
                            rest_lengths=np.ones(v, np.float32), follow_root_offsets=np.zeros((s, 4), np.float32),
                            bone_skinning=np.tile(np.array([0, 0, 0, 0, 1, 0, 0, 0], np.float32), (s, 1)))
    margin = margin if np.isinf(margin) else float(np.float32(margin * cell))
    ora = oracle.OracleHair(asset)
    ora.prev[...] = prev.reshape(ora.prev.shape)
    hair, sdf = HairObject(ctx, asset), SDFCollision(ctx, g.num_cells)
    hair.write(A.BUF_POSITIONS_PREV, prev)
    sdf.write(words)
    sdf.collide(hair, g, margin)
    oracle.sdf_collide(g, words, margin, ora)
    got = [hair.read(b).reshape(-1) for b in (A.BUF_POSITIONS, A.BUF_POSITIONS_PREV)]
    want = [np.ascontiguousarray(a, dtype=np.float32).reshape(-1) for a in (ora.pos, ora.prev)]
    sdf.close()
    moved = (want[0] != pos.reshape(-1)).any()
    assert moved, "no vertex collided"
    for a, b in zip(got, want):
        same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
        assert same.all(), f"{int((~same).sum())} of {same.size} words differ"
