"""k_follow_collide on whole strand groups: a class with at least four groups for every resident block (155,648 strands
on GB300) is not cut into chunks, and no other test has so many strands with follow hairs.  A partial last group,
one and two follow hairs, groups of 32 x 8 and 32 x 4 vertices, with corner-expanded grids and without, against the
oracle bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,guides,follows,expand", [(8, 156001, 1, 0), (8, 156001, 1, 1), (4, 160007, 2, 2)])
def test_whole_groups_with_follow_hairs(ctx, n, guides, follows, expand):
    from oracle.scene_driver import OraclePipeline
    from test_batched_gpu import assert_same
    from tressfx_gb300.headless import BatchedPipeline
    from tressfx_gb300.synthetic import scene_head
    sc = scene_head(seed=5 + n, num_guides=guides, n=n, follows=follows, triangles=1500, sdf_cells=32, frames=4)
    gpu = BatchedPipeline(ctx, sc)
    try:
        gpu.batch.set_option(gpu.batch.EXPANDED_GRIDS, expand)
        ora = OraclePipeline(sc)
        for f in range(4):
            fin = gpu.step(f)
            ora.step(fin)
        assert_same(gpu.hair[0], ora.hair[0], f"n={n} follows={follows} expand={expand}")
    finally:
        gpu.close()
