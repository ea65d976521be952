"""What the host side launches, and what it does when device memory runs out: the library's own objects linked
against a stand-in for the CUDA runtime (tests/cpp/fake_cudart.cpp), on the CPU."""
import os
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from tressfx_gb300 import build as B
    B.build()
    out = tmp_path_factory.mktemp("fake") / "libfake.so"
    objects = sorted(B.BUILD_DIR / (s.name + ".o") for s in B._sources())
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{B._cuda_home() / 'include'}",
                    str(ROOT / "tests" / "cpp" / "fake_cudart.cpp"), *map(str, objects), "-Wl,-Bsymbolic", "-Wl,--no-undefined",
                    "-lpthread", "-ldl", "-lrt", "-o", str(out)], check=True)
    return out


PRELUDE = """
import ctypes as C, sys
from pathlib import Path
from tressfx_gb300 import _capi as A
A.LIB_PATH = Path(sys.argv[1])
from tressfx_gb300.api import Batch, Context
from tressfx_gb300.headless import BatchedPipeline, FrameInputs
from tressfx_gb300.synthetic import scene_head
L = A.lib()
L.fake_launches.restype = C.c_char_p
L.fake_malloc_limit.argtypes = [C.c_size_t]
def launches():
    rows = [r.split() for r in L.fake_launches().decode().splitlines()]
    L.fake_forget()
    return [(r[0], int(r[1]), int(r[2])) for r in rows]
def named(rows, part):   # their block sizes
    return {r[2] for r in rows if part in r[0]}
def batch(triangles):
    return BatchedPipeline(Context(0), scene_head(seed=7, num_guides=64, n=16, follows=1, triangles=triangles, sdf_cells=32, frames=1))
"""


def run(fake, code, **more):
    env = dict(os.environ, PYTHONPATH=str(ROOT), **more)
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code), str(fake)], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_batch_builds_without_its_job_array(fake):
    """A batch whose job array (256 bytes a triangle) cannot be had builds, and makes its jobs in shared memory."""
    run(fake, """
    p = batch(6000)
    rows = launches()
    assert named(rows, "k_batch_sdf_jobs") and not named(rows, "construct_chunks")
    p.close()
    whole = Batch.build
    def build(self):   # the objects are there; what the batch asks for from 1 MB on fails (its job array takes 1.5)
        L.fake_malloc_limit(1 << 20)
        whole(self)
    Batch.build = build
    p = batch(6000)
    rows = launches()
    assert named(rows, "construct_chunks") and not named(rows, "k_batch_sdf_jobs")
    p.step(0)
    p.close()
    """)


@pytest.mark.parametrize("triangles,kernel", [(1500, "construct_chunks"), (6000, "k_batch_sdf_construct")])
def test_sdf_block_is_the_construct_block(fake, triangles, kernel):
    """TFX_BATCH_SDF_BLOCK is the block size of the construct, with a job array and without."""
    run(fake, f"""
    p = batch({triangles})
    assert named(launches(), "{kernel}") == {{128}}
    for threads in (64, 256, 128):
        p.batch.set_option(Batch.SDF_BLOCK, threads)
        rows = launches()
        assert named(rows, "{kernel}") == {{threads}}, rows
        warps = max(b * t // 32 for n, b, t in rows if "{kernel}" in n)
        assert warps >= {triangles} // 16
    p.close()
    """)


def test_objects_may_go_before_the_batch(fake):
    """Destroying a batch reads nothing of the objects that it held, which a program may have destroyed before it
    (freed memory is overwritten here, so that reading it shows)."""
    run(fake, """
    p = batch(1500)
    for x in p.hair + p.sdfs + p.meshes:
        x.close()
    p.batch.close()
    """, MALLOC_PERTURB_="165", GLIBC_TUNABLES="glibc.malloc.tcache_count=0")
