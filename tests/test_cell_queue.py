"""The SDF construct's queue of cells to evaluate, run on host threads that record which entries the lanes touch
between two warp synchronisations: no cell lost or doubled, and no unordered accesses to one entry."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_lanes_touch_an_entry_in_order(tmp_path):
    from tressfx_gb300 import build as B
    exe = tmp_path / "cell_queue"
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", f"-I{ROOT / 'tressfx_gb300' / 'csrc'}",
                    f"-I{B._cuda_home() / 'include'}", str(ROOT / "tests" / "cpp" / "cell_queue.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300).stdout.split()
    assert out == ["0", "0"], f"cells lost or doubled: {out[0]}, unordered accesses: {out[1]}"
