"""Kernels that are let in while the launch before them still writes (tfx_launch.cuh) read what a launch may write
after their wait and by plain loads.  A load by __ldg or through a `const ... __restrict__` parameter of the
kernel promises that the words stay as they are for the kernel's whole lifetime, which here overlaps the
producer's, and leaves the compiler free to move it above the wait; what is read before the wait has no promise
of being visible.  No run can show either as long as a compiler's schedule happens to be kind, so this reads the
sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tressfx_gb300" / "csrc"
# what no launch writes: a batch's tables and the training samples (parameters), and a batch's bind poses, skin
# weights, rest data and indices (the argument of __ldg)
CONSTANT_PARAMETERS = {"objs", "items", "sdfs", "meshes", "expSdf", "expFirst", "pool"}
CONSTANT_LOADS = ("h.init", "h.skin", "h.rest", "init ", "m.bind", "m.skin", "s.indices", "expFirst", "expSdf")


def block(text, start, pair):
    """text[start..] from its first pair[0] to the matching pair[1], and the index behind it."""
    i = text.index(pair[0], start)
    depth, k = 0, i
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[k], 0)
        k += 1
        if depth == 0:
            return text[i:k], k


def kernels(text):
    """(name, parameters, body, begin, end) of every kernel defined in a source."""
    for m in re.finditer(r"__global__", text):
        n = re.compile(r"\b(k_\w+)\s*\(").search(text, m.end())
        params, at = block(text, n.end() - 1, "()")
        if text[at:].lstrip()[:1] != "{":
            continue
        body, end = block(text, at, "{}")
        yield n.group(1), params, body, m.start(), end


def source(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


FILES = sorted(p for p in CSRC.glob("*.cu") if "after_previous()" in p.read_text())
DEPENDENT = [(p.name, k) for p in FILES for k in kernels(source(p)) if "after_previous()" in k[2]]


def test_sources_are_found():
    assert len(DEPENDENT) >= 20 and {"k_fused_strands", "k_nsdf_adam", "k_sdf_collide", "k_batch_sdf_jobs"} <= {k[0] for _, k in DEPENDENT}


@pytest.mark.parametrize("file,kernel", DEPENDENT, ids=[k[0] for _, k in DEPENDENT])
def test_kernel_reads_by_plain_loads_behind_its_wait(file, kernel):
    name, params, body, _, _ = kernel
    assert "ReadOnlyLoad" not in body
    readonly = set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params))
    assert readonly <= CONSTANT_PARAMETERS, (file, name, readonly - CONSTANT_PARAMETERS)
    assert not re.search(r"const\s+[\w:]+\s*\*\s*__restrict__\s+\w+\s*=", body), (file, name)
    before = body[:body.index("after_previous()")]
    for p in re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)\s*[,)]", params):
        if p not in CONSTANT_PARAMETERS:
            assert not re.search(rf"(?<![\w.]){p}\s*\[|\*\s*{p}\b(?!\s*[,)])|{p}->", before), (file, name, p)


@pytest.mark.parametrize("path", FILES + [CSRC / "tfx_device_math.cuh", CSRC / "tfx_sdf_math.cuh"], ids=lambda p: p.name)
def test_read_only_loads_are_of_constants(path):
    text = source(path)
    for name, _, body, begin, end in reversed(list(kernels(text))):
        if "after_previous()" not in body:   # launched plainly
            text = text[:begin] + text[end:]
    for plain in ("struct ReadOnlyLoad", "struct GroupCorners"):   # used by kernels launched plainly alone
        if plain in text:
            _, end = block(text, text.index(plain), "{}")
            text = text[:text.index(plain)] + text[end:]
    loads = re.findall(r"__ldg\(([^;]*)", text)
    bad = [a for a in loads if not a.startswith(CONSTANT_LOADS)]
    assert not bad, bad
