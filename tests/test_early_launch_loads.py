"""Kernels that are placed while the ones before them still run (launch.cuh) read
what those write with plain loads only: read-only loads are for memory that
nothing writes while the kernel exists.  Read from the sources, on the CPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nbodysimulation_gb300", "csrc")
READ_ONLY = re.compile(r"__ldg\s*\(|__restrict__|ld\.global\.nc")


def source(path):
    with open(path) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def kernels(text):
    """(name, text) of every __global__ function, its parameters and its body."""
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        at = text.index("{", m.end())
        depth = 0
        for end in range(at, len(text)):
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            if depth == 0:
                break
        yield m.group(1), text[m.start():end + 1]


def test_early_kernels_use_plain_loads():
    found = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for name, body in kernels(source(path)):
            found[name] = body
    early = {name for name, body in found.items() if "wait_for_previous()" in body}
    assert {"k_direct", "k_force", "k_path", "k_cells", "k_link", "k_top", "k_grid_rest", "k_batch_link"} <= early
    for name in sorted(early):
        assert not READ_ONLY.search(found[name]), name


def test_device_functions_use_plain_loads():
    for path in sorted(glob.glob(os.path.join(CSRC, "*_device.cuh"))):
        assert not READ_ONLY.search(source(path)), os.path.basename(path)


def test_only_kernels_that_wait_are_launched_early():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = source(path)
        bodies = dict(kernels(text))
        for m in re.finditer(r"launch_next(?:_shared)?\(\s*(k_\w+)", text):
            assert re.search(r"\{\s*wait_for_previous\(\);", bodies[m.group(1)]), m.group(1)
