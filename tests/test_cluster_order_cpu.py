"""Thread-block clusters: a block's shared memory may be touched by its neighbours only once it is known to run, which takes a
cluster barrier that all blocks have passed (griddepcontrol.wait orders against earlier grids, not against the blocks of this one).
Read from the sources: in every kernel the first access to another block's shared memory stands behind such a barrier."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rusty_b200", "csrc")
REMOTE = re.compile(r"\b(st_cluster_u32|mapa_u32|map_shared_rank)\s*\(")
PASSED = re.compile(r"\b(cluster_sync_all|cluster_wait|cl\.sync|barrier_wait)\s*\(")


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        text = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text)
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\((?=[^;{]*\)\s*\{)", text):
            start = text.index("{", m.end())
            depth, at = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
                if depth == 0:
                    break
            yield os.path.basename(path), m.group(1), text[start:at]


ACCESSING = [(f, name, body) for f, name, body in _kernels() if REMOTE.search(body)]


def test_the_kernels_are_found():
    names = {name for _, name, _ in ACCESSING}
    assert {"digitize_x_kernel", "qlinear_i8_tc_kernel", "qlinear_gc_tc_kernel", "qlinear_gc_wide_kernel", "logits_rows_kernel",
            "argmax_rows_kernel", "gemv_affine_kernel"} <= names


@pytest.mark.parametrize("file,name,body", ACCESSING, ids=[n for _, n, _ in ACCESSING])
def test_no_remote_access_before_the_blocks_have_met(file, name, body):
    met = PASSED.search(body)
    assert met is not None and met.start() < REMOTE.search(body).start(), f"{file}: {name}"
