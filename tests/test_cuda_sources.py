"""Rules that the CUDA sources keep and that no run can be relied on to show."""
import re
from pathlib import Path

import pytest

GPU = Path(__file__).resolve().parent.parent / "csrc" / "gpu"


def _kernels():
    """(file, name, body) of every kernel."""
    for path in sorted(GPU.rglob("*.cu*")):
        text = re.sub(r"//[^\n]*|__(launch_bounds|cluster_dims)__\s*\([^()]*\)", "", path.read_text())
        for m in re.finditer(r"__global__[^{;]*?(\w+)\s*\([^{;]*\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield path.name, m.group(1), text[m.end():end]


@pytest.mark.parametrize("kernel", [k for k in _kernels() if "st_cluster_" in k[2]], ids=lambda k: f"{k[0]}:{k[1]}")
def test_other_blocks_shared_memory_is_written_between_cluster_barriers(kernel):
    """A block's shared memory may be written by others once it runs and until it ends: a cluster barrier lies in front of the first
    remote store and one behind the last."""
    body = kernel[2]
    barriers = [m.start() for m in re.finditer(r"\bcluster_(sync_all|wait)\(", body)]
    stores = [m.start() for m in re.finditer(r"\bst_cluster_\w+\(", body)]
    assert barriers and barriers[0] < stores[0] and barriers[-1] > stores[-1]


def test_the_kernels_with_remote_stores_are_found():
    names = {k[1] for k in _kernels() if "st_cluster_" in k[2]}
    assert {"route_one_launch_kernel", "gemm_small_kernel", "gemm2sm_kernel"} <= names


@pytest.mark.parametrize("kernel", [k for k in _kernels() if "tmem_ld_32x" in k[2]], ids=lambda k: f"{k[0]}:{k[1]}")
def test_warps_that_read_accumulators_give_up_together(kernel):
    """Another role's failure is seen lane by lane: a warp that goes on with instructions of whole warps asks for all of its lanes."""
    epilogue = kernel[2][kernel[2].index("const int q = warp & 3"):]
    assert "!*abort_flag" not in epilogue and not re.search(r"\bmbar_wait\(", epilogue)
    assert "mbar_wait(&tfull" not in kernel[2] and "mbar_wait(tfull" not in kernel[2]
