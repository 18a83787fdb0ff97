"""Rules of the tensor-core kernels that only their source shows: a run that broke them would need a wait to
run out."""
import glob
import os
import re

import pytest

from conftest import PKG


def _kernels():
    """(file, name, body) of every kernel that owns tensor memory."""
    for f in sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu"))):
        for part in re.split(r"(?=__global__ void)", open(f).read())[1:]:
            body = part[: part.index("\n}\n")]
            if "tcgen05.alloc" in body:
                name = re.search(r"(\w+)\s*\(BlockSource|(\w+)\s*\(const float\*", body)
                yield os.path.basename(f), next(g for g in name.groups() if g), body


@pytest.mark.parametrize("file,name,body", [pytest.param(*k, id=k[1]) for k in _kernels()])
def test_tensor_memory_is_released_behind_the_issuing_lane(file, name, body):
    """tcgen05.commit covers the MMAs of the thread that issues it, so the elected lane (the same one at every election of
    a whole warp) issues every MMA and every commit, the one before the release of tensor memory included."""
    assert not re.search(r"umma_(commit|bf16|tf32)\(", body)
    assert set(re.findall(r"umma_\w+_by\((\w+)", body)) == {"leader", "elect_one"}
    assert set(re.findall(r"leader = ([^;]+);", body)) == {"elect_one()"}
    last = [m.start() for m in re.finditer(r"umma_commit_by\(elect_one\(\),", body)][-1]
    assert body.rindex("umma_") == last < body.index("tcgen05.dealloc")


def test_every_kernel_with_tensor_memory_is_looked_at():
    assert [k[1] for k in _kernels()] == ["conv3d_tc_kernel", "conv3d_run_kernel", "conv3d_wgrad_tc_kernel",
                                          "llr_gram_tc_kernel"]
