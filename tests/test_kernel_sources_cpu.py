"""What the kernels' sources have to keep to where no run on a GPU would show it."""
import glob
import os
import re

import pytest

from mindspeed_mm_b200.ops import build


def _kernels():
    """(file, name, body) of every kernel."""
    for path in sorted(glob.glob(os.path.join(build.CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s*(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth = end = 0
            for end in range(start, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            yield os.path.basename(path), m.group(1), text[start:end]


KERNELS = list(_kernels())
EARLY = {name for path in glob.glob(os.path.join(build.CSRC, "*.cu*")) for name in re.findall(r"launch_after(?:_if)?\((?:[^,()]*,\s*)?(\w+_kernel)\b", open(path).read())}


def test_the_sources_were_read():
    assert len(KERNELS) > 60 and {"fmha_bwd_dq_kernel", "fmha_fwd_alt_kernel", "gemv_rows_kernel"} <= EARLY
    assert {"gemm_kernel", "grouped_gemm_kernel", "gdn_fwd_kernel"} <= {name for _, name, _ in KERNELS}


@pytest.mark.parametrize("file,name,body", KERNELS, ids=[f"{f}:{n}" for f, n, _ in KERNELS])
def test_a_successor_is_let_start_when_it_can_do_no_harm(file, name, body):
    """Behind the wait, and behind the allocation of tensor memory: a successor that starts early takes its columns before it waits, and a
    block that it waits for could be left without."""
    trigger, wait, alloc = (body.find(w) for w in ("let_successor_start(", "wait_for_predecessor(", "tmem_alloc"))
    if name in EARLY or (file, name) == ("gemm.cu", "gemm_kernel"):
        assert wait >= 0
    if trigger >= 0:
        assert trigger > wait and trigger > alloc
