"""Tensor memory is read and written by the tensor core out of the threads' order: an access behind a barrier on which its
MMAs (or another warp's accesses) were waited for needs ``tcgen05.fence::after_thread_sync`` between the two, stores that
overwrite an operand as well as loads and MMAs.  No run can show a missing fence for sure; the text of the kernels can."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "boostr_b200", "csrc")
EVENT = re.compile(r"(?<!\w)(?P<wait>(?:i8_wait|pf_wait|mbar_wait|wait|wait_cluster|take)\()|(?P<fence>tc_(?:fence_)?after\(\)|tcgen05\.fence::after_thread_sync)"
                   r"|(?P<access>tmem_st\d+\(|tmem_ld\d+(?:_async)?\(|tc_mma_\w+\(|mma_\w+_ts\()")


def _unfenced(text):
    """Line numbers of accesses whose last wait before them has no fence behind it (in the order of the text, kernel by kernel)."""
    bad = []
    start = text.find("__global__")
    while start >= 0:
        end = text.find("__global__", start + 1)
        fenced = False
        for m in EVENT.finditer(text, start, end if end >= 0 else len(text)):
            if m["access"]:
                if not fenced:
                    bad.append(text.count("\n", 0, m.start()) + 1)
            else:
                fenced = m["fence"] is not None
        start = end
    return bad


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu"))))
def test_accesses_are_fenced_behind_waits(name):
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert _unfenced(text) == []
