"""The contraction kernels' waits are bounded; no warp may then wait for one that gave up.
Such a hang is not provoked on a GPU, so this looks at the kernels' text: the draining
warps meet at no named barrier, and a warp's lanes leave a wait with one outcome (the
TMEM loads after it are warp-collective)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scp3_b200", "csrc")


@pytest.mark.parametrize("name,kernel", [("contract_i8.cu", "contract_i8_kernel"), ("contract_tc.cu", "contract_n256_kernel")])
def test_draining_warps(name, kernel):
    text = open(os.path.join(CSRC, name)).read()
    body = text[text.index(" " + kernel + "("):]
    body = body[:body.index("\n}\n")]
    assert "tcgen05.dealloc" in body
    assert "bar.sync" not in body and "barrier.sync" not in body
    drain = body[body.index("mma_commit(drain)"):]
    waits = re.findall(r"if \(!(.*?)mbar_wait\(acc_full", drain)
    assert waits and all("__all_sync" in w for w in waits)
