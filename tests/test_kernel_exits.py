"""A block of a tcgen05 product whose bounded wait ran out leaves through the common exit.  No wait can be made to run out without a
fault, so this reads the source: every role that sends for copies or issues products waits for them before that exit."""
import os
import re

import pytest

from mashbox_b200.ops.build import CSRC


@pytest.mark.parametrize("source", ["gemm_f32_tc5.cu", "gemm_experts.cu"])
def test_roles_wait_for_what_they_sent_for(source):
    text = open(os.path.join(CSRC, source)).read()
    text = text[:text.index("// common exit")]
    body = text[text.rindex("__global__"):]
    roles = re.split(r"\n {4,8}(?:\} else )?if \(warp (?:<|==|>=)", body)
    sends = [r for r in roles if re.search(r"tma_load_2d\(", r)]
    issues = [r for r in roles if re.search(r"umma_f16(_warp)?\(", r)]
    assert sends and issues
    for r in sends:
        assert r.rindex("copies_landed(") > r.rindex("tma_load_2d(")
    for r in issues:
        assert r.rindex("products_landed<") > r.rindex("umma_f16")
