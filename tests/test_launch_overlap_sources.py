"""Kernels that become resident while the launch in front of them still writes (launch_pdl): what that launch may be writing
does not come by the read-only path, which const __restrict__ pointers ask for (common.h).  A stale read cannot be provoked,
so the sources are looked at."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lapis_b200", "csrc")


@pytest.mark.parametrize("source,function,constant", [
    ("pcg.cu", "mht_piece", {"crd", "val", "mask"}),
    ("pcg.cu", "mht_row", {"crd", "val", "mask"}),
    ("pcg.cu", "mht_rows", {"pos", "crd", "val", "d", "mask"}),
    ("pcg.cu", "mht_operator_kernel", {"pos", "crd", "val", "d", "mask"}),
    ("pcg.cu", "mht_residual_kernel", {"d"}),
    ("gemm_split.cu", "split_kernel", set()),
])
def test_read_only_path_is_for_what_stays(source, function, constant):
    """`constant`: what no kernel of the solve writes."""
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    heads = re.findall(r"\b%s\(([^;{]*)\)\s*\{" % function, text)
    assert len(heads) == 1, function
    body = text[text.index(heads[0]):]
    body = body[:body.index("\n}\n")]
    read_only = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", body))
    assert read_only == constant
    assert "__ldg" not in body
