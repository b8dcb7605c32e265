"""Barriers of warps with different roles: __syncthreads() asks that all threads of the block come to the same one."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lapis_b200", "csrc")


def test_long_row_roles_meet_at_a_counted_barrier():
    """spmm_long_kernel: feeders and adders are the two branches of one if; each meets the other once a tile."""
    with open(os.path.join(CSRC, "spmm.cu")) as f:
        text = f.read()
    roles = text[text.index("if (feeder >= 0) {"):]
    roles = re.split(r"\n    if \(end\) break;", roles)[0]
    assert "__syncthreads" not in roles
    assert roles.count("tile_barrier();") == 3  # two tiles a turn of the feeders' loop, one of the adders'
    assert 'asm volatile("barrier.sync 1, %0;" ::"n"(SPMM_LONG_THREADS) : "memory");' in text
