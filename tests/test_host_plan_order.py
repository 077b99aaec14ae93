"""Which requests of a host step share memory (``ops.HostStepPlan`` orders those), on plain CPU tensors."""

import torch


def test_overlapping_requests_are_found():
    from liquidgemm_b200 import ops
    buf = torch.zeros(64, 8)
    x, y, z = buf[:4], buf[4:8], buf[8:12]
    other = torch.zeros(4, 8)
    assert ops._overlaps([(x, None, y), (x, None, z)]) == set()                    # a shared input is no conflict
    assert ops._overlaps([(x, None, y), (y, None, z)]) == {("yx", 0, 1)}
    assert ops._overlaps([(x, None, y), (buf[6:10], None, other)]) == {("yx", 0, 1)}   # a part of it
    assert ops._overlaps([(x, None, y), (z, None, x)]) == {("xy", 0, 1)}
    assert ops._overlaps([(x, None, y), (z, None, y)]) == {("yy", 0, 1)}
    assert ops._overlaps([(x, None, y), (y, None, x)]) == {("yx", 0, 1), ("xy", 0, 1)}
    assert ops._overlaps([(buf[:0], None, y), (z, None, buf[64:])]) == set()       # no bytes, no conflict
    assert ops._overlaps([(x, None, x)]) == set()                                  # a request in place is ordered by itself
