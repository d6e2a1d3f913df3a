"""vlxb_fockBuild declines builds whose shared preparations would not leave room
on the device: it says so before it touches the device (no GPU needed here)."""
import pytest

from vlxb._lib import VlxbFockBuild, lib


@pytest.mark.parametrize("l,j,k", [(0, [], ["ssss"]), (1, [], ["pppp"]), (2, [], ["dddd"]), (0, ["ssss"], [])])
def test_large_builds_go_class_by_class(l, j, k):
    b = VlxbFockBuild()
    for t in range(3):
        b.prim_count[t] = 1 if t != l else 80000
    assert not lib().fock_build(b, j, k, 0)
