"""The multiply lane kernel with the product in an operand's place: the order of
its loads and stores, replayed, never reads a group after storing it, and its
loads do not go through the read-only path, which takes memory that the kernel
does not write."""
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _kernel():
    with open(os.path.join(ROOT, "xmp_b200", "csrc", "mul.cu")) as f:
        text = f.read()
    body = text[text.index("void __launch_bounds__(256) mul_lanes_kernel"):]
    return body[:body.index("\n}\n")]


def test_loads_are_plain_and_ordered():
    body = _kernel()
    assert "load_group_rw(a, ea" in body and "load_group_rw(b, eb" in body
    for read_only in ("__ldg", "load_group(", "load_limb(", "load_lane_limbs"):
        assert read_only not in body
    # every lane has passed its loads before lane 0 stores a group
    assert body.index("__syncwarp();") < body.index("store_group(c.limbs")


@pytest.mark.parametrize("L", [8, 12, 16])
@pytest.mark.parametrize("nb,nc", [(1, 33), (33, 33), (48, 48), (64, 64), (65, 96), (128, 128), (131, 512), (512, 512)])
def test_no_group_is_read_after_it_is_stored(L, nb, nc):
    stored = set()
    next_load = 0

    def load(g):
        nonlocal next_load
        assert g == next_load and g not in stored
        next_load += 1

    load(0)
    for base in range(0, nb, L):
        for m in range(L // 4):
            load(base // 4 + m + 1)
            if base + 4 * m < nc:
                stored.add(base // 4 + m)
    assert next_load * 4 >= nb
