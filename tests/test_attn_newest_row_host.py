"""The row of the newest token in a warp's shared memory is first filled with zeros by asynchronous copies, whose end a lane can only wait for where it issued
them itself.  So the lane that copied 16 bytes of that row is the one that writes the newest key or value there.  Read from the source, which lanes these are
is worked out here."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc", "attention.cu")


def _text():
    return re.sub(r"//[^\n]*", "", open(SOURCE).read())


def test_stores_follow_the_wait_of_the_copying_lane():
    stores = re.findall(r'cp\.async\.wait_group 1;"[^\n]*\n\s*if \(newest && ([^\n]*)\) store8\((sK|sV) \+ slot \* LD \+ (\w+) \* 8, load8\(sm\.fresh\[\d\] \+ (\w+) \* 8\)\);', _text())
    assert len(stores) == 2
    for lanes, _, unit, same in stores:
        assert lanes == "lane_row == slot % (32 / U)" and unit == same == "lane_unit"


@pytest.mark.parametrize("H", [64, 128])
def test_that_lane_is_the_copying_one(H):
    text = _text()
    assert "lane_row = lane / U, lane_unit = lane % U;" in text and "const int r = i * (32 / U);" in text and "(dst + (8 * e + r) * LD * 2)" in text
    assert "smem_u32(which ? sV : sK) + (lane_row * LD + lane_unit * 8) * 2" in text
    U, keys = H // 8, 2048 // H
    copied = {(8 * e + i * (32 // U) + lane // U, lane % U): lane for lane in range(32) for e in range(keys // 8) for i in range(U // 4)}
    assert len(copied) == keys * U
    for slot in range(keys):
        for lane in range(32):
            if lane // U == slot % (32 // U):
                assert copied[slot, lane % U] == lane
