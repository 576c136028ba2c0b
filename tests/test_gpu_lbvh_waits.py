"""LBVH hierarchy: node boxes taken from the leaves, as after a sibling's box that did not arrive
(RG_HIER_POLL_LIMIT=0 takes every box of another block's node that way), are the climb's, byte for byte."""
import numpy as np
import pytest

from test_gpu_lbvh import boxes_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 513, 1025, 8193, 65537, 140001])
@pytest.mark.parametrize("kind", ["clusters", "line", "equal", "holes", "nan"])
def test_boxes_from_the_leaves(rg, monkeypatch, kind, n):
    boxes = boxes_of("line" if kind == "nan" else kind, n)
    if kind == "nan":  # whole subtrees without a number, and single corners
        boxes[n // 4:n // 2] = np.nan
        boxes[::5, 4] = np.nan
    ctx = rg.Context()
    want = ctx.lbvh_build_host(boxes)
    monkeypatch.setenv("RG_HIER_POLL_LIMIT", "0")
    got = ctx.lbvh_build_host(boxes)
    ctx.close()
    for k in ("morton", "order", "left", "right", "nodeboxes"):
        assert got[k].tobytes() == want[k].tobytes(), k
