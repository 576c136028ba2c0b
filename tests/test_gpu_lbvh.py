"""LBVH builds at the edges of their forms: one cluster's sort (1 to 16 blocks of 1, 2 or 4 keys a thread)
or the tiled one, the hierarchy's blocks of leaves; distributions whose nodes cross the blocks' borders,
equal codes, empty and NaN boxes.  Codes, order, nodes and boxes equal the oracle's."""
import numpy as np
import pytest

from raygun_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def boxes_of(kind, n):
    u = S.Rng(n + 3)
    if kind == "equal":
        return np.tile(np.array([[0, 0, 0, 1, 1, 1]], np.float32), (n, 1))
    if kind == "line":  # codes in input order: long runs share their leading bits
        c = np.zeros((n, 3))
        c[:, 0] = np.arange(n) * 0.25
    else:
        centre = u.uniform(96, 0, 100).reshape(32, 3)
        c = centre[(u.u64(n) % np.uint64(32)).astype(np.int64)] + u.normal(3 * n, 4.0).reshape(n, 3)
    h = u.uniform(3 * n, 0, 0.2).reshape(n, 3)
    b = np.concatenate([c - h, c + h], 1).astype(np.float32)
    if kind == "holes":
        b[::7, :3], b[::7, 3:] = np.inf, -np.inf
    return b


def unions(boxes, r):
    """The node boxes of a tree over boxes, children first (reverse of a pre-order walk)."""
    out = np.zeros_like(r["nodeboxes"])
    walk, stack = [], [0] if len(out) else []
    while stack:
        i = stack.pop()
        walk.append(i)
        stack += [int(c) for c in (r["left"][i], r["right"][i]) if not c >> 31]
    for i in reversed(walk):
        a, b = (boxes[r["order"][c & 0x7FFFFFFF]] if c >> 31 else out[c] for c in (int(r["left"][i]), int(r["right"][i])))
        out[i, :3], out[i, 3:] = np.minimum(a[:3], b[:3]), np.maximum(a[3:], b[3:])
    return out


@pytest.mark.parametrize("n", [1, 2, 3, 33, 511, 512, 513, 1024, 1025, 2049, 8193, 16384, 16385, 32768, 32769, 65535, 65536, 65537, 140001])
@pytest.mark.parametrize("kind", ["clusters", "line", "equal", "holes"])
def test_lbvh_equals_oracle(rg, orc, kind, n):
    boxes = boxes_of(kind, n)
    ctx = rg.Context()
    g = ctx.lbvh_build_host(boxes)
    ctx.close()
    empty = ~(boxes[:, 0] <= boxes[:, 3])
    r = orc.lbvh(np.where(empty[:, None], np.float32(0.0), boxes))  # empty boxes are keyed at the origin
    if empty.any():
        r["nodeboxes"] = unions(boxes, r)
    for k in ("morton", "order", "left", "right"):
        assert np.array_equal(g[k], r[k]), k
    assert g["nodeboxes"].tobytes() == r["nodeboxes"].tobytes()
