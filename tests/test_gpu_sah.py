"""Binned-SAH builds at the edges of their forms (two primitives, a warp's subtree, one CTA with its
primitives in shared memory, level kernels, several CTAs a task) over distributions that steer the binning:
scattered and clustered triangles, a lattice full of equal costs, coincident ones, chains that peel.
The tree is the oracle's."""
import numpy as np
import pytest

from raygun_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def soup(kind, n):
    u = S.Rng(n + 17)
    if kind == "lattice":
        s = int(np.ceil(n ** (1 / 3)))
        k = np.arange(n)
        c = np.stack([k % s, k // s % s, k // (s * s)], 1).astype(np.float64)
    elif kind == "same":
        c = np.zeros((n, 3))
    elif kind == "chain":  # a surface-area split peels a few off the far end
        c = np.zeros((n, 3))
        c[:, 0] = 1.07 ** (np.arange(n) % 400)
    else:
        centre = u.uniform(48, 0, 60).reshape(16, 3)
        c = centre[(np.arange(n) * 16 // n)] + u.normal(3 * n, 2.0).reshape(n, 3)  # runs of neighbours, as in a mesh
    d = np.array([[0, 0, 0], [0.4, 0, 0.1], [0.1, 0.3, 0.2]])
    if kind == "clusters":
        d = d[None] * (0.5 + u.uniform(n)[:, None, None])
    return (c[:, None, :] + d).astype(np.float32)


@pytest.mark.parametrize("n", [2, 3, 4, 16, 17, 32, 33, 64, 65, 255, 1023, 1025, 4096, 4097, 32767, 32768, 70001])
@pytest.mark.parametrize("kind", ["clusters", "lattice", "same", "chain"])
def test_sah_equals_oracle(rg, orc, kind, n):
    tri = soup(kind, n)
    sc = S.spheres_scene(n_spheres=1, width=8, height=8)
    verts = np.zeros(3 * n, sc.vertices.dtype)
    verts["position"] = tri.reshape(-1, 3)
    verts["normal"] = (0, 1, 0)
    ctx = rg.Context()
    ctx.upload_geometry(verts, np.arange(3 * n, dtype=np.uint32), sc.materials)
    b = ctx.build_blas(0, 0, n)
    got = ctx.bvh(b)
    ctx.close()
    ref = orc.sah(np.ascontiguousarray(np.concatenate([tri.min(1), tri.max(1)], 1)))
    assert orc.same_tree(got, ref)
    ids = np.concatenate([r[~(r >> 31).astype(bool)] for r in (got["left"], got["right"])])
    assert np.array_equal(np.sort(ids), np.arange(1, n - 1))  # every node but the root is one node's child
