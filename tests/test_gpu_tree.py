"""Frames through ray trees (breadth-first expansion, check, bottom-up composition) against the
megakernel, which runs the shaders depth first, and against the oracle; spread traversal launches.

The scenes are hard on the expansion's assumptions: overlapping glass of several refractive indices
(curIOR left behind by a reflection's subtree), a grid-effect floor seen through it (refDepth), shadows
through glass, materials that consume several recursion levels."""
import numpy as np
import pytest

from raygun_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def glass_scene(width, height, spp, depth, seed=11, spheres=14):
    sc = S.spheres_scene(n_spheres=spheres, width=width, height=height, num_samples=spp, max_recursions=depth, seed=seed,
                         slices=16, stacks=8)
    rng = S.Rng(seed + 1)
    for k in range(1, len(sc.materials)):
        u, v = rng.uniform(2)
        m = S._material(rng.uniform(3), transparency=0.98 if u < 0.8 else 0.0, reflectivity=0.9 if u < 0.7 else 0.4, roughness=float(v) * 0.5,
                        ior=(1.5, 1.3, 2.4, 1.0)[k % 4], ray_consumption=1 + k % 3, effect_id=1 if k % 5 == 0 else 0)
        sc.materials[k] = m[0]
    # pull the spheres together so that they overlap
    p = sc.vertices["position"]
    p[4:] *= np.float32(0.55)
    p[4:, 1] += np.float32(0.4)
    return sc


def render(rg, sc, flags=0, glossy=0):
    rt = rg.Raytracer(sc, flags=flags).prepare()
    if glossy:
        rt.ctx.set_glossy(glossy)
    img = rt.render()
    g = [rt.ctx.download_image(k) for k in ("normal", "rough")]
    st = rt.ctx.stats()
    rt.ctx.close()
    return [img, *g], {k: st[k] for k in ("primary", "shadow", "secondary", "masked")}


@pytest.mark.parametrize("w,h,spp,depth,glossy", [(97, 55, 2, 0, 0), (97, 55, 2, 1, 0), (160, 90, 1, 2, 0), (161, 91, 2, 4, 0),
                                                  (120, 67, 3, 8, 0), (96, 54, 2, 5, 7), (1, 1, 1, 8, 0)])
def test_trees_equal_depth_first(rg, w, h, spp, depth, glossy):
    sc = glass_scene(w, h, spp, depth)
    a, sa = render(rg, sc, glossy=glossy)
    b, sb = render(rg, sc, flags=rg.RG_FLAG_MEGAKERNEL, glossy=glossy)
    assert sa == sb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("pool", [4700, 20000, 60000])
def test_full_node_pool(rg, monkeypatch, pool):
    """A pool that holds a fraction of the frame's nodes: the samples go in smaller and smaller chunks."""
    sc = glass_scene(160, 90, 2, 5)
    ref, sr = render(rg, sc)
    monkeypatch.setenv("RG_TREE_POOL", str(pool))
    got, sg = render(rg, sc)
    assert sg == sr
    for x, y in zip(got, ref):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("pool", [None, 2000000])
def test_two_lanes(rg, monkeypatch, pool):
    """A frame large enough for two lanes of chunks, with a pool that holds all trees or a fraction of them."""
    sc = glass_scene(1283, 409, 2, 3)
    ref, sr = render(rg, sc, flags=rg.RG_FLAG_MEGAKERNEL)
    if pool:
        monkeypatch.setenv("RG_TREE_POOL", str(pool))
    for _ in range(2):
        got, sg = render(rg, sc)
        assert sg == sr
        for x, y in zip(got, ref):
            assert np.array_equal(x, y)


def test_trees_equal_oracle(rg, orc):
    sc = glass_scene(128, 72, 1, 6)
    (img, _, _), st = render(rg, sc)
    b, n, r, ost = orc.OracleScene(sc).render()
    assert {k: ost[k] for k in st} == st
    ref = orc.post(sc.ubo, b, n, r)
    assert np.mean((np.abs(img - ref) <= 2.0 / 255.0).all(-1)) >= 0.999


@pytest.mark.parametrize("n", [1, 31, 4256, 4257, 40001, 136191, 136193, 200000])
def test_query_sizes(rg, n):
    """Spread launches (fewer rays than lanes, idle lanes joining) and full ones give the hits of the
    one-ray-per-thread kernel."""
    import torch
    ctx = rg.Context()
    rg.load_scene(ctx, S.instanced_scene(width=64, height=36, counts=(12, 10, 6, 2, 6, 6, 2, 2), hf_n=64, ico_levels=(2, 3, 3, 4)))
    u = S.Rng(5)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = np.stack([u.uniform(n, -70, 70), u.uniform(n, 0.0, 20), u.uniform(n, -70, 70)], 1)
    d = np.stack([u.normal(n), u.normal(n) * 0.3, u.normal(n)], 1)
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 3], rays[:, 7] = 0.01, 1000.0
    tuv, ids = ctx.trace_rays(rays)
    d_rays = torch.from_numpy(rays).cuda()
    d_tuv, d_ids = torch.full((n, 3), -1.0, device="cuda"), torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.trace_rays_device(d_rays.data_ptr(), n, d_tuv.data_ptr(), d_ids.data_ptr())
    ctx.synchronize()
    assert np.array_equal(d_ids.cpu().numpy().view(np.uint32), ids) and np.array_equal(d_tuv.cpu().numpy(), tuv)
    ctx.close()


@pytest.mark.parametrize("pool", [None, 4608, 30000])
@pytest.mark.parametrize("host_loop,sort", [(False, "none"), (False, "morton"), (True, "octant")])
def test_batch_trees(rg, monkeypatch, pool, host_loop, sort):
    """A batch of scenes of different recursion limits (0 to 8) and sizes through ray trees, its loops on the
    device or on the host, in chunks that fill the node pool, equals the scenes' own frames."""
    scs = [glass_scene(97, 55, 2, 5, seed=3), glass_scene(40, 30, 1, 0, seed=4), glass_scene(64, 64, 1, 8, seed=5, spheres=24),
           glass_scene(1, 1, 3, 2, seed=6)]
    ref = [render(rg, sc) for sc in scs]
    if pool:
        monkeypatch.setenv("RG_TREE_POOL", str(pool))
    br = rg.BatchRenderer(scs, flags=rg.RG_FLAG_HOST_LOOP if host_loop else 0)
    br.ctx.set_batch_tune(128, 48, sort)
    for _ in range(2):
        for img, (r, _) in zip(br.render(), ref):
            assert np.array_equal(img, r[0])
        st = br.ctx.stats()
        assert {k: st[k] for k in ("primary", "shadow", "secondary", "masked")} == \
            {k: sum(s[k] for _, s in ref) for k in ("primary", "shadow", "secondary", "masked")}
        assert st["iterations"] >= 9  # the largest recursion limit + 1
    br.ctx.close()
