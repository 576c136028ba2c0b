"""Traversal: the box terms' reciprocals, the shear set up before a BLAS's first triangle and the box
tests of empty slots, against the oracle's hits (exact: culling never drops a hit, whatever the rounding
of 1/d, and the triangle test's arithmetic is the oracle's)."""
import numpy as np
import pytest

from raygun_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def edge_rays(kind, n=6000):
    u = S.Rng(23)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = np.stack([u.uniform(n, -70, 70), u.uniform(n, 0.0, 16), u.uniform(n, -70, 70)], 1) * (0.7, 1, 0.7)
    d = np.stack([u.normal(n), u.normal(n) * 0.3 - 0.3, u.normal(n)], 1).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True).astype(np.float32)
    if kind == "axis":  # one direction component, the others zero of both signs
        k = np.arange(n) % 3
        m = np.where(u.uniform(n) < 0.5, np.float32(-0.0), np.float32(0.0)).astype(np.float32)
        d = np.where(np.arange(3)[None] == k[:, None], np.sign(d) + (d == 0), m[:, None])
        rays[: n // 2, :3] = np.round(rays[: n // 2, :3])  # starts on grid planes
    elif kind == "tiny":  # components down to subnormal numbers
        d[np.arange(n), np.arange(n) % 3] *= np.float32(10.0) ** (-(np.arange(n) % 44)).astype(np.float32)
    elif kind == "scale":  # |d| far from 1: t scales with it
        s = (np.float32(2.0) ** (np.arange(n) % 41 - 20)).astype(np.float32)
        d *= s[:, None]
    rays[:, 4:7] = d
    rays[:, 3], rays[:, 7] = 0.001, np.where(np.arange(n) % 4 == 0, 5.0, 1e9)
    return rays.astype(np.float32)


@pytest.mark.parametrize("kind", ["plain", "axis", "tiny", "scale"])
def test_edge_rays_equal_oracle(rg, orc, kind):
    import torch
    sc = S.instanced_scene(width=64, height=36, counts=(12, 10, 6, 2, 6, 6, 2, 2), hf_n=64, ico_levels=(2, 3, 3, 4))
    rays = edge_rays(kind)
    tuv, ids = orc.OracleScene(sc).trace(rays)
    assert (ids[:, 0] != 0xFFFFFFFF).sum() > 200  # of 6000 rays in an open scene
    ctx = rg.Context()
    rg.load_scene(ctx, sc)
    th, ih = ctx.trace_rays(rays)
    d_rays = torch.from_numpy(rays).cuda()
    d_tuv, d_ids = torch.full((len(rays), 3), -1.0, device="cuda"), torch.zeros((len(rays), 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.trace_rays_device(d_rays.data_ptr(), len(rays), d_tuv.data_ptr(), d_ids.data_ptr())
    ctx.synchronize()
    for t, i in ((th, ih), (d_tuv.cpu().numpy(), d_ids.cpu().numpy().view(np.uint32))):
        assert np.array_equal(i, ids) and np.array_equal(t, tuv)
    ctx.close()


@pytest.mark.parametrize("n", [1, 12288, 12289, 172032, 172033])
def test_host_query_routes(rg, n):
    """rg_trace_rays at the edges of its routes (page-locked rays; device copies; two launches whose overflow
    lists lie in each other's buffers), one ray in 50 overflowing a 16-word stack, against the
    device query."""
    import torch
    from test_gpu_parity import camera_rays, stacked_scene
    sc = stacked_scene(4096)
    ctx = rg.Context()
    rg.load_scene(ctx, sc)
    ctx.set_batch_tune(128, 16, "none")
    cam = camera_rays(sc)
    rays = np.ascontiguousarray(cam[(np.arange(n) * 7) % len(cam)], np.float32)
    rays[np.arange(n) % 50 != 0, 4:7] *= np.float32(-1.0)
    rays[::50] = cam[len(cam) // 2 + 24]  # the image's middle
    tuv, ids = ctx.trace_rays(rays)
    st = ctx.stats()
    hits = int((ids[:, 0] != 0xFFFFFFFF).sum())
    assert st["stack_overflows"] == hits == -(-n // 50) and st["deep_overflows"] == 0
    d_rays = torch.from_numpy(rays).cuda()
    d_tuv, d_ids = torch.full((n, 3), -1.0, device="cuda"), torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.trace_rays_device(d_rays.data_ptr(), n, d_tuv.data_ptr(), d_ids.data_ptr())
    ctx.synchronize()
    assert np.array_equal(d_ids.cpu().numpy().view(np.uint32), ids) and np.array_equal(d_tuv.cpu().numpy(), tuv)
    ctx.close()
