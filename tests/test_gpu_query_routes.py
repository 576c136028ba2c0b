"""Ray queries against the oracle at the sizes where their forms meet (spread and full launches, page-locked rays and
device copies, one launch and two), and rays written by earlier work of the context's stream."""
import numpy as np
import pytest

from raygun_gb300 import scenes as S
from test_gpu_traverse import edge_rays

pytestmark = pytest.mark.gpu


def both(rg, ctx, rays):
    """Hits of rg_trace_rays and of rg_trace_rays_device, as (tuv, ids) each."""
    import torch
    n = len(rays)
    host = ctx.trace_rays(rays)
    d_rays = torch.from_numpy(rays).cuda()
    d_tuv, d_ids = torch.full((n, 3), -1.0, device="cuda"), torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.trace_rays_device(d_rays.data_ptr(), n, d_tuv.data_ptr(), d_ids.data_ptr())
    ctx.synchronize()
    return host, (d_tuv.cpu().numpy(), d_ids.cpu().numpy().view(np.uint32))


# 136192 lanes on 152 SMs: from there on a launch is no longer spread; 12288 and 172032: rg_trace_rays' routes
@pytest.mark.parametrize("n", [1, 2, 31, 33, 4256, 4257, 12288, 12289, 40001, 136191, 136192, 136193, 172032, 172033, 200000])
def test_query_sizes_equal_oracle(rg, orc, n):
    sc = S.instanced_scene(width=64, height=36, counts=(12, 10, 6, 2, 6, 6, 2, 2), hf_n=64, ico_levels=(2, 3, 3, 4))
    ctx = rg.Context()
    rg.load_scene(ctx, sc)
    rays = edge_rays("plain", n)
    tuv, ids = orc.OracleScene(sc).trace(rays)
    assert n < 50 or (ids[:, 0] != 0xFFFFFFFF).any()
    for t, i in both(rg, ctx, rays):
        assert np.array_equal(i, ids) and np.array_equal(t, tuv)
    ctx.close()


@pytest.mark.parametrize("n", [1, 77, 5000, 12289, 140000, 172033])
def test_overflowing_rays_equal_oracle(rg, orc, n):
    """Rays that overflow a 16-word stack, traced again by the launch's last block, among rays that miss."""
    from test_gpu_parity import camera_rays, stacked_scene
    sc = stacked_scene(4096)
    ctx = rg.Context()
    rg.load_scene(ctx, sc)
    ctx.set_batch_tune(128, 16, "none")
    cam = np.ascontiguousarray(camera_rays(sc), np.float32)
    away = cam.copy()
    away[:, 4:7] *= np.float32(-1.0)
    kinds = np.concatenate([cam, away])
    k = (np.arange(n) * 7) % len(cam) + np.where(np.arange(n) % 61 == 0, 0, len(cam))
    k[::61] = len(cam) // 2 + 24 + np.arange(len(k[::61])) % 3  # the image's middle, which the triangles cover
    tuv, ids = orc.OracleScene(sc).trace(kinds)
    got = both(rg, ctx, np.ascontiguousarray(kinds[k]))
    st = ctx.stats()
    assert st["stack_overflows"] == (ids[k, 0] != 0xFFFFFFFF).sum() == -(-n // 61) and st["deep_overflows"] == 0
    for t, i in got:
        assert np.array_equal(i, ids[k]) and np.array_equal(t, tuv[k])
    ctx.close()


@pytest.mark.parametrize("n", [50, 1000, 12288, 13000])
def test_rays_written_on_the_stream(rg, n):
    """Page-locked rays that a copy on the context's stream fills: the call reads them after that copy, on either side
    of the size (12288) up to which the kernel reads page-locked memory itself."""
    import torch
    sc = S.instanced_scene(width=64, height=36, counts=(12, 10, 6, 2, 6, 6, 2, 2), hf_n=64, ico_levels=(2, 3, 3, 4))
    ctx = rg.Context()
    rg.load_scene(ctx, sc)
    rays = edge_rays("plain", n)
    want = ctx.trace_rays(rays)
    assert (want[1][:, 0] != 0xFFFFFFFF).any()
    src = torch.from_numpy(rays).cuda()
    buf = torch.zeros(n, 8).pin_memory()  # zero directions: no hits
    torch.cuda.synchronize()
    stream = torch.cuda.ExternalStream(ctx.stream())
    with torch.cuda.stream(stream):
        torch.cuda._sleep(40_000_000)  # some 20 ms
        buf.copy_(src, non_blocking=True)
    got = ctx.trace_rays(buf.numpy())
    del buf  # while its stream exists
    ctx.close()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_overflowing_rays_share_the_chip(rg):
    """Many rays that overflow the short stack are traced again side by side: 12000 of them take no more than a few times
    as long as 100 (87 times when one block did them all)."""
    import time
    from test_gpu_parity import camera_rays, stacked_scene
    sc = stacked_scene()
    ctx = rg.Context()
    rg.load_scene(ctx, sc)
    ctx.set_batch_tune(128, 16, "none")
    cam = np.ascontiguousarray(camera_rays(sc), np.float32)
    cam = cam[ctx.trace_rays(cam)[1][:, 0] != 0xFFFFFFFF]

    def best(n):
        rays = np.ascontiguousarray(np.tile(cam, (n // len(cam) + 1, 1))[:n])
        times = []
        for _ in range(3):
            t = time.perf_counter()
            ctx.trace_rays(rays)
            times.append(time.perf_counter() - t)
        assert ctx.stats()["stack_overflows"] == n
        return min(times)

    assert best(12000) < 12 * best(100)
    ctx.close()
