"""rg_trace_rays: rays written by earlier work of the context's stream."""
import numpy as np
import pytest

from raygun_gb300 import scenes as S
from test_gpu_traverse import edge_rays

pytestmark = pytest.mark.gpu


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
