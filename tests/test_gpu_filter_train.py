"""The training step's weight-gradient and finishing kernels at sizes on the edges of their tiles: runs
that end inside a strip, CTAs without a row, one-pixel images, several strips and images."""
import numpy as np
import pytest

from test_gpu_filter import F, random_input, st_round, torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (1, 3, 127), (2, 5, 128), (1, 2, 129), (3, 61, 131), (1, 400, 257)])
def test_gradients_at_tile_edges(rg, B, H, W):
    """Bars of the existing gradient test: cosine >= 0.99 and norm within 5 % per layer against autograd
    with the same BF16 roundings."""
    ctx = rg.Context()
    flt = rg.Filter(ctx, seed=B + H)
    x = random_input(B, H, W, H)
    target = torch.zeros(B, H, W, 4)
    target[..., :3] = torch.rand(B, H, W, 3, generator=torch.Generator().manual_seed(9))
    d_in, d_t = x.to(torch.bfloat16).cuda(), target.cuda()
    torch.cuda.synchronize()
    flt.train_step(d_in.data_ptr(), d_t.data_ptr(), B, H, W, 0.0)
    grads = flt.grads().astype(np.float64)
    p = torch.tensor(flt.params(), device="cuda", dtype=torch.float64, requires_grad=True)
    layers, off = [], 0
    for co, ci in rg.FILTER_LAYERS:
        layers.append((p[off:off + co * ci * 9].view(co, ci, 3, 3), p[off + co * ci * 9:off + co * ci * 9 + co]))
        off += co * ci * 9 + co
    xx = x[..., :12].permute(0, 3, 1, 2).cuda().double()
    rnd = lambda t: st_round(t.float()).double()
    conv = lambda t, wb: F.conv2d(t, rnd(wb[0]), wb[1], padding=1)
    y1 = rnd(F.relu(conv(xx, layers[0])))
    y = rnd(F.relu(conv(y1, layers[1])))
    y = rnd(F.relu(conv(y, layers[2])))
    y = rnd(F.relu(conv(y, layers[3])))
    ((conv(rnd(y + y1), layers[4]).permute(0, 2, 3, 1) - target[..., :3].cuda().double()) ** 2).mean().backward()
    ref = p.grad.cpu().numpy()
    off = 0
    for co, ci in rg.FILTER_LAYERS:
        for n in (co * ci * 9, co):  # weights, then biases
            a, r = grads[off:off + n], ref[off:off + n]
            off += n
            if np.linalg.norm(r) == 0:
                assert np.linalg.norm(a) == 0
                continue
            assert a @ r / (np.linalg.norm(a) * np.linalg.norm(r)) >= 0.99
            assert abs(np.linalg.norm(a) - np.linalg.norm(r)) <= 0.05 * np.linalg.norm(r)


def test_step_updates_every_copy_of_the_weights(rg):
    """After a step the FP32 parameters follow Adam's formula (bar: a few FP32 roundings), and the packed
    forward and transposed weights are those of a filter given the same parameters: same gradients, bit
    for bit."""
    ctx = rg.Context()
    a, b = rg.Filter(ctx, seed=2), rg.Filter(ctx, seed=3)
    B, H, W = 2, 20, 140
    d_in = random_input(B, H, W, 1).to(torch.bfloat16).cuda()
    d_t = torch.rand(B, H, W, 4, generator=torch.Generator().manual_seed(1)).cuda()
    torch.cuda.synchronize()
    w0 = a.params().astype(np.float64)
    a.train_step(d_in.data_ptr(), d_t.data_ptr(), B, H, W, 1e-3)
    g = a.grads().astype(np.float64)
    m, v = (1 - np.float64(np.float32(0.9))) * g, (1 - np.float64(np.float32(0.999))) * g * g
    want = w0 - 1e-3 * (m / (1 - np.float64(np.float32(0.9)))) / (np.sqrt(v / (1 - np.float64(np.float32(0.999)))) + 1e-8)
    assert np.abs(a.params() - want).max() <= 1e-6
    b.set_params(a.params())
    la = a.train_step(d_in.data_ptr(), d_t.data_ptr(), B, H, W, 0.0)
    lb = b.train_step(d_in.data_ptr(), d_t.data_ptr(), B, H, W, 0.0)
    assert la == lb and np.array_equal(a.grads(), b.grads())
