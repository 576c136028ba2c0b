"""Batches at the edges of their loops: what new device memory holds, loops that give up, many chunks, samples
whose trees exceed the node pool."""
import numpy as np
import pytest

from test_gpu_tree import glass_scene, render

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def glass(rg):
    scs = [glass_scene(97, 55, 2, 5, seed=3), glass_scene(40, 30, 1, 0, seed=4), glass_scene(64, 64, 1, 8, seed=5, spheres=24)]
    return scs, [render(rg, sc)[0][0] for sc in scs]


@pytest.mark.parametrize("host_loop", [False, True])
@pytest.mark.parametrize("sort", ["none", "octant", "morton"])
def test_first_batch_in_filled_memory(rg, glass, monkeypatch, sort, host_loop):
    """The first batch of a context whose buffers do not start as zeros (the ray sort's bucket counts are added to)."""
    scs, ref = glass
    br = rg.BatchRenderer(scs, flags=rg.RG_FLAG_HOST_LOOP if host_loop else 0)
    br.ctx.set_batch_tune(128, 48, sort)
    monkeypatch.setenv("RG_FILL_ALLOC", "0x3c")
    for _ in range(2):
        for img, r in zip(br.render(), ref):
            assert np.array_equal(img, r)
    br.ctx.close()


def test_host_loop_limit_is_reported(rg, glass, monkeypatch):
    """The host loop that stops at its limit returns the error itself, and leaves nothing behind for the
    batches after it, in either form."""
    scs, ref = glass
    br = rg.BatchRenderer(scs, flags=rg.RG_FLAG_HOST_LOOP)
    br.ctx.set_batch_slots(1024)
    monkeypatch.setenv("RG_BATCH_LOOP_LIMIT", "1")
    with pytest.raises(rg.RgError) as e:
        br.ctx.render_batch(br.jobs())
    assert e.value.code == -2 and "iteration limit" in str(e.value), str(e.value)
    monkeypatch.delenv("RG_BATCH_LOOP_LIMIT")
    for flags in (0, rg.RG_FLAG_HOST_LOOP):
        br.ctx.set_flags(flags)
        for img, r in zip(br.render(), ref):
            assert np.array_equal(img, r)
    br.ctx.close()


@pytest.mark.parametrize("host_loop", [False, True])
def test_loop_limit_counts_a_chunk(rg, glass, monkeypatch, host_loop):
    """The limit of the loops bounds the work on a chunk, not the number of chunks: a batch of hundreds of them passes
    with a limit of 40 runs."""
    scs, ref = glass
    br = rg.BatchRenderer(scs, flags=rg.RG_FLAG_HOST_LOOP if host_loop else 0)
    br.ctx.set_batch_slots(1024)
    monkeypatch.setenv("RG_TREE_POOL", "4700")
    monkeypatch.setenv("RG_BATCH_LOOP_LIMIT", "40")
    for img, r in zip(br.render(), ref):
        assert np.array_equal(img, r)
    br.ctx.close()


def dense_scene(width, height, spp, depth, seed):
    """Large glass spheres through each other: 8 to 9 rays a sample on average, hundreds for some."""
    sc = glass_scene(width, height, spp, depth, seed=seed, spheres=24)
    p = sc.vertices["position"]
    p[4:] = (p[4:] - p[4:].mean(0)) * np.float32(2.7) + p[4:].mean(0)
    m = sc.materials[1:]
    m["transparency"], m["reflectivity"], m["rayConsumption"] = 0.98, 0.9, 1
    return sc


@pytest.mark.parametrize("pool", [8, 40])
def test_samples_larger_than_the_pool(rg, monkeypatch, pool):
    """Samples whose trees no pool holds are rendered depth first: frames and both loop forms of a batch equal the
    megakernel's images and ray counts."""
    scs = [dense_scene(33, 17, 1, 8, 5), dense_scene(24, 16, 2, 6, 6), glass_scene(9, 7, 1, 0)]
    ref = [render(rg, sc, flags=rg.RG_FLAG_MEGAKERNEL) for sc in scs]
    count = ref[0][1]
    assert sum(count.values()) - count["masked"] > 8 * count["primary"]  # so a tree of more than 8 nodes is among them
    monkeypatch.setenv("RG_TREE_POOL", str(pool))
    for sc, (want, st) in zip(scs, ref):
        got, sg = render(rg, sc)
        assert sg == st
        for x, y in zip(got, want):
            assert np.array_equal(x, y)
    for flags in (0, rg.RG_FLAG_HOST_LOOP):
        br = rg.BatchRenderer(scs, flags=flags)
        for img, (want, _) in zip(br.render(), ref):
            assert np.array_equal(img, want[0])
        st = br.ctx.stats()
        assert {k: st[k] for k in count} == {k: sum(s[k] for _, s in ref) for k in count}
        br.ctx.close()


def test_glossy_sample_larger_than_the_pool(rg, monkeypatch):
    """The same with glossy reference shading, whose directions hang on the sample's seed."""
    sc = dense_scene(24, 16, 1, 7, 5)
    want, st = render(rg, sc, flags=rg.RG_FLAG_MEGAKERNEL, glossy=9)
    monkeypatch.setenv("RG_TREE_POOL", "8")
    got, sg = render(rg, sc, glossy=9)
    assert sg == st
    for x, y in zip(got, want):
        assert np.array_equal(x, y)


def test_chunks_grow_again(rg):
    """A batch with few slots: chunks shrink where samples need many rays and grow again behind them (the rounds of all chunks
    stay below those of chunks of one sample a slot)."""
    from raygun_gb300 import scenes as S
    scs = [dense_scene(64, 64, 1, 8, 5), S.spheres_scene(n_spheres=8, width=640, height=360, num_samples=1, max_recursions=2, seed=3)]
    ref = [render(rg, sc)[0][0] for sc in scs]
    br = rg.BatchRenderer(scs)
    br.ctx.set_batch_slots(1024)
    for img, r in zip(br.render(), ref):
        assert np.array_equal(img, r)
    # 9 rounds a chunk, and 9 for each of up to 8 repetitions in the dense job's
    assert br.ctx.stats()["iterations"] <= 9 * (640 * 360 // 1024) + 9 * 9 * (64 * 64 // 64)
    br.ctx.close()


@pytest.mark.parametrize("w,h,spp,swell,budget,rounds", [(160, 90, 1, 1.5, 0, 60), (160, 90, 1, 1.5, 1 << 30, 60), (1283, 409, 2, 2.5, 0, 250)])
def test_frames_of_many_rays_a_sample(rg, w, h, spp, swell, budget, rounds):
    """Frames with more nodes than the pool holds: images as the megakernel's from the first on, and later frames in few chunks
    that fit (9 rounds a chunk and those of replaced rays; 131, 131 and 371 rounds with a pool filled in vain first)."""
    sc = dense_scene(w, h, spp, 8, 5)
    p = sc.vertices["position"]
    p[4:] = (p[4:] - p[4:].mean(0)) * np.float32(swell) + p[4:].mean(0)
    (want, *_), st = render(rg, sc, flags=rg.RG_FLAG_MEGAKERNEL)
    assert sum(st.values()) - st["masked"] > 7 * st["primary"]  # so the first pool is too small
    rt = rg.Raytracer(sc, hbm_budget_bytes=budget).prepare()
    for k in range(4):
        assert np.array_equal(rt.render(), want)
        got = rt.ctx.stats()
        assert {x: got[x] for x in st} == st
    assert got["iterations"] <= rounds
    rt.ctx.close()


@pytest.mark.parametrize("host_loop", [False, True])
@pytest.mark.parametrize("budget", [0, 1 << 30])
def test_batches_of_many_rays_a_sample(rg, budget, host_loop):
    """The same for a batch, whose later launches take the chunks that fit in the last one; then a batch of as many samples
    and far fewer rays through the same context."""
    sc = dense_scene(160, 90, 1, 8, 5)
    p = sc.vertices["position"]
    p[4:] = (p[4:] - p[4:].mean(0)) * np.float32(1.5) + p[4:].mean(0)
    light = glass_scene(160, 90, 1, 8, seed=2, spheres=1)
    want = [render(rg, s)[0][0] for s in (sc, light)]
    br = rg.BatchRenderer([sc, light], flags=rg.RG_FLAG_HOST_LOOP if host_loop else 0, hbm_budget_bytes=budget)
    jobs = br.jobs()
    for k in (0, 0, 0, 0, 1, 1, 0):
        assert np.array_equal(br.render(jobs[k:k + 1])[0], want[k])
        its = br.ctx.stats()["iterations"]
        if k == 0:
            last = its
    assert last <= 60
    br.ctx.close()


def test_pool_falls_back_within_the_budget(rg):
    """A budget that holds 7 nodes a slot but not the 13 that a batch of few slots asks for first."""
    sc = glass_scene(640, 360, 1, 3)
    want = render(rg, sc)[0][0]
    slots = 1 << 16

    def batch(budget):
        br = rg.BatchRenderer([sc], hbm_budget_bytes=budget)
        br.ctx.set_batch_slots(slots)
        for _ in range(2):
            assert np.array_equal(br.render()[0], want)
        held = br.ctx.memory()[0]
        br.ctx.close()
        return held

    held = batch(0)
    assert held > 13 * 112 * slots
    budget = held - 5 * 112 * slots
    assert batch(budget) <= budget
