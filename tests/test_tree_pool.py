"""The size of the ray trees' node pool (host code): links hold 29 bits for a node, so a pool asked for more
samples than that holds fewer nodes, never nodes that a link cannot name."""
import os
import subprocess

import pytest

from raygun_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pool_stays_within_the_links(tmp_path):
    exe = os.path.join(tmp_path, "tree_pool_dump")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", build.CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "tree_pool_dump.cu")], check=True)
    ask = [(1, 7, 4608), (658, 7, 4608), (659, 7, 4608), (1 << 25, 7, 4608), (1 << 25, 13, 4608), (41297762, 13, 4608), (41297763, 13, 4608),
           (76695844, 7, 4608), (76695845, 7, 4608), (1 << 31, 13, 4608), (1 << 62, 13, 4608), (1 << 40, 1, 4608), (0, 1, 4608)]
    out = subprocess.run([exe, *(str(v) for a in ask for v in a)], check=True, capture_output=True, text=True).stdout
    *got, last = (int(v) for v in out.split())
    assert got == [min(max(r * p, m), last) for r, p, m in ask]
    assert last < (1 << 29) - 3  # the links' values for no node


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = os.path.join(tmp_path_factory.mktemp("plan"), "tree_plan_sim")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", build.CSRC, "-o", exe, os.path.join(ROOT, "tests", "cpp", "tree_plan_sim.cpp")],
                   check=True)

    def run(work, lanes, pool, density, frames=3):
        out = subprocess.run([exe, *(str(v) for v in (work, lanes, pool, pool // 7, frames, *density))], check=True, capture_output=True,
                             text=True).stdout
        return [tuple(int(v) for v in line.split()) for line in out.splitlines()]

    return run


SKY_TO_GLASS = (1, 1, 2, 4, 12, 60, 40, 9)


@pytest.mark.parametrize("lanes", [1, 2])
@pytest.mark.parametrize("work", [1, 31, 32, 33, 1000, 14400, 100001])
@pytest.mark.parametrize("pool", [4, 8, 40, 4700, 100000, 1300013])
@pytest.mark.parametrize("density", [(1,) * 8, (3,) * 8, SKY_TO_GLASS, (500,) * 8])
def test_every_sample_once_in_chunks_that_fit(plan, work, lanes, pool, density):
    """Each sample is rendered once, no chunk has more roots than the pool nodes (exit code of the simulation)."""
    for done, full, samples, largest in plan(work, lanes, pool, density):
        assert samples == work and largest <= pool


@pytest.mark.parametrize("lanes", [1, 2])
@pytest.mark.parametrize("density", [(2.5,) * 8, (6,) * 8, (12,) * 8, (18,) * 8, (39,) * 8, SKY_TO_GLASS, SKY_TO_GLASS[::-1]])
def test_planned_frames_fill_no_pool(plan, lanes, density):
    """From the second frame on chunks fit (13 nodes a sample), and there are hardly more than their nodes need."""
    work = 230400
    pool = 13 * work // lanes
    nodes = sum(density) / 8 * work
    first, *rest = plan(work, lanes, pool, density, frames=4)
    for done, full, _, _ in rest[1:]:
        assert full == 0
        assert done <= max(lanes, int(nodes / (pool * 0.875)) + 1 + lanes)
