"""The size of the ray trees' node pool (host code): links hold 29 bits for a node, so a pool asked for more
samples than that holds fewer nodes, never nodes that a link cannot name."""
import os
import subprocess

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
