"""Rules the kernels follow that can be checked without a GPU: compiled from the headers the kernels
include, or read from their sources.
"""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "trl_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def body(src, head):
    """The text from `head` to the closing brace of the block that follows it."""
    at = src.index(head)
    depth, i = 0, src.index("{", at)
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[at : j + 1]
    raise AssertionError(head)


def test_every_pair_of_the_tridiagonalisation_is_waited_for(tmp_path):
    exe = str(tmp_path / "tridiag_schedule")
    src = os.path.join(ROOT, "tests", "host", "tridiag_schedule.cc")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O2", f"-I{CSRC}", src, "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()
    assert out == [f"steps {sum(N - 1 for N in range(3, 1025))}"]
    # the kernel decides by the function that was checked, and expects a pair per row >= s
    steps = body(source("small.cu"), "__device__ __forceinline__ bool tri_steps(")
    assert steps.count("st_async_pair(") == 1
    assert re.search(r"if \(tri_sends\(N, g, lane, s\)\)\s*st_async_pair\(", steps)
    assert "static_cast<uint32_t>(N - s) * 16u" in steps
