"""Rules the kernels follow that can be checked without a GPU: compiled from the headers the kernels
include, or read from their sources.
"""
import os
import re
import subprocess

import numpy as np
import pytest

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


@pytest.fixture(scope="module")
def largest_overlaps(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host") / "orthonormal_limit")
    src = os.path.join(ROOT, "tests", "host", "orthonormal_limit.cc")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", f"-I{CSRC}", src, "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [(int(k), float(e)) for k, e in (ln.split() for ln in out.splitlines())]


@pytest.mark.parametrize("signs", ["equal", "random"])
def test_second_orthonormalisation_step_ends_at_rounding(largest_overlaps, signs):
    """The step z_j - E_jj / 2 z_j - sum_{i<j} E_ij z_i in extended precision on a Gram matrix I + E with every
    overlap at the largest that is let through. It leaves (S^T (I + E) S) - I with S = I - D / 2 - U: -E_ij E_ik
    summed over K vectors, and E^2 once for the diagonal's share: (K + 1) E^2 <= 2 eps."""
    for K, e in largest_overlaps:
        E = np.full((K, K), e, dtype=np.longdouble)
        if signs == "random":
            E *= np.sign(np.random.default_rng(K).standard_normal((K, K)))
            E = np.triu(E) + np.triu(E, 1).T
        S = np.eye(K, dtype=np.longdouble) - np.triu(E, 1) - np.diag(np.diag(E)) / 2
        left = S.T @ (np.eye(K, dtype=np.longdouble) + E) @ S - np.eye(K, dtype=np.longdouble)
        assert np.abs(left).max() <= 2 * np.finfo(np.float64).eps, K


def test_orthonormalisation_decides_by_the_checked_limit():
    launches = re.findall(r"launch\((?:k_gs_apply|k_tri_gs),[^;]*;", source("small.cu"))
    assert len(launches) == 2 and all("gs_limit(K)" in ln for ln in launches)


def test_kernels_of_one_type_have_their_own_ctas_per_sm(tmp_path):
    from trl_b200 import build

    exe = str(tmp_path / "resident_ctas")
    src = os.path.join(ROOT, "tests", "host", "resident_ctas.cu")
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", f"-I{CSRC}", f"-I{ROOT}/include", src, "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, env=dict(os.environ, CUDA_VISIBLE_DEVICES="")).stdout
    assert out.split() == ["4", "2", "4", "2", "3"]
    # no cache beside it that is shared between kernels of one type
    for name in ("sell.cu", "spmm.cu"):
        assert "cudaOccupancyMaxActiveBlocksPerMultiprocessor" not in source(name)


def test_no_unguarded_static_state():
    """What a function keeps for the process is atomic or behind a lock: host threads with a handle each call the
    library at the same time."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        src = source(name)
        kept = [ln.strip() for ln in src.splitlines() if re.match(r"\s+static (?!constexpr|const |std::atomic|std::mutex|__device__|_?assert)(?!.*\()", ln)]
        if name == "small.cu":  # tri_variant's, behind its lock
            assert "static std::mutex lock;" in body(src, "const TriVariant* tri_variant(")
            kept = [ln for ln in kept if ln not in ("static int ok[64][kNumTriVariants];", "static bool checked[64];")]
        assert kept == [], name
