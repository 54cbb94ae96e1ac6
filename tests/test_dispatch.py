"""Which FP64 kernel a launch with one grid takes (hxg_dispatch.cuh, host code): the
one-grid kernels need records on 32-byte lines and fewer than 2^32 of them; other
records, which only hxg_write_grid_noalloc can bring, go to the general kernel.
tests/test_fp64_loop.py runs that route on misaligned records."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CASES = [
    # groups, address, nx, ny, nz, groups of the instantiation
    (0, 0, 0, 0, 0, 0),
    (1, 0, 64, 64, 64, 1),
    (1, 32, 64, 64, 64, 1),
    (1, 16, 64, 64, 64, 2),
    (2, 16, 64, 64, 64, 2),
    (4, 0, 64, 64, 64, 4),
    (1, 0, 65535, 65537, 1, 1),          # 2^32 - 1 records
    (1, 0, 65536, 65536, 1, 2),          # 2^32
    (1, 0, 1626, 1626, 1626, 2),         # 4.299e9 records, 137.6 GB
    (1, 0, 1625, 1625, 1625, 1),
    (1, 0, 2 ** 31 - 1, 2 ** 31 - 1, 2 ** 31 - 1, 2),
    (3, 0, 1626, 1626, 1626, 3),
]


@pytest.fixture(scope="module")
def groups(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("dispatch")
    src = d / "groups.cc"
    src.write_text("""
#include <cstdio>
#include "hxg_dispatch.cuh"
int main() {
  long long n, at, nx, ny, nz;
  while (std::scanf("%lld %lld %lld %lld %lld", &n, &at, &nx, &ny, &nz) == 5)
    std::printf("%d\\n", hxg::fp64_groups((int)n, (const void *)at, (int)nx, (int)ny, (int)nz));
}
""")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "hammurabix_b200", "csrc"), "-I",
                    inc, "-o", str(d / "groups"), str(src)], check=True)
    text = "\n".join(" ".join(map(str, c[:5])) for c in CASES)
    out = subprocess.run([str(d / "groups")], input=text, capture_output=True, text=True,
                         check=True).stdout.split()
    return [int(v) for v in out]


@pytest.mark.parametrize("k", range(len(CASES)))
def test_groups_of_the_instantiation(groups, k):
    assert groups[k] == CASES[k][5], CASES[k]
