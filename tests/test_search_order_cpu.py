"""Which matrices one thread group searches in discovery order from the first
pass on (csrc/search.h), compiled with the host compiler: wide stencils and
rows longer than an unordered pass puts together."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "parallelbatchrcm_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "search.h"
int main(int, char** a)
{
    const uint32_t n = (uint32_t)strtoul(a[1], nullptr, 10), nnz = (uint32_t)strtoul(a[2], nullptr, 10),
                   maxdeg = (uint32_t)strtoul(a[3], nullptr, 10);
    printf("%d %d\n", (int)pbrcm::wide_stencil(n, nnz, maxdeg), (int)pbrcm::long_rows(maxdeg));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "rule.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(d / "rule"), str(d / "rule.cpp")], check=True)
    return lambda *a: subprocess.run([str(d / "rule"), *map(str, a)], capture_output=True, text=True).stdout.split()


@pytest.mark.parametrize("n,nnz,maxdeg,want", [
    (4096, 20224, 5, "00"),                # 64 x 64 5-point grid
    (2097152, 14581760, 7, "00"),          # 128^3 7-point grid
    (20000, 218000, 19, "00"),             # geometric graph of 4-12 neighbours
    (20000, 300000, 31, "00"), (20000, 300000, 32, "01"),
    (20000, 708000, 52, "01"),             # geometric graph of 20-40 neighbours
    (20000, 820000, 68, "01"),             # random graph of 41 entries a row
    (4010, 12028, 403, "01"),              # path of hubs
    (7200, 177000, 27, "10"),              # 27-point mesh
    (1000000, 8988004, 9, "10"),           # 9-point mesh
    (8000, 830000, 125, "11"),             # 125-point mesh
    (4000000, 4294967280, 1100, "11"),     # 64-bit products
])
def test_order_rule(rule, n, nnz, maxdeg, want):
    assert "".join(rule(n, nnz, maxdeg)) == want
