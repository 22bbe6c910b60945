"""The walk of a warp over a tile's entries (csrc/entries.h), compiled with
the host compiler: every entry once, in order of steps and lanes, and an end
to the walk, up to the largest entry count a pattern may have."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "parallelbatchrcm_b200", "csrc")
MAX_NNZ = 0xFFFFFFF0

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "entries.h"
int main(int, char** a)
{
    constexpr int U = 4;
    const uint32_t beg = (uint32_t)strtoul(a[1], nullptr, 10), end = (uint32_t)strtoul(a[2], nullptr, 10);
    const uint64_t most = ((uint64_t)(end - beg) + 32 * U - 1) / (32 * U);  // steps that cover the tile
    uint64_t next = beg, steps = 0;
    for (pbrcm::EntrySteps<U> es(beg, end); es.more(); es.next()) {
        if (++steps > most)
            return puts("endless"), 1;
        for (int i = 0; i < U; ++i)
            for (uint32_t lane = 0; lane < 32; ++lane) {
                uint32_t k = 0;
                if (!es.entry(i, lane, k))
                    continue;
                if (k != next++)
                    return puts("entry"), 1;
            }
    }
    return next == end && steps == most ? puts("ok"), 0 : (puts("short"), 1);
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("entries")
    (d / "walk.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(d / "walk"), str(d / "walk.cpp")], check=True)
    return str(d / "walk")


@pytest.mark.parametrize("length", [0, 1, 31, 32, 33, 127, 128, 129, 1000])
@pytest.mark.parametrize("end", [1000, 1 << 31, MAX_NNZ - 127, MAX_NNZ - 112, MAX_NNZ - 111, MAX_NNZ - 1, MAX_NNZ])
def test_every_entry_once(walk, end, length):
    out = subprocess.run([walk, str(end - length), str(end)], capture_output=True, text=True)
    assert out.stdout == "ok\n" and out.returncode == 0, out.stdout
