"""The end of a team's pass (csrc/search.h) with host threads for CTAs: the
first one runs every pass alone and hands it over at a gate, as a team does
while levels are small, and starts the next pass as soon as it may; one of
the others lags behind by far more than a pass before it looks at the queue.
Every thread has to see what the pass of that number left there."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "parallelbatchrcm_b200", "csrc")

PROGRAM = r"""
#include <pthread.h>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#include "search.h"

struct HostTeam {
    unsigned size, rank;
    pthread_barrier_t* bar;
    std::atomic<bool>* stop;
    bool sync(unsigned)
    {
        pthread_barrier_wait(bar);
        return !stop->load();
    }
};

int main(int, char** a)
{
    const unsigned size = (unsigned)atoi(a[1]), lag = (unsigned)atoi(a[2]), passes = 6;
    pthread_barrier_t bar;
    pthread_barrier_init(&bar, nullptr, size);
    std::atomic<unsigned> queue{0}, gate{0}, wrong{0};
    std::atomic<bool> stop{false};
    std::vector<std::thread> ts;
    for (unsigned r = 0; r < size; ++r)
        ts.emplace_back([&, r] {
            HostTeam team{size, r, &bar, &stop};
            for (unsigned p = 1; p <= passes; ++p) {
                if (r == 0) {
                    queue.store(p);  // the pass
                    gate.store(p);
                } else {
                    while (gate.load() < p)
                        std::this_thread::yield();
                }
                unsigned seen = 0;
                pbrcm::end_pass(team, [&] {
                    if (r == lag)
                        std::this_thread::sleep_for(std::chrono::milliseconds(20));
                    seen = queue.load();
                });
                if (seen != p)
                    ++wrong;
            }
        });
    for (auto& t : ts)
        t.join();
    // a team of one never waits; a stop is handed on
    HostTeam one{1, 0, nullptr, &stop}, two{2, 0, &bar, &stop};
    bool alone = pbrcm::end_pass(one, [] {});
    stop = true;
    pthread_barrier_t b1;
    pthread_barrier_init(&b1, nullptr, 1);
    two.bar = &b1;
    bool stopped = !pbrcm::end_pass(two, [] {});
    printf("%u %d %d\n", wrong.load(), alone, stopped);
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("end_pass")
    (d / "run.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(d / "run"), str(d / "run.cpp")], check=True)
    return lambda *a: subprocess.run([str(d / "run"), *map(str, a)], capture_output=True, text=True, timeout=60).stdout


@pytest.mark.parametrize("size,lag", [(2, 1), (4, 1), (4, 3), (8, 5)])
def test_every_cta_sees_the_pass_it_ended(run, size, lag):
    assert run(size, lag) == "0 1 1\n"
