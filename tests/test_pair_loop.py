"""The loop in which two warps take groups together, run on two host threads: a warp whose
bounded wait ran out must not leave the other one at a barrier that it never reaches."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gravity-sim_gb300", "csrc")
HOST = r"""
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include "pair_loop.h"

// a barrier of two; a thread that waits 5 s for the other ends the program
struct Barrier {
    std::mutex m;
    std::condition_variable c;
    unsigned arrived = 0;
    void wait() {
        std::unique_lock<std::mutex> l(m);
        const unsigned phase = arrived++ / 2;
        c.notify_all();
        if (!c.wait_for(l, std::chrono::seconds(5), [&] { return arrived / 2 > phase; })) {
            std::puts("a warp waits for one that has left");
            std::_Exit(1);
        }
    }
};

int main(int argc, char** argv) {
    const uint32_t total = 40, at = std::atoi(argv[1]);  // the unit whose walk fails
    const int who = std::atoi(argv[2]);                  // bit w: on warp w
    uint32_t next = 0;
    gsim::PairTurn turn{0u, 0u};
    Barrier b;
    uint32_t walked[2] = {0, 0};
    auto warp = [&](int w) {
        gsim::pair_loop(turn, w == 0, total, [&] { return next < total ? next++ : total; }, [&] { b.wait(); },
                        [&](uint32_t u) {
                            if (u != walked[w]) std::_Exit(2);  // every unit once, in order
                            ++walked[w];
                            if ((u + w) % 3 == 0) std::this_thread::sleep_for(std::chrono::microseconds(200));
                            return !(u == at && (who >> w & 1));
                        });
    };
    std::thread other(warp, 1);
    warp(0);
    other.join();
    std::printf("%u %u\n", walked[0], walked[1]);
    return 0;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair")
    (d / "host.cpp").write_text(HOST)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + CSRC, str(d / "host.cpp"), "-o", str(d / "host")],
                   check=True)
    return str(d / "host")


@pytest.mark.parametrize("unit", [0, 17, 39])
@pytest.mark.parametrize("who", [1, 2, 3])
def test_a_failed_walk_ends_both_warps(host, unit, who):
    r = subprocess.run([host, str(unit), str(who)], capture_output=True, text=True, timeout=60)
    assert (r.returncode, r.stdout.split()) == (0, [str(unit + 1)] * 2)


def test_every_unit_without_a_failure(host):
    r = subprocess.run([host, "99", "3"], capture_output=True, text=True, timeout=60)
    assert (r.returncode, r.stdout.split()) == (0, ["40", "40"])
