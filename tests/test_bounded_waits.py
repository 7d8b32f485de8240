"""The bookkeeping of the gather's bounded waits (csrc/waits.h), compiled for
the host: a wait that never ends is given up at the limit and reported by
then, whatever the number of polls after which it is to be reported; one that
ends is reported exactly when it took at least that many polls."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "waits.h"
using namespace nufft3d;

// polls a copy that lands at poll `lands` (-1: never); prints reports, polls
// made and whether the wait was given up
int main(int, char **argv)
{
    const int polls = atoi(argv[1]), limit = atoi(argv[2]), lands = atoi(argv[3]);
    BoundedWait w;
    int reports = 0, made = 0, first = -1;
    bool gave_up = false;
    for (;;) {
        const WaitTurn t = wait_turn(w, polls, limit);
        if (t != kWaitOn) {
            if (first < 0) first = made;
            ++reports;
        }
        if (t == kWaitGiveUp) {
            gave_up = true;
            break;
        }
        if (made++ == lands) break;
        ++w.failed;
    }
    printf("%d %d %d %d\n", reports, first, made, (int)gave_up);
}
"""

LIMIT = 1 << 12


@pytest.fixture(scope="module")
def waits(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("waits")
    src, exe = d / "w.cpp", d / "w"
    src.write_text(SRC)
    subprocess.check_call([cxx, "-std=c++17", "-Wall", "-Werror", "-I",
                           os.path.join(ROOT, "nufft_3d_gb300", "csrc"), str(src), "-o", str(exe)])

    def run(polls, limit, lands):
        return tuple(int(v) for v in subprocess.check_output([str(exe), str(polls), str(limit), str(lands)]).split())

    return run


@pytest.mark.parametrize("polls", [0, 1, LIMIT - 1, LIMIT, LIMIT + 1, 2 ** 31 - 1])
def test_endless_wait_is_reported_and_given_up(waits, polls):
    reports, first, made, gave_up = waits(polls, LIMIT, -1)
    assert gave_up and made == LIMIT
    assert reports >= 1 and first == min(polls, LIMIT)


@pytest.mark.parametrize("polls", [0, 1, 7, LIMIT - 1, LIMIT])
@pytest.mark.parametrize("lands", [0, 1, 6, 7, 8, LIMIT - 2, LIMIT - 1])
def test_wait_that_ends(waits, polls, lands):
    reports, first, made, gave_up = waits(polls, LIMIT, lands)
    assert not gave_up and made == lands + 1
    assert reports == (1 if lands >= polls else 0)
    assert first == (polls if reports else -1)
