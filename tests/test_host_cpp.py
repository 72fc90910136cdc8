"""Host code of csrc/ that needs no CUDA, compiled by g++ and checked here against plain restatements."""

import heapq
import random
import subprocess

import numpy as np
import pytest

from kohaku_tt_b200 import _lib


def run(tmp_path, source, *args):
    """Output lines of `source` (C++17, csrc/ on its include path)."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", _lib.CSRC, "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True, text=True).stdout.split("\n")


@pytest.mark.parametrize("answers,want,asked", [
    ([5], [5, 5, 5], 1),            # asked once
    ([0], [0, 0, 0], 1),            # 0 is an answer
    ([-1, -1, 7], [-1, -1, 7, 7], 3),   # a failure is not one: the next caller asks again
])
def test_kept_answers(tmp_path, answers, want, asked):
    lines = run(tmp_path, '''
#include <cstdio>
#include <cstdlib>
#include "kept.h"
int main(int argc, char** argv) {
    std::atomic<int> slot{0};
    const int calls = std::atoi(argv[1]);
    int asked = 0;
    for (int i = 0; i < calls; ++i) std::printf("%d\\n", ktt::kept(slot, [&]() { return std::atoi(argv[2 + asked++]); }));
    std::printf("%d\\n", asked);
}
''', len(want), *answers)
    assert [int(x) for x in lines[:-1]] == want + [asked]


def _list_schedule(cost, count, machines):
    free = [np.float32(0)] * machines
    for c, n in zip(cost, count):
        for _ in range(n):
            heapq.heapreplace(free, np.float32(free[0] + c))
    return max(free)


# Up to 128 levels (and as many groups of machines), equal and unequal costs, more and fewer items than machines.
@pytest.mark.parametrize("levels,most,machines,steps", [
    (1, 400, 148, 1), (4, 60, 148, 3), (64, 40, 148, 1000), (128, 3, 296, 10**6), (128, 30, 148, 10**6), (128, 9, 7, 10**6), (65, 1, 148, 2), (64, 300, 1, 50),
])
def test_makespan_is_list_scheduling(tmp_path, levels, most, machines, steps):
    rng = random.Random(levels * machines)
    cost = np.array(sorted((rng.randint(1, steps) * 0.37 for _ in range(levels)), reverse=True), dtype=np.float32)
    count = [rng.randint(0, most) for _ in range(levels)]
    lines = run(tmp_path, '''
#include <cstdio>
#include <cstdlib>
#include "rounds.h"
int main(int argc, char** argv) {
    const int levels = (argc - 2) / 2;
    static float cost[2 * ktt::kMostLevels];
    static int64_t count[2 * ktt::kMostLevels];
    for (int i = 0; i < levels; ++i) {
        cost[i] = std::strtof(argv[2 + 2 * i], nullptr);
        count[i] = std::atoll(argv[3 + 2 * i]);
    }
    std::printf("%.9g\\n", static_cast<double>(ktt::makespan(cost, count, levels, std::atoll(argv[1]))));
}
''', machines, *(x for c, n in zip(cost, count) for x in ("%.9g" % c, n)))
    assert np.float32(lines[0]) == _list_schedule(cost, count, machines)
