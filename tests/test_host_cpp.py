"""Host code of csrc/ that needs no CUDA, compiled by g++ and checked here against plain restatements."""

import os
import subprocess

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
