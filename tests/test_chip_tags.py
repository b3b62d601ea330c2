"""The tags of the face words of solves held in shared memory: whatever eager launches and replays of
captured ones follow one another, a launch finds none of its tags in the words. The words are modelled on
the CPU: the tags that launches have left there since they were last cleared."""
import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "hns_chip_tags.hpp"

struct Range { uint64_t first, last; };

int main(int, char** argv) {
    std::mt19937_64 rng(std::stoul(argv[1]));
    hns::ChipTags tags;
    std::vector<Range> left{{0, 0xFFFFFFFFull}};  // not cleared yet: anything
    std::vector<Range> graphs;
    int eager = 0, cleared = 0;
    for (int k = 0; k < 20000; ++k) {
        const uint32_t n = rng() % 3 ? (uint32_t)(rng() % 400) : (uint32_t)(rng() % 0x7FFFFFF0u) >> (rng() % 24);
        Range r;
        bool clear = true;
        if (rng() % 8 == 0) {  // captured: runs when it is replayed
            const auto t = tags.take(n, true);
            if (!t.clear || t.first == 0) return std::printf("captured launch %d\n", k), 1;
            graphs.push_back({t.first, (uint64_t)t.first + n});
            continue;
        }
        if (!graphs.empty() && rng() % 4 == 0) {
            r = graphs[rng() % graphs.size()];
        } else {
            const auto t = tags.take(n, false);
            clear = t.clear;
            r = {t.first, (uint64_t)t.first + n};
            ++eager, cleared += clear;
        }
        if (r.first == 0 || r.last > 0xFFFFFFFFull) return std::printf("launch %d: tags %llu..%llu\n", k, (unsigned long long)r.first, (unsigned long long)r.last), 1;
        if (clear) left.clear();
        for (const Range& q : left)
            if (r.first <= q.last && q.first <= r.last) return std::printf("launch %d: tag still in the words\n", k), 1;
        left.push_back(r);
    }
    if (cleared < 3 || cleared > eager / 2) return std::printf("%d of %d eager launches clear\n", cleared, eager), 1;
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("chip_tags")
    (d / "tags.cpp").write_text("#include <string>\n" + PROGRAM)
    exe = str(d / "tags")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "hnanosolver_b200", "csrc"), str(d / "tags.cpp"),
                    "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("seed", range(4))
def test_no_launch_finds_its_tags_in_the_words(program, seed):
    r = subprocess.run([program, str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
