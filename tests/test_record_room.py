"""The record buffer's bookkeeping (st_room.h) over ranks whose buffers differ.

The kernels store records below the capacity they are given, so at every launch that capacity must
fit the rank's own buffer, whatever the other ranks' buffers hold; an overflow on one rank makes all
ranks start again, with room for the largest count.  Compiled for the host and driven with a fake
buffer through the batches of a run.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "soltrace_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "st_room.h"

struct Buf {
    size_t bytes = 0;
    int ensure(size_t b) {
        if (b > bytes) bytes = b + b / 4;
        return 0;
    }
    int grow_keep(size_t b, size_t, int) {
        if (b > bytes) bytes = b;
        return 0;
    }
};

// argv: record bytes, then per rank: records of its earlier runs, then ':' and per batch the records of
// each rank.  A batch asks for `planned` records a rank, fewer than it leaves where that is possible.
int main(int argc, char **argv) {
    const size_t one = strtoull(argv[1], 0, 10);
    const int ranks = atoi(argv[2]);
    std::vector<Buf> buf(ranks);
    std::vector<stb::RecordRoom<Buf>> room;
    int at = 3;
    for (int k = 0; k < ranks; ++k) buf[k].ensure(strtoull(argv[at++], 0, 10) * one);
    for (int k = 0; k < ranks; ++k) room.emplace_back(buf[k], one);
    for (int attempt = 0; attempt < 4; ++attempt) {
        std::vector<unsigned long long> n(ranks, 0);
        for (int k = 0; k < ranks; ++k) room[k].begin(4096);
        bool again = false;
        for (int a = at; a + ranks < argc && !again; a += ranks + 1) {
            const unsigned long long planned = strtoull(argv[a], 0, 10);
            std::vector<unsigned long long> reports;
            for (int k = 0; k < ranks; ++k) {
                room[k].room(n[k] + planned + 4096, n[k], 0);
                if (room[k].cap * one > buf[k].bytes) return printf("rank %d may store past its buffer\n", k), 1;
                n[k] += strtoull(argv[a + 1 + k], 0, 10);
                for (unsigned long long v : room[k].report(n[k])) reports.push_back(v);
            }
            for (int k = 0; k < ranks; ++k) {
                const bool over = room[k].overflowed(reports.data(), ranks);
                if (k && over != again) return printf("ranks disagree\n"), 1;
                again = over;
            }
        }
        if (again) continue;
        for (int k = 0; k < ranks; ++k)
            if (n[k] > room[k].cap || room[k].cap * one > buf[k].bytes) return printf("records lost\n"), 1;
        return printf("ok %d\n", attempt), 0;
    }
    return printf("never sized\n"), 1;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("room")
    src, exe = d / "room.cpp", d / "room"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


CASES = [  # ranks' earlier records; batches of (planned records, records left on each rank); re-runs
    ([0], [(1000, 1500)], 0),
    ([0], [(1000, 900), (50_000, 90_000)], 1),
    ([1_000_000, 0], [(2000, 1800, 1700), (500_000, 400_000, 400_000)], 0),  # a small pilot, then a large batch
    ([0, 1_000_000, 10], [(2000, 1800, 1700, 0), (300_000, 1, 290_000, 290_000)], 0),
    ([1_000_000, 0], [(2000, 1800, 1700), (100_000, 90_000, 200_000)], 1),   # the small rank overflows
]


@pytest.mark.parametrize("earlier,batches,reruns", CASES)
def test_capacity_is_the_ranks_own(driver, earlier, batches, reruns):
    args = [driver, "72", str(len(earlier)), *map(str, earlier), *(str(v) for b in batches for v in b)]
    r = subprocess.run(args, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == f"ok {reruns}", r.stdout
