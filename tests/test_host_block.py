"""Host memory that a run reads its results into (st_hostblock.h): page-locked where it can be had,
ordinary memory otherwise, each given back the way it was taken.  Compiled for the host with a fake
of the page-locked allocation that can fail."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "soltrace_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "st_hostblock.h"

static bool refuse = false;
static int taken = 0, given = 0;
struct Fake {
    static bool alloc(void **p, size_t b) {
        if (refuse) return false;
        ++taken;
        *p = malloc(b);
        return true;
    }
    static void free(void *p) {
        ++given;
        ::free(p);
    }
};
#define CHECK(x) if (!(x)) return printf("line %d: %s\n", __LINE__, #x), 1
int main() {
    {
        stb::HostBlock<Fake> b;
        void *p = b.take(1 << 19);
        CHECK(p && b.pinned() && taken == 1);
        CHECK(b.take(1 << 19) == p && taken == 1);
    }
    CHECK(given == 1);
    refuse = true;
    {
        stb::HostBlock<Fake> b;
        void *p = b.take(1 << 19);
        CHECK(p && !b.pinned());
        memset(p, 1, 1 << 19);
        CHECK(b.take(1 << 19) == p);
    }
    CHECK(taken == 1 && given == 1);
    { stb::HostBlock<Fake> unused; }
    CHECK(given == 1);
    puts("ok");
    return 0;
}
"""


def test_ordinary_memory_stands_in_for_page_locked(tmp_path):
    src, exe = tmp_path / "block.cpp", tmp_path / "block"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
