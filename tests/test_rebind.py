"""A workspace that moves to another device (st_rebind.h) leaves that device selected.

Compiled for the host with a fake workspace, whose destructor selects the device it frees on, as
the library's does; runs over several devices need one GPU each, so the sequence is checked here.
"""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "soltrace_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include "st_rebind.h"

static int current = 0, made = 0, freed_on = -1;
struct Workspace {
    int device = -1;
    int stream_device = -1;   // where the buffers and the stream were made
    unsigned long long scene = 0;
    ~Workspace() {
        if (device >= 0) current = device;
        freed_on = current;
    }
};
static int select_device(int d) {
    if (d > 3) return 101;
    current = d;
    return 0;
}
static int run(Workspace &ws, int device) {
    if (int e = stb::rebind(ws, device, select_device)) return e;
    if (ws.stream_device < 0) {
        ws.stream_device = current;
        ++made;
    }
    ws.scene = 7;
    return 0;
}
#define CHECK(x) if (!(x)) return printf("line %d: %s\n", __LINE__, #x), 1
int main() {
    Workspace ws;
    CHECK(run(ws, 0) == 0 && ws.stream_device == 0 && made == 1);
    CHECK(run(ws, 0) == 0 && made == 1 && ws.scene == 7);
    CHECK(run(ws, 2) == 0);
    CHECK(freed_on == 0);                 // the old device's buffers went there
    CHECK(current == 2 && ws.device == 2 && ws.stream_device == 2 && made == 2);
    CHECK(run(ws, 2) == 0 && made == 2 && current == 2);
    CHECK(run(ws, 9) == 101 && ws.device == 2 && ws.scene == 7);  // refused: the workspace stays
    CHECK(run(ws, 0) == 0 && current == 0 && ws.stream_device == 0);
    puts("ok");
    return 0;
}
"""


def test_moved_workspace_leaves_its_device_selected(tmp_path):
    src, exe = tmp_path / "rebind.cpp", tmp_path / "rebind"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
