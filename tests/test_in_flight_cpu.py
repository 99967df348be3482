"""The list of outputs that launches in flight may be writing (csrc/in_flight.h): a weight written by any call since the last ordered
launch is found, however many calls lie between."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "in_flight.h"
#include <cstdio>
using nnb::InFlight;
static char* at(size_t a) { return (char*)a; }
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
    InFlight f;
    CHECK(!f.may_write(at(4096), 64));
    f.wrote(at(4096), 64);
    for (int rep = 0; rep < 50; ++rep)   // six q/k/v calls, then fifty: the first output stays known
        for (int i = 0; i < 20; ++i) f.wrote(at(1 << 20) + i * 4096, 4096);
    CHECK(f.out.size() == 21 && !f.more);
    CHECK(f.may_write(at(4096), 64) && f.may_write(at(4096 + 63), 1) && f.may_write(at(1), 4096));
    CHECK(!f.may_write(at(4096 + 64), 64) && !f.may_write(at(1), 4095));
    f.wrote(at(4096 + 16), 16);          // inside a known one
    f.wrote(at(4000), 400);              // around it
    CHECK(f.out.size() == 21 && f.may_write(at(4000), 1) && f.may_write(at(4399), 1) && !f.may_write(at(4400), 1));
    f.wrote(nullptr, 64);
    f.wrote(at(64), 0);
    CHECK(f.out.size() == 21 && !f.may_write(nullptr, 64));
    f.ordered();
    CHECK(!f.may_write(at(4096), 64));
    for (size_t i = 0; i < InFlight::MAX; ++i) f.wrote(at(4096) + i * 128, 64);
    CHECK(!f.more && !f.may_write(at(1 << 30), 64));
    f.wrote(at(1 << 20), 64);            // one more than fit: everything may be in flight
    CHECK(f.may_write(at(1 << 30), 64) && f.may_write(at(4096), 64));
    f.ordered();
    CHECK(!f.may_write(at(1 << 30), 64));
    f.wrote_unknown();
    CHECK(f.may_write(at(1 << 30), 64));
    f.ordered();
    f.limit = (size_t)-1;                // a recording
    for (size_t i = 0; i < 10 * InFlight::MAX; ++i) f.wrote(at(4096) + i * 128, 64);
    CHECK(!f.more && f.may_write(at(4096), 64) && f.may_write(at(4096 + 639 * 128), 1) && !f.may_write(at(4096 + 64), 64));
    return 0;
}
"""


def test_outputs_in_flight(tmp_path):
    src, exe = tmp_path / "in_flight.cpp", tmp_path / "in_flight"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(REPO, "adreno-llms_b200", "csrc"), str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
