"""CPU: the marks that say whether the host's mirror of the lengths is behind the device (csrc/len_mirror.h), with other threads stepping in at every place
of a step.  The header is compiled alone; `device` and `mirror` stand for one length on either side."""
import os
import subprocess

import pytest

import __graft_entry__ as entry

PROGRAM = r"""
#include "len_mirror.h"
#include <cstdio>
#include <cstring>
#include <thread>
using b200::MirrorMarks;

static MirrorMarks marks;
static int device = 0, mirror = 0;
static int refresh() { return marks.refresh([] { mirror = device; return 0; }); }
static void launch(int tokens, int layers = 1) { device += tokens; for (int l = 0; l < layers; ++l) marks.mark(); }
template <typename F> static void elsewhere(F&& f) { std::thread(f).join(); }

int main(int, char** argv) {
    const char* when = argv[1];
    const auto is = [&](const char* s) { return std::strcmp(when, s) == 0; };
    launch(3);
    if (!is("behind")) refresh();
    const auto at = marks.here();
    if (is("launch before")) elsewhere([] { launch(5); });
    if (is("read before")) elsewhere([] { refresh(); });
    launch(1, 4);                                        // this thread's step marks once a layer
    if (is("launch during")) elsewhere([] { launch(5); });
    if (is("read during")) elsewhere([] { refresh(); });
    if (is("both during")) elsewhere([] { launch(5); refresh(); });
    if (is("clear during")) elsewhere([] { marks.set_both([] { device = mirror = 0; }); });
    marks.enter_own(at, [] { mirror += 1; });
    if (is("launch after")) elsewhere([] { launch(5); });
    if (is("launch while reading")) {
        launch(1);
        marks.refresh([] { mirror = device; elsewhere([] { launch(5); }); return 0; });
    }
    std::printf("%d ", (int)marks.behind());
    refresh();
    std::printf("%d %d\n", device, mirror);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    where = tmp_path_factory.mktemp("mirror")
    src, exe = where / "t.cpp", where / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(entry.PKG_DIR, "csrc"), "-o", str(exe), str(src)], check=True)
    return str(exe)


@pytest.mark.parametrize("when,behind", [
    ("alone", 0), ("behind", 1), ("launch before", 1), ("read before", 0), ("launch during", 1), ("read during", 0), ("both during", 0), ("clear during", 0),
    ("launch after", 1), ("launch while reading", 1),
])
def test_a_step_enters_its_own_tokens_and_nobody_elses(program, when, behind):
    got = subprocess.run([program, when], check=True, capture_output=True, text=True).stdout.split()
    assert int(got[0]) == behind
    assert got[1] == got[2]               # what the next reader is told is what the device holds
