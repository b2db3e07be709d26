"""The pinned words that contexts share (gell_b200/csrc/count_words.h), on the CPU against a fake of the
runtime: words are distinct while they are held, pages come and go, an allocation that fails gives no word, and
a word whose page went with a device reset is not given back to the page that now has its address."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cassert>
#include <cstdlib>
#include <set>
#include "count_words.h"
static int buffers[4][1024];
static bool held[4];
static int room = 4;
struct Fake {
    static bool known(const int* p) {
        for (int k = 0; k < 4; ++k)
            if (p == buffers[k]) return held[k];
        return false;
    }
    static int* alloc(size_t bytes) {
        if (bytes > sizeof buffers[0]) abort();
        for (int k = 0; k < room; ++k)
            if (!held[k]) {
                held[k] = true;
                return buffers[k];
            }
        return nullptr;
    }
    static void release(int* p) {
        if (!known(p)) abort();
        held[(p - buffers[0]) / 1024] = false;
    }
};
static int pages() { return held[0] + held[1] + held[2] + held[3]; }
#define CHECK(x) do { if (!(x)) return __LINE__ & 0xff; } while (0)
int main() {
    gell::CountWords<Fake> w;
    std::set<int*> seen;
    gell::CountWord a[130];
    for (auto& x : a) {
        x = w.take();
        CHECK(x.at && seen.insert(x.at).second);
    }
    CHECK(pages() == 3);
    for (int k = 64; k < 130; ++k) w.give(a[k]);
    CHECK(pages() == 1);
    for (int k = 0; k < 64; ++k) w.give(a[k]);
    CHECK(pages() == 1);  // the last page stays
    // a reset: the page is gone, and the next one comes at its address
    gell::CountWord old = w.take();
    held[0] = false;
    gell::CountWord now = w.take();
    CHECK(now.at == old.at);
    w.give(old);
    CHECK(w.take().at != now.at);
    w.give(gell::CountWord{});
    // no memory
    gell::CountWords<Fake> v;
    room = 0;
    CHECK(!v.take().at);
    room = 4;
    CHECK(v.take().at);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_words_of_pages_that_come_and_go(tmp_path):
    src, exe = tmp_path / "words.cpp", tmp_path / "words"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "gell_b200", "csrc"), str(src), "-o", str(exe),
                    "-pthread"], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
