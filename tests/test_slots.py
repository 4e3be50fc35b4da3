"""The places that concurrent calls take in turn (litiv_gb300/csrc/slots.h), compiled for the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "slots.h"
#include <atomic>
#include <chrono>
#include <stdio.h>
#include <thread>
using namespace lvbgs;
static int bad = 0;
#define CHECK(c) do { if (!(c)) { printf("%d: %s\n", __LINE__, #c); ++bad; } } while (0)
int main() {
    {   // a place given back is taken again; one whose call did not end is not
        SlotPool pool(2);
        int first;
        { SlotLease a(pool); first = a.slot(); a.done(); }
        { SlotLease a(pool); CHECK(a.slot() == first); }  // no done(): retired
        for (int i = 0; i < 5; ++i) { SlotLease a(pool); CHECK(a.slot() == 1 - first); a.done(); }
        { SlotLease a(pool); CHECK(a.slot() == 1 - first); }
        { SlotLease a(pool); CHECK(a.slot() == -1); a.done(); }  // all retired: no wait without end
        CHECK(pool.take() == -1);
    }
    {   // a call that waits for a place goes on when the last one is retired
        SlotPool pool(1);
        std::atomic<int> got{7};
        const int held = pool.take();
        std::thread t([&] { got = pool.take(); });
        std::this_thread::sleep_for(std::chrono::milliseconds(20));
        CHECK(held == 0 && got == 7);
        pool.retire();
        t.join();
        CHECK(got == -1);
    }
    {   // eight threads over three places: no place is held twice
        SlotPool pool(3);
        std::atomic<int> users[3] = {{0}, {0}, {0}}, clashes{0};
        std::thread ts[8];
        for (auto& t : ts)
            t = std::thread([&] {
                for (int i = 0; i < 2000; ++i) {
                    SlotLease a(pool);
                    if (users[a.slot()]++ != 0) ++clashes;
                    --users[a.slot()];
                    a.done();
                }
            });
        for (auto& t : ts) t.join();
        CHECK(clashes == 0);
    }
    return bad;
}
"""


def test_places_are_given_back_or_retired(tmp_path):
    src, exe = tmp_path / "slots_test.cpp", tmp_path / "slots_test"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I" + os.path.join(ROOT, "litiv_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
