"""CPU test of the turns of the allocation-free step's control sets (st_turns.h): whatever calls
overlapped or failed before, a call that runs alone works in a set that was reset, and one that
follows complete, lone calls needs no reset kernel for it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "st_turns.h"

struct Call {
    st::Turns::Turn turn;
    int left;      /* kernels still to run: step (2), conversion (1) */
    bool alone;
};

int main()
{
    st::Turns t;
    bool used[2] = {false, false};   /* what the device's sets hold */
    std::vector<Call> run;
    int lone = 0, resets = 0, extra = 0;
    bool before = true;              /* every earlier call was complete and alone */
    srand(5);
    for (int k = 0; k < 200000; ++k) {
        const bool begin = run.empty() || (rand() % 8 == 0 && run.size() < 3);
        if (begin) {
            Call c = {t.begin(), 2, run.empty()};
            if (run.empty()) {
                if (c.turn.reset) used[0] = used[1] = false;
                assert(!used[c.turn.set]);
                ++lone;
                resets += c.turn.reset;
                extra += c.turn.reset && before;
                before = true;
            } else {
                assert(!c.turn.reset);
                for (Call& o : run) o.alone = false;
                before = false;
            }
            run.push_back(c);
            continue;
        }
        const int i = rand() % (int)run.size();
        Call& c = run[i];
        const bool fails = rand() % 50 == 0;
        if (!fails && c.left == 2) {
            used[c.turn.set] = true;           /* probe and step */
        } else if (!fails && c.left == 1) {
            used[c.turn.set ^ 1] = false;      /* the conversion resets the other set */
        }
        if (fails || --c.left == 0) {
            before = before && !fails && c.alone;
            t.end(!fails);
            run.erase(run.begin() + i);
        }
    }
    assert(lone > 1000 && resets > 100 && extra == 0);
    puts("ok");
    return 0;
}
"""


def test_lone_calls_get_a_reset_set(tmp_path):
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "driver"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I",
                           os.path.join(ROOT, "scale-track_b200", "csrc"), str(src), "-o",
                           str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stderr
