"""The MMA warp's looks ahead at barriers: whichever lane issues the MMA afterwards must itself have seen
every barrier complete that the look stands for (or have waited for it), since a vote between lanes is no
memory order. 32 lanes are played one after the other on the host, for every way in which two barriers can
complete while the lanes look."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "f2k_cuda_b200" / "csrc"

PROGRAM = r"""
#include "barrier_look.h"
#include <cstdio>
#include <initializer_list>
using namespace f2k;
// Barrier b completes before lane done[b] looks (0: before all of them, 32: after all of them).
struct Warp {
    int lane, done[2];
    bool vote;                    // result of the vote, the same in every lane
    bool* acquired;               // [2], of this lane
    bool one(uint32_t bar, uint32_t par) const {
        const bool complete = par == bar && lane >= done[bar];      // barrier b is waited for with parity b
        if (complete) acquired[bar] = true;
        return complete;
    }
    bool test(uint32_t a, uint32_t pa, uint32_t b, uint32_t pb) const {
        const bool sa = one(a, pa);
        return b == a ? sa : one(b, pb) && sa;
    }
    bool all(bool) const { return vote; }
    bool wait(uint32_t bar, uint32_t par) const { return acquired[bar] = par == bar; }
};
int main() {
    for (int two : {0, 1})
        for (int a = 0; a <= 32; ++a)
            for (int b = 0; b <= 32; ++b) {
                bool acquired[32][2] = {}, vote = true;
                Look look[32];
                for (int lane = 0; lane < 32; ++lane) {
                    const Warp w{lane, {a, b}, false, acquired[lane]};
                    look[lane] = two ? look_at(w, 0, 0, 1, 1) : look_at(w, 0, 0);
                    vote = vote && look[lane].seen;
                }
                if (vote != (a == 0 && (!two || b == 0))) { std::printf("vote: two %d a %d b %d\n", two, a, b); return 1; }
                for (int lane = 0; lane < 32; ++lane) {
                    if (!finish(Warp{lane, {a, b}, vote, acquired[lane]}, look[lane])) { std::printf("gave up\n"); return 1; }
                    for (int k = 0; k <= two; ++k)
                        if (!acquired[lane][k]) { std::printf("lane %d goes on without barrier %d: two %d a %d b %d\n", lane, k, two, a, b); return 1; }
                }
            }
    return 0;
}
"""


def test_every_lane_is_behind_every_barrier(tmp_path):
    src, exe = tmp_path / "look.cpp", tmp_path / "look"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
