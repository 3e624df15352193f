"""Host logic of the attention grid: every query tile of every (batch, head) group is taken by exactly
one CTA, pairs of tiles come before single ones, and splitting the last pairs never makes the grid longer
than one round of all SMs behind the full waves."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "f2k_cuda_b200" / "csrc"

PROGRAM = r"""
#include "attn_params.h"
#include <cstdio>
#include <vector>
using namespace f2k;
int main() {
    const CtaPlan ragged = cta_plan(17, 24, 148), ordinary = cta_plan(9, 32, 148);
    if (ragged.n_pairs != 148 || ragged.n_split != 44 || ragged.n_ctas != 148 + 2 * 44 + 24 ||
        ordinary.n_pairs != 128 || ordinary.n_split != 0 || ordinary.n_ctas != 128 + 32) { std::printf("known plans\n"); return 1; }
    for (int sms : {1, 7, 148})
        for (int tiles = 1; tiles <= 140; tiles += (tiles < 40 ? 1 : 7))
            for (int groups : {1, 2, 3, 4, 12, 24, 31, 32, 64, 128}) {
                const CtaPlan c = cta_plan(tiles, groups, sms);
                std::vector<int> seen(tiles * groups, 0);
                bool single = false;
                for (int i = 0; i < c.n_ctas; ++i) {
                    const CtaWork w = cta_work(c, tiles, i);
                    if (w.group < 0 || w.group >= groups || w.tile < 0 || w.tile + (w.two ? 1 : 0) >= tiles) {
                        std::printf("out of range: sms %d tiles %d groups %d cta %d\n", sms, tiles, groups, i);
                        return 1;
                    }
                    if (w.two && single) { std::printf("a pair behind a single tile\n"); return 1; }
                    single |= !w.two;
                    ++seen[w.group * tiles + w.tile];
                    if (w.two) ++seen[w.group * tiles + w.tile + 1];
                }
                for (int n : seen)
                    if (n != 1) { std::printf("sms %d tiles %d groups %d: a tile %d times\n", sms, tiles, groups, n); return 1; }
                const int rest = tiles / 2 * groups % sms, odd = tiles % 2 * groups;
                if (c.n_split != (2 * rest + odd <= sms ? rest : 0)) { std::printf("split rule\n"); return 1; }
                if (c.n_split > 0 && (c.n_pairs % sms != 0 || c.n_ctas - c.n_pairs > sms)) { std::printf("split\n"); return 1; }
            }
    return 0;
}
"""


def test_every_tile_is_taken_once(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(PROGRAM)
    cuda = Path("/usr/local/cuda/include")
    if not (cuda / "cuda.h").exists():
        pytest.skip("no CUDA headers")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-I", str(cuda), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
