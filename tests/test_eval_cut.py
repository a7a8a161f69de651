"""How the FP64 evaluation pass deals a unit's pairs to the warps of its CTA
(csrc/eval_cut.hpp, the code the kernel runs, compiled for the host): for every
number of targets and of sources of a stage, each (target, source) pair belongs
to exactly one lane, and the sum at the end meets every lane's part once.  Built
with and without fused multiply-adds: nothing may hang on how a compiler rounds.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sal-fort_b200", "csrc")

PROGRAM = r"""
#include "eval_cut.hpp"
#include <cstdio>
#include <vector>
using namespace sal;
int main() {
    for (int nt = 1; nt <= 256; ++nt) {
        const EvalCut cut(nt, eval_fold(nt));
        // per (warp, slot, lane): what its share is, and whether the end's sum takes it
        std::vector<EvalShare> sh;
        std::vector<int> target(kEvalWarps * kEvalSlots * 32, -1), taken(kEvalWarps * kEvalSlots * 32, 0);
        for (int w = 0; w < kEvalWarps; ++w)
            for (int i = 0; i < kEvalSlots; ++i)
                for (int l = 0; l < 32; ++l) sh.push_back(eval_share(cut, w, l, i));
        for (int id = 0; id < cut.nid; ++id) {   // as eval_kernel's end: lane id of the folded set
            const int c = id >> 5, last = c == cut.nch - 1, n = last ? cut.nlast : 32, r = last ? cut.rlast : 1;
            for (int w = 0; w < kEvalWarps; ++w) {
                const int i = cut.slot_of(w, c);
                if (i < 0 || i >= kEvalSlots) continue;
                for (int k = 0; k < r; ++k) {
                    const int at = (w * kEvalSlots + i) * 32 + (id & 31) + k * n;
                    ++taken[at];
                    target[at] = id % nt;
                }
            }
        }
        for (int n = 1; n <= 256; ++n) {
            std::vector<unsigned char> seen((size_t)nt * n, 0);
            for (size_t at = 0; at < sh.size(); ++at) {
                if (!sh[at].work) continue;
                int s, e;
                sh[at].sources(n, s, e);
                if (s < e && (taken[at] != 1 || target[at] != sh[at].ti)) { printf("nt %d: a lane's sum is lost\n", nt); return 1; }
                for (; s < e; s += sh[at].step) {
                    if (s < 0) { printf("nt %d n %d: source %d\n", nt, n, s); return 1; }
                    ++seen[(size_t)sh[at].ti * n + s];
                }
            }
            for (unsigned char v : seen)
                if (v != 1) { printf("nt %d n %d: a pair is taken %d times\n", nt, n, v); return 1; }
        }
    }
    return 0;
}
"""


@pytest.mark.parametrize("flags", [["-ffp-contract=off"], ["-mfma", "-ffp-contract=fast"]])
def test_every_pair_is_taken_once(tmp_path, flags):
    src = tmp_path / "cut.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "cut"
    subprocess.run(["g++", "-O2", "-std=c++17", *flags, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
