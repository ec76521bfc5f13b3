"""The loop that runs the buckets of a sweep side by side, on the CPU with buckets that
fail on purpose: the others still deliver their results."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <memory>
#include <vector>
#include "cg_wave.h"
struct B { bool done = false; int id, need, steps = 0, asked = 0, delivered = 0; };
int main(int argc, char **argv) {
    // five buckets of 1 .. 5 steps; number `bad` fails with 2 in its step `at` (0: when it delivers)
    const int bad = atoi(argv[1]), at = atoi(argv[2]);
    std::vector<std::unique_ptr<B>> wave;
    for (int i = 0; i < 5; i++) {
        wave.push_back(std::make_unique<B>());
        wave[i]->id = i, wave[i]->need = i + 1;
    }
    const int st = cg::run_side_by_side(
        wave, [](B &b, bool last, bool *go) { *go = last || (b.asked++ & 1); return 0; },
        [&](B &b) {
            if (b.id == bad && at > 0 && b.steps + 1 == at) return 2;
            b.done = ++b.steps == b.need;
            return 0;
        },
        [&](B &b) {
            if (b.id == bad && at == 0) return 2;
            b.delivered++;
            return 0;
        });
    printf("%d", st);
    for (auto &b : wave) printf(" %d", b->delivered);
}
"""


def test_a_failing_bucket_leaves_the_others_their_results(tmp_path):
    src, exe = tmp_path / "wave.cpp", tmp_path / "wave"
    src.write_text(PROGRAM.replace("#include <cstdio>", "#include <cstdio>\n#include <cstdlib>"))
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "cugmres_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True, timeout=120)

    def run(bad, at):
        out = subprocess.run([str(exe), str(bad), str(at)], capture_output=True, text=True, timeout=20, check=True)
        return [int(v) for v in out.stdout.split()]

    assert run(-1, 0) == [0, 1, 1, 1, 1, 1]
    for bad in range(5):
        for at in (0, 1, bad + 1):
            assert run(bad, at) == [2] + [int(i != bad) for i in range(5)]
