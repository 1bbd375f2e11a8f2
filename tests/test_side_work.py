"""The order of a step with work on a side stream (csrc/side_work.hpp): whichever part of it fails, what was started on
the side is joined before the step returns, and the first failure is what it returns.  Compiled for the host with parts
that fail on request; no GPU."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <string>
#include "side_work.hpp"
int main() {
    for (int fails = 0; fails < 4; fails++) { // part 1, 2 or 3, or none
        std::string order;
        auto part = [&](char name, int k) { order += name; return fails == k ? 10 + k : 0; };
        const int s = hp::with_side_work(0, [&] { return part('b', 1); }, [&] { return part('w', 2); },
                                         [&] { return part('e', 3); }, [&] { order += 'j'; });
        std::printf("%d %s\n", s, order.c_str());
    }
}
"""


def test_a_failing_step_joins_its_side_work(tmp_path):
    src, exe = tmp_path / "side.cpp", tmp_path / "side"
    src.write_text(PROGRAM)
    inc = os.path.join(REPO, "hybrid-final_b200", "csrc")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", inc, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    assert out[:4] == ["0 bwe", "11 bj", "12 bwj", "13 bwej"]


def test_every_forking_step_goes_through_it():
    """fluid_begin and fluid_end have no caller outside a with_side_work."""
    for name in ("batch.cu", "capi.cu"):
        text = open(os.path.join(REPO, "hybrid-final_b200", "csrc", name)).read()
        assert text.count("fluid_begin(") == text.count("fluid_end(") == text.count("fluid_join(") == 1
        assert text.index("fluid_begin(") < text.index("fluid_end(") < text.index("with_side_work(HP_OK") < text.index("fluid_join(")
