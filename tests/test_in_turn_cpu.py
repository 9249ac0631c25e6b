"""Host control flow of the ensemble's calls (csrc/in_turn.hpp), compiled by g++: what is completed when a step
throws.  The four lanes of an ensemble are stood in for by counters (no GPU needed)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "in_turn.hpp"
#include <cstdio>
#include <stdexcept>
using namespace mf3d;
#define EXPECT(c) if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; }
template <class F> int thrown(F&& f) { try { f(); } catch (int e) { return e; } return 0; }
int main() {
    int flags[5] = {0, 1, 0, 1, 0}, seen = 0; // each flag is cleared, the first is reported
    EXPECT(thrown([&] { each_then_throw(5, [&](size_t i) { ++seen; if (flags[i]) { flags[i] = 0; throw (int)i; } }); }) == 1);
    EXPECT(seen == 5 && !flags[1] && !flags[3]);
    EXPECT(thrown([&] { each_then_throw(0, [&](size_t) { throw 1; }); }) == 0);
    // work started on lanes 0 and 1 when lane 2 fails: every lane is joined, and waited for
    int joined = 0, waited = 0, started = 0;
    auto join = [&](bool failed) { for (int l = 0; l < 4; ++l) { ++joined; waited += failed; } };
    EXPECT(thrown([&] { then_always([&] { for (int l = 0; l < 4; ++l) { if (l == 2) throw 7; ++started; } }, join); }) == 7);
    EXPECT(started == 2 && joined == 4 && waited == 4);
    EXPECT(thrown([&] { then_always([&] { started = 4; }, join); }) == 0);
    EXPECT(started == 4 && joined == 8 && waited == 4);
    // the first failure is reported, a failure of the joining only when nothing failed before it
    EXPECT(thrown([&] { then_always([] { throw 3; }, [](bool) { throw 4; }); }) == 3);
    EXPECT(thrown([&] { then_always([] {}, [](bool) { throw 4; }); }) == 4);
    std::puts("ok");
}
"""


def test_steps_are_completed_and_the_first_error_is_thrown(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "macroflow3d_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout
