"""The protocol of a CTA's waits for its bulk copies (csrc/amrlbm_wait.h) where
one does not land in time, on the host: the header is compiled with a model of
an mbarrier (a wait on a parity is over once the phase of that parity is), whose
copies land at a given wait or never."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "amr-lbm-openmp-2d_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "amrlbm_wait.h"
struct Barrier {
    int lands_at;  // wait during which the copy lands (0: before the first; -1: never)
    int waits = 0, phases = 0;
    bool wait(unsigned parity) {
        ++waits;
        if (phases == 0 && lands_at >= 0 && waits > lands_at) ++phases;
        return (phases & 1u) != parity;  // the phase of this parity is over
    }
};
int main(int, char** v) {
    Barrier bar[2] = {{atoi(v[1])}, {atoi(v[2])}};
    const int b = atoi(v[3]);
    CopyWaits w;
    auto on = [&](int b, unsigned p) { return bar[b].wait(p); };
    const bool ok = w.landed(b, atoi(v[4]), on, [](bool x) { return x; });
    printf("%d %u %d %d\n", ok, w.parity, bar[0].waits, bar[1].waits);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("copy_waits")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, "-o", str(d / "main"),
                    str(d / "main.cpp")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("lands,wait,in_flight,want", [
    # in time: one wait, the awaited barrier's parity advances
    ((0, 0), 0, 3, (1, 1, 1, 0)),
    ((0, -1), 0, 1, (1, 1, 1, 0)),
    ((-1, 0), 1, 2, (1, 2, 0, 1)),
    # late: the caller must not go on, though the copy has landed by now
    ((1, 0), 0, 1, (0, 0, 2, 0)),
    ((0, 1), 1, 2, (0, 0, 0, 2)),
    # never: the parity stays, or the next wait would pass at once
    ((-1, -1), 0, 1, (0, 0, 2, 0)),
    # the copies behind the other barrier are waited for too, where some are
    # in flight
    ((-1, 0), 0, 3, (0, 0, 2, 1)),
    ((1, -1), 0, 3, (0, 0, 2, 1)),
    ((0, -1), 1, 3, (0, 0, 1, 2)),
])
def test_late_copies(program, lands, wait, in_flight, want):
    out = subprocess.run([program, *map(str, (*lands, wait, in_flight))], check=True,
                         capture_output=True, text=True).stdout
    assert tuple(map(int, out.split())) == want
