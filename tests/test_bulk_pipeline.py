"""The row-major fill's copies and reductions (gbx_bulk.h) on the host, with
copies that arrive late or never: every item added once and in order while all
arrive; after a wait that gave up nothing is started any more, no buffer is
filled while its copy or a reduction still uses it, every copy under way is
waited for again, and the result says that bins are missing."""

import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "gbx_bulk.h"

// a barrier of one expected copy per phase, as the hardware's
struct Stage { int item = -1; bool flying = false; unsigned phase = 0; int waits = 0; };

int main(int, char **v)
{
    constexpr int S = 4;
    const int items = atoi(v[1]), stuck = atoi(v[2]);
    std::vector<Stage> st(S);
    std::vector<int> reading;                        // stages whose reduction has not read yet
    int given = 0, added = 0, faults = 0, gave_up = 0, waited_again = 0;
    auto next = [&](int &it) { if (given == items) return false; it = given++; return true; };
    auto load = [&](int k, const int &it) {
        for (int r : reading) faults += r == k;      // still read by a reduction
        faults += st[k].flying || gave_up;           // still filled, or started after giving up
        st[k].item = it;
        st[k].flying = true;
    };
    auto loaded = [&](int k, unsigned parity) {
        Stage &s = st[k];
        if (gave_up) waited_again++;
        if (s.flying && s.item != stuck) { s.flying = false; s.phase ^= 1; }     // arrives
        const bool ok = (s.phase & 1) != parity;     // the phase of that parity is over
        if (!ok) { gave_up++; s.waits++; }
        return ok;
    };
    auto add = [&](int k, const int &it) {
        faults += st[k].flying || st[k].item != it || it != added;
        added++;
        reading.push_back(k);
    };
    auto read = [&]() { while (reading.size() > 1) reading.erase(reading.begin()); };
    const bool ok = gbx::bulk_pipeline<S, int>(next, load, loaded, add, read);
    int flying = 0, unwaited = 0;
    for (auto &s : st) { flying += s.flying; unwaited += s.flying && s.waits < 2; }
    printf("%d %d %d %d %d %d %d\n", ok, added, given, faults, flying, unwaited, waited_again);
}
'''


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("bulk")
    (d / "p.cpp").write_text(PROGRAM)
    exe = str(d / "p")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "gbgpu_gb300", "csrc"),
                    str(d / "p.cpp"), "-o", exe], check=True)
    return exe


def run(program, items, stuck):
    out = subprocess.run([program, str(items), str(stuck)], capture_output=True, text=True, check=True)
    return tuple(map(int, out.stdout.split()))


@pytest.mark.parametrize("items", [0, 1, 2, 3, 4, 5, 8, 9, 100])
def test_all_arrive(program, items):
    assert run(program, items, -1) == (1, items, items, 0, 0, 0, 0)


@pytest.mark.parametrize("items,stuck", [(n, k) for n in (1, 3, 4, 9, 100)
                                         for k in (0, 1, 3, 4, 7, 8, 50, 99) if k < n])
def test_one_never_arrives(program, items, stuck):
    ok, added, given, faults, flying, unwaited, again = run(program, items, stuck)
    # everything before it is added, at most three copies were under way, and all of
    # them, the late one included, were waited for once more
    assert (ok, added, faults, flying, unwaited) == (0, stuck, 0, 1, 0)
    assert given == min(items, stuck + 3) and again == given - stuck
