"""The order in which the hierarchy build looks at the pairs of a frontier
(csrc/tlfr_common.cuh): every pair once, by i and then j, also for frontiers of more
than 65536 nodes (one grid cell can hold that many)."""
import os
import subprocess

from tlfr_testutil import ROOT

PROGRAM = r"""
#include "tlfr_common.cuh"
#include <cstdio>
using namespace tlfr;

static int fail(const char* what, int size, int step)
{
    std::printf("%s: size %d, %d at a time\n", what, size, step);
    return 1;
}

int main()
{
    const int steps[] = { 1, 8, 32 };
    for (int step : steps)
        for (int size = 0; size < 45; size++)
        {
            int total = 0;
            for (int first = 0; first < step; first++)
            {
                PairWalk w(size, first);
                int flat = 0;
                for (int i = 0; i < size - 1; i++)
                    for (int j = i + 1; j < size; j++, flat++)
                        if (flat % step == first)
                        {
                            if (w.done() || w.i != i || w.j != j)
                                return fail("pair", size, step);
                            w.advance(step);
                            total++;
                        }
                if (!w.done())
                    return fail("end", size, step);
            }
            if (total != (size > 1 ? size * (size - 1) / 2 : 0))
                return fail("count", size, step);
        }
    // more than 2^31 pairs
    const int size = 70000, step = 32;
    const long long pairs = (long long)size * (size - 1) / 2;
    const int lanes[] = { 0, 31 };
    for (int first : lanes)
    {
        long long count = 0;
        int last_i = -1, last_j = -1;
        for (PairWalk w(size, first); !w.done(); w.advance(step))
        {
            if (w.i >= w.j || w.j >= size || w.i < last_i || (w.i == last_i && w.j <= last_j))
                return fail("order", size, step);
            last_i = w.i;
            last_j = w.j;
            count++;
        }
        if (count != (pairs - first + step - 1) / step)
            return fail("count", size, step);
    }
    std::puts("ok");
    return 0;
}
"""


def test_pairs_in_order(tmp_path):
    src = tmp_path / "pairs.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "pairs"
    csrc = os.path.join(ROOT, "temporal-lightfield-reconstruction_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", csrc, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
