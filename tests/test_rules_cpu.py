"""The size-independent rules of the kernels (csrc/sg_rules.h), compiled for the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "simbuca_gb300", "csrc")


def run(tmp_path, body):
    src = tmp_path / "rules.cpp"
    src.write_text('#include <cstdio>\n#include <set>\n#include "sg_rules.h"\n'
                   "int main() {\n" + body + "\nreturn 0;\n}\n")
    exe = tmp_path / "rules"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout


def test_fills_of_a_ragged_leaf_meet_no_padding_ion(tmp_path):
    """A fill of the last leaf's unused lanes on the same point as a padding ion would be a
    close pair of indices that no list holds (10,000 ions: padding ion 10,000 at 2.0e4)."""
    assert run(tmp_path, """
    const float fj = sg_leaf_fill(false), fi = sg_leaf_fill(true);
    // every padding ion of clouds of up to 2^21 ions; close pairs are within a few 1e-1
    for (int g = 1; g <= (1 << 21); g++) {
        const float p = sg_pad_frame(g);
        if (!(p - fj > 1.0f || fj - p > 1.0f) || !(p - fi > 1.0f || fi - p > 1.0f)) printf("%d\\n", g);
    }
    if (!(fi - fj > 1.0f || fj - fi > 1.0f)) printf("fills\\n");
    """) == ""


@pytest.mark.parametrize("n", [9984, 9985, 10000, 10001, 20000, 128, 1])
def test_only_real_ions_are_listed(tmp_path, n):
    assert run(tmp_path, f"""
    const int poff = 4096, n = {n}, end = poff + n, leaf0 = poff + (n - 1) / 128 * 128;
    for (int i = leaf0; i < leaf0 + 128; i++)
        for (int j = leaf0; j < leaf0 + 128; j++)
            if (sg_lists_pair(i, j, end) != (i != j && i < poff + n && j < poff + n)) printf("%d %d\\n", i, j);
    """) == ""


@pytest.mark.parametrize("blocks,past", [(152, 0), (152, 1), (1, 0), (160, 0)])
def test_a_barrier_count_may_wrap(tmp_path, blocks, past):
    """A block waits for every arrival of its barrier, and no longer, wherever the count
    stands: at the start, across 2^31 and across 2^32."""
    assert run(tmp_path, f"""
    const unsigned R = {blocks}, past = {past};
    for (unsigned base : {{0u, 0x7fffffffu - R, 0x7fffffffu, 0x80000000u, 0xffffffffu - R, 0xffffffffu}}) {{
        const unsigned target = base + R;
        for (unsigned a = 0; a < R + past; a++)
            if (sg_reached(base + a, target + past)) printf("early %u %u\\n", base, a);
        // the others may be one barrier further on
        for (unsigned a = R + past; a <= 2 * R; a++)
            if (!sg_reached(base + a, target + past)) printf("late %u %u\\n", base, a);
    }}
    """) == ""
