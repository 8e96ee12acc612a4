"""CPU: the host rules of the activation quantizer's launches, as the library is compiled with."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ruquant_b200", "csrc")


def run(tmp_path, body):
    (tmp_path / "p.cpp").write_text('#include <stdio.h>\n#include "rq_act_plan.h"\nint main() {\n' + body + "\nreturn 0; }\n")
    subprocess.check_call(["g++", "-std=c++17", "-fsanitize=address", "-I", CSRC, str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")])
    return subprocess.check_output([str(tmp_path / "p")], text=True)


@pytest.mark.parametrize("asked", [-5, 0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 64, 1000, 2147483647])
def test_cluster_width(tmp_path, asked):
    """whatever RQ_TUNE_ACT_CMAX holds: a power of two up to 8 whose clusters all fit; no other entry of the table is read
    (9 entries, the ones between hold a number that would let anything pass)"""
    out = run(tmp_path, """
    int * t = new int[9];
    for (int i = 0; i < 9; ++i) t[i] = 1 << 30;
    t[2] = 70; t[4] = 33; t[8] = 15;
    for (int units = 1; units < 40; ++units)
        for (int M = 1; M < 90; ++M) printf("%%d %%d %%d\\n", units, M, rq_act_cluster(rq_act_cluster_cap(%d), units, M, t));
    delete[] t;""" % asked)
    fits = {1: 1 << 30, 2: 70, 4: 33, 8: 15}
    rows = [tuple(int(v) for v in line.split()) for line in out.split("\n") if line]
    assert len(rows) == 39 * 89
    for units, M, c in rows:
        ok = [w for w in (1, 2, 4, 8) if w == 1 or (w <= asked and units >= 2 * w and M <= fits[w])]
        assert c == max(ok), (asked, units, M)


def test_threads_of_a_prefill_cta(tmp_path):
    """256 threads while the tokens are few, never again once 128 have been taken; at the sizes both forms were measured at"""
    out = run(tmp_path, """
    const int p[6] = { 12, 12, 20, 12, 44, 60 }, K[6] = { 768, 3072, 5120, 6144, 11264, 15360 };
    for (int i = 0; i < 6; ++i) {
        for (int M = 1; M < 2000; ++M) putchar(rq_act_256(p[i], K[i], M, 148) ? '1' : '0');
        putchar('\\n');
    }""")
    rows = out.split()
    last = [row.rfind("1") + 1 for row in rows]
    assert all(row == "1" * n + "0" * (1999 - n) for row, n in zip(rows, last))
    assert last == [444, 444, 592, 592, 444, 444]
