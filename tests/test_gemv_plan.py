"""CPU: which kernel takes 9 to 16 tokens, as the library is compiled: the line lies where both kernels were measured."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ruquant_b200", "csrc")
GEMV, TENSOR_CORES = 1, 0
# inputs, rows, CTAs of the GEMV at once (288 without weight multipliers, 140 with them), tokens
MEASURED = [(256, 16, 288, 16, GEMV), (1024, 4096, 288, 9, GEMV), (1024, 4096, 140, 9, GEMV), (4096, 2048, 140, 16, GEMV), (6144, 4096, 288, 16, GEMV),
            (5120, 1024, 288, 12, GEMV), (1024, 8192, 288, 16, GEMV), (4096, 8192, 288, 9, GEMV),
            (256, 8192, 288, 9, TENSOR_CORES), (1024, 12288, 288, 9, TENSOR_CORES), (1024, 8192, 140, 9, TENSOR_CORES), (5120, 8192, 288, 9, TENSOR_CORES),
            (6144, 512, 288, 9, TENSOR_CORES), (6144, 1024, 288, 16, TENSOR_CORES), (11264, 4096, 288, 16, TENSOR_CORES),
            (17408, 5120, 288, 9, TENSOR_CORES), (5120, 17408, 288, 16, TENSOR_CORES)]


@pytest.fixture(scope="module")
def takes(tmp_path_factory):
    d = tmp_path_factory.mktemp("gemv")
    (d / "p.cpp").write_text('#include <stdio.h>\n#include "rq_gemv_plan.h"\nint main() { long long k, t, c, m, g;\n'
                             'while (scanf("%lld %lld %lld %lld %lld", &k, &t, &c, &m, &g) == 5) printf("%d\\n", (int) rq_gemv_takes_16(k, t, c, m, (int) g, c == 140)); return 0; }\n')
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, str(d / "p.cpp"), "-o", str(d / "p")])

    def ask(points, group=64):
        text = "\n".join("%d %d %d %d %d" % (K, (N + 15) // 16, ctas, M, group) for K, N, ctas, M in points)
        return [int(v) for v in subprocess.run([str(d / "p")], input=text, capture_output=True, text=True, check=True).stdout.split()]

    return ask


def test_where_it_was_measured(takes):
    assert takes([p[:4] for p in MEASURED]) == [p[4] for p in MEASURED]
    assert takes([(6144, 4096, 288, 16), (5120, 8192, 288, 16), (8192, 4096, 288, 16), (17408, 2048, 140, 9), (17408, 17408, 288, 9)], 256) == [
        GEMV, GEMV, GEMV, TENSOR_CORES, TENSOR_CORES]


def test_more_tokens_inputs_or_rows_never_come_back_to_the_gemv(takes):
    ks = [512, 1024, 4096, 4352, 5120, 8192, 11264, 32768]
    for N in (16, 1024, 2048, 4096):
        for M in (9, 16):
            got = takes([(K, N, 288, M) for K in ks])
            assert got == sorted(got, reverse=True)
    for K in ks:
        got = takes([(K, 2048, 288, M) for M in range(9, 17)])
        assert got == sorted(got, reverse=True)
