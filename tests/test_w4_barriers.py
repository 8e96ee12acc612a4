"""CPU: the barriers on which the fold warps of the 9-to-64-token kernel wait.  A wait names a phase by its parity, so it is sound
only for a warp that has seen every earlier phase of that barrier end: the constants the kernel is compiled with, walked for
every tile width, activation group and team of fold warps."""
import os
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ruquant_b200", "csrc", "rq_gemm_w4_plan.h")
PROGRAM = r"""
#include <stdio.h>
#include "rq_gemm_w4_plan.h"
int main() {
    for (int nt = 16; nt <= 64; nt += 16)
        for (int gsteps = 1; gsteps <= 4; gsteps *= 2)
            printf("%d %d %d %d %d %d %d\n", nt, gsteps, rq_w4_nd(nt), rq_w4_full_bars(nt), rq_w4_slice_sets(nt, gsteps), RQ_W4_M_STAGES,
                   RQ_W4_FOLD_TEAMS);
    return 0;
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("w4")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-I", os.path.dirname(HEADER), str(d / "plan.cpp"), "-o", str(d / "plan")])
    lines = subprocess.check_output([str(d / "plan")], text=True).split("\n")
    return [tuple(int(v) for v in line.split()) for line in lines if line]


def waits_see_every_phase(visits):
    """visits: (barrier, phase) in the order one warp waits for them"""
    seen = {}
    for barrier, phase in visits:
        if phase != seen.get(barrier, -1) + 1:
            return False
        seen[barrier] = phase
    return True


def test_the_rule_itself():
    assert waits_see_every_phase([(s % 4, s // 4) for s in range(0, 40, 2)])
    assert not waits_see_every_phase([(s % 3, s // 3) for s in range(0, 40, 2)])      # three barriers, every second set


def test_fold_warps_see_every_phase(plans):
    assert len(plans) == 12
    for nt, gsteps, nd, bars, sets, m_stages, teams in plans:
        assert nd >= 2 and bars >= nd
        for team in range(teams):
            own = range(team, 240, teams)
            assert waits_see_every_phase([(s % bars, s // bars) for s in own]), (nt, "accumulator sets")
            # the multiplier ring: a slot per slice, waited for once per own set of the slice (again for the same phase is harmless)
            slices = sorted({s // sets for s in own})
            assert waits_see_every_phase([(i % m_stages, i // m_stages) for i in slices]), (nt, gsteps, "multipliers")
