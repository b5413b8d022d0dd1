"""The shares of a batched launch's later rounds (team_sync.cuh): every block
makes them for itself, so they must not depend on what teams of the same round
store meanwhile."""
from __future__ import annotations

import os
import subprocess

import pytest

from sfr3d_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SYSTEMS, GRID = 41, 96
FIRST = [sum(3 + (i * 37) % 90 for i in range(s)) for s in range(SYSTEMS + 1)]


def test_shares_of_a_round_do_not_follow_its_own_results(cuda, tmp_path):
    exe = tmp_path / "team_rounds"
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-ccbin", build._host_cxx(),
                    "--expt-relaxed-constexpr", "-I", build.INCLUDE, "-I", build.CSRC,
                    os.path.join(HERE, "team_rounds.cu"), "-o", str(exe)], check=True)
    text = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    plans = {}
    for line in text.splitlines():
        rnd, late, block, *rest = map(int, line.split())
        plans.setdefault((rnd, late), []).append(rest)
    done = set()
    for rnd in (1, 2, 3):
        plan = plans[rnd, 0]
        assert plans[rnd, 1] == plan
        # one team of neighbouring blocks a system left, its slices in order
        teams = {}
        for block, (any_left, sys_, s0, s1, b0, b1) in enumerate(plan):
            assert any_left == 1
            if sys_ >= 0:
                assert b0 <= block < b1 <= GRID
                teams.setdefault(sys_, []).append((block, s0, s1, b0, b1))
        assert set(teams) == set(range(SYSTEMS)) - done
        for sys_, blocks in teams.items():
            assert [b[0] for b in blocks] == list(range(blocks[0][3], blocks[0][4]))
            assert len({b[3:] for b in blocks}) == 1
            edges = [blocks[0][1]] + [b[2] for b in blocks]
            assert [b[1] for b in blocks] == edges[:-1]
            assert (edges[0], edges[-1]) == (FIRST[sys_], FIRST[sys_ + 1])
        done |= {i for i in range(SYSTEMS) if i % 3 == rnd % 3}
    # the rounds after take the stores in
    assert plans[1, 0] != plans[2, 0] != plans[3, 0]
