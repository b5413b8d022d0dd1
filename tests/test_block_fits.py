"""Shared memory a block of a batched launch takes for its slots
(team_sync.cuh): exact also where the bytes of very wide rows pass 2^31."""
from __future__ import annotations

import os
import subprocess

from sfr3d_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
LEFT = 231000


def test_slot_bytes_past_31_bits(tmp_path):
    exe = tmp_path / "block_fits"
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-ccbin", build._host_cxx(),
                    "--expt-relaxed-constexpr", "-I", build.INCLUDE, "-I", build.CSRC,
                    os.path.join(HERE, "block_fits.cu"), "-o", str(exe)], check=True)
    text = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert len(text.splitlines()) == 7
    for line in text.splitlines():
        slots, *got = map(int, line.split())
        need = [32 * 40 + slots * 10, 32 * 40 + slots * 12, slots * 2, slots * 4]
        fits = [int(n <= LEFT) for n in need]
        left = [LEFT - (n + 7) // 8 * 8 * f for n, f in zip(need[2:], fits[2:])]
        assert got == fits + left
