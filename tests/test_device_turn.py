"""The order of grids whose blocks wait for one another (csrc/device_turn.hpp),
on the CPU: two threads launch finite grids, two others step without a pause
and stay on the device where they may. No two grids overlap, none overlaps a
stay, every launch gets its turn, and stepping goes on meanwhile."""

import os
import subprocess

import nemo_b200.build as b

HERE = os.path.dirname(os.path.abspath(__file__))


def test_waiting_grids_never_overlap(tmp_path):
    exe = str(tmp_path / "device_turn_check")
    subprocess.check_call([b.CXX, "-std=c++17", "-O1", "-g", "-pthread", "-Wall", *b.INCLUDES,
                           os.path.join(HERE, "device_turn_check.cpp"), os.path.join(b.CSRC, "device_turn.cpp"),
                           "-o", exe])
    for _ in range(3):
        r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
        assert r.stdout.strip() == "ok", r.stdout + r.stderr
