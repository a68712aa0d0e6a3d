"""The decisions of a one-launch solve, compiled for the host: CTAs that leave a grid barrier at
different times take the same ones (the reference decides on the host, GraphCut.pyx:348-418)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cl-util_b200", "csrc")


def test_ctas_agree_on_every_step(tmp_path):
    exe = str(tmp_path / "solve_schedule_sim")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "solve_schedule_sim.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
