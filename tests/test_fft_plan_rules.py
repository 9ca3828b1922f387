"""Host rules over FFT plans at the shortest transform (length 1 has no stage):
tests/cuda/plan_checks.cu evaluates them at compile time, where reading outside a
plan's arrays is an error (no GPU needed)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_rules_stay_inside_the_plan(tmp_path):
    from phaser_b200 import build
    cmd = [build.nvcc()] + build.ARCH + build.NVCC_FLAGS + ["-c", os.path.join(HERE, "cuda", "plan_checks.cu"), "-o",
                                                            str(tmp_path / "plan_checks.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
