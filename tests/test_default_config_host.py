"""CPU check of the configuration rule of new FP64 handles (no GPU): its edges,
and that every sector has a two-pass configuration where the fused form, which
needs thread-block clusters, cannot run."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "dmrgpp_b200", "csrc")


def test_default_configuration_rule(tmp_path):
    exe = str(tmp_path / "default_config_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    os.path.join(HERE, "default_config_check.cpp"), os.path.join(CSRC, "kron_plan.cpp"),
                    "-o", exe, "-lpthread"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
