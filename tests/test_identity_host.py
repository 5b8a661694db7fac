"""CPU check of the FP64 H*x on sectors with identity blocks (no GPU): the work
list, in which a term with an identity factor is one product that skips
pass 1, replayed by identity_schedule_check.cpp against H*x with the
identities multiplied out."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "dmrgpp_b200", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("identity") / "identity_schedule_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    os.path.join(HERE, "identity_schedule_check.cpp"),
                    os.path.join(CSRC, "kron_plan.cpp"), "-o", exe, "-lpthread"], check=True)
    return exe


# one state; whole tiles and their edges; many small patches; wide ones
@pytest.mark.parametrize("seed,np_,maxs", [(1, 1, 1), (2, 3, 9), (3, 5, 33), (4, 3, 65), (5, 14, 12), (6, 2, 140)])
def test_identity_terms(checker, seed, np_, maxs):
    out = subprocess.run([checker, str(seed), str(np_), str(maxs)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
    if maxs > 1:
        assert int(out.stdout.split()[2]) > 0
