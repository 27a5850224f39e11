"""Row masks of the small closure's cluster (csrc/cluster_rows.cuh) simulated on
the CPU: every warp of every CTA must count the same rows after a cluster barrier,
since it decides from them whether to leave or to wait at the next one."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def simulate(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("cluster") / "cluster_rows")
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "cfpq-on-gpgpu_b200", "csrc"), "-o",
                    exe, os.path.join(ROOT, "tests", "cpp", "cluster_rows_main.cpp")], check=True)

    def run(*args):
        p = subprocess.run([exe, *args], capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stdout
        return tuple(map(int, p.stdout.split()))

    return run


def test_every_warp_decides_alike(simulate):
    decisions, wrong = simulate("2000")
    assert decisions == 2000 * 8 * 6 and wrong == 0


def test_the_simulation_sees_masks_written_from_outside(simulate):
    """The mistake that the protocol rules out, planted in the simulation."""
    assert simulate("2000", "shared")[1] > 0
