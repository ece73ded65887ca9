"""The one-kernel repair in states that the public calls do not reach: started
from lists of the test's own, and with a barrier across the grid that gives up
(its failure word is set before the call, so its waits end at once)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "streamgc_b200", "lib")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    """tests/native/repair_probe.cu, built against the library."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("probe") / "repair_probe")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-o", exe, os.path.join(ROOT, "tests", "native", "repair_probe.cu"), "-L" + LIB, "-lstreamgc_b200",
                    "-Xlinker", "-rpath=" + LIB], check=True)

    def run(what):
        r = subprocess.run([exe, what], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr
    return run


def test_a_given_up_repair_is_an_error(probe):
    probe("status")


@pytest.mark.gpu
def test_publish_core_coloring_and_ticks_report_it_and_recover(probe):
    probe("give_up")


@pytest.mark.gpu
def test_lists_of_winners_and_lists_that_grow_again(probe):
    probe("lists")
