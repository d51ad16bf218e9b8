"""The drain of a TMA ring after a bounded wait ran out: no load may still be in
flight when the CTA ends (its shared memory goes to the next one).  A host
model of the stage barriers, built with g++ on the kernels' own bookkeeping
(spk_ring.cuh): no GPU, and no failing wait, is involved."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("kernel", ["line", "axis"])
def test_drain_covers_the_loads_in_flight(kernel, tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "ring_drain")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "spooky-git_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "ring_drain.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, kernel], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["in_flight", "0", "idle_waits", "0"]
