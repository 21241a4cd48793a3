"""The fixed-point words that the pair kernels add to their histograms
(corr_pc_gb300/csrc/df32.cuh), built for the host: terms within half a quantum,
words within the range that a bin's term limit relies on, and a bin filled to that
limit with the largest words read back exactly."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_fixed_point_words(tmp_path):
    exe = str(tmp_path / "fixed_words")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "corr_pc_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "fixed_words_driver.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "BAD" not in r.stdout, r.stdout + r.stderr
