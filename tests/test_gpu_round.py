"""The mixed factorisation's square roots and quotients (cg_round.cuh) round like sqrtf and divisions: every root of
[2^-60, 2^60] with its reciprocal, the values outside that are left to the library, and every divisor's significand
by 256 numerators, random ones and those at the ends of their binades."""
import os
import subprocess

import pytest

from conftest import ROOT

from cosmopp_gb300 import build

pytestmark = pytest.mark.gpu


def test_roots_and_quotients_are_rounded_to_the_nearest(tmp_path):
    exe = str(tmp_path / "test_round")
    subprocess.check_call([build._nvcc()] + build.ARCH + ["-O2", "-std=c++17", "-o", exe,
                                                          os.path.join(ROOT, "tests", "cxx", "test_round.cu")])
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stderr
    assert p.stdout.split() == ["0", "0", "0"]
