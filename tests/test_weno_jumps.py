"""The reconstructions beside jumps (csrc/weno_fixed.cuh), compiled for the host, against long double."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("wj") / "driver")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "weno_jumps_driver.cpp")], check=True)
    out = subprocess.run([exe], check=True, stdout=subprocess.PIPE).stdout.decode()
    return [x.split() for x in out.splitlines()]


@pytest.mark.parametrize("z", [0, 1])
def test_between_two_jumps(lines, z):
    """A smooth middle between two jumps of different sizes: 16 x 2^-53 of the largest value, as for any
    stencil (test_weno_fixed.py), and never smooth to AdaWENO's switch."""
    ((worst, smooth),) = [x[2:] for x in lines if x[0] == "between" and x[1] == str(z)]
    assert float(worst) <= 16 * 2.0 ** -53
    assert int(smooth) == 0
