"""The integer WENO reconstructions (csrc/weno_fixed.cuh), compiled for the host, against long
double and beside the FP64 form (csrc/weno_fast.cuh): no less exact over smooth, discontinuous and
rough stencils, and the same answers in every form an input can take."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("wf") / "driver")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "weno_fixed_driver.cpp")], check=True)
    out = subprocess.run([exe], check=True, stdout=subprocess.PIPE).stdout.decode()
    return [x.split() for x in out.splitlines()]


def test_reciprocal(lines):
    (worst,) = [float(x[1]) for x in lines if x[0] == "reciprocal"]
    assert worst <= 2.0 ** -58


@pytest.mark.parametrize("kind", range(5))
@pytest.mark.parametrize("z", [0, 1])
def test_accuracy(lines, kind, z):
    """In units of the stencils' largest value S: the centres' sum rounds by 2^-52, the result (at
    most 4.3 S) by 2.2 x 2^-52, the differences by 2^-52 each with sensitivities of 4 in all: 16 x
    2^-53. The rms no larger than the FP64 form's on the same stencils."""
    _, _, _, worst, rms, worst64, rms64 = [x for x in lines if x[0] == "accuracy" and x[1:3] == [str(z), str(kind)]][0]
    assert float(worst) <= 16 * 2.0 ** -53
    assert float(rms) <= float(rms64)


@pytest.mark.parametrize("z", [0, 1])
def test_forms(lines, z):
    """Signs and the two stencils' order leave the bits alone, flat stencils give their centre, a
    NaN or infinity gives NaN, and magnitudes from 1e-180 to 1e90 keep their accuracy."""
    _, _, odd, swap, flat, bad, n, scale_err = [x for x in lines if x[0] == "forms" and x[1] == str(z)][0]
    assert (int(odd), int(swap), int(flat), int(bad)) == (0, 0, 0, 0)
    assert int(n) > 1000 and float(scale_err) <= 1.0


def test_adaptive(lines):
    """AdaWENO's switch equals theta > delta away from the threshold (within the rounding of the
    surrogate's values), delta's two ends and a NaN decide it, and a stencil reconstructed with the
    surrogate's weights is exact to a few roundings."""
    n, wrong, near, ends, nans, smooth, worst = [float(v) for v in [x for x in lines if x[0] == "adaptive"][0][1:]]
    assert (wrong, ends, nans) == (0, 0, 0)
    assert near < 0.1 * n and 0.05 * n < smooth < 0.95 * n
    assert worst <= 16 * 2.0 ** -53


def test_roots(lines):
    """Reciprocal, inverse square root and square root: values good to 2^-58, rounded once, so half an
    ulp and 2^-5 of one; a NaN outside their ranges."""
    (row,) = [x[1:] for x in lines if x[0] == "roots"]
    assert max(float(v) for v in row[:3]) <= 0.5 + 2.0 ** -5 and int(row[3]) == 0


def test_flux_change(lines):
    """The update's dt/dx dh_xi + dt/dy dh_eta: the rates' own rounding aside, truncations of 2^-57 and
    one rounding of the result, half an ulp; twice that bounds it. Odd in the fluxes and under a
    mirror image, zero for equal fluxes, NaN for what is not finite."""
    ((worst, odd, bad),) = [x[1:] for x in lines if x[0] == "change"]
    assert float(worst) <= 2.0 and int(odd) == 0 and int(bad) == 0


def test_conversion(lines):
    """Fixed point to double is a nearest rounding at every width, up to the next power of two too."""
    assert [x[1] for x in lines if x[0] == "conversion"] == ["0"]


@pytest.mark.parametrize("kind", range(5))
@pytest.mark.parametrize("z", [0, 1])
def test_gradient(lines, kind, z):
    """The taped gradient's rms error is that of weno_grad or less, up to a quarter more (its fixed-point
    differences know a stencil's smoothest part to 2^-55 of the largest one's, kRough bits less than
    FP64's 2^-53 of themselves); the value is the plain sweep's to the bit; the gradient is even."""
    (row,) = [x[3:] for x in lines if x[0] == "gradient" and x[1:3] == [str(z), str(kind)]]
    assert float(row[0]) <= 1.25 * float(row[1])
    assert int(row[3]) == 0 and int(row[4]) == 0
