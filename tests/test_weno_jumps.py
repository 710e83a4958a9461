"""The reconstructions beside jumps (csrc/weno_fixed.cuh, csrc/weno_value.cuh), compiled for the host,
against long double."""
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


@pytest.mark.parametrize("decades", [-3, 0, 1, 2, 4, 6, 10, 14])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("z", [0, 1])
def test_small_side(lines, z, kind, decades):
    """A face's value on the small side of a jump, relative to that side: as exact as in FP64 (the rms
    over the same 20,000 stencils, whose scatter is 1 %; the worst of them to a factor of two)."""
    ((rms, rms64, worst, worst64),) = [[float(v) for v in x[4:]] for x in lines
                                       if x[0] == "sided" and x[1:4] == [str(z), str(kind), str(decades)]]
    assert rms <= 1.02 * rms64
    assert worst <= 2.0 * worst64


@pytest.mark.parametrize("z", [0, 1])
def test_forms(lines, z):
    """Odd, the same in either order, and a flat stencil's centre, in both arithmetics."""
    (row,) = [[int(v) for v in x[2:]] for x in lines if x[0] == "forms" and x[1] == str(z)]
    assert row[:3] == [0, 0, 0] and row[3] > 10000


@pytest.mark.parametrize("ratio", ["0.1", "2", "8", "100", "10000", "1e+08"])
def test_characteristic_fluxes(lines, ratio):
    """The characteristic schemes' fluxes beside jumps, each relative to its own small side: no less exact
    than an FP64 reconstruction of the fields' values (the worst to a factor of two)."""
    rows = [[float(v) for v in x[3:]] for x in lines if x[0] == "fields" and x[1] == ratio]
    assert len(rows) == 4
    for rms, rms64, worst, worst64 in rows:
        assert rms <= 1.02 * rms64
        assert worst <= 2.0 * worst64


@pytest.mark.parametrize("decades", [-3, 0, 2, 6, 10])
@pytest.mark.parametrize("delta", ["0", "0.001", "0.01", "0.5", "0.9"])
def test_borrowed_weights(lines, delta, decades):
    """AdaWENO's smooth branch, a component beside a jump with a smooth surrogate's weights (or, delta 0,
    with any surrogate's): no less exact than in FP64, as test_small_side."""
    ((rms, rms64, worst, worst64),) = [[float(v) for v in x[3:]] for x in lines
                                       if x[0] == "borrowed" and x[1:3] == [delta, str(decades)]]
    assert rms <= 1.02 * rms64
    assert worst <= 2.0 * worst64


@pytest.mark.parametrize("kind", range(4))
def test_flux_change(lines, kind):
    """The update's dt/dx dh_xi + dt/dy dh_eta, whatever lies between the directions' fluxes, differences
    and rates: no less exact than in FP64 relative to the larger product (two roundings there, one
    here), odd, and towards infinity where the result leaves the doubles' range."""
    ((odd, *errors),) = [x[2:] for x in lines if x[0] == "change" and x[1] == str(kind)]
    rms, rms64, worst, worst64 = map(float, errors)
    assert int(odd) == 0
    assert rms <= 1.02 * rms64
    assert worst <= 2.0 * worst64


@pytest.mark.parametrize("decades", [-2, -1, 0, 1, 4])
@pytest.mark.parametrize("kind", range(4))
@pytest.mark.parametrize("z", [0, 1])
def test_taped_gradient(lines, z, kind, decades):
    """The taped gradient on the exponent two stencils share: smooth ones, a jump in its own stencil, one
    in its partner, and rough ones, no less exact than weno_grad's (the worst to a factor of two)."""
    ((rms, rms64, worst, worst64),) = [[float(v) for v in x[4:]] for x in lines
                                       if x[0] == "taped" and x[1:4] == [str(z), str(kind), str(decades)]]
    assert rms <= 1.02 * rms64
    assert worst <= 2.0 * worst64


@pytest.mark.parametrize("decades", [0, 2, 4, 8])
def test_roe_means(lines, decades):
    """The Roe averages of two cells of very different density, relative to the mean of the magnitudes: two
    products and a sum, a sum and its reciprocal, their product, half an ulp each: 6 x 2^-53."""
    ((worst,),) = [x[2:] for x in lines if x[0] == "means" and x[1] == str(decades)]
    assert float(worst) <= 6.0
