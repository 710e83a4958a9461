"""The register bounds of the launch configurations were chosen on the fast kernels; the strict 104 sweeps,
four-thread component-wise sweeps and update keep theirs. Read from the compiler's resource report of the build."""
import os
import re

import pytest


def spills(dense, unit, kernel):
    log = os.path.join(os.path.dirname(dense.__file__), "csrc", "_build", f"ptxas_{unit}.log")
    if not os.path.exists(log):
        pytest.skip("the library was not built here")
    with open(log) as f:
        text = f.read()
    out = {}
    for m in re.finditer(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores", text, re.S):
        if kernel in m.group(1):
            out[m.group(1)] = int(m.group(2))
    assert out
    return out


# (k_flux_char<DIR, ADAPT = false, ...>: 104; AdaWENO's 80 registers bind every variant, as measured)
@pytest.mark.parametrize("kernel", ["k_flux_charILi0ELb0", "k_flux_charILi1ELb0", "9k_flux_cw", "8k_update"])
def test_strict_kernels_do_not_spill(dense, kernel):
    assert set(spills(dense, "kernels_strict", kernel).values()) == {0}
