"""The sweeps' tiles and threads per interface follow the grid's size; the arithmetic of an interface
does not, so every choice must give the same bits: at the sizes around each line of the choice and with
the last tile of a line holding one interface, few, or all."""
import ctypes

import numpy as np
import pytest

from conftest import interior
from test_gpu_batch import batch_cfgs, plain

pytestmark = pytest.mark.gpu


# component-wise: the batch's own tiles against the single solve's, either side of its line
@pytest.mark.parametrize("split,recon,sizes", [
    (101, 253, [(359, 359), (360, 360), (383, 351), (321, 415)]),
    (102, 255, [(383, 352), (320, 407)]),
    (101, 253, [(16, 131075)]),  # more rows of tiles than a grid's y holds
    (103, 255, [(258, 258), (260, 258), (319, 287)]),
])
def test_component_wise_tiles(dense, split, recon, sizes):
    cfgs = batch_cfgs(dense, split, recon, sizes)
    with dense.BatchSolver.from_setups(cfgs) as b:
        b.steps(2)
        for i, cfg in enumerate(cfgs):
            ref = plain(dense, cfg, 2)[0]
            np.testing.assert_array_equal(interior(b.download(i)), interior(ref), err_msg=str(sizes[i]))


# AdaWENO: counting the branches takes the small-grid tiles on every grid
@pytest.mark.parametrize("ni,nj", [(283, 283), (319, 255), (320, 256), (1921, 47)])
def test_adaptive_tiles(dense, ni, nj):
    cfg = dense.config_default(ni=ni, nj=nj, benchmark=5, splitting=105, recon=0, cfl=0.5)
    out = []
    for counting in (0, 1):
        c, cons, prim, x, y = dense.init_general(cfg)
        with dense.Solver(c) as s:
            s.upload(cons, prim, x, y)
            s.lib.dense_count_branches(s.h, counting)
            s.steps(3)
            out.append(interior(s.download(False)).copy())
            counts = (ctypes.c_ulonglong * 8)()
            s.lib.dense_get_branch_counts(s.h, counts)
    np.testing.assert_array_equal(out[0], out[1])
    # every interface and sign of three steps' nine stages was counted once
    assert counts[0] + counts[1] == 18 * (ni + 1) * nj and counts[4] + counts[5] == 18 * ni * (nj + 1)
