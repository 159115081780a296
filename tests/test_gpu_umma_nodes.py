"""The FP32 form's dense I2O per receiving node on the tcgen05 tensor cores (GPU): chunk counts and tiles.

Blocks of an odd number of 32-value chunks keep this form, since an accumulation segment of two
chunks runs on into the next pair. Three moment warps take every third chunk each, so a warp skips
pairs of one chunk (8 and 27 real coefficients, 8 complex ones) and starts those of seven (216
real) at its first, second or third chunk; an interaction list may be shorter than three chunks.
Right-hand sides below, at and past a tile's 64 (complex: 32), both orientations, with and without
permutations. Compared with the FP64 form: FP32 storage and TF32-split products with 64-value FP32 segments keep 1e-6.
"""

import copy

import numpy as np
import pytest

import h2factory_b200 as h2
from h2factory_b200 import _abi
from test_gpu_pairs_i2o import _core, _product, _x, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,cplx,symmetry,widths", [(2, False, False, (5, 64)), (2, True, True, (3, 33)),
                                                    (3, False, True, (5, 17)), (6, False, True, (5, 12, 65)),
                                                    (6, False, False, (16,))])
def test_chunk_counts_match_fp64(p, cplx, symmetry, widths):
    core = _core(p, 900, cplx, symmetry)
    c32 = copy.copy(core)
    c32.precision = "fp32"
    timeouts = _abi.tensor_wait_timeouts(0)
    for nrhs in widths:
        w64, w32 = h2.H2Workspace(core, max_nrhs=nrhs), h2.H2Workspace(c32, max_nrhs=nrhs)
        x = _x(core, nrhs, nrhs)
        for view in (lambda w: w, h2.transpose, h2.adjoint):
            y = _product(h2.mul_, view(w32), core, x)
            assert rel(y, _product(h2.mul_, view(w64), core, x)) < 1e-6, nrhs
            assert np.array_equal(y, _product(h2.mul_, view(w32), core, x)), nrhs  # the same bits again
        w64.close()
        w32.close()
    assert _abi.tensor_wait_timeouts(0) == timeouts  # no bounded wait gave up
