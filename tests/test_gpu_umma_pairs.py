"""The FP32 form's dense I2O by stored block on the tcgen05 tensor cores (GPU): edges of its tiles.

An item is a tile of pairs that read one block through one permutation: 128 rows of the block, 64
product columns (pairs x right-hand sides; Re and Im columns in complex maps). The sizes here are
those where a tile can go wrong: one partial row tile (64 and 125 coefficients), two (216), block
columns that are not whole 16-byte multiples (125: copied with padded columns), items of 2, 4, 8 and
14 chunks, column counts below one tile, filling it and running into further ones, every
orientation, with and without permutations; and several units of receiving nodes
(h2b_farmul_noalloc). Compared with the FP64 form: FP32 storage and TF32-split products with
64-value FP32 segments keep 1e-6.
"""

import copy
import ctypes as C

import numpy as np
import pytest
import torch

import h2factory_b200 as h2
from h2factory_b200 import _abi, methods
from h2factory_b200.trees import build_tree
from test_gpu_pairs_i2o import _core, _product, _x, rel

pytestmark = pytest.mark.gpu


def _fp32(core):
    c = copy.copy(core)
    c.precision = "fp32"
    return c


@pytest.mark.parametrize("p,cplx,symmetry,widths", [(4, False, False, (5, 32, 33)), (4, True, True, (3, 16, 17)),
                                                    (5, False, True, (6, 64)), (5, True, True, (5, 33)),
                                                    (6, True, True, (3, 8, 33))])
def test_tile_edges_match_fp64(p, cplx, symmetry, widths):
    core = _core(p, 900, cplx, symmetry)
    timeouts = _abi.tensor_wait_timeouts(0)
    for nrhs in widths:
        w64, w32 = h2.H2Workspace(core, max_nrhs=nrhs), h2.H2Workspace(_fp32(core), max_nrhs=nrhs)
        x = _x(core, nrhs, nrhs)
        for view in (lambda w: w, h2.transpose, h2.adjoint):
            y = _product(h2.mul_, view(w32), core, x)
            assert rel(y, _product(h2.mul_, view(w64), core, x)) < 1e-6, nrhs
            assert np.array_equal(y, _product(h2.mul_, view(w32), core, x)), nrhs  # the same bits again
        w64.close()
        w32.close()
    assert _abi.tensor_wait_timeouts(0) == timeouts  # no bounded wait gave up


def test_units_of_receiving_nodes():
    rng = np.random.default_rng(9)
    tree = build_tree(rng.random((6000, 3)), maxvalues=48, root_center=[0.5] * 3, root_halfsize=0.5)
    core = methods.interpolation_core(tree, methods.helmholtz(2.0), 4, symmetry=True, precision="fp32")
    assert len(core.plans.far) * 64 * 16 > 2 * (4 << 20)
    ws = h2.H2Workspace(core, max_nrhs=3)
    x = _x(core, 3, 4)
    lib = _abi.load_library()
    n = core.trial.npoints
    for mode, A in ((0, ws), (1, h2.transpose(ws)), (2, h2.adjoint(ws))):

        def noalloc(y, _, xd):
            st = lib.h2b_farmul_noalloc(ws.dcore.handle, mode, 3, C.c_void_p(xd.data_ptr()), n,
                                        C.c_void_p(y.data_ptr()), n, None, None,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0, lib.h2b_last_error().decode()

        # the same segments; FP64 sums in another order before one rounding to FP32
        assert rel(_product(noalloc, None, core, x), _product(h2.farmul_, A, core, x)) < 1e-9, mode
    ws.close()
