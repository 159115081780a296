"""The dense I2O by stored block with FP64 sums (GPU): edges of its tiles.

Every stored block is multiplied by the moments of all the pairs that read it, 72 rows and 64
columns (pairs x right-hand sides) at a time, 8 or 16 coefficients of k per stage, and every
receiving node then adds its pairs' products. The maps here take the sizes where that can go wrong:
coefficient counts below one row tile (8, 27), at 64, above it with a partial last 8-row block
(125) and of three whole tiles (216), none of 8, 27 and 125 a multiple of the stage; column counts
of 1, of a partial and of several column tiles; both orientations of the block, with and without
permutations; the storage types of both forms. FP64 against the oracle, the FP32 form (FP64 sums of
FP32 moments and blocks) against FP64.

Tolerances: FP64 sums of at most 216 x 189 products of O(1) terms keep 1e-12 relative by three
orders of magnitude; FP32 storage rounds moments, blocks and collections once each (6e-8), so 1e-6.
"""

import copy
import ctypes as C

import numpy as np
import pytest
import torch

import h2factory_b200 as h2
from h2factory_b200 import _abi, methods
from h2factory_b200.trees import build_tree
from oracle import oracle

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _core(p, n, cplx, symmetry, leaf=16):
    rng = np.random.default_rng(100 * p + n)
    tree = build_tree(rng.random((n, 3)) * [1.0, 0.9, 0.3], maxvalues=leaf, root_center=[0.5] * 3, root_halfsize=0.5)
    kernel = methods.helmholtz(3.0) if cplx else methods.laplace
    return methods.interpolation_core(tree, kernel, p, symmetry=symmetry, transfers="separable")


def _product(fn, A, core, x):
    dt = torch.complex128 if core.field == "complex" else torch.float64
    xd = torch.from_numpy(np.ascontiguousarray(x.T)).to(DEV).t()
    y = torch.zeros((x.shape[1], core.test.npoints), dtype=dt, device=DEV).t()
    fn(y, A, xd)
    torch.cuda.synchronize()
    return y.cpu().numpy()


def _x(core, k, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((core.trial.npoints, k))
    return x + 1j * rng.standard_normal(x.shape) if core.field == "complex" else x


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("p,symmetry,nrhs", [(2, False, 5), (3, True, 1), (4, False, 33), (5, True, 7), (6, True, 65)])
def test_tile_edges_match_oracle(p, symmetry, nrhs, cplx):
    core = _core(p, 900, cplx, symmetry)
    ws = h2.H2Workspace(core, max_nrhs=nrhs)
    x = _x(core, nrhs, p)
    for mode, A in ((0, ws), (1, h2.transpose(ws)), (2, h2.adjoint(ws))):
        y = _product(h2.mul_, A, core, x)
        assert rel(y, oracle.matvec(core, x, mode)) < 1e-12, mode
        assert np.array_equal(y, _product(h2.mul_, A, core, x)), mode  # no atomics: the same bits again
    ws.close()


@pytest.mark.parametrize("cplx", [False, True])
def test_fp32_storage_with_fp64_sums(cplx):
    core = _core(5, 900, cplx, True)
    c32 = copy.copy(core)
    c32.precision = "fp32"
    for nrhs in (1, 2) if cplx else (1, 3, 4):
        x = _x(core, nrhs, nrhs)
        w64, w32 = h2.H2Workspace(core, max_nrhs=nrhs), h2.H2Workspace(c32, max_nrhs=nrhs)
        for view in (lambda w: w, h2.transpose, h2.adjoint):
            assert rel(_product(h2.mul_, view(w32), c32, x), _product(h2.mul_, view(w64), core, x)) < 1e-6
        w64.close()
        w32.close()


def test_units_of_receiving_nodes():
    """More pair products than the allocation-free call's buffer holds: several units of receiving
    nodes, each with its own tiles, give the workspace call's far product."""
    core = _core(4, 6000, False, False, leaf=32)
    assert len(core.plans.far) * 64 * 8 > 2 * (4 << 20)
    ws = h2.H2Workspace(core, max_nrhs=2)
    x = _x(core, 2, 3)
    lib = _abi.load_library()
    n = core.trial.npoints
    for mode, A in ((0, ws), (1, h2.transpose(ws)), (2, h2.adjoint(ws))):
        want = _product(h2.farmul_, A, core, x)

        def noalloc(y, _, xd):
            st = lib.h2b_farmul_noalloc(ws.dcore.handle, mode, 2, C.c_void_p(xd.data_ptr()), n,
                                        C.c_void_p(y.data_ptr()), n, None, None,
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0, lib.h2b_last_error().decode()

        assert rel(_product(noalloc, None, core, x), want) < 1e-14 * 100, mode
    ws.close()
