"""The buffer of pair products of a workspace: its share of a nearly full device, its bound, and the
dense I2O in every form that a smaller buffer selects (GPU).

A block of right-hand sides takes the plan of the largest units whose products fit the buffer for all
of them, then smaller units, then some right-hand sides at a time, and where that takes too many
passes, or there is no room for the smallest units, the kernels per receiving node. The bounds below
select each of these on maps of 47 and 57 MiB of products a right-hand side (units of all pairs, 32,
16 and 4 MiB).

Tolerances: FP64 sums of O(1) terms keep 1e-12 relative by three orders of magnitude, in whatever
order; FP32 storage and TF32-split products with 64-value FP32 segments keep 1e-6.
"""

import copy

import numpy as np
import pytest
import torch

import h2factory_b200 as h2
from h2factory_b200 import _abi
from oracle import oracle
from test_gpu_pairs_i2o import _core, _product, _x, rel

pytestmark = pytest.mark.gpu

MIB = 1 << 20
VIEWS = (lambda w: w, h2.transpose, h2.adjoint)


def _fp32(core):
    c = copy.copy(core)
    c.precision = "fp32"
    return c


def test_nearly_full_device_keeps_its_free_memory():
    """What a program allocates after the workspace still finds room."""
    nrhs = 64
    core = _core(6, 900, True, True)
    dcore = h2.DeviceCore(core)
    x = _x(core, nrhs, 1)
    ws = h2.H2Workspace(dcore, max_nrhs=nrhs)
    want = _product(h2.mul_, ws, core, x)
    ws.close()
    n = core.test.npoints
    arenas = (2 * dcore.info().moment_elems + 4 * n) * nrhs * 16 + 32 * MIB
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 1536 * MIB, dtype=torch.uint8, device="cuda")
    try:
        before = torch.cuda.mem_get_info()[0]
        ws = h2.H2Workspace(dcore, max_nrhs=nrhs)
        assert before - torch.cuda.mem_get_info()[0] < arenas + before // 8
        assert 0 < ws.product_bytes <= before // 16
        assert rel(_product(h2.mul_, ws, core, x), want) < 1e-12
        ws.close()
    finally:
        del fill
        torch.cuda.empty_cache()


def test_bound_and_size():
    core = _core(6, 900, True, True)
    dcore = h2.DeviceCore(core)
    for limit, least in ((0, 0), (5 * MIB, 5 * MIB), (1 << 62, 15 * MIB)):
        ws = h2.H2Workspace(dcore, max_nrhs=1, max_product_bytes=limit)
        assert least <= ws.product_bytes <= min(limit, 20 * MIB)
        twin = h2.similarworkspace(ws)
        assert twin.product_bytes == ws.product_bytes
        twin.close()
        ws.close()
    with pytest.raises(_abi.H2BError) as err:
        h2.H2Workspace(dcore, max_nrhs=1, max_product_bytes=-1)
    assert err.value.status == _abi.H2B_ERR_INVALID


@pytest.mark.parametrize("p,n,cplx,symmetry", [(6, 1800, True, True), (4, 6000, False, False)])
def test_smaller_buffers_give_the_same_product(p, n, cplx, symmetry):
    nrhs = 16
    core = _core(p, n, cplx, symmetry, leaf=16 if p == 6 else 32)
    x = _x(core, nrhs, 5)
    for c in (core, _fp32(core)):
        dcore = h2.DeviceCore(c)
        full = h2.H2Workspace(dcore, max_nrhs=nrhs)
        for mode, view in enumerate(VIEWS):
            want = _product(h2.mul_, view(full), c, x)
            if c is core:
                assert rel(want[:, :2], oracle.matvec(core, np.asfortranarray(x[:, :2]), mode)) < 1e-12, mode
            for mib in (256, 64, 32, 12, 5, 0):
                ws = h2.H2Workspace(dcore, max_nrhs=nrhs, max_product_bytes=mib * MIB)
                got = _product(h2.mul_, view(ws), c, x)
                assert rel(got, want) < (1e-12 if c is core else 1e-6), (c.precision, mode, mib)
                ws.close()
        full.close()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("p,symmetry", [(2, True), (3, False), (4, True), (5, False), (6, True)])
def test_kernels_per_receiving_node(p, symmetry, cplx):
    """No buffer: FP64 sums per receiving node in the FP64 form and for few columns of the FP32 form, the
    tcgen05 kernel for wider blocks of it."""
    core = _core(p, 900, cplx, symmetry)
    for nrhs in (1, 5, 17):
        x = _x(core, nrhs, nrhs)
        w64, w32 = (h2.H2Workspace(c, max_nrhs=nrhs, max_product_bytes=0) for c in (core, _fp32(core)))
        for mode, view in enumerate(VIEWS):
            y = _product(h2.mul_, view(w64), core, x)
            assert rel(y, oracle.matvec(core, x, mode)) < 1e-12, (nrhs, mode)
            assert rel(_product(h2.mul_, view(w32), core, x), y) < 1e-6, (nrhs, mode)
        w64.close()
        w32.close()
