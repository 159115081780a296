"""The buffer of pair products of a workspace: its share of a nearly full device and its bound (GPU)."""

import pytest
import torch

import h2factory_b200 as h2
from h2factory_b200 import _abi
from test_gpu_pairs_i2o import _core, _product, _x, rel

pytestmark = pytest.mark.gpu

MIB = 1 << 20


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
        ws.close()
    with pytest.raises(_abi.H2BError) as err:
        h2.H2Workspace(dcore, max_nrhs=1, max_product_bytes=-1)
    assert err.value.status == _abi.H2B_ERR_INVALID
