"""A batch's buffers of pair products share a part of the free device memory (GPU).

Every map of a batch holds its own buffer, up to 512 MiB: a batch of hundreds of maps must not spend
on them what its further workspaces need. The device's free memory is reported small here, as it is to
the batch beside many maps.

Tolerance: FP64 sums of O(1) terms keep 1e-12 relative by three orders of magnitude.
"""

import numpy as np
import pytest
import torch

from h2factory_b200 import batch
from oracle import oracle
from test_gpu_pairs_i2o import _core, _x, rel

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def test_buffers_stay_within_a_share_of_the_free_memory(monkeypatch):
    cores = [_core(p, 900, cplx, True) for p, cplx in ((6, True), (6, False), (5, True), (5, False))]
    nrhs = [3, 4, 5, 6]
    free = 64 * MIB
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (free, 180 << 30))
    maps = batch.BatchedMaps(cores, nrhs)
    sizes = [ws.product_bytes for ws in maps.ws]
    assert min(sizes) > 0 and sum(sizes) <= free // 4
    xs = [_x(c, r, r) for c, r in zip(cores, nrhs)]
    maps.set_inputs([torch.from_numpy(np.ascontiguousarray(x)) for x in xs])
    maps.capture()
    maps.replay()
    torch.cuda.synchronize()
    for core, x, y in zip(cores, xs, maps.outputs):
        assert rel(y.cpu().numpy(), oracle.matvec(core, x, 0)) < 1e-12
    maps.close()
