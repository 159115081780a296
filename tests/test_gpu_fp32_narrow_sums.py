"""Up to 4 field columns of the FP32 form have FP64 sums (GPU).

A column's sums run over the same terms in the same order whatever stands beside it, so the first
columns of blocks of 2, 3 and 4 real right-hand sides have equal bits: with the
FP32 segments of the tcgen05 kernels, which take wider blocks, they differ. The dispatch is what is
tested, so nothing is left to a tolerance.
"""

import copy

import numpy as np
import pytest

import h2factory_b200 as h2
from test_gpu_pairs_i2o import _core, _product, _x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [4, 5, 6])
def test_columns_keep_their_bits_up_to_four(p):
    core = copy.copy(_core(p, 900, False, True))
    core.precision = "fp32"
    x = _x(core, 5, 3)
    ws = h2.H2Workspace(core, max_nrhs=5)
    for view in (lambda w: w, h2.transpose):
        outs = [_product(h2.farmul_, view(ws), core, x[:, :r]) for r in (2, 3, 4, 5)]
        for y in outs[1:-1]:
            assert np.array_equal(y[:, :2], outs[0][:, :2])
        assert not np.array_equal(outs[-1][:, :2], outs[0][:, :2])
    ws.close()
