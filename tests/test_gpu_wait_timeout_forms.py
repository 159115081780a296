"""The timeout path of the bounded waits in every form of the tcgen05 I2O (GPU).

The forms differ in the warps that wait and in the copies that have to land before a CTA may leave:
per receiving node with columns by TMA gather (216 real coefficients) and with columns read from
global memory (27), by stored block with moments by TMA (64) and by cp.async (125). The bound is
lowered to one attempt, so that waits give up; nothing faults or hangs. The product has to be reported
as incomplete, and the same workspace has to give a correct one again with the default bound.

Tolerance: FP32 storage and TF32-split products with 64-value FP32 segments keep 1e-6 of the FP64 form.
"""

import copy

import numpy as np
import pytest

import h2factory_b200 as h2
from h2factory_b200 import _abi
from test_gpu_pairs_i2o import _core, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [3, 4, 5, 6])
def test_timeout_reported_and_recovered(p):
    core = _core(p, 2000, False, True)
    c32 = copy.copy(core)
    c32.precision = "fp32"
    x = np.asfortranarray(np.random.default_rng(p).standard_normal((2000, 12)))
    ws64, ws32 = h2.H2Workspace(core, max_nrhs=12), h2.H2Workspace(c32, max_nrhs=12)
    want = ws64.matvec_host(x)
    before = _abi.tensor_wait_timeouts(0)
    try:
        _abi.set_tensor_wait_limit(1)
        with pytest.raises(_abi.H2BError) as err:
            ws32.matvec_host(x)
        assert err.value.status == _abi.H2B_ERR_CUDA and "gave up" in str(err.value)
        assert _abi.tensor_wait_timeouts(0) > before
    finally:
        _abi.set_tensor_wait_limit(0)
    after = _abi.tensor_wait_timeouts(0)
    assert rel(ws32.matvec_host(x), want) < 1e-6
    assert _abi.tensor_wait_timeouts(0) == after
    ws64.close()
    ws32.close()
