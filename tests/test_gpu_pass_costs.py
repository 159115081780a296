"""The dense I2O never takes more passes over a small buffer of pair products than pay (GPU).

Far products whose buffer holds few products (h2b_farmul_noalloc's scratch), and wide blocks of small
coefficient counts in the FP32 form, against the kernels per receiving node (a workspace without a
buffer), which such products fall back to: at most a quarter longer. Passes that do not pay are 1.5 to
14 times as long on these maps (55,748 pairs).
"""

import ctypes as C

import numpy as np
import pytest
import torch

import h2factory_b200 as h2
from h2factory_b200 import methods
from h2factory_b200.trees import build_tree

pytestmark = pytest.mark.gpu


def _case(p, cplx, precision, nrhs):
    tree = build_tree(np.random.default_rng(0).random((6000, 3)), maxvalues=64, root_center=[0.5] * 3, root_halfsize=0.5)
    core = methods.interpolation_core(tree, methods.helmholtz(3.0) if cplx else methods.laplace, p, symmetry=True,
                                      precision=precision, near="free")
    dt = torch.complex128 if cplx else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((nrhs, 6000), dtype=dt, device="cuda", generator=gen).t()
    return h2.DeviceCore(core), x, torch.zeros((nrhs, 6000), dtype=dt, device="cuda").t()


def _ms(call):
    times = []
    for _ in range(12):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        call()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return min(times[2:])


def _far(dcore, x, y, limit):
    ws = h2.H2Workspace(dcore, max_nrhs=x.shape[1], max_product_bytes=limit)
    ms = _ms(lambda: h2.farmul_(y, ws, x))
    out = y.clone()
    ws.close()
    return ms, out


def _close(a, b, precision):
    return torch.linalg.vector_norm(a - b) < (1e-12 if precision == "fp64" else 1e-6) * torch.linalg.vector_norm(b)


@pytest.mark.parametrize("p,cplx,precision,nrhs", [
    (2, False, "fp64", 16), (3, True, "fp64", 16), (4, False, "fp64", 16), (4, True, "fp64", 8),
    (3, True, "fp32", 32), (4, False, "fp32", 32), (4, True, "fp32", 5), (5, False, "fp32", 16)])
def test_noalloc_against_the_kernels_per_node(p, cplx, precision, nrhs):
    dcore, x, y = _case(p, cplx, precision, nrhs)
    node, want = _far(dcore, x, y, 0)

    def noalloc():
        assert dcore.lib.h2b_farmul_noalloc(dcore.handle, 0, nrhs, C.c_void_p(x.data_ptr()), 6000, C.c_void_p(y.data_ptr()),
                                            6000, None, None,
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0

    assert _ms(noalloc) < 1.25 * node
    assert _close(y, want, precision)


def test_whole_buffer_for_wide_blocks_of_many_coefficients():
    """Several passes that do pay: about four fifths of the time per receiving node."""
    dcore, x, y = _case(6, True, "fp32", 64)
    node, want = _far(dcore, x, y, 0)
    full, got = _far(dcore, x, y, 1 << 62)
    assert full < node
    assert _close(got, want, "fp32")


def test_wide_blocks_of_few_coefficients():
    dcore, x, y = _case(3, True, "fp32", 32)
    node, want = _far(dcore, x, y, 0)
    full, got = _far(dcore, x, y, 1 << 62)
    assert full < 1.25 * node
    assert _close(got, want, "fp32")
