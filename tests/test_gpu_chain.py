"""One-column products whose far passes are launched ahead of each other (GPU).

The kernels of such a product start while the one before still runs and wait for it before they read
its results, so products queued back to back, eager and from a graph, each have to see their own
moments. Maps of one level of transfers and of several, dense and separable, with launches below and
above the limit on blocks (the product kernel of 30,000 points has more than 2,368).

Tolerance: FP64 sums of at most 216 x 189 products of O(1) terms keep 1e-12 relative by three orders
of magnitude.
"""

import numpy as np
import pytest
import torch

import h2factory_b200 as h2
from h2factory_b200 import methods
from h2factory_b200.trees import build_tree
from oracle import oracle

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("n,leaf,cplx,transfers", [(150, 16, False, "dense"), (3000, 8, True, "separable"),
                                                   (3000, 8, False, "dense"), (30000, 16, False, "separable")])
def test_queued_products_see_their_own_moments(n, leaf, cplx, transfers):
    rng = np.random.default_rng(n)
    tree = build_tree(rng.random((n, 3)), maxvalues=leaf, root_center=[0.5] * 3, root_halfsize=0.5)
    core = methods.interpolation_core(tree, methods.helmholtz(3.0) if cplx else methods.laplace, 3, transfers=transfers)
    ws = h2.H2Workspace(core, max_nrhs=1)
    x = rng.standard_normal((n, 4))
    if cplx:
        x = x + 1j * rng.standard_normal(x.shape)
    for mode, A in ((0, ws), (2, h2.adjoint(ws))):
        want = oracle.matvec(core, x, mode)
        xd = [torch.from_numpy(np.ascontiguousarray(x[:, k])).to(DEV) for k in range(4)]
        ys = [torch.zeros_like(xd[0]) for _ in range(24)]
        for k, y in enumerate(ys):
            h2.mul_(y, A, xd[k % 4])
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        g, xin, yout = torch.cuda.CUDAGraph(), xd[0].clone(), torch.zeros_like(xd[0])
        with torch.cuda.graph(g, stream=s):
            h2.mul_(yout, A, xin)
        for k in range(4):
            xin.copy_(xd[k])
            g.replay()
            ys.append(yout.clone())
        torch.cuda.synchronize()
        for k, y in enumerate(ys):
            got = y.cpu().numpy()
            assert np.linalg.norm(got - want[:, k % 4]) < 1e-12 * np.linalg.norm(want[:, k % 4]), (mode, k)
    ws.close()
