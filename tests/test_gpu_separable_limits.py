"""Separable transfers whose children do not fit an SM's shared memory side by side (GPU).

At 10 points an axis in complex FP64 a moment column takes 16 KB, two buffers of eight children's 256
KB: the upward pass contracts five children, then the other three, and keeps their sum in a buffer of
its own. Two clusters in boxes of one level, each split into eight leaves, give parents with all their
children.

Tolerance: FP64 sums of at most 1,000 x 16 products of O(1) terms keep 1e-12 relative; the FP32
form's storage 1e-6.
"""

import copy

import numpy as np
import pytest

import h2factory_b200 as h2
from h2factory_b200 import methods
from h2factory_b200.trees import build_tree
from oracle import oracle
from test_gpu_pairs_i2o import _product, _x, rel

pytestmark = pytest.mark.gpu


def _clusters(p):
    corners = np.array([[i, j, k] for i in (0, 1) for j in (0, 1) for k in (0, 1)])
    rng = np.random.default_rng(p)
    box = np.concatenate([0.125 * (corners + 0.1 + 0.8 * rng.random((8, 3))) for _ in range(2)])
    tree = build_tree(np.concatenate([box, box + [0.75, 0.0, 0.0]]), maxvalues=4, root_center=[0.5] * 3,
                      root_halfsize=0.5)
    core = methods.interpolation_core(tree, methods.helmholtz(2.0), p, symmetry=True, transfers="separable")
    parents = np.unique(core.plans.far)
    assert all(np.count_nonzero(tree.parent == b) == 8 for b in parents)
    return core


@pytest.mark.parametrize("p", [9, 10])
def test_children_in_parts_match_oracle(p):
    core = _clusters(p)
    c32 = copy.copy(core)
    c32.precision = "fp32"
    for nrhs in (1, 3):
        x = _x(core, nrhs, nrhs)
        w64, w32 = h2.H2Workspace(core, max_nrhs=nrhs), h2.H2Workspace(c32, max_nrhs=nrhs)
        for mode, view in enumerate((lambda w: w, h2.transpose, h2.adjoint)):
            y = _product(h2.mul_, view(w64), core, x)
            assert rel(y, oracle.matvec(core, x, mode)) < 1e-12, (nrhs, mode)
            assert rel(_product(h2.mul_, view(w32), core, x), y) < 1e-6, (nrhs, mode)
        w64.close()
        w32.close()
