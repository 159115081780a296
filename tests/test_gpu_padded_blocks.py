"""FP32 blocks whose columns are not whole 16 bytes: padded copies for the tcgen05 I2O (GPU).

The copies are made on the device when the core is made, from the stored blocks for forward products
and from their transposes for the others. A map whose sides have different coefficient counts (125
and 64) tells rows from columns. Compared with the FP64 form: FP32 storage and TF32-split products
with 64-value FP32 segments keep 1e-6.
"""

import copy

import numpy as np
import pytest

import h2factory_b200 as h2
from h2factory_b200.core import H2Core
from h2factory_b200.trees import build_plans, build_tree
from test_gpu_pairs_i2o import _product, rel

pytestmark = pytest.mark.gpu


def _two_shapes(test, trial, cplx):
    """Four leaves a side on a line, far pairs between leaves only, three random blocks."""
    rng = np.random.default_rng(3)
    points = np.full((64, 3), 0.3)
    points[:, 0] = (np.arange(64) + 0.5) / 64
    tree = build_tree(points, maxvalues=16, root_center=[0.5] * 3, root_halfsize=0.5)
    plans = build_plans(tree)
    assert len(plans.far) > 0 and not np.intersect1d(plans.far, tree.parent).size

    def draw(*shape):
        a = rng.standard_normal(shape)
        return a + 1j * rng.standard_normal(shape) if cplx else a

    def shape(n):
        sh = np.ones((tree.nlevels + 1, 3), np.int32)
        sh[:] = n
        return sh

    def colls(n):
        return {int(l): draw(1, int(np.prod(n)), tree.values(int(l)).size) for l in tree.leaves()}

    core = H2Core(field="complex" if cplx else "real", test=tree, trial=tree, plans=plans, ncomp=1, dim=3,
                  shape_test=shape(test), shape_trial=shape(trial), collections_test=colls(test),
                  collections_trial=colls(trial), transfers_test={}, transfers_trial={}, transfer_kind="dense",
                  coupling_kind="dense", couplings=[draw(int(np.prod(test)), int(np.prod(trial))) for _ in range(3)],
                  pair_coupling=np.arange(len(plans.far)) % 3)
    core.set_near_blocks([np.zeros((16, 16), core.dtype) for _ in plans.near])
    return core


@pytest.mark.parametrize("cplx,nrhs", [(False, 6), (False, 70), (True, 3), (True, 33)])
def test_sides_of_different_shapes(cplx, nrhs):
    core = _two_shapes((5, 5, 5), (4, 4, 4), cplx)
    c32 = copy.copy(core)
    c32.precision = "fp32"
    rng = np.random.default_rng(nrhs)
    x = rng.standard_normal((64, nrhs)) + (1j * rng.standard_normal((64, nrhs)) if cplx else 0)
    w64, w32 = h2.H2Workspace(core, max_nrhs=nrhs), h2.H2Workspace(c32, max_nrhs=nrhs)
    for view in (lambda w: w, h2.transpose, h2.adjoint):
        assert rel(_product(h2.mul_, view(w32), core, x), _product(h2.mul_, view(w64), core, x)) < 1e-6
    w64.close()
    w32.close()
