"""The server's estimate of a map's device memory counts what the dense I2O keeps per pair (CPU)."""

import copy

import numpy as np

from h2factory_b200 import methods, serving
from h2factory_b200.trees import build_tree


def test_dense_map_counts_its_plans_and_products():
    rng = np.random.default_rng(1)
    tree = build_tree(rng.random((1500, 3)), maxvalues=16, root_center=[0.5] * 3, root_halfsize=0.5)
    core = methods.interpolation_core(tree, methods.laplace, 2)
    other = copy.copy(core)
    other.coupling_kind = "toeplitz"
    pairs, executor = len(core.plans.far), serving.GpuExecutor()
    # five plans a side, a 16-byte record per pair each
    assert executor.footprint(core, 4, 0) - executor.footprint(other, 4, 0) == 2 * 5 * 16 * pairs
    # and, per slot, the products of all pairs (8 coefficients, 4 right-hand sides)
    slot = [executor.footprint(c, 4, 1) - executor.footprint(c, 4, 0) for c in (core, other)]
    assert slot[0] - slot[1] == pairs * 8 * 8 * 4
