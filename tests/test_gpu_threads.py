"""Two host threads multiply different maps at once, each on a workspace and stream of its own (GPU).

Any host thread may call; only a workspace belongs to one call at a time. A kernel's limit on dynamic
shared memory, though, is one value per device for all threads, so a launcher must not make it follow
its own map. The pairs of maps here share a kernel and need different amounts for it: separable
transfers of 4 and 6 points an axis, the tcgen05 I2O per receiving node with 5 and 60 right-hand
sides, Toeplitz transforms of 5 and 8 points an axis. They are small, so that the threads spend their
time in launches.

Every product has to succeed, and the last one's bits have to be those of the same call made alone
(no atomics, so equal calls give equal bits).
"""

import copy
import threading

import numpy as np
import pytest
import torch

import h2factory_b200 as h2
from h2factory_b200 import methods
from h2factory_b200.trees import build_tree

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
ROUNDS, QUEUED = 50, 20


def _chebyshev(p, cplx, precision="fp64", transfers="separable"):
    rng = np.random.default_rng(p)
    tree = build_tree(rng.random((300, 3)), maxvalues=4, root_center=[0.5] * 3, root_halfsize=0.5)
    kernel = methods.helmholtz(3.0) if cplx else methods.laplace
    core = methods.interpolation_core(tree, kernel, p, symmetry=True, transfers=transfers)
    core = copy.copy(core)
    core.precision = precision
    return core


def _toeplitz(p):
    rng = np.random.default_rng(p)
    tree = build_tree(rng.random((200, 3)), depth=3, root_center=[0.5] * 3, root_halfsize=0.5)
    return methods.interpolation_core(tree, methods.helmholtz(3.0), p, nodes="equispaced", couplings="toeplitz")


PAIRS = {
    "separable": lambda: ((_chebyshev(4, True), 1), (_chebyshev(6, True), 4)),
    "per-node-tcgen05": lambda: tuple((_chebyshev(3, False, "fp32", "dense"), nrhs) for nrhs in (5, 60)),
    "toeplitz": lambda: ((_toeplitz(5), 1), (_toeplitz(8), 1)),
}


@pytest.mark.parametrize("name", sorted(PAIRS))
def test_threads_with_different_maps(name):
    jobs = []
    for core, nrhs in PAIRS[name]():
        ws = h2.H2Workspace(core, max_nrhs=nrhs)
        dt = torch.complex128 if core.field == "complex" else torch.float64
        x = torch.randn((nrhs, core.trial.npoints), dtype=dt, device=DEV).t()
        alone = torch.zeros((nrhs, core.test.npoints), dtype=dt, device=DEV).t()
        h2.mul_(alone, ws, x)
        jobs.append((ws, x, alone, torch.empty_like(alone), torch.cuda.Stream(DEV)))
    torch.cuda.synchronize()
    start, errors = threading.Barrier(len(jobs)), []

    def work(ws, x, alone, y, stream):
        try:
            start.wait(timeout=60)
            for _ in range(ROUNDS):
                for _ in range(QUEUED):
                    h2.mul_(y, ws, x, stream=stream.cuda_stream)
                stream.synchronize()
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    torch.cuda.synchronize()
    assert not errors, errors[0]
    for ws, x, alone, y, _ in jobs:
        assert torch.equal(y, alone)
        ws.close()
