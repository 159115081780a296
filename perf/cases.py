"""The H2 matrix-vector products that this framework is timed on.

Each case is a map (geometry, kernel, interpolation order, storage, far-field precision) and one
product with it (orientation, right-hand sides, call). The sizes are those of the benchmark's and
tests' workloads: the small plain Laplace map, the Toeplitz map, the Helmholtz sphere, the uneven
batch and the serving requests. A program builds a map once and multiplies by new vectors, as an
iterative solver does: `prepare` makes the device core, a workspace and the vectors, `run` is one
product. The geometry belongs to the case, the vectors to the seed.
"""

from __future__ import annotations

import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MODES = {"forward": 0, "transpose": 1, "adjoint": 2}


def _package():
    if "h2factory_b200" not in sys.modules:
        pkg = os.path.join(ROOT, "h2factory.jl_b200")
        spec = importlib.util.spec_from_file_location("h2factory_b200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["h2factory_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["h2factory_b200"]


def _case(name=None, *, call="mul", mode="forward", nrhs=1, precision="fp64", geometry="cube", n=2048, leaf=64,
          kernel="laplace", wavenumber=0.0, p=4, storage="dense", transfers="dense", near="stored", points=0, maps=1):
    case = dict(call=call, mode=mode, nrhs=nrhs, precision=precision, geometry=geometry, n=n, leaf=leaf,
                kernel=kernel, wavenumber=wavenumber, p=p, storage=storage, transfers=transfers, near=near,
                points=points, maps=maps)
    return case if name is None else dict(case, name=name)


def listed():
    sphere = dict(geometry="sphere", leaf=128, kernel="helmholtz", wavenumber=8 * math.pi * 0.45, p=6,
                  storage="symmetric", transfers="separable")
    toeplitz = dict(geometry="cube", n=262144, leaf=0, p=4, storage="toeplitz")
    return [
        # the smallest map: one Krylov step of a small problem, where launches count
        _case("laplace-2k-1", n=2048),
        # the plain Laplace configuration: 8,192 points, FP64, one vector
        _case("laplace-8k-1", n=8192),
        # one adjoint step on a thin surface of odd size (least-squares solvers, sensitivities)
        _case("ellipsoid-20k-1-adjoint", mode="adjoint", geometry="ellipsoid", n=20011, kernel="helmholtz",
              wavenumber=7.3, p=5, storage="symmetric", transfers="separable"),
        # a few vectors on the reduced-precision form, transposed
        _case("cube-12k-3-transpose-f32", mode="transpose", nrhs=3, precision="fp32", n=12289, p=5,
              storage="symmetric", transfers="separable"),
        # a block of vectors held by a host program: copied in, multiplied, copied out
        _case("cube-30k-16-host", call="host", nrhs=16, n=30011, p=5, storage="symmetric", transfers="separable"),
        # one Krylov step on the Helmholtz sphere, FP64
        _case("sphere-65k-1", n=65536, **sphere),
        # a serving request of 8 vectors on the reduced-precision form, transposed
        _case("sphere-65k-8-transpose-f32", mode="transpose", nrhs=8, precision="fp32", n=65536, **sphere),
        # a full block of 32 excitations on the reduced-precision form, adjoint
        _case("sphere-65k-32-adjoint-f32", mode="adjoint", nrhs=32, precision="fp32", n=65536, **sphere),
        # the largest: 32 excitations in FP64
        _case("sphere-262k-32", nrhs=32, n=262144, **sphere),
        # the Toeplitz configuration, FP64, one vector
        _case("toeplitz-262k-1", **toeplitz),
        # the Toeplitz configuration, reduced precision, a block of vectors, transposed
        _case("toeplitz-262k-16-transpose-f32", mode="transpose", nrhs=16, precision="fp32", **toeplitz),
        # twelve uneven maps with 1-16 vectors each, one CUDA graph replay (many bodies, one solve)
        _case("batch-12", call="batch", maps=12, precision="fp32", n=16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["mul"] * 8 + ["host", "batch"])
    points = rng.randrange(1 << 20)
    mode = rng.choice(["forward", "forward", "transpose", "adjoint"])
    precision = rng.choice(["fp64", "fp32"])
    if call == "batch":
        return _case(call="batch", maps=rng.randint(4, 12), precision=precision, n=_log_int(rng, 4096, 16384),
                     points=points)
    if rng.random() < 0.25:
        n = _log_int(rng, 8192, 262144)
        return _case(call=call, mode=mode, nrhs=rng.choice([1, 1, rng.randint(2, 16)]), precision=precision, n=n,
                     leaf=0, p=4, storage="toeplitz", points=points)
    geometry = rng.choice(["cube", "sphere", "ellipsoid"])
    kernel = rng.choice(["laplace", "helmholtz"])
    p = rng.choice([4, 5, 6])
    storage = rng.choice(["dense", "symmetric"]) if p == 4 and geometry == "cube" else "symmetric"
    return _case(call=call, mode=mode, nrhs=rng.choice([1, rng.randint(1, 16), rng.randint(1, 32)]) if geometry != "cube"
                 else rng.choice([1, rng.randint(1, 16)]), precision=precision, geometry=geometry,
                 n=_log_int(rng, 2048, 20000 if geometry == "cube" else 65536), leaf=rng.choice([64, 64, 128]),
                 kernel=kernel, wavenumber=round(rng.uniform(1.0, 12.0), 3) if kernel == "helmholtz" else 0.0, p=p,
                 storage=storage, transfers=rng.choice(["dense", "separable", "separable"]),
                 near=rng.choice(["stored"] * 5 + ["free"]), points=points)


# ---------------------------------------------------------------------------------------------
# the maps
# ---------------------------------------------------------------------------------------------
def _points(geometry, n, seed):
    """Points of a volume, or of a jittered Fibonacci lattice on a surface, in the unit cube."""
    rng = np.random.default_rng(seed)
    if geometry == "cube":
        return rng.random((n, 3))
    i = np.arange(n) + 0.5
    phi, th = np.arccos(1 - 2 * i / n), math.pi * (1 + 5 ** 0.5) * i
    pts = np.stack([np.cos(th) * np.sin(phi), np.sin(th) * np.sin(phi), np.cos(phi)], axis=1)
    pts = pts + 0.1 * math.sqrt(4 * math.pi / n) * rng.standard_normal(pts.shape)
    axes = np.array([1.0, 1.0, 1.0] if geometry == "sphere" else [1.0, 0.25, 0.25])
    return 0.5 + 0.45 * pts * axes


def _members(case):
    """The maps of a case: itself, or the uneven maps of a batch."""
    if case["call"] != "batch":
        return [case]
    rng = np.random.default_rng(1000 + case["points"])
    out = []
    for _ in range(case["maps"]):
        helm = bool(rng.integers(2))
        n = int(round(math.exp(rng.uniform(math.log(2048), math.log(case["n"])))))
        out.append(_case(mode=["forward", "transpose", "adjoint"][int(rng.integers(3))], nrhs=int(rng.integers(1, 17)),
                         precision=case["precision"], geometry=["cube", "sphere", "ellipsoid"][int(rng.integers(3))],
                         n=n, kernel="helmholtz" if helm else "laplace",
                         wavenumber=float(rng.uniform(1, 20)) if helm else 0.0, p=int(rng.integers(4, 7)),
                         storage="symmetric", transfers="separable", points=int(rng.integers(1 << 20))))
    return out


def _tree(case):
    from h2factory_b200 import trees

    pts = _points(case["geometry"], case["n"], case["points"])
    if case["storage"] == "toeplitz":  # uniform octree, about 64 points a leaf, points in Morton order
        pts = pts[trees.morton_order(pts)]
        depth = 1 + max(2, round(math.log(case["n"] / 64, 8)))
        return trees.build_tree(pts, depth=depth, root_center=[0.5] * 3, root_halfsize=0.5)
    return trees.build_tree(pts, maxvalues=case["leaf"], root_center=[0.5] * 3, root_halfsize=0.5)


@functools.lru_cache(maxsize=12)
def _host_map(items):
    """The method's data of a map on the host: trees, plans, collections, transfers, couplings."""
    _package()
    from h2factory_b200 import methods

    case = dict(items)
    toeplitz = case["storage"] == "toeplitz"
    kernel = methods.laplace if case["kernel"] == "laplace" else methods.helmholtz(case["wavenumber"])
    return methods.interpolation_core(
        _tree(case), kernel, case["p"], nodes="equispaced" if toeplitz else "chebyshev",
        transfers=case["transfers"], couplings="toeplitz" if toeplitz else "dense",
        symmetry=case["storage"] == "symmetric", precision=case["precision"],
        near="free" if case["near"] == "free" else "none")


def _map(case):
    """The host map of `case`, with its near blocks assembled on the device where they are stored."""
    core = _host_map(tuple(sorted((k, v) for k, v in case.items() if k not in ("call", "mode", "nrhs", "name"))))
    if case["near"] == "stored":
        from h2factory_b200 import assembly

        assembly.near_blocks_device(core, case["kernel"], wavenumber=case["wavenumber"], batch_entries=1 << 24)
    return core


def _release(core):
    """The device core holds its own copy of the near blocks."""
    core.near_device = None


def _vectors(case, seed, k=0):
    """The k-th map's vectors, N(0, 1), real or complex Gaussian, one column each."""
    g = torch.Generator(device="cuda").manual_seed(seed * 64 + k)
    dt = torch.complex128 if case["kernel"] == "helmholtz" else torch.float64
    return torch.randn((case["nrhs"], case["n"]), dtype=dt, device="cuda", generator=g).t()


def prepare(case, seed):
    h2 = _package()
    if case["call"] == "batch":
        members = _members(case)
        cores = [_map(c) for c in members]
        maps = h2.batch.BatchedMaps(cores, [c["nrhs"] for c in members], modes=[MODES[c["mode"]] for c in members])
        maps.capture()
        for core in cores:
            _release(core)
        return {"call": "batch", "maps": maps, "x": [_vectors(c, seed, k) for k, c in enumerate(members)]}
    core = _map(case)
    ws = h2.H2Workspace(h2.DeviceCore(core), max_nrhs=case["nrhs"])
    _release(core)
    x = _vectors(case, seed)
    if case["call"] == "host":
        xh = np.asfortranarray(x.cpu().numpy())
        return {"call": "host", "ws": ws, "mode": MODES[case["mode"]], "x": xh, "y": np.zeros_like(xh, order="F")}
    op = {"forward": lambda a: a, "transpose": h2.transpose, "adjoint": h2.adjoint}[case["mode"]](ws)
    if case["nrhs"] == 1:
        x = x[:, 0].contiguous()
        y = torch.zeros_like(x)
    else:
        y = torch.zeros((case["nrhs"], case["n"]), dtype=x.dtype, device="cuda").t()
    return {"call": "mul", "mul": h2.mul_, "op": op, "x": x, "y": y}


def run(state):
    if state["call"] == "batch":
        state["maps"].set_inputs(state["x"])
        state["maps"].replay()
        return list(state["maps"].outputs)
    if state["call"] == "host":
        return state["ws"].matvec_host(state["x"], state["mode"], y=state["y"])
    return state["mul"](state["y"], state["op"], state["x"])


# ---------------------------------------------------------------------------------------------
# what a product cannot do without, and its value in 64 bits
# ---------------------------------------------------------------------------------------------
def _work(case):
    core = _host_map(tuple(sorted((k, v) for k, v in case.items() if k not in ("call", "mode", "nrhs", "name"))))
    cplx, r, tree = core.field == "complex", case["nrhs"], core.test
    mac, entry, far = (8 if cplx else 2), (16 if cplx else 8), (8 if case["precision"] == "fp64" else 4)
    far *= 2 if cplx else 1
    nv = np.diff(tree.value_ptr).astype(np.int64)
    near = int((nv[core.plans.near[:, 0]] * nv[core.plans.near[:, 1]]).sum())
    q, dim = case["p"] ** tree.dim, tree.dim
    edges = 2 * int((core.plans.test.agg_node.size + core.plans.test.dis_node.size) / 2)
    leaf = case["n"] * q
    per_edge = dim * case["p"] ** (dim + 1) if case["transfers"] == "separable" else q * q
    if case["storage"] == "toeplitz":  # one product per frequency, half of them in a real map
        half = case["p"] * (2 * case["p"] - 1) ** 2
        m2l, unique = 8 * half * len(core.plans.far) * r, len(core.couplings) * half * 2 * (8 if case["precision"] == "fp64" else 4)
    else:
        m2l, unique = mac * q * q * len(core.plans.far) * r, sum(b.size for b in core.couplings) * far
    stored = near * entry if case["near"] == "stored" else 0
    return {"bytes": stored + unique + leaf * far + 2 * case["n"] * r * entry,
            "flops": mac * r * (near + 2 * leaf + edges * per_edge) + m2l}


def work(case):
    parts = [_work(c) for c in _members(case)]
    return {k: float(sum(w[k] for w in parts)) for k in ("bytes", "flops")}


def _kernel(case, r):
    """The point kernel at distances r, 0 at r = 0."""
    safe = torch.where(r > 0, r, torch.ones_like(r))
    if case["kernel"] == "laplace":
        return torch.where(r > 0, 1.0 / (4.0 * math.pi * safe), torch.zeros_like(r))
    phase = case["wavenumber"] * safe
    return torch.polar(torch.where(r > 0, 1.0 / (4.0 * math.pi * safe), torch.zeros_like(r)), phase)


def _interp(nodes, t):
    """Lagrange polynomials of `nodes` at t (..., points, 3): (..., p^3, points), axis 0 fastest."""
    diff = t.unsqueeze(-1) - nodes                              # (..., points, 3, p)
    cols = []
    for k in range(nodes.numel()):
        others = [m for m in range(nodes.numel()) if m != k]
        cols.append((diff[..., others] / (nodes[k] - nodes[others])).prod(-1))
    a = torch.stack(cols, -1).transpose(-3, -2).transpose(-2, -1)  # (..., 3, p, points)
    out = a[..., 2, :, None, None, :] * a[..., 1, None, :, None, :] * a[..., 0, None, None, :, :]
    return out.flatten(-4, -2)


def _exact(case, x):
    """op(A) x of the map's definition, summed in 64 bits: near leaf pairs by the point kernel, far
    pairs by interpolating both boxes, each box's moments straight from the points it holds."""
    core = _host_map(tuple(sorted((k, v) for k, v in case.items() if k not in ("call", "mode", "nrhs", "name"))))
    tree, dev, p = core.test, "cuda", case["p"]
    up = lambda a, dt=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(dev, dt)  # noqa: E731
    if case["mode"] == "adjoint":
        x = x.conj()
    dt = x.dtype
    k = torch.arange(p, dtype=torch.float64, device=dev)
    toeplitz = case["storage"] == "toeplitz"
    xi = -1 + (2 * k + 1) / p if toeplitz else torch.cos((2 * k + 1) * math.pi / (2 * p))
    grid = torch.cartesian_prod(xi, xi, xi).flip(-1)            # axis 0 fastest
    leaves = tree.leaves()
    m = int(np.diff(tree.value_ptr).max())
    idx = np.full((tree.nnodes, m), -1, np.int64)
    for leaf in leaves:
        v = tree.values(int(leaf))
        idx[leaf, :v.size] = v
    idx = up(idx, torch.int64)
    valid = idx >= 0
    pts, safe = up(tree.points), idx.clamp(min=0)
    center, half = up(tree.center), up(tree.halfsize)
    y = torch.zeros((case["n"], x.shape[1]), dtype=dt, device=dev)
    # near field
    a, b = (0, 1) if case["mode"] == "forward" else (1, 0)
    near, far = up(core.plans.near, torch.int64), up(core.plans.far, torch.int64)
    step = max(1, (1 << 24) // (m * max(m, 2 * x.shape[1])))
    for s in range(0, near.shape[0], step):
        r, c = near[s:s + step, a], near[s:s + step, b]
        d = pts[safe[r]][:, :, None, :] - pts[safe[c]][:, None, :, :]
        block = _kernel(case, d.square().sum(-1).sqrt())
        block = block * (valid[r][:, :, None] & valid[c][:, None, :])
        out = block.to(dt) @ x[safe[c]]
        y.index_add_(0, safe[r].flatten(), out.flatten(0, 1) * valid[r].flatten()[:, None])
    # the ancestors of every leaf
    level = tree.level
    chain = np.full((leaves.size, int(level.max()) + 1), -1, np.int64)
    node = leaves.astype(np.int64)
    while (node >= 0).any():
        ok = node >= 0
        chain[np.nonzero(ok)[0], level[node[ok]]] = node[ok]
        node = np.where(ok, tree.parent[np.maximum(node, 0)], -1)
    used = np.unique(core.plans.far)
    leaves_t = up(leaves, torch.int64)

    def walk(visit):
        """visit(leaves, box at one level, interpolation matrix of the leaves' points in it)."""
        for lvl in range(1, chain.shape[1]):
            sel = np.nonzero((chain[:, lvl] >= 0) & np.isin(chain[:, lvl], used))[0]
            for s in range(0, sel.size, max(1, (1 << 25) // (m * p ** 3 + p ** 3 * 2 * x.shape[1]))):
                part = up(sel[s:s + max(1, (1 << 25) // (m * p ** 3 + p ** 3 * 2 * x.shape[1]))], torch.int64)
                n, box = leaves_t[part], up(chain[part.cpu().numpy(), lvl], torch.int64)
                t = (pts[safe[n]] - center[box][:, None]) / half[box][:, None, None]
                visit(n, box, (_interp(xi, t) * valid[n][:, None, :]).to(dt))

    moments = torch.zeros((tree.nnodes, p ** 3, x.shape[1]), dtype=dt, device=dev)
    local = torch.zeros_like(moments)
    walk(lambda n, box, c: moments.index_add_(0, box, c @ x[safe[n]]))
    keys = core.pair_coupling
    order = np.argsort(keys, kind="stable")
    first = np.nonzero(np.diff(keys[order], prepend=-1))[0]
    for group in np.split(order, first[1:]):                    # pairs of equal geometry share one block
        r, c = int(core.plans.far[group[0], a]), int(core.plans.far[group[0], b])
        d = (center[r] - center[c]) + (half[r] * grid)[:, None, :] - (half[c] * grid)[None, :, :]
        block = _kernel(case, d.square().sum(-1).sqrt()).to(dt)
        pair = far[up(group, torch.int64)]
        for s in range(0, pair.shape[0], 4096):
            r, c = pair[s:s + 4096, a], pair[s:s + 4096, b]
            src = moments[c].transpose(0, 1).flatten(1)         # one product for the whole group
            local.index_add_(0, r, (block @ src).unflatten(1, (r.numel(), -1)).transpose(0, 1))

    def scatter(n, box, c):
        out = c.transpose(1, 2) @ local[box]
        y.index_add_(0, safe[n].flatten(), out.flatten(0, 1) * valid[n].flatten()[:, None])

    walk(scatter)
    return y.conj().resolve_conj() if case["mode"] == "adjoint" else y


def exact(case, seed):
    found = [_exact(c, _vectors(c, seed, k)) for k, c in enumerate(_members(case))]
    if case["call"] == "batch":
        return found
    y = found[0][:, 0] if case["nrhs"] == 1 and case["call"] == "mul" else found[0]
    return y.cpu().numpy() if case["call"] == "host" else y
