"""The timed cases of the H-matrix framework: products and assembly as a
program calls them.

A case is a dict of plain values.  Its "kind":

  product    y = H x on one H-matrix that the program keeps (an operator of a
             Krylov solve, a boundary-integral operator, a covariance matrix)
  batch      the products of several forests of independent H-matrices, one
             captured graph launched once
  assembly   HMatrix.build (device partialACA and the layout of the leaves) on
             a cluster tree the program has, and the first product with it

prepare() makes the points and right-hand sides of a seed and builds what such
a program keeps; run() is one pass; exact() is the dense product in 64 bits.
"""
import math

import numpy as np
import torch

import htool_gb300 as H
from htool_gb300 import geometry as G

#: wave number, admissibility and tolerance of the two kinds of operators
HELMHOLTZ_K = 20.0
LAPLACE_ETA, LAPLACE_EPS = 10.0, 1e-6
HELMHOLTZ_ETA, HELMHOLTZ_EPS = 3.0, 1e-5

#: exact() takes on at most this many kernel entries (about 20 s)
EXACT_ENTRIES = 8e10


def product(name=None, **over):
    """A product case: the defaults, with `over` in place."""
    case = {
        "kind": "product",
        "shape": "sphere",  # point set (htool_gb300.geometry)
        "kernel": "laplace",
        "n": 100000,
        "mu": 1,  # right-hand sides
        "storage": "fp64",  # low-rank factors of products: fp64 or mixed
        "layout": "real",  # of complex H-matrices: real (form) or native
        "symmetry": "N",
        "op": "N",  # N: H x, T: its transpose
        "arrays": "device",  # device pointers on the current stream, or host arrays
        "planes": False,  # set_digit_planes: what a program with many right-hand sides turns on
        "tuned": False,  # autotune(mu) after the build
    }
    case.update(over)
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # the smallest calls: one product of the 4 000-point cylinder on host
        # arrays, as htool's users call it
        product("cylinder_4k_host", shape="cylinder", kernel="inv_r_eps", n=4000, arrays="host"),
        # one matvec of a Krylov step, FP64, at an ordinary size and at the
        # size of the headline benchmark
        product("sphere_100k", n=100000),
        product("sphere_1m", n=1000000),
        # the same with reduced-precision factors; an odd size
        product("sphere_200k_mixed", n=200003, storage="mixed"),
        # a block of right-hand sides: block Krylov methods, several loads
        product("sphere_100k_4rhs", n=100000, mu=4, tuned=True),
        product("sphere_100k_mixed_8rhs", n=100000, mu=8, storage="mixed"),
        # many right-hand sides: multi-source solves
        product("sphere_60k_64rhs", n=60000, mu=64, planes=True),
        product("helmholtz_30k_mixed_64rhs", shape="cube", kernel="helmholtz", n=30000, mu=64, storage="mixed", planes=True),
        # one complex right-hand side, factors at 16 bytes an entry
        product("helmholtz_60k_native", shape="cube", kernel="helmholtz", n=60000, layout="native"),
        # H^T x on host arrays (least squares, adjoint solves)
        product("ellipsoid_20k_transposed", shape="ellipsoid", n=20000, mu=2, op="T", arrays="host"),
        # many independent operators with 1 to 8 right-hand sides each
        {"name": "batch_24", "kind": "batch", "members": 24, "nmin": 2000, "nmax": 12000, "storage": "fp64"},
        # a new operator: assembly and its first product
        {"name": "assembly_50k", "kind": "assembly", "shape": "sphere", "n": 50000, "symmetry": "N"},
    ]


def _log(rng, lo, hi):
    """An odd or even integer of [lo, hi], its logarithm uniform."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    shape = rng.choice(["sphere", "ellipsoid", "cylinder", "cube"])
    what = rng.choice(["small", "one", "one", "mixed", "few", "few_mixed", "many", "helmholtz", "native", "twin", "batch", "assembly"])
    if what == "small":
        return product(shape=shape, kernel=rng.choice(["laplace", "inv_r_eps"]), n=_log(rng, 1500, 20000), mu=rng.choice([1, 1, 2]), arrays=rng.choice(["host", "device"]))
    if what == "one":
        return product(shape=shape, n=_log(rng, 20000, 500000))
    if what == "mixed":
        return product(shape=shape, n=_log(rng, 20000, 500000), storage="mixed")
    if what == "few":
        return product(shape=shape, n=_log(rng, 15000, 150000), mu=rng.randint(2, 8), tuned=True)
    if what == "few_mixed":
        return product(shape=shape, n=_log(rng, 15000, 150000), mu=rng.randint(2, 8), storage="mixed")
    if what == "many":
        return product(shape=shape, n=_log(rng, 8000, 80000), mu=_log(rng, 9, 64), planes=True)
    if what == "helmholtz":
        return product(shape="cube", kernel="helmholtz", n=_log(rng, 4000, 30000), mu=_log(rng, 8, 64), storage=rng.choice(["fp64", "mixed"]), planes=True)
    if what == "native":
        return product(shape="cube", kernel="helmholtz", n=_log(rng, 8000, 80000), mu=rng.randint(1, 3), layout="native")
    if what == "twin":
        transposed = rng.random() < 0.5
        return product(shape=shape, n=_log(rng, 4000, 60000), mu=rng.randint(1, 4), symmetry="N" if transposed else "S", op="T" if transposed else "N", arrays="host" if transposed else "device")
    if what == "batch":
        return {"kind": "batch", "members": rng.randint(6, 24), "nmin": 2000, "nmax": _log(rng, 4000, 14000), "storage": rng.choice(["fp64", "mixed"])}
    return {"kind": "assembly", "shape": shape, "n": _log(rng, 5000, 60000), "symmetry": rng.choice(["N", "S"])}


# ---------------------------------------------------------------------------
# inputs


def _points(shape, n, seed):
    if shape == "sphere":
        return G.sphere(n, seed=seed)
    if shape == "cylinder":
        return G.cylinder(n, seed=seed)
    if shape == "cube":
        return G.cube_surface(n, seed=seed)
    axes = np.random.default_rng([seed, n]).uniform(0.5, 2.0, 3)
    return G.ellipsoid(n, axes, seed=seed)


def _params(case):
    if case.get("kernel") == "helmholtz":
        return HELMHOLTZ_EPS, HELMHOLTZ_ETA, HELMHOLTZ_K
    return LAPLACE_EPS, LAPLACE_ETA, 0.0


def _rhs(n, mu, seed, dtype):
    """N(0, 1) right-hand sides, column-major n x mu."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 77)
    return torch.randn(mu, n, dtype=dtype, device="cuda", generator=g)


def _build(case, seed):
    """The points and the H-matrix of a product case."""
    pts = _points(case["shape"], case["n"], seed)
    eps, eta, k = _params(case)
    is_complex = case["kernel"] == "helmholtz"
    sym = case["symmetry"]
    t = H.Cluster().build(case["n"], pts)
    hm = H.HMatrix(t, t, eps, eta, symmetry=sym, UPLO="L" if sym == "S" else "N", dtype=np.complex128 if is_complex else np.float64, complex_layout=case["layout"])
    hm.build(case["kernel"], pts, kernel_param=k)
    return pts, hm


def _members(case, seed):
    """(right-hand sides, points) of every member of a batch: the sizes are
    the case's, the ellipsoids and their points the seed's."""
    sizes = np.random.default_rng([case["members"], case["nmin"], case["nmax"]])
    axes = np.random.default_rng([seed, 4])
    out = []
    for k in range(case["members"]):
        n = int(round(np.exp(sizes.uniform(np.log(case["nmin"]), np.log(case["nmax"])))))
        out.append(((1, 2, 4, 8)[k % 4], G.ellipsoid(n, axes.uniform(0.5, 2.0, 3), seed=1000 * seed + k)))
    return out


def _forests(case, seed):
    """Members with the same number of right-hand sides as one forest each."""
    by_mu = {}
    for mu, pts in _members(case, seed):
        by_mu.setdefault(mu, []).append(pts)
    forests = []
    for mu, sets in sorted(by_mu.items()):
        t = H.Cluster.forest([H.Cluster().build(len(p), p) for p in sets])
        hm = H.HMatrix(t, t, LAPLACE_EPS, LAPLACE_ETA).build(H.LAPLACE, t.points)
        if case["storage"] != "fp64":
            hm.set_precision(case["storage"], 1.0)
        forests.append((mu, sets, t, hm))
    return forests


def prepare(case, seed):
    if case["kind"] == "assembly":
        pts = _points(case["shape"], case["n"], seed)
        return {"case": case, "points": pts, "tree": H.Cluster().build(case["n"], pts), "x": _rhs(case["n"], 1, seed, torch.float64), "y": torch.zeros(1, case["n"], dtype=torch.float64, device="cuda")}
    if case["kind"] == "batch":
        batch, xs, ys = H.HBatch(), [], []
        for mu, _, t, hm in _forests(case, seed):
            n = t.get_size()
            xs.append(_rhs(n, mu, seed + mu, torch.float64))
            ys.append(torch.zeros(mu, n, dtype=torch.float64, device="cuda"))
            torch.cuda.synchronize()
            batch.add(hm, xs[-1].data_ptr(), ys[-1].data_ptr(), mu, keep=(t, xs[-1], ys[-1]))
        batch.capture()
        return {"case": case, "batch": batch, "ys": ys}
    _, hm = _build(case, seed)
    if case["storage"] != "fp64":
        hm.set_precision(case["storage"], 1.0)
    if case["planes"]:
        hm.set_digit_planes(True)
    if case["tuned"]:
        hm.autotune(case["mu"])
    x = _rhs(case["n"], case["mu"], seed, torch.complex128 if case["kernel"] == "helmholtz" else torch.float64)
    if case["arrays"] == "host":
        return {"case": case, "hm": hm, "x": x.cpu().numpy()}
    return {"case": case, "hm": hm, "x": x, "y": torch.zeros_like(x)}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].launch(torch.cuda.current_stream().cuda_stream)
        return state["ys"]
    if case["kind"] == "assembly":
        sym = case["symmetry"]
        hm = H.HMatrix(state["tree"], state["tree"], LAPLACE_EPS, LAPLACE_ETA, symmetry=sym, UPLO="L" if sym == "S" else "N")
        hm.build(H.LAPLACE, state["points"])
        state["hm"] = hm  # the operator is kept, as its product is still under way
        hm.mvprod_ptr(state["x"].data_ptr(), state["y"].data_ptr(), 1, 0, torch.cuda.current_stream().cuda_stream)
        info = hm.get_infos()  # htool's print_infos: the numbers of leaves, the ranks
        return {"y": state["y"], "infos": [int(info[key]) for key in ("Number_of_lrmat", "Number_of_dmat", "Number_of_false_positive", "Rank_max")]}
    hm = state["hm"]
    if case["arrays"] == "host":
        if case["op"] == "T":
            return hm.mvprod_transp_global_to_global(state["x"], case["mu"])
        return hm.mvprod_global_to_global(state["x"], case["mu"])
    hm.mvprod_ptr(state["x"].data_ptr(), state["y"].data_ptr(), case["mu"], 0, torch.cuda.current_stream().cuda_stream)
    return state["y"]


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _leaf_sums(hm):
    """Entries of the low-rank factors and of the dense leaves, and the
    entries times ranks that an assembly's corrections take."""
    lr, dn = (a.astype(np.int64) for a in hm.get_leaves())
    factors = lr[:, 4] * (lr[:, 2] + lr[:, 3])
    dense = dn[:, 2] * dn[:, 3]
    return int(factors.sum()), int(dense.sum()), int((factors * lr[:, 4]).sum())


def work(case):
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for mu, _, t, hm in _forests(case, 1):
            factors, dense, _ = _leaf_sums(hm)
            stored = hm.precision_info()["stored_bytes"] if case["storage"] != "fp64" else 8 * (factors + dense)
            total["bytes"] += stored + 16 * mu * t.get_size()
            total["flops"] += 2 * mu * (factors + dense)
        return total
    full = product(**case) if case["kind"] == "product" else product(shape=case["shape"], n=case["n"], symmetry=case["symmetry"])
    _, hm = _build(full, 1)
    factors, dense, cross = _leaf_sums(hm)
    if case["kind"] == "assembly":
        # an entry of the kernel: three differences, a square root, a division
        # (about 30 operations); a cross of rank k is corrected by the k before
        # it and its norm estimate takes as much again
        return {"bytes": 8 * (factors + dense) + 48 * case["n"], "flops": 30 * (factors + dense) + 2 * cross}
    twice = 2 if case["symmetry"] == "S" else 1
    cplx = case["kernel"] == "helmholtz"
    entry = 16 if cplx else 8
    if cplx and case["layout"] == "real":
        factors, dense = factors // 4, dense // 4  # reported with doubled sizes and ranks
    stored = entry * (factors + dense)
    if case["storage"] != "fp64":
        hm.set_precision(case["storage"], 1.0)
        stored = hm.precision_info()["stored_bytes"] // (2 if cplx and case["layout"] == "real" else 1)
    return {"bytes": stored + 2 * entry * case["mu"] * case["n"], "flops": twice * (8 if cplx else 2) * case["mu"] * (factors + dense)}


# ---------------------------------------------------------------------------
# the dense product in 64 bits


def _dense_product(kernel, pts, x, transposed=False):
    """(mu x n) rows of the dense kernel matrix applied to x; the kernels are
    symmetric, so the transposed product is the same."""
    P = torch.from_numpy(pts).cuda()
    n, mu = P.shape[0], x.shape[0]
    y = torch.empty_like(x)
    step = max(1, min(n, int(6e7 // n)))
    for a in range(0, n, step):
        b = min(n, a + step)
        d2 = torch.zeros(b - a, n, dtype=torch.float64, device="cuda")
        for c in range(3):
            d2 += (P[a:b, c, None] - P[None, :, c]).square_()
        r = d2.sqrt_()
        if kernel == "inv_r_eps":
            k = r.add_(1e-5).reciprocal_()
        else:
            k = (4 * math.pi * r).reciprocal_()
            k.masked_fill_(r == 0, 0.0)
        if kernel == "helmholtz":
            re, im = torch.cos(HELMHOLTZ_K * r).mul_(k), torch.sin(HELMHOLTZ_K * r).mul_(k)
            y[:, a:b] = torch.complex(x.real @ re.T - x.imag @ im.T, x.real @ im.T + x.imag @ re.T)
        else:
            y[:, a:b] = x @ k.T
    return y


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        by_mu = {}
        for mu, pts in _members(case, seed):
            by_mu.setdefault(mu, []).append(pts)
        for mu, sets in sorted(by_mu.items()):
            n = sum(len(p) for p in sets)
            x = _rhs(n, mu, seed + mu, torch.float64)
            parts, o = [], 0
            for p in sets:
                parts.append(_dense_product("laplace", p, x[:, o:o + len(p)].contiguous()))
                o += len(p)
            out.append(torch.cat(parts, 1))
        return out
    n = case["n"]
    if n * n * (4.0 if case.get("kernel") == "helmholtz" else 1.0) > EXACT_ENTRIES:
        return None
    pts = _points(case["shape"], n, seed)
    if case["kind"] == "assembly":
        return {"y": _dense_product("laplace", pts, _rhs(n, 1, seed, torch.float64)), "infos": None}
    x = _rhs(n, case["mu"], seed, torch.complex128 if case["kernel"] == "helmholtz" else torch.float64)
    y = _dense_product(case["kernel"], pts, x)
    return y.reshape(-1).cpu().numpy() if case["arrays"] == "host" else y
