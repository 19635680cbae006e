"""The performance cases of sp2b: what its users have it do, over the range of sizes.

Every case goes through the public entry points: the C ABI of include/sp2b.h with device
pointers (what a resident simulation code calls), the numpy functions of ``sp2b`` and the
torch function ``sp2b.autograd.sp2_density``.  Hamiltonians are the repository's model
systems (``sp2b.modelham``) with seeded disorder:

* ``two_band`` chains, gapped, 11 to 15 SP2 steps;
* ``cubic`` lattices, nearly gapless, 35 to 70 SP2 steps.

Kinds of cases: ``dense`` (one density matrix from device arrays), ``host`` (the same from
numpy arrays), ``response`` (density and first-order response), ``gradient`` (density and
dL/dH of L = Tr(D A) through autograd) and ``subgraph`` (all core+halo parts of a lattice).
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("qmd-progress_b200")   # the working folder is the repository's root
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sp2b                                              # noqa: E402
from sp2b import _lib, autograd, graph, modelham         # noqa: E402

PRECISIONS = {"fp64": sp2b.PREC_FP64, "mixed_fp16": sp2b.PREC_MIXED_FP16,
              "mixed_bf16": sp2b.PREC_MIXED_BF16, "exact_int8": sp2b.PREC_EXACT_INT8}
IDEMTOL = 1e-10
MAXITER = 100
# SP2 steps of a solve, for the operation counts
STEPS = {"two_band": 14, "cubic": 50}
# |H^2| above this connects two sites of the sub-graph cases (core+halo 100 to 500 sites at
# 64 to 150 core sites per part)
GRAPH_THRESHOLD = 0.6


def listed():
    return [
        # a molecule of a few dozen atoms in an MD step: launches and host latency only
        {"name": "fp64_100", "kind": "dense", "model": "two_band", "n": 100,
         "precision": "fp64", "algorithm": "alg2"},
        # an ordinary small system in the parity form, with its branch sequence kept
        {"name": "fp64_1000_genseq", "kind": "dense", "model": "two_band", "n": 1000,
         "precision": "fp64", "algorithm": "alg2_genseq"},
        # a large system in the parity form, a size that is no multiple of the tiles
        {"name": "fp64_3500_alg1", "kind": "dense", "model": "two_band", "n": 3500,
         "precision": "fp64", "algorithm": "alg1"},
        # an ordinary small system in split precision (padded to 1024)
        {"name": "mixed_1000", "kind": "dense", "model": "two_band", "n": 1000,
         "precision": "mixed_fp16", "algorithm": "alg2"},
        # the benchmark's dense workload
        {"name": "mixed_8192_genseq", "kind": "dense", "model": "two_band", "n": 8192,
         "precision": "mixed_fp16", "algorithm": "alg2_genseq"},
        # a nearly gapless lattice (14^3 sites) in the exact form, many steps
        {"name": "exact_cubic_2744", "kind": "dense", "model": "cubic", "n": 2744,
         "precision": "exact_int8", "algorithm": "alg2_genseq"},
        # the numpy call of a Python user: host arrays in and out
        {"name": "host_mixed_2000", "kind": "host", "model": "two_band", "n": 2000,
         "precision": "mixed_fp16", "algorithm": "alg2"},
        # density-matrix perturbation theory, an odd size
        {"name": "response_777", "kind": "response", "model": "two_band", "n": 777,
         "precision": "fp64"},
        # one training step's density and gradient, the benchmark's adjoint size
        {"name": "gradient_2048", "kind": "gradient", "model": "two_band", "n": 2048},
        # the benchmark's graph-partitioned lattice: 256 parts of a 32^3 lattice
        {"name": "subgraph_int8_32", "kind": "subgraph", "edge": 32, "parts": 256,
         "precision": "exact_int8"},
        # a small graph-partitioned lattice in the parity form
        {"name": "subgraph_fp64_16", "kind": "subgraph", "edge": 16, "parts": 32,
         "precision": "fp64"},
        # the split form on a middle-sized lattice with uneven parts
        {"name": "subgraph_fp16_20", "kind": "subgraph", "edge": 20, "parts": 60,
         "precision": "mixed_fp16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense_fp64", "dense_fp64", "mixed", "mixed", "exact", "host", "response",
                       "gradient", "subgraph", "subgraph"])
    if kind == "dense_fp64":
        return {"kind": "dense", "model": "two_band", "n": _log_int(rng, 64, 3500),
                "precision": "fp64",
                "algorithm": rng.choice(["alg2", "alg2_genseq", "alg1"])}
    if kind == "mixed":
        return {"kind": "dense", "model": "two_band", "n": _log_int(rng, 200, 8192),
                "precision": rng.choice(["mixed_fp16", "mixed_fp16", "mixed_bf16"]),
                "algorithm": rng.choice(["alg2", "alg2_genseq"])}
    if kind == "exact":
        if rng.random() < 0.5:
            return {"kind": "dense", "model": "cubic", "n": rng.randint(6, 14) ** 3,
                    "precision": "exact_int8", "algorithm": "alg2_genseq"}
        return {"kind": "dense", "model": "two_band", "n": _log_int(rng, 300, 6000),
                "precision": "exact_int8", "algorithm": "alg2"}
    if kind == "host":
        return {"kind": "host", "model": "two_band", "n": _log_int(rng, 64, 2000),
                "precision": rng.choice(["fp64", "mixed_fp16"]), "algorithm": "alg2"}
    if kind == "response":
        return {"kind": "response", "model": "two_band", "n": _log_int(rng, 64, 1500),
                "precision": "fp64"}
    if kind == "gradient":
        return {"kind": "gradient", "model": "two_band", "n": _log_int(rng, 200, 2048)}
    edge = rng.randint(10, 32)
    return {"kind": "subgraph", "edge": edge,
            "parts": max(4, int(edge ** 3 / rng.uniform(100, 160))),
            "precision": rng.choice(["exact_int8", "exact_int8", "fp64", "mixed_fp16"])}


# ----------------------------------------------------------------------------------
# Inputs
# ----------------------------------------------------------------------------------

def _hamiltonian(case, seed):
    """(H as a dense numpy array, bndfil): half filling, rounded up for odd sizes (the
    lower band of an odd two-band chain has one site more)."""
    n = case["n"]
    if case["model"] == "two_band":
        h = modelham.two_band_1d(n, seed=seed)
    else:
        h = modelham.cubic_3d(round(n ** (1.0 / 3.0)), seed=seed)
    return h, ((n + 1) // 2) / n


@functools.lru_cache(maxsize=8)
def _subgraph_parts(edge, parts, on_gpu):
    """Halo lists and sizes of the parts, from the H^2 graph of one configuration: a
    program keeps them while the disorder (the atoms' positions) changes."""
    n = edge ** 3
    build = graph.square_graph_gpu if on_gpu else graph.thresholded_square_graph
    g = build(modelham.cubic_3d_csr(edge, seed=0), n, GRAPH_THRESHOLD)
    nodes = graph.rcb_partition(graph.lattice_coords(edge), parts, seed=0, lo=0.4, hi=0.6)
    return sp2b.subgraph_halos(n, g, nodes, None, double_jump=False)


def _subgraph_problem(edge, parts, seed, on_gpu=True):
    """The flattened sub-graph problem of the edge^3 lattice: CSR H, halo lists, core
    sizes, branch sequence and bounds.  The chemical potential is that of an 8^3 lattice,
    the gap 5e-5 of the spectral width (the 32^3 lattice's), and the branch sequence
    prg_sp2sequence's for them."""
    n = edge ** 3
    rp, col, val = modelham.cubic_3d_csr(edge, seed=seed)
    rows = np.repeat(np.arange(n), np.diff(rp))
    diag = np.zeros(n)
    diag[rows[rows == col]] = val[rows == col]
    radius = np.bincount(rows, weights=np.abs(val), minlength=n) - np.abs(diag)
    emin, emax = float(np.min(diag - radius)), float(np.max(diag + radius))
    levels = np.linalg.eigvalsh(modelham.cubic_3d(8, seed=seed))
    mu = 0.5 * (levels[255] + levels[256])
    half_gap = 2.5e-5 * (emax - emin)
    pp, maxiter = sp2b.sp2sequence(emin, emax, mu - half_gap, mu + half_gap, 1e-12)
    halo_ptr, halo_idx, lsize, llsize = _subgraph_parts(edge, parts, on_gpu)
    return {"n": n, "rp": rp, "col": col, "val": val, "halo_ptr": halo_ptr, "halo_idx": halo_idx,
            "lsize": lsize, "llsize": llsize, "pp": np.array(pp, dtype=np.int32),
            "maxiter": maxiter, "emin": emin, "emax": emax}


def _gradient_inputs(case, seed):
    h, bndfil = _hamiltonian(case, seed)
    return h, modelham.random_symmetric(case["n"], seed=seed + 1), bndfil


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind, "precision": PRECISIONS.get(case.get("precision"))}
    if kind in ("dense", "host", "response"):
        h, s["bndfil"] = _hamiltonian(case, seed)
        n = s["n"] = case["n"]
        if kind == "host":
            s["h"] = h
            return s
        s["h"] = torch.from_numpy(h).cuda()
        s["rho"] = torch.empty_like(s["h"])
        s["pp"] = np.zeros(MAXITER + 2, dtype=np.int32)
        s["vv"] = np.zeros(MAXITER + 2)
        if kind == "response":
            h1 = modelham.random_symmetric(n, seed=seed + 1)
            s["h1"] = torch.from_numpy(h1).cuda()
            s["rho1"] = torch.empty_like(s["h"])
        return s
    if kind == "gradient":
        h, a, bndfil = _gradient_inputs(case, seed)
        s["h"] = torch.from_numpy(h).float().cuda()
        s["a"] = torch.from_numpy(a).float().cuda()
        s["pp"], s["emin"], s["emax"] = autograd.sequence_and_bounds(s["h"], bndfil)
        return s
    p = _subgraph_problem(case["edge"], case["parts"], seed)
    s.update({k: p[k] for k in ("n", "pp", "maxiter", "emin", "emax")})
    for k in ("rp", "col", "val", "halo_ptr", "halo_idx", "llsize"):
        s[k] = torch.from_numpy(p[k]).cuda()
    s["nparts"] = len(p["llsize"])
    s["core"] = torch.empty(int(np.sum(p["llsize"].astype(np.int64) * p["lsize"])),
                            dtype=torch.float64, device="cuda")
    s["vv"] = np.zeros(max(p["maxiter"], 1))
    return s


# ----------------------------------------------------------------------------------
# One pass
# ----------------------------------------------------------------------------------

def _device_opts(s):
    return _lib.make_opts(precision=s["precision"], device_ptrs=True,
                          stream=torch.cuda.current_stream().cuda_stream)


def _run_dense(s):
    L, o, n = _lib.lib(), _device_opts(s), s["n"]
    count = C.c_int(0)
    h, rho = s["h"].data_ptr(), s["rho"].data_ptr()
    if s["case"]["algorithm"] == "alg2_genseq":
        s["pp"][:] = 0
        s["vv"][:] = 0
        _lib.check(L.sp2b_sp2_alg2_genseq(h, rho, n, 0.0, s["bndfil"], 0, MAXITER, b"None", IDEMTOL,
                                          s["pp"].ctypes.data, C.byref(count), s["vv"].ctypes.data,
                                          0, C.byref(o)), "sp2_alg2_genseq")
        return s["rho"], s["pp"], s["vv"]
    solve = L.sp2b_sp2_alg1 if s["case"]["algorithm"] == "alg1" else L.sp2b_sp2_alg2
    _lib.check(solve(h, rho, n, 0.0, s["bndfil"], 0, MAXITER, b"None", IDEMTOL, 0, C.byref(o),
                     C.byref(count)), s["case"]["algorithm"])
    return s["rho"]


def _run_response(s):
    o = _device_opts(s)
    count = C.c_int(0)
    _lib.check(_lib.lib().sp2b_compute_response_sp2(
        s["h"].data_ptr(), s["h1"].data_ptr(), s["rho1"].data_ptr(), s["rho"].data_ptr(), s["n"], 0.0,
        s["bndfil"], 0, MAXITER, b"None", IDEMTOL, 0.0, 0, s["pp"].ctypes.data, C.byref(count),
        C.byref(o)), "compute_response_sp2")
    return s["rho"], s["rho1"]


def _run_gradient(s):
    h = s["h"].detach().requires_grad_(True)
    d = autograd.sp2_density(h, s["pp"], s["emin"], s["emax"])
    (d * s["a"]).sum().backward()
    return d.detach(), h.grad


def _run_subgraph(s):
    o = _device_opts(s)
    _lib.check(_lib.lib().sp2b_subgraph_sp2_loop(
        s["n"], s["rp"].data_ptr(), s["col"].data_ptr(), s["val"].data_ptr(), s["nparts"],
        s["halo_ptr"].data_ptr(), s["halo_idx"].data_ptr(), s["llsize"].data_ptr(),
        s["pp"].ctypes.data, s["maxiter"], s["emin"], s["emax"], s["core"].data_ptr(), None,
        s["vv"].ctypes.data, C.byref(o)), "subgraph_sp2_loop")
    return s["core"], s["vv"]


def run(state):
    kind = state["kind"]
    if kind == "dense":
        return _run_dense(state)
    if kind == "host":
        return sp2b.sp2_alg2(state["h"], state["bndfil"], 0, MAXITER, "None", IDEMTOL,
                             precision=state["precision"]).rho
    if kind == "response":
        return _run_response(state)
    if kind == "gradient":
        return _run_gradient(state)
    return _run_subgraph(state)


# ----------------------------------------------------------------------------------
# What a pass cannot do without, and how far correct results may lie apart
# ----------------------------------------------------------------------------------

def work(case):
    """One product of symmetric matrices with a symmetric result (n^2 (n + 1) operations)
    per SP2 step; a response or reverse step adds two products with one symmetric result.
    H is read once and each result written once."""
    kind = case["kind"]
    if kind == "subgraph":
        p = _subgraph_problem(case["edge"], case["parts"], 0, on_gpu=False)
        size = p["lsize"].astype(np.float64)
        core = float(np.sum(p["llsize"] * size))
        return {"bytes": float(12 * len(p["val"]) + 4 * len(p["halo_idx"])) + 8.0 * core,
                "flops": p["maxiter"] * float(np.sum(size * size * (size + 1.0)))}
    n = float(case["n"])
    product = n * n * (n + 1.0)
    steps = STEPS[case["model"]]
    if kind == "response":
        return {"bytes": 32.0 * n * n, "flops": 3.0 * steps * product}
    if kind == "gradient":
        return {"bytes": 16.0 * n * n, "flops": 3.0 * steps * product}
    return {"bytes": 16.0 * n * n, "flops": steps * product}


def tolerance(case):
    kind = case["kind"]
    precision = case.get("precision")
    if kind == "gradient":
        return {"rel": 2e-6}
    if kind == "subgraph":
        # states within rounding of the chemical potential decide the size of these
        return {"rel": {"fp64": 1e-11, "exact_int8": 4e-6, "mixed_fp16": 4e-3}[precision]}
    rel = {"fp64": 1e-12, "mixed_fp16": 3e-7, "mixed_bf16": 1e-5, "exact_int8": 1e-7}[precision]
    if case.get("algorithm") != "alg2_genseq":
        return {"rel": rel}
    # vv is summed from the split products' residuals; the last branches of a converged
    # solve are ties (X^2 and 2X - X^2 leave the same trace), and the split form stops up to
    # three steps before FP64
    return {"rel": max(rel, {"mixed_fp16": 1e-5, "mixed_bf16": 5e-5}.get(precision, 0.0)),
            "differ": 0.05}


# ----------------------------------------------------------------------------------
# The same results in plain FP64
# ----------------------------------------------------------------------------------

def _normalised(h):
    d = torch.diagonal(h)
    radius = h.abs().sum(1) - d.abs()
    emin, emax = float((d - radius).min()), float((d + radius).max())
    return _normalise(h, emin, emax), emin, emax


def _normalise(h, emin, emax):
    x = -h / (emax - emin)
    torch.diagonal(x).add_(emax / (emax - emin))
    return x


def _alg2(h, bndfil, d=None):
    """The alg2 recursion in FP64, with a first-order response when d is given: X, response,
    ||X_k - X_k^2||_F and branch of every step."""
    occ = bndfil * h.shape[0]
    x, emin, emax = _normalised(h)
    if d is not None:
        d = -d / (emax - emin)
    vv, pp = [], []
    for _ in range(MAXITER):
        x2 = x @ x
        tr, tr2 = float(torch.trace(x)), float(torch.trace(x2))
        diff = abs(tr2 - occ) - abs(2.0 * tr - tr2 - occ)
        if abs(diff) < IDEMTOL:
            break
        vv.append(float((x - x2).norm()))
        pp.append(0 if diff > 0 else 1)
        if d is not None:
            xd = x @ d
            anti = xd + xd.T
            d = 2.0 * d - anti if diff > 0 else anti
        x = 2.0 * x - x2 if diff > 0 else x2
    return x, d, vv, pp, emin, emax


def _exact_subgraph(case, seed):
    p = _subgraph_problem(case["edge"], case["parts"], seed)
    n = p["n"]
    rows = np.repeat(np.arange(n), np.diff(p["rp"]))
    h = torch.sparse_coo_tensor(torch.from_numpy(np.stack([rows, p["col"].astype(np.int64)])),
                                torch.from_numpy(p["val"]), (n, n)).cuda().coalesce()
    core, vv = [], torch.zeros(p["maxiter"], dtype=torch.float64, device="cuda")
    (hr, hc), hv = h.indices(), h.values()
    where = torch.empty(n, dtype=torch.int64, device="cuda")
    for q in range(len(p["llsize"])):
        nodes = torch.from_numpy(p["halo_idx"][p["halo_ptr"][q]:p["halo_ptr"][q + 1]]).cuda().long()
        m, mc = len(nodes), int(p["llsize"][q])
        where.fill_(-1)
        where[nodes] = torch.arange(m, device="cuda")
        keep = (where[hr] >= 0) & (where[hc] >= 0)
        x = torch.zeros(m, m, dtype=torch.float64, device="cuda")
        x[where[hr[keep]], where[hc[keep]]] = hv[keep]
        x = _normalise(x, p["emin"], p["emax"])
        for k in range(p["maxiter"]):
            y = x - x @ x
            vv[k] += (y[:mc] ** 2).sum()
            x = x - y if p["pp"][k] == 1 else x + y
        core.append(2.0 * x[:mc].reshape(-1))
    return torch.cat(core), vv.sqrt().cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "subgraph":
        return _exact_subgraph(case, seed)
    if kind == "gradient":
        h, a, bndfil = _gradient_inputs(case, seed)
        h = torch.from_numpy(h).float().double().cuda()
        a = torch.from_numpy(a).float().double().cuda()
        _, _, _, pp, emin, emax = _alg2(h, bndfil)
        h.requires_grad_(True)
        x = -h / (emax - emin) + torch.eye(case["n"], dtype=h.dtype, device=h.device) * (emax / (emax - emin))
        for b in pp:
            x2 = x @ x
            x = x2 if b == 1 else 2.0 * x - x2
        d = 2.0 * x
        (d * a).sum().backward()
        return d.detach(), h.grad
    h, bndfil = _hamiltonian(case, seed)
    h = torch.from_numpy(h).cuda()
    if kind == "response":
        h1 = torch.from_numpy(modelham.random_symmetric(case["n"], seed=seed + 1)).cuda()
        x, d, _, _, _, _ = _alg2(h, bndfil, h1)
        return 2.0 * x, 2.0 * d
    x, _, vv, pp, _, _ = _alg2(h, bndfil)
    rho = 2.0 * x
    if kind == "host":
        return rho.cpu().numpy()
    if case["algorithm"] != "alg2_genseq":
        return rho
    full_pp = np.zeros(MAXITER + 2, dtype=np.int32)
    full_vv = np.zeros(MAXITER + 2)
    full_pp[:len(pp)] = pp
    full_vv[:len(vv)] = vv
    return rho, full_pp, full_vv
