"""Workloads of the library as its users run them, through the public Python entry points.

Every case names one call: a block solve (`gpu_solve_sources`), one application of the operator
(`GPUDielectricOperator.matvec_device`, `op @ X`), potentials at probe points (`laplace3d_pottrg`),
or a burst of requests to the request server (`SolveServer`). What a program keeps between
calls (mesh, near-field blocks, device geometry, server) is made by `prepare`; sources, charges and
densities come from the seed. `exact` gives the same result from a dense FP64 matrix in plain torch;
the mesh and the correction blocks are inputs there, as they are for the operator.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    name = "dielectricbie_jl_b200"  # the package's folder name is not a Python identifier
    if name not in sys.modules:
        folder = os.path.abspath("dielectricbie.jl_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


def listed():
    return [
        # One plain FP64 solve on a small box, one source, to 1e-12: the smallest call, where the
        # iteration's launches and host checks count.
        _solve("solve_small_fp64", 1.2, 0.8, 0.6, 4, 0.2, 4.0, 1, "fp64", False, 1e-12),
        # A few sources in a small box: what a request of a parameter study looks like.
        _solve("solve_small_block", 1.0, 0.9, 0.7, 4, 0.25, 4.0, 8, "bf16x3", True, 1e-10),
        # One source in a medium box with the FP32 operator inside the refinement.
        _solve("solve_single_fp32", 1.1, 0.9, 0.6, 6, 0.12, 4.0, 1, "fp32", False, 1e-10),
        # An odd number of sources, one Arnoldi process per column (the default of gpu_solve).
        _solve("solve_columns_odd", 1.3, 0.9, 0.7, 6, 0.1, 3.0, 19, "bf16x3", False, 1e-10),
        # The benchmark's box: 64 sources at once, refined.
        _solve("solve_block_refined", 1.5, 1.0, 0.8, 6, 0.08, 4.0, 64, "bf16x3", True, 1e-10),
        # The same in plain FP64, the form that needs no trust in a reduced precision.
        _solve("solve_block_fp64", 1.5, 1.0, 0.8, 6, 0.08, 4.0, 64, "fp64", True, 1e-10),
        # A finer box and a stronger contrast, 8 sources.
        _solve("solve_large_refined", 2.0, 1.0, 1.0, 6, 0.05, 10.0, 8, "bf16x3", True, 1e-10),
        # A lattice of eight dielectric cubes, 16 sources between them: the largest call.
        dict(_solve("solve_lattice", 0.5, 0.5, 0.5, 6, 0.05, 4.0, 16, "bf16x3", True, 1e-10), cubes=2, gap=0.2),
        # One FP64 operator application on device vectors: the step of a caller's own Krylov loop.
        _case("matvec", "matvec_single", 1.5, 1.0, 0.8, 6, 0.08, 4.0, k=1, host=False),
        # mul! on host arrays, as the Julia solvers call it, with an odd block of columns.
        _case("matvec", "matvec_host_block", 1.1, 0.9, 0.6, 6, 0.12, 4.0, k=13, host=True),
        # Potentials of 64 densities at 1,000 exterior probes.
        _case("potential", "potential_probes", 1.5, 1.0, 0.8, 6, 0.08, 4.0, k=64, probes=1000),
        # A burst of requests over boxes of uneven size, 1 to 6 sources each, to the server.
        _case("serve", "serve_burst", 1.1, 0.9, 0.6, 6, 0.12, 4.0, requests=24),
    ]


def _case(kind, name, lx, ly, lz, n_quad, l_ec, eps, **more):
    return dict(name=name, kind=kind, lx=lx, ly=ly, lz=lz, n_quad=n_quad, l_ec=l_ec, eps=eps, cubes=0, gap=0.0, **more)


def _solve(name, lx, ly, lz, n_quad, l_ec, eps, k, precision, block, rtol):
    return _case("solve", name, lx, ly, lz, n_quad, l_ec, eps, k=k, precision=precision, block=block, rtol=rtol)


def draw(rng):
    """Boxes of about 1,500 to 75,000 nodes with sides in [0.6, 1.8] and contrasts of 2 to 10, 1 to 96 columns."""
    kind = rng.choice(["solve", "solve", "solve", "solve", "matvec", "matvec", "potential", "serve"])
    n_quad = rng.choice([4, 6])
    lx, ly, lz = (round(rng.uniform(0.6, 1.8), 3) for _ in range(3))
    area = 2 * (lx * ly + ly * lz + lx * lz)
    nodes = math.exp(rng.uniform(math.log(1500), math.log(20000 if kind == "serve" else 50000)))
    l_ec = round(math.sqrt(area * n_quad ** 2 / nodes), 4)
    eps = round(math.exp(rng.uniform(math.log(2.0), math.log(10.0))), 3)
    k = int(round(math.exp(rng.uniform(0.0, math.log(96.0)))))
    if kind == "solve":
        precision = rng.choice(["fp64", "fp32", "bf16x3", "bf16x3", "bf16x6"])
        if precision == "fp32":
            k = min(k, 4)  # the FP32 operator is the one for few columns
        return {x: v for x, v in _solve("", lx, ly, lz, n_quad, l_ec, eps, k, precision, rng.random() < 0.5,
                                        1e-10).items() if x != "name"}
    more = {"matvec": dict(k=k, host=rng.random() < 0.5), "potential": dict(k=k, probes=rng.randrange(100, 3000)),
            "serve": dict(requests=rng.randrange(6, 32))}[kind]
    return {x: v for x, v in _case(kind, "", lx, ly, lz, n_quad, l_ec, eps, **more).items() if x != "name"}


def _interface(case, scale=1.0, l_ec=None):
    bie = _package()
    l_ec = case["l_ec"] if l_ec is None else l_ec
    if case["cubes"]:
        m, pitch = case["cubes"], case["lx"] + case["gap"]
        boxes = [((a * pitch, b * pitch, c * pitch), case["lx"], case["ly"], case["lz"])
                 for a in range(m) for b in range(m) for c in range(m)]
        return bie.multi_dielectric_box3d(case["n_quad"], l_ec, boxes, [case["eps"]] * len(boxes), 1.0)
    return bie.single_dielectric_box3d(case["lx"] * scale, case["ly"] * scale, case["lz"], case["n_quad"], l_ec,
                                       case["eps"], 1.0)


def _sources(case, rng, k, scale=1.0):
    """Positions (k, 3), charges (k) and the permittivity at the sources."""
    if case["cubes"]:
        # centres of the gaps between the cubes, shifted a little; charges +-1
        m, pitch = case["cubes"], case["lx"] + case["gap"]
        cell = rng.integers(0, 2 * m - 1, size=(k, 3))
        cell[np.arange(k), rng.integers(0, 3, size=k)] = 2 * rng.integers(0, m - 1, size=k) + 1
        pos = cell * (pitch / 2) + rng.uniform(-0.1, 0.1, size=(k, 3)) * case["gap"]
        return pos, rng.choice([-1.0, 1.0], size=k), 1.0
    half = np.array([case["lx"] * scale, case["ly"] * scale, case["lz"]]) / 2 * 0.8
    return rng.uniform(-half, half, size=(k, 3)), rng.standard_normal(k), case["eps"]


def _operator(itf, precision="fp64"):
    return _package().lhs_dielectric_box3d_fmm3d_corrected(itf, 1e-12, 1e-9, 8, precision=precision)


def _point_sources(pos, q):
    bie = _package()
    return [bie.PointSource(tuple(map(float, p)), float(c)) for p, c in zip(pos, q)]


def _probes(itf, rng, count):
    """Exterior points 0.1 to 0.5 off a random surface node."""
    at = rng.integers(0, itf.n, size=count)
    return itf.points[at] + itf.normals[at] * rng.uniform(0.1, 0.5, size=count)[:, None]


# Uneven boxes of the server's burst: sides and mesh size relative to the case's own.
SERVED = ((1.0, 1.0), (0.9, 1.6), (0.8, 2.0), (0.7, 2.6), (0.6, 3.0))


def _requests(case, rng):
    """(box, positions, charges) of each request: repeated boxes in a mixed order, 1 to 6 sources."""
    out = []
    for i in range(case["requests"]):
        box = (i * 7 + i // 3) % len(SERVED)
        pos, q, _ = _sources(case, rng, 1 + (i * 5 + i // 4) % 6, SERVED[box][0])
        out.append((box, pos, q))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    state = {"case": case}
    if case["kind"] == "serve":
        state["itfs"] = [_interface(case, s, case["l_ec"] * f) for s, f in SERVED]
        state["ops"] = [_operator(i, "bf16x3") for i in state["itfs"]]
        state["requests"] = [(box, _point_sources(pos, q)) for box, pos, q in _requests(case, rng)]
        state["server"] = _package().SolveServer(hbm_fraction=0.2)
        return state
    itf = state["itf"] = _interface(case)
    if case["kind"] == "solve":
        pos, q, state["eps_src"] = _sources(case, rng, case["k"])
        state["op"] = _operator(itf, case["precision"])
        state["sources"] = _point_sources(pos, q)
    elif case["kind"] == "matvec":
        state["op"] = _operator(itf)
        x = rng.standard_normal((itf.n, case["k"]))
        if case["host"]:
            state["X"] = np.asfortranarray(x)
        else:
            state["X"] = torch.from_numpy(x).cuda()  # node-major, the layout of the device entry
            state["Y"] = torch.empty_like(state["X"])
            state["stream"] = torch.cuda.Stream()
    else:
        state["S"] = np.asfortranarray(rng.standard_normal((itf.n, case["k"])))
        state["op"] = _package().laplace3d_pottrg(itf, _probes(itf, rng, case["probes"]))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        return _package().gpu_solve_sources(state["op"], state["sources"], state["eps_src"], rtol=case["rtol"],
                                            block=case["block"])[0]
    if case["kind"] == "matvec":
        if case["host"]:
            return state["op"] @ state["X"]
        state["op"].matvec_device(state["X"].data_ptr(), state["Y"].data_ptr(), case["k"],
                                  stream=state["stream"].cuda_stream)
        return state["Y"]
    if case["kind"] == "potential":
        return state["op"] @ state["S"]
    server = state["server"]
    tickets = [server.submit_sources(state["ops"][box], sources, case["eps"], rtol=1e-10)
               for box, sources in state["requests"]]
    return [server.result(t)[0] for t in tickets]


_nodes = {}


def _size(case, scale=1.0, factor=1.0):
    key = (case["cubes"], case["gap"], case["lx"] * scale, case["ly"] * scale, case["lz"], case["n_quad"],
           case["l_ec"] * factor)
    if key not in _nodes:
        _nodes[key] = _interface(case, scale, case["l_ec"] * factor).n
    return _nodes[key]


def work(case):
    """Nodes and correction blocks (about 7 of n_quad^4 values a panel) read once, inputs read and
    results written once; 20 operations a kernel value and 2 a column, in each operator application. A
    solve to 1e-10 applies the operator about 16 times."""
    def one(n, k, applied):
        blocks = 7.0 * n * case["n_quad"] ** 2 * 8
        return 8.0 * (8 * n + 2 * n * k) + blocks, applied * float(n) ** 2 * (20 + 2 * k)

    if case["kind"] == "serve":
        share = case["requests"] / len(SERVED)
        total = [one(_size(case, s, f), 3.5 * share, 16) for s, f in SERVED]
        return {"bytes": sum(t[0] for t in total), "flops": sum(t[1] for t in total)}
    n, k = _size(case), case["k"]
    if case["kind"] == "potential":
        return {"bytes": 8.0 * (4 * n + n * k + case["probes"] * (3 + k)), "flops": float(n) * case["probes"] * (14 + 2 * k)}
    b, f = one(n, k, 16 if case["kind"] == "solve" else 1)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------------
# The same results from a dense matrix in plain FP64.
# ---------------------------------------------------------------------------------------------
def _dense(itf):
    """D^T (j != i), diagonal and correction blocks as one N x N matrix on the GPU."""
    x, nrm, w, diag = (torch.from_numpy(v).cuda() for v in (itf.points, itf.normals, itf.weights, itf.diag))
    n = itf.n
    A = torch.empty((n, n), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // n)
    for lo in range(0, n, step):
        hi = min(n, lo + step)
        num, r2 = None, None
        for a in range(3):
            d = x[lo:hi, a, None] - x[None, :, a]
            num = nrm[lo:hi, a, None] * d if num is None else num + nrm[lo:hi, a, None] * d
            r2 = d * d if r2 is None else r2 + d * d
        own = torch.arange(lo, hi, device="cuda")
        r2[own - lo, own] = 1.0
        v = num / (r2 * r2.sqrt()) * (w / (4 * math.pi))
        v[own - lo, own] = diag[lo:hi]
        A[lo:hi] = v
    near = itf.near(8, 1e-9, True, _package().AdaptiveConfig(1e-9))
    nb = near.nb
    rows = np.repeat(np.arange(itf.npanels), np.diff(near.rowptr))
    blocks = torch.from_numpy(near.val.reshape(-1, nb, nb)).cuda()  # [block][column][row]
    view = A.view(itf.npanels, nb, itf.npanels, nb)
    p, q = torch.from_numpy(rows).cuda(), torch.from_numpy(near.col.astype(np.int64)).cuda()
    for lo in range(0, len(rows), 2000):
        s = slice(lo, lo + 2000)
        view[p[s], :, q[s], :] += blocks[s].transpose(1, 2)
    return A


def _rhs(itf, pos, q, eps):
    x, nrm = torch.from_numpy(itf.points).cuda(), torch.from_numpy(itf.normals).cuda()
    d = x[:, None, :] - torch.from_numpy(pos).cuda()[None]
    r2 = (d * d).sum(-1)
    return -(d * nrm[:, None, :]).sum(-1) / (r2 * r2.sqrt()) / (4 * math.pi * eps) * torch.from_numpy(q).cuda()


def _solution(A, F):
    LU = torch.linalg.lu_factor(A)
    S = torch.linalg.lu_solve(*LU, F)
    return S + torch.linalg.lu_solve(*LU, F - A @ S)


def exact(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "serve":
        todo = _requests(case, rng)
        out = [None] * len(todo)
        for box, (s, f) in enumerate(SERVED):
            mine = [i for i, t in enumerate(todo) if t[0] == box]
            if not mine:
                continue
            itf = _interface(case, s, case["l_ec"] * f)
            F = torch.cat([_rhs(itf, todo[i][1], todo[i][2], case["eps"]) for i in mine], 1)
            S = _solution(_dense(itf), F).cpu().numpy()
            at = 0
            for i in mine:
                k = len(todo[i][2])
                out[i] = S[:, at:at + k]
                at += k
        return out
    itf = _interface(case)
    if case["kind"] == "potential":
        S = rng.standard_normal((itf.n, case["k"]))
        at = torch.from_numpy(_probes(itf, rng, case["probes"])).cuda()
        x, w = torch.from_numpy(itf.points).cuda(), torch.from_numpy(itf.weights).cuda()
        r2 = sum((at[:, a, None] - x[None, :, a]) ** 2 for a in range(3))
        return ((w / (4 * math.pi)) / r2.sqrt() @ torch.from_numpy(S).cuda()).cpu().numpy()
    if itf.n > 50000:
        return None  # the factorisation takes too long
    if case["kind"] == "matvec":
        Y = _dense(itf) @ torch.from_numpy(rng.standard_normal((itf.n, case["k"]))).cuda()
        return Y.cpu().numpy()
    pos, q, eps = _sources(case, rng, case["k"])
    return _solution(_dense(itf), _rhs(itf, pos, q, eps)).cpu().numpy()
