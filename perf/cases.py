"""Workloads of the BorderedCR solver on the GPU.

A case is one pass of the work a caller repeats, through the public Python
classes of ``alglin_b200.bcr``:

* ``step``  -- the Newton step: factorize the loaded matrix and solve for new
  right-hand sides (``factorize_solve_device``), everything on the device;
* ``graph`` -- the same step as a captured CUDA graph (``graph_launch``), for
  systems so small that the launches count;
* ``solve`` -- a simplified Newton step: the factors are kept, only the
  right-hand sides are new (``solve_device``);
* ``host``  -- the call a program ported from the C++ class makes: matrix in the
  object's host blocks, right-hand side in host memory, one
  ``factorize_solve``;
* ``batch`` -- many uneven systems (multiple BVPs, or the subproblems of a
  parametric study) in one ``Batch`` step.

The matrices are trapezoid collocations (``alglin_b200.synth``): D = -I - hJ/2,
E = I - hJ/2 with borders, h = 1/nblock.  The right-hand side is A*x for an x
drawn from N(0,1), so the exact solution is known; A*x is formed with torch in
64 bits.  ``mixed`` cases ask the refinement for the accuracy of the FP64 path
(1e-15 instead of the default 1e-12).
"""
from __future__ import annotations

import random

import numpy as np
import torch

from alglin_b200 import bcr, synth

F64 = torch.float64
REFINE_TOL = 1e-15


def _case(name, op, nblock, n, qr=0, qx=0, nr=0, nx=0, nrhs=1, select="LU", mixed=False):
    return {"name": name, "op": op, "nblock": nblock, "n": n, "qr": qr, "qx": qx, "nr": nr, "nx": nx,
            "nrhs": nrhs, "select": select, "mixed": mixed}


def listed():
    return [
        # a single shooting/collocation BVP with 8 states inside a Newton loop:
        # about 40 dependent kernels, nothing but latency
        _case("graph_n8", "graph", 1000, 8, nr=2, nx=2),
        # the largest mesh at the common block size: an optimal-control problem
        # with 8 states and 8 costates, parameters and control borders
        _case("step_n16", "step", 100000, 16, 2, 2, 4, 4),
        # the same with several right-hand sides (sensitivities)
        _case("step_n16_rhs8", "step", 30000, 16, 2, 2, 4, 4, nrhs=8),
        # simplified Newton: old factors, new right-hand side
        _case("solve_n16", "solve", 50000, 16, 2, 2, 4, 4),
        # Householder panels, for users who do not trust partial pivoting
        _case("step_n16_qr", "step", 20011, 16, 2, 2, 4, 4, select="QR"),
        # 6 states + 6 costates: block sizes of real problems are no powers of two
        _case("step_n12", "step", 20011, 12, 1, 2, 4, 3),
        # larger state vectors, factors in FP64 and in FP32 with refinement
        _case("step_n32", "step", 16384, 32, nr=8, nx=8),
        _case("mixed_n32", "step", 16384, 32, nr=8, nx=8, mixed=True),
        # semi-discretised PDEs: large blocks, factors in FP64 and in FP32
        _case("step_n128", "step", 1024, 128, 4, 4, 16, 16),
        _case("mixed_n128", "step", 1024, 128, 4, 4, 16, 16, mixed=True),
        # the Newton steps of 512 independent BVPs, nblock in [64, 1024],
        # n in {4, 8, 16, 32}
        {"name": "batch_512", "op": "batch", "systems": 512, "lo": 64, "hi": 1024, "mixed": False},
        # a caller of the C++ class who changes nothing but the library
        _case("host_n16", "host", 20000, 16, 2, 2, 4, 4),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng: random.Random):
    op = rng.choice(["step"] * 8 + ["graph", "graph", "solve", "solve", "host", "batch"])
    if op == "batch":
        lo = _log_int(rng, 16, 256)
        return {"op": "batch", "systems": _log_int(rng, 60, 512), "lo": lo, "hi": _log_int(rng, 2 * lo, 1024),
                "mixed": False}
    select = rng.choice(["LU"] * 5 + ["QR"])
    mixed = op == "step" and select == "LU" and rng.random() < 0.25
    if select == "QR":
        n = _log_int(rng, 2, 24)
    elif op == "host":
        n = _log_int(rng, 4, 32)
    else:
        n = rng.choice([8, 16, 32, 64, 128] + [_log_int(rng, 2, 128) for _ in range(5)])
    # at most the matrix of 100000 blocks of order 16, fewer for larger blocks
    # (the work per entry grows with n); the smallest meshes have a few blocks
    most = {"graph": 2000, "host": 20000}.get(op, 100000)
    most = min(most, int(25_600_000 / (n * n)), int(2.2e9 / n ** 3))
    if select == "QR":
        most = min(most, 20000)
    nblock = _log_int(rng, min(64, most), most)
    nr, nx = rng.randint(0, 8), rng.randint(0, 8)
    if n > 32 and rng.random() < 0.5:
        nr, nx = rng.randint(9, 16), rng.randint(9, 16)
    extra = rng.choice([0, 0, 1, 2])  # square: n + qr + nr rows against n + qx + nx columns
    qr, qx = extra + max(0, nx - nr), extra + max(0, nr - nx)
    nrhs = rng.choice([1, 1, 1, 2, 5, 8, 16]) if op in ("step", "solve") and not mixed else 1
    c = _case("", op, nblock, n, qr, qx, nr, nx, nrhs, select, mixed)
    del c["name"]
    return c


def _batch_dims(case, seed):
    # one seed of the sizes for all inputs of a case: the batch's plan is kept,
    # its matrices change
    return synth.batch_dims(case["systems"], case["lo"], case["hi"], seed=case["systems"])


def _dims(case):
    return tuple(case[k] for k in ("nblock", "n", "qr", "qx", "nr", "nx"))


def _times(dims, blocks, x):
    """A * x for x of shape (nrhs, ncols), in 64 bits."""
    nb, n, qr, qx, nr, nx = dims
    D, E, B, C, Cq, F, H = blocks
    r = x.shape[0]
    xs = x[:, :(nb + 1) * n].reshape(r, nb + 1, n)
    xq = x[:, (nb + 1) * n:(nb + 1) * n + qx]
    xb = x[:, (nb + 1) * n + qx:]
    rows = torch.einsum("kji,rkj->rki", D, xs[:, :-1]) + torch.einsum("kji,rkj->rki", E, xs[:, 1:])
    rows = rows + torch.einsum("kji,rj->rki", B, xb)
    ends = torch.cat([xs[:, 0], xs[:, nb], xq, xb], dim=1)
    bottom = ends @ H
    border = torch.einsum("kjr,skj->sr", C, xs) + xq @ Cq + xb @ F
    return torch.cat([rows.reshape(r, nb * n), bottom, border], dim=1)


def _system(dims, seed, nrhs):
    blocks = synth.collocation_torch(torch, *dims, seed=seed)
    nb, n, _, qx, _, nx = dims
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)
    x = torch.randn((nrhs, (nb + 1) * n + qx + nx), generator=g, device="cuda", dtype=F64)
    return blocks, x


class _DeviceArray:
    """A device vector of the library as torch can view it."""

    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _prepare_batch(case, seed):
    dims = _batch_dims(case, seed)
    b = bcr.Batch()
    for d in dims:
        b.add_device(*d)
    if case["mixed"]:
        b.set_precision(bcr.PRECISION_MIXED)
        b.set_refinement(REFINE_TOL, 30)
    b.prepare()
    views = []
    for i, d in enumerate(dims):
        blocks, x = _system(d, 1000 * seed + i, 1)
        rhs = _times(d, blocks, x)[0]
        torch.cuda.synchronize()
        b.load_device(i, *[t.data_ptr() if t.numel() else 0 for t in blocks])
        torch.as_tensor(_DeviceArray(b.device_b(i), rhs.numel()), device="cuda").copy_(rhs)
        views.append(torch.as_tensor(_DeviceArray(b.device_x(i), rhs.numel()), device="cuda"))
    torch.cuda.synchronize()
    b.graph_capture()
    return {"op": "batch", "batch": b, "views": views, "stream": torch.cuda.ExternalStream(b.stream())}


def prepare(case, seed):
    if case["op"] == "batch":
        return _prepare_batch(case, seed)
    dims, nrhs = _dims(case), case["nrhs"]
    blocks, x = _system(dims, seed, nrhs)
    rhs = _times(dims, blocks, x).contiguous()
    h = bcr.BorderedCR()
    stream = torch.cuda.Stream()
    h.set_stream(stream.cuda_stream)
    h.load_system(synth.BABD(*dims, *[t.cpu().numpy() for t in blocks]))
    h.select(case["select"])
    h.select_last("LU")
    if case["mixed"]:
        h.set_precision(bcr.PRECISION_MIXED)
        h.set_refinement(REFINE_TOL, 10)
    state = {"op": case["op"], "solver": h, "stream": stream, "nrhs": nrhs, "ld": rhs.shape[1]}
    if case["op"] == "host":
        # right-hand side and solution in page-locked memory of the caller
        state["rhs"] = rhs.cpu().numpy()
        state["x"] = torch.empty(rhs.shape, dtype=F64, pin_memory=True).numpy()
        return state
    state["rhs"], state["x"] = rhs, torch.empty_like(rhs)
    h.upload()
    torch.cuda.synchronize()
    if case["op"] == "graph":
        h.graph_capture(bcr.GRAPH_STEP, nrhs, state["x"].data_ptr(), state["ld"], rhs.data_ptr())
    elif case["op"] == "solve":
        h.factorize_device()
    return state


def run(state):
    op = state["op"]
    if op == "batch":
        state["batch"].graph_launch()
        with torch.cuda.stream(state["stream"]):
            return torch.cat(state["views"])
    h, x = state["solver"], state["x"]
    if op == "graph":
        h.graph_launch(bcr.GRAPH_STEP)
    elif op == "host":
        np.copyto(x, state["rhs"])
        h.factorize_solve(state["nrhs"], x.reshape(-1), state["ld"])
    else:
        with torch.cuda.stream(state["stream"]):
            x.copy_(state["rhs"])
        if op == "step":
            h.factorize_solve_device(state["nrhs"], x.data_ptr(), state["ld"])
        else:
            h.solve_device(state["nrhs"], x.data_ptr(), state["ld"])
    return x


def _system_work(dims, nrhs, solve_only=False):
    nb, n, qr, qx, nr, nx = dims
    per_matrix = 2 * n * n + n * nx + nr * n
    cols = (nb + 1) * n + qx + nx
    if solve_only:
        # the factors (2n x n panel, U row of 2n + nx columns, border row) and
        # the vectors in and out
        entries = nb * (4 * n * n + n * nx + nr * n)
        flops = 2.0 * nb * nrhs * (2 * n * n + 2 * n * n + n * nx + nr * n)
        return 8.0 * (entries + 2 * cols * nrhs), flops
    # one elimination per block: n rank-one updates of a (2n + nr) x (3n + nx)
    # work matrix of which a third is zero, then the sweeps
    flops = nb * sum(2.0 * (2 * n + nr - i - 1) * (n - i - 1) + (2 * n + nr - i) for i in range(n))
    flops += nb * 2.0 * n * (n + nr) * (2 * n + nx) + nb * 1.0 * n * n * (2 * n + nx)
    flops += 2.0 * nb * nrhs * (4 * n * n + n * nx + nr * n)
    return 8.0 * (nb * per_matrix + 2 * cols * nrhs), flops


def work(case):
    """Matrix, right-hand sides and solution once; the eliminations of the reduction."""
    if case["op"] == "batch":
        w = [_system_work(d, 1) for d in _batch_dims(case, 0)]
        return {"bytes": sum(a for a, _ in w), "flops": sum(b for _, b in w)}
    b, f = _system_work(_dims(case), case["nrhs"], case["op"] == "solve")
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """The x the right-hand sides were made from."""
    if case["op"] == "batch":
        return torch.cat([_system(d, 1000 * seed + i, 1)[1][0] for i, d in enumerate(_batch_dims(case, seed))])
    x = _system(_dims(case), seed, case["nrhs"])[1]
    return x.cpu().numpy() if case["op"] == "host" else x
