"""The calls whose time matters, over the range of orders, batch sizes, matrix classes, data types
and entry points that this library is used with.

A case is one pass through a public entry point of ``tokura_zgeev_batched_gb300``, as a program
calls it with its matrices on the GPU, a handle, and (where the entry point takes one) a workspace
kept from call to call:

* ``zgeev``: ``api.zgeev_batched``, complex128 matrices of one order;
* ``cgeev``: ``api.cgeev_batched``, complex64 in and out;
* ``strided``: ``api.zgeev_strided`` on blocks of larger matrices, read in place;
* ``ragged``: ``api.zgeev_ragged``, an order per matrix;
* ``dgeev``, ``sgeev``: ``api.dgeev_batched`` on float64 / float32 matrices;
* ``vectors``: ``api.zgeev_vectors``, eigenvalues with left and right eigenvectors;
* ``grad``: forward and backward of ``autograd.eigvals`` under a smooth loss;
* ``ragged_grad``: a gradient-descent step through ``autograd.eigvals_ragged``.

A QR iteration returns a matrix's eigenvalues in the order in which they deflate, which rounding
may change, so every pass ends as a program that compares or tracks spectra does: the eigenvalues
of each matrix are put in order, by Re + 0.618 Im (which also separates conjugate pairs).
"""
from __future__ import annotations

import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from tokura_zgeev_batched_gb300 import api
from tokura_zgeev_batched_gb300 import autograd as ag
from tokura_zgeev_batched_gb300 import workloads as wl

# Weight of the imaginary part in the order that a pass puts eigenvalues in.
ORDER_IM = 0.618
# Smallest distance between two eigenvalues of a matrix that is differentiated.
MIN_SEP = 0.05
# Step length of the gradient-descent case.
LEARNING_RATE = 1e-2


def listed():
    return [
        # One control problem at a time: a handful of small matrices, where latency counts.
        {"name": "zgeev n8 b16", "kind": "zgeev", "dist": "gaussian", "n": 8, "batch": 16},
        # Very many tiny matrices (per-pixel, per-cell problems).
        {"name": "zgeev n4 b1048576", "kind": "zgeev", "dist": "gaussian", "n": 4, "batch": 1048576},
        # A full batch of a small order, matrices with prescribed spectra V diag V^-1.
        {"name": "zgeev n16 b65536 vdv", "kind": "zgeev", "dist": "vdv", "n": 16, "batch": 65536},
        # The benchmark's first configuration: a batch that does not fill the GPU.
        {"name": "zgeev n32 b10000", "kind": "zgeev", "dist": "gaussian", "n": 32, "batch": 10000},
        # The benchmark's default workload: the largest order at a full batch (4 GiB).
        {"name": "zgeev n64 b65536", "kind": "zgeev", "dist": "gaussian", "n": 64, "batch": 65536},
        # Polynomial roots: odd order, odd batch of a few matrices per SM, sparse structured input.
        {"name": "zgeev n47 b1003 companion", "kind": "zgeev", "dist": "companion", "n": 47, "batch": 1003},
        # Single-precision complex data, solved in double precision.
        {"name": "cgeev n24 b30000", "kind": "cgeev", "dist": "gaussian", "n": 24, "batch": 30000},
        # Mixed orders in one call.
        {"name": "ragged 1-64 b20000", "kind": "ragged", "dist": "gaussian", "nmin": 1, "nmax": 64, "batch": 20000},
        # Real matrices (the dgeev entry point).
        {"name": "dgeev n64 b16384", "kind": "dgeev", "dist": "gaussian", "n": 64, "batch": 16384},
        # Modal analysis: eigenvalues with both sets of eigenvectors.
        {"name": "vectors n32 b8192", "kind": "vectors", "dist": "gaussian", "n": 32, "batch": 8192},
        # Training through eigenvalues: forward and backward.
        {"name": "grad n48 b8192", "kind": "grad", "dist": "vdv", "n": 48, "batch": 8192},
        # A gradient-descent step on matrices of mixed orders.
        {"name": "ragged_grad 8-64 b4000", "kind": "ragged_grad", "dist": "vdv", "nmin": 8, "nmax": 64, "batch": 4000},
    ]


# Relative cost of a pass of each kind against the eigenvalues of complex matrices of one order.
_COST = {"zgeev": 1.0, "cgeev": 1.0, "strided": 1.0, "ragged": 1.2, "dgeev": 0.6, "sgeev": 0.6, "vectors": 3.0,
         "grad": 3.0, "ragged_grad": 3.0}
# Weights of a drawn case's kind: the plain call most often.
_DRAW = [("zgeev", 6), ("cgeev", 1), ("strided", 1), ("ragged", 2), ("dgeev", 2), ("sgeev", 1), ("vectors", 2),
         ("grad", 2), ("ragged_grad", 1)]


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, math.floor(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choices([k for k, _ in _DRAW], [w for _, w in _DRAW])[0]
    differentiated = kind in ("grad", "ragged_grad")
    case = {"kind": kind, "dist": "vdv" if differentiated else
            rng.choice(["gaussian", "uniform"]) if kind in ("dgeev", "sgeev", "ragged") else
            rng.choice(["gaussian", "gaussian", "vdv", "companion", "uniform"])}
    if kind in ("ragged", "ragged_grad"):
        lo = _log_int(rng, 2 if differentiated else 1, 32)
        case["nmin"], case["nmax"] = lo, rng.randint(lo, 64)
        size = case["nmax"]
    else:
        case["n"] = size = _log_int(rng, 2, 64)
    # At most an eighth of the largest listed case's operations, and of its bytes; a small order's
    # cost is not all in n^3, hence n (n + 8)^2.
    most = min(65536 * 64 ** 3 / 8 / (_COST[kind] * size * (size + 8) ** 2), 2.0 ** 29 / (16 * size * size))
    if kind in ("ragged", "ragged_grad"):
        most = min(most, 30000)
    case["batch"] = _log_int(rng, 8, int(max(8, most)))
    return case


def _real_dtype(case):
    return torch.float32 if case["kind"] in ("cgeev", "sgeev") else torch.float64


def _matrices(case, n, batch, seed):
    """``[batch, n, n]`` complex128 (float64 for the real entry points) matrices on the GPU."""
    real = case["kind"] in ("dgeev", "sgeev")
    dist = case["dist"]
    if real or dist == "uniform":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        shape = (batch, n, n) if real else (batch, n, n, 2)
        if dist == "uniform":
            A = 2 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 1
        else:
            A = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
        return A if real else torch.view_as_complex(A)
    if case["kind"] in ("grad", "ragged_grad"):
        return wl.torch_vdv_separated(batch, n, seed=seed, min_sep=MIN_SEP)[0]
    return wl.TORCH_GENERATORS[dist](batch, n, seed=seed)


def _orders(case):
    """A case's orders: the layout of the packed buffers, as a program has it before the entries."""
    return wl.ragged_sizes(case["batch"], case["nmin"], case["nmax"], seed=case["batch"])


def _packed(case, seed):
    """Orders, element offsets and the packed matrices of a ragged case (grouped draws, then placed)."""
    orders = torch.from_numpy(_orders(case)).cuda()
    n64 = orders.to(torch.int64)
    offsets = torch.cumsum(n64 * n64, 0) - n64 * n64
    out = torch.empty(int((n64 * n64).sum()), dtype=torch.complex128, device="cuda")
    for n in range(case["nmin"], case["nmax"] + 1):
        at = offsets[orders == n]
        if at.numel():
            block = _matrices(case, n, at.numel(), seed + 7919 * n)
            out[(at[:, None] + torch.arange(n * n, device="cuda")).reshape(-1)] = block.reshape(-1)
    return orders, offsets, out


def prepare(case, seed):
    kind, batch = case["kind"], case["batch"]
    state = {"kind": kind, "handle": api.Handle()}
    if kind in ("ragged", "ragged_grad"):
        orders, offsets, A = _packed(case, seed)
        n64 = orders.to(torch.int64)
        state.update(A=A, orders=orders, offsets=offsets, total=int(n64.sum()),
                     segment=torch.repeat_interleave(torch.arange(batch, device="cuda"), n64))
        state["work"] = torch.empty(api.tokura_get_zgeev_ragged_workspacesize(batch, A.numel()), dtype=torch.uint8,
                                    device="cuda")
        if kind == "ragged_grad":
            state["work_bwd"] = torch.empty(api.tokura_get_zgeev_ragged_backward_workspacesize(batch, A.numel()),
                                            dtype=torch.uint8, device="cuda")
            state["A"] = A.requires_grad_(True)
        return state
    n = case["n"]
    if kind == "strided":  # blocks of larger matrices
        big = _matrices(case, n + 5, batch, seed)
        state["A"] = big[:, 2:n + 2, 3:n + 3]
    else:
        A = _matrices(case, n, batch, seed)
        if kind in ("cgeev", "sgeev"):
            A = A.to(torch.complex64 if kind == "cgeev" else torch.float32)
        state["A"] = A.requires_grad_(True) if kind == "grad" else A
    if kind in ("zgeev", "cgeev", "strided"):
        state["work"] = torch.empty(api.tokura_get_zgeeveigenvaluesgetworspacesize(n, batch), dtype=torch.uint8,
                                    device="cuda")
    elif kind in ("dgeev", "sgeev"):
        state["work"] = torch.empty(api.tokura_get_dgeev_workspacesize(n, batch), dtype=torch.uint8, device="cuda")
    return state


def _in_order(w):
    """The order of each row's eigenvalues."""
    return torch.argsort(w.real.double() + ORDER_IM * w.imag.double(), dim=-1)


def _loss(w):
    """A smooth loss of the eigenvalues whose gradient is exp(Re w) + 2 w."""
    return torch.sum(torch.exp(w.real) + w.real ** 2 + w.imag ** 2)


def _segments_in_order(w, segment):
    by_key = torch.argsort(w.real + ORDER_IM * w.imag)
    return w[by_key[torch.argsort(segment[by_key], stable=True)]]


def run(state):
    kind, A, h = state["kind"], state["A"], state["handle"]
    if kind in ("zgeev", "cgeev", "strided"):
        call = {"zgeev": api.zgeev_batched, "cgeev": api.cgeev_batched, "strided": api.zgeev_strided}[kind]
        w, flag = call(A, handle=h, work=state["work"])
        return {"w": torch.gather(w, -1, _in_order(w)), "flag": flag}
    if kind in ("dgeev", "sgeev"):
        wr, wi, flag = api.dgeev_batched(A, handle=h, work=state["work"])
        w = torch.complex(wr, wi)
        return {"w": torch.gather(w, -1, _in_order(w)), "flag": flag}
    if kind == "vectors":
        w, VL, VR, flag = api.zgeev_vectors(A, handle=h)
        order = _in_order(w)
        columns = order[:, None, :].expand(VR.shape)
        return {"w": torch.gather(w, -1, order), "VL": torch.gather(VL, -1, columns),
                "VR": torch.gather(VR, -1, columns), "flag": flag}
    if kind == "grad":
        w = ag.eigvals(A, handle=h)
        (grad,) = torch.autograd.grad(_loss(w), A)
        w = w.detach()
        return {"w": torch.gather(w, -1, _in_order(w)), "grad": grad}
    if kind == "ragged":
        w, flag = api.zgeev_ragged(A, state["orders"], offsets=state["offsets"], handle=h, work=state["work"],
                                   total_eigenvalues=state["total"])
        return {"w": _segments_in_order(w, state["segment"]), "flag": flag}
    w = ag.eigvals_ragged(A, state["orders"], state["offsets"], handle=h, work_fwd=state["work"],
                          work_bwd=state["work_bwd"], total_eigenvalues=state["total"])
    (grad,) = torch.autograd.grad(_loss(w), A)
    return {"w": _segments_in_order(w.detach(), state["segment"]), "A": A.detach() - LEARNING_RATE * grad}


def _sum_of(case, f):
    """Sum of f(n) over the matrices (ragged orders: U{nmin..nmax})."""
    if "n" in case:
        return case["batch"] * f(case["n"])
    sizes = range(case["nmin"], case["nmax"] + 1)
    return case["batch"] * sum(f(n) for n in sizes) / len(sizes)


def work(case):
    """Operations by the usual counts (a multiply-add is two): 40 n^3 for the eigenvalues of a
    complex matrix (Hessenberg reduction 40/3 n^3 and QR), 10 n^3 real; 54.7 n^3 for a gradient;
    100 n^3 in all with both sets of eigenvectors."""
    kind = case["kind"]
    flops = {"dgeev": 10.0, "sgeev": 10.0, "vectors": 100.0, "grad": 94.7, "ragged_grad": 94.7}.get(kind, 40.0)
    item = {"cgeev": 8, "dgeev": 8, "sgeev": 4}.get(kind, 16)
    pair = 2 * _real_dtype(case).itemsize  # an eigenvalue
    times = {"vectors": 3, "grad": 2, "ragged_grad": 2}.get(kind, 1)  # matrices in, vectors or gradients out
    return {"bytes": _sum_of(case, lambda n: times * item * n * n + pair * n + 1),
            "flops": flops * _sum_of(case, lambda n: n ** 3)}


def _cpu(A, f):
    """f over slices of the batch, on all cores."""
    parts = min(len(A), 4 * (os.cpu_count() or 1))
    cuts = [len(A) * k // parts for k in range(parts + 1)]
    with ThreadPoolExecutor() as pool:
        return list(pool.map(lambda k: f(A[cuts[k]:cuts[k + 1]]), range(parts)))


def _np_in_order(w, *arrays):
    at = np.argsort(w.real.astype(np.float64) + ORDER_IM * w.imag.astype(np.float64), axis=-1, kind="stable")
    return np.take_along_axis(w, at, -1), [np.take_along_axis(a, at[:, None, :], -1) for a in arrays]


def _np_eigvals(A, dtype=np.complex128):
    w = np.concatenate(_cpu(A, np.linalg.eigvals)).astype(dtype)
    return _np_in_order(w)[0]


def _normalised(V):
    """Columns of unit length with the largest component real."""
    V = V / np.linalg.norm(V, axis=-2, keepdims=True)
    top = np.take_along_axis(V, np.argmax(np.abs(V), axis=-2)[:, None, :], -2)
    return V * (np.conj(top) / np.abs(top))


def _np_gradient(A):
    """Eigenvalues and the gradient of the loss: V^-H diag(exp(Re w) + 2 w) V^H."""
    def part(a):
        w, V = np.linalg.eig(a)
        Vh = np.conj(np.swapaxes(V, -1, -2))
        return w, np.linalg.solve(Vh, (np.exp(w.real) + 2 * w)[:, :, None] * Vh)
    got = _cpu(A, part)
    w, g = np.concatenate([p[0] for p in got]), np.concatenate([p[1] for p in got])
    return _np_in_order(w)[0], g


# Sum of n^3 + 1500 n over a batch whose spectra the cores give in some seconds; eigenvectors and gradients take
# about four times as long for each matrix.
_EXACT_MOST = 2.5e10


def exact(case, seed):
    kind = case["kind"]
    heavy = kind in ("vectors", "grad", "ragged_grad")
    if _sum_of(case, lambda n: n ** 3 + 1500 * n) * (4 if heavy else 1) > _EXACT_MOST:
        return None
    if kind in ("ragged", "ragged_grad"):
        orders, offsets, A = _packed(case, seed)
        orders, offsets, A = orders.cpu().numpy(), offsets.cpu().numpy(), A.cpu().numpy()
        first = np.cumsum(orders, dtype=np.int64) - orders
        w, moved = np.empty(int(orders.sum()), np.complex128), np.empty_like(A)
        for n in np.unique(orders):
            at = np.nonzero(orders == n)[0]
            places = offsets[at][:, None] + np.arange(n * n)
            M = A[places].reshape(-1, n, n)
            if kind == "ragged":
                v = _np_eigvals(M)
            else:  # the packed matrices are column-major: M is the transpose, and so is its gradient
                v, g = _np_gradient(M)
                moved[places] = (M - LEARNING_RATE * g).reshape(len(at), -1)
            w[first[at][:, None] + np.arange(n)] = v
        return {"w": w, "flag": None} if kind == "ragged" else {"w": w, "A": moved}
    A = prepare(case, seed)["A"].detach()
    A = A.to(torch.complex128 if A.is_complex() else torch.float64).cpu().numpy()
    if kind == "vectors":
        def part(a):
            w, V = np.linalg.eig(a)
            return w, V, np.conj(np.swapaxes(np.linalg.inv(V), -1, -2))
        got = _cpu(A, part)
        w, VR, VL = (np.concatenate([p[k] for p in got]) for k in range(3))
        w, (VL, VR) = _np_in_order(w, _normalised(VL), _normalised(VR))
        return {"w": w, "VL": VL, "VR": VR, "flag": None}
    if kind == "grad":
        w, g = _np_gradient(A)
        return {"w": w, "grad": g}
    # Rounded to the output's type before ordering, as the entry point does.
    return {"w": _np_eigvals(A, np.complex64 if kind in ("cgeev", "sgeev") else np.complex128), "flag": None}
