"""Runs the bounds-checked library (TOKURA_ZGEEV_DEBUG_BOUNDS=1) over every launch shape of the fixed-point kernels, and
the FP64 kernels of the entry points that start in fixed point. Prints one JSON object: violations, and the accesses that
the fixed-point kernels' checked pointers made, for each case. Started as a subprocess by
tests/test_debug_bounds_fixed_gpu.py."""
import ctypes
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def main():
    assert os.environ.get("TOKURA_ZGEEV_DEBUG_BOUNDS") == "1"
    import torch

    from tokura_zgeev_batched_gb300 import api, autograd, build
    from tokura_zgeev_batched_gb300 import workloads as wl

    lib = api.lib()
    assert lib._name == build.DEBUG_LIB_PATH, lib._name
    rec = torch.zeros(6, dtype=torch.int64, device="cuda")
    assert lib.tokuraDebugAttach(rec.data_ptr()) == 0
    out = {}

    def checks():
        n = ctypes.c_ulonglong()
        assert lib.tokuraDebugChecks(ctypes.byref(n)) == 0
        return n.value

    def check(name, fn):
        rec[0] = 0
        torch.cuda.synchronize()
        before = checks()
        fn()
        torch.cuda.synchronize()
        r = rec.cpu().tolist()
        out[name] = {"violations": int(r[0]), "first": r[1:4], "checks": checks() - before}

    def handle(hints=False, real=0):
        """hints: the FP64 kernels; real: those of real matrices of that order."""
        h = api.Handle()
        assert not hints or h.set_shift_hints(1) == 0
        assert real == 0 or h.set_real_config(real, 4, 32) == 0
        return h

    def orders(batch, lo, hi, hints=False):
        ns = wl.ragged_sizes(batch, lo, hi, seed=batch)
        n64 = torch.from_numpy(ns).to(torch.int64)
        g = torch.Generator(device="cuda").manual_seed(batch)
        A = torch.view_as_complex(torch.randn(int((n64 * n64).sum()), 2, dtype=torch.float64, device="cuda", generator=g))
        return A, torch.from_numpy(ns).cuda(), handle(hints)

    def ragged(batch, lo, hi, hints=False):
        A, ns, h = orders(batch, lo, hi, hints)
        api.zgeev_ragged(A, ns, handle=h)

    def ragged_gradient(batch, lo, hi, hints=False):
        A, ns, h = orders(batch, lo, hi, hints)
        n64 = ns.to(torch.int64)
        w = autograd.eigvals_ragged(A.requires_grad_(True), ns, torch.cumsum(n64 * n64, 0) - n64 * n64, handle=h)
        torch.autograd.grad(torch.sum(w.real ** 2 + w.imag), A)

    # Every width of the launch rule: few, some, many matrices (zgeev_fixed_launch.cuh).
    for n, batches in ((2, (97, 12000, 60001)), (4, (97, 12000, 60001)), (5, (97, 8000)), (8, (97, 8000, 20001)),
                       (13, (97,)), (16, (97, 4000, 10001)), (20, (97,)), (24, (97, 5001)), (30, (97,)), (32, (97, 2001)),
                       (40, (97, 1500, 4001)), (48, (97,)), (49, (97,)), (64, (97, 1001))):
        for batch in batches:
            A = wl.torch_gaussian(batch, n, seed=n)
            check(f"plain n={n} b={batch}", lambda: api.zgeev_batched(A, handle=handle()))
    for n, batches in ((3, (97, 12000, 60001)), (8, (97, 8000)), (16, (97, 10001)), (31, (97, 2001)), (33, (97,)),
                       (42, (8001,)), (64, (97, 5001))):
        for batch in batches:
            A = torch.randn(batch, n, n, dtype=torch.float64, device="cuda")
            check(f"real n={n} b={batch}", lambda: api.dgeev_batched(A, handle=handle()))
    for n in (5, 8, 9, 16, 17, 32, 33, 64):
        A = wl.torch_gaussian(65, n, seed=n)
        check(f"vectors n={n}", lambda: api.zgeev_vectors(A, handle=handle()))
        check(f"vectors FP64 n={n}", lambda: api.zgeev_vectors(A, handle=handle(True)))
    for batch, lo, hi in ((300, 1, 64), (4000, 1, 20), (31000, 33, 35)):
        check(f"ragged {lo}-{hi} b={batch}", lambda: ragged(batch, lo, hi))
    check("ragged gradient", lambda: ragged_gradient(300, 2, 64))
    # The FP64 kernels behind the same entry points.
    check("ragged FP64", lambda: ragged(300, 1, 64, hints=True))
    check("ragged gradient FP64", lambda: ragged_gradient(300, 2, 64, hints=True))
    for n in (3, 16, 45):
        A = torch.randn(96, n, n, dtype=torch.float64, device="cuda")
        check(f"real FP64 n={n}", lambda: api.dgeev_batched(A, handle=handle(real=n)))
    big = wl.torch_gaussian(40, 48, seed=8)
    for hints, name in ((False, ""), (True, " FP64")):
        check("strided" + name, lambda: api.zgeev_strided(big[:, 5:37, 3:35], handle=handle(hints)))
        check("pointers" + name, lambda: api.zgeev_pointers([big[k] for k in range(40)], handle=handle(hints)))
        check("complex64" + name, lambda: api.cgeev_batched(big.to(torch.complex64), handle=handle(hints)))
        h = handle(hints)
        w, f = torch.empty(40, 48, dtype=torch.complex128, device="cuda"), torch.empty(40, dtype=torch.int8, device="cuda")
        check("noalloc" + name, lambda: lib.tokura_zgeev_batched_gpu_noalloc(
            h.value, 48, 40, big.data_ptr(), w.data_ptr(), f.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert lib.tokuraDebugAttach(None) == 0
    print(json.dumps(out))


if __name__ == "__main__":
    main()
