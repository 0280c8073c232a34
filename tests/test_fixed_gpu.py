"""Eigenvalues in 64-bit fixed point (the default path of the plain entry points).

Every launch shape of the dispatch does the same arithmetic on a matrix, so a batch must give
bitwise what its slices give in other shapes; parity with LAPACK at the edges of the order
classes; graded and triangular matrices are left to the FP64 kernels, bitwise.
"""
import numpy as np
import pytest

from oracle import lapack_oracle as lo
from tokura_zgeev_batched_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def solve(A, handle=None):
    import torch
    from tokura_zgeev_batched_gb300 import api

    w, f = api.zgeev_batched(A, handle=handle)
    torch.cuda.synchronize()
    return w.cpu().numpy(), f.cpu().numpy()


@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49, 63, 64])
def test_parity_at_class_edges(cuda, n):
    import torch

    for cls in ("gaussian", "vdv", "companion"):
        A = wl.GENERATORS[cls](65, n, seed=5000 + n)
        w, f = solve(torch.from_numpy(A).cuda())
        rep = lo.parity_report(A, w, f)
        assert rep["flag_mismatch"] == 0 and (f == 0).all(), (cls, rep)
        if rep["well_conditioned"]:
            assert rep["max_rel_err_well"] <= lo.TOL_REL_FRO, (cls, rep["max_rel_err_well"])


@pytest.mark.parametrize("n,batches", [(4, (9000, 40000, 60001)), (7, (4000, 12000, 30001)), (13, (2000, 9000, 12001)),
                                       (21, (1100, 4000, 6001)), (30, (1100, 4001)), (40, (700, 1500, 4001)),
                                       (48, (900, 4001)), (61, (800, 1001, 4001))])
def test_every_launch_shape_gives_the_same_bits(cuda, n, batches):
    A = wl.torch_gaussian(max(batches), n, seed=5100 + n)
    few = [solve(A[k:k + 5])[0] for k in (0, 3)]
    for batch in batches:
        w, f = solve(A[:batch])
        assert (f == 0).all()
        assert np.array_equal(w[:5].view(np.uint64), few[0].view(np.uint64)), batch
        assert np.array_equal(w[3:8].view(np.uint64), few[1].view(np.uint64)), batch
        tail = solve(A[batch - 6:batch])[0]
        assert np.array_equal(w[-6:].view(np.uint64), tail.view(np.uint64)), batch


@pytest.mark.parametrize("n", [3, 8, 20, 50])
def test_graded_and_triangular_matrices_are_left_to_fp64(cuda, n):
    import torch
    from tokura_zgeev_batched_gb300 import api

    A = wl.gaussian(12, n, seed=5200 + n)
    d = 2.0 ** np.linspace(0, -40, n)
    A[1] *= d[:, None] * d[None, :]  # graded rows and columns
    A[4] = np.triu(A[4])
    A[7] *= d[:, None]
    A[9] = np.diag(d)
    At = torch.from_numpy(A).cuda()
    w, f = solve(At)
    h = api.Handle()
    assert h.set_shift_hints(0) == 0  # the FP64 iteration without hints
    w64, f64 = solve(At, h)
    left = [1, 4, 7, 9]
    assert np.array_equal(w[left].view(np.uint64), w64[left].view(np.uint64))
    assert np.array_equal(f, f64)
    assert np.array_equal(np.sort(w[9].real), np.sort(d))


def test_extreme_scales_and_exact_rows(cuda):
    """The exponent of a matrix may be anything; eigenvalues scale with it exactly."""
    import torch

    A = wl.gaussian(8, 19, seed=5300)
    w, _ = solve(torch.from_numpy(A).cuda())
    for e in (-900, -300, 300, 900):
        ws, f = solve(torch.from_numpy(np.ldexp(A.view(np.float64), e).view(np.complex128)).cuda())
        assert (f == 0).all()
        assert np.array_equal(np.ldexp(ws.view(np.float64), -e), w.view(np.float64))


@pytest.mark.parametrize("batch,lo_n,hi_n", [(40, 1, 64), (700, 1, 64), (2500, 1, 33), (6000, 1, 17), (31000, 32, 34)])
def test_ragged_gives_the_bits_of_the_uniform_calls(cuda, batch, lo_n, hi_n):
    """Few and many matrices (both sets of launch shapes), every order, a graded one among them."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    ns = wl.ragged_sizes(batch, lo_n, hi_n, seed=5400 + batch)
    mats = [wl.gaussian(1, int(n), seed=5500 + k)[0] for k, n in enumerate(ns)]
    d = 2.0 ** np.linspace(0, -40, int(ns[5]))
    mats[5] = mats[5] * d[:, None]
    buf, n32, offs, eoffs = wl.pack_ragged(mats)
    w, f = api.zgeev_ragged(torch.from_numpy(buf).cuda(), torch.from_numpy(n32))
    w, f = w.cpu().numpy(), f.cpu().numpy()
    assert (f == 0).all()
    for n in np.unique(ns):
        at = [k for k in np.nonzero(ns == n)[0] if k != 5]
        if not at:
            continue
        wu, fu = solve(torch.from_numpy(np.stack([mats[k] for k in at])).cuda())
        got = np.stack([w[eoffs[k]:eoffs[k] + n] for k in at])
        assert np.array_equal(got.view(np.uint64), wu.view(np.uint64)), n
    n = int(ns[5])
    ref = lo.zgeev(mats[5][None])[0]
    err = lo.matched_abs_errors(w[eoffs[5]:eoffs[5] + n][None], ref).max()
    assert err <= lo.TOL_REL_FRO * np.linalg.norm(mats[5])


def ragged_backward(A, w, g, handle=None):
    """A, w, g: tensors [batch, n, n], [batch, n], [batch, n]; through the ragged entry point."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    batch, n = w.shape
    ns = torch.full((batch,), n, dtype=torch.int32, device="cuda")
    offs = torch.arange(batch, dtype=torch.int64, device="cuda") * (n * n)
    work = torch.empty(api.tokura_get_zgeev_ragged_backward_workspacesize(batch, A.numel()), dtype=torch.uint8,
                       device="cuda")
    A, w, g = A.contiguous(), w.contiguous(), g.contiguous()
    gA, flag = torch.empty_like(A), torch.empty(batch, dtype=torch.int8, device="cuda")
    h = handle if handle is not None else api.default_handle()
    st = api.tokura_zgeev_ragged_backward_gpu(h, batch, ns.data_ptr(), offs.data_ptr(), None, A.numel(), A.data_ptr(),
                                              w.data_ptr(), g.data_ptr(), gA.data_ptr(), work.data_ptr(),
                                              flag.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    return gA, flag


@pytest.mark.parametrize("n", [4, 5, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49, 64])
def test_ragged_gradients_from_fixed_point_schur_forms(cuda, n):
    """Against torch's gradient; matrices left to the FP64 kernel among the others."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    A_np = wl.vdv(37, n, seed=5600 + n, min_sep=0.05)
    A_np[3] = np.tril(A_np[3])  # triangular as stored
    A_np[3] += np.diag(np.arange(n))  # well separated
    Ac = torch.from_numpy(A_np).requires_grad_(True)
    lam = torch.linalg.eigvals(Ac)
    torch.sum(torch.exp(lam.real) + lam.real ** 2 + lam.imag ** 2).backward()
    ref = Ac.grad.numpy()
    A = torch.from_numpy(A_np).cuda()
    w, f = api.zgeev_batched(A)
    gbar = torch.exp(w.real) + 2 * w
    g, fg = ragged_backward(A, w, gbar)
    assert (fg == 0).all()
    # relative error as the FP64 kernels are tested: 1e-9 on separated spectra
    err = np.linalg.norm(g.cpu().numpy() - ref, axis=(1, 2)) / np.linalg.norm(ref, axis=(1, 2))
    assert err.max() < 1e-9, err.max()
    bad = A.clone()
    bad[5, 1, 2] = complex("nan")
    gb, fb = ragged_backward(bad, w, gbar)
    assert fb[5] == 2 and torch.isnan(gb[5].real).all()
    keep = [k for k in range(37) if k != 5]
    assert torch.equal(torch.view_as_real(gb[keep]), torch.view_as_real(g[keep])) and (fb[keep] == 0).all()
    lam_bad = w.clone()
    lam_bad[6, 0] = complex("inf")  # first shifts that fixed point does not hold
    gi, fi = ragged_backward(A, lam_bad, gbar)
    assert torch.equal(torch.view_as_real(gi[7:]), torch.view_as_real(g[7:]))


@pytest.mark.parametrize("n", [4, 5, 8, 9, 16, 17, 32, 33, 64])
def test_eigenvectors_from_fixed_point_schur_forms(cuda, n):
    import torch
    from tokura_zgeev_batched_gb300 import api

    for k in (0, 1):
        A = wl.vdv(37, n, seed=5700 + n) if k == 0 else wl.gaussian(37, n, seed=5700 + n)
        A[3] = np.tril(A[3]) + np.diag(np.arange(n))
        M = torch.from_numpy(A).cuda()
        w, VL, VR, f = api.zgeev_vectors(M)
        assert (f == 0).all()
        fro = torch.linalg.norm(M, dim=(1, 2))[:, None, None]
        assert float(((M @ VR - VR * w[:, None, :]).abs() / fro).max()) <= 1e-12 * n
        assert float(((VL.mH @ M - w[:, :, None] * VL.mH).abs() / fro).max()) <= 1e-12 * n
        assert torch.allclose(torch.linalg.norm(VR, dim=1), torch.ones_like(w.real), atol=1e-13)
        rep = lo.parity_report(A, w.cpu().numpy(), f.cpu().numpy())
        assert rep["max_rel_err_well"] <= lo.TOL_REL_FRO or not rep["well_conditioned"]
    bad = M.clone()
    bad[5, 1, 2] = complex("nan")
    wb, VLb, VRb, fb = api.zgeev_vectors(bad)
    keep = [k for k in range(37) if k != 5]
    assert fb[5] == 2 and torch.isnan(wb[5].real).all() and torch.isnan(VRb[5].real).all()
    assert torch.equal(torch.view_as_real(VRb[keep].contiguous()), torch.view_as_real(VR[keep].contiguous()))


def test_schur_sweep_cap(cuda):
    import torch
    from tokura_zgeev_batched_gb300 import api

    A = torch.from_numpy(wl.gaussian(20, 24, seed=5800)).cuda()
    h = api.Handle()
    assert h.set_sweep_cap(1) == 0
    w, VL, VR, f = api.zgeev_vectors(A, handle=h)
    assert (f == 1).all() and bool(torch.isfinite(torch.view_as_real(w)).all())
    w0, _ = api.zgeev_batched(A)
    g, fg = ragged_backward(A, torch.zeros_like(w0), w0, handle=h)  # useless first shifts
    assert (fg == 1).all() and torch.isnan(g.real).all()


def test_fp64_call_is_the_hinted_fp64_path(cuda):
    import torch
    from tokura_zgeev_batched_gb300 import api

    A = torch.from_numpy(wl.gaussian(50, 20, seed=5900)).cuda()
    w, f = api.zgeev_batched(A, fp64=True)
    h = api.Handle()
    assert h.set_shift_hints(1) == 0
    w1, f1 = api.zgeev_batched(A, handle=h)
    assert torch.equal(torch.view_as_real(w), torch.view_as_real(w1)) and (f == 0).all()


def solve_real(A, handle=None):
    import torch
    from tokura_zgeev_batched_gb300 import api

    wr, wi, f = api.dgeev_batched(A, handle=handle)
    torch.cuda.synchronize()
    return torch.complex(wr, wi).cpu().numpy(), f.cpu().numpy()


@pytest.mark.parametrize("n,batches", [(3, (9000, 60001)), (4, (12000, 40001)), (7, (4000, 30001)), (13, (2000, 9001)),
                                       (21, (1100, 4000, 6001)), (30, (1100, 4001)), (33, (1001,)), (40, (12001,)), (48, (1700, 8001)),
                                       (61, (1001, 5001)), (64, (6001,))])
def test_real_matrices_at_every_launch_shape(cuda, n, batches):
    """The same bits in every shape; parity and conjugate pairs are checked on a slice."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(5700 + n)
    A = torch.randn(max(batches), n, n, dtype=torch.float64, device="cuda", generator=gen)
    few, f = solve_real(A[3:40])
    rep = lo.real_parity_report(A[3:40].cpu().numpy(), few.real.copy(), few.imag.copy(), f)
    assert rep["flag_mismatch"] == 0 and rep["pairs_ok"]
    assert rep["max_rel_err_well"] <= lo.TOL_REL_FRO, rep["max_rel_err_well"]
    for batch in batches:
        w, f = solve_real(A[:batch])
        assert (f == 0).all()
        assert np.array_equal(w[3:40].view(np.uint64), few.view(np.uint64)), batch
        tail = solve_real(A[batch - 6:batch])[0]
        assert np.array_equal(w[-6:].view(np.uint64), tail.view(np.uint64)), batch


@pytest.mark.parametrize("n", [3, 8, 20, 50])
def test_real_matrices_left_to_fp64(cuda, n):
    """Graded, triangular, and spectra whose conjugates can't be told apart."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    A = np.random.default_rng(5800 + n).standard_normal((12, n, n))
    d = 2.0 ** np.linspace(0, -40, n)
    A[1] *= d[:, None] * d[None, :]
    A[4] = np.triu(A[4])
    A[7] = 1.0  # n - 1 zero eigenvalues
    A[9] = A[9] @ np.diag(np.r_[2.0, 2.0, np.arange(n - 2)]) @ np.linalg.inv(A[9])  # a double one
    A[10] = 0.0
    A[11, 1, 2] = np.inf
    At = torch.from_numpy(A).cuda()
    w, f = solve_real(At)
    h = api.Handle()
    assert h.set_real_config(n, 8 if n >= 16 else 4, 32) == 0  # what so small a batch uses
    w64, f64 = solve_real(At, h)
    left = [1, 4, 7, 9]
    assert np.array_equal(w[left].view(np.uint64), w64[left].view(np.uint64))
    assert np.array_equal(f, f64) and f[11] == 2
    assert (w[10] == 0).all() and np.isnan(w[11].real).all()


@pytest.mark.parametrize("n,batch", [(5, 8191), (5, 29183), (12, 30001)])
def test_host_chunks_solved_in_turn_give_the_device_call(cuda, n, batch):
    from tokura_zgeev_batched_gb300 import api

    A = wl.torch_gaussian(batch, n, seed=5900 + batch)
    w, f = api.zgeev_batched_host(A.cpu())
    wd, fd = solve(A)
    assert np.array_equal(np.ascontiguousarray(w).view(np.uint64), wd.view(np.uint64)) and np.array_equal(f, fd)
