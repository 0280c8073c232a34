"""Matrices that fixed point leaves to the FP64 kernels because of their entries' sizes: every entry point
gives the FP64 kernels' results for them, whatever else is in the batch."""
import numpy as np
import pytest

from oracle import lapack_oracle as lo
from tokura_zgeev_batched_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def bits(t):
    import torch

    a = t.detach()
    a = torch.view_as_real(a) if a.is_complex() else a
    return a.cpu().numpy().view(np.uint64)


def fp64_handle():
    from tokura_zgeev_batched_gb300 import api

    h = api.Handle()
    assert h.set_shift_hints(0) == 0  # the FP64 iteration without hints
    return h


def block_diagonal(seed, n, scale):
    """diag(B, scale B'), with its blocks' spectra by LAPACK."""
    A = np.zeros((n, n), dtype=np.complex128)
    k = n // 2
    A[:k, :k] = wl.gaussian(1, k, seed=seed)[0]
    small = wl.gaussian(1, n - k, seed=seed + 1)[0]
    A[k:, k:] = np.ldexp(small.view(np.float64), scale).view(np.complex128)
    return A, [(A[:k, :k], 0), (small, scale)]


def below_the_unit(n, seed, real=False):
    """Graded ones at places 1, 4 and 6: a block, and one diagonal entry, below 2^-61 of the norm."""
    A = wl.gaussian(9, n, seed=seed)
    A[1], blocks = block_diagonal(seed + 10, n, -70)
    A[4] = block_diagonal(seed + 20, n, -200)[0]
    A[6, n - 1] = 0
    A[6, :, n - 1] = 0
    A[6, n - 1, n - 1] = 2.0 ** -90 * 3
    return (np.ascontiguousarray(A.real) if real else A), blocks


LEFT = [1, 4, 6]


@pytest.mark.parametrize("n", [4, 7, 16, 20, 33, 64])
def test_what_is_below_the_unit_is_not_lost(cuda, n):
    import torch
    from tokura_zgeev_batched_gb300 import api

    A, blocks = below_the_unit(n, 6100 + n)
    M = torch.from_numpy(A).cuda()
    w, f = api.zgeev_batched(M)
    w64, f64 = api.zgeev_batched(M, handle=fp64_handle())
    assert np.array_equal(bits(w[LEFT]), bits(w64[LEFT])) and torch.equal(f[LEFT], f64[LEFT])
    assert f[1] == 0 and f[6] == 0
    assert float((w[6] - 3 * 2.0 ** -90).abs().min()) <= 3 * 2.0 ** -90 * 1e-14
    # the small block's eigenvalues to the parity bound of its own norm
    got = w[1].cpu().numpy()
    got = got[np.argsort(np.abs(got))]
    small, scale = blocks[1]
    k = len(small)
    ref = lo.zgeev(small[None])[0]
    err = lo.matched_abs_errors(np.ldexp(got[:k].copy().view(np.float64), -scale).view(np.complex128)[None], ref)
    assert err.max() <= lo.TOL_REL_FRO * np.linalg.norm(small)


@pytest.mark.parametrize("n", [4, 7, 16, 20, 33, 64])
def test_what_is_below_the_unit_is_not_lost_in_real_matrices(cuda, n):
    import torch
    from tokura_zgeev_batched_gb300 import api

    A, _ = below_the_unit(n, 6200 + n, real=True)
    M = torch.from_numpy(A).cuda()
    h = api.Handle()
    assert h.set_real_config(n, 8 if n >= 16 else 4, 32) == 0  # what so small a batch uses
    for got, ref in zip(api.dgeev_batched(M), api.dgeev_batched(M, handle=h)):
        assert torch.equal(got[LEFT], ref[LEFT])


def packed(A):
    import torch

    ns = torch.full((len(A),), A.shape[1], dtype=torch.int32)
    return torch.from_numpy(A).cuda().reshape(-1), ns


@pytest.mark.parametrize("n", [4, 7, 16, 20, 33])
def test_what_is_below_the_unit_is_not_lost_in_ragged_calls(cuda, n):
    """Orders below those that the FP64 path has shift hints for."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    A, _ = below_the_unit(n, 6300 + n)
    buf, ns = packed(A)
    w, f = api.zgeev_ragged(buf, ns)
    w64, f64 = api.zgeev_ragged(buf, ns, handle=fp64_handle())
    assert torch.equal(f, f64)
    assert np.array_equal(bits(w.reshape(-1, n)[LEFT]), bits(w64.reshape(-1, n)[LEFT]))


@pytest.mark.parametrize("n", [5, 7, 16, 20, 33, 64])
def test_what_is_below_the_unit_is_not_lost_in_schur_forms(cuda, n):
    import torch
    from tokura_zgeev_batched_gb300 import api

    A, blocks = below_the_unit(n, 6400 + n)
    M = torch.from_numpy(A).cuda()
    w, VL, VR, f = api.zgeev_vectors(M)
    assert f[1] == 0
    got = w[1].cpu().numpy()
    got = got[np.argsort(np.abs(got))]
    small, scale = blocks[1]
    ref = lo.zgeev(small[None])[0]
    k = len(small)
    err = lo.matched_abs_errors(np.ldexp(got[:k].copy().view(np.float64), -scale).view(np.complex128)[None], ref)
    assert err.max() <= lo.TOL_REL_FRO * np.linalg.norm(small)
    # gradients: the FP64 kernel's, from the same eigenvalues
    lam, _ = api.zgeev_batched(M, handle=fp64_handle())
    gbar = (torch.exp(lam.real) + 2 * lam).contiguous()
    out = []
    for h in (api.default_handle(), fp64_handle()):
        ns = torch.full((len(A),), n, dtype=torch.int32, device="cuda")
        offs = torch.arange(len(A), dtype=torch.int64, device="cuda") * (n * n)
        work = torch.empty(api.tokura_get_zgeev_ragged_backward_workspacesize(len(A), M.numel()), dtype=torch.uint8,
                           device="cuda")
        g, flag = torch.empty_like(M), torch.empty(len(A), dtype=torch.int8, device="cuda")
        assert api.tokura_zgeev_ragged_backward_gpu(h, len(A), ns.data_ptr(), offs.data_ptr(), None, M.numel(),
                                                    M.data_ptr(), lam.data_ptr(), gbar.data_ptr(), g.data_ptr(),
                                                    work.data_ptr(), flag.data_ptr(),
                                                    torch.cuda.current_stream().cuda_stream) == 0
        out.append((bits(g[LEFT]), flag[LEFT].cpu()))
    assert np.array_equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def graded_a_little(n, seed, real=False):
    """Matrices whose small eigenvalues FP64 holds to their relative precision and an absolute unit does not."""
    A = wl.gaussian(12, n, seed=seed)
    k = n // 2
    down = 2.0 ** np.linspace(0, -9, n)
    for j, s in ((1, 7), (2, 11)):  # two blocks
        A[j, :k, k:] = 0
        A[j, k:, :k] = 0
        A[j, k:, k:] = np.ldexp(A[j, k:, k:].copy().view(np.float64), -s).view(np.complex128)
    A[4] *= down[:, None] * down  # rows and columns
    A[5, n - 1] *= 2.0 ** -8  # one row and column
    A[5, :, n - 1] *= 2.0 ** -8
    A[7] *= 2.0 ** np.linspace(0, -12, n)  # rows (of the column-major matrix)
    return np.ascontiguousarray(A.real) if real else A


GRADED = [1, 2, 4, 5, 7]


@pytest.mark.parametrize("n", [2, 4, 9, 20, 50])
def test_slightly_graded_matrices_are_left_to_fp64(cuda, n):
    import torch
    from tokura_zgeev_batched_gb300 import api

    M = torch.from_numpy(graded_a_little(n, 6500 + n)).cuda()
    w, f = api.zgeev_batched(M)
    w64, f64 = api.zgeev_batched(M, handle=fp64_handle())
    assert np.array_equal(bits(w[GRADED]), bits(w64[GRADED])) and torch.equal(f, f64)
    if n > 2:
        R = torch.from_numpy(graded_a_little(n, 6500 + n, real=True)).cuda()
        h = api.Handle()
        assert h.set_real_config(n, 8 if n >= 16 else 4, 32) == 0
        for got, ref in zip(api.dgeev_batched(R), api.dgeev_batched(R, handle=h)):
            assert torch.equal(got[GRADED], ref[GRADED])


def badly_balanced(n, seed, real=False):
    """Tridiagonal ones 2^k, 1, 2^-k (places 0 and 1, spectra known) and D^-1 B D."""
    A = np.empty((5, n, n), dtype=np.complex128)
    for j, k in ((0, 4), (1, 8)):
        A[j] = np.diag(np.full(n - 1, 2.0 ** k), 1) + np.diag(np.full(n - 1, 2.0 ** -k), -1) + np.eye(n)
    d = 2.0 ** np.linspace(0, 11, n)
    A[2:] = wl.gaussian(3, n, seed=seed) * d / d[:, None]
    A[3] = np.swapaxes(A[3], 0, 1)
    if real:
        A = A.real + A.imag
    return np.ascontiguousarray(A)


@pytest.mark.parametrize("n", [4, 6, 16, 33, 64])
def test_badly_balanced_matrices_are_left_to_fp64(cuda, n):
    import torch
    from tokura_zgeev_batched_gb300 import api

    A = badly_balanced(n, 6600 + n)
    M = torch.from_numpy(A).cuda()
    w, f = api.zgeev_batched(M)
    w64, f64 = api.zgeev_batched(M, handle=fp64_handle())
    assert np.array_equal(bits(w), bits(w64)) and torch.equal(f, f64)
    if n <= 6:  # (above, FP64 without balancing does not hold them either)
        exact = 1 + 2 * np.cos(np.arange(1, n + 1) * np.pi / (n + 1))
        err = lo.matched_abs_errors(w[:2].cpu().numpy(), np.stack([exact, exact]).astype(np.complex128))
        assert err.max() <= lo.TOL_REL_FRO * np.linalg.norm(A[0])
    R = torch.from_numpy(badly_balanced(n, 6600 + n, real=True)).cuda()
    h = api.Handle()
    assert h.set_real_config(n, 8 if n >= 16 else 4, 32) == 0
    for got, ref in zip(api.dgeev_batched(R), api.dgeev_batched(R, handle=h)):
        assert torch.equal(got, ref)


@pytest.mark.parametrize("n", [33, 47, 64])
def test_real_matrices_with_repeated_eigenvalues(cuda, n):
    """Given up as soon as two eigenvalues have one place: the FP64 kernel's results, the others as without them."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    rng = np.random.default_rng(6800 + n)
    A = rng.standard_normal((40, n, n))
    Q = np.linalg.qr(A)[0]
    A[3] = Q[3][:, : n // 2] @ Q[3][:, : n // 2].T  # a projection
    A[8] = np.eye(n)[rng.permutation(n)]
    A[9] = np.kron(np.eye(n // 2 + 1), [[0.5, 2.0], [-1.0, 0.25]])[:n, :n]  # one pair many times
    A[11] = 0.0
    A[11, np.arange(1, n), np.arange(n - 1)] = 1.0  # a cycle: no two alike
    A[11, 0, n - 1] = 1.0
    M = torch.from_numpy(A).cuda()
    h = api.Handle()
    assert h.set_real_config(n, 8, 32) == 0  # what so small a batch uses
    got, ref = api.dgeev_batched(M), api.dgeev_batched(M, handle=h)
    for g, r in zip(got, ref):
        assert torch.equal(g[[3, 8, 9]], r[[3, 8, 9]])
    others = [k for k in range(40) if k not in (3, 8, 9)]
    for g, r in zip(got, api.dgeev_batched(M[others].contiguous())):
        assert torch.equal(g[others], r)
    wr, wi, f = got
    assert not f.any()
    err = lo.matched_abs_errors(torch.complex(wr, wi)[11:12].cpu().numpy(), np.exp(2j * np.pi * np.arange(n) / n)[None])
    assert err.max() <= lo.TOL_REL_FRO * np.sqrt(n)


@pytest.mark.parametrize("n,batch", [(5, 40001), (9, 40001), (16, 20001), (20, 9801), (33, 9801), (64, 9801)])
def test_few_left_matrices_in_a_large_batch(cuda, n, batch):
    """Alone or one in eight of a warp's tile: the bits of a small FP64 batch; more of them: parity, as the batch's."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    M = wl.torch_gaussian(batch, n, seed=6900 + n)
    d = torch.from_numpy(2.0 ** np.linspace(0, -30, n)).cuda()
    few, many = [3, 9000, batch - 1], list(range(640, 672))
    plain = api.zgeev_batched(M)[0]
    for j in few + many:
        M[j] *= d[:, None] * d
    w, f = api.zgeev_batched(M)
    assert not f.any()
    alone = api.zgeev_batched(M[few].contiguous(), handle=fp64_handle())[0]
    assert np.array_equal(bits(w[few]), bits(alone))
    others = torch.ones(batch, dtype=torch.bool, device="cuda")
    others[few + many] = False
    assert torch.equal(torch.view_as_real(w[others]), torch.view_as_real(plain[others]))
    err = lo.matched_abs_errors(w[many].cpu().numpy(), lo.zgeev(M[many].cpu().numpy())[0])
    assert (err.max(1) <= lo.TOL_REL_FRO * torch.linalg.norm(M[many], dim=(1, 2)).cpu().numpy()).all()
