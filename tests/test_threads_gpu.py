"""Calls of different orders from several host threads at once, each with a handle and a stream of its own."""
import threading

import numpy as np
import pytest

from tokura_zgeev_batched_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def test_orders_with_different_shared_memory(cuda):
    """The reduction takes more than the default shared memory from order 55 on, a different amount for each order.
    Triangular matrices: as launches they are like all others, and the kernels are done with them at once."""
    import torch
    from tokura_zgeev_batched_gb300 import api

    lib = api.lib()
    failed = []

    def loop(n, A, h, stream, w, flag, work):
        for k in range(3000):
            st = lib.tokura_zgeev_batched_gpu(h.value, n, 2, A.data_ptr(), w.data_ptr(), work.data_ptr(),
                                              flag.data_ptr(), stream.cuda_stream)
            if st != 0:
                failed.append((n, k, st))
                return
            if k % 100 == 0:
                stream.synchronize()
        stream.synchronize()

    threads, runs = [], []
    for n in (56, 64, 60, 62):
        M = np.swapaxes(np.triu(wl.gaussian(2, n, seed=6700 + n)), 1, 2)  # upper triangular where it is column-major
        A = torch.from_numpy(np.ascontiguousarray(M)).cuda()
        w, flag = torch.empty(2, n, dtype=torch.complex128, device="cuda"), torch.ones(2, dtype=torch.int8, device="cuda")
        work = torch.empty(api.tokura_get_zgeeveigenvaluesgetworspacesize(n, 2), dtype=torch.uint8, device="cuda")
        runs.append((n, A, api.Handle(), torch.cuda.Stream(), w, flag, work))
    torch.cuda.synchronize()
    for run in runs:
        threads.append(threading.Thread(target=loop, args=run, daemon=True))
        threads[-1].start()
    for t in threads:
        t.join(60)
    assert not failed, failed
    assert not any(t.is_alive() for t in threads)
    for n, A, _, _, w, flag, _ in runs:
        assert not flag.any() and torch.equal(w, torch.diagonal(A, dim1=1, dim2=2))
