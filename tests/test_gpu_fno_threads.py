"""he4_fno_contract from several host threads at once, with sizes that need
different amounts of shared memory of one kernel: no call fails and the results
are those of one thread (the same bits)."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_contract_sizes_in_threads(pkg):
    import torch
    L = pkg.load_library()
    f = L.he4_fno_contract
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p] + [C.c_int32] * 7 + [C.c_void_p]
    jobs = []
    gen = torch.Generator(device="cuda").manual_seed(3)
    # complex in and out, 16 modes: 80, 72 and 64 KB of one kernel
    for J, K in ((384, 16), (320, 16), (256, 16)):
        x = torch.randn(2, J, 32, 2, device="cuda", generator=gen)
        A = torch.randn(K, J, 2, device="cuda", generator=gen)
        a2, x2 = torch.view_as_complex(A.double()), torch.view_as_complex(x.double())
        want = torch.einsum("kj,bjr->bkr", a2, x2)
        # the bound of test_gpu_fno_kernels.py for 2 J real products
        tol = (4 * J + 4) * 2.0 ** -24 * 2 * torch.einsum("kj,bjr->bkr", a2.abs(), x2.abs())
        jobs.append((J, K, x, A, want, tol))
    torch.cuda.synchronize()
    fails, outs = [], [None] * len(jobs)

    def work(i):
        J, K, x, A = jobs[i][:4]
        s = torch.cuda.Stream()
        y = torch.empty(2, K, 32, 2, device="cuda")
        s.wait_stream(torch.cuda.default_stream())
        for _ in range(4000):
            rc = f(x.data_ptr(), y.data_ptr(), A.data_ptr(), 2, J, K, 32, 0, 0, 0, s.cuda_stream)
            if rc:
                fails.append((J, rc, L.he4_last_error()))
                break
        s.synchronize()
        outs[i] = y

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not fails, fails
    for (J, K, _, _, want, tol), y in zip(jobs, outs):
        assert bool(((torch.view_as_complex(y.double()) - want).abs() <= tol).all()), J
