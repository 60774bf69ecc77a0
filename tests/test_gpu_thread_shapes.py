"""Host threads with a handle each launch the same kernels in different shapes
at once: no call is refused for the shared memory of another thread's shape,
and the results are those of a call alone.  The threads call the C ABI on
buffers of their own, so that their launches follow each other closely."""
import ctypes as C
import threading

import numpy as np
import pytest

from hiten_gb300.workloads import MU_EM, section_states, stm_fixed_batch

pytestmark = pytest.mark.gpu

CALLS = 10000


def run_threads(*workers):
    """worker: (call(stream), check()) -- `call` is repeated on a stream of
    the thread's own."""
    import torch
    failures = []

    def body(make):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                call, check = make()
                stream.synchronize()
                ready.wait()
                for _ in range(CALLS):
                    call(C.c_void_p(stream.cuda_stream))
                stream.synchronize()
                check()
        except Exception as e:  # noqa: BLE001
            ready.abort()
            failures.append(f"{type(e).__name__}: {e}")

    ready = threading.Barrier(len(workers))
    threads = [threading.Thread(target=body, args=(w,)) for w in workers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]


def soa(y):
    import torch
    return torch.as_tensor(y, device="cuda").t().contiguous()


def ptr(t):
    return C.c_void_p(t.data_ptr())


def tuned(**keys):
    from hiten_gb300 import _lib
    H = _lib.handle(0)
    for k, v in keys.items():
        H.set_tuning(getattr(_lib, "HG_TUNE_" + k), v)
    return H


def test_fixed_pair_batches_of_two_sizes(gpu):
    """One block an SM (it takes over half of the SM's shared memory) beside
    several."""
    import torch
    t = np.linspace(0.0, 0.003, 3)

    def worker(n):
        y = stm_fixed_batch(n, seed=n)
        alone = gpu.propagate_fixed(y, t, MU_EM, order=4, out_every=2)[1].cpu()

        def make():
            H = tuned(BLOCK_THREADS=128, LANES_D42=12)
            y0, tv, out = soa(y), torch.as_tensor(t, device="cuda"), soa(np.zeros((n, 84)))

            def call(st):
                H.check(H.lib.hg_propagate_fixed(H.ptr, MU_EM, 4, 42, n, ptr(y0), n, ptr(tv), 3, 2, ptr(out), n, 1,
                                                 0, 42, None, st))
            return call, lambda: np.testing.assert_array_equal(out[42:].t().cpu(), alone)
        return make

    run_threads(worker(60), worker(2000))


def test_dop853_spread_beside_plain_blocks(gpu):
    import torch
    from hiten_gb300 import _lib
    opts = _lib.hg_dop853_opts(1e-12, 1e-12, 1e4, 1e-15, 100000, 1, 0, 6)

    def worker(n, **tune):
        y = section_states(n, seed=n)
        alone = gpu.propagate_dop853(y, 0.0, 0.01, MU_EM, scheduled=False).y_end.cpu()

        def make():
            H = tuned(DOP853_LANES_D6=2, **tune)
            y0, end = soa(y), soa(np.zeros((n, 6)))
            t_end, ints = torch.zeros(n, dtype=torch.float64, device="cuda"), soa(np.zeros((n, 3), dtype=np.int32))

            def call(st):
                H.check(H.lib.hg_propagate_dop853(H.ptr, MU_EM, 6, n, ptr(y0), n, None, None, 0.0, 0.01,
                                                  C.byref(opts), None, 0, 0, None, ptr(end), ptr(t_end), None, None,
                                                  None, ptr(ints[0]), ptr(ints[1]), ptr(ints[2]), st))
            return call, lambda: np.testing.assert_array_equal(end.t().cpu(), alone)
        return make

    run_threads(worker(200, BLOCK_THREADS=128, SPREAD=1), worker(300, BLOCK_THREADS=128),
                worker(100, BLOCK_THREADS=64))
