"""Calls of different sizes from several host threads at once: a kernel's shared
memory limit is the process's, so no call may set it to its own need only."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _both(a, b):
    errors = []

    def run(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 -- reported by the assertion below
            errors.append(repr(e))

    threads = [threading.Thread(target=run, args=(f,)) for f in (a, b)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_unwrap_of_two_sizes_from_two_threads():
    import torch
    from als_speckle_b200._lib import call, ptr

    def calls(N, reps):
        m = torch.rand((N, N), device="cuda")
        work = torch.empty((N, N), dtype=torch.float64, device="cuda")
        mean = torch.empty(4, device="cuda")
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())

        def f():
            for _ in range(reps):
                call("sp_unwrap", ptr(m), N, 0, 4, float(N // 2), float(N // 2), 0, ptr(work), None,
                     ptr(mean), s.cuda_stream)
            s.synchronize()
        return f

    _both(calls(8192, 200), calls(512, 2000))


def test_registration_of_two_upsamplings_from_two_threads():
    """Both run one instantiation (7 column groups), at 222 and 194 points."""
    import torch
    from als_speckle_b200.phasing import align_frames_subpixel

    def calls(U):
        f = torch.randn((1, 16, 16), dtype=torch.complex64, device="cuda")

        def g():
            for _ in range(2000):
                align_frames_subpixel(f, upsample=U)
        return g

    _both(calls(148), calls(129))
