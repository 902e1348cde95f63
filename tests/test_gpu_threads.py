"""Calls of different sizes from several host threads, each on its own stream: what a launch needs of a kernel's settings
(its dynamic shared memory's limit) holds for every size, whatever another thread has set in between."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


def _threads(jobs, reps):
    """Each job (a function that makes a call) reps times in its own thread and stream, all at once; their errors."""
    errors, ready = [], threading.Barrier(len(jobs))

    def body(make):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                call, checked = make()
                torch.cuda.current_stream().synchronize()
                ready.wait(60)
                for i in range(reps):
                    call()
                    if i % 16 == 15:                        # (no thread far ahead of the device)
                        torch.cuda.current_stream().synchronize()
                torch.cuda.current_stream().synchronize()
                checked()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(repr(e))
            ready.abort()
    ts = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    return errors


def _solver(n, nrhs, what):
    """A diagonal factor of n unknowns: its preparation, or a solve with it."""
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib

    def make():
        d = torch.linspace(1, 2, n, device='cuda')
        A = torch.zeros((n, n), dtype=torch.complex64, device='cuda')
        A.diagonal().copy_(d)
        piv = torch.arange(n, dtype=torch.int32, device='cuda')
        aux = torch.empty(int(lib().m25_getrs_aux_bytes(n, 1)), dtype=torch.uint8, device='cuda')
        B = torch.ones((n, nrhs), dtype=torch.complex64, device='cuda')
        X, s = B.clone(), _lib.stream_ptr()

        def prepare():
            check(lib().m25_getrs_prepare(P(A), ctypes.c_long(n), n, P(piv), 1, P(aux), ctypes.c_size_t(aux.numel()), s),
                  'm25_getrs_prepare')

        def solve():
            X.copy_(B)
            check(lib().m25_getrs_aux(P(A), ctypes.c_long(n), n, 1, P(aux), P(X), nrhs, s), 'm25_getrs_aux')

        def checked():
            solve()
            torch.cuda.current_stream().synchronize()
            assert float((X * d[:, None] - 1).abs().max()) <= 1e-6
        prepare()
        return (prepare if what == 'prepare' else solve), checked
    return make


def _spline(n):
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib

    def make():
        x = np.linspace(0, 1, n)
        y = np.stack([x ** 2 + 1j * x, 1 - x + 0j])
        d_x, d_y = _lib.dev(x), _lib.dev(y)
        out, s = torch.empty((2, 64), dtype=torch.complex128, device='cuda'), _lib.stream_ptr()

        def call():
            check(lib().m25_spline_uniform(P(d_x), P(d_y), 2, n, ctypes.c_double(1 / 63), 64, P(out), 0, ctypes.c_long(64),
                                           ctypes.c_long(0), 1, s), 'm25_spline_uniform')

        def checked():                                     # quadratics come back to rounding
            t = np.linspace(0, 1, 64)
            assert np.abs(out.cpu().numpy() - np.stack([t ** 2 + 1j * t, 1 - t + 0j])).max() <= 1e-11
        return call, checked
    return make


@pytest.mark.parametrize('what', ['prepare', 'solve', 'spline'])
def test_sizes_in_threads(what):
    """prepare: 72 and 52 KB of shared memory for the rows of 18,000 and 13,000 unknowns beside 600; solve (above 8
    right-hand sides): two blocks of 64 rows a CTA beside one; spline: 176 KB of 2,000 knots beside 53 of 600."""
    if what == 'spline':
        jobs, reps = [_spline(n) for n in (600, 2000, 700, 1500)], 1500
    else:
        jobs, reps = [_solver(n, 12, what) for n in (600, 18000, 650, 13000)], 300
    assert _threads(jobs, reps) == []
