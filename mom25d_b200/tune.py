"""
mom25d_b200.tune - the autotuner of the LU's tile parameters, and timings of the hot path's kernels on this GPU.

    python -m mom25d_b200.tune --autotune [--sizes 1000 2000 ... 40000] [--write]
    python -m mom25d_b200.tune --lu 8192 [--single] [--tf32] [--reps 3]     # the LU alone, CUDA events
    python -m mom25d_b200.tune --update 4096 4096 256                        # the tensor-core trailing update
    python -m mom25d_b200.tune --solve 18788 [--single]                      # the triangular solves, 8 columns
    python -m mom25d_b200.tune --dense 18788 8                               # the dense double product

Times are CUDA-event measurements on the launching stream after a warm-up, the matrix a random complex one with a
dominant diagonal (pivots away from it as well).

The autotuner fills the LU's table from the smallest size up. A factorisation takes, for each outer block, the width of
the entry nearest (in log n) to the size that is left, so the entry of a size decides the blocks down to the line with
the entry below (their geometric mean), and what is left below that line is factored as the entries found before say:
each candidate is timed as the whole table it would make, the candidates of a size in turn, several times over. The sizes
are therefore where the widths may change: with the default ones (SIZES) at 1,414, 2,828, 5,099 and 8,062 rows left
and above in complex64, at 1,414, 2,828, 5,477, 8,660 and above in complex128.

Searched is the outer width; the CTAs of the cooperative panel kernel (16 to 64) only with M25_PANEL_CLUSTER=0 (the panels
that have more rows than a thread-block cluster takes need more CTAs than that for their shared memory). Widths: 64 to
256 for the complex128 LU (the drop-in); of times within TIE the widest. For the complex64 LU with tensor-core updates (the mixed path's factorisation) 256, or 64,
where every update is in FP32: the widths between leave more of the factor's updates to 3xTF32 instead of FP32 and cost
the factor its use as a preconditioner at the low-frequency end (measured on the routed board: with 128, the fresh
factor at 0.67 GHz no longer converged). With at most FP32_ROWS rows left the next block's columns too are updated in
FP32, which makes up for it (n = 4,977: residual of the factor 0.9e-4 with 128 against 1.7e-4 with 256 and the next
block's columns in 3xTF32): 128 is searched for the entries whose lines lie below that. The widths then differ little (64,
128, 256: 2.20, 2.20, 2.19 ms at 1,000; 4.47, 4.46, 4.55 at 2,000; 10.38, 9.41, 9.49 at 4,000; 1% either way on another
GPU), and of times within TIE the narrowest is taken, which leaves more of the factor to FP32. (128 up to 6,847 rows left
was measured too: 17.30 against 17.25 ms at 6,250, 33.5 against 33.0 at 9,601.)

The winners go into TUNING_FILE ({"device", "sms", "complex64": [{"n", "nb2", "blocks", "ms"}], "complex128": [...]}; ms:
the LU of that size with the table), which the library reads at load (_lib.apply_tuning -> m25_set_lu_tuning). The
tensor-core kernel's stage count is a compile-time choice (two stages, two CTAs an SM) and is not searched.
"""
import os
import argparse
import ctypes
import json
import time

import numpy as np
import torch

from . import _lib
from ._lib import P, check, lib


def random_matrix(n, dtype, seed=0):
    g = torch.Generator(device='cuda').manual_seed(seed)
    rdt = torch.float32 if dtype == torch.complex64 else torch.float64
    Z = torch.complex(torch.randn(n, n, generator=g, device='cuda', dtype=rdt),
                      torch.randn(n, n, generator=g, device='cuda', dtype=rdt))
    Z.diagonal().add_(4 * n ** 0.5)
    return Z


TUNING_FILE = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'tuning_b200.json')
SIZES = {True: [1000, 2000, 4000, 6500, 10000, 20000, 40000], False: [1000, 2000, 4000, 7500, 10000, 20000]}
FP32_ROWS = 8000               # lu.cu WIN_ROWS: rows left at which the next block's columns go to FP32 (complex64)
TIE = {True: 0.015, False: 0.005}      # times within this of the shortest count as equal


def candidates(n, above, single):
    """The (width, panel CTAs) tried at size n when the next larger entry is at `above` (None: there is none), of equal
    ones the preferred first."""
    if single:
        line = (n * above) ** 0.5 if above else float('inf')
        widths = (64, 128, 256) if line <= FP32_ROWS else (64, 256)
    else:
        widths = (256, 192, 128, 64)
    blocks = (32 if single or n < 4000 else 16,)
    if os.environ.get('M25_PANEL_CLUSTER') == '0':
        blocks = (16, 24, 32, 48, 64) if n <= 20000 else (32, 48)
    return [(w, b) for w in widths for b in blocks if w > 64 or n <= 20000]    # (above, 64 is seconds a try)


def set_table(entries, single=True):
    """The LU's tuning table in the library: [(n, nb2, blocks)] for complex64 (single) or complex128."""
    arr = lambda i: (ctypes.c_int * max(1, len(entries)))(*[e[i] for e in entries])
    check(lib().m25_set_lu_tuning(int(single), arr(0), arr(1), arr(2), len(entries)), 'm25_set_lu_tuning')


def autotune(sizes, single=True, reps=2, log=print):
    """The table of the complex64 (tensor-core) or complex128 LU, left set in the library: [{n, nb2, blocks, ms, grid:
    {"nb2/blocks": ms}}] by rising n."""
    out, sizes = [], sorted(sizes)
    entry = lambda e: (e['n'], e['nb2'], e['blocks'])
    for i, n in enumerate(sizes):
        above = sizes[i + 1] if i + 1 < len(sizes) else None
        times = {c: [] for c in candidates(n, above, single)}
        for _ in range(reps if n > 10000 else 3 * reps):
            for b2, bl in times:
                set_table([entry(e) for e in out] + [(int(n), b2, bl)], single)
                times[b2, bl].append(time_lu(n, single=single, tf32=single, reps=1 if n > 10000 else 5)['ms'])
        times = {c: float(np.median(t)) for c, t in times.items()}
        b2, bl = next(c for c in times if times[c] <= (1 + TIE[single]) * min(times.values()))
        out.append(dict(n=int(n), nb2=b2, blocks=bl, ms=round(times[b2, bl], 2),
                        grid={f'{w}/{b}': round(v, 2) for (w, b), v in times.items()}))
        if log:
            log(f"{'complex64' if single else 'complex128'} n={n}: nb2 {b2}, panel blocks {bl}: {times[b2, bl]:.2f} ms "
                f"of {out[-1]['grid']}")
    set_table([entry(e) for e in out], single)
    return out


def write_tuning(c64, c128, path=TUNING_FILE):
    import torch
    props = torch.cuda.get_device_properties(0)
    keep = lambda es: [{k: e[k] for k in ('n', 'nb2', 'blocks', 'ms')} for e in es]
    doc = dict(device=props.name, sms=props.multi_processor_count, complex64=keep(c64), complex128=keep(c128))
    with open(path, 'w') as fh:
        json.dump(doc, fh, indent=1)
    return path


def time_lu(n, single=False, tf32=False, reps=3):
    dtype = torch.complex64 if single else torch.complex128
    Z0 = random_matrix(n, dtype)
    Z = torch.empty_like(Z0)
    ipiv = torch.empty(n, dtype=torch.int32, device='cuda')
    nb = int(lib().m25_getrf_workspace(n, int(single)))
    work = torch.empty(nb, dtype=torch.uint8, device='cuda')
    out = []
    for r in range(reps + 1):
        Z.copy_(Z0)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s = torch.cuda.current_stream()
        a.record(s)
        check(lib().m25_getrf(P(Z), ctypes.c_long(n), n, P(ipiv), int(single), int(tf32), P(work), ctypes.c_size_t(nb),
                              _lib.stream_ptr()), 'm25_getrf')
        b.record(s)
        _lib.sync_check()
        if r:
            out.append(a.elapsed_time(b))
    ms = float(np.median(out))
    flops = 8.0 / 3.0 * n ** 3
    return dict(n=n, single=single, tf32=tf32, ms=ms, tflops=flops / ms / 1e9)


def time_update(M, N, K, reps=5):
    """The complex64 trailing update C -= L U alone: tensor cores (3xTF32) and, for comparison, the LU's SIMT
    kernel through a factorisation-free call are both timed with CUDA events. 8 M N K flops."""
    ld = max(M, K)
    C = random_matrix(max(ld, N), torch.complex64)[:N, :].contiguous()          # N columns of ld
    L = random_matrix(max(ld, K), torch.complex64, seed=1)[:K, :].contiguous()
    U = random_matrix(max(ld, N), torch.complex64, seed=2)[:N, :].contiguous()
    nb = int((2 * 2 * M * 512 + 2 * N * 512) * 4 + 4096)
    work = torch.empty(nb, dtype=torch.uint8, device='cuda')
    s = torch.cuda.current_stream()
    out = []
    for r in range(reps + 1):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        check(lib().m25_cgemm_update_tf32(P(C), ctypes.c_long(C.shape[1]), M, N, K, P(L), P(U), P(work),
                                          ctypes.c_size_t(nb), _lib.stream_ptr()), 'm25_cgemm_update_tf32')
        b.record(s)
        _lib.sync_check()
        if r:
            out.append(a.elapsed_time(b))
    ms = float(np.median(out))
    return dict(M=M, N=N, K=K, ms=ms, tflops_complex=8.0 * M * N * K / ms / 1e9,
                tflops_tf32_issued=3 * 8.0 * M * N * K / ms / 1e9)


def time_solve(n, nrhs=8, single=True, reps=5):
    """The triangular solves with a factor (m25_getrs_aux, diagonal-block inverses prepared once)."""
    dtype = torch.complex64 if single else torch.complex128
    Z = random_matrix(n, dtype)
    ipiv = torch.empty(n, dtype=torch.int32, device='cuda')
    nb = int(lib().m25_getrf_workspace(n, int(single)))
    work = torch.empty(nb, dtype=torch.uint8, device='cuda')
    check(lib().m25_getrf(P(Z), ctypes.c_long(n), n, P(ipiv), int(single), int(single), P(work), ctypes.c_size_t(nb),
                          _lib.stream_ptr()), 'm25_getrf')
    na = int(lib().m25_getrs_aux_bytes(n, int(single)))
    aux = torch.empty(na, dtype=torch.uint8, device='cuda')
    check(lib().m25_getrs_prepare(P(Z), ctypes.c_long(n), n, P(ipiv), int(single), P(aux), ctypes.c_size_t(na),
                                  _lib.stream_ptr()), 'm25_getrs_prepare')
    B = random_matrix(max(n, nrhs), dtype, seed=3)[:n, :nrhs].contiguous()
    s = torch.cuda.current_stream()
    out = []
    for r in range(reps + 1):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        check(lib().m25_getrs_aux(P(Z), ctypes.c_long(n), n, int(single), P(aux), P(B), nrhs, _lib.stream_ptr()),
              'm25_getrs_aux')
        b.record(s)
        _lib.sync_check()
        if r:
            out.append(a.elapsed_time(b))
    ms = float(np.median(out))
    return dict(n=n, nrhs=nrhs, single=single, ms=ms, factor_GBps=n * n * (8 if single else 16) / ms / 1e6)


def time_dense(n, k=8, reps=5):
    """The refinement's dense double product Y = Z X (m25_zgemm_skinny): HBM-bound, 16 n^2 bytes of Z a call."""
    Z = random_matrix(n, torch.complex128)
    X = random_matrix(max(n, k), torch.complex128, seed=3)[:n, :k].contiguous()
    Y = torch.empty_like(X)
    s = torch.cuda.current_stream()
    out = []
    for r in range(reps + 1):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        check(lib().m25_zgemm_skinny(P(Z), ctypes.c_long(n), n, P(X), k, P(Y), _lib.stream_ptr()), 'm25_zgemm_skinny')
        b.record(s)
        _lib.sync_check()
        if r:
            out.append(a.elapsed_time(b))
    ms = float(np.median(out))
    return dict(n=n, k=k, ms=ms, GBps=16.0 * n * n / ms / 1e6)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument('--update', type=int, nargs=3, default=None, metavar=('M', 'N', 'K'))
    ap.add_argument('--solve', type=int, default=0)
    ap.add_argument('--dense', type=int, nargs=2, default=None, metavar=('N', 'K'))
    ap.add_argument('--lu', type=int, default=0)
    ap.add_argument('--single', action='store_true')
    ap.add_argument('--tf32', action='store_true')
    ap.add_argument('--reps', type=int, default=3)
    ap.add_argument('--autotune', action='store_true')
    ap.add_argument('--sizes', type=int, nargs='+', default=None)
    ap.add_argument('--write', action='store_true', help='write the autotuner\'s table to ' + TUNING_FILE)
    a = ap.parse_args()
    _lib.require_cuda()
    if a.autotune:
        c64 = autotune(a.sizes or SIZES[True], single=True, reps=max(1, min(a.reps, 2)))
        c128 = autotune([n for n in a.sizes or SIZES[False] if n <= 20000], single=False, reps=1)
        print(json.dumps(dict(complex64=c64, complex128=c128)))
        if a.write:
            print('wrote', write_tuning(c64, c128))
    if a.lu:
        print(json.dumps(time_lu(a.lu, a.single, a.tf32, a.reps)))
    if a.update:
        print(json.dumps(time_update(*a.update, reps=a.reps)))
    if a.dense:
        print(json.dumps(time_dense(*a.dense, reps=a.reps)))
    if a.solve:
        print(json.dumps(time_solve(a.solve, single=a.single, reps=a.reps)))


if __name__ == '__main__':
    main()
