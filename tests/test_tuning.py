"""The LU's tuning table (m25_set_lu_tuning / m25_get_lu_tuning, filled by the autotuner mom25d_b200.tune): entry
lookup by size, the defaults without entries, argument checks, and the table file the library applies at load.
Host-side only: no kernel runs."""
import ctypes
import json

import pytest

from mom25d_b200 import _lib


def _get(L, n, single=1):
    a, b = ctypes.c_int(), ctypes.c_int()
    assert L.m25_get_lu_tuning(n, single, ctypes.byref(a), ctypes.byref(b)) == 0
    return a.value, b.value


def test_table_lookup_and_defaults(monkeypatch):
    monkeypatch.delenv('M25_NB2', raising=False)
    monkeypatch.delenv('M25_PANEL_BLOCKS', raising=False)
    from mom25d_b200 import tune
    L = _lib.lib()
    tune.set_table([(15000, 192, 48), (1000, 128, 16)])
    try:
        assert _get(L, 500) == (128, 16)                   # the entry nearest in log n
        assert _get(L, 3800) == (128, 16) and _get(L, 4000) == (192, 48)
        assert _get(L, 18788) == (192, 48)
        assert _get(L, 18788, single=0) == (256, min(32, _get(L, 18788, single=0)[1]))   # complex128: its own table
        monkeypatch.setenv('M25_NB2', '64')
        assert _get(L, 18788)[0] == 64                     # the environment overrides
        monkeypatch.delenv('M25_NB2')
        bad = (ctypes.c_int * 1)
        assert L.m25_set_lu_tuning(1, bad(5), bad(100), bad(3), 1) == 1   # nb2 not a multiple of 64
        assert _get(L, 18788) == (192, 48)                 # a refused table leaves the last one
    finally:
        tune.set_table([])
    nb2, blocks = _get(L, 5000)
    assert nb2 == 256 and 1 <= blocks <= 32


def test_tuning_file_is_applied(tmp_path):
    L = _lib.lib()
    f = tmp_path / 't.json'
    f.write_text(json.dumps(dict(device='test', sms=None, complex64=[dict(n=1, nb2=256, blocks=24, ms=1.0)],
                                 complex128=[dict(n=1, nb2=192, blocks=16, ms=1.0)])))
    try:
        assert _lib.apply_tuning(L, str(f))
        assert _get(L, 20000) == (256, 24) and _get(L, 20000, single=0) == (192, 16)
    finally:
        L.m25_set_lu_tuning(1, None, None, None, 0)
        L.m25_set_lu_tuning(0, None, None, None, 0)
        _lib.apply_tuning(L)                               # back to the committed table, if any


def _lu_model(lines, tried):
    """A stand-in for tune.time_lu: a factorisation's outer blocks are walked as m25_getrf walks them, each at the width
    the library's table has for the size left; a row costs 1 at the best width there (lines: {width: rows left above
    which it is the best}), more the further its width is from that."""
    def time_lu(n, single=False, tf32=False, reps=3):
        ms, left = 0.0, n
        while left > 0:
            w = _get(_lib.lib(), left, int(single))[0]
            best = max((b for b in lines if left > lines[b]), key=lambda b: lines[b])
            ms += min(w, left) * (1 + abs(w - best) / 64) * 1e-3
            tried.append((single, left, w))
            left -= w
        return dict(ms=ms)
    return time_lu


@pytest.mark.parametrize('single,lines,want', [
    (True, {64: 0, 128: 2828, 256: 5000}, {500: 64, 2700: 64, 2900: 128, 4900: 128, 5100: 256, 18788: 256}),
    (False, {64: 0, 128: 2828, 256: 5477}, {500: 64, 2700: 64, 2900: 128, 5400: 128, 5600: 256, 18788: 256}),
    (False, {128: 0, 192: 5477, 256: 8660}, {500: 128, 5400: 128, 5600: 192, 8600: 192, 8700: 256, 18788: 256})])
def test_autotuner_finds_the_lines(single, lines, want, monkeypatch):
    """The autotuner times the tables a factorisation uses: with costs that change at the lines between its sizes it
    finds the widths on both sides of each, the 128 columns of the complex64 table among them."""
    from mom25d_b200 import tune
    monkeypatch.delenv('M25_NB2', raising=False)
    monkeypatch.delenv('M25_PANEL_BLOCKS', raising=False)
    tried = []
    monkeypatch.setattr(tune, 'time_lu', _lu_model(lines, tried))
    L = _lib.lib()
    try:
        out = tune.autotune(tune.SIZES[single], single=single, log=None)
        assert {n: _get(L, n, int(single))[0] for n in want} == want
        assert all(set(e) >= {'n', 'nb2', 'blocks', 'ms'} for e in out)
        if single:                                         # 3xTF32 on the next block's columns: 64 or 256 only
            assert all(w in (64, 256) for s, left, w in tried if left > tune.FP32_ROWS)
    finally:
        _lib.apply_tuning(L)


def test_committed_table():
    """The committed table is of the autotuner's own form: its sizes, its candidates, a time each."""
    from mom25d_b200 import tune
    doc = json.load(open(tune.TUNING_FILE))
    for key, single in (('complex64', True), ('complex128', False)):
        es = doc[key]
        ns = [e['n'] for e in es]
        assert ns == tune.SIZES[single] and all(e['ms'] > 0 for e in es)
        for e, above in zip(es, ns[1:] + [None]):
            assert (e['nb2'], e['blocks']) in tune.candidates(e['n'], above, single)
