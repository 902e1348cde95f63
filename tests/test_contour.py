"""The host's Sommerfeld contour against the oracle's, for cut-offs K past the lifted part, on its end and before it;
and a frequency's tables' contour as host arrays."""
import numpy as np
import pytest

from oracle import green


@pytest.mark.parametrize('K', [None, 3.0, 1.0 + 1e-9, 1.0, 0.999, 0.2])
@pytest.mark.parametrize('f', [0.1e9, 3.0e9, 10.0e9])
def test_host_contour(K, f):
    """K in units of the lifted part's end t1 (None: the default)."""
    from mom25d_b200 import board as B, device
    st = B.microstrip_board(dmax=0.6e-3, length=10e-3).stack
    t1, *_ = device.contour_path(f, st, 0.02)
    K = None if K is None else K * t1
    kr, dk, K1 = device.sommerfeld_contour(f, st, 0.02, K)
    kr0, dk0, K0 = green.sommerfeld_contour(f, st, 0.02, K)
    m1, n2 = device.contour_path(f, st, 0.02, K)[4:]
    assert K1 == K0 and len(kr) == len(kr0) == 8 * (m1 + n2)
    # breakpoints of m1 + n2 steps: a few ulp of the path's end in a node and in a weight
    tol = 16 * 2.0 ** -53 * max(K1, t1)
    assert np.abs(kr - kr0).max() <= tol and np.abs(dk - dk0).max() <= tol


@pytest.mark.gpu
def test_tables_have_their_contour():
    from mom25d_b200 import board as B, device, geometry as G
    geo = G.Geometry(B.microstrip_board(dmax=0.6e-3, length=10e-3))
    tb = device.DeviceTables(device.DeviceGeometry(geo), 2.0e9)
    kr, dk, K = green.sommerfeld_contour(2.0e9, geo.st, geo.rho_max)
    tol = 16 * 2.0 ** -53 * K
    assert tb.npts == len(tb.kr) == len(tb.dk) == len(kr)
    assert np.abs(tb.kr - kr).max() <= tol and np.abs(tb.dk - dk).max() <= tol
