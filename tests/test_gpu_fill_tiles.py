"""The far fill at the edges of its 32 x 32 tiles (one edge, a tile, a tile and one, several), with the edges in mesh
order and shuffled (the tile's distinct triangle pairs then exceed the shared-memory budget), against the oracle; Z is
exactly symmetric and nothing outside the block is written."""
import importlib.util
import os

import numpy as np
import pytest

import oracle
from oracle import solve as osolve

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.fixture(scope='module')
def case():
    from mom25d_b200 import board as B, geometry as G
    spec = importlib.util.spec_from_file_location('mg', os.path.join(os.path.dirname(__file__), 'golden',
                                                                     'make_golden.py'))
    mg = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mg)
    geo = G.Geometry(mg.small_board(B))
    od = osolve.Direct(geo)
    od.setup(3e9)
    return geo, od


@pytest.mark.parametrize('shuffled', [False, True])
@pytest.mark.parametrize('Ne', [1, 31, 32, 33, 64, 65, 200])
def test_fill_tiles(case, Ne, shuffled):
    from mom25d_b200 import core
    geo, od = case
    pick = np.random.default_rng(Ne).permutation(geo.Ne)[:Ne] if shuffled else np.arange(Ne)
    g = dict(geo.g)
    for k in ('ep', 'em', 'ap', 'am'):
        g[k] = np.ascontiguousarray(np.asarray(geo.g[k])[pick])
    for k in ('vp', 'vm'):
        g[k] = np.ascontiguousarray(np.asarray(geo.g[k]).reshape(-1, 2)[pick])
    Z = np.full((Ne + 1, Ne + 1), 7 + 1j)
    Zo = Z.copy()
    core.fill_far(Z, g, od.tb, od.w)
    oracle.fill_far(Zo, g, od.tb, od.w)
    # two orders of about 40 roundings an entry; entries near zero are differences of the two halves' terms
    assert np.abs(Z - Zo).max() <= 1e-13 * np.abs(Zo[:Ne, :Ne]).max()
    assert np.array_equal(Z[:Ne, :Ne], Z[:Ne, :Ne].T)
    assert np.all(Z[Ne] == 7 + 1j) and np.all(Z[:, Ne] == 7 + 1j)
