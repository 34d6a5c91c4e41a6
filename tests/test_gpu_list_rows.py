"""Neighbour lists of boxes with at least seven cells per axis and 5,000 atoms,
pair for pair against a k-d tree in FP64: unequal edges and cell edges from the smallest to
nearly the largest, atom counts that leave a short last block, atoms outside the
box, a clump so dense that a lane's share of a row does not fit its buffer, and
cutoffs at which some lanes' shares or nearly all do not (each size of buffer), so
that a row is finished from the middle, or at which a smaller system's rows go to
a warp per atom.
Pairs within 1e-9 A of the list radius may be on either side.
"""
import dataclasses

import numpy as np
import pytest
from scipy.spatial import cKDTree

pytestmark = pytest.mark.gpu


def reference(pos, box, r):
    tree = cKDTree(np.mod(pos, box) % box, boxsize=box)
    p = tree.query_pairs(r, output_type="ndarray")
    p.sort(axis=1)
    return p[np.lexsort((p[:, 1], p[:, 0]))]


def keys(p, n):
    return p[:, 0].astype(np.int64) * n + p[:, 1]


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("nw,stretch,clump", [(1667, (1.0, 1.15, 1.3), 1.0), (1701, (1.0, 1.0, 1.0), 1.0),
                                              (3001, (1.2, 1.0, 1.07), 1.0), (7001, (1.0, 1.1, 1.0), 1.0),
                                              (1701, (1.0, 1.0, 1.0), 0.6)])
def test_rows_match_tree(thp, nw, stretch, clump, precision):
    from tinker_hp_b200 import lib
    ws = thp.water.make_water_box(nw, cfg=0)
    box = np.array(ws.box) * stretch
    rng = np.random.default_rng(nw)
    pos = ws.positions() * stretch * clump + 0.37 * box[0]
    pos += rng.integers(-1, 2, pos.shape) * box  # images of the box
    ws = dataclasses.replace(ws.with_positions(pos), box=tuple(box))
    ctx = lib.Context(ws, precision=getattr(lib, precision), max_neighbors=1600)
    ctx.nblist()
    r = ws.ewaldcut + ws.lbuffer
    got = keys(ctx.pairs(1600), ws.n)
    assert len(np.unique(got)) == len(got)
    assert np.isin(keys(reference(pos, box, r - 1e-9), ws.n), got).all()
    assert np.isin(got, keys(reference(pos, box, r + 1e-9), ws.n)).all()
    if clump < 1.0:
        assert 2 * len(got) > 5 * 64 * ws.n  # on average more than the five lanes' buffers hold


@pytest.mark.parametrize("nw,cut", [(3001, 7.5), (3001, 8.5), (7001, 8.0), (7001, 9.0), (7001, 9.5),
                                    (7001, 11.0)])
def test_rows_past_the_buffer_match_tree(thp, nw, cut):
    from tinker_hp_b200 import lib
    ws = dataclasses.replace(thp.water.make_water_box(nw, cfg=0), ewaldcut=cut, vdw=None)
    ctx = lib.Context(ws, precision=lib.FP64, max_neighbors=1000)
    assert all(e >= 7 * (0.5 * (cut + ws.lbuffer) + 1e-6) for e in ws.box)
    ctx.nblist()
    r, box = cut + ws.lbuffer, np.array(ws.box)
    pairs = ctx.pairs(1000)
    got = keys(pairs, ws.n)
    assert len(np.unique(got)) == len(got)
    assert np.isin(keys(reference(ws.positions(), box, r - 1e-9), ws.n), got).all()
    assert np.isin(got, keys(reference(ws.positions(), box, r + 1e-9), ws.n)).all()
