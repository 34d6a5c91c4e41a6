"""The single-field CG (systems whose d and p scales agree, as water) against the
two-field one, which a caller's guess selects: sizes on both sides of the
small/large limit, with short last groups and blocks, and grid lengths whose
rows are multiples of four and of two.

Both run to the same residual, so the dipoles agree to the CG's own error: the
stop at poleps leaves a few poleps (e A) per component, against dipoles of
about 0.1 e A.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def compare(lib, ws, precision):
    poleps = 1e-11 if precision == "FP64" else 1e-7
    bound = 1e-9 if precision == "FP64" else 2e-5
    ctx = lib.Context(ws, precision=getattr(lib, precision), poleps=poleps)
    one = ctx.solve()
    u1, p1 = ctx.dipoles()
    assert np.array_equal(u1, p1)
    ctx.set_guess(np.zeros((ws.n, 2, 3)))
    two = ctx.solve(lib.GUESS_HOST)
    u2, p2 = ctx.dipoles()
    assert one["converged"] and two["converged"]
    scale = np.abs(u2).max()
    assert np.abs(u1 - u2).max() < bound * scale and np.abs(u1 - p2).max() < bound * scale
    assert abs(one["epol"] - two["epol"]) < bound * abs(two["epol"])
    assert np.allclose(one["ene"], two["ene"], rtol=bound)
    # a warm start from the two-field dipoles, back in the single-field form
    again = ctx.solve(lib.GUESS_PREVIOUS)
    assert again["niter"] <= 2 and abs(again["epol"] - one["epol"]) < bound * abs(one["epol"])


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("nw", [216, 1001, 6667, 7001])
def test_single_field_matches_two_fields(thp, nw, precision):
    from tinker_hp_b200 import lib
    compare(lib, thp.water.make_water_box(nw, cfg=0), precision)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("nw,nfft", [(216, 18), (216, 54), (216, 100), (7001, 50), (7001, 64), (7001, 90)])
def test_single_field_grid_lengths(thp, nw, nfft, precision):
    from tinker_hp_b200 import lib
    compare(lib, dataclasses.replace(thp.water.make_water_box(nw, cfg=0), nfft=(nfft,) * 3), precision)
