"""The single-field CG (systems whose d and p scales agree, as water) against the
two-field one, which a caller's guess selects: sizes on both sides of the
small/large limit and past the one where the pair stream leaves L1 (32,001
waters), with short last groups and blocks, and grid lengths whose rows are
multiples of four and of two.  On a grid that is no cube a system solves two
fields over cuFFT whatever its scales: against the CPU oracle.

Both run to the same residual, so the dipoles agree to the CG's own error: the
stop at poleps leaves a few poleps (e A) per component, against dipoles of
about 0.1 e A.
"""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def compare(lib, ws, precision, poleps=None):
    poleps = poleps or (1e-11 if precision == "FP64" else 1e-7)
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


@pytest.mark.parametrize("precision,poleps", [("FP64", 1e-13), ("MIXED", 1e-7)])
def test_single_field_matches_two_fields_past_l1(thp, precision, poleps):
    # 96,003 atoms: the largest component's error is up to 90 poleps where the
    # two solves stop at different iterations (FP64, both against 1e-14: 3e-10
    # and 9e-10 at 1e-11, 3.6e-12 each at 1e-13), so the FP64 form stops at 1e-13
    from tinker_hp_b200 import lib
    compare(lib, thp.water.make_water_box(32001, cfg=0), precision, poleps)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("nw,nfft", [(216, 18), (216, 54), (216, 100), (7001, 50), (7001, 64), (7001, 90)])
def test_single_field_grid_lengths(thp, nw, nfft, precision):
    from tinker_hp_b200 import lib
    compare(lib, dataclasses.replace(thp.water.make_water_box(nw, cfg=0), nfft=(nfft,) * 3), precision)


@pytest.mark.parametrize("nw,nfft", [(216, (20, 24, 18)), (7001, (60, 64, 54))])
def test_grid_that_is_no_cube_matches_oracle(thp, nw, nfft):
    from tinker_hp_b200 import lib
    ws = dataclasses.replace(thp.water.make_water_box(nw, cfg=0), nfft=nfft)
    orc = O.Oracle(ws, poleps=1e-6)
    assert orc.mlistcell()[0] == 0
    ref = orc.solve()
    e_ref, _ = orc.epolar(ref["uind"])
    for precision, dipole, energy in (("FP64", 1e-6, 1e-8), ("MIXED", 1e-5, 6e-7)):  # D, relative: the forms' bounds
        ctx = lib.Context(ws, precision=getattr(lib, precision), poleps=1e-6)
        res = ctx.solve()
        assert res["converged"]
        for got, want in zip(ctx.dipoles(), (ref["uind"], ref["uinp"])):
            assert np.sqrt(np.mean(np.sum((got - want) ** 2, axis=1))) * 4.80321 < dipole, precision
        assert abs(res["epol"] - e_ref) < energy * abs(e_ref), precision
