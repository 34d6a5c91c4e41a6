"""The three-kernel PME convolution against the CPU oracle's FFT path, at every
grid length it covers (FP64: as far as a plane fits in shared memory), and the
grids it leaves to cuFFT (a length outside its list, a grid that is no cube).

thp_tmatxbrecip spreads the dipoles, convolves and gathers the field, so every
grid point and frequency enters.  FP64: sums of order-one terms through about
seven radix stages, within 1e-12 of the largest component; FP32: 24-bit sums
over 125 stencil points and the stages, within 2e-5.
"""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = (16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 150, 160)


@pytest.mark.parametrize("nfft", [(n, n, n) for n in LENGTHS] + [(162, 162, 162), (24, 30, 20)],
                         ids=lambda g: "x".join(map(str, g)))
def test_reciprocal_field_matches_oracle(thp, nfft):
    from tinker_hp_b200 import lib
    ws = dataclasses.replace(thp.water.make_water_box(216, cfg=0), nfft=nfft)
    orc = O.Oracle(ws)
    mu = np.random.default_rng(5).normal(0.0, 0.1, (ws.n, 2, 3))
    ref = orc.tmatxbrecip(mu)
    scale = np.abs(ref).max()
    for precision, bound in (("FP64", 1e-12), ("MIXED", 2e-5)):
        ctx = lib.Context(ws, precision=getattr(lib, precision))
        for _ in range(2):  # the second call spreads into the grid the first one left
            assert np.abs(ctx.tmatxbrecip(mu) - ref).max() < bound * scale, precision


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_virial_leaves_the_grid_ready(thp, precision):
    """The virial's transforms run through cuFFT in the spread grid; the solve
    after them must not see what they leave."""
    from tinker_hp_b200 import lib
    ws = thp.water.make_water_box(216, cfg=0)
    ctx = lib.Context(ws, precision=getattr(lib, precision))
    first = ctx.solve()["epol"]
    ctx.set_virial(True)
    ctx.gradient()
    ctx.empole1()
    assert abs(ctx.solve()["epol"] - first) < (1e-12 if precision == "FP64" else 1e-6) * abs(first)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_batch_of_both_kinds_of_grid(thp, precision):
    """A batch plan whose systems share neither grid shape nor convolution."""
    from tinker_hp_b200 import lib
    base = thp.water.make_water_box(216, cfg=0)
    boxes = [dataclasses.replace(base, nfft=g) for g in ((20, 20, 20), (20, 24, 20), (20, 20, 20), (162, 16, 16))]
    ctxs = [lib.Context(b, precision=getattr(lib, precision)) for b in boxes]
    alone = []
    for c in ctxs:
        c.solve()
        alone.append(c.dipoles()[0])
    plan = lib.Batch(ctxs)
    for _ in range(8):  # through the tuning solves
        plan.solve()
        for c, ref in zip(ctxs, alone):
            got = c.dipoles()[0]
            assert np.abs(got - ref).max() < (1e-10 if precision == "FP64" else 2e-6) * np.abs(ref).max()
