"""Pair terms with more scaled partners than the kernels hold in registers
(four) and with scale factors that differ between the d and p fields, against
the CPU oracle: two neighbouring waters form one polarization group (five
partners per atom), and the atoms of the second are 1-4 and 1-5 neighbours of
the first.  Sizes with a short last group of four sites and a short last block
of sixteen.

FP64: the gradients within 1e-9 of their largest component (the bound of the
plain water boxes).  Mixed: FP32 pair terms, force RMS within 5e-5
(polarization, which includes the CG stop), 1e-5 (multipoles, van der Waals).
"""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def csr(rows):
    off = np.zeros(len(rows) + 1, np.int32)
    off[1:] = np.cumsum([len(r) for r in rows])
    return off, np.array([v for r in rows for v in r], dtype=np.int32)


def paired_waters(thp, nw):
    """Waters 2m and 2m+1 joined: one polarization group, 1-4 between their
    oxygens and 1-5 between the other atoms of the two."""
    ws = thp.water.make_water_box(nw, cfg=0, edge=21.0)
    n = ws.n
    i14, i15, ip11 = [], [], []
    for i in range(n):
        m = i // 3
        other = m ^ 1
        group = list(range(3 * m, 3 * m + 3))
        if other < nw:
            far = list(range(3 * other, 3 * other + 3))
            i14.append([far[0]] if i % 3 == 0 else [])
            i15.append(far[1:] if i % 3 == 0 else far)
            group = sorted(group + far)
        else:
            i14.append([])
            i15.append([])
        ip11.append(group)
    conn = dict(ws.conn, i14=csr(i14), i15=csr(i15), ip11=csr(ip11))
    scales = dict(ws.scales, p_scale=(0.0, 0.0, 0.7, 0.9), pi_scale=(0.0, 0.1, 0.4, 0.8), d_scale=(0.3, 1.0, 1.0, 1.0),
                  u_scale=(0.6, 1.0, 1.0, 1.0))
    vdw = dict(ws.vdw, v_scale=(0.0, 0.0, 0.6, 0.9))
    return dataclasses.replace(ws, conn=conn, scales=scales, vdw=vdw)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("nw", [217, 222])
def test_gradients_with_many_scaled_partners(thp, nw, precision):
    from tinker_hp_b200 import lib
    ws = paired_waters(thp, nw)
    orc = O.Oracle(ws, poleps=1e-9)
    assert orc.mlistcell()[0] == 0
    ctx = lib.Context(ws, precision=getattr(lib, precision), poleps=1e-9 if precision == "FP64" else 1e-6)
    assert ctx.solve()["converged"]
    _, dep = ctx.gradient()
    uind, uinp = ctx.dipoles()
    if precision == "FP64":
        ref = orc.epolar1(uind, uinp)[1]
    else:
        sol = orc.solve()
        ref = orc.epolar1(sol["uind"], sol["uinp"])[1]
    assert np.abs(uind - uinp).max() > 1e-3  # the two fields do differ here
    got = {"dep": (dep, ref, 5e-5), "dem": (ctx.empole1()[1], orc.empole1()[1], 1e-5),
           "dev": (ctx.ehal1()[1], orc.ehal1()[1], 1e-5)}
    for name, (a, b, rms) in got.items():
        if precision == "FP64":
            assert np.abs(a - b).max() < 1e-9 * np.abs(b).max(), (name, np.abs(a - b).max() / np.abs(b).max())
        else:
            assert np.sqrt(np.mean((a - b) ** 2)) < rms * np.sqrt(np.mean(b ** 2)), name
