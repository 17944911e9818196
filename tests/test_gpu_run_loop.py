"""The persistent loop kernel against the same loop launched kernel by kernel
(smd_use_graphs off), over the sizes where its split changes: the fewest beads
per CTA, each lane count, remainders, thin list grids, a sparse vesicle, BOND
and BEND terms, both forms, and stretches cut at odd steps (mirror parity,
barostat trials at a stretch's first and last step).  The mixed form's sums are
exact in any order, so its runs are bitwise equal; the plain form's differ by
the order of FP64 sums (1e-9 over 40 steps, the suite's trajectory bound).
"""
import numpy as np
import pytest
from conftest import load_golden, mpd_from_golden

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu


def _system(tmp_path, shape, lipids):
    p = str(tmp_path / "r.mpd")
    if shape == "vesicle":
        smd.synth_vesicle(p, 5, lipids, 3.45, 60.0)
    elif shape == "thin":  # 2 list cells along z
        smd.synth_bilayer(p, 5, lipids, 3.45, 6.5, 0.01, 0.1)
    else:
        smd.synth_bilayer(p, 5, lipids, 3.45, 15.0, 0.01, 0.1)
    return smd.read_mpd(p)


def _run(m, persistent, precision, cuts):
    s = smd.System(m, precision=precision)
    s.use_graphs(persistent)
    s.prepare()
    l0 = s.launches()
    for k in cuts:
        s.advance(k)
    out = s.state() + (s.box(), s.mc_stats(), s.rebuilds(), s.forces(), s.launches() - l0)
    s.close()
    return out


CASES = [("bilayer", 150), ("bilayer", 401), ("bilayer", 1300), ("bilayer", 2601), ("bilayer", 9000), ("thin", 700),
         ("vesicle", 300), ("vesicle", 4999), ("vesicle", 13001), ("bilayer", 21650)]


@pytest.mark.parametrize("shape,lipids", CASES)
def test_mixed_loop_bitwise(built, tmp_path, shape, lipids):
    m = _system(tmp_path, shape, lipids)
    cuts = (1, 7, 9, 16, 27, 64)
    a = _run(m, True, smd.MIXED, cuts)
    b = _run(m, False, smd.MIXED, cuts)
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x, y)
    assert a[3] == b[3] and a[4] == b[4] > 0
    assert np.array_equal(a[5], b[5])  # the list and state it leaves serve the other calls
    assert a[6] < b[6] / 10


@pytest.mark.parametrize("shape,lipids", [("bilayer", 150), ("bilayer", 1300), ("thin", 700), ("vesicle", 2999)])
def test_plain_loop(built, tmp_path, shape, lipids):
    m = _system(tmp_path, shape, lipids)
    a = _run(m, True, smd.PLAIN_FP64, (3, 37))
    b = _run(m, False, smd.PLAIN_FP64, (3, 37))
    for x, y in zip(a[:3], b[:3]):
        assert np.abs(x - y).max() < 1e-9
    assert a[3]["trials"] == b[3]["trials"] and a[3]["accepted"] == b[3]["accepted"]


def test_terms(built):
    m = mpd_from_golden(load_golden("net400"))  # BOND and BEND residues
    a, b = _run(m, True, smd.MIXED, (24, 9)), _run(m, False, smd.MIXED, (24, 9))
    for x, y in zip(a[:3], b[:3]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", [smd.MIXED, smd.PLAIN_FP64])
@pytest.mark.parametrize("sizes", [(150, 401, 126, 1300), (2600, 300, 4999, 700), (130,) * 40])
def test_batch_loop(built, tmp_path, sizes, precision):
    """A batch's replicas on CTAs of their own: uneven sizes,
    one replica without a barostat, and few CTAs for many replicas."""
    ms = []
    for k, lipids in enumerate(sizes):
        p = str(tmp_path / f"b{k}.mpd")
        smd.synth_bilayer(p, 7 + k, lipids, 3.45, 15.0, 0.0 if k == 1 else 0.01, 0.1 * (k % 3))
        ms.append(smd.read_mpd(p))
    outs = []
    for persistent in (True, False):
        s = smd.System(ms, precision=precision)
        s.use_graphs(persistent)
        s.prepare()
        l0 = s.launches()
        for k in (1, 8, 31):
            s.advance(k)
        outs.append(s.state() + (np.array([s.box(r) for r in range(len(ms))]), s.launches() - l0,
                                 [s.mc_stats(r) for r in range(len(ms))], s.rebuilds()))
        s.close()
    a, b = outs
    for x, y in zip(a[:3], b[:3]):
        if precision == smd.MIXED:
            assert np.array_equal(x, y)
        else:
            assert np.abs(x - y).max() < 1e-9
    assert a[3] < b[3] / 10
    assert [m["accepted"] for m in a[4]] == [m["accepted"] for m in b[4]]
    assert a[5] == b[5] > 0
