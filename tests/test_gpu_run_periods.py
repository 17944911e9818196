"""The persistent loop at barostat periods other than the usual 8, against the
same loop launched kernel by kernel (smd_use_graphs off).  At a period of 1 a
trial follows a trial with no step between them, so the words that carry a
trial's largest displacement and list slack are cleared behind that trial's own
barrier; at 2 and 3 the trials alternate with one and two plain steps.  The
mixed form's sums are exact in any order, so its runs are bitwise equal.
"""
import numpy as np
import pytest

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu


class _Rate:
    """The library with another barostat period in every descriptor."""

    def __init__(self, rate):
        self._lib, self._rate = smd.lib(), rate

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def smd_create_batch(self, descs, n, precision, out):
        for r in range(n):
            descs[r].resize_rate = self._rate
        return self._lib.smd_create_batch(descs, n, precision, out)


@pytest.mark.parametrize("rate", [1, 2, 3])
@pytest.mark.parametrize("sizes", [(150,), (2601,), (300, 401, 700)])
def test_short_barostat_periods(built, tmp_path, monkeypatch, rate, sizes):
    ms = []
    for k, lipids in enumerate(sizes):
        p = str(tmp_path / f"p{k}.mpd")
        smd.synth_bilayer(p, 3 + k, lipids, 3.45, 15.0, 0.01, 0.1 * k)
        ms.append(smd.read_mpd(p))
    proxy = _Rate(rate)
    monkeypatch.setattr(smd, "lib", lambda: proxy)
    outs = []
    for persistent in (True, False):
        s = smd.System(ms)
        s.use_graphs(persistent)
        s.prepare()
        l0 = s.launches()
        for k in (1, 8, 61, 90):
            s.advance(k)
        outs.append((s.state() + tuple(s.box(r) for r in range(len(ms))), s.rebuilds(),
                     [s.mc_stats(r) for r in range(len(ms))], s.launches() - l0))
        s.close()
    a, b = outs
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)
    assert a[1] == b[1] > 0 and a[2] == b[2]
    assert all(m["trials"] == 159 // rate for m in a[2])
    assert a[3] < b[3] / 10  # (the loop was taken)
