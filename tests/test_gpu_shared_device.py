"""Several handles advancing at once: from the third on (or the second, for large
systems) their advances launch kernel by kernel and run side by side, where
persistent loops would queue behind one another; a handle alone takes the loop
again.  The choice changes no bit of a mixed run.  The launch counts tell which
way was taken: two or more launches a step, or a handful per call.
"""
import threading

import numpy as np
import pytest

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu

STEPS = 400


def _handles(tmp_path):
    hs = []
    for k in range(4):
        p = str(tmp_path / f"h{k}.mpd")
        if k % 2:
            smd.synth_vesicle(p, 5 + k, 300 + 17 * k, 3.45, 30.0)
        else:
            smd.synth_bilayer(p, 5 + k, 300 + 17 * k, 3.45, 15.0, 0.01, 0.0)
        s = smd.System(smd.read_mpd(p))
        s.prepare()
        s.autotune()
        hs.append(s)
    return hs


def _rounds(hs, mode):
    """Three rounds of every handle's advance; launches of each handle in the last round."""
    for _ in range(3):
        l0 = [s.launches() for s in hs]
        if mode == "alone":
            for s in hs:
                s.advance(STEPS)
        elif mode == "queued":
            for s in hs:
                s.advance(STEPS, asynchronous=True)
            for s in hs:
                s.sync()
        else:
            ts = [threading.Thread(target=s.advance, args=(STEPS,)) for s in hs]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
    return [s.launches() - l for s, l in zip(hs, l0)]


def test_handles_side_by_side(built, tmp_path):
    out = {}
    for mode in ("alone", "queued", "threads"):
        hs = _handles(tmp_path)
        n = _rounds(hs, mode)
        if mode == "alone":
            assert max(n) < STEPS / 10
        elif mode == "queued":
            assert min(n) > STEPS
            l0 = hs[0].launches()
            hs[0].advance(STEPS)  # still counts the round before
            hs[0].advance(STEPS)  # nobody beside it since: the loop again
            assert hs[0].launches() - l0 > STEPS
            l0 = hs[0].launches()
            hs[0].advance(STEPS)
            assert hs[0].launches() - l0 < STEPS / 10
            hs[0].close()
            hs = hs[1:]
        out[mode] = [s.state() for s in hs]
        for s in hs:
            s.close()
    for mode, skip in (("queued", 1), ("threads", 0)):
        for a, b in zip(out["alone"][skip:], out[mode]):
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_adjoint_beside_others(built, tmp_path):
    """The adjoint's forward and recompute choose the same way: its end state is the same bits."""
    p = str(tmp_path / "a.mpd")
    smd.synth_bilayer(p, 5, 400, 3.45, 15.0, 0.0, 0.0)
    m = smd.read_mpd(p)
    others = _handles(tmp_path)
    res = []
    for beside in (False, True):
        s = smd.System(m)
        s.prepare()
        if beside:
            for h in others:
                h.advance(4 * STEPS, asynchronous=True)
        r = s.adjoint(40, checkpoint_every=20)
        res.append(s.state() + (r["grad"], r["mean_potential"]))
        s.close()
    for h in others:
        h.sync()
        h.close()
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1])
    assert np.allclose(res[0][2], res[1][2], rtol=1e-9) and np.isclose(res[0][3], res[1][3], rtol=1e-12)
