"""Handles made and first used while the legacy stream is busy: every array of a
handle is cleared and filled on the handle's own stream, which does not wait
for the legacy one, so nothing that a user's other work delays can fall between
an array's contents and their use.  (An array cleared on the legacy stream lost
its contents when the clear came late: gradients without their Umin component,
now and then.)  Compared with the same calls on an idle device; the mixed form
is bitwise reproducible, its gradients' atomic sums to 1e-9.
"""
import numpy as np
import pytest
from conftest import load_golden, mpd_from_golden

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu


def _calls(m, busy):
    s = smd.System(m, precision=smd.MIXED)
    out = []
    for k in range(3):
        busy()
        s.prepare()
        s.advance(5 + 8 * k)
        busy()
        out += list(s.state())
        busy()
        out.append(s.forces())
    s.advance(3, stop_at_measure=True)
    busy()
    q = s.measure()
    out.append(np.concatenate([[q["kinetic"]], q["lo"], q["hi"]]))
    busy()
    r = s.adjoint(300, checkpoint_every=50, umin_types=(3, 3), segment_local=True)
    s.close()
    return out, np.append(r["grad"], r["mean_potential"])


@pytest.mark.parametrize("ms", [1, 4, 16])
def test_first_calls_beside_a_busy_legacy_stream(built, ms):
    torch = pytest.importorskip("torch")
    m = mpd_from_golden(load_golden("bil400"))
    m.delta_lxy = 0.0
    want, grad = _calls(m, lambda: None)
    assert np.all(grad != 0.0)
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()

    def busy():
        torch.cuda._sleep(int(ms * 1.9e6))  # on torch's default stream, the legacy one

    busy()
    got, ggrad = _calls(m, busy)
    torch.cuda.synchronize()
    for x, y in zip(want, got):
        assert np.allclose(x, y, rtol=1e-13, atol=0) if x.ndim == 1 else np.array_equal(x, y)
    assert np.allclose(grad, ggrad, rtol=1e-9, atol=0)
