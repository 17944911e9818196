"""The adjoint pair pass walks a list in stretches of 128 queued entries: the
Hessian-vector product must not depend on how long the list is.  A skin of 0.4
gives one stretch per bead (about 90 entries), 1.6 two (about 220).  The terms
in range are the same bits, so only the order of sums that carry more than 45
bits differs: 1e-11 of the largest component.
"""
import numpy as np
import pytest
from conftest import load_golden, mpd_from_golden

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [smd.MIXED, smd.PLAIN_FP64])
def test_hessian_vector_over_long_lists(built, precision):
    m = mpd_from_golden(load_golden("bil400"))
    w = np.random.default_rng(7).standard_normal((len(m.type), 3))
    out = []
    for skin in (0.4, 1.6):
        s = smd.System(m, precision=precision, skin=skin)
        out.append(s.hessian_vector(w))
        s.close()
    assert np.abs(out[0] - out[1]).max() <= 1e-11 * np.abs(out[0]).max()
