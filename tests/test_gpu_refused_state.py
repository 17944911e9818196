"""A refused smd_set_state does nothing: state, forces (the plain form's to the
bit, so no bead was reordered), rebuild count and a pending list rebuild are
those of before, and the run goes on as if the call had not been made.
"""
import numpy as np
import pytest
from conftest import load_golden, mpd_from_golden

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["outside", "nan", "velocity"])
@pytest.mark.parametrize("precision", [smd.PLAIN_FP64, smd.MIXED])
def test_refused_state_leaves_everything(built, precision, what):
    m = mpd_from_golden(load_golden("bil400"))
    runs = []
    for refuse in (True, False):
        s = smd.System(m, precision=precision)
        s.prepare()
        counts = []
        for _ in range(12):  # a list lasts about two steps, so some steps leave a rebuild pending
            s.advance(1)
            if refuse:
                pos, vel = s.state()
                before = s.rebuilds()
                bad, badv = pos.copy(), vel.copy()
                if what == "outside":
                    bad[7, 1] = m.box[1] + 3.0
                elif what == "nan":
                    bad[7, 1] = np.nan
                else:
                    badv[7, 1] = np.inf
                with pytest.raises(smd.SmdError):
                    s.set_state(bad, badv)
                assert s.rebuilds() == before
                after = s.state()
                assert np.array_equal(after[0], pos) and np.array_equal(after[1], vel)
            counts.append(s.rebuilds())
        f = s.forces()
        with pytest.raises(smd.SmdError):
            s.set_state(np.full_like(m.pos, np.nan))
        assert np.array_equal(s.forces(), f)
        runs.append((s.state(), counts))
        s.close()
    assert runs[0][1] == runs[1][1] and runs[0][1][-1] > 2
    for a, b in zip(runs[0][0], runs[1][0]):
        assert np.array_equal(a, b) if precision == smd.MIXED else np.abs(a - b).max() < 1e-9
