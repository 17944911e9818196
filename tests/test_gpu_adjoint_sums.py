"""The mixed form's Hessian-vector product adds its FP32 pair terms in no fewer
bits than FP64 additions would.

Bead 0 sits between twenty mirrored pairs of neighbours, whose w are opposite
and large, and twelve neighbours with w of order one.  Positions are exact on
the 32-bit mirror, so the terms of a mirrored pair are each other's negatives,
bit for bit, and the large part leaves no trace in the exact sum.  What is left
of it is at most one FP64 rounding of the terms' total, 2^-53 (their measure
with FP64 additions: 0.42 of that at most, with two FP32 words up to 21).
"""
import numpy as np
import pytest

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu

BOX, RC = 16.0, 2.0


def _system(rng):
    d = rng.standard_normal((32, 3))
    d *= (rng.uniform(0.6, 1.9, 32) / np.sqrt((d * d).sum(1)))[:, None]
    d = np.round(d * 2.0**20) / 2.0**20  # 2^-28 of a box edge per mirror unit: exact
    pos = 8.0 + np.concatenate([np.zeros((1, 3)), d[:20], -d[:20], d[20:]])
    row = [1.0, 2.0 * 100.0, 0.0, RC, 6.0 * -6.0, 6.0 * -6.0]
    pot = [1.0, 106.0, -6.0, RC, 3.0 * -6.0, 2.0 * -6.0]
    n = len(pos)
    return smd.Mpd(n_types=1, pos=pos, vel=np.zeros((n, 3)), type=np.zeros(n, np.int32), box=np.full(3, BOX),
                   cutoff=RC, fconst=np.array(row), uconst=np.array(pot), chain_blocks=np.zeros((0, 3), np.int32),
                   chain_consts=np.zeros((0, 4)), dt=0.01, gamma=1.0, temperature=1.0, seed=3, tension=0.0,
                   delta_lxy=0.0, initial_time=0.0, final_time=1.0)


def _terms_total(m, w):
    """Sum of the magnitudes of bead 0's terms, per component."""
    d, e = m.pos[0] - m.pos[1:], w[0] - w[1:]
    r = np.sqrt((d * d).sum(1))
    c = m.fconst
    k = 3 * (r >= c[0])
    q = c[k] - r
    g = (c[k + 1] - c[k + 2] * q) * q / r
    s = -((c[k + 1] - 2.0 * c[k + 2] * q) + g) / (r * r)
    return np.abs(g[:, None] * e + (s * (d * e).sum(1))[:, None] * d).sum(0)


@pytest.mark.parametrize("scale", [2.0**20, 2.0**30, 2.0**40])
def test_mixed_sums_keep_fp64_bits(built, scale):
    worst = 0.0
    for seed in range(8):
        rng = np.random.default_rng(seed)
        m = _system(rng)
        w = np.zeros((53, 3))
        w[41:] = rng.standard_normal((12, 3)).astype(np.float32)
        s = smd.System(m, precision=smd.MIXED)
        small = s.hessian_vector(w)[0]
        big = (rng.standard_normal((20, 3)) * scale).astype(np.float32)
        w[1:21], w[21:41] = big, -big
        worst = max(worst, float((np.abs(s.hessian_vector(w)[0] - small) / _terms_total(m, w)).max()))
        s.close()
    assert worst <= 2.0**-53
