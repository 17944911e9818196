"""The CHAIN part of the plain form's Hessian-vector product rounds no worse than
a square root and divisions do.

20,000 three-bead chains without bending terms, the first bond of each at a
random orientation and stretched along itself (w = the bond vector d on its
first bead), with a rest length of 64 against bonds of 0.5 to 1:
K w = (l/r - 1) d - (l/r) (u . d) u is -d exactly, and what the unit vector u
and l/r lack of the correctly rounded ones is magnified.  Its rms error is held
to that of the same formula in numpy, whose root and divisions are correctly
rounded, and 1 %: three times the spread of an rms over 60,000 roundings.
"""
import numpy as np
import pytest

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu

N, REST = 20000, 64.0


def _fma(a, b, c):
    a, b, c = (np.asarray(v, np.longdouble) for v in (a, b, c))
    return (a * b + c).astype(np.float64)


def test_chain_derivative_rounds_as_divisions_do(built):
    rng = np.random.default_rng(1)
    d = rng.standard_normal((N, 3))
    d *= (rng.uniform(0.5, 1.0, N) / np.sqrt((d * d).sum(1)))[:, None]
    k = np.arange(N)
    first = 2.0 + 2.0 * np.stack([k % 28, k // 28 % 28, k // 784], 1)
    n = 3 * N
    pos, w = np.empty((n, 3)), np.zeros((n, 3))
    pos[0::3], pos[1::3], pos[2::3] = first, first - d, first - d + np.array([0.3, 0.0, 0.0])
    d = pos[0::3] - pos[1::3]
    w[0::3] = d
    m = smd.Mpd(n_types=1, pos=pos, vel=np.zeros((n, 3)), type=np.zeros(n, np.int32), box=np.full(3, 60.0), cutoff=2.0,
                fconst=np.array([1.0, 0, 0, 2.0, 0, 0]), uconst=np.array([1.0, 0, 0, 2.0, 0, 0]),
                chain_blocks=np.array([[0, N, 3]], np.int32), chain_consts=np.array([[REST, 1.0, 0.0, 0.0]]), dt=0.01,
                gamma=1.0, temperature=1.0, seed=3, tension=0.0, delta_lxy=0.0, initial_time=0.0, final_time=1.0)
    s = smd.System(m, precision=smd.PLAIN_FP64)
    got = s.hessian_vector(w)[0::3]
    s.close()
    r = np.sqrt(_fma(d[:, 2], d[:, 2], _fma(d[:, 1], d[:, 1], d[:, 0] * d[:, 0])))
    u, lr = d / r[:, None], REST / r
    b = lr * _fma(u[:, 2], d[:, 2], _fma(u[:, 1], d[:, 1], u[:, 0] * d[:, 0]))
    ref = _fma((lr - 1.0)[:, None], d, -b[:, None] * u)

    def rms(v):  # the exact value is -d
        return float(np.sqrt(((v + d) ** 2).mean()))

    assert 0.0 < rms(got) <= 1.01 * rms(ref)
