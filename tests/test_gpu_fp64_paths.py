"""The list build and the pair passes (both forms, and smd_pair_forces_static)
against a direct FP64 sum over all pairs.

The FP64 passes queue the entries that an FP32 test keeps and evaluate those in
FP64, and the list comes from matrix tiles of 16 beads by 8 candidates, so the
sizes are the ones where that can go wrong: a single bead, group and tile
remainders, boxes of exactly three cutoffs, thin list grids (minimum image per
candidate), cells of more than 32 beads, stencils of more than one chunk of
1,024, more neighbours than a queue or a list buffer holds, cells wider than
twice the list cut, and beads on the faces 0 and L.  A bead's force sums at most
a few hundred terms of a few roundings each, so 1e-12 of max |F| (the suite's
plain-form tolerance) leaves a decade; 1e-5 is the suite's for the mixed form.
"""
import ctypes

import numpy as np
import pytest

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu

RC = 2.0
# beads, box
CASES = [(1, (6.5, 6.5, 6.5)), (37, (6.0, 6.0, 6.0)), (613, (6.0, 17.3, 9.9)), (1500, (6.5, 6.5, 6.5)),
         (2501, (31.0, 14.2, 9.1)), (3000, (7.6, 7.7, 7.8)), (1901, (7.6, 7.6, 23.0))]


def _system(n, box):
    rng = np.random.default_rng(n)
    umax = np.array([[100.0, 90.0], [90.0, 200.0]])
    umin = np.array([[0.0, -2.0], [-2.0, -6.0]])
    fc, uc = [], []
    for a in range(2):
        for b in range(2):
            hi, lo = umax[a, b], umin[a, b]
            fc += [1.0, 2.0 * (hi - lo), 0.0, RC, 6.0 * lo, 6.0 * lo]
            uc += [1.0, hi - lo, lo, RC, 3.0 * lo, 2.0 * lo]
    pos = rng.uniform(0.0, 1.0, (n, 3)) * np.array(box)
    for k in range(min(n // 4, 6)):  # on the faces
        pos[k, k % 3] = 0.0 if k < 3 else box[k % 3]
    z = np.zeros((n, 3))
    return smd.Mpd(n_types=2, pos=pos, vel=z, type=rng.integers(0, 2, n).astype(np.int32), box=np.array(box, float),
                   cutoff=RC, fconst=np.array(fc), uconst=np.array(uc), chain_blocks=np.zeros((0, 3), np.int32),
                   chain_consts=np.zeros((0, 4)), dt=0.01, gamma=1.0, temperature=1.0, seed=3, tension=0.0,
                   delta_lxy=0.0, initial_time=0.0, final_time=1.0)


def _direct(m):
    """Forces and potential over all pairs with the minimum image."""
    f, u = np.zeros_like(m.pos), 0.0
    fc, uc = m.fconst.reshape(-1, 6), m.uconst.reshape(-1, 6)
    for i in range(len(m.pos)):
        d = m.pos[i] - m.pos
        d -= np.where(d > m.box / 2, m.box, 0.0) - np.where(d < -m.box / 2, m.box, 0.0)
        r2 = (d * d).sum(1)
        r2[i] = np.inf
        near = r2 < RC * RC
        d, r = d[near], np.sqrt(r2[near])
        row = m.type[i] * 2 + m.type[near]
        c, p = fc[row], uc[row]
        out = (r >= c[:, 0]).astype(int) * 3
        k = np.arange(len(r))
        w = c[k, out] - r
        f[i] = (d * (((c[k, out + 1] - c[k, out + 2] * w) * w) / r)[:, None]).sum(0)
        v, q = p[:, 3] - r, p[:, 0] - r
        u += 0.5 * np.where(r <= p[:, 0], p[:, 1] * q * q + p[:, 2], v * v * (p[:, 4] - v * p[:, 5])).sum()
    return f, u


@pytest.mark.parametrize("n,box", CASES)
def test_fp64_pair_passes_against_all_pairs(built, n, box):
    torch = pytest.importorskip("torch")
    m = _system(n, box)
    want, energy = _direct(m)
    scale = max(np.abs(want).max(), 1.0)
    s = smd.System(m, precision=smd.PLAIN_FP64)
    assert np.abs(s.forces() - want).max() <= 1e-12 * scale
    assert abs(s.energy()[0]["pair"] - energy) <= 1e-12 * max(abs(energy), 1.0)
    s.close()
    s = smd.System(m, precision=smd.MIXED)
    for kern in range(3):
        s.set_tuning(8, kern)
        s.set_state(m.pos)  # builds the list with this kernel
        assert np.abs(s.forces() - want).max() <= 1e-5 * scale
    s.close()
    pos = torch.from_numpy(m.pos).cuda()
    typ = torch.from_numpy(m.type).cuda()
    fc = torch.from_numpy(m.fconst).cuda()
    out = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    b = np.ascontiguousarray(m.box)
    rc = smd.lib().smd_pair_forces_static(pos.data_ptr(), typ.data_ptr(), n, b.ctypes.data, RC, 2, fc.data_ptr(),
                                          out.data_ptr(), ctypes.c_void_p(0))
    assert rc == 0, smd.last_error()
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - want).max() <= 1e-12 * scale


@pytest.mark.parametrize("prec,tol", [(smd.PLAIN_FP64, 1e-12), (smd.MIXED, 1e-5)])
def test_list_of_cells_wider_than_twice_the_cut(built, prec, tol):
    """A box set far larger than the handle's cell grid was sized for."""
    m = _system(700, (7.6, 7.6, 7.6))
    s = smd.System(m, precision=prec)
    m.box = np.array([30.0, 30.0, 30.0])
    s.set_box(m.box)
    want, _ = _direct(m)
    assert np.abs(s.forces() - want).max() <= tol * np.abs(want).max()
    s.close()
