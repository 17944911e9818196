"""Branches of the persistent loop and of the list build that the other tests pass by.

* Boxes set far larger than the handle's cell grid was sized for: list cells of
  2.6 and 3 list cuts, where the loop tests candidates by the expanded square
  (five or more cells on every axis) or by differences (fewer).
* Diffusion tracked from the middle of a run on: its steps leave the loop.
* What the loop does not take: BOND and BEND residues, tracked steps.
* Stencils around the list kernel's stage of 640 candidates, on a grid of three
  cells per axis, whose beads per cell leave warps 1, 2, 3 and 4 at a time.

Against the separate kernels (mixed bitwise, plain to 1e-9 over a short run, the
bounds of the loop's other tests) or the FP64 sum over all pairs (1e-12 and 1e-5
of max |F|, the bounds of the pair passes' tests).
"""
import numpy as np
import pytest
from conftest import load_golden, mpd_from_golden
from test_gpu_fp64_paths import _direct, _system

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [smd.MIXED, smd.PLAIN_FP64])
@pytest.mark.parametrize("n,small,big", [(3000, 13.0, 39.0), (900, 8.0, 30.0), (701, 13.0, 39.0), (150, 13.0, 39.0)])
def test_loop_on_wide_cells(built, n, small, big, precision):
    m = _system(n, (small,) * 3)
    m.dt = 0.001
    outs = []
    for persistent in (True, False):
        s = smd.System(m, precision=precision)
        s.set_box(np.full(3, big))
        s.use_graphs(persistent)
        s.prepare()
        l0 = s.launches()
        for k in (1, 5, 20):
            s.advance(k)
        outs.append(s.state() + (s.forces(), s.launches() - l0))
        s.close()
    a, b = outs
    for x, y in zip(a[:3], b[:3]):
        if precision == smd.MIXED:
            assert np.array_equal(x, y)
        else:
            assert np.abs(x - y).max() < 1e-9 * max(1.0, np.abs(y).max())
    assert a[3] < b[3] / 2


@pytest.mark.parametrize("precision", [smd.MIXED, smd.PLAIN_FP64])
def test_diffusion_from_the_middle_of_a_run(built, tmp_path, precision):
    p = str(tmp_path / "d.mpd")
    smd.synth_vesicle(p, 5, 700, 3.45, 30.0)
    m = smd.read_mpd(p)
    n = len(m.type)
    outs = []
    for persistent in (True, False):
        s = smd.System(m, precision=precision)
        s.use_graphs(persistent)
        s.set_msd_groups([0, n // 2, n], np.arange(n))
        s.prepare()
        l0 = s.launches()
        s.advance(19)
        l1 = s.launches()
        s.start_diffusion()
        s.advance(17)
        l2 = s.launches()
        s.advance(4, stop_at_measure=True)
        outs.append((s.state(), s.measure(2)["msd_sum"], l1 - l0, l2 - l1))
        s.close()
    a, b = outs
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y) if precision == smd.MIXED else np.abs(x - y).max() < 1e-9
    assert np.allclose(a[1], b[1], rtol=1e-12 if precision == smd.MIXED else 1e-8, atol=0) and a[1].min() > 0
    assert a[2] < 19 <= b[2] and a[3] >= 17  # the loop, and out of it


@pytest.mark.parametrize("precision", [smd.MIXED, smd.PLAIN_FP64])
def test_who_takes_the_loop(built, precision):
    for name, taken in (("bil400", True), ("net400", False)):
        s = smd.System(mpd_from_golden(load_golden(name)), precision=precision)
        s.prepare()
        s.advance(1)
        l0 = s.launches()
        s.advance(40)
        assert (s.launches() - l0 < 10) == taken
        s.close()


@pytest.mark.parametrize("n", [1, 30, 81, 163, 639, 640, 641, 672, 1279, 1281])
def test_stencils_around_the_stage(built, n):
    m = _system(n, (7.6, 7.6, 7.6))  # three cells per axis: every bead is in every stencil
    want, _ = _direct(m)
    scale = max(np.abs(want).max(), 1.0)
    for precision, tol in ((smd.PLAIN_FP64, 1e-12), (smd.MIXED, 1e-5)):
        s = smd.System(m, precision=precision)
        assert np.abs(s.forces() - want).max() <= tol * scale
        s.close()
