"""An asynchronous advance captured by the caller as a CUDA graph: its replays go
on from the state that each finds, step number and rebuild flag included.  Four
steps per capture (an even number keeps the mirror's parity, fewer than a
barostat period launch kernel by kernel), bitwise against the same steps
advanced without a capture.
"""
import numpy as np
import pytest

import softmold_gb300 as smd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("lipids", [300, 1501])
def test_replayed_advance(built, tmp_path, graphs, lipids):
    torch = pytest.importorskip("torch")
    p = str(tmp_path / "c.mpd")
    smd.synth_vesicle(p, 3, lipids, 3.45, 40.0)
    m = smd.read_mpd(p)
    torch.cuda.synchronize()
    outs = []
    for captured in (False, True):
        s = smd.System(m)
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        s.use_graphs(graphs)
        s.prepare()
        s.advance(6)
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                s.advance(4, asynchronous=True)
            with torch.cuda.stream(stream):
                for _ in range(25):
                    g.replay()
            s.sync()
        else:
            for _ in range(25):
                s.advance(4)
        outs.append(s.state())
        s.close()
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
