"""One frame a call under every way its stages are launched: the default
schedules (the frame's job travels as the kernels' argument), a changed one
(the job table), and both with captured graphs on, for host and device frames;
each call against the oracle, with other frames in between."""

import numpy as np
import pytest

from goav1_b200 import abi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("schedule", [None, (abi.PF_TUNE_CDEF, dict(units_per_cta=2)),
                                      (abi.PF_TUNE_FILM_GRAIN, dict(tile=1)),
                                      (abi.PF_TUNE_RESTORATION, dict(ctas=3))],
                         ids=["default", "chunks", "rows", "persistent"])
def test_single_frames(graphs, schedule):
    import oracle_ctypes
    from goav1_b200.postfilter import DeviceFrame, PostFilterRunner, device_side

    r = PostFilterRunner()
    try:
        r.batch_graphs(graphs)
        if schedule:
            r.set_schedule(schedule[0], **schedule[1])
        frames = [synth.make_frame(1, 60 + i, **kw) for i, kw in
                  enumerate((dict(width=200, height=136), dict(width=200, height=136),
                             dict(width=137, height=72, bit_depth=10, ss=(0, 0))))]
        for call in range(2):
            for i, (fr, si) in enumerate(frames):
                ref, rdisp = fr.copy(), fr.like()
                assert oracle_ctypes.frame_apply(ref.pf(), si.side, rdisp.pf()) == 0
                out, disp = fr.copy(), fr.like()
                r.apply(out.pf(), si.side, disp.pf())
                d, dd, ds = DeviceFrame(fr), DeviceFrame(fr.like()), device_side(si, fr)
                r.apply(d.pf(), ds.side, dd.pf())
                r.sync()
                for name, want, got in (("reference", ref, out), ("display", rdisp, disp),
                                        ("device reference", ref, d.download()),
                                        ("device display", rdisp, dd.download())):
                    for p, (a, b) in enumerate(zip(want.planes, got.planes)):
                        assert np.array_equal(a, b), "call %d frame %d %s plane %d" % (call, i, name, p)
    finally:
        r.close()


def test_host_batch_after_a_single_host_frame():
    """A batch of host frames on a context whose copy streams an earlier
    single-frame call made."""
    import oracle_ctypes
    from goav1_b200.postfilter import PostFilterRunner

    r = PostFilterRunner()
    try:
        frames = [synth.make_frame(1, 80 + i, width=200, height=136) for i in range(6)]
        fr, si = frames[0]
        one, one_disp = fr.copy(), fr.like()  # pf() does not own the planes
        r.apply(one.pf(), si.side, one_disp.pf())
        out = [(fr.copy(), fr.like()) for fr, _ in frames]
        r.apply_batch([(o.pf(), si.side, d.pf()) for (o, d), (_, si) in zip(out, frames)])
        for (fr, si), got in zip(frames, out):
            ref, rdisp = fr.copy(), fr.like()
            assert oracle_ctypes.frame_apply(ref.pf(), si.side, rdisp.pf()) == 0
            for want, g in zip((ref, rdisp), got):
                assert all(np.array_equal(a, b) for a, b in zip(want.planes, g.planes))
    finally:
        r.close()
