"""Film grain alone against the oracle at the edges of its 4x4-sample quads:
widths and heights off the quad, block and tile grid, every chroma layout and
depth, scaling from luma, restricted range, no overlap, inactive planes, and
planes whose rows start on no word boundary.  Integer arithmetic: tolerance
zero."""

import ctypes as C

import numpy as np
import pytest

from goav1_b200 import abi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def runner():
    from goav1_b200.postfilter import PostFilterRunner

    r = PostFilterRunner()
    yield r
    r.close()


def oracle(fr, si):
    import oracle_ctypes

    ref, disp = fr.copy(), fr.like()
    assert oracle_ctypes.frame_apply(ref.pf(), si.side, disp.pf()) == 0
    return disp


OPTIONS = {
    "plain": {},
    "from_luma": dict(chroma_scaling_from_luma=1, num_cb_points=0, num_cr_points=0),
    "restricted": dict(clip_to_restricted_range=1),
    "no_overlap": dict(overlap=0),
    "no_luma": dict(num_y_points=0),
}


@pytest.mark.parametrize("w,h", [(33, 31), (64, 64), (67, 35), (130, 97)])
@pytest.mark.parametrize("ss", [(1, 1), (1, 0), (0, 0), (0, 1)], ids=["420", "422", "444", "440"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_quads(runner, w, h, ss, bd):
    fr, si = synth.make_frame(1, w + 5 * h + bd, width=w, height=h, bit_depth=bd, ss=ss,
                              stages=abi.PF_STAGE_FILM_GRAIN)
    for name, fields in OPTIONS.items():
        saved = {k: getattr(si.side.fg, k) for k in fields}
        for k, v in fields.items():
            setattr(si.side.fg, k, v)
        want, out, disp = oracle(fr, si), fr.copy(), fr.like()
        runner.apply(out.pf(), si.side, disp.pf())
        for p, (a, b) in enumerate(zip(want.planes, disp.planes)):
            assert np.array_equal(a, b), "%s: plane %d differs in %d samples" % (name, p, int((a != b).sum()))
        for k, v in saved.items():
            setattr(si.side.fg, k, v)


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("ss", [(1, 1), (0, 0)], ids=["420", "444"])
def test_rows_off_word_boundaries(runner, bd, ss):
    import torch

    fr, si = synth.make_frame(1, 17 + bd, width=131, height=70, bit_depth=bd, ss=ss, stages=abi.PF_STAGE_FILM_GRAIN)
    want, keep = oracle(fr, si), []

    def device(host, fill):
        f, ts = host.pf(memory=abi.PF_MEM_DEVICE, ptrs=[0, 0, 0]), []
        for p, a in enumerate(host.planes):
            t = torch.zeros((a.shape[0], a.shape[1] + 3), dtype=torch.uint8 if bd == 8 else torch.int16, device="cuda")
            if fill:
                t[:, 1:1 + a.shape[1]] = torch.from_numpy(a if bd == 8 else a.view(np.int16)).cuda()
            ts.append(t)
            f.plane[p].data = t.data_ptr() + t.element_size()
            f.plane[p].stride = t.stride(0) * t.element_size()
        keep.append(ts)
        return f

    f, d = device(fr, True), device(fr.like(), False)
    torch.cuda.synchronize()
    runner.apply(f, si.side, d)
    runner.sync()
    for p, a in enumerate(want.planes):
        got = keep[1][p][:, 1:1 + a.shape[1]].cpu().numpy()
        assert np.array_equal(a, got if bd == 8 else got.view(np.uint16)), "plane %d" % p


@pytest.mark.parametrize("w", [7, 63, 71])
@pytest.mark.parametrize("ss", [(1, 1), (1, 0)], ids=["420", "422"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_last_chroma_column_without_a_right_luma_neighbour(runner, w, ss, bd):
    """Odd widths whose chroma width is a multiple of four: the last quad ends
    at the crop and its last column's scaling index is one luma sample's.  The
    luma padding holds other values than the last column, and no border
    extension makes it alike."""
    import goav1_b200
    from goav1_b200.postfilter import DeviceFrame

    fr, si = synth.make_frame(1, 3 * w + bd, width=w, height=34, bit_depth=bd, ss=ss, stages=abi.PF_STAGE_FILM_GRAIN)
    luma = fr.planes[0]
    luma[:, w:] = ((1 << bd) - 1) - luma[:, w - 1:w]
    for name, fields in OPTIONS.items():
        saved = {k: getattr(si.side.fg, k) for k in fields}
        for k, v in fields.items():
            setattr(si.side.fg, k, v)
        want, out, disp = oracle(fr, si), fr.copy(), fr.like()
        runner.apply(out.pf(), si.side, disp.pf())
        dev, still = DeviceFrame(fr), DeviceFrame(fr.like())
        assert goav1_b200.lib().pf_film_grain_static(C.byref(dev.pf()), C.byref(si.side.fg), C.byref(still.pf()),
                                                     None) == abi.PF_OK
        for p, (a, b, c) in enumerate(zip(want.planes, disp.planes, still.download().planes)):
            assert np.array_equal(a, b), "%s: plane %d differs in %d samples" % (name, p, int((a != b).sum()))
            assert np.array_equal(a, c), "%s, static: plane %d differs in %d samples" % (name, p, int((a != c).sum()))
        for k, v in saved.items():
            setattr(si.side.fg, k, v)
