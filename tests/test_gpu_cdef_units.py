"""CDEF alone against the oracle at the edges of its units and forms: frames
smaller than a unit, one 8x8 block past a unit, every chroma layout (4:2:0
stages its planes together, the others one by one), 8 and 10 bits (packed
fp16 pairs), 12 bits and 10-bit frames holding longer samples (integers), and
planes whose rows start on no 4-sample boundary.  Integer arithmetic:
tolerance zero."""

import numpy as np
import pytest

from goav1_b200 import abi, synth

pytestmark = pytest.mark.gpu

STAGES = abi.PF_STAGE_CDEF


@pytest.fixture(scope="module")
def runner():
    from goav1_b200.postfilter import PostFilterRunner

    r = PostFilterRunner()
    yield r
    r.close()


def oracle(fr, si):
    import oracle_ctypes

    ref = fr.copy()
    assert oracle_ctypes.frame_apply(ref.pf(), si.side, None) == 0
    return ref


@pytest.mark.parametrize("w,h", [(8, 8), (64, 64), (72, 72), (130, 66), (200, 136)])
@pytest.mark.parametrize("ss", [(1, 1), (1, 0), (0, 0), (0, 1)], ids=["420", "422", "444", "440"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_units(runner, w, h, ss, bd):
    fr, si = synth.make_frame(1, w + 3 * h + bd, width=w, height=h, bit_depth=bd, ss=ss, stages=STAGES)
    ref, out = oracle(fr, si), fr.copy()
    runner.apply(out.pf(), si.side)
    for p, (a, b) in enumerate(zip(ref.planes, out.planes)):
        assert np.array_equal(a, b), "plane %d differs in %d samples" % (p, int((a != b).sum()))


@pytest.mark.parametrize("plane", [0, 1, 2])
@pytest.mark.parametrize("ss", [(1, 1), (0, 0)], ids=["420", "444"])
def test_samples_longer_than_ten_bits(runner, plane, ss):
    fr, si = synth.make_frame(1, 77 + plane, width=200, height=136, bit_depth=10, ss=ss, stages=STAGES)
    rng = np.random.default_rng(plane)
    at = rng.random(fr.planes[plane].shape) < 0.02
    fr.planes[plane][at] = rng.integers(1024, 1100, size=int(at.sum()))
    ref, out = oracle(fr, si), fr.copy()
    runner.apply(out.pf(), si.side)
    for p, (a, b) in enumerate(zip(ref.planes, out.planes)):
        assert np.array_equal(a, b), "plane %d differs in %d samples" % (p, int((a != b).sum()))


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("ss", [(1, 1), (0, 0)], ids=["420", "444"])
def test_rows_off_word_boundaries(runner, bd, ss):
    import torch

    fr, si = synth.make_frame(1, 91 + bd, width=200, height=136, bit_depth=bd, ss=ss, stages=STAGES)
    ref = oracle(fr, si)
    f, keep = fr.pf(memory=abi.PF_MEM_DEVICE, ptrs=[0, 0, 0]), []
    for p, a in enumerate(fr.planes):
        t = torch.zeros((a.shape[0], a.shape[1] + 3), dtype=torch.uint8 if bd == 8 else torch.int16, device="cuda")
        t[:, 1:1 + a.shape[1]] = torch.from_numpy(a if bd == 8 else a.view(np.int16)).cuda()
        keep.append(t)
        f.plane[p].data = t.data_ptr() + t.element_size()
        f.plane[p].stride = t.stride(0) * t.element_size()
    torch.cuda.synchronize()
    runner.apply(f, si.side)
    runner.sync()
    for p, a in enumerate(ref.planes):
        got = keep[p][:, 1:1 + a.shape[1]].cpu().numpy()
        assert np.array_equal(a, got if bd == 8 else got.view(np.uint16)), "plane %d" % p


@pytest.mark.parametrize("plane", [0, 1, 2])
@pytest.mark.parametrize("ss", [(1, 1), (1, 0), (0, 0)], ids=["420", "422", "444"])
@pytest.mark.parametrize("bd", [10, 12])
def test_samples_longer_than_twelve_bits(runner, plane, ss, bd):
    """16-bit words that hold more than 12 bits, in units with and without a
    frame border.  Luma's stay where the direction costs of a block with one
    of them fit 32 bits; with secondary strengths only, and in chroma, which
    have no direction search of their own, they take the whole range."""
    for secondary in (False, True):
        fr, si = synth.make_frame(1, 31 + plane, width=264, height=200, bit_depth=bd, ss=ss, stages=STAGES)
        whole = secondary or plane > 0
        if secondary:
            for i in range(8):
                si.side.cdef.y_strength[i] = 1 + i % 3
                si.side.cdef.uv_strength[i] = 1 + (i + 1) % 3
        rng = np.random.default_rng([plane, bd])
        px = fr.planes[plane]
        at = rng.random(px.shape) < (0.02 if whole else 0.002)
        n = int(at.sum())
        if whole:
            long = rng.integers(1 << 12, 1 << 16, size=n)
            edge = rng.integers(0x3f00, 0x4100, size=n)  # around the value that stands for an absent sample
            px[at] = np.where(rng.random(n) < 0.5, long, edge)
        else:
            px[at] = rng.integers(1 << 12, 0x1400 if bd == 10 else 0x4100, size=n)
        ref, out = oracle(fr, si), fr.copy()
        runner.apply(out.pf(), si.side)
        for p, (a, b) in enumerate(zip(ref.planes, out.planes)):
            assert np.array_equal(a, b), "secondary %s: plane %d differs in %d samples" % (
                secondary, p, int((a != b).sum()))
