"""Deblocking alone against the oracle at the edges of its forms: frames
smaller than a tile and one unit past it, every chroma layout, smooth planes
(the wide filters' flat tests pass) and noisy ones (the narrow filter and its
clamps at both ends of the range), 8 and 10 bits (packed pairs of lines), 12
bits, 10-bit frames holding longer samples and levels above 63 (line by line),
and planes whose rows start on no 4-sample boundary.  Integer arithmetic:
tolerance zero."""

import numpy as np
import pytest

from goav1_b200 import abi, synth

pytestmark = pytest.mark.gpu

STAGES = abi.PF_STAGE_LOOP_FILTER


@pytest.fixture(scope="module")
def runner():
    from goav1_b200.postfilter import PostFilterRunner

    r = PostFilterRunner()
    yield r
    r.close()


def frame(seed, w, h, bd, ss, content):
    """A deblocking-only frame of one of three kinds of samples."""
    fr, si = synth.make_frame(1, seed, width=w, height=h, bit_depth=bd, ss=ss, stages=STAGES)
    rng = np.random.default_rng([seed, 5])
    top = (1 << bd) - 1
    for p in fr.planes:
        if content == "smooth":  # flat blocks, small steps, noise within the flat bound
            y, x = np.indices(p.shape)
            step = rng.integers(0, 4 << (bd - 8), size=((p.shape[0] + 7) // 8, (p.shape[1] + 7) // 8))
            v = (top >> 1) + step[y // 8, x // 8] + rng.integers(0, 2, p.shape)
            p[:] = np.where(rng.random(p.shape) < 0.01, rng.integers(0, top + 1, p.shape), v)
        elif content == "ends":  # both ends of the range, close together
            y, x = np.indices(p.shape)
            side = rng.integers(0, 2, size=((p.shape[0] + 15) // 16, (p.shape[1] + 15) // 16))
            d = rng.integers(0, 6 << (bd - 8), p.shape)
            p[:] = np.where(side[y // 16, x // 16] == 1, top - d, d)
    return fr, si


def check(runner, fr, si):
    import oracle_ctypes

    ref, out = fr.copy(), fr.copy()
    assert oracle_ctypes.frame_apply(ref.pf(), si.side, None) == 0
    runner.apply(out.pf(), si.side)
    for p, (a, b) in enumerate(zip(ref.planes, out.planes)):
        assert np.array_equal(a, b), "plane %d differs in %d samples" % (p, int((a != b).sum()))
    return ref


@pytest.mark.parametrize("w,h", [(8, 8), (64, 64), (132, 36), (200, 136)])
@pytest.mark.parametrize("ss", [(1, 1), (1, 0), (0, 0), (0, 1)], ids=["420", "422", "444", "440"])
@pytest.mark.parametrize("bd", [8, 10, 12])
@pytest.mark.parametrize("content", ["texture", "smooth", "ends"])
def test_units(runner, w, h, ss, bd, content):
    for seed in range(4):
        check(runner, *frame(w + 3 * h + bd + 1000 * seed, w, h, bd, ss, content))


@pytest.mark.parametrize("plane", [0, 1, 2])
def test_samples_longer_than_ten_bits(runner, plane):
    for seed in range(4):
        fr, si = frame(77 + plane + 10 * seed, 200, 136, 10, (1, 1), "smooth")
        rng = np.random.default_rng(plane)
        at = rng.random(fr.planes[plane].shape) < 0.02
        fr.planes[plane][at] = rng.integers(1024, 1100, size=int(at.sum()))
        check(runner, fr, si)


@pytest.mark.parametrize("bd", [8, 10])
def test_rows_off_word_boundaries(runner, bd):
    import oracle_ctypes
    import torch

    fr, si = frame(91 + bd, 200, 136, bd, (1, 1), "smooth")
    ref = fr.copy()
    assert oracle_ctypes.frame_apply(ref.pf(), si.side, None) == 0
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


@pytest.mark.parametrize("bd", [8, 10])
def test_wide_edge_that_ends_with_the_allocated_row(runner, bd):
    """A 14-tap edge (from a malformed mask: its transforms are too narrow)
    whose last tap is the last sample of the allocated row, in a buffer that
    ends there: filtered without touching the word's fourth sample."""
    import oracle_ctypes
    import torch

    w, h, aw, pitch = 16, 16, 19, 20
    fr, si = frame(5, w, h, bd, (1, 1), "smooth")
    fr.planes[0] = np.ascontiguousarray(fr.planes[0][:, :aw])
    fr.planes[0][:] = (1 << (bd - 1)) + np.random.default_rng(bd).integers(0, 2, fr.planes[0].shape)
    masks = np.zeros(abi.PF_LF_MASK_WORDS, np.uint16)
    masks[(3 * 3 + 2) * 2] = 0xf  # vertical edges at column 12, widest class, the four unit rows
    levels = np.full((h // 4, w // 4, 4), 40, np.uint8)
    si.side.lf.masks, si.side.lf.level_cache = masks.ctypes.data, levels.ctypes.data
    ref = fr.copy()
    assert oracle_ctypes.frame_apply(ref.pf(), si.side, None) == 0
    assert not np.array_equal(ref.planes[0], fr.planes[0])
    f, keep = fr.pf(memory=abi.PF_MEM_DEVICE, ptrs=[0, 0, 0]), []
    for p, a in enumerate(fr.planes):
        rows, cols = a.shape
        n = pitch if p == 0 else cols
        flat = torch.zeros(n * (rows - 1) + cols, dtype=torch.uint8 if bd == 8 else torch.int16, device="cuda")
        t = flat.as_strided((rows, cols), (n, 1))
        t.copy_(torch.from_numpy(a if bd == 8 else a.view(np.int16)))
        keep.append(t)
        f.plane[p].data = t.data_ptr()
        f.plane[p].stride = n * t.element_size()
    torch.cuda.synchronize()
    runner.apply(f, si.side)
    runner.sync()
    for p, a in enumerate(ref.planes):
        got = keep[p].cpu().numpy()
        assert np.array_equal(a, got if bd == 8 else got.view(np.uint16)), "plane %d" % p


@pytest.fixture(params=[1, 2, 3], ids=["32x8", "32x16", "32x32"])
def tiled(request):
    """A runner for each tile size (a small frame takes the smallest by itself)."""
    from goav1_b200.postfilter import PostFilterRunner

    r = PostFilterRunner()
    r.set_schedule(abi.PF_TUNE_DEBLOCK, tile=request.param)
    yield r
    r.close()


@pytest.mark.parametrize("w,h", [(132, 36), (200, 136), (264, 330)])
@pytest.mark.parametrize("ss", [(1, 1), (1, 0), (0, 0), (0, 1)], ids=["420", "422", "444", "440"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_tile_sizes(tiled, w, h, ss, bd):
    """One, two and four units a thread on tiles that the frame ends inside:
    shared mask words, the class lists filled from both ends, the level rows."""
    for content in ("texture", "smooth", "ends"):
        check(tiled, *frame(w + 3 * h + bd, w, h, bd, ss, content))


@pytest.mark.parametrize("plane", [0, 1, 2])
def test_tile_sizes_with_samples_longer_than_ten_bits(tiled, plane):
    fr, si = frame(77 + plane, 264, 330, 10, (1, 1), "smooth")
    rng = np.random.default_rng(plane)
    at = rng.random(fr.planes[plane].shape) < 0.02
    fr.planes[plane][at] = rng.integers(1024, 1 << 16, size=int(at.sum()))
    check(tiled, fr, si)


def on_device(fr, bd, gap):
    """A device copy of a frame, each row `gap` samples past a 4-sample boundary."""
    import torch

    f, keep = fr.pf(memory=abi.PF_MEM_DEVICE, ptrs=[0, 0, 0]), []
    for p, a in enumerate(fr.planes):
        t = torch.zeros((a.shape[0], a.shape[1] + 4), dtype=torch.uint8 if bd == 8 else torch.int16, device="cuda")
        t[:, gap:gap + a.shape[1]] = torch.from_numpy(a if bd == 8 else a.view(np.int16)).cuda()
        keep.append(t)
        f.plane[p].data = t.data_ptr() + gap * t.element_size()
        f.plane[p].stride = t.stride(0) * t.element_size()
    torch.cuda.synchronize()
    return f, keep


@pytest.mark.parametrize("bd", [8, 10])
def test_tile_sizes_with_rows_off_word_boundaries(tiled, bd):
    import oracle_ctypes

    fr, si = frame(91 + bd, 264, 330, bd, (1, 1), "smooth")
    ref = fr.copy()
    assert oracle_ctypes.frame_apply(ref.pf(), si.side, None) == 0
    f, keep = on_device(fr, bd, 1)
    tiled.apply(f, si.side)
    tiled.sync()
    for p, a in enumerate(ref.planes):
        got = keep[p][:, 1:1 + a.shape[1]].cpu().numpy()
        assert np.array_equal(a, got if bd == 8 else got.view(np.uint16)), "plane %d" % p


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("content", ["smooth", "ends"])
def test_levels_above_63(tiled, bd, content):
    """A device-side level cache is not looked over: cells above 63 (no
    bitstream has them) go line by line beside others that do not."""
    import ctypes as C

    import oracle_ctypes
    from goav1_b200.postfilter import device_side

    fr, si = frame(19 + bd, 200, 136, bd, (1, 1), content)
    lf = si.side.lf
    levels = np.ctypeslib.as_array(C.cast(lf.level_cache, C.POINTER(C.c_uint8)), (4 * lf.mi_cols * lf.mi_rows,)).copy()
    rng = np.random.default_rng(bd)
    at = rng.random(levels.size) < 0.2
    levels[at] = rng.integers(64, 256, size=int(at.sum()))
    lf.level_cache = levels.ctypes.data
    ref = fr.copy()
    assert oracle_ctypes.lib().oracle_loop_filter(C.byref(ref.pf()), C.byref(si.side)) == 0
    f, keep = on_device(fr, bd, 0)
    tiled.apply(f, device_side(si, fr).side)
    tiled.sync()
    for p, a in enumerate(ref.planes):
        got = keep[p][:, :a.shape[1]].cpu().numpy()
        assert np.array_equal(a, got if bd == 8 else got.view(np.uint16)), "plane %d" % p
