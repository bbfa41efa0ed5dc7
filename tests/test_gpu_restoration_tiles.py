"""Loop restoration alone against the oracle at the edges of its tiles: sizes
off the pair, word and stripe grid, every chroma layout and depth, all-Wiener,
all-self-guided (every parameter set) and mixed units, chroma units of 32
(whose tiles are one processing column wide) and larger ones, and planes whose
rows start on no word boundary.  Integer arithmetic: tolerance zero."""

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

    ref = fr.copy()
    assert oracle_ctypes.frame_apply(ref.pf(), si.side, None) == 0
    return ref


def frame(w, h, bd, ss, kind, uv):
    """A frame whose units are of one kind; chroma units of `uv` samples."""
    fr, si = synth.make_frame(1, w + 7 * h + bd, width=w, height=h, bit_depth=bd, ss=ss,
                              stages=abi.PF_STAGE_LOOP_RESTORATION)
    rng = np.random.default_rng([w, h, bd, uv])
    lr = si.side.lr
    lr.unit_size_y, lr.unit_size_uv = 64, uv
    for p in range(3):
        us = 64 if p == 0 else uv
        pw, ph = fr.crop[p]
        n = max(1, (pw + us // 2) // us) * max(1, (ph + us // 2) // us)
        units = (abi.pf_lr_unit * n)()
        for i in range(n):
            u = units[i]
            u.type = {"wiener": abi.PF_LR_WIENER, "sgr": abi.PF_LR_SGRPROJ,
                      "mixed": int(rng.choice([abi.PF_LR_NONE, abi.PF_LR_WIENER, abi.PF_LR_SGRPROJ]))}[kind]
            for t in (u.wiener_v, u.wiener_h):
                t[0] = 0 if p else int(rng.integers(-5, 11))
                t[1], t[2] = int(rng.integers(-23, 9)), int(rng.integers(-17, 47))
            u.sgr_set = (i + p * 5) % 16
            u.sgr_xqd[0], u.sgr_xqd[1] = int(rng.integers(-96, 32)), int(rng.integers(-32, 96))
        si.keep.append(units)
        lr.units[p], lr.unit_count[p] = C.addressof(units), n
    return fr, si


@pytest.mark.parametrize("w,h", [(8, 8), (63, 61), (66, 130), (141, 75)])
@pytest.mark.parametrize("ss,uv", [((1, 1), 32), ((1, 1), 64), ((1, 0), 64), ((0, 0), 64), ((0, 1), 64)],
                         ids=["420-32", "420-64", "422", "444", "440"])
@pytest.mark.parametrize("bd", [8, 10, 12])
def test_tiles(runner, w, h, ss, uv, bd):
    for kind in ("wiener", "sgr", "mixed"):
        fr, si = frame(w, h, bd, ss, kind, uv)
        ref, out = oracle(fr, si), fr.copy()
        stats = runner.apply(out.pf(), si.side)
        for p, (a, b) in enumerate(zip(ref.planes, out.planes)):
            assert np.array_equal(a, b), "%s: plane %d differs in %d samples" % (kind, p, int((a != b).sum()))
        # Counted as processing units, whatever the tiles' width.
        want = 0
        for p in range(3):
            sx, sy = ss if p else (0, 0)
            aw, ah = ((w + 7) & ~7) >> sx, ((h + 7) & ~7) >> sy
            want += -(-aw // (64 >> sx)) * -(-(ah + (8 >> sy)) // (64 >> sy))
        assert stats.lr_units == want


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("kind", ["wiener", "sgr"])
def test_rows_off_word_boundaries(runner, bd, kind):
    import torch

    fr, si = frame(131, 70, bd, (1, 1), kind, 64)
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


@pytest.mark.parametrize("w,h", [(63, 61), (141, 130)])
@pytest.mark.parametrize("ss", [(1, 1), (0, 0)], ids=["420", "444"])
@pytest.mark.parametrize("bd", [10, 12])
@pytest.mark.parametrize("kind", ["wiener", "sgr"])
@pytest.mark.parametrize("content", ["spots", "level"])
def test_samples_longer_than_twelve_bits(runner, w, h, ss, bd, kind, content):
    """16-bit words that hold more than 12 bits: single ones, at most one in a
    box (none on a row or column that a border repeats), and whole planes of
    them.  Every box's sum of squares fits 32 bits."""
    fr, si = frame(w, h, bd, ss, kind, 64)
    rng = np.random.default_rng([w, bd])
    for p in fr.planes:
        if content == "spots":
            spots = p[3::8, 3::8]
            spots[:] = rng.integers(1 << 12, 45000 if bd == 10 else 40000, size=spots.shape)
        else:
            p[:] = 8000 + p // (1 << (bd - 9))
    ref, out = oracle(fr, si), fr.copy()
    runner.apply(out.pf(), si.side)
    for p, (a, b) in enumerate(zip(ref.planes, out.planes)):
        assert np.array_equal(a, b), "plane %d differs in %d samples" % (p, int((a != b).sum()))
