"""The super-resolution upscale against the oracle at the edges of its tiles
(256 output columns by 8 rows), and more super-resolved frames in a batch than
one launch takes.  Integer results: tolerance zero."""

import ctypes as C

import numpy as np
import pytest

from goav1_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def runner():
    from goav1_b200.postfilter import PostFilterRunner

    r = PostFilterRunner()
    yield r
    r.close()


@pytest.mark.parametrize("w", [17, 255, 256, 257, 513])
@pytest.mark.parametrize("h", [1, 7, 8, 9, 65])
@pytest.mark.parametrize("bd", [8, 12])
def test_upscale_tiles(runner, w, h, bd):
    import oracle_ctypes

    rng = np.random.default_rng([w, h, bd])
    for denom in (9, 16):
        coded = synth.HostFrame.alloc((8 * w + denom // 2) // denom, h, bd)
        for p in coded.planes:
            p[:] = rng.integers(0, 1 << bd, size=p.shape)
        up = synth.HostFrame.alloc(w, h, bd)
        want = up.copy()
        assert oracle_ctypes.lib().oracle_superres_upscale(C.byref(coded.pf()), C.byref(want.pf())) == 0
        runner.superres_upscale(coded.pf(), up.pf())
        for p, (a, b) in enumerate(zip(want.planes, up.planes)):
            assert np.array_equal(a, b), "denominator %d: plane %d differs" % (denom, p)


def test_more_frames_than_a_launch_takes(runner):
    import test_gpu_superres_chain as chain
    from goav1_b200.postfilter import DeviceFrame

    cases = [chain.SuperResCase(128 + 32 * (i % 3), 72 + 8 * (i % 4), 9 + i % 8, seed=900 + i) for i in range(11)]
    dev = [[DeviceFrame(f) for f in (c.coded, c.up, c.up.like())] for c in cases]
    runner.apply_batch_superres([(a.pf(), c.side, b.pf(), d.pf()) for c, (a, b, d) in zip(cases, dev)])
    runner.sync()
    for i, (c, frames) in enumerate(zip(cases, dev)):
        for name, want, got in zip(("coded", "upscaled", "display"), chain.run_oracle(c), frames):
            chain.assert_same(want, got.download(), "frame %d %s" % (i, name))
