"""GPU encoder CDEF search vs the CPU oracle (oracle/cdef_search_oracle.cpp):
the per-block SSE table, the chosen presets and the per-block preset index
must be identical (integer path, tolerance zero)."""

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


def _oracle(src, rec, noskip, qindex, lam, max_presets):
    import oracle_ctypes

    w, h = rec.width, rec.height
    mi_cols, mi_rows = ((w + 7) >> 3) << 1, ((h + 7) >> 3) << 1
    nfb = ((mi_cols + 15) // 16) * ((mi_rows + 15) // 16)
    mse = np.zeros((2, nfb, 64), np.uint64)
    idx = np.zeros(nfb, np.uint8)
    res = abi.pf_cdef_search_result()
    prm = abi.pf_cdef_search_params(qindex=qindex, damping=0, max_presets=max_presets, lam=lam)
    st = oracle_ctypes.lib().oracle_cdef_search(C.byref(src.pf()), C.byref(rec.pf()),
                                                noskip.ctypes.data if noskip is not None else None, C.byref(prm),
                                                mse.ctypes.data, idx.ctypes.data, C.byref(res))
    assert st == 0
    return res, mse, idx


def _noskip(side, fr):
    ucols, urows = (fr.width + 63) // 64, (fr.height + 63) // 64
    return np.ctypeslib.as_array((C.c_uint8 * (ucols * urows * 8)).from_address(side.side.cdef.noskip)).copy()


@pytest.mark.parametrize("w,h,qindex,lam", [(256, 192, 100, 2000.0), (640, 360, 180, 9000.0), (200, 130, 40, 300.0)])
def test_search_matches_oracle(runner, w, h, qindex, lam):
    src, rec, side, _ = synth.make_search_pair(7 + w, w, h)
    ns = _noskip(side, rec)
    r0, m0, i0 = _oracle(src, rec, ns, qindex, lam, 8)
    r1, m1, i1 = runner.cdef_search(src.pf(), rec.pf(), ns, qindex, lam)
    assert np.array_equal(m0, m1), "SSE tables differ in %d entries" % int((m0 != m1).sum())
    assert np.array_equal(i0, i1)
    assert (r0.bits, r0.strength_count) == (r1.bits, r1.strength_count)
    assert list(r0.y_strength) == list(r1.y_strength) and list(r0.uv_strength) == list(r1.uv_strength)
    assert r0.cost == r1.cost


def test_search_all_blocks_without_noskip(runner):
    src, rec, _, _ = synth.make_search_pair(3, 192, 128)
    r0, m0, i0 = _oracle(src, rec, None, 128, 4000.0, 4)
    r1, m1, i1 = runner.cdef_search(src.pf(), rec.pf(), None, 128, 4000.0, max_presets=4)
    assert np.array_equal(m0, m1) and np.array_equal(i0, i1)
    assert list(r0.y_strength) == list(r1.y_strength) and r0.bits == r1.bits


@pytest.mark.parametrize("blocks", ["all", "some"])
def test_selection_of_sums_past_32_bits(runner, blocks):
    """240 blocks, most of them as far from their source as samples go: a
    cluster CTA's share of the savings no longer fits 32 bits and is handed
    over in 64 ("some": of part of the CTAs only)."""
    src, rec, _, _ = synth.make_search_pair(5, 1280, 768)
    rng = np.random.default_rng(11)
    for s, r in zip(src.planes, rec.planes):
        far = rng.random(s.shape) < 0.5
        rows = s.shape[0] if blocks == "all" else s.shape[0] // 2
        r[:rows][far[:rows]] = 255
        r[:rows][~far[:rows]] = 0
        s[:rows] = 255 - r[:rows]
    r0, m0, i0 = _oracle(src, rec, None, 128, 4000.0, 8)
    r1, m1, i1 = runner.cdef_search(src.pf(), rec.pf(), None, 128, 4000.0)
    assert m0.max(axis=2).sum(axis=0)[:15].sum() >= 1 << 32  # one CTA's 15 blocks
    assert np.array_equal(m0, m1) and np.array_equal(i0, i1)
    assert (r0.bits, r0.cost) == (r1.bits, r1.cost)
    assert list(r0.y_strength) == list(r1.y_strength) and list(r0.uv_strength) == list(r1.uv_strength)


def test_selection_of_more_blocks_than_shared_memory_holds(runner):
    """2,916 filter blocks, of which about 150 count: the SSE rows are read
    from the table instead of shared memory."""
    w = h = 3456
    src, rec, _, _ = synth.make_search_pair(9, w, h)
    rng = np.random.default_rng(2)
    ns = np.zeros((54 * 54, 8), np.uint8)
    ns[rng.random(54 * 54) < 0.05] = 0xFF
    ns = ns.reshape(-1)
    r0, m0, i0 = _oracle(src, rec, ns, 100, 2000.0, 8)
    r1, m1, i1 = runner.cdef_search(src.pf(), rec.pf(), ns, 100, 2000.0)
    assert np.array_equal(m0, m1) and np.array_equal(i0, i1)
    assert (r0.bits, r0.cost) == (r1.bits, r1.cost)
    assert list(r0.y_strength) == list(r1.y_strength) and list(r0.uv_strength) == list(r1.uv_strength)


def test_search_rejects_unsupported_formats(runner):
    from goav1_b200.postfilter import ErrUnsupportedPostFilter

    fr = synth.HostFrame.alloc(64, 64, 10)
    with pytest.raises(ErrUnsupportedPostFilter):
        runner.cdef_search(fr.pf(), fr.pf(), None, 100, 1000.0)


def test_search_under_a_deadline():
    """A context with a wait limit: a search that meets it gives the oracle's
    table; one that gives up leaves work that pf_sync waits for, the table's
    copy on the second stream included, after which another search is right."""
    import time

    from goav1_b200.postfilter import ErrTimeout, PostFilterRunner

    big = synth.make_search_pair(6, 1920, 1080)
    src, rec, side, _ = synth.make_search_pair(7, 256, 192)
    ns = _noskip(side, rec)
    r0, m0, i0 = _oracle(src, rec, ns, 100, 2000.0, 8)
    hasty, patient = PostFilterRunner(wait_timeout_us=1), PostFilterRunner(wait_timeout_us=10_000_000)

    def finished(f):
        for _ in range(20000):  # bounded: the work takes less than a millisecond
            try:
                return f()
            except ErrTimeout:
                time.sleep(0.0005)
        pytest.fail("still waiting")

    try:
        for _ in range(3):
            with pytest.raises(ErrTimeout):
                hasty.cdef_search(big[0].pf(), big[1].pf(), None, 128, 4000.0)
            finished(hasty.sync)
            with pytest.raises(ErrTimeout):
                hasty.cdef_search(src.pf(), rec.pf(), ns, 100, 2000.0)
            finished(hasty.sync)
            r1, m1, i1 = patient.cdef_search(src.pf(), rec.pf(), ns, 100, 2000.0)
            assert np.array_equal(m0, m1) and np.array_equal(i0, i1) and r0.cost == r1.cost
    finally:
        hasty.close()
        patient.close()
