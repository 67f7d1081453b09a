"""GPU parity of the paired-tap bicubic RGC (magnifications 2 and 4, launches without drift) against the
per-pixel kernel with the reference's arithmetic: the smallest frames, ragged strips and rows, the
shortest and longest discs it takes, several segments, uneven pushes, the sweep's per-frame mode.

Tolerance: 1e-4 of each slice's range, the engine's bar (both sides are FP32 with different orders of
summation, about 1e-6 apart; a column, row or strip misplaced is above 1e-2).
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-4


def block(esrrf, frames, M, fwhm, S, kernel, intw=True, mp=True, chunks=None, gradients=False):
    eng = esrrf.LiveSRRF_CL()
    n = frames.shape[0]
    eng.initialise(frames.shape[2], frames.shape[1], M, fwhm, S, n, n, intWeighting=intw, kernel=kernel,
                   doMPmapCorrection=mp, doFHTinterpolation=False)
    launches = 0
    try:
        eng.resetFramePosition()
        s = 0
        for c in chunks or [n]:
            assert not eng.calculateSRRF(frames[s:s + c])
            launches = eng.lastTiming()[2]
            s += c
        out = eng.readSRRFbuffer().copy()
        if not gradients:
            return out, launches
        g = np.empty((2, 2 * frames.shape[1], 2 * frames.shape[2]), np.float32)
        import ctypes
        esrrf._lib.check(eng.handle, esrrf.lib().esrrf_read_gradients(
            eng.handle, g.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(g.size)))
        return out, g
    finally:
        eng.release()


@pytest.mark.parametrize("M,fwhm,w,h,paired", [
    (2, 1.0, 6, 5, True), (4, 0.5, 120, 77, True), (2, 0.5, 61, 140, True), (4, 1.5, 150, 131, True),
    (2, 3.0, 103, 97, True), (4, 3.0, 161, 150, True), (4, 3.6, 90, 80, False), (3, 1.5, 90, 80, False),
    (4, 1.0, 4, 4, True)])
def test_bic_pair_sizes(esrrf_mod, M, fwhm, w, h, paired):
    from esrrf import synth
    raw = synth.small_stack(30 + M, 24, h, w, emitters=60).astype(np.float32)
    raw[5] = 321.0  # a frame without any gradient
    got, n = block(esrrf_mod, raw, M, fwhm, 2, "fused", mp=False)
    ref, _ = block(esrrf_mod, raw, M, fwhm, 2, "plain", mp=False)
    # per launch the nodes, the paired kernel and its cumulants; the tabulated form has five kernels
    assert (n % 3 == 0 and n % 5 != 0) == paired, "the launch took the other form"
    for k in range(4):
        assert rel_err(got[k], ref[k]) < TOL, k


@pytest.mark.parametrize("S,intw", [(1, True), (3, True), (5, False)])
def test_bic_pair_pushes_options_and_gradients(esrrf_mod, S, intw):
    """Pushes of 1 (tabulated), 22 and 18 frames of uint16; the gradient read-back after a paired launch is
    that of the last launch's first frame."""
    from esrrf import synth
    raw = synth.small_stack(77, 41, 113, 140, emitters=60)
    got, g = block(esrrf_mod, raw, 4, 1.5, S, "fused", intw, chunks=[1, 22, 18], gradients=True)
    ref, h = block(esrrf_mod, raw, 4, 1.5, S, "plain", intw, chunks=[1, 22, 18], gradients=True)
    for k in range(4):
        assert rel_err(got[k], ref[k]) < TOL, k
    np.testing.assert_array_equal(g, h)


def test_bic_pair_nan_and_infinity(esrrf_mod):
    """A NaN and an infinity in a float frame reach the outputs they reach in the per-pixel kernel."""
    from esrrf import synth
    raw = synth.small_stack(78, 12, 100, 120, emitters=60).astype(np.float32)
    raw[3, 40, 50] = np.nan
    raw[4, 20, 90] = np.inf
    got, _ = block(esrrf_mod, raw, 4, 1.5, 1, "fused", mp=False)
    ref, _ = block(esrrf_mod, raw, 4, 1.5, 1, "plain", mp=False)
    for k in range(4):
        np.testing.assert_array_equal(np.isfinite(got[k]), np.isfinite(ref[k]))
        ok = np.isfinite(ref[k])
        assert np.abs(got[k][ok] - ref[k][ok]).max() < TOL * np.ptp(ref[k][ok])


def test_bic_pair_sweep(esrrf_mod):
    """The bicubic sweep with both forms among its (magnification, radius) pairs."""
    from esrrf import synth
    raw = synth.small_stack(79, 24, 101, 120, emitters=60)
    sw = esrrf_mod.Sweep(120, 101, 24, [2, 3, 4], [1.0, 1.5], [1, 2], [(0, 24), (3, 11)], interpolation="bicubic")
    try:
        out = {k: v.copy() for k, v in sw.run(raw).items()}
    finally:
        sw.release()
    for (M, r, S, (st, ln)), got in out.items():
        ref, _ = block(esrrf_mod, raw[st:st + ln], M, r, S, "plain")
        for k in range(4):
            assert rel_err(got[k], ref[k]) < TOL, (M, r, S, st, k)
