"""The paired-tap Fourier kernel on frames whose last strip of 32 columns is not full: lanes right of the image have no
gradient, but need no check of it (rgc_pair.cuh), which cost a frame with such a strip more than a wider one
without."""
import ctypes

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-4


def rgc_us(esrrf, w, h, M, fwhm, n):
    """Device time of the RGC of one launch of n frames, the lower quartile of 16."""
    import torch
    raw = torch.from_numpy(np.random.default_rng(1).poisson(300, (n, h, w)).astype(np.int16)).cuda()
    L = esrrf.lib()
    eng = esrrf.LiveSRRF_CL()
    eng.initialise(w, h, M, fwhm, 2, n, n, framesPerLaunch=n)
    try:
        eng.setTiming(True)
        ts = []
        for _ in range(16):
            eng.resetFramePosition()
            assert L.esrrf_calculate_srrf_u16_device(eng.handle, ctypes.c_void_p(raw.data_ptr()), n) == 0
            ts.append(eng.lastTiming()[1] * 1e3)
        return sorted(ts)[3]
    finally:
        eng.release()


def test_ragged_frame_is_no_slower_than_a_wider_whole_one(esrrf_mod):
    """36 against 64 output columns, two strips each (196 against 119 us with the check)."""
    assert rgc_us(esrrf_mod, 9, 394, 4, 1.5, 6) <= 1.15 * rgc_us(esrrf_mod, 16, 394, 4, 1.5, 6)


# output widths around a strip, heights around one, two and three blocks of rows (12; 8 above radius 8)
@pytest.mark.parametrize("M,fwhm", [(1, 1.0), (4, 1.5), (5, 2.0)])
@pytest.mark.parametrize("W", [31, 32, 33, 63, 65])
@pytest.mark.parametrize("H", [5, 8, 13, 17, 25, 37])
def test_strip_and_block_edges(esrrf_mod, M, fwhm, W, H):
    """Against the per-pixel kernel; a frame without gradient, and a column and a row without in the others."""
    from esrrf import synth
    w, h = max(4, -(-W // M)), max(4, -(-H // M))
    raw = synth.small_stack(50 + M, 24, h, w, emitters=12).astype(np.float32)
    raw[7] = 321.0
    raw[9, :, w // 2:] = 100.0
    raw[11, h // 2:] = 100.0
    out = {}
    for kernel in ("fused", "plain"):
        eng = esrrf_mod.LiveSRRF_CL()
        eng.initialise(w, h, M, fwhm, 2, 24, 24, kernel=kernel)
        try:
            eng.resetFramePosition()
            assert not eng.calculateSRRF(raw)
            out[kernel] = eng.readSRRFbuffer().copy(), eng.lastTiming()[2]
        finally:
            eng.release()
    assert out["fused"][1] == out["plain"][1], "the launch took the fused kernel"
    for k in range(4):
        assert rel_err(out["fused"][0][k], out["plain"][0][k]) < TOL, k
