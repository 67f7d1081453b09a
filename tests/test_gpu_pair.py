"""GPU parity of the paired-tap RGC (two opposite taps at a time, launches without drift) against the
per-pixel kernel with the reference's arithmetic, over the tap boxes it has instantiations for and
frame sizes that leave ragged strips, several row segments and a last, shorter one.

Tolerance: 1e-4 of each slice's range, the engine's bar; a strip's edge column, a row of a chunk or
a tap left out is two orders of magnitude above it.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-4


def block(esrrf, frames, M, fwhm, S, kernel, intw=True, chunks=None):
    eng = esrrf.LiveSRRF_CL()
    n = frames.shape[0]
    eng.initialise(frames.shape[2], frames.shape[1], M, fwhm, S, n, n, intWeighting=intw, kernel=kernel)
    launches = 0
    try:
        eng.resetFramePosition()
        s = 0
        for c in chunks or [n]:
            assert not eng.calculateSRRF(frames[s:s + c])
            launches += eng.lastTiming()[2]
            s += c
        return eng.readSRRFbuffer().copy(), launches
    finally:
        eng.release()


# (M, radius): loop radius R = M (int(2 radius / 2.354) + 1) = 1 .. 15; the disc clipped by the box
# (M 4, radius 3), reaching the corner of the box's unpaired row and column (M 4, radius 1), or with
# no unpaired column at all (M 1, radius 0.5)
@pytest.mark.parametrize("M,fwhm,w,h", [
    (1, 0.5, 200, 180), (1, 2.0, 260, 190), (3, 1.0, 61, 83), (4, 1.0, 75, 50), (5, 0.9, 63, 41),
    (2, 2.5, 97, 111), (7, 1.1, 45, 33), (4, 1.5, 81, 77), (3, 2.5, 67, 59), (5, 2.0, 53, 49),
    (11, 1.0, 45, 41), (4, 3.0, 111, 105), (13, 1.0, 80, 70), (7, 2.0, 140, 130), (5, 3.0, 130, 120)])
def test_pair_every_box(esrrf_mod, M, fwhm, w, h):
    from esrrf import synth
    raw = synth.small_stack(40 + M, 30, h, w, emitters=60).astype(np.float32)
    raw[7] = 321.0  # a frame without any gradient
    got, n = block(esrrf_mod, raw, M, fwhm, 2, "fused")
    ref, n_plain = block(esrrf_mod, raw, M, fwhm, 2, "plain")
    # the paired kernel and its cumulants are two launches, as the plain path's; the fused kernel is one
    assert n == n_plain, "the launch took the fused kernel"
    for k in range(4):
        assert rel_err(got[k], ref[k]) < TOL, k


@pytest.mark.parametrize("S,intw", [(1, True), (3, True), (5, False)])
def test_pair_pushes_and_options(esrrf_mod, S, intw):
    """Uneven pushes carry TAC2's previous value across launches, some of them small enough for the
    fused kernel; sensitivities with and without an instantiation; no intensity weighting."""
    from esrrf import synth
    raw = synth.small_stack(77, 41, 57, 90, emitters=60)
    got, _ = block(esrrf_mod, raw, 4, 1.5, S, "fused", intw, chunks=[1, 22, 18])
    ref, _ = block(esrrf_mod, raw, 4, 1.5, S, "plain", intw)
    for k in range(4):
        assert rel_err(got[k], ref[k]) < TOL, k


def test_pair_sweep_planes(esrrf_mod):
    """The per-frame mode (CGLH over the sum of weights) against the per-pixel kernel's blocks."""
    from esrrf import synth
    raw = synth.small_stack(78, 24, 61, 70, emitters=60)
    sw = esrrf_mod.Sweep(70, 61, 24, [4], [1.0, 1.5], [1, 2], [(0, 24), (3, 11)])
    try:
        res = sw.run(raw)
        # per radius: interpolation once, the paired kernel, its normalisation and one cumulant launch
        out = {k: v.copy() for k, v in res.items()}
    finally:
        sw.release()
    for (M, r, S, (st, ln)), got in out.items():
        ref, _ = block(esrrf_mod, raw[st:st + ln], M, r, S, "plain")
        for k in range(4):
            assert rel_err(got[k], ref[k]) < TOL, (r, S, st, k)


def test_pair_edges_of_a_wide_frame(esrrf_mod, oracle_mod):
    """A few rows of many strips against the oracle."""
    from esrrf import synth
    raw = synth.small_stack(79, 24, 8, 150, emitters=40).astype(np.float32)
    ref = oracle_mod.fht_block(oracle_mod.fht_interpolate(raw, 4), 4, 1.5, 1)
    got, _ = block(esrrf_mod, raw, 4, 1.5, 1, "fused")
    for k in range(4):
        assert rel_err(got[k], ref[k]) < TOL, k


@pytest.mark.parametrize("M,fwhm", [(2, 7.7), (2, 1.1), (3, 4.4), (4, 3.0), (1, 8.5), (5, 1.1), (4, 1.4), (4, 2.3)])
def test_pair_against_the_fused_kernel(esrrf_mod, M, fwhm):
    """Every tap is there once: against the fused kernel (the allocation-free entry point runs it, on the
    same FP32 interpolation at this padded size).  The two sum the same FP32 terms in another order:
    n terms differ by up to sqrt(n) 2^-24 of the sum, 1.6e-6 at 700 taps, so 5e-6 of AVG's range; a row of
    the box's outermost taps is worth 5e-5 at M 2, radius 7.7."""
    import ctypes

    import torch
    from esrrf import synth
    raw = synth.small_stack(60 + M, 24, 50, 61, emitters=60).astype(np.float32)
    got, n = block(esrrf_mod, raw, M, fwhm, 1, "fused", intw=False)
    d = torch.from_numpy(raw).cuda()
    out = torch.empty((4, 50 * M, 61 * M), device="cuda")
    err = ctypes.create_string_buffer(200)
    rc = esrrf_mod.lib().esrrf_fht_block_noalloc(
        ctypes.c_void_p(d.data_ptr()), 0, 24, 61, 50, M, ctypes.c_float(fwhm), 1, 0,
        ctypes.c_void_p(out.data_ptr()), None, err, 200)
    assert rc == 0, err.value
    torch.cuda.synchronize()
    assert rel_err(got[0], out[0].cpu().numpy()) < 5e-6
