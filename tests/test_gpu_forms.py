"""Which kernel a launch without drift takes is a rule on its size; these tests reach each of them on purpose and
check, by the launch count, that they did: the fused kernel with several frame groups, the paired-tap kernel in the
engine and with a plane per frame (the sweep), and both bicubic forms.

Per push the Fourier engine counts the interpolation's kernels and the RGC's: one fused, or two paired or plain; the
bicubic engine three paired or five tabulated.  The sweep counts two kernels per (magnification, radius) with one
sensitivity and block on the fused kernel, three on the paired one.

Tolerance: 1e-4 of each slice's range, the engine's bar.
"""
import ctypes

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-4


def block(esrrf, frames, M, fwhm, S, kernel="fused", intw=True, chunks=None, fpl=0, fht=True):
    """The block and every push's launch count."""
    eng = esrrf.LiveSRRF_CL()
    n = frames.shape[0]
    eng.initialise(frames.shape[2], frames.shape[1], M, fwhm, S, n, n, intWeighting=intw, kernel=kernel,
                   framesPerLaunch=fpl, doFHTinterpolation=fht)
    counts, s = [], 0
    try:
        eng.resetFramePosition()
        for c in chunks or [n]:
            assert not eng.calculateSRRF(frames[s:s + c])
            counts.append(eng.lastTiming()[2])
            s += c
        return eng.readSRRFbuffer().copy(), counts
    finally:
        eng.release()


def per_pair(esrrf, w, h, n, M, r, frames):
    """Kernels of one (magnification, radius) of a sweep with one sensitivity and block."""
    def count(radii):
        sw = esrrf.Sweep(w, h, n, [M], radii, [1], [(0, n)])
        try:
            sw.run(frames)
            c = ctypes.c_int()
            assert esrrf.lib().esrrf_sweep_launch_count(sw._h, ctypes.byref(c)) == 0
            return c.value
        finally:
            sw.release()
    return count([r, r]) - count([r])


def check_sweep(esrrf, raw, M, r, blocks, sens):
    h, w = raw.shape[1:]
    sw = esrrf.Sweep(w, h, len(raw), [M], [r], sens, blocks)
    try:
        res = sw.run(raw)
    finally:
        sw.release()
    for (_, _, S, (st, ln)), got in res.items():
        ref, _ = block(esrrf, raw[st:st + ln], M, r, S, "plain")
        for k in range(4):
            assert rel_err(got[k], ref[k]) < TOL, (S, st, k)


def test_fused_kernel_with_frame_groups(esrrf_mod, oracle_mod):
    """A 240 x 200 output is 32 CTA tiles (32 x 64) on 296 slots: 20-frame launches split their frames into 5
    groups, each later group re-running the frame before it for TAC2's previous value, sums folded
    atomically, the last values handed to the next launch.  Against the oracle and 3-frame launches (one
    group)."""
    from esrrf import synth
    raw = synth.small_stack(91, 40, 40, 48).astype(np.float32)
    ref = oracle_mod.fht_block(oracle_mod.fht_interpolate(raw, 5), 5, 3.0, 2)
    _, plain = block(esrrf_mod, raw, 5, 3.0, 2, "plain", chunks=[20, 20], fpl=20)
    grouped, n = block(esrrf_mod, raw, 5, 3.0, 2, chunks=[20, 20], fpl=20)
    assert [a + 1 for a in n] == plain, "the launches took the paired kernel"
    _, plain = block(esrrf_mod, raw, 5, 3.0, 2, "plain", chunks=[3] * 13 + [1], fpl=3)
    single, n = block(esrrf_mod, raw, 5, 3.0, 2, chunks=[3] * 13 + [1], fpl=3)
    assert [a + 1 for a in n] == plain
    for k in range(4):
        assert rel_err(grouped[k], ref[k]) < TOL, k
        assert rel_err(grouped[k], single[k]) < 1e-5, k
    assert np.abs(grouped[2]).max() > 0


@pytest.mark.parametrize("w,h,M,r,kernels", [(48, 40, 2, 1.5, 2), (64, 50, 5, 3.0, 2), (100, 90, 4, 1.5, 3),
                                             (161, 120, 4, 1.0, 3)])
def test_sweep_planes_of_both_kernels(esrrf_mod, w, h, M, r, kernels):
    from esrrf import synth
    raw = synth.small_stack(78, 24, h, w, emitters=60)
    assert per_pair(esrrf_mod, w, h, 24, M, r, raw) == kernels
    check_sweep(esrrf_mod, raw, M, r, [(0, 24), (3, 11)], [1, 2])


@pytest.mark.parametrize("S,intw", [(1, True), (3, True), (0, True), (0, False)])
def test_fourier_pushes_of_both_kernels(esrrf_mod, S, intw):
    """A push of 1 on the fused kernel, of 22 and 18 on the paired one: the previous value goes from one to the
    other; sensitivity 0 (every power 1) has no instantiation of its own."""
    from esrrf import synth
    raw = synth.small_stack(77, 41, 57, 90, emitters=60)
    got, n = block(esrrf_mod, raw, 4, 1.5, S, intw=intw, chunks=[1, 22, 18])
    ref, plain = block(esrrf_mod, raw, 4, 1.5, S, "plain", intw=intw, chunks=[1, 22, 18])
    assert [n[0] + 1, n[1], n[2]] == plain
    for k in range(4):
        if S == 0 and not intw and k < 3:  # every value is 1
            np.testing.assert_allclose(got[k], ref[k], atol=1e-5)
        else:
            assert rel_err(got[k], ref[k]) < TOL, k


def test_bicubic_pushes_of_both_forms(esrrf_mod):
    """A push of 1 on the tabulated form, of 22 and 18 on the paired one; then the gradients of the last push's
    first frame, which a paired launch does not leave behind, and the same after a tabulated push."""
    from esrrf import synth
    raw = synth.small_stack(77, 42, 113, 140, emitters=60)
    grads, outs = {}, {}
    for kernel in ("fused", "plain"):
        eng = esrrf_mod.LiveSRRF_CL()
        eng.initialise(140, 113, 4, 1.5, 2, 42, 42, kernel=kernel, doFHTinterpolation=False, framesPerLaunch=22)
        grads[kernel] = []
        try:
            eng.resetFramePosition()
            s = 0
            for c, count in ((1, 5), (22, 3), (18, 3), (1, 5)):
                assert not eng.calculateSRRF(raw[s:s + c])
                s += c
                if kernel == "fused":
                    assert eng.lastTiming()[2] == count, c
                g = np.empty((2, 2 * 113, 2 * 140), np.float32)
                for _ in range(2):
                    esrrf_mod._lib.check(eng.handle, esrrf_mod.lib().esrrf_read_gradients(
                        eng.handle, g.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(g.size)))
                    grads[kernel].append(g.copy())
            outs[kernel] = eng.readSRRFbuffer().copy()
        finally:
            eng.release()
    for a, b in zip(grads["fused"], grads["plain"]):
        np.testing.assert_array_equal(a, b)
    for k in range(4):
        assert rel_err(outs["fused"][k], outs["plain"][k]) < TOL, k


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("intw", [True, False])
def test_paired_fourier_kernel_with_a_frame_that_is_not_finite(esrrf_mod, bad, intw):
    """One such pixel makes its whole interpolated frame NaN: no gradient and no convergence anywhere in it,
    which without intensity weighting leaves AVG, VAR and TAC2 finite."""
    from esrrf import synth
    raw = synth.small_stack(81, 24, 60, 90, emitters=60).astype(np.float32)
    raw[5, 20, 30] = bad
    got, n = block(esrrf_mod, raw, 4, 1.5, 2, intw=intw)
    ref, plain = block(esrrf_mod, raw, 4, 1.5, 2, "plain", intw=intw)
    assert n == plain
    for k in range(4):
        np.testing.assert_array_equal(np.isfinite(got[k]), np.isfinite(ref[k]))
        assert rel_err(got[k], ref[k]) < TOL, k
    assert intw or np.ptp(got[0]) > 0


def test_paired_fourier_kernel_with_gradients_beyond_fp32(esrrf_mod):
    """Intensities around 1e20, the squares of whose larger gradients overflow: such a source has no direction, as
    in the fused kernel (which the allocation-free entry point runs).  5e-6 of AVG's range: the same terms
    summed in another order."""
    import torch
    from esrrf import synth
    raw = synth.small_stack(82, 24, 50, 61, emitters=60).astype(np.float32) * np.float32(1e17)
    got, n = block(esrrf_mod, raw, 4, 1.5, 1, intw=False)
    _, plain = block(esrrf_mod, raw, 4, 1.5, 1, "plain", intw=False)
    assert n == plain
    d = torch.from_numpy(raw).cuda()
    out = torch.empty((4, 200, 244), device="cuda")
    err = ctypes.create_string_buffer(200)
    rc = esrrf_mod.lib().esrrf_fht_block_noalloc(
        ctypes.c_void_p(d.data_ptr()), 0, 24, 61, 50, 4, ctypes.c_float(1.5), 1, 0,
        ctypes.c_void_p(out.data_ptr()), None, err, 200)
    assert rc == 0, err.value
    torch.cuda.synchronize()
    assert np.ptp(got[0]) > 0
    assert rel_err(got[0], out[0].cpu().numpy()) < 5e-6
