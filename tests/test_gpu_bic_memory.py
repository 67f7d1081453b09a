"""The bicubic path's paired-tap form needs buffers that a handle can do without: where the GPU has no room
for them the tabulated form takes every launch, and they never take the room of something needed.

The GPU's free memory is brought down by an ordinary allocation.  Output tolerance as for the paired
form against the per-pixel kernel: 1e-4 of each slice's range.
"""
import contextlib

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-4
MB = 1 << 20


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def only(free):
    """Leaves about `free` bytes of the GPU's memory to the code inside."""
    import torch
    torch.cuda.empty_cache()
    hold = torch.empty(free_bytes() - int(free), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hold
        torch.cuda.empty_cache()


def engine(esrrf, w, h, M, n, **kw):
    eng = esrrf.LiveSRRF_CL()
    eng.initialise(w, h, M, 1.5, 2, n, n, doMPmapCorrection=True, doFHTinterpolation=False, **kw)
    return eng


def block(eng, frames):
    """The block and how many kernels its one launch took (paired 3, tabulated 5)."""
    eng.resetFramePosition()
    assert not eng.calculateSRRF(frames)
    return eng.readSRRFbuffer().copy(), eng.lastTiming()[2]


def test_handle_without_room_for_the_paired_form(esrrf_mod):
    """256 x 256 at M4, 25 frames a launch.  The two planes of the paired form take 210 MB, what the handle
    allocates besides its per-frame buffers (accumulators, previous values, output) 55 MB."""
    import torch
    from esrrf import synth
    torch.zeros(1, device="cuda")
    raw = synth.small_stack(90, 25, 256, 256, emitters=80)
    px = 1024 * 1024
    engine(esrrf_mod, 256, 256, 4, 25).release()  # whatever the first handle of a process loads
    before = free_bytes()
    eng = engine(esrrf_mod, 256, 256, 4, 25)
    whole = before - free_bytes()
    ref, n = block(eng, raw)
    assert n == 3
    eng.release()
    planes = 2 * 25 * 4 * px
    # one plane too few; and all of them but with half of the accumulators and the output missing
    for free in (whole - planes // 2, whole - 26 * px):
        with only(free):
            eng = engine(esrrf_mod, 256, 256, 4, 25)
            try:
                got, n = block(eng, raw)
            finally:
                eng.release()
        assert n == 5, "the tabulated form takes the launches"
        for k in range(4):
            assert rel_err(got[k], ref[k]) < TOL, k


def test_planes_are_given_back_for_a_queued_read(esrrf_mod):
    """The second output of a queued read-back is allocated by the first one: if there is no room left by
    then, the handle gives up the paired form's planes (105 MB here against 17 MB)."""
    import torch
    from esrrf import synth
    raw = synth.small_stack(91, 50, 256, 256, emitters=80)
    eng = engine(esrrf_mod, 256, 256, 4, 25, framesPerLaunch=13)
    out = np.empty((2, 4, 1024, 1024), np.float32)
    try:
        ref, n = block(eng, raw[:25])
        assert n == 6
        block(eng, raw[25:])
        with only(8 * MB):
            eng.readSRRFbufferAsync(out[0])
            eng.finishQueue()
        got, n = block(eng, raw[:25])
        assert n == 10
    finally:
        eng.release()
    for k in range(4):
        assert rel_err(got[k], ref[k]) < TOL, k
    eng = engine(esrrf_mod, 256, 256, 4, 25)
    try:
        want, _ = block(eng, raw[25:])
    finally:
        eng.release()
    for k in range(4):
        assert rel_err(out[0][k], want[k]) < TOL, k


def test_launch_size_counts_the_paired_forms_planes(esrrf_mod, tmp_path, monkeypatch):
    """A launch's frames are limited by the memory that they hold in the form they take: 19 input planes and the
    paired form's 2 M^2, 4 GB in all.  What the handle holds besides is counted from its arrays: accumulators
    (4 x 8 bytes an output pixel), previous values, output and sums of weights (6 floats), and the staging."""
    import torch
    torch.zeros(1, device="cuda")
    engine(esrrf_mod, 64, 64, 4, 25).release()
    for w, h, M in ((1024, 1024, 4), (1300, 900, 2)):
        before = free_bytes()
        eng = engine(esrrf_mod, w, h, M, 100)
        held, F = before - free_bytes(), eng.framesPerLaunch()
        eng.release()
        rest = (4 * 8 + 6 * 4) * w * h * M * M + 2 * F * 4 * w * h
        assert held <= 4e9 + rest + 64 * MB, (held, F)
        assert F >= 17  # and still long enough launches
    monkeypatch.setenv("ESRRF_TUNE_CACHE", str(tmp_path / "tune.txt"))
    eng = engine(esrrf_mod, 1024, 1024, 4, 100, framesPerLaunch=-1)
    try:
        tried = [c["frames_per_launch"] for c in eng.tuneReport()["candidates"]]
    finally:
        eng.release()
    assert max(tried) * (19 + 2 * 16) * 4 * 1024 * 1024 <= 4e9, tried
