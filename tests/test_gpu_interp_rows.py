"""The tensor-core interpolation of a large launch (the last five) contracts each row of the frame once and
writes the result at every padded row that mirrors it: frames whose padded square repeats a row many
times, once or not at all, row counts around a tile of 128 and a K block of 16, against the float64 interpolation of the padded frame.
Tolerance: 2e-6 of the slice's range, as for square frames (the sums are the same)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,M,n", [(300, 20, 2, 2), (9, 200, 3, 2), (129, 127, 2, 2), (255, 129, 4, 2),
                                     (65, 33, 4, 2), (161, 144, 3, 2), (128, 128, 2, 2),
                                     (300, 110, 2, 26), (400, 129, 2, 20), (640, 260, 2, 8), (97, 600, 2, 38),
                                     (270, 97, 4, 20)])
def test_rows_once(esrrf_mod, w, h, M, n):
    from esrrf import synth
    from oracle import adjoint_oracle as A
    raw = synth.small_stack(200 + w + h + M, n, h, w)
    ref = A.interpolate_f64(raw.astype(np.float64), M).mean(axis=0)
    for frames in (raw, raw.astype(np.float32)):
        eng = esrrf_mod.LiveSRRF_CL()
        eng.initialise(w, h, M, 1.0, 1, n, n)
        try:
            eng.resetFramePosition()
            assert not eng.calculateSRRF(frames)
            got = eng.readSRRFbuffer()[3].copy()
        finally:
            eng.release()
        assert rel_err(got, ref) < 2e-6
