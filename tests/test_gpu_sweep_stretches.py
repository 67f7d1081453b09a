"""The sweep's cumulants sum the stretches between block bounds and add them to the blocks around them:
blocks that overlap, nest, repeat, touch, leave frames out or hold one frame, more of them and more
sensitivities than a launch takes, against each block and sensitivity alone (one stretch).  The FP64 sums
differ in their grouping only, so the FP32 results are within one rounding of each other, and within the
cancellation of 1e-10 of the slice's range where a value is the difference of two sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks,sens", [
    ([(0, 10), (10, 20), (0, 30)], [1, 2, 3]),
    ([(3, 1), (7, 9), (8, 3), (20, 10), (7, 9)], [2, 1, 3, 4, 5]),
    ([(0, 30), (29, 1), (12, 8), (12, 9)], [1, 2]),
    ([(25, 5), (0, 2), (5, 1)], [2]),
])
@pytest.mark.parametrize("weighting", [True, False])
def test_stretches(esrrf_mod, blocks, sens, weighting):
    from esrrf import synth
    raw = synth.small_stack(60, 30, 37, 29, emitters=16)
    kw = dict(int_weighting=weighting)
    sw = esrrf_mod.Sweep(29, 37, 30, [2], [1.0], sens, blocks, **kw)
    try:
        res = sw.run(raw)
    finally:
        sw.release()
    for st, ln in set(blocks):
        for S in sens:
            one = esrrf_mod.Sweep(29, 37, 30, [2], [1.0], [S], [(st, ln)], **kw)
            try:
                ref = one.run(raw)[(2, 1.0, S, (st, ln))]
            finally:
                one.release()
            got = res[(2, 1.0, S, (st, ln))]
            for k in range(4):
                np.testing.assert_allclose(got[k], ref[k], rtol=2.4e-7, atol=1e-10 * np.abs(ref[k]).max())
