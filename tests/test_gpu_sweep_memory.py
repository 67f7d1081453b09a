"""A sweep's optional plane (the paired-tap kernels' second one) never takes the room of what the sweep cannot do
without: two shards on one device, whose planes and host-run staging come out of the same memory.

The GPU's free memory is brought down by an ordinary allocation.  Output tolerance as for the paired kernels
against the others: 1e-4 of each slice's range.
"""
import numpy as np
import pytest

from conftest import rel_err
from test_gpu_bic_memory import free_bytes, only

pytestmark = pytest.mark.gpu
TOL = 1e-4
BLOCKS = [(k, 20) for k in range(8)] + [(30 + k, 20) for k in range(8)]  # two runs of 27 frames


def sweep(esrrf, interpolation):
    return esrrf.Sweep(256, 256, 57, [4], [1.5], [1, 2, 3], BLOCKS, interpolation=interpolation, devices=[0, 0])


@pytest.mark.parametrize("interpolation", ["fht", "bicubic"])
def test_two_shards_on_one_device(esrrf_mod, interpolation):
    """Room for everything that both shards need and half a plane: a shard that looks at its own needs alone
    takes a plane, and the other's staging then fails."""
    import torch
    from esrrf import synth
    torch.zeros(1, device="cuda")
    raw = synth.small_stack(92, 57, 256, 256, emitters=80)
    P = 4 * 1024 * 1024  # bytes of an output plane
    plane, staging = 27 * P, 3 * 8 * 4 * P + 27 * 4 * 256 * 256
    sweep(esrrf_mod, interpolation).release()  # whatever the first sweep of a process loads
    before = free_bytes()
    sw = sweep(esrrf_mod, interpolation)
    whole = before - free_bytes()
    try:
        ref = {k: v.copy() for k, v in sw.run(raw).items()}
    finally:
        sw.release()
    with only(whole - 2 * plane + 2 * staging + plane // 2):
        sw = sweep(esrrf_mod, interpolation)
        try:
            got = sw.run(raw)
            again = sw.run(raw)
        finally:
            sw.release()
    assert set(got) == set(ref)
    for key in ref:
        np.testing.assert_array_equal(got[key], again[key])
        for k in range(4):
            assert rel_err(got[key][k], ref[key][k]) < TOL, (key, k)


@pytest.mark.parametrize("interpolation", ["fht", "bicubic"])
def test_plane_is_given_back_for_the_staging(esrrf_mod, interpolation):
    """A host run of a sweep whose memory ran short after it was created gives up the plane."""
    import torch
    from esrrf import synth
    torch.zeros(1, device="cuda")
    raw = synth.small_stack(93, 30, 256, 256, emitters=80)
    sw = esrrf_mod.Sweep(256, 256, 30, [4], [1.5], [2], [(0, 30)], interpolation=interpolation)
    try:
        with only(4 << 20):  # the staging is 24 MB, the plane 126
            got = {k: v.copy() for k, v in sw.run(raw).items()}
    finally:
        sw.release()
    sw = esrrf_mod.Sweep(256, 256, 30, [4], [1.5], [2], [(0, 30)], interpolation=interpolation)
    try:
        ref = sw.run(raw)
        for key in ref:
            for k in range(4):
                assert rel_err(got[key][k], ref[key][k]) < TOL, (key, k)
    finally:
        sw.release()
