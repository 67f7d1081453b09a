"""The autotuner's cache does not hand out launch sizes that were measured with other kernels: entries written
before the paired-tap kernels carry another version."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fht", [True, False])
def test_entries_of_the_earlier_kernels_are_measured_again(esrrf_mod, tmp_path, monkeypatch, fht):
    path = tmp_path / "tune.txt"
    monkeypatch.setenv("ESRRF_TUNE_CACHE", str(path))

    def report():
        eng = esrrf_mod.LiveSRRF_CL()
        eng.initialise(64, 48, 2, 1.5, 1, 30, 30, framesPerLaunch="auto", doFHTinterpolation=fht)
        try:
            return eng.tuneReport()
        finally:
            eng.release()

    first = report()
    assert first["source"] == "measured"
    version, key = first["key"].split("|", 1)
    path.write_text(f"v1|{key} 3 0 0.5\n")
    again = report()
    assert again["source"] == "measured" and again["frames_per_launch"] != 3
    assert report()["source"] == "cache"
