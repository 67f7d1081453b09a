"""CPU tests of what bench.py says about the kernels that it timed: the RGC form comes from the engine's launch
counts, not from the flags, and a summary's counts are quoted only for the form, and the sources, they were taken of."""
import importlib.util
import os
import re
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_forms_under_test", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    argv = sys.argv
    sys.argv = ["bench.py"]
    try:
        spec.loader.exec_module(mod)
    finally:
        sys.argv = argv
    return mod


@pytest.mark.parametrize("bic,kernel,drift,counts,form", [
    (False, "fused", False, {21}, "fht_rgc_pair"), (False, "fused", False, {18}, "fht_rgc_fused"),
    (False, "fused", False, {20}, "several forms"), (False, "fused", False, {18, 21}, "several forms"),
    (False, "plain", False, {21}, "fht_rgc_plain"), (False, "fused", True, {21}, "fht_rgc_fused"),
    (True, "fused", False, {9}, "bic_pair"), (True, "fused", False, {15}, "bic_tab"),
    (True, "fused", False, {13}, "several forms"), (True, "plain", False, {12}, "bic_rgc"),
    (True, "fused", True, {12}, "bic_rgc")])
def test_form_from_the_launch_counts(bench, bic, kernel, drift, counts, form):
    assert bench.rgc_form(bic, kernel, drift, counts, 3, 7) == form


@pytest.mark.parametrize("kernel", ["rgc_fused_fht512", "rgc_fused_bic512"])
def test_summary_depends_on_the_launch_layout_too(bench, monkeypatch, kernel):
    """The rows a warp walks, and with them instructions and traffic, are set by the host code."""
    real = bench._code_only
    for name in ("pair_shape.cu", {"rgc_fused_fht512": "rgc_pair.cu", "rgc_fused_bic512": "bic_pair.cu"}[kernel]):
        with open(os.path.join(ROOT, "nanoj-esrrf_b200", "csrc", name)) as f:
            text = f.read()
        monkeypatch.setattr(bench, "_code_only", lambda s: real(s + ";") if s == text else real(s))
        assert bench.summary_stale(kernel), name
        monkeypatch.setattr(bench, "_code_only", real)


@pytest.mark.parametrize("kernel,names", [("rgc_fused_fht512", ["fht_rgc_pair", "pair_cumulants"]),
                                          ("rgc_fused_bic512", ["bic_pair", "bic_cumulants"])])
def test_summary_counts_every_timed_kernel(bench, kernel, names):
    """The engine's RGC time spans the paired kernel and its cumulants: the totals are the sums over both."""
    with open(os.path.join(ROOT, "profiles", bench.TRAFFIC_SUMMARIES[kernel])) as f:
        text = f.read()
    rows = {n: re.search(rf"^\| {n}_kernel[^|]*\|([^|]*)\|([^|]*)\|([^|]*)\|", text, flags=re.M) for n in names}
    frames = int(re.search(r"\((\d+) frames; the engine splits", text).group(1))
    inst = sum(float(r.group(1)) for r in rows.values())
    dram = sum(float(r.group(i)) for r in rows.values() for i in (2, 3))
    assert bench.read_traffic_summary(kernel, "warp_instructions_per_frame") == pytest.approx(inst / frames, rel=1e-6)
    assert bench.read_traffic_summary(kernel) == pytest.approx(dram, rel=1e-6)
