"""bench.py's roofline is a utilisation: lane instructions that the named
kernels execute, by the committed profiles, over the time of the stage they
make up (CPU only, on the counts of the full length-2 enumeration)."""
import importlib.util
import os

import pytest

from conftest import ROOT

COUNTS = {"targets": 7633612, "pairs": 7633612 * 2863, "qc_hits": 6757313, "mid_hits": 5373297, "exh_passed": 1075805,
          "exh_items": 72782}
PEAK = 148 * 128 * 1965e6


def _bench():
    spec = importlib.util.spec_from_file_location("bench_under_test", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("qc_ms,exh_ms,kernels", [(0.84, 0.75, "k_qc_join+k_expand"), (0.84, 1.12, "k_small+k_exhaustive+k_exh_items")])
def test_longest_stage_stays_below_the_peak(qc_ms, exh_ms, kernels):
    b = _bench()
    figs, source = b.load_profile_figures()
    r = b.stage_roofline(COUNTS, {"qc": qc_ms, "exhaustive": exh_ms}, figs, PEAK)
    assert r["kernel"] == kernels and source
    assert 0 < r["frac"] <= 1 and r["frac"] == pytest.approx(r["achieved"] / r["peak"])
    assert r["kernel_ms_per_step"] == max(qc_ms, exh_ms) and r["traffic"] > 0
    assert set(r["issue_active_from_profile"]) == set(kernels.split("+"))


def test_lane_instructions_are_counted_by_their_units():
    b = _bench()
    figs = {k: {"traffic": 1, "issue_active": 0.5, "lane_insts": n} for k, n in (("k_qc_join", 100.0), ("k_expand", 1000.0))}
    r = b.stage_roofline({"targets": 30, "mid_hits": 7}, {"qc": 1.0, "exhaustive": 0.5}, figs, 1e9)
    assert r["frac"] == pytest.approx((100 * 30 + 1000 * 7) / 1e-3 / 1e9)


def test_without_profiles_nothing_is_claimed():
    b = _bench()
    r = b.stage_roofline(COUNTS, {"qc": 1.0, "exhaustive": 0.5}, {}, PEAK)
    assert r["achieved"] is None and r["frac"] is None and r["traffic"] is None
