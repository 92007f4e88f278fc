"""Candidates that are one function on every compared output (CandGroups):
the join searches and verifies one member per group and emits the rules of
all.  The scan of every pair knows no groups; rules and stage counts must be
the same at masks with no group, groups of two, and groups of 256."""
import numpy as np
import pytest

import oracle
from m6502 import _lib, inst

pytestmark = pytest.mark.gpu

OP = {n: i for i, n in enumerate(inst.OP_NAMES)}
COUNTS = ("targets", "pairs", "qc_hits", "mid_hits", "exh_checked", "exh_passed", "rules", "exh_algo_ops", "exh_undecided")


def _targets(tlen):
    """Targets that change no live output at some mask (compares and flag
    instructions, reading A, X, Y or M), and seeded random ones."""
    rng = np.random.default_rng(tlen)
    quiet = [OP["CMP_IMM"] | 7 << 8, OP["CMP_IMM"] | 0x80 << 8, OP["CPX_IMM"], OP["CPY_IMM"] | 255 << 8, OP["CMP_M"], OP["CPX_M"],
             OP["BIT_M"], OP["CLC"], OP["SEC"], OP["CLV"], OP["CLD"], OP["SEI"], OP["STA_M"], OP["INX"]]
    made = [[quiet[int(k)] for k in rng.integers(0, len(quiet), tlen)] for _ in range(60)]
    drawn = np.asarray(oracle.draw_targets(tlen, tlen, 120))
    return np.concatenate([np.asarray(made, dtype=np.uint16), drawn.astype(np.uint16)])


@pytest.mark.parametrize("probe", [0, 1])
@pytest.mark.parametrize("mask", [0x00, 0x01, 0x0C, 0x40, 0x41, 0x82, 0x83, 0xC3, 0xCF, 0xFF])
def test_grouped_join_equals_scan(engine, mask, probe):
    saved = engine.tune
    try:
        engine.tune = {"join_probe": probe}
        for tlen, sweep in ((1, _lib.SWEEP_FULL), (2, _lib.SWEEP_FULL), (2, _lib.SWEEP_REFERENCE), (3, _lib.SWEEP_REFERENCE)):
            t = _targets(tlen)
            for mode in ((_lib.EXH_CONES, _lib.EXH_BRUTE) if tlen == 2 and sweep == _lib.SWEEP_REFERENCE else (_lib.EXH_CONES,)):
                a, sa = engine.search(t, dead_flags=mask, sweep=sweep, exh_mode=mode, cap=1 << 20)
                b, sb = engine.search(t, dead_flags=mask, sweep=sweep, exh_mode=mode, cap=1 << 20, qc_scan=True)
                assert np.array_equal(np.sort(a, order=["target", "cand"]), np.sort(b, order=["target", "cand"]))
                assert {k: sa[k] for k in COUNTS} == {k: sb[k] for k in COUNTS}
                n, sc = engine.search(t, dead_flags=mask, sweep=sweep, exh_mode=mode, count_only=True)
                assert n == len(a) and sc["exh_passed"] == sa["exh_passed"]
    finally:
        engine.tune = saved


def test_group_rules_past_the_buffer_stay_staged(engine):
    """A group's 256 rules may straddle the caller's buffer; none is lost."""
    t = np.asarray([[OP["CMP_M"], OP["CMP_IMM"] | 7 << 8]] * 3, dtype=np.uint16)
    full, _ = engine.search(t, dead_flags=0xFF, cap=1 << 14)
    cut, _ = engine.search(t, dead_flags=0xFF, cap=300)
    assert len(full) > 900
    assert np.array_equal(np.sort(full, order=["target", "cand"]), np.sort(cut, order=["target", "cand"]))
