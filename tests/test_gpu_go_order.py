"""Go semantics: the joins number a target's survivors in Go order as they
meet them, and the first 64 of each pass skip the survivor list.  The scan
sorts its survivors instead; both give the same rules and verify the same
pairs, with up to several hundred survivors per target and pass."""
import numpy as np
import pytest

import oracle
from m6502 import _lib, inst

pytestmark = pytest.mark.gpu

OP = {n: i for i, n in enumerate(inst.OP_NAMES)}


def _targets(tlen):
    """Targets with one, tens and hundreds of survivors: compares of a register
    against nearby operands, flag instructions, dead loads, random ones."""
    rng = np.random.default_rng(17 + tlen)
    some = [OP["CMP_IMM"] | v << 8 for v in (0, 3, 0x41, 0x90, 255)] + [OP["CPX_IMM"] | 9 << 8, OP["CPY_M"], OP["CLC"], OP["SED"],
            OP["CLV"], OP["STA_M"], OP["LDA_IMM"], OP["LDX_M"], OP["TAY"], OP["INX"], OP["ASL_A"]]
    made = np.asarray([[some[int(k)] for k in rng.integers(0, len(some), tlen)] for _ in range(200)], dtype=np.uint16)
    return np.concatenate([made, np.asarray(oracle.draw_targets(tlen, tlen, 300), dtype=np.uint16)])


@pytest.mark.parametrize("mask", [0x00, 0x01, 0x42, 0x81, 0x83, 0xC3, 0xFF])
@pytest.mark.parametrize("tlen", [1, 2, 3])
def test_join_and_scan_verify_in_the_same_order(engine, tlen, mask):
    t = _targets(tlen)
    for sweep in (_lib.SWEEP_REFERENCE, _lib.SWEEP_FULL):
        a, sa = engine.search(t, dead_flags=mask, semantics=_lib.SEM_GO, sweep=sweep)
        b, sb = engine.search(t, dead_flags=mask, semantics=_lib.SEM_GO, sweep=sweep, qc_scan=True)
        order = ["target", "cand", "dead_flags"]
        assert np.array_equal(np.sort(a, order=order), np.sort(b, order=order))
        for k in ("qc_hits", "mid_hits", "exh_checked", "rules"):
            assert sa[k] == sb[k], (k, sweep)
    c, sc = engine.search(t, dead_flags=mask, semantics=_lib.SEM_GO, stages=_lib.CHECK_QC)
    d, sd = engine.search(t, dead_flags=mask, semantics=_lib.SEM_GO, stages=_lib.CHECK_QC, qc_scan=True)
    assert np.array_equal(np.sort(c, order=["target", "cand"]), np.sort(d, order=["target", "cand"]))
    assert sc["qc_hits"] == sd["qc_hits"]


@pytest.mark.parametrize("mask", [0x00, 0x83])
def test_length2_candidates_against_the_oracle(engine, mask):
    """Length-2 candidates: ranges within a chunk, across chunks, and past the first round."""
    t = _targets(3)[::9]
    want, _ = oracle.search_go(t, dead=mask, max_cand_len=2)
    rules, _ = engine.search(t, dead_flags=mask, semantics=_lib.SEM_GO, sweep=_lib.SWEEP_REFERENCE, max_cand_len=2)
    got = sorted((int(r["target"]), tuple(int(x) for x in r["cand"][:int(r["cand_len"])]), int(r["dead_flags"])) for r in rules)
    assert got == sorted(want)
