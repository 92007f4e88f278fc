"""The length-1 join takes 1..32 targets per warp, by how many there are.
At the edges of that range, and for targets in enumeration and in random
order (lanes whose opcodes differ), it gives the scan's rules and counts."""
import numpy as np
import pytest

import oracle
from m6502 import _lib

pytestmark = pytest.mark.gpu

COUNTS = ("targets", "pairs", "qc_hits", "mid_hits", "exh_checked", "exh_passed", "rules")


def _same(engine, targets, **kw):
    a, sa = engine.search(targets, cap=1 << 21, **kw)
    b, sb = engine.search(targets, cap=1 << 21, qc_scan=True, **kw)
    order = ["target", "cand", "dead_flags"]
    assert np.array_equal(np.sort(a, order=order), np.sort(b, order=order))
    assert {k: sa[k] for k in COUNTS} == {k: sb[k] for k in COUNTS}
    return len(a)


@pytest.mark.parametrize("n", [1, 31, 33, 4736, 4737, 151553])
@pytest.mark.parametrize("tlen", [1, 2, 3])
def test_join_chunk_edges(engine, n, tlen):
    """4,736 = resident warps of 148 SMs; 151,553 = 32 targets for each and one more."""
    if tlen == 1:
        t = np.resize(oracle.insn_table().astype(np.uint16), n)[:, None]
    else:
        t = np.asarray(oracle.draw_targets(n, tlen, n), dtype=np.uint16)
    for dead in (0x00, 0x82):
        _same(engine, t, dead_flags=dead, sweep=_lib.SWEEP_REFERENCE)
    _same(engine, t, dead_flags=0x00, sweep=_lib.SWEEP_REFERENCE, stages=_lib.CHECK_QC)
    if n <= 4737:
        _same(engine, t, dead_flags=0x41, sweep=_lib.SWEEP_REFERENCE, semantics=_lib.SEM_GO)


@pytest.mark.parametrize("shuffled", [False, True])
def test_join_in_any_target_order(engine, shuffled):
    tab = oracle.insn_table()
    t = np.stack([np.repeat(tab[20:84], 2863), np.tile(tab, 64)], axis=1).astype(np.uint16)
    if shuffled:
        t = t[np.random.default_rng(3).permutation(len(t))]
    assert _same(engine, t, dead_flags=0x00, sweep=_lib.SWEEP_REFERENCE) > 0
    assert _same(engine, t, dead_flags=0x01, sweep=_lib.SWEEP_REFERENCE, stages=_lib.CHECK_QC | _lib.CHECK_MID) > 0
