"""exh_probe_rejects counts every pair that the line states reject before the
cone analysis, also where no filter ran with the join: the candidates of
length 2, the scan's survivors and the Go rounds."""
import numpy as np
import pytest

import m6502
import oracle
from m6502 import _lib

pytestmark = pytest.mark.gpu

P = m6502.inst.parse_assembly
# The flags of the last compare depend on A, M and the carry (17 bits); the
# test vectors leave many operands of it in, all but one of them wrong.
TARGETS = [P(f"ADC M : CMP #${k ^ 0x5A:02X} : CMP #${k:02X}") for k in (0x05, 0x41, 0x77, 0xC8)]


def _differ_on_line_states(t, c):
    """A = i, M = 77 i + 196 ... : the line states of pairs that read A, M and the carry."""
    for i in range(256):
        state = (i, 0, 0, bin(i).count("1") & 1, 0xFD, (77 * i + 196) & 0xFF, 0, 0)
        if oracle.exec_seq(state, t) != oracle.exec_seq(state, c):
            return True
    return False


@pytest.mark.parametrize("sem,scan", [(_lib.SEM_CUDA, False), (_lib.SEM_GO, False), (_lib.SEM_CUDA, True)])
def test_line_rejects_are_counted(engine, sem, scan):
    t = np.asarray(TARGETS, dtype=np.uint16)
    kw = dict(semantics=sem, sweep=_lib.SWEEP_FULL, max_cand_len=2, qc_scan=scan)
    if sem == _lib.SEM_GO:   # what precedes the first passing candidate in its rounds is not known here
        _, st = engine.search(t, **kw)
        assert 0 < st["exh_probe_rejects"] <= st["exh_checked"] - st["exh_passed"]
        return
    rules, st = engine.search(t, **kw)
    pairs, _ = engine.search(t, stages=_lib.CHECK_QC | _lib.CHECK_MID, **kw)
    right = {(int(r["target"]), tuple(r["cand"][:r["cand_len"]].tolist())) for r in rules}
    line = sum(_differ_on_line_states(TARGETS[k], list(c)) for k, c in
               {(int(r["target"]), tuple(r["cand"][:r["cand_len"]].tolist())) for r in pairs} - right
               if c[0] & 0xFF == P("ADC M")[0] and len(c) == 2)
    assert line > 0   # the targets do have such pairs
    assert line <= st["exh_probe_rejects"] <= st["exh_checked"] - st["exh_passed"]
