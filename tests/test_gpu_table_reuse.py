"""Length-2 candidate tables are kept for four masks: a search whose table was
rebuilt in another's place gives what it gave, in both semantics."""
import numpy as np
import pytest

import oracle
from m6502 import _lib

pytestmark = pytest.mark.gpu

MASKS = (0x00, 0x01, 0x42, 0x81, 0x83, 0xC3)


@pytest.mark.parametrize("sem", [_lib.SEM_CUDA, _lib.SEM_GO])
def test_masks_in_turn(engine, sem):
    t = np.asarray(oracle.draw_targets(7, 3, 12), dtype=np.uint16)
    order = ["target", "cand", "cand_len", "dead_flags"]
    first = {}
    for turn in range(2):
        for mask in MASKS:
            rules, st = engine.search(t, dead_flags=mask, semantics=sem, sweep=_lib.SWEEP_REFERENCE, max_cand_len=2)
            got = (np.sort(rules, order=order).tobytes(), st["qc_hits"], st["mid_hits"])
            assert first.setdefault(mask, got) == got, (turn, mask)
    if sem == _lib.SEM_GO:
        for mask in (0x42, 0xC3):
            want, _ = oracle.search_go(t, dead=mask, max_cand_len=2)
            rules, _ = engine.search(t, dead_flags=mask, semantics=sem, sweep=_lib.SWEEP_REFERENCE, max_cand_len=2)
            got = sorted((int(r["target"]), tuple(int(x) for x in r["cand"][:int(r["cand_len"])]), int(r["dead_flags"])) for r in rules)
            assert got == sorted(want), mask
