"""A chain's course depends on its seed alone: not on how many chains share
its warp (one to four, by how many are searching), nor on their number."""
import pytest

import m6502
from m6502 import _lib

pytestmark = pytest.mark.gpu

P = m6502.inst.parse_assembly
TARGET = P("LDA #$05 : TAX : LDA #$07 : STA M : LDX M")


def _first_chain(engine, chains, targets, cost):
    _, proofs, st = engine.stoke([TARGET] * targets, chains_per_target=chains, steps=600, steps_per_epoch=200, seed=11, cost=cost)
    return [(p["step"], tuple(p["cand"]), p["dead_flags"]) for p in proofs if p["target"] == 0 and p["chain"] == 0]


@pytest.mark.parametrize("cost", [_lib.COST_REF, _lib.COST_HAMMING])
def test_first_chain_is_the_same_among_any_number(engine, cost):
    want = _first_chain(engine, 1, 1, cost)
    assert want
    for chains, targets in ((2, 1), (3, 1), (5, 1), (7, 9), (33, 3), (1777, 2), (2000, 4)):
        assert _first_chain(engine, chains, targets, cost) == want, (chains, targets)
