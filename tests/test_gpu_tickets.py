"""Which warp takes which pair: counts around one pair per block, one per warp
and several per warp of the verification's grids, and lists that are mostly
pairs for the exhaustive kernel.  Every verdict is the oracle's for that pair,
whatever the list's length and order."""
import functools

import pytest

import oracle
from m6502 import _lib, inst

pytestmark = pytest.mark.gpu

P = inst.parse_assembly

# equal and unequal pairs, decided at nine input bits or fewer and beyond
PAIRS = [(P(t), P(c)) for t, c in [
    ("LDA #$05 : LDA #$07", "LDA #$07"), ("TAX : TXA", "TAX"), ("INX : DEX : INX", "INX"), ("ROL A : NOP", "ROL A"),
    ("ADC M", "ADC M"), ("INX : INY", "INX : INY"), ("TXA : TAY : LDA M : LDX #$01", "TXA : TAY : LDA M : LDX #$01"),
    ("INX : INY", "INX : DEY"), ("ADC M", "SBC M"), ("LDA #$05", "LDA #$06"), ("ASL A : ASL A", "ASL A"),
]]


@functools.lru_cache(maxsize=None)
def _want():
    return [oracle.exhaustive(t, c, 0, oracle.SWEEP_REFERENCE) for t, c in PAIRS]


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 147, 149, 443, 444, 445, 591, 593, 3551, 3553, 4735, 4737, 9475, 38001])
def test_counts(engine, n):
    want = _want()
    idx = [(i * 7 + i // 11) % len(PAIRS) for i in range(n)]
    got = engine.check_pairs([PAIRS[i][0] for i in idx], [PAIRS[i][1] for i in idx], 0, _lib.CHECK_EXH,
                             _lib.SWEEP_REFERENCE)
    assert [bool(o & 4) for o in got] == [want[i] for i in idx]


@pytest.mark.parametrize("n", [1, 9, 593, 4737, 9475])
def test_only_wide_pairs(engine, n):
    want = _want()
    wide = [i for i, (t, c) in enumerate(PAIRS) if 4 <= i <= 8]
    idx = [wide[i % len(wide)] for i in range(n)]
    got = engine.check_pairs([PAIRS[i][0] for i in idx], [PAIRS[i][1] for i in idx], 0, _lib.CHECK_EXH, _lib.SWEEP_FULL)
    assert [bool(o & 4) for o in got] == [want[i] for i in idx]
