"""Pairs decided a lane each (k_small): the compared outputs depend on nothing,
the carry, one register (eight bits, or five under the reduced sweep) or one
register and the carry.  Every register and both sides of the nine-bit line,
against the oracle's sweep of the whole domain; and the search's line filter
against brute force, which does without both."""
import numpy as np
import pytest

import m6502
import oracle
from m6502 import _lib, inst

pytestmark = pytest.mark.gpu

P = inst.parse_assembly

# (target, an equivalent candidate): what the outputs depend on in the comment
EQUAL = [
    ("LDA #$05 : LDA #$07", "LDA #$07"),                                  # nothing
    ("CLC : SEC", "SEC"),                                                 # nothing
    ("LDA #$00 : ROL A : LDA #$01", "LDA #$00 : ROL A : LDA #$01"),       # nothing that is compared but C
    ("LDA #$40 : ROL A", "LDA #$40 : ROL A"),                             # carry
    ("TAX : TXA", "TAX"), ("ASL A : ASL A", "ASL A : ASL A"),             # A
    ("INX : DEX : INX", "INX"), ("TXA : TAX", "TXA"),                     # X
    ("INY : INY : DEY", "INY"), ("TYA : TAY", "TYA"),                     # Y
    ("TSX : TXS", "TSX"),                                                 # S
    ("LDA M : STA M", "LDA M"), ("INC M : DEC M : INC M", "INC M"),   # M
    ("PLA : PLA : LDA #$01", "PLA : PLA : LDA #$01"),                     # S0, S1
    ("ROL A : NOP", "ROL A"), ("ADC #$13 : TAX", "ADC #$13 : TAX"),       # A and carry
    ("TXA : ROL A", "TXA : ROL A"), ("LDA M : ROR A", "LDA M : ROR A"),   # X / M and carry
    ("ADC M", "ADC M"), ("INX : INY", "INX : INY"),                   # beyond nine bits
    ("TXA : TAY : LDA M : LDX #$01", "TXA : TAY : LDA M : LDX #$01"),
]


def _variants():
    """Each equivalent pair, and the candidate with one operand or opcode off."""
    ts, cs = [], []
    tab = [int(x) for x in oracle.insn_table()]
    rng = np.random.default_rng(11)
    for t, c in EQUAL:
        t, c = P(t), P(c)
        ts.append(t)
        cs.append(c)
        for _ in range(6):
            d = list(c)
            k = int(rng.integers(len(d)))
            d[k] = d[k] ^ (1 << int(rng.integers(8, 16))) if 26 <= d[k] & 0xFF <= 36 else tab[int(rng.integers(len(tab)))]
            ts.append(t)
            cs.append(d)
    return ts, cs


@pytest.mark.parametrize("dead", [0x00, 0x01, 0x82, 0xFF])
def test_pairs_against_the_oracle(engine, dead):
    ts, cs = _variants()
    got = engine.check_pairs(ts, cs, dead, _lib.CHECK_EXH, _lib.SWEEP_REFERENCE)
    for t, c, o in zip(ts, cs, got):
        assert bool(o & 4) == oracle.exhaustive(t, c, dead, oracle.SWEEP_REFERENCE), (t, c, dead)
    pad = [P("CLD")[0]]   # the same pairs at the longest length, D cleared on both sides
    long_t, long_c = [t + pad * (16 - len(t)) for t in ts], [c + pad * (16 - len(c)) for c in cs]
    again = engine.check_pairs(long_t, long_c, dead, _lib.CHECK_EXH, _lib.SWEEP_REFERENCE)
    assert np.array_equal(again & 4, got & 4)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 4097])
def test_pair_counts_at_warp_and_block_edges(engine, n):
    ts, cs = _variants()
    want = engine.check_pairs(ts, cs, 0, _lib.CHECK_EXH) & 4
    k = np.arange(n) % len(ts)
    assert np.array_equal(engine.check_pairs([ts[i] for i in k], [cs[i] for i in k], 0, _lib.CHECK_EXH) & 4, want[k])


@pytest.mark.parametrize("dead", [0x00, 0x01, 0x40, 0x82, 0xCF])
def test_line_filter_against_brute_force(engine, dead):
    """Targets that read no, one, two and (reduced sweep) three extra registers."""
    t2 = np.asarray([[a, b] for a in range(0, 58, 1) for b in (3, 7, 11, 27 | 9 << 8, 34 | 64 << 8, 35 | 1 << 8, 38, 48, 56)
                     if a != 25 and not 26 <= a <= 36], dtype=np.uint16)
    rules, st = engine.search(t2, dead_flags=dead, sweep=_lib.SWEEP_REFERENCE, cap=1 << 20)
    brute, sb = engine.search(t2, dead_flags=dead, sweep=_lib.SWEEP_REFERENCE, cap=1 << 20, exh_mode=_lib.EXH_BRUTE)
    order = ["target", "cand"]
    assert np.array_equal(np.sort(rules, order=order), np.sort(brute, order=order))
    for k in ("qc_hits", "mid_hits", "exh_checked", "exh_passed", "exh_algo_ops"):
        assert st[k] == sb[k]
