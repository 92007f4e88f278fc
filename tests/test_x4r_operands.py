"""Words with an operand byte on an instruction that takes none (the C ABI and
Instruction(INX, 5) build them): every executor ignores the byte, the STOKE
chains' table-driven one too."""
import os
import subprocess

import pytest

import m6502
from conftest import PKG_DIR, ROOT
from m6502 import _lib


def test_table_driven_exec_ignores_unused_operand_bytes(tmp_path):
    exe = str(tmp_path / "x4r_operands")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "x4r_operands.cpp")], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("cost", [_lib.COST_REF, _lib.COST_HAMMING])
def test_stoke_ignores_unused_operand_bytes(engine, cost):
    """A chain's course is the one of the plain words; what it keeps of the
    target keeps its byte."""
    plain = [m6502.inst.parse_assembly(s) for s in ("LDA #$05 : TAX : INX : DEY : INC M", "TXA : TAX : INY : DEC M : DEX")]
    marked = [[w | (0x5A << 8) if not m6502.inst.imm_of(w) else w for w in t] for t in plain]
    runs = []
    for targets in (plain, marked):
        _, proofs, st = engine.stoke(targets, chains_per_target=16, steps=600, steps_per_epoch=200, seed=5, cost=cost)
        runs.append(([(p["target"], p["chain"], p["step"], tuple(w & 0xFF for w in p["cand"])) for p in proofs],
                     st["accepted"], st["candidates"]))
    assert runs[0][0] and runs[0] == runs[1]
