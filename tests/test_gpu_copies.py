"""Inputs and results on their way: host targets copied pass by pass beside
the kernels, rules straight into the caller's buffer, pairs in one block each
way (page-locked up to 64 MiB, from the caller's arrays beyond)."""
import ctypes

import numpy as np
import pytest

import m6502
import oracle
from m6502 import _lib

pytestmark = pytest.mark.gpu

ORDER = ["target", "cand", "dead_flags"]


@pytest.mark.parametrize("semantics,cand", [(_lib.SEM_CUDA, 1), (_lib.SEM_GO, 1), (_lib.SEM_CUDA, 2)])
def test_many_passes_equal_one(engine, semantics, cand):
    t = np.asarray(oracle.draw_targets(9, 2, 2500), dtype=np.uint16)
    kw = dict(dead_flags=0x01, semantics=semantics, sweep=_lib.SWEEP_REFERENCE, max_cand_len=cand)
    want, ws = engine.search(t, **kw)
    small = m6502.Engine(targets_per_pass=600)
    try:
        for _ in range(2):   # recorded, then replayed
            got, st = small.search(t, **kw)
            assert st["passes"] == 5 and st["rules"] == len(got) == ws["rules"]
            assert np.array_equal(np.sort(got, order=ORDER), np.sort(want, order=ORDER))
        cut, _ = small.search(t, cap=len(want) // 2 + 1, **kw)   # the rest is staged and fetched
        assert np.array_equal(np.sort(cut, order=ORDER), np.sort(want, order=ORDER))
        for at in (0, 1300, 2499):   # an opcode outside the table, in any pass
            bad = t.copy()
            bad[at, 1] = 0x3A
            with pytest.raises(m6502.M6502Error):
                small.search(bad, **kw)
        again, _ = small.search(t, **kw)
        assert np.array_equal(np.sort(again, order=ORDER), np.sort(want, order=ORDER))
    finally:
        small.close()


@pytest.mark.parametrize("checks", [0, _lib.CHECK_QC, _lib.CHECK_MID, _lib.CHECK_EXH, _lib.CHECK_QC | _lib.CHECK_EXH, _lib.CHECK_ALL])
def test_pair_checks_one_by_one(engine, checks):
    tab = [int(x) for x in oracle.insn_table()]
    rng = np.random.default_rng(checks)
    ts = [[tab[k] for k in rng.integers(0, 2863, 2)] for _ in range(300)]
    cs = [[t[int(rng.integers(2))]] for t in ts]
    every, fd = engine.check_pairs(ts, cs, 0x01, _lib.CHECK_ALL, flagdiff=True)
    assert np.array_equal(engine.check_pairs(ts, cs, 0x01, checks), every & checks)
    some, fd2 = engine.check_pairs(ts, cs, 0x01, checks, flagdiff=True)
    assert np.array_equal(some, every & checks) and np.array_equal(fd, fd2)


def test_pairs_beyond_the_staging_buffer(engine):
    n, k = 4_900_000, 2863
    tab = oracle.insn_table().astype(np.uint16)
    t = np.resize(tab, n)
    c = np.resize(np.roll(tab, 1), n)
    c[::3] = t[::3]
    offs = np.arange(n + 1, dtype=np.uint32)
    out, fd = np.full(n, 0x55, dtype=np.uint8), np.full(n, 0x55, dtype=np.uint8)

    def check(m):
        p16, p32, p8 = ctypes.c_uint16, ctypes.c_uint32, ctypes.c_uint8
        rc = engine._L.m6502_check_pairs(engine._ctx, m, _lib.ptr(t, p16), _lib.ptr(offs, p32), _lib.ptr(c, p16),
                                         _lib.ptr(offs, p32), 0, _lib.CHECK_ALL, _lib.SWEEP_REFERENCE, _lib.EXH_CONES,
                                         _lib.ptr(out, p8), _lib.ptr(fd, p8))
        assert rc == _lib.M6502_OK
        return out[:m].copy(), fd[:m].copy()

    few = check(3 * k)      # the pairs repeat after 3 k
    many = check(n)
    for a, b in zip(few, many):
        assert np.array_equal(np.resize(a, n), b)
