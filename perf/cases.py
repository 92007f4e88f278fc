"""The work that users have this engine do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a program holds before the call, `run` is
one pass through the public entry points (the Python mirror, or the C ABI where a program holds
flat buffers).  Rules come back in no particular order, so a pass sorts them, as the rule tables
of the command line do, and pads them to a length that the case alone decides.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "6502-optimizer_b200"))

import m6502  # noqa: E402
from m6502 import _lib, inst  # noqa: E402

NI = 2863                       # instructions; candidates of length 1
MASKS = (0x00, 0x01, 0xC3, 0xFF)
# What m6502_autotune picks on a B200 for the full length-2 enumeration: a program that
# enumerates at length tunes its engine once and keeps it.
TUNED = {"exh_minb": 4, "ticket_batch": 8, "chunk_log2": 12, "join_probe": 0}


def listed():
    return [
        # A few rewrites checked one by one from a script (the Go verifier API): latency.
        {"name": "verify_48", "kind": "verify_list", "pairs": 48, "min_len": 2, "max_len": 4, "mask": 0x00},
        # A rule file re-checked (verify-jsonl): QuickCheck, MidCheck and ExhaustiveCheck of each line.
        {"name": "verify_20k", "kind": "verify", "pairs": 20011, "min_len": 2, "max_len": 4, "mask": 0x00},
        # `target "..."`: one sequence against all candidates of length 1 and 2, Go semantics.
        {"name": "target_one", "kind": "target", "calls": 1, "mask": 0x00},
        # A batch of length-2 targets (a compiler's peephole windows), CUDA semantics.
        {"name": "search_256", "kind": "search", "n": 256, "len": 2, "go": False, "cand": 1, "mask": 0x00},
        # Length-3 targets against every candidate of length 1 and 2, the four condition flags dead.
        {"name": "search_len3_4096", "kind": "search", "n": 4096, "len": 3, "go": True, "cand": 2, "mask": 0xC3},
        # All 7.6 million length-2 targets from host memory, the full sweep: the headline enumeration.
        {"name": "search_len2_all", "kind": "shard", "stride": 1, "mask": 0x00},
        # The Go tool's own run: length-2 enumeration, first rule per target in Go order, reduced sweep.
        {"name": "enumerate_len2_go", "kind": "enumerate", "len": 2, "width": 2800, "go": True, "mask": 0x00},
        # One first instruction's slice of the length-3 enumeration (the unit it is sharded by).
        {"name": "enumerate_len3_op", "kind": "enumerate", "len": 3, "width": 1, "go": False, "mask": 0x00},
        # Stage statistics with every flag dead: 480 million survivors, counted, not returned.
        {"name": "count_len2_ff", "kind": "count", "width": 2800, "mask": 0xFF},
        # STOKE over a batch of longer targets until each is proved or the steps run out.
        {"name": "stoke_256", "kind": "stoke", "targets": 256, "chains": 128, "steps": 4000, "cost": 1, "mask": 0x00},
        # The learned proposal scoring the moves it is validated on.
        {"name": "mlp_predict_4000", "kind": "predict", "n": 4000},
        # Loss and gradient of one batch: the forward and backward pass of training.
        {"name": "mlp_gradients_10k", "kind": "gradients", "n": 10007},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["verify_list", "verify", "target", "search", "search3", "shard", "enumerate", "enumerate3",
                       "count", "stoke", "predict", "gradients"])
    mask = rng.choice(MASKS + (rng.randrange(256) & 0xCF,))
    if kind == "verify_list":
        lo = rng.randint(1, 3)
        return {"kind": kind, "pairs": _log_int(rng, 16, 600), "min_len": lo + 1, "max_len": lo + rng.randint(1, 2), "mask": mask}
    if kind == "verify":
        lo = rng.randint(1, 3)
        return {"kind": kind, "pairs": _log_int(rng, 1000, 30000), "min_len": lo + 1, "max_len": lo + rng.randint(1, 2), "mask": mask}
    if kind == "target":
        return {"kind": kind, "calls": rng.randint(1, 12), "mask": rng.randrange(256) & 0xCF}
    if kind == "search":
        go = rng.random() < 0.5
        return {"kind": kind, "n": _log_int(rng, 1, 20000), "len": rng.choice([2, 3]), "go": go, "cand": 1, "mask": mask}
    if kind == "search3":
        return {"kind": "search", "n": _log_int(rng, 16, 4096), "len": 3, "go": True, "cand": 2, "mask": rng.choice((0x00, 0x01, 0xC3))}
    if kind == "shard":
        return {"kind": kind, "stride": _log_int(rng, 1, 64), "mask": 0x00}
    if kind == "enumerate":
        return {"kind": kind, "len": 2, "width": _log_int(rng, 4, 2800), "go": rng.random() < 0.5, "mask": rng.choice((0x00, 0x0C))}
    if kind == "enumerate3":
        return {"kind": "enumerate", "len": 3, "width": 1, "go": False, "mask": rng.choice((0x00, 0x04, 0x08))}
    if kind == "count":
        return {"kind": kind, "width": _log_int(rng, 40, 2800), "mask": rng.choice((0x01, 0x40, 0x83, 0xC3, 0xFF))}
    if kind == "stoke":
        return {"kind": kind, "targets": _log_int(rng, 1, 256), "chains": rng.choice([32, 64, 128]), "steps": rng.randint(500, 4000),
                "cost": rng.randrange(2), "mask": rng.choice((0x00, 0x01, 0xC3))}
    return {"kind": kind, "n": _log_int(rng, 128, 12000)}


# ---- what a program keeps: one engine, one tuned engine, one C handle, one model ----

@functools.lru_cache(maxsize=None)
def _tuned_engine():
    e = m6502.Engine()
    e.tune = TUNED
    return e


@functools.lru_cache(maxsize=None)
def _handle():
    """A context of the C ABI, as a host program written against it holds one."""
    ctx = ctypes.c_void_p()
    opts = _lib.Opts(0, 0, 0)
    rc = _lib.lib().m6502_create(ctypes.byref(ctx), ctypes.byref(opts))
    if rc:
        raise m6502.M6502Error(rc, "m6502_create")
    return ctx


SHAPES = [(314, 128), (8, 128), (314, 128), (16, 128), (512, 448), (1, 512), (512, 512), (1, 512), (512, 512), (1, 512),
          (384, 512), (1, 384)]     # E_T P_T E_C P_C W1 b1 W2 b2 W3 b3 W4 b4


@functools.lru_cache(maxsize=None)
def _weights():
    """The model's parameters: the spread of a trained proposal's, the same in every run."""
    rng = np.random.default_rng(6502)
    parts = []
    for i, (r, c) in enumerate(SHAPES):
        scale = 0.5 if i < 4 else 0.05 if r == 1 else math.sqrt(6.0 / c)
        parts.append(rng.uniform(-scale, scale, r * c))
    return np.concatenate(parts).astype(np.float32)


@functools.lru_cache(maxsize=None)
def _model():
    m = m6502.mlp.MLP(_tuned_engine())
    m.set_params(_weights())
    return m


# ---- inputs ----

@functools.lru_cache(maxsize=None)
def _table():
    return np.asarray(inst.insn_table(), dtype=np.uint16)


@functools.lru_cache(maxsize=None)
def _len2_targets():
    """Every pruned length-2 target in enumeration order."""
    L = _lib.lib()
    n = L.m6502_enumerate_targets(2, 0, NI, None, 0)
    out = np.empty((n, 2), dtype=np.uint16)
    L.m6502_enumerate_targets(2, 0, NI, _lib.ptr(out, ctypes.c_uint16), n)
    return out


def _op(name):
    return inst.OP_NAMES.index(name)


# Loads overwrite a register and N, Z without reading them, so an instruction that only
# touches those, put in front, is dead: (load, instructions that are dead before it).
def _dead_pairs():
    imm = {n: _op(n + "_IMM") for n in ("LDA", "LDX", "LDY")}
    return [(imm["LDA"], [imm["LDA"], _op("LDA_M"), _op("TXA"), _op("TYA")]),
            (imm["LDX"], [imm["LDX"], _op("LDX_M"), _op("TAX"), _op("INX"), _op("DEX")]),
            (imm["LDY"], [imm["LDY"], _op("LDY_M"), _op("TAY"), _op("INY"), _op("DEY")]),
            (_op("LDA_M"), [imm["LDA"], _op("TXA"), _op("TYA")])]


def _insn(rng, op):
    return op | (int(rng.integers(256)) << 8 if 26 <= op <= 36 else 0)


def _pairs(case, seed):
    """Targets and their proposed rewrites, one instruction shorter: half of them right (a dead
    instruction left out), half as a search proposes them (any one instruction left out)."""
    rng = np.random.default_rng(seed)
    tab, dead = _table(), _dead_pairs()
    ts, cs = [], []
    for _ in range(case["pairs"]):
        n = int(rng.integers(case["min_len"], case["max_len"] + 1))
        c = [int(x) for x in tab[rng.integers(0, NI, n - 1)]]
        if rng.random() < 0.5:
            load, befores = dead[int(rng.integers(len(dead)))]
            k = int(rng.integers(n - 1))
            c[k] = _insn(rng, load)
            t = c[:k] + [_insn(rng, befores[int(rng.integers(len(befores)))])] + c[k:]
        else:
            k = int(rng.integers(n))
            t = c[:k] + [int(tab[int(rng.integers(NI))])] + c[k:]
        ts.append(t)
        cs.append(c)
    return ts, cs


def _csr(seqs):
    offs = np.zeros(len(seqs) + 1, dtype=np.uint32)
    offs[1:] = np.cumsum([len(s) for s in seqs])
    return np.concatenate([np.asarray(s, dtype=np.uint16) for s in seqs]), offs


def _draw_targets(seed, lo, hi, n, prune):
    insns, offs = np.zeros(n * hi, dtype=np.uint16), np.zeros(n + 1, dtype=np.uint32)
    rc = _lib.lib().m6502_draw_targets(seed, lo, hi, n, int(prune), _lib.ptr(insns, ctypes.c_uint16),
                                       _lib.ptr(offs, ctypes.c_uint32))
    if rc:
        raise m6502.M6502Error(rc, "m6502_draw_targets")
    return insns[:int(offs[-1])].copy(), offs


def _examples(case, seed):
    """Moves of a search: a target, a candidate some edits away from it, the move that was taken."""
    rng = np.random.default_rng(seed)
    n, tab = case["n"], _table()
    arr = np.zeros(n, dtype=np.dtype([("target", "<u2", 8), ("cand", "<u2", 16), ("diff", "<u4"), ("tlen", "u1"), ("clen", "u1"),
                                      ("pos", "u1"), ("op", "u1"), ("imm", "u1"), ("weight", "u1"), ("reserved", "u1", 6)]))
    tlen = rng.integers(2, 9, n)
    t = tab[rng.integers(0, NI, (n, 8))]
    c = np.zeros((n, 16), dtype=np.uint16)
    c[:, :8] = t
    c[:, 8:10] = tab[rng.integers(0, NI, (n, 2))]
    edit = rng.random((n, 16)) < 0.25
    c = np.where(edit, tab[rng.integers(0, NI, (n, 16))], c)
    clen = np.clip(tlen + rng.integers(-1, 3, n), 1, 10)
    arr["target"] = np.where(np.arange(8) < tlen[:, None], t, 0)
    arr["cand"] = np.where(np.arange(16) < clen[:, None], c, 0)
    arr["diff"] = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    arr["tlen"], arr["clen"] = tlen, clen
    arr["pos"] = rng.integers(0, clen)
    move = tab[rng.integers(0, NI, n)]
    arr["op"], arr["imm"] = move & 0xFF, move >> 8
    arr["weight"] = 1
    return arr


def prepare(case, seed):
    s = dict(case)
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "verify_list":
        s["targets"], s["cands"] = _pairs(case, seed)
        s["engine"] = m6502.default_engine()
    elif kind == "verify":
        ts, cs = _pairs(case, seed)
        s["t"], s["c"] = _csr(ts), _csr(cs)
        s["out"], s["fd"] = np.zeros(len(ts), dtype=np.uint8), np.zeros(len(ts), dtype=np.uint8)
        s["ctx"] = _handle()
    elif kind == "target":   # constants folded: LDA #a : op #b : store or move
        s["seqs"] = []
        for _ in range(case["calls"]):
            op = _op(("AND_IMM", "ORA_IMM", "EOR_IMM")[int(rng.integers(3))])
            last = _op(("TAX", "TAY", "STA_M", "PHA")[int(rng.integers(4))])
            s["seqs"].append([_insn(rng, _op("LDA_IMM")), _insn(rng, op), last])
        s["engine"] = m6502.default_engine()
    elif kind == "search":
        insns, _ = _draw_targets(seed, case["len"], case["len"], case["n"], True)
        s["targets"] = insns.reshape(case["n"], case["len"])
        s["engine"] = m6502.default_engine()
    elif kind == "shard":    # a rank's strided share, from some place of the list on
        t = _len2_targets()
        s["targets"] = np.roll(t[seed % case["stride"]::case["stride"]], int(rng.integers(1, len(t))), axis=0)
        n = len(t) // case["stride"]      # the same for every seed
        s["targets"] = np.ascontiguousarray(s["targets"][:n])
        s["engine"] = _tuned_engine()
    elif kind in ("enumerate", "count"):
        s["first"] = int(rng.integers(0, NI - case["width"] + 1))
        s["engine"] = m6502.default_engine() if case.get("go") else _tuned_engine()
    elif kind == "stoke":
        s["insns"], s["offs"] = _draw_targets(seed, 4, 8, case["targets"], False)
        s["results"] = (_lib.StokeResult * case["targets"])()
        s["cap"] = case["targets"] * case["chains"] * 4 + 4096
        s["proofs"] = (_lib.StokeProof * s["cap"])()
        s["seed"] = int(seed) & 0x7FFFFFFF
        s["ctx"] = _handle()
    else:
        s["ex"] = _examples(case, seed)
        s["model"] = _model()
        s["probs"] = np.empty((case["n"], _lib.MLP_OUT), dtype=np.float32) if kind == "predict" else None
        s["grads"] = np.empty(s["model"].n_params, dtype=np.float32) if kind == "gradients" else None
    return s


# ---- one pass ----

def _sorted_rules(rules, rows):
    """The rule records (target, then candidate, length and dead flags in one word), sorted and
    padded with -1 to `rows`."""
    out = torch.full((rows, 2), -1, dtype=torch.int64, device="cuda")
    n = len(rules)
    if n > rows:
        raise ValueError("%d rules: more than the %d that fit" % (n, rows))
    if n:
        r = torch.from_numpy(np.ascontiguousarray(rules).view(np.int64).reshape(-1, 2)).cuda()
        cand = r[:, 1] & 0xFFFFFFF           # one instruction and most of the next: unique within a target
        order = torch.sort((r[:, 0] << 28) | cand).indices
        out[:n] = r[order]
    return out


def _rows(case):
    """How many rules a case can give at most, or a bound that real targets stay far below."""
    if case["kind"] == "shard":
        return 1200000 // case["stride"] + 4096
    if case["kind"] == "enumerate":
        if case["len"] == 3:
            return 12000000
        targets = case["width"] * NI
        return targets + 4096
    if case["go"]:
        return 2 * case["n"]
    return case["n"] * 160 + 4096


def _sequences(words, at):
    """Clears what lies past the end of each row's 16-instruction sequence (at word `at`, its
    length in the byte behind it): only the instructions it has are written."""
    words[:, at:at + 16] *= np.arange(16) < (words[:, at + 16] & 0xFF)[:, None]
    return words


def run(s):
    kind = s["kind"]
    L = _lib.lib()
    if kind == "verify_list":
        return s["engine"].check_pairs(s["targets"], s["cands"], dead_flags=s["mask"], flagdiff=True)
    if kind == "verify":
        (ti, to), (ci, co) = s["t"], s["c"]
        p16, p32, p8 = ctypes.c_uint16, ctypes.c_uint32, ctypes.c_uint8
        rc = L.m6502_check_pairs(s["ctx"], len(s["out"]), _lib.ptr(ti, p16), _lib.ptr(to, p32), _lib.ptr(ci, p16),
                                 _lib.ptr(co, p32), s["mask"], _lib.CHECK_ALL, _lib.SWEEP_REFERENCE, _lib.EXH_CONES,
                                 _lib.ptr(s["out"], p8), _lib.ptr(s["fd"], p8))
        if rc:
            raise m6502.M6502Error(rc, "m6502_check_pairs")
        return s["out"], s["fd"]
    if kind == "target":
        got = np.full((s["calls"], 7), -1, dtype=np.int64)
        for row, seq in zip(got, s["seqs"]):
            rule = m6502.SearchSingleMasked(seq, 2, s["mask"], engine=s["engine"])
            if rule is not None:
                row[:3] = rule.BytesSaved, rule.CyclesSaved, rule.DeadFlags
                row[3:3 + len(rule.Replacement)] = rule.Replacement
        return got
    if kind == "search":
        rules, _ = s["engine"].search(s["targets"], dead_flags=s["mask"], semantics=_lib.SEM_GO if s["go"] else _lib.SEM_CUDA,
                                      sweep=_lib.SWEEP_FULL, max_cand_len=s["cand"], cap=_rows(s))
        return _sorted_rules(rules, _rows(s))
    if kind == "shard":
        rules, _ = s["engine"].search(s["targets"], dead_flags=s["mask"])
        return _sorted_rules(rules, _rows(s))
    if kind == "enumerate":
        rules, _ = s["engine"].enumerate(s["len"], s["mask"], _lib.SEM_GO if s["go"] else _lib.SEM_CUDA,
                                         sweep=_lib.SWEEP_REFERENCE if s["go"] else _lib.SWEEP_FULL,
                                         first=s["first"], last=s["first"] + s["width"])
        return _sorted_rules(rules, _rows(s))
    if kind == "count":
        n, st = s["engine"].enumerate(2, s["mask"], first=s["first"], last=s["first"] + s["width"], count_only=True)
        return [n] + [st[k] for k in ("targets", "pairs", "qc_hits", "mid_hits", "exh_checked", "exh_passed", "rules",
                                      "exh_algo_ops", "exh_undecided")]
    if kind == "stoke":
        cfg = _lib.StokeCfg()
        cfg.chains_per_target, cfg.steps, cfg.steps_per_epoch, cfg.first_epoch = s["chains"], s["steps"], 2000, 64
        cfg.seed, cfg.cost, cfg.dead_flags = s["seed"], s["cost"], s["mask"]
        cfg.sweep, cfg.stop_on_proof = _lib.SWEEP_REFERENCE, 1
        n_out, st = ctypes.c_uint64(0), _lib.StokeStats()
        rc = L.m6502_stoke_run(s["ctx"], ctypes.byref(cfg), _lib.ptr(s["insns"], ctypes.c_uint16),
                               _lib.ptr(s["offs"], ctypes.c_uint32), s["targets"], s["results"], s["proofs"], s["cap"],
                               ctypes.byref(n_out), ctypes.byref(st))
        if rc:
            raise m6502.M6502Error(rc, "m6502_stoke_run")
        # everything but the times: what was proved, when in steps, by which chain, and the best rewrites
        n = int(n_out.value)
        res = _sequences(np.frombuffer(s["results"], dtype=np.uint16).reshape(-1, 32)[:, 4:].copy(), 8)
        prf = np.zeros((s["cap"], 32), dtype=np.uint16)
        prf[:n] = np.frombuffer(s["proofs"], dtype=np.uint16).reshape(-1, 32)[:n]
        prf[:n, 8:12] = 0
        _sequences(prf[:n], 12)
        return {"results": res, "proofs": prf, "n": n, "accepted": int(st.accepted), "candidates": int(st.candidates),
                "proven": int(st.targets_proven)}
    ex = s["ex"].ctypes.data_as(ctypes.POINTER(_lib.MlpExample))
    if kind == "predict":
        rc = L.m6502_mlp_predict(s["model"].handle, ex, len(s["ex"]), s["probs"].ctypes.data_as(ctypes.c_void_p))
        if rc:
            raise m6502.M6502Error(rc, "m6502_mlp_predict")
        return s["probs"]
    loss = ctypes.c_float(0)
    rc = L.m6502_mlp_gradients(s["model"].handle, ex, len(s["ex"]), ctypes.byref(loss), s["grads"].ctypes.data_as(ctypes.c_void_p))
    if rc:
        raise m6502.M6502Error(rc, "m6502_mlp_gradients")
    return {"loss": float(loss.value), "grads": _by_tensor(s["grads"])}


def _by_tensor(flat):
    out, o = [], 0
    for r, c in SHAPES:
        out.append(flat[o:o + r * c].reshape(r, c))
        o += r * c
    return out


# ---- the least work of a pass ----

# Executing one instruction on one state, by the fixed convention of the benchmark: 10 integer
# operations; comparing two states 3.
def work(case):
    kind = case["kind"]
    if kind in ("predict", "gradients"):
        n, dense = case["n"], 512 * (448 + 512 + 512 + 384)
        params = 4 * sum(r * c for r, c in SHAPES)
        if kind == "predict":
            return {"bytes": n * (64 + 4 * _lib.MLP_OUT) + params, "flops": 2 * n * dense}
        return {"bytes": n * 64 + 2 * params, "flops": 6 * n * dense}
    if kind in ("verify", "verify_list"):
        n, length = case["pairs"], case["min_len"] + case["max_len"] - 1
        return {"bytes": n * (2 * length + 8 + 2), "flops": n * (32 + 512) * (10 * length + 3)}
    if kind == "stoke":   # a step: a sequence of about six instructions on the 32 vectors; most targets fall early
        steps = case["targets"] * case["chains"] * case["steps"]
        return {"bytes": case["targets"] * (24 + 64 + 64 * 16), "flops": steps * 32 * 63 * 0.25}
    length = case.get("len", 2)
    if kind == "target":
        n, length, rules = case["calls"], 3, case["calls"]
    elif kind == "search":
        n, rules = case["n"], case["n"]
    elif kind == "shard":
        n = len(_len2_targets()) // case["stride"]
        rules = n // 7
    elif kind == "count":
        n, rules = case["width"] * 2666, 0
    else:
        n = case["width"] * (2666 if length == 2 else 2666 * 2666)
        rules = n // 7
    survivors = n * (0.7 if case["mask"] == 0 else 63 if case["mask"] == 0xFF else 4)
    if kind == "search" and case["cand"] == 2 or kind == "target":
        survivors += n * 100
    flops = n * 32 * 10 * length + survivors * 256 * (10 * (length + 1) + 3) / 4   # a quarter needs a byte-wide cone
    return {"bytes": n * length * 2 + rules * 16, "flops": flops}


# ---- what the numbers are in 64 bits ----

def _features64(ex, P, dev):
    """The network's input: summed embeddings of target and candidate, and the marks of where they differ."""
    n = len(ex)
    x = torch.zeros((n, 448), dtype=torch.float64, device=dev)
    t = torch.from_numpy(ex["target"].astype(np.int64)).to(dev)
    c = torch.from_numpy(ex["cand"].astype(np.int64)).to(dev)
    tl = torch.from_numpy(ex["tlen"].astype(np.int64)).to(dev)
    cl = torch.from_numpy(ex["clen"].astype(np.int64)).to(dev)

    def has_imm(op):
        return (op >= 26) & (op <= 36)

    for seq, ln, col, emb, pos in ((t, tl, 0, P[0], P[1]), (c, cl, 128, P[2], P[3])):
        for p in range(seq.shape[1]):
            live = (p < ln).double()[:, None]
            op, imm = seq[:, p] & 0xFF, seq[:, p] >> 8
            row = emb[op] + torch.where(has_imm(op)[:, None], emb[58 + imm], torch.zeros_like(emb[op])) + pos[p]
            x[:, col:col + 128] = x[:, col:col + 128] + live * row
    diff = torch.from_numpy(ex["diff"].astype(np.int64)).to(dev)
    with torch.no_grad():
        for b in range(32):
            x[:, 256 + b] = (diff >> b & 1).double()
        for p in range(16):
            x[:, 288 + p], x[:, 304 + p] = (tl == p).double(), (cl == p).double()
            tp = t[:, p] if p < 8 else torch.full_like(tl, -1)
            x[:, 320 + p] = ((p < cl) & (p < tl) & (c[:, p] != tp)).double()
            tn = t[:, p + 1] if p + 1 < 8 else torch.full_like(tl, -1)
            x[:, 336 + p] = ((p < cl) & (p + 1 < tl) & (c[:, p] == tn)).double()
            if p >= 1:
                tb = t[:, p - 1] if p - 1 < 8 else torch.full_like(tl, -1)
                x[:, 352 + p] = ((p < cl) & (p - 1 < tl) & (c[:, p] == tb)).double()
        away = torch.full_like(tl, -1)
        for p in reversed(range(8)):
            out = (p < tl) & ((p >= cl) | (c[:, p] != t[:, p]))
            away = torch.where(out, torch.full_like(away, t.new_tensor(p)), away)
        there = away >= 0
        first = t.gather(1, away.clamp(min=0)[:, None])[:, 0]
        op, imm = first & 0xFF, first >> 8
        for k in range(58):
            x[:, 368 + k] = (there & (op == k)).double()
        for b in range(8):
            x[:, 426 + b] = (there & has_imm(op) & ((imm >> b & 1) == 1)).double()
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("predict", "gradients"):
        return None          # verdicts, rules and counts are whole numbers
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ex = _examples(case, seed)
    flat = torch.from_numpy(_weights()).double().to(dev)
    P = [p.clone().requires_grad_(kind == "gradients") for p in _by_tensor(flat)]
    h = _features64(ex, P, dev)
    for k in (4, 6, 8):
        h = torch.relu(h @ P[k].T + P[k + 1])
    z = h @ P[10].T + P[11]
    heads = [torch.log_softmax(z[:, a:b], dim=1) for a, b in ((0, 16), (16, 74), (74, 330))]
    if kind == "predict":
        return torch.cat(heads, dim=1).exp()
    rows = torch.arange(len(ex), device=dev)
    pos, op, imm = (torch.from_numpy(ex[k].astype(np.int64)).to(dev) for k in ("pos", "op", "imm"))
    weight = torch.from_numpy(ex["weight"].astype(np.float64)).to(dev)
    each = -heads[0][rows, pos] - heads[1][rows, op] - torch.where((op >= 26) & (op <= 36), heads[2][rows, imm], 0.0 * heads[2][rows, imm])
    loss = (each * weight).sum() / weight.sum()
    grads = torch.autograd.grad(loss, P)
    return {"loss": float(loss.detach()), "grads": [g.detach() for g in grads]}
