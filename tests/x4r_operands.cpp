// An operand byte on an instruction that takes none changes nothing: the
// table-driven executor (exec_x4r) against exec_x4 for every opcode with every
// operand byte, and for sequences of such words.  Built and run by
// tests/test_x4r_operands.py.
#include <cstdio>
#include <cstdint>

#include "isa.cuh"

using namespace m6502;

static uint64_t rng = 0x0502;
static uint32_t next32() {
    uint64_t z = (rng += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (uint32_t)((z ^ (z >> 31)) >> 32);
}

// One run of `n` words by both executors from one random state.
static bool agree(const uint32_t* insn, int n) {
    St s{next32(), next32(), next32(), next32(), next32(), next32(), next32(), next32()};
    uint32_t st[X4S_COUNT] = {s.a, s.x, s.y, s.s, s.m, s.s0, s.s1}, p = s.p;
    for (int i = 0; i < n; i++) {
        exec_x4r(st, 1, p, x4_row(insn[i] & 0xFFu), insn[i]);
        exec_x4(s, insn[i]);
    }
    return st[X4S_A] == s.a && st[X4S_X] == s.x && st[X4S_Y] == s.y && st[X4S_S] == s.s && st[X4S_M] == s.m &&
           st[X4S_S0] == s.s0 && st[X4S_S1] == s.s1 && p == s.p;
}

int main() {
    long bad = 0;
    for (uint32_t op = 0; op < NUM_OPS; op++)
        for (uint32_t imm = 0; imm < 256; imm++)
            for (int trial = 0; trial < 20; trial++) {
                const uint32_t insn = op | imm << 8;
                if (!agree(&insn, 1) && bad++ < 10) std::printf("op %u operand byte %u\n", op, imm);
            }
    for (int trial = 0; trial < 20000; trial++) {
        uint32_t seq[16];
        for (uint32_t& w : seq) w = next32() % NUM_OPS | (next32() & 0xFFu) << 8;
        if (!agree(seq, 16) && bad++ < 10) std::printf("sequence %d\n", trial);
    }
    std::printf("%ld mismatches\n", bad);
    return bad ? 1 : 0;
}
