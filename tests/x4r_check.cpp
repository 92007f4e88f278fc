// Checks the table-driven executor (exec_x4r with the rows of x4_row) against
// exec_x4 for every instruction of the table, and against scalar exec calls
// for sequences, on seeded random states.  Built and run by tests/test_x4r.py.
#include <cstdio>
#include <cstdint>

#include "isa.cuh"

using namespace m6502;

static uint64_t rng = 0x6502;
static uint32_t next32() {
    uint64_t z = (rng += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (uint32_t)((z ^ (z >> 31)) >> 32);
}
constexpr int kStride = 3;   // slots apart, as lanes' are

static void put(uint32_t* st, const St& s) {
    const uint32_t f[7] = {s.a, s.x, s.y, s.s, s.m, s.s0, s.s1};
    for (int i = 0; i < 7; i++) st[i * kStride] = f[i];
}
static bool same(const uint32_t* st, uint32_t p, const St& s) {
    const uint32_t f[7] = {s.a, s.x, s.y, s.s, s.m, s.s0, s.s1};
    for (int i = 0; i < 7; i++)
        if (st[i * kStride] != f[i]) return false;
    return p == s.p;
}

int main() {
    long checked = 0, bad = 0;
    for (uint32_t op = 0; op < NUM_OPS; op++)
        for (uint32_t imm = 0; imm < (has_imm(op) ? 256u : 1u); imm++)
            for (int trial = 0; trial < 200; trial++) {
                St s{next32(), next32(), next32(), next32(), next32(), next32(), next32(), next32()};
                if (trial < 8) { s.a = 0x80FF0001u; s.m = 0x00FF8001u; s.x = 0; s.y = 0xFFFFFFFFu; }   // edges
                uint32_t st[X4S_COUNT * kStride] = {}, p = s.p;
                put(st, s);
                exec_x4r(st, kStride, p, x4_row(op), op | imm << 8);
                exec_x4(s, op | imm << 8);
                if (!same(st, p, s) && bad++ < 10) std::printf("op %u imm %u\n", op, imm);
                checked++;
            }
    for (int trial = 0; trial < 20000; trial++) {   // sequences of 16: what one instruction leaves, the next takes
        St s{next32(), next32(), next32(), next32(), next32(), next32(), next32(), next32()};
        uint32_t st[X4S_COUNT * kStride] = {}, p = s.p;
        put(st, s);
        for (int i = 0; i < 16; i++) {
            const uint32_t op = next32() % NUM_OPS, insn = op | (has_imm(op) ? (next32() & 0xFFu) << 8 : 0u);
            exec_x4r(st, kStride, p, x4_row(op), insn);
            exec_x4(s, insn);
        }
        if (!same(st, p, s) && bad++ < 10) std::printf("sequence %d\n", trial);
        checked++;
    }
    std::printf("checked %ld, %ld mismatches\n", checked, bad);
    return bad ? 1 : 0;
}
