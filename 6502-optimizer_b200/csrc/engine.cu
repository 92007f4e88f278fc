// engine.cu -- B200 kernels and the C ABI of libm6502gpu.so.
//
// Pipeline of a search (all on one stream; a CUDA-semantics search with
// length-1 candidates queues every pass and syncs once at the end):
//
//   k_check_ops     every opcode of a pass's targets, before the rest of it.
//   k_qc_join       (default) lane per target: its 8 masked QC outputs are
//                   hashed and looked up among the candidates' distinct
//                   outputs (keys and bucket directory in shared memory);
//                   only a match runs the 24 MidCheck vectors.
//   k_fingerprint + k_qc1  (M6502_QC_SCAN) 32 packed output states per
//                   target, then a tile of 64 targets x all 2,863
//                   candidates per CTA with one masked 64-bit compare per
//                   pair; the same survivors as the join.
//   k_expand        matching targets x their candidates -> survivors; those
//                   that differ on the line states are rejected here.
//   k_small         lane per pair; decides the pairs whose outputs depend on
//                   at most nine input bits, lists the rest for k_exhaustive.
//   k_exhaustive    persistent; a warp takes one listed pair from a device
//                   ticket, derives the pair's swept input space (reference
//                   rule) and the input cone of every output location, and
//                   sweeps each maximal cone; large cones are probed in-warp
//                   and the rest is split into work items.
//   k_exh_items     persistent; warps drain the work-item queue; a failing
//                   item raises the pair's fail flag, which the others poll.
//   k_emit_*        passing pairs -> rules (CUDA semantics: all of them; Go
//                   semantics: first candidate in Go order per target).
#include <cuda_runtime.h>

#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>

#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <cctype>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "internal.h"
#include "isa.cuh"
#include "m6502.h"

using namespace m6502;

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kMaxSeq = 16;          // longest sequence the pairwise API takes
constexpr int kWarpsPerBlock = 8;    // 256-thread CTAs
constexpr uint64_t kSmallSweep = 1ull << 13;  // sweep in-warp up to this many states
constexpr uint64_t kProbe = 1ull << 12;       // in-warp probe of a large cone
constexpr uint64_t kChunk = 1ull << 11;       // states per work item (at least)
constexpr uint64_t kMaxItemsPerCone = 1ull << 16;   // larger cones get larger items
// Largest cone a pair may need swept (2^34 states, about 0.1 s of the whole
// GPU).  Pairs of long sequences that read many registers can need far
// more; they get the verdict "undecided" instead of an endless sweep.
constexpr uint32_t kMaxConeBits = 34;
constexpr unsigned kTicketBatch = 4;           // pairs a warp takes per ticket atomic
constexpr int kDirBits = 12;                   // key-bucket directory of the length-1 join (4,096 buckets)
constexpr size_t kPairsStaged = 64u << 20;     // m6502_check_pairs: page-locked staging, at most
constexpr int kMaxAsyncPasses = 64;            // passes of one search queued without a host round trip

// Test vectors: TestVectors + MidCheckVectors of pkg/search/verifier.go:18-67
// (A, X, Y, P, S, M, S0, S1).  Vectors 0..7 are QuickCheck's.
const uint8_t kVectors[32][8] = {
    {0x00, 0x00, 0x00, 0x00, 0xFD, 0x42, 0x00, 0x00}, {0xFF, 0xFF, 0xFF, 0xFF, 0xFF, 0xBD, 0xFF, 0xFF},
    {0x01, 0x02, 0x03, 0x00, 0xFD, 0x13, 0x10, 0x20}, {0x80, 0x40, 0x20, 0x01, 0xFC, 0x7E, 0x30, 0x40},
    {0x55, 0xAA, 0x55, 0x00, 0xFE, 0xA5, 0x55, 0xAA}, {0xAA, 0x55, 0xAA, 0x01, 0xFD, 0x5A, 0xAA, 0x55},
    {0x0F, 0xF0, 0x0F, 0x00, 0xFB, 0xE1, 0x0F, 0xF0}, {0x7F, 0x80, 0x7F, 0x01, 0xFD, 0x33, 0x80, 0x7F},
    {0x02, 0x01, 0x04, 0x00, 0xFD, 0x91, 0x11, 0x22}, {0x04, 0x08, 0x10, 0x01, 0xFD, 0x48, 0x33, 0x44},
    {0x08, 0x10, 0x20, 0x00, 0xFD, 0x24, 0x55, 0x66}, {0x10, 0x20, 0x40, 0x01, 0xFD, 0xD7, 0x77, 0x88},
    {0x20, 0x40, 0x80, 0x00, 0xFD, 0x6B, 0x99, 0xBB}, {0x40, 0x80, 0x01, 0x01, 0xFD, 0xB2, 0xCC, 0xDD},
    {0x03, 0x05, 0x09, 0x00, 0xFD, 0x0F, 0xEE, 0x11}, {0x05, 0x0A, 0x14, 0x01, 0xFD, 0xF0, 0x22, 0x33},
    {0xFE, 0x7F, 0x80, 0x00, 0xFD, 0x01, 0x44, 0x55}, {0x81, 0xFE, 0x01, 0x01, 0xFD, 0xFE, 0x66, 0x77},
    {0x7E, 0x81, 0x42, 0x00, 0xFD, 0x80, 0x88, 0x99}, {0xBF, 0x40, 0xBF, 0x01, 0xFD, 0x40, 0xAA, 0xBB},
    {0xC0, 0x3F, 0xC0, 0x00, 0xFD, 0x1F, 0xCC, 0xDD}, {0xE0, 0x1F, 0xE0, 0x01, 0xFD, 0xEF, 0xEE, 0x00},
    {0xF0, 0x0F, 0xF0, 0x00, 0xFD, 0x55, 0x11, 0x22}, {0x0E, 0xE0, 0x0E, 0x01, 0xFD, 0xAA, 0x33, 0x44},
    {0x11, 0x22, 0x33, 0x00, 0xFE, 0xC3, 0x00, 0x00}, {0x22, 0x33, 0x44, 0x01, 0xFF, 0x3C, 0x55, 0x66},
    {0x44, 0x55, 0x66, 0x00, 0xFC, 0x87, 0x77, 0x88}, {0x88, 0x99, 0xAA, 0x01, 0xFB, 0x69, 0x99, 0xAA},
    {0x33, 0x44, 0x55, 0x00, 0xFD, 0xAE, 0xBB, 0xCC}, {0xCC, 0xDD, 0xEE, 0x01, 0xFD, 0x51, 0xDD, 0xEE},
    {0x66, 0x77, 0x88, 0x00, 0xFD, 0xDA, 0x12, 0x34}, {0x99, 0xAA, 0xBB, 0x01, 0xFD, 0x25, 0x56, 0x78},
};

// Representative values of the reduced sweep (pkg/search/verifier.go:378-383).
const uint8_t kRepValues[32] = {
    0x00, 0x01, 0x02, 0x0F, 0x10, 0x1F, 0x20, 0x3F, 0x40, 0x55, 0x7E, 0x7F, 0x80, 0x81, 0xAA, 0xBF,
    0xC0, 0xD5, 0xE0, 0xEF, 0xF0, 0xF7, 0xFE, 0xFF, 0x03, 0x07, 0x11, 0x33, 0x77, 0xBB, 0xDD, 0xEE,
};

__constant__ uint64_t c_vec[32];             // packed test vectors
__constant__ uint32_t c_vec4[8][8];           // the same, vectors 4 g .. 4 g + 3 one per byte of each field (A X Y P S M S0 S1)
__constant__ uint32_t c_line[64][8];         // the 256 line states (see k_expand), four per word, by field
__constant__ uint16_t c_dep[NUM_OPS][NUM_LOCS];
__constant__ uint16_t c_wr[NUM_OPS];          // written locations per opcode
__constant__ uint16_t c_sweep[NUM_OPS];       // swept locations implied by opReads
__constant__ uint32_t c_x4d[NUM_OPS];         // packed-executor descriptors (x4_desc)
__constant__ uint16_t c_tab[kNumInsns];       // instructions, CUDA order
__constant__ uint16_t c_gotab[kNumInsns];     // instructions, Go order
__constant__ uint32_t c_gorank[kNumInsns];    // Go-order rank of CUDA index i
__constant__ uint16_t c_goidx[kNumInsns];     // CUDA index of Go rank r
__constant__ uint32_t c_rep[32];
__device__ uint4 g_dep16[NUM_OPS * 2];         // c_dep padded to 16 entries per opcode, for copies into shared memory
__device__ uint4 g_x4row[NUM_OPS * 3];        // X4Row by opcode (the STOKE chains' executor)

// Packed-executor descriptor of an instruction (an opcode outside the table
// runs as NOP, as exec leaves the state unchanged for it).
__device__ __forceinline__ uint32_t desc_x4(uint32_t insn) {
    const uint32_t op = insn & 0xFFu;
    return op < NUM_OPS ? c_x4d[op] : (uint32_t)X4_NOP;
}

// ---------------------------------------------------------------------------
// Host tables
// ---------------------------------------------------------------------------
void host_tables(uint16_t* cuda_tab, uint16_t* go_tab, uint32_t* gorank) {
    int k = 0;
    for (uint32_t op = 0; op < NUM_OPS; op++) {
        if (has_imm(op)) for (uint32_t v = 0; v < 256; v++) cuda_tab[k++] = (uint16_t)(op | (v << 8));
        else cuda_tab[k++] = (uint16_t)op;
    }
    k = 0;
    for (uint32_t op = 0; op < NUM_OPS; op++) if (!has_imm(op)) go_tab[k++] = (uint16_t)op;
    for (uint32_t op = 0; op < NUM_OPS; op++)
        if (has_imm(op)) for (uint32_t v = 0; v < 256; v++) go_tab[k++] = (uint16_t)(op | (v << 8));
    // rank of each CUDA-order instruction in Go order
    for (int i = 0; i < kNumInsns; i++) {
        uint32_t op = cuda_tab[i] & 0xFF, imm = cuda_tab[i] >> 8;
        uint32_t r;
        if (!has_imm(op)) {
            r = 0;
            for (uint32_t o = 0; o < op; o++) r += has_imm(o) ? 0 : 1;
        } else {
            r = 47;
            for (uint32_t o = 0; o < op; o++) r += has_imm(o) ? 256 : 0;
            r += imm;
        }
        gorank[i] = r;
    }
}

uint32_t sweep_locs_of_reads(uint32_t reads) {
    uint32_t l = 0;
    if (reads & R_X) l |= LB(L_X);
    if (reads & R_Y) l |= LB(L_Y);
    if (reads & R_M) l |= LB(L_M);
    if (reads & R_S) l |= LB(L_S);
    if (reads & R_S0) l |= LB(L_S0);
    if (reads & R_S1) l |= LB(L_S1);
    return l;
}

// ---------------------------------------------------------------------------
// Device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t fp_of(const St& s) {
    return pack(s) & ~((uint64_t)(~kPMask & 0xFFu) << 24);   // P & PMask
}

// Join key of a sequence: a 64-bit hash of its 8 QuickCheck outputs under
// the run's mask.  Pairs passing QuickCheck have equal keys; equal keys are
// re-checked vector by vector, so a hash collision costs only time.
__host__ __device__ __forceinline__ uint64_t key_mix(uint64_t z) {
    z ^= z >> 33; z *= 0xFF51AFD7ED558CCDull;
    z ^= z >> 33; z *= 0xC4CEB9FE1A85EC53ull;
    z ^= z >> 33;
    return z;
}
// key = mix(0x6502 ^ XOR over vectors v of mix(masked output v + (v + 1) * phi)):
// the per-vector terms are independent, so a warp computes them on 8 lanes at
// once and combines them with 3 shuffles.
__host__ __device__ __forceinline__ uint64_t key_term(uint64_t masked_out, int v) {
    return key_mix(masked_out + (uint64_t)(v + 1) * 0x9E3779B97F4A7C15ull);
}
__host__ __device__ __forceinline__ uint64_t key_final(uint64_t x) { return key_mix(x ^ 0x6502ull); }

// Key of the length-1 join: a hash of the 8 QuickCheck outputs as 16 packed
// words (fields A X Y P S M S0 S1 of vectors 0-3, then of vectors 4-7, one
// vector per byte; P masked), one 32 x 32 + 64 bit multiply-add per word.
__host__ __device__ __forceinline__ uint64_t join_key(const uint32_t (&w)[16]) {
    constexpr uint32_t kMul[16] = {0x9E3779B1u, 0x85EBCA77u, 0xC2B2AE3Du, 0x27D4EB2Fu, 0x165667B1u, 0xD3A2646Du,
                                   0xFD7046C5u, 0xB55A4F09u, 0x8DA6B343u, 0xD8163841u, 0xCB1AB31Fu, 0xA2C2A7D5u,
                                   0x91E10DA5u, 0xE7037ED1u, 0xF4914F6Du, 0xAF251AF3u};
    uint64_t h = 0x6502;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < 16; i++) h += (uint64_t)w[i] * kMul[i];
    h ^= h >> 29;
    h *= 0xFF51AFD7ED558CCDull;
    return h ^ (h >> 32);
}

// The length-1 join's table for one dead-flags mask.  The non-pruned
// candidates fall into classes of equal QuickCheck outputs (1,883 at mask
// 0x00) and those into subclasses of equal MidCheck outputs (2,032): a class
// is an entry, by the directory's buckets (two entries may share a key), and a target's
// outputs are compared once per class and subclass, not once per candidate
// (runs of up to 43 compare operands share a class).  `key` and `dir`, a
// directory of the keys' top bits, are copied into shared memory; the rest
// is read for the targets that match (15 %).
struct alignas(16) JoinTable {
    uint64_t key[kNumInsns + 1];
    uint16_t dir[(1u << kDirBits) + 8];    // first entry whose key's top kDirBits bits are >= b
    uint16_t sub[kNumInsns + 1];           // subclasses of entry u: sub[u] .. sub[u + 1]
    uint16_t start[kNumInsns + 1];         // candidates of subclass j: cand[start[j] .. start[j + 1])
    uint16_t cand[kNumInsns + 1];          // index | byte size << 12
    uint16_t weight[kNumInsns + 1][2];     // pairs (CandGroups) of entry u's candidates of 1 byte, of at most 2
};
constexpr size_t kJoinShared = offsetof(JoinTable, sub);
static_assert(kJoinShared % 16 == 0 && kNumInsns < (1 << 12), "copied in 16-byte words; 12-bit indices");

// Warp-collective key of the outputs held by lanes 0..7 (lane v: vector v).
__device__ __forceinline__ uint64_t warp_key(uint64_t tv, uint64_t mask, uint64_t salt, int lane) {
    uint64_t h = lane < 8 ? key_term((tv & mask) + salt, lane) : 0ull;
    h ^= __shfl_xor_sync(kFull, h, 1);
    h ^= __shfl_xor_sync(kFull, h, 2);
    h ^= __shfl_xor_sync(kFull, h, 4);
    return key_final(__shfl_sync(kFull, h, 0));
}

// First index of a sorted array with keys[i] >= key; the warp splits the
// range 33 ways per step (one load per lane).
__device__ __forceinline__ uint32_t warp_lower_bound(const uint64_t* __restrict__ keys, uint32_t n, uint64_t key,
                                                     int lane) {
    uint32_t lo = 0, hi = n;   // the answer lies in [lo, hi]
    while (hi - lo > 32) {
        const uint32_t piv = lo + (uint32_t)(((uint64_t)(hi - lo) * (uint64_t)(lane + 1)) / 33u);
        const unsigned less = __ballot_sync(kFull, keys[piv] < key);
        const int k = __popc(less);   // pivots ascend, so the lanes below k are exactly the ones below key
        const uint32_t plo = __shfl_sync(kFull, piv, k > 0 ? k - 1 : 0);
        const uint32_t phi = __shfl_sync(kFull, piv, k < 32 ? k : 31);
        const uint32_t nlo = k > 0 ? plo + 1 : lo;
        hi = k < 32 ? phi : hi;
        lo = nlo;
    }
    const uint32_t i = lo + (uint32_t)lane;
    return lo + (uint32_t)__popc(__ballot_sync(kFull, i < hi && keys[i] < key));
}

// Survivor record: target (index within the pass) and candidate code:
// bits 0..22 candidate index, bit 23 length-2 candidate, bit 24 Go masked
// pass (k_go_emit computes the winner's FlagDiff).
struct Surv {
    uint32_t t;
    uint32_t c;
};
constexpr uint32_t kSurvLen2 = 1u << 23, kSurvMasked = 1u << 24;
// target_id of a pair source whose pairs do not share targets.
constexpr uint64_t kNoTarget = ~0ull;

// fail[] of a pair: 0 passed, 3 undecided, 4 deferred (STOKE), kFailLine
// rejected by k_small's line states, anything else rejected.  The kernels that
// read the verdicts count the line states' rejects: a counter in k_small made
// its callers up to 1 % slower.
constexpr uint32_t kFailLine = 5u;

// Counters of one verification (k_small, k_exhaustive, k_exh_items over one
// list of pairs); zero at its start.
constexpr uint32_t kGoBlock = 64;    // survivors of a (target, pass) in the first Go-order round
struct VerifyCounters {
    unsigned long long n;            // pairs listed (Go-order rounds)
    unsigned long long exh_ticket, items, item_ticket, small_ticket, small_left;
};
constexpr int kMaxRounds = 8;        // Go-order rounds per phase: 64 x 8^r ordinals each, 19 M before the last

struct Counters {
    unsigned long long qc, mid;
    // restart with the length-2 phase
    unsigned long long surv, max_ord;      // max_ord: largest ordinal among the survivors (Go semantics)
    unsigned long long join_items;         // chunks of long length-2 equal ranges
    unsigned long long rules, exh_pass, states, algo, probe_rejects;
    unsigned long long undecided;          // pairs left undecided (a cone beyond the sweep cap)
    unsigned long long round_rejects;      // pairs of a first round that the line filter settled
    unsigned long long surv1;              // survivors of the length-1 phase
    unsigned long long join_ticket, matches;   // k_qc_join: claimed chunks of targets, matching targets
    VerifyCounters v[2][kMaxRounds];       // by phase and round (CUDA semantics: round 0)
};
constexpr int kPhaseCounters = 3;   // surv, max_ord, join_items

struct Item {   // one chunk of a large cone sweep
    uint32_t pair;
    uint16_t cone;
    uint8_t rep;
    uint8_t pad;
    uint64_t outmask;
    uint64_t start;
    uint64_t count;
};

// A pair as the exhaustive kernels see it, staged in shared memory.
struct PairView {
    const uint16_t* t;
    const uint16_t* c;
    int tn, cn;
    uint32_t dead;
};

// Groups of length-1 candidates that are the same function of the state on
// every output the run compares (CUDA semantics, per dead-flags mask): one
// member stands for all of them in the join's table and in every survivor
// record, and k_emit_all gives each passing record's rules member by member.
// At mask 0xFF the 600,000 targets that change no live output each match 779
// candidates that change none either (CMP, CPX and CPY with any operand, the
// flag instructions); they fall into 8 records instead, and the full length-2
// enumeration at that mask, which is bound by the records it verifies, takes
// 21.4 ms instead of 441 by this alone (482 M records before, 8 M now), 6.2 ms
// with the kernels that verify them.
struct CandGroups {
    uint16_t mult[kNumInsns];    // members of the group that candidate c stands for (0: another stands for c)
    uint16_t first[kNumInsns];   // index of its first member in `member`
    uint16_t member[kNumInsns];  // candidate indices, group by group
};

__device__ __forceinline__ uint32_t surv_weight(uint32_t code, const uint16_t* mult) {
    return mult && !(code & kSurvLen2) ? mult[code & 0x7FFFFFu] : 1u;
}

// Pair sources: survivors of the enumeration pipeline, or explicit CSR pairs.
struct SurvSource {
    static constexpr int kMaxT = 3, kMaxC = 2;   // longest target and candidate
    const Surv* surv;
    const uint16_t* targets;
    uint32_t tlen;
    uint32_t run_dead;
    int go;
    const uint16_t* mult;   // CandGroups::mult of the run's mask, or null: every record is one pair
    __device__ void load(uint64_t p, uint16_t* st, uint16_t* sc, int& tn, int& cn, uint32_t& dead,
                         int lane) const {
        Surv s = surv[p];
        tn = (int)tlen;
        if (lane < (int)tlen) st[lane] = targets[(uint64_t)s.t * tlen + lane];
        uint32_t idx = s.c & 0x7FFFFFu;
        if (s.c & kSurvLen2) {
            cn = 2;
            if (lane == 0) { sc[0] = c_tab[idx / kNumInsns]; sc[1] = c_tab[idx % kNumInsns]; }
        } else {
            cn = 1;
            if (lane == 0) sc[0] = c_tab[idx];
        }
        dead = go ? ((s.c & kSurvMasked) ? run_dead : 0u) : run_dead;
    }
    // Pair p into a lane's column of the staging array (instruction i at st[i * ld]).
    __device__ void load_lane(uint64_t p, uint16_t* st, uint16_t* sc, int ld, int& tn, int& cn, uint32_t& dead) const {
        const Surv s = surv[p];
        tn = (int)tlen;
        for (int i = 0; i < tn; i++) st[i * ld] = targets[(uint64_t)s.t * tlen + i];
        const uint32_t idx = s.c & 0x7FFFFFu;
        cn = (s.c & kSurvLen2) ? 2 : 1;
        sc[0] = c_tab[cn == 2 ? idx / kNumInsns : idx];
        if (cn == 2) sc[ld] = c_tab[idx % kNumInsns];
        dead = go && !(s.c & kSurvMasked) ? 0u : run_dead;
    }
    // Pairs with the same id share their target (the probe reuses its outputs).
    __device__ uint64_t target_id(uint64_t p) const { return surv[p].t; }
    // Pairs that record p stands for.
    __device__ uint32_t weight(uint64_t p) const { return surv_weight(surv[p].c, mult); }
};

struct CsrSource {
    static constexpr int kMaxT = kMaxSeq, kMaxC = kMaxSeq;
    const uint16_t* t_ins;
    const uint32_t* t_off;
    const uint16_t* c_ins;
    const uint32_t* c_off;
    uint32_t dead_;
    __device__ void load(uint64_t p, uint16_t* st, uint16_t* sc, int& tn, int& cn, uint32_t& dead,
                         int lane) const {
        uint32_t t0 = t_off[p], c0 = c_off[p];
        tn = (int)(t_off[p + 1] - t0);
        cn = (int)(c_off[p + 1] - c0);
        if (lane < tn) st[lane] = t_ins[t0 + lane];
        if (lane < cn) sc[lane] = c_ins[c0 + lane];
        dead = dead_;
    }
    __device__ void load_lane(uint64_t p, uint16_t* st, uint16_t* sc, int ld, int& tn, int& cn, uint32_t& dead) const {
        const uint32_t t0 = t_off[p], c0 = c_off[p];
        tn = (int)(t_off[p + 1] - t0);
        cn = (int)(c_off[p + 1] - c0);
        for (int i = 0; i < tn; i++) st[i * ld] = t_ins[t0 + i];
        for (int i = 0; i < cn; i++) sc[i * ld] = c_ins[c0 + i];
        dead = dead_;
    }
    __device__ uint64_t target_id(uint64_t) const { return kNoTarget; }
    __device__ uint32_t weight(uint64_t) const { return 1u; }
};

// Decode parameters of one cone sweep.  State index bits: A (8, if in the
// cone), carry (1), then each swept extra register in the cone (8 bits, or 5
// bits indexing the representative values).
struct Fields {
    uint32_t sh[8], mk[8], base[8];   // order: A, X, Y, S, M, S0, S1, carry
    uint32_t rep_mask;                // fields translated through c_rep
    uint32_t bits;
    int low;                          // the field at bit 0 if it is at least 2 bits wide, else -1
    uint32_t low_mk;                  // its mask (its values are state & low_mk)
};

__device__ __forceinline__ Fields make_fields(uint32_t cone, uint32_t swept, bool rep) {
    Fields f;
    uint32_t bit = 0;
    const uint32_t locs[8] = {L_A, L_X, L_Y, L_S, L_M, L_S0, L_S1, L_C};
    f.rep_mask = 0;
    f.low = -1;
    f.low_mk = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint32_t l = locs[i];
        f.sh[i] = 0; f.mk[i] = 0;
        f.base[i] = (l == L_S && !(swept & LB(L_S))) ? 0xFDu : 0u;
        if (cone & LB(l)) {
            uint32_t w = (l == L_C) ? 1u : ((rep && l != L_A) ? 5u : 8u);
            if (bit == 0) { f.low = w >= 2 ? i : -1; f.low_mk = (1u << w) - 1u; }
            f.sh[i] = bit; f.mk[i] = (1u << w) - 1u; f.base[i] = 0;
            if (rep && l != L_A && l != L_C) f.rep_mask |= 1u << i;
            bit += w;
        }
    }
    f.bits = bit;
    return f;
}

__device__ __forceinline__ uint32_t fld(const Fields& f, int i, uint64_t s) {
    uint32_t v = (uint32_t)(s >> f.sh[i]) & f.mk[i];
    if (f.rep_mask & (1u << i)) v = c_rep[v];
    return v | f.base[i];
}

// Per-byte compare masks of a packed output mask.
struct OutMask {
    uint32_t a, x, y, p, s, m, s0, s1;
};
__device__ __forceinline__ OutMask out_mask(uint64_t om) {
    return OutMask{(uint32_t)om & 0xFFu,         (uint32_t)(om >> 8) & 0xFFu,  (uint32_t)(om >> 16) & 0xFFu,
                   (uint32_t)(om >> 24) & 0xFFu, (uint32_t)(om >> 32) & 0xFFu, (uint32_t)(om >> 40) & 0xFFu,
                   (uint32_t)(om >> 48) & 0xFFu, (uint32_t)(om >> 56) & 0xFFu};
}

// Nonzero when target and candidate disagree on a compared output from
// the input state with index s.
__device__ __forceinline__ St decode_state(const Fields& f, uint64_t s) {
    St in;
    in.a = fld(f, 0, s); in.x = fld(f, 1, s); in.y = fld(f, 2, s); in.s = fld(f, 3, s);
    in.m = fld(f, 4, s); in.s0 = fld(f, 5, s); in.s1 = fld(f, 6, s); in.p = fld(f, 7, s);
    return in;
}

__device__ __forceinline__ uint32_t out_diff(const St& t, const St& c, const OutMask& m) {
    return ((t.a ^ c.a) & m.a) | ((t.x ^ c.x) & m.x) | ((t.y ^ c.y) & m.y) | ((t.p ^ c.p) & m.p) |
           ((t.s ^ c.s) & m.s) | ((t.m ^ c.m) & m.m) | ((t.s0 ^ c.s0) & m.s0) | ((t.s1 ^ c.s1) & m.s1);
}

// Target and candidate on one state: one loop over target then candidate (a
// single inlined copy of the opcode switch per call site keeps the code, and
// instruction-cache misses, small).
__device__ __forceinline__ uint32_t state_diff_in(const PairView& pv, const OutMask& m, const St& in) {
    St c = in, t = in;
    const int n = pv.tn + pv.cn;
    for (int i = 0; i < n; i++) {
        if (i == pv.tn) { t = c; c = in; }
        exec(c, i < pv.tn ? pv.t[i] : pv.c[i - pv.tn]);
    }
    if (pv.cn == 0) { t = c; c = in; }
    return out_diff(t, c, m);
}
__device__ __forceinline__ uint32_t state_diff(const PairView& pv, const Fields& f, const OutMask& m, uint64_t s) {
    return state_diff_in(pv, m, decode_state(f, s));
}

// One uniformly random state of a pair's whole sweep domain, from 64 random
// bits: every swept register takes its own byte of z (its representative
// value, c_rep[byte & 31], under the reduced sweep, A excepted), the carry
// bit 63; the others hold the sweep's fixed values (S = 0xFD, the rest 0,
// the other flags clear) -- the same domain make_fields(swept, swept, rep)
// enumerates, drawn without packing a state index.
__device__ __forceinline__ St probe_state(uint32_t swept, bool rep, uint64_t z) {
    const uint32_t lo = (uint32_t)z, hi = (uint32_t)(z >> 32);
    auto reg = [&](uint32_t loc, uint32_t byte, uint32_t fixed) -> uint32_t {
        if (!(swept & LB(loc))) return fixed;
        return rep ? c_rep[byte & 31u] : byte;
    };
    St in;
    in.a = lo & 0xFFu;
    in.x = reg(L_X, (lo >> 8) & 0xFFu, 0u);
    in.y = reg(L_Y, (lo >> 16) & 0xFFu, 0u);
    in.s = reg(L_S, lo >> 24, 0xFDu);
    in.m = reg(L_M, hi & 0xFFu, 0u);
    in.s0 = reg(L_S0, (hi >> 8) & 0xFFu, 0u);
    in.s1 = reg(L_S1, (hi >> 16) & 0xFFu, 0u);
    in.p = hi >> 31;
    return in;
}

// The i-th random word of a probe with the given salt (splitmix64 output
// mixing of salt + i * golden ratio).
__device__ __forceinline__ uint64_t probe_z(uint64_t salt, int i) {
    uint64_t z = salt + (uint64_t)i * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Per-warp memory of the target last probed and composed, in shared memory
// so that nothing of it stays in registers across the pair loop.  The probe
// states are stored field-major (field f of lane l at [f][l]): one
// conflict-free 32-bit access per field.
struct TargetCache {
    uint64_t probe_id;        // target whose probe states `in4` / `out4` hold (kNoTarget: none)
    uint64_t flow_id;         // target whose composition `dt` / wt / st hold
    uint32_t in4[8][32];      // per lane: four probe input states packed one per byte
    uint32_t out4[8][32];     // per lane: the target's outputs on them, packed the same way
    uint32_t dt[32];          // per lane: the target's composed dependencies
    uint32_t wt, st;          // locations the target writes / sweeps
};

__device__ __forceinline__ St st_load(const uint32_t (*a)[32], int lane) {
    St s;
    s.a = a[0][lane]; s.x = a[1][lane]; s.y = a[2][lane]; s.p = a[3][lane];
    s.s = a[4][lane]; s.m = a[5][lane]; s.s0 = a[6][lane]; s.s1 = a[7][lane];
    return s;
}
__device__ __forceinline__ void st_store(uint32_t (*a)[32], int lane, const St& s) {
    a[0][lane] = s.a; a[1][lane] = s.x; a[2][lane] = s.y; a[3][lane] = s.p;
    a[4][lane] = s.s; a[5][lane] = s.m; a[6][lane] = s.s0; a[7][lane] = s.s1;
}

// 128 random states of a pair's sweep domain, four per lane packed one per
// byte (state k in byte k of every field; see exec_x4).  Under the full
// sweep every packed field of a swept register is 32 random bits (four
// independent uniform bytes), the carry one random bit per byte, and the
// other fields hold the sweep's fixed values (S = 0xFD, the rest 0, the
// other flags clear): four splitmix64 words per lane.  Under the reduced
// sweep each byte of an extra register is a representative value
// (c_rep[byte & 31]), drawn state by state through probe_state.
__device__ __forceinline__ St probe_state_x4(uint32_t swept, bool rep, uint64_t salt, int lane) {
    St o{0, 0, 0, 0, 0, 0, 0, 0};
    if (rep) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const St s = probe_state(swept, true, probe_z(salt, lane + 32 * k));
            const int sh = 8 * k;
            o.a |= s.a << sh; o.x |= s.x << sh; o.y |= s.y << sh; o.p |= s.p << sh;
            o.s |= s.s << sh; o.m |= s.m << sh; o.s0 |= s.s0 << sh; o.s1 |= s.s1 << sh;
        }
        return o;
    }
    const uint64_t z0 = probe_z(salt, lane), z1 = probe_z(salt, lane + 32), z2 = probe_z(salt, lane + 64),
                   z3 = probe_z(salt, lane + 96);
    o.a = (uint32_t)z0;
    o.x = (swept & LB(L_X)) ? (uint32_t)(z0 >> 32) : 0u;
    o.y = (swept & LB(L_Y)) ? (uint32_t)z1 : 0u;
    o.s = (swept & LB(L_S)) ? (uint32_t)(z1 >> 32) : 0xFDu * kB1;
    o.m = (swept & LB(L_M)) ? (uint32_t)z2 : 0u;
    o.s0 = (swept & LB(L_S0)) ? (uint32_t)(z2 >> 32) : 0u;
    o.s1 = (swept & LB(L_S1)) ? (uint32_t)z3 : 0u;
    o.p = (uint32_t)(z3 >> 32) & kB1;
    return o;
}

// The probe of one pair: 128 pseudo-random states of its whole sweep domain,
// four per lane packed one per byte (one exec_x4 dispatch per instruction
// for four states), drawn from the target's salt when the source says which
// pairs share a target (`tid`), else from the pair's.  When the pair's
// domain is the target's own (the candidate reads no other register) the
// packed input states and the target's outputs on them are kept in the
// warp's cache; a later pair of the same target then loads its inputs and
// runs only its candidate.  One exec site.  False when a state differs.
__device__ __forceinline__ bool probe_pair(const PairView& pv, uint32_t sw_t, uint32_t sw_c, bool rep, uint64_t tid,
                                           uint64_t p, TargetCache& tc, int lane) {
    const uint64_t salt = tid != kNoTarget ? tid * 0xD1B54A32D192ED03ull + 0x632BE59BD9B4E019ull : p;
    const bool same = tid != kNoTarget && (sw_c & ~sw_t) == 0;   // uniform
    const bool hit = same && tc.probe_id == tid;                  // uniform
    const uint32_t swu = sw_t | sw_c | LB(L_A) | LB(L_C);
    const int n = pv.tn + pv.cn;
    const St in = hit ? st_load(tc.in4, lane) : probe_state_x4(swu, rep, salt, lane);
    St ps = in, ts = in;
    for (int i = hit ? pv.tn : 0; i < n; i++) {
        if (i == pv.tn && !hit) { ts = ps; ps = in; }   // the target is done: the candidate starts
        const uint32_t insn = i < pv.tn ? pv.t[i] : pv.c[i - pv.tn];
        exec_x4d(ps, insn, desc_x4(insn));
    }
    if (pv.cn == 0 && !hit) { ts = ps; ps = in; }
    if (hit) ts = st_load(tc.out4, lane);
    if (same && !hit) {   // every lane read probe_id above, before this sync
        st_store(tc.in4, lane, in);
        st_store(tc.out4, lane, ts);
        __syncwarp();
        if (lane == 0) tc.probe_id = tid;
        __syncwarp();
    }
    OutMask m = out_mask(cmp_mask(pv.dead));
    m.a *= kB1; m.x *= kB1; m.y *= kB1; m.p *= kB1; m.s *= kB1; m.m *= kB1; m.s0 *= kB1; m.s1 *= kB1;
    return !__any_sync(kFull, out_diff(ts, ps, m) != 0);
}

// Four consecutive states s..s+3 (s a multiple of 4) packed one per byte
// (see exec_x4).  They differ only in the low two bits of the lowest field,
// so one scalar decode plus that field's four values builds them.
__device__ __forceinline__ St decode_x4(const Fields& f, uint64_t s) {
    const St in = decode_state(f, s);
    St o;
    o.a = in.a * kB1; o.x = in.x * kB1; o.y = in.y * kB1; o.s = in.s * kB1;
    o.m = in.m * kB1; o.s0 = in.s0 * kB1; o.s1 = in.s1 * kB1; o.p = in.p * kB1;
    uint32_t low;
    const uint32_t i0 = (uint32_t)s & f.low_mk;   // the lowest field starts at bit 0 and has base 0
    if (f.rep_mask & (1u << f.low))
        low = c_rep[i0] | (c_rep[i0 + 1] << 8) | (c_rep[i0 + 2] << 16) | (c_rep[i0 + 3] << 24);
    else
        low = i0 * kB1 + 0x03020100u;
    switch (f.low) {   // warp-uniform
    case 0: o.a = low; break;
    case 1: o.x = low; break;
    case 2: o.y = low; break;
    case 3: o.s = low; break;
    case 4: o.m = low; break;
    case 5: o.s0 = low; break;
    default: o.s1 = low; break;
    }
    return o;
}

__device__ __forceinline__ uint32_t state_diff_x4(const PairView& pv, const Fields& f, const OutMask& m4, uint64_t s) {
    St c = decode_x4(f, s), t = c;
    const int n = pv.tn + pv.cn;
    for (int i = 0; i < n; i++) {
        if (i == pv.tn) { t = c; c = decode_x4(f, s); }
        exec_x4(c, i < pv.tn ? pv.t[i] : pv.c[i - pv.tn]);
    }
    if (pv.cn == 0) { t = c; c = decode_x4(f, s); }
    return out_diff(t, c, m4);
}

// Sweeps states [s0, s1) of one cone; true when target and candidate agree
// on the compared outputs in every state.  Warp-collective.  When `stop`
// becomes nonzero (another item of the same pair failed) the sweep ends
// early; its result is then irrelevant.
// PER_LANE = 4: four consecutive states per lane packed one per byte
// (exec_x4: one dispatch, byte-parallel arithmetic); 1: one.  The packed path
// needs 4-aligned ranges and a lowest field of at least 2 bits, and falls
// back to one state per lane.
template <int PER_LANE>
__device__ __forceinline__ bool sweep_states(const PairView& pv, const Fields& f, uint64_t om, uint64_t s0,
                                             uint64_t s1, const volatile uint32_t* stop, unsigned long long* nstates,
                                             int lane) {
    if (PER_LANE == 4 && (f.low < 0 || (s0 & 3) || (s1 & 3)))   // packed sweep needs 4-aligned runs
        return sweep_states<1>(pv, f, om, s0, s1, stop, nstates, lane);
    OutMask m = out_mask(om);
    if (PER_LANE == 4) {
        m.a *= kB1; m.x *= kB1; m.y *= kB1; m.p *= kB1; m.s *= kB1; m.m *= kB1; m.s0 *= kB1; m.s1 *= kB1;
    }
    uint64_t iter = 0;
    constexpr uint64_t kStep = 32 * PER_LANE;
    for (uint64_t b = s0; b < s1; b += kStep, iter++) {
        const uint64_t s = b + PER_LANE * (uint64_t)lane;
        uint32_t d = 0;
        if (s < s1) d = PER_LANE == 4 ? state_diff_x4(pv, f, m, s) : state_diff(pv, f, m, s);
        if (__any_sync(kFull, d != 0)) {
            if (lane == 0) *nstates += min((b - s0) + kStep, s1 - s0);
            return false;
        }
        if ((iter & (255 / PER_LANE)) == (255 / PER_LANE) && stop) {
            uint32_t sv = lane == 0 ? *stop : 0u;   // one read, broadcast: keeps the warp uniform
            if (__shfl_sync(kFull, sv, 0)) break;
        }
    }
    if (lane == 0) *nstates += s1 - s0;
    return true;
}
__device__ __noinline__ bool sweep_general(const PairView& pv, uint32_t cone, uint32_t swept, bool rep, uint64_t om,
                                           uint64_t s0, uint64_t s1, const volatile uint32_t* stop,
                                           unsigned long long* nstates, int lane) {
    return sweep_states<4>(pv, make_fields(cone, swept, rep), om, s0, s1, stop, nstates, lane);
}

// A row's state: the values of the locations of `high` from its index `bits`,
// the same in every byte; the others at the first value of their range.
__device__ __forceinline__ St row_state(uint32_t bits, uint32_t high, uint32_t bs, bool rep) {
    auto field = [&](uint32_t l, uint32_t fixed) -> uint32_t {
        if (!(high & LB(l))) return fixed * kB1;
        const uint32_t w = rep ? 5u : 8u, x = bits & ((1u << w) - 1u);
        bits >>= w;
        return (rep ? c_rep[x] : x) * kB1;
    };
    St in;
    in.a = 0;
    in.x = field(L_X, 0); in.y = field(L_Y, 0); in.s = field(L_S, bs); in.m = field(L_M, 0);
    in.s0 = field(L_S0, 0); in.s1 = field(L_S1, 0);
    in.p = (high & LB(L_C)) ? (bits & 1u) * kB1 : 0u;
    return in;
}
__device__ __forceinline__ void put_reg(St& s, uint32_t loc, uint32_t v) {
    if (loc == LB(L_A)) s.a = v;
    else if (loc == LB(L_X)) s.x = v;
    else if (loc == LB(L_Y)) s.y = v;
    else if (loc == LB(L_S)) s.s = v;
    else if (loc == LB(L_M)) s.m = v;
    else if (loc == LB(L_S0)) s.s0 = v;
    else s.s1 = v;
}
__device__ __forceinline__ OutMask out_mask4(uint64_t om) {
    OutMask m = out_mask(om);
    m.a *= kB1; m.x *= kB1; m.y *= kB1; m.p *= kB1; m.s *= kB1; m.m *= kB1; m.s0 *= kB1; m.s1 *= kB1;
    return m;
}
// Target and candidate on two packed words: nonzero where they differ.
__device__ __forceinline__ uint32_t words_differ(const PairView& pv, const St (&in)[2], const OutMask& m) {
    St t[2] = {in[0], in[1]}, c[2] = {in[0], in[1]};
    for (int i = 0; i < pv.tn; i++) exec_x4n(t, pv.t[i]);
    for (int i = 0; i < pv.cn; i++) exec_x4n(c, pv.c[i]);
    return out_diff(t[0], c[0], m) | out_diff(t[1], c[1], m);
}

// The reduced sweep of a cone without A: its registers have 32 values each (8
// words).  Rows are the 1,024 states of the two lowest, in 4 steps of two
// words; lane l holds the lowest one's word l % 8 for good and takes values
// l / 8 + 4 j of the next.  Where the general sweep takes its place k_exhaustive
// needs 1.8 ms for a STOKE run's proofs (256 targets of 4 to 8 instructions)
// instead of 0.7.
__device__ __noinline__ bool sweep_narrow(const PairView& pv, uint32_t cone, uint32_t low, uint32_t next, uint32_t bs,
                                          uint64_t om, uint64_t s0, uint64_t s1, const volatile uint32_t* stop,
                                          unsigned long long* nstates, int lane) {
    const uint32_t i0 = 4u * ((uint32_t)lane & 7u);
    const uint32_t v = c_rep[i0] | (c_rep[i0 + 1] << 8) | (c_rep[i0 + 2] << 16) | (c_rep[i0 + 3] << 24);
    const OutMask m = out_mask4(om);
    const uint32_t q1 = (uint32_t)(s1 >> 8);
    for (uint32_t q = (uint32_t)(s0 >> 8); q < q1; q++) {   // steps of 256 states
        const St row = row_state(q >> 2, cone & ~(low | next), bs, true);
        St in[2] = {row, row};
#pragma unroll
        for (int k = 0; k < 2; k++) {
            put_reg(in[k], low, v);
            put_reg(in[k], next, c_rep[((uint32_t)lane >> 3) + 4u * (2u * (q & 3u) + (uint32_t)k)] * kB1);
        }
        if (__any_sync(kFull, words_differ(pv, in, m) != 0)) {
            if (lane == 0) *nstates += ((uint64_t)(q + 1) << 8) - s0;
            return false;
        }
        if ((q & 31) == 31 && stop) {
            const uint32_t sv = lane == 0 ? *stop : 0u;   // one read, broadcast: keeps the warp uniform
            if (__shfl_sync(kFull, sv, 0)) break;
        }
    }
    if (lane == 0) *nstates += s1 - s0;
    return true;
}

// The same sweep by rows of 256 states when the cone's lowest field is a
// whole register (A, or any register under the full sweep) and the range is
// made of rows.  Lane l holds values 4 l .. 4 l + 3 and 4 l + 128 .. of that
// register in two packed words for good; a row sets the other fields, the
// same in every lane, and runs both words with one dispatch per instruction.
// The general sweep decodes 8 fields with 64-bit shifts for every word and
// sequence: 300 warp instructions per word, against 85 here (the work items
// of the full length-2 enumeration: 0.60 -> 0.28 ms).
__device__ __forceinline__ bool sweep_cone(const PairView& pv, uint32_t cone, uint32_t swept, bool rep, uint64_t om,
                                           uint64_t s0, uint64_t s1, const volatile uint32_t* stop,
                                           unsigned long long* nstates, int lane) {
    const uint32_t regs = cone & ~LB(L_C);
    const uint32_t low = (cone & LB(L_A)) ? LB(L_A) : (regs & (0u - regs));   // A first, then X Y S M S0 S1
    const uint32_t bs = (swept & LB(L_S)) ? 0u : 0xFDu;   // S outside the cone: its first value
    if (low == 0 || (rep && low != LB(L_A)) || ((s0 | s1) & 255)) {
        const uint32_t rest = regs & ~low, next = rest & (0u - rest);
        if (next && !((s0 | s1) & 1023)) return sweep_narrow(pv, cone, low, next, bs, om, s0, s1, stop, nstates, lane);
        return sweep_general(pv, cone, swept, rep, om, s0, s1, stop, nstates, lane);
    }
    const uint32_t high = cone & ~low;
    const uint32_t v0 = 4u * (uint32_t)lane * kB1 + 0x03020100u, v1 = v0 + 0x80808080u;
    const OutMask m = out_mask4(om);
    const uint32_t r1 = (uint32_t)(s1 >> 8);
    for (uint32_t row = (uint32_t)(s0 >> 8); row < r1; row++) {
        const St at = row_state(row, high, bs, rep);
        St in[2] = {at, at};
        put_reg(in[0], low, v0);
        put_reg(in[1], low, v1);
        if (__any_sync(kFull, words_differ(pv, in, m) != 0)) {
            if (lane == 0) *nstates += ((uint64_t)(row + 1) << 8) - s0;
            return false;
        }
        if ((row & 31) == 31 && stop) {
            const uint32_t sv = lane == 0 ? *stop : 0u;   // one read, broadcast: keeps the warp uniform
            if (__shfl_sync(kFull, sv, 0)) break;
        }
    }
    if (lane == 0) *nstates += s1 - s0;
    return true;
}

// Swept locations, written locations and input cones of a pair.  Lane l
// (l < 13) ends with the cone of output location l.
struct Flow {
    uint32_t swept;      // A, carry and the extra registers opReads implies
    uint32_t written;    // locations either sequence writes
    uint32_t cone;       // this lane's output cone (within `swept`)
    int k;               // extra registers swept
};

__device__ __forceinline__ uint32_t compose(uint32_t D, const uint16_t* seq, int n, int lane,
                                            uint32_t& written, uint32_t& sweep) {
    for (int i = 0; i < n; i++) {
        uint32_t op = seq[i] & 0xFFu;
        uint32_t dep = (lane < NUM_LOCS) ? c_dep[op][lane] : 0u;
        uint32_t nd = 0;
#pragma unroll
        for (int l = 0; l < NUM_LOCS; l++) {
            uint32_t x = __shfl_sync(kFull, D, l);
            if (dep & (1u << l)) nd |= x;
        }
        D = nd;
        written |= c_wr[op];
        sweep |= c_sweep[op];
    }
    return D;
}

__device__ __forceinline__ Flow dataflow(const PairView& pv, int lane) {
    Flow fl;
    uint32_t wt = 0, wc = 0, sw = 0;
    uint32_t id = (lane < NUM_LOCS) ? (1u << lane) : 0u;
    uint32_t dt = compose(id, pv.t, pv.tn, lane, wt, sw);
    uint32_t dc = compose(id, pv.c, pv.cn, lane, wc, sw);
    fl.k = __popc(sw);
    fl.swept = sw | LB(L_A) | LB(L_C);
    fl.written = wt | wc;
    fl.cone = (dt | dc) & fl.swept;
    return fl;
}

// Groups of a pair: maximal cones among the compared outputs; each group
// compares every output whose cone it contains.
struct Groups {
    int n;
    uint16_t cone[NUM_LOCS];
    uint64_t mask[NUM_LOCS];
    uint32_t bits[NUM_LOCS];
};

__device__ __forceinline__ uint32_t cone_bits(uint32_t cone, bool rep) {
    uint32_t b = 0;
    if (cone & LB(L_A)) b += 8;
    if (cone & LB(L_C)) b += 1;
    uint32_t extra = cone & ~(LB(L_A) | LB(L_C));
    b += (uint32_t)__popc(extra) * (rep ? 5u : 8u);
    return b;
}

__device__ Groups make_groups(const Flow& fl, uint32_t dead, bool rep, bool brute, int lane) {
    Groups g;
    g.n = 0;
    if (brute) {
        g.n = 1;
        g.cone[0] = (uint16_t)fl.swept;
        g.mask[0] = cmp_mask(dead);
        g.bits[0] = cone_bits(fl.swept, rep);
        return g;
    }
    uint32_t deadlocs = 0;
    for (uint32_t l = L_C; l <= L_N; l++) if (dead & flag_bit(l)) deadlocs |= LB(l);
    uint32_t active = fl.written & ~deadlocs;
    uint32_t cones[NUM_LOCS];
#pragma unroll
    for (int l = 0; l < NUM_LOCS; l++) cones[l] = __shfl_sync(kFull, fl.cone, l);
    for (int o = 0; o < NUM_LOCS; o++) {
        if (!(active & (1u << o))) continue;
        bool maximal = true;
        for (int q = 0; q < NUM_LOCS && maximal; q++) {
            if (q == o || !(active & (1u << q))) continue;
            bool sup = (cones[q] & cones[o]) == cones[o];
            if (sup && (cones[q] != cones[o] || q < o)) maximal = false;
        }
        if (!maximal) continue;
        uint64_t m = 0;
        for (int q = 0; q < NUM_LOCS; q++)
            if ((active & (1u << q)) && (cones[q] & cones[o]) == cones[q]) m |= loc_mask64((uint32_t)q);
        g.cone[g.n] = (uint16_t)cones[o];
        g.mask[g.n] = m;
        g.bits[g.n] = cone_bits(cones[o], rep);
        g.n++;
    }
    // smallest sweeps first: cheap groups reject failing pairs early
    for (int i = 1; i < g.n; i++)
        for (int j = i; j > 0 && g.bits[j] < g.bits[j - 1]; j--) {
            uint16_t tc = g.cone[j]; g.cone[j] = g.cone[j - 1]; g.cone[j - 1] = tc;
            uint64_t tm = g.mask[j]; g.mask[j] = g.mask[j - 1]; g.mask[j - 1] = tm;
            uint32_t tb = g.bits[j]; g.bits[j] = g.bits[j - 1]; g.bits[j - 1] = tb;
        }
    (void)lane;
    return g;
}

// The same composition reading the dependency table from shared memory
// (13 lanes read 13 different entries: constant memory would serialise).
// Most locations of an instruction depend on nothing or on themselves only,
// so only the locations that feed another one (`cross`, a few per
// instruction) are fetched from their lanes.
__device__ __forceinline__ uint32_t compose_s(uint32_t D, const uint16_t* seq, int n, int lane, uint32_t& written,
                                              uint32_t& sweep, const uint16_t (*dep_tab)[16]) {
    for (int i = 0; i < n; i++) {
        uint32_t op = seq[i] & 0xFFu;
        uint32_t dep = (lane < NUM_LOCS) ? dep_tab[op][lane] : 0u;
        const uint32_t self = 1u << lane;
        uint32_t nd = (dep & self) ? D : 0u;
        for (uint32_t cross = __reduce_or_sync(kFull, dep & ~self); cross; cross &= cross - 1) {
            const int l = __ffs(cross) - 1;
            const uint32_t x = __shfl_sync(kFull, D, l);
            if (dep & (1u << l)) nd |= x;
        }
        D = nd;
        written |= c_wr[op];
        sweep |= c_sweep[op];
    }
    return D;
}

// The same composition with the target's half kept in the warp's cache:
// pairs of one target (consecutive survivors) compose only their candidate.
// The two halves are independent: each starts from the identity.
__device__ __forceinline__ Flow dataflow_cached(const PairView& pv, int lane, const uint16_t (*dep_tab)[16],
                                                uint64_t tid, TargetCache& tc) {
    const uint32_t id = (lane < NUM_LOCS) ? (1u << lane) : 0u;
    uint32_t dt, wt, st;
    if (tid == kNoTarget || tc.flow_id != tid) {   // warp-uniform
        wt = 0; st = 0;
        dt = compose_s(id, pv.t, pv.tn, lane, wt, st, dep_tab);
        if (tid != kNoTarget) {
            __syncwarp();
            tc.dt[lane] = dt;
            if (lane == 0) { tc.wt = wt; tc.st = st; tc.flow_id = tid; }
            __syncwarp();
        }
    } else {
        dt = tc.dt[lane]; wt = tc.wt; st = tc.st;
    }
    Flow fl;
    uint32_t wc = 0, sw = st;
    const uint32_t dc = compose_s(id, pv.c, pv.cn, lane, wc, sw, dep_tab);
    fl.k = __popc(sw);
    fl.swept = sw | LB(L_A) | LB(L_C);
    fl.written = wt | wc;
    fl.cone = (dt | dc) & fl.swept;
    return fl;
}

// Lane-distributed groups: lane o (< 13) keeps the cone of output o; the
// maximal cones are found with shuffles and visited smallest first with warp
// reductions, so no per-thread arrays (local memory) are needed.
struct LaneGroups {
    uint32_t my;        // this lane's cone (0 when its output is not compared)
    uint32_t active;    // compared outputs (uniform)
    uint32_t maxm;      // outputs whose cone is maximal (uniform)
    uint32_t mybits;    // this lane's sweep bits when maximal
};

__device__ __forceinline__ LaneGroups lane_groups(const Flow& fl, uint32_t dead, bool rep, int lane) {
    LaneGroups g;
    uint32_t deadlocs = 0;
    for (uint32_t l = L_C; l <= L_N; l++) if (dead & flag_bit(l)) deadlocs |= LB(l);
    g.active = fl.written & ~deadlocs;
    const bool act = lane < NUM_LOCS && ((g.active >> lane) & 1u);
    g.my = act ? fl.cone : 0u;
    bool ismax = act;
    for (uint32_t rest = g.active & ((1u << NUM_LOCS) - 1u); rest; rest &= rest - 1) {   // compared outputs only
        const int q = __ffs(rest) - 1;
        const uint32_t cq = __shfl_sync(kFull, g.my, q);
        if (q != lane && (cq & g.my) == g.my && (cq != g.my || q < lane)) ismax = false;
    }
    g.maxm = __ballot_sync(kFull, ismax);
    g.mybits = ismax ? cone_bits(g.my, rep) : 0xFFu;
    return g;
}

// Next group (smallest sweep first) of `remaining`: its output lane, bits,
// cone and compare mask (outputs whose cone it contains).
__device__ __forceinline__ void next_group(const LaneGroups& g, uint32_t remaining, int lane, int& o, uint32_t& bits,
                                           uint32_t& cone, uint64_t& mask) {
    const uint32_t key = ((remaining >> lane) & 1u) ? ((g.mybits << 5) | (uint32_t)lane) : 0xFFFFFFFFu;
    const uint32_t kmin = __reduce_min_sync(kFull, key);
    o = (int)(kmin & 31u);
    bits = kmin >> 5;
    cone = __shfl_sync(kFull, g.my, o);
    const bool act = lane < NUM_LOCS && ((g.active >> lane) & 1u);
    const uint64_t contrib = (act && (g.my & cone) == g.my) ? loc_mask64((uint32_t)lane) : 0ull;
    const uint32_t lo = __reduce_or_sync(kFull, (uint32_t)contrib), hi = __reduce_or_sync(kFull, (uint32_t)(contrib >> 32));
    mask = (uint64_t)lo | ((uint64_t)hi << 32);
}

struct ExhArgs {
    uint32_t* fail;              // per pair: 1 = not equivalent
    Item* items;
    uint64_t item_cap;
    Counters* cnt;
    VerifyCounters* v;           // this verification's counters
    uint32_t sweep;              // M6502_SWEEP_*
    uint32_t brute;
    uint32_t defer_bits;         // > 0: pairs with a cone above 2^defer_bits states get fail = 4 (deferred)
    uint32_t ticket_batch;       // pairs a warp claims per ticket atomic (0 = kTicketBatch)
    uint32_t chunk_log2;         // states per work item, at least (0 = kChunk)
    const uint32_t* order;       // non-null: ticket q sweeps pair order[q] (the pairs k_small left);
                                 // null: ticket q is pair q
};

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// Fingerprints: warp per sequence, lane v = test vector v.  out: 32 packed
// states per sequence (P & PMask); meta (optional): CUDA bytes | Go bytes << 4.
struct FixedSeqs {
    const uint16_t* p;
    uint32_t len;
    __device__ int load(uint64_t i, uint16_t* dst, int lane) const {
        if (lane < (int)len) dst[lane] = p[i * len + lane];
        return (int)len;
    }
};
struct CsrSeqs {
    const uint16_t* ins;
    const uint32_t* off;
    __device__ int load(uint64_t i, uint16_t* dst, int lane) const {
        uint32_t a = off[i], n = off[i + 1] - a;
        if (lane < (int)n) dst[lane] = ins[a + lane];
        return (int)n;
    }
};
struct CandSeqs {
    uint32_t len;
    __device__ int load(uint64_t i, uint16_t* dst, int lane) const {
        if (lane == 0) {
            if (len == 1) dst[0] = c_tab[i];
            else { dst[0] = c_tab[i / kNumInsns]; dst[1] = c_tab[i % kNumInsns]; }
        }
        return (int)len;
    }
};

template <class Src>
__global__ void __launch_bounds__(256) k_fingerprint(Src src, uint64_t n, uint64_t* __restrict__ out,
                                                      uint8_t* __restrict__ meta) {
    __shared__ uint16_t s_seq[kWarpsPerBlock][kMaxSeq];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t nw = (uint64_t)gridDim.x * kWarpsPerBlock;
    for (uint64_t i = (uint64_t)blockIdx.x * kWarpsPerBlock + w; i < n; i += nw) {
        int len = src.load(i, s_seq[w], lane);
        __syncwarp();
        St s = unpack(c_vec[lane]);
        for (int k = 0; k < len; k++) exec(s, s_seq[w][k]);
        out[i * 32 + lane] = fp_of(s);
        if (meta && lane == 0) {
            uint32_t bc = 0, bg = 0;
            for (int k = 0; k < len; k++) { bc += bytes_cuda(s_seq[w][k] & 0xFFu); bg += bytes_go(s_seq[w][k] & 0xFFu); }
            meta[i] = (uint8_t)(min(bc, 15u) | (min(bg, 15u) << 4));
        }
        __syncwarp();
    }
}

// Survivor appends staged per warp in shared memory: one global atomic per
// flush of up to kStage records instead of one per warp-iteration with a hit
// (a single hot counter otherwise serialises millions of appends).
constexpr int kStage = 64;
__device__ __forceinline__ void stage_flush(Surv* buf, int& n, Surv* out, uint64_t cap,
                                            unsigned long long* counter, int lane) {
    if (n == 0) return;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(counter, (unsigned long long)n);
    base = __shfl_sync(kFull, base, 0);
    for (int i = lane; i < n; i += 32)
        if (base + (unsigned long long)i < cap) out[base + i] = buf[i];
    __syncwarp();
    n = 0;
}
__device__ __forceinline__ void stage_push(bool pass, Surv rec, Surv* buf, int& n, Surv* out, uint64_t cap,
                                           unsigned long long* counter, int lane) {
    unsigned vote = __ballot_sync(kFull, pass);
    if (!vote) return;
    if (pass) buf[n + __popc(vote & ((1u << lane) - 1u))] = rec;
    __syncwarp();
    n += __popc(vote);
    if (n > kStage - 32) stage_flush(buf, n, out, cap, counter, lane);
}

// Everything after a vector-0 match for one (target, candidate) pair: byte
// filter, pruner, QC vectors 1-7, then MidCheck vectors 8-31 (CUDA pipeline)
// or the Go worker's unmasked / masked split with FlagDiff.  Returns true
// and the survivor code when the pair goes on to ExhaustiveCheck.
template <bool GO>
__device__ __forceinline__ bool qc_candidate(const uint64_t* __restrict__ trow, uint64_t t0, uint64_t c0, uint32_t tb,
                                             uint32_t cm, uint32_t c, const uint64_t* __restrict__ cfp,
                                             uint64_t loose, uint64_t exact, uint32_t dead, uint32_t stages,
                                             unsigned long long& nqc, unsigned long long& nmid, uint32_t& code) {
    const uint32_t cb = GO ? ((cm >> 2) & 3u) : (cm & 3u);
    if ((cm & 0x90u) || cb >= tb) return false;   // pruned, padding, or not shorter
    bool qc = true, ex = ((t0 ^ c0) & exact) == 0;
    for (int v = 1; v < 8 && qc; v++) {
        uint64_t x = trow[v] ^ cfp[(uint64_t)v * kNumInsns + c];
        qc = (x & loose) == 0;
        ex = ex && (x & exact) == 0;
    }
    if (!qc) return false;
    if (!GO) {
        nqc++;
        bool mid = true;
        if (stages & M6502_CHECK_MID)
            for (int v = 8; v < 32 && mid; v++)
                mid = ((trow[v] ^ cfp[(uint64_t)v * kNumInsns + c]) & loose) == 0;
        if (!mid) return false;
        nmid++;
        code = c;
        return true;
    }
    if (ex) {           // processTask: unmasked QC passes
        nqc++; nmid++;
        code = c;
        return true;
    }
    if (dead) {         // processTaskMasked: masked QC passes, unmasked does not
        uint32_t fd = 0;
        for (int v = 0; v < 8; v++) fd |= (uint32_t)((trow[v] ^ cfp[(uint64_t)v * kNumInsns + c]) >> 24) & kPMask;
        if (fd) {
            nqc++; nmid++;
            code = c | kSurvMasked;
            return true;
        }
    }
    return false;
}

// QC (+ MidCheck) of targets x all length-1 candidates, scanning: every
// pair gets one masked 64-bit compare of its vector-0 outputs.
constexpr int kQcTile = 64;
constexpr int kQcPerThread = 12;   // 256 x 12 = 3072 >= 2863 candidates

template <bool GO>
__global__ void __launch_bounds__(256) k_qc1(const uint64_t* __restrict__ tfp, const uint8_t* __restrict__ tmeta,
                                              uint32_t nt, const uint64_t* __restrict__ cfp,
                                              const uint8_t* __restrict__ cmeta, uint32_t dead,
                                              uint32_t stages, Surv* __restrict__ surv, uint64_t cap,
                                              Counters* __restrict__ cnt, const uint32_t* __restrict__ bad = nullptr) {
    if (bad && *bad) return;
    __shared__ uint64_t s_t0[kQcTile];
    __shared__ uint8_t s_tb[kQcTile];
    __shared__ Surv s_stage[kWarpsPerBlock][kStage];
    const int lane = threadIdx.x & 31;
    Surv* stage = s_stage[threadIdx.x >> 5];
    int nstage = 0;
    const uint64_t loose = cmp_mask(dead), exact = cmp_mask(0);
    uint64_t c0[kQcPerThread];
    uint32_t cm[kQcPerThread];
#pragma unroll
    for (int j = 0; j < kQcPerThread; j++) {
        uint32_t c = threadIdx.x + 256u * (uint32_t)j;
        if (c < (uint32_t)kNumInsns) { c0[j] = cfp[c]; cm[j] = cmeta[c]; }
        else { c0[j] = 0; cm[j] = 0x80u; }   // padding lane: always filtered
    }
    unsigned long long nqc = 0, nmid = 0;
    const uint32_t ntiles = (nt + kQcTile - 1) / kQcTile;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        __syncthreads();
        if (threadIdx.x < kQcTile) {
            uint32_t t = tile * kQcTile + threadIdx.x;
            s_t0[threadIdx.x] = t < nt ? tfp[(uint64_t)t * 32] : 0;
            s_tb[threadIdx.x] = t < nt ? tmeta[t] : 0;
        }
        __syncthreads();
        const int tcount = (int)min((uint32_t)kQcTile, nt - tile * kQcTile);
        for (int k = 0; k < tcount; k++) {
            const uint64_t t0 = s_t0[k];
            uint32_t hm = 0;
#pragma unroll
            for (int j = 0; j < kQcPerThread; j++) hm |= (((t0 ^ c0[j]) & loose) == 0 ? 1u : 0u) << j;
            if (!__any_sync(kFull, hm != 0)) continue;
            const uint32_t t = tile * kQcTile + (uint32_t)k;
            const uint32_t tb = GO ? (s_tb[k] >> 4) : (s_tb[k] & 15u);
            const uint64_t* trow = tfp + (uint64_t)t * 32;
#pragma unroll
            for (int j = 0; j < kQcPerThread; j++) {
                bool pass = false;
                uint32_t code = 0;
                const uint32_t c = threadIdx.x + 256u * (uint32_t)j;
                if (hm & (1u << j))
                    pass = qc_candidate<GO>(trow, t0, c0[j], tb, cm[j], c, cfp, loose, exact, dead, stages,
                                            nqc, nmid, code);
                stage_push(pass, Surv{t, code}, stage, nstage, surv, cap, &cnt->surv, lane);
            }
        }
    }
    stage_flush(stage, nstage, surv, cap, &cnt->surv, lane);
    // one atomic per warp for the stage counters
    for (int o = 16; o; o >>= 1) {
        nqc += __shfl_down_sync(kFull, nqc, o);
        nmid += __shfl_down_sync(kFull, nmid, o);
    }
    if (lane == 0) {
        if (nqc) atomicAdd(&cnt->qc, nqc);
        if (nmid) atomicAdd(&cnt->mid, nmid);
    }
}

// QC (+ MidCheck) of targets x all length-1 candidates as an exact join
// through the mask's JoinTable.  A warp takes `chunk` (1..32) consecutive
// targets, a lane each: it runs its target on the 8 QuickCheck vectors (two
// packed words of four states), hashes the outputs, finds the key's entry
// and checks the outputs against it (cfp4: 256 packed bytes per candidate),
// then runs it on the 24 MidCheck vectors and finds its subclass.  A match is
// written as {target, first candidate in JoinTable::cand | count << 16};
// k_expand turns matches into the survivors that k_qc1 finds.
// Bound by integer issue: a warp per target with a
// lane per vector spent 400 warp instructions per target, most of them on
// dispatch, hashing and ballots for 32 states of two instructions; here those
// are paid once for 32 targets with four states per register.  Lanes whose
// targets differ in opcode diverge, which the enumeration's order makes rare
// and the packed words cheap.
// 1.9 M length-2 targets (every fourth), mask 0x00: 945 -> 138 us; 60 M warp
// instructions, latency bound now (38 % of issue slots).
template <bool GO>
__global__ void __launch_bounds__(256, 4) k_qc_join(const uint16_t* __restrict__ targets, uint32_t tlen, uint32_t nt,
                                                  uint32_t chunk, const uint4* __restrict__ cfp4,
                                                  const JoinTable* __restrict__ table, uint32_t dead,
                                                  uint32_t stages, Surv* __restrict__ match,
                                                  Counters* __restrict__ cnt, const uint32_t* __restrict__ bad) {
    if (bad && *bad) return;   // an opcode outside the table: nothing of this search counts
    __shared__ alignas(16) uint8_t s_raw[kJoinShared];
    const JoinTable& s_tab = *reinterpret_cast<const JoinTable*>(s_raw);   // key and dir only
    __shared__ Surv s_stage[kWarpsPerBlock][kStage];
    for (uint32_t i = threadIdx.x; i < kJoinShared / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(s_raw)[i] = reinterpret_cast<const uint4*>(table)[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Surv* stage = s_stage[w];
    int nstage = 0;
    const uint32_t pm = (kPMask & ~dead & 0xFFu) * kB1;   // compared bits of a packed P word
    unsigned long long nqc = 0;
    // Chunks come from a ticket, claimed one ahead: their hits are uneven, and
    // a fixed stride left some SMs with half the work of others.
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(&cnt->join_ticket, 1ull);
    for (;;) {
        const uint64_t base = __shfl_sync(kFull, next, 0) * chunk;
        if (base >= nt) break;
        if (lane == 0) next = atomicAdd(&cnt->join_ticket, 1ull);
        const bool have = (uint32_t)lane < chunk && base + lane < nt;
        const uint16_t* tp = targets + (base + (have ? lane : 0)) * tlen;
        uint32_t ins01 = tp[0], ins2 = 0;   // its instructions: two in the first word, the third in the second
        if (tlen > 1) ins01 |= (uint32_t)tp[1] << 16;
        if (tlen > 2) ins2 = tp[2];
        uint32_t tb = 0, lo = 0, n = 0;
        // Its outputs on vectors 8 r .. 8 r + 7 against candidate c's.
        auto run = [&](St (&v)[2], int r) {
#pragma unroll
            for (int g = 0; g < 2; g++)
                v[g] = St{c_vec4[2 * r + g][0], c_vec4[2 * r + g][1], c_vec4[2 * r + g][2], c_vec4[2 * r + g][3],
                          c_vec4[2 * r + g][4], c_vec4[2 * r + g][5], c_vec4[2 * r + g][6], c_vec4[2 * r + g][7]};
            for (uint32_t i = 0; i < tlen; i++) exec_x4n(v, i == 0 ? ins01 & 0xFFFFu : i == 1 ? ins01 >> 16 : ins2);
        };
        auto differ = [&](const St (&v)[2], int r, uint32_t c) -> uint32_t {
            const uint4* row = cfp4 + (size_t)c * 16 + r * 4;
            uint32_t d = 0;
#pragma unroll
            for (int g = 0; g < 2; g++) {
                const uint4 q0 = __ldg(row + 2 * g), q1 = __ldg(row + 2 * g + 1);
                d |= (v[g].a ^ q0.x) | (v[g].x ^ q0.y) | (v[g].y ^ q0.z) | ((v[g].p ^ q0.w) & pm) | (v[g].s ^ q1.x) |
                     (v[g].m ^ q1.y) | (v[g].s0 ^ q1.z) | (v[g].s1 ^ q1.w);
            }
            return d;
        };
        {
            St v[2];
            run(v, 0);
            for (uint32_t i = 0; i < tlen; i++) {
                const uint32_t op = (i == 0 ? ins01 : i == 1 ? ins01 >> 16 : ins2) & 0xFFu;
                tb += GO ? bytes_go(op) : bytes_cuda(op);
            }
            const uint32_t words[16] = {v[0].a, v[0].x, v[0].y, v[0].p & pm, v[0].s, v[0].m, v[0].s0, v[0].s1,
                                        v[1].a, v[1].x, v[1].y, v[1].p & pm, v[1].s, v[1].m, v[1].s0, v[1].s1};
            const uint64_t key = join_key(words);
            const uint32_t b = (uint32_t)(key >> (64 - kDirBits));
            uint32_t j0 = 0, j1 = 0;   // subclasses of the entry that matches
            for (uint32_t u = s_tab.dir[b], e = s_tab.dir[b + 1]; have && u < e; u++) {
                if (s_tab.key[u] != key) continue;
                const uint32_t j = table->sub[u];
                if (differ(v, 0, table->cand[table->start[j]] & 0xFFFu)) continue;
                j0 = j;
                j1 = table->sub[u + 1];
                if (!GO && tb > 1) nqc += table->weight[u][tb > 2];
                break;
            }
            if (GO || !(stages & M6502_CHECK_MID)) {   // every candidate of the entry
                lo = table->start[j0];
                n = table->start[j1] - lo;
            } else if (tb <= 1) {
                j1 = j0;                               // nothing is shorter
            }
            if (!GO && (stages & M6502_CHECK_MID)) {   // the subclass with the target's outputs, if any
                for (; j0 < j1; j0++) {
                    const uint32_t c = table->cand[table->start[j0]] & 0xFFFu;
                    bool equal = true;
                    for (int r = 1; r < 4 && equal; r++) {
                        run(v, r);
                        equal = differ(v, r, c) == 0;
                    }
                    if (!equal) continue;
                    lo = table->start[j0];
                    n = table->start[j0 + 1] - lo;
                    break;
                }
            }
        }
        stage_push(n > 0, Surv{(uint32_t)base + (uint32_t)lane, lo | n << 16}, stage, nstage, match, nt, &cnt->matches, lane);
    }
    stage_flush(stage, nstage, match, nt, &cnt->matches, lane);
    for (int o = 16; o; o >>= 1) nqc += __shfl_down_sync(kFull, nqc, o);
    if (lane == 0 && nqc) atomicAdd(&cnt->qc, nqc);
}

// ---- Matches to survivors ----
//
// A target that passes MidCheck with a run of compare operands (CMP #k for
// the k that no test vector tells apart) matches up to 43 candidates of which
// one is right, and a random state of the sweep domain tells two of them
// apart with a chance of a few in 256.  The line states do so for all of them
// at once: 256 states in which A and every register that the target reads
// take each value once (c_line: a permutation per register), the carry both
// values, and the others the sweep's fixed ones.  They lie in the sweep
// domain of every pair whose candidate reads no other register, so a pair
// whose outputs differ there is rejected, as ExhaustiveCheck would.  The
// outputs are compared by a 32-bit hash of the compared fields: the target's
// is computed once for all its candidates, the candidates' are tabulated per
// set of swept registers (k_line_hash, 64 x 2,863 per mask).  Unequal hashes
// come from unequal outputs only; equal ones are left to ExhaustiveCheck.
// Not filtered: pairs whose candidate reads a register the target does not,
// pairs swept over representative values (three or more extra registers
// under the reduced sweep), and targets for which it does not pay: those with
// one candidate, which costs as much to sweep, and those that write no live
// output, whose candidates are nearly all right (counting at 0xFF: 7.28 -> 6.42 ms).

// Bits 0..5 of a register set: X, Y, S, M, S0, S1 (the swept locations less A and carry).
__host__ __device__ __forceinline__ uint32_t extra_bits(uint32_t swept) { return (swept >> 1) & 0x3Fu; }

// Hash of the outputs of a sequence on the line states of register set
// `regs`: the sum of a term per packed word, of which this call adds words
// 2 sub, 2 sub + 1, then every 2 << g further on (2^g lanes share a
// sequence); run(v) executes it on two words.
template <class Run>
__device__ __forceinline__ uint32_t line_hash(uint32_t regs, uint32_t pm, const Run& run, uint32_t sub = 0, int g = 0) {
    auto mask = [&](uint32_t l) { return (regs & LB(l)) ? 0xFFFFFFFFu : 0u; };
    const uint32_t mx = mask(L_X), my = mask(L_Y), ms = mask(L_S), mm = mask(L_M), m0 = mask(L_S0), m1 = mask(L_S1);
    const uint32_t bs = ms ? 0u : 0xFDu * kB1;
    uint32_t h = 0;
    for (uint32_t j = 2 * sub; j < 64; j += 2u << g) {
        St v[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t* w = c_line[j + k];
            v[k] = St{w[0], w[1] & mx, w[2] & my, w[3], (w[4] & ms) | bs, w[5] & mm, w[6] & m0, w[7] & m1};
        }
        run(v);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const St& s = v[k];
            uint32_t x = (j + k) * 0x2C1B3C6Du + s.a * 0x9E3779B1u + s.x * 0x85EBCA77u + s.y * 0xC2B2AE3Du +
                         (s.p & pm) * 0x27D4EB2Fu + s.s * 0x165667B1u + s.m * 0xD3A2646Du + s.s0 * 0xFD7046C5u +
                         s.s1 * 0xB55A4F09u;
            x = (x ^ (x >> 15)) * 0x2C1B3C6Du;
            h += x ^ (x >> 13);
        }
    }
    return h;
}

// Thread per (register set, candidate): the candidates' hashes for one mask.
__global__ void __launch_bounds__(256) k_line_hash(uint32_t dead, uint32_t* __restrict__ out) {
    const uint32_t pm = (kPMask & ~dead & 0xFFu) * kB1;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 64u * kNumInsns; i += gridDim.x * blockDim.x) {
        const uint32_t insn = c_tab[i % kNumInsns];
        out[i] = line_hash((i / kNumInsns) << 1, pm, [&](St (&v)[2]) { exec_x4n(v, insn); });
    }
}

// Go semantics: ordinals of survivors met in Go order, 32 at a time.
struct GoCount {
    uint32_t run0 = 0, run1 = 0;   // unmasked and masked survivors so far of the target that lane 31 was at
    // This lane's ordinal within its target and pass.  `seg`: the first lane of
    // its target in this step; `cont`: the target began in an earlier step.
    __device__ __forceinline__ uint32_t step(bool take, bool masked, uint32_t seg, bool cont, int lane) {
        const unsigned b0 = __ballot_sync(kFull, take && !masked), b1 = __ballot_sync(kFull, take && masked);
        const unsigned span = (kFull << seg) & ((1u << lane) - 1u);
        const uint32_t k0 = (cont ? run0 : 0u) + __popc(b0 & span), k1 = (cont ? run1 : 0u) + __popc(b1 & span);
        run0 = __shfl_sync(kFull, k0, 31) + (b0 >> 31);
        run1 = __shfl_sync(kFull, k1, 31) + (b1 >> 31);
        return masked ? k1 : k0;
    }
};
// Survivors past the first round: kept with their ordinals.
__device__ __forceinline__ void go_late(bool late, Surv rec, uint32_t at, Surv* __restrict__ surv,
                                        uint32_t* __restrict__ ord, uint64_t cap, Counters* __restrict__ cnt, int lane) {
    const unsigned vote = __ballot_sync(kFull, late);
    if (!vote) return;
    const uint32_t top = __reduce_max_sync(kFull, late ? at : 0u);
    unsigned long long b = 0;
    if (lane == 0) {
        b = atomicAdd(&cnt->surv, (unsigned long long)__popc(vote));
        atomicMax(&cnt->max_ord, (unsigned long long)top);
    }
    b = __shfl_sync(kFull, b, 0) + __popc(vote & ((1u << lane) - 1u));
    if (late && b < cap) {
        surv[b] = rec;
        ord[b] = at;
    }
}

// A lane per match, or 2^g lanes while the matches alone do not fill the
// chip; a static stride, since each costs about the same.  FILTER computes
// the target's line hash; then the candidates of the warp's matches, numbered
// through, go round the lanes, and those that are shorter and not rejected
// are appended as survivors.
// The filter leaves 1.1 of the 5.4 M MidCheck survivors of the full length-2
// enumeration (mask 0x00); the random probe it replaces (128 states, a warp
// per pair) left 1.36 M in 2.42 ms.  Here, candidates and survivors included:
// 0.48 ms.
// Go semantics: the candidates of a match come in Go order, so a survivor's
// ordinal within its (target, pass) is a running count.  The first `block` of
// each go straight to the first round's list (there the line filter applies,
// on the run's mask in both passes: what differs under the mask differs
// without it), the others to `surv` with their ordinals.
template <bool GO, bool FILTER>
__global__ void __launch_bounds__(256, 4) k_expand(const Surv* __restrict__ match, const uint16_t* __restrict__ targets,
                                                 uint32_t tlen, const uint4* __restrict__ cfp4,
                                                 const JoinTable* __restrict__ table, uint32_t dead, uint32_t sweep,
                                                 const uint16_t* __restrict__ mult, const uint32_t* __restrict__ lines,
                                                 Surv* __restrict__ surv, uint64_t cap, Counters* __restrict__ cnt,
                                                 Surv* __restrict__ first, uint32_t* __restrict__ ord, uint32_t block) {
    __shared__ Surv s_stage[kWarpsPerBlock][kStage];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Surv* stage = s_stage[w];
    int nstage = 0;
    const uint32_t pm = (kPMask & ~dead & 0xFFu) * kB1;   // compared bits of a packed P word
    unsigned long long nqc = 0, nmid = 0, nrej = 0;
    const uint32_t nmatch = (uint32_t)cnt->matches;
    int g = 5;   // lanes per match, log2
    for (uint64_t warps = (uint64_t)gridDim.x * kWarpsPerBlock; g > 0 && nmatch > warps; g--) warps <<= 1;
    const uint32_t sub = (uint32_t)lane & ((1u << g) - 1u), per = 32u >> g;
    for (uint64_t base = ((uint64_t)blockIdx.x * kWarpsPerBlock + w) * per; base < nmatch;
         base += (uint64_t)gridDim.x * kWarpsPerBlock * per) {
        const uint64_t mi = base + (uint32_t)(lane >> g);
        const bool have = mi < nmatch && sub == 0;   // the lane that stands for the match
        const Surv m = match[mi < nmatch ? mi : base];
        const uint16_t* tp = targets + (uint64_t)m.t * tlen;
        uint32_t ins01 = tp[0], ins2 = 0;
        if (tlen > 1) ins01 |= (uint32_t)tp[1] << 16;
        if (tlen > 2) ins2 = tp[2];
        const uint32_t lo = m.c & 0xFFFFu, n = have ? m.c >> 16 : 0u;
        auto run = [&](St (&v)[2]) {
            for (uint32_t i = 0; i < tlen; i++) exec_x4n(v, i == 0 ? ins01 & 0xFFFFu : i == 1 ? ins01 >> 16 : ins2);
        };
        uint32_t tb = 0, regs = 0, live = 0;   // live: compared locations that it writes
        for (uint32_t i = 0; i < tlen; i++) {
            const uint32_t op = (i == 0 ? ins01 : i == 1 ? ins01 >> 16 : ins2) & 0xFFu;
            tb += GO ? bytes_go(op) : bytes_cuda(op);
            regs |= c_sweep[op];
            live |= c_wr[op];
        }
        live &= ~(((dead & 0x0Fu) << L_C) | ((dead >> 6) << L_V));
        uint32_t hash = 0, tp0 = 0, tp1 = 0;   // tp: P after the QuickCheck vectors (Go semantics)
        bool filter = FILTER && n > 1 && live && !(sweep == M6502_SWEEP_REFERENCE && __popc(regs) >= 3);
        if (FILTER && __any_sync(kFull, filter)) {
            hash = line_hash(regs, pm, run, sub, g);
            for (int o = 0; o < g; o++) hash += __shfl_xor_sync(kFull, hash, 1 << o);
        }
        if (GO) {
            St v[2];
#pragma unroll
            for (int g = 0; g < 2; g++)
                v[g] = St{c_vec4[g][0], c_vec4[g][1], c_vec4[g][2], c_vec4[g][3],
                          c_vec4[g][4], c_vec4[g][5], c_vec4[g][6], c_vec4[g][7]};
            run(v);
            tp0 = v[0].p;
            tp1 = v[1].p;
        }
        uint32_t upto = n;   // candidates of this lane's match and the lanes' below
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(kFull, upto, o);
            upto += lane >= o ? x : 0u;
        }
        const uint32_t total = __shfl_sync(kFull, upto, 31);
        GoCount count;
        for (uint32_t h0 = 0; h0 < total; h0 += 32) {
            const uint32_t h = h0 + (uint32_t)lane;
            uint32_t own = 0;   // lanes whose candidates end at or before h
#pragma unroll
            for (uint32_t o = 16; o; o >>= 1) {
                const uint32_t x = __shfl_sync(kFull, upto, (int)(own + o - 1));
                own += x <= h ? o : 0u;
            }
            const uint32_t end = __shfl_sync(kFull, upto, (int)own), cnt_o = __shfl_sync(kFull, n, (int)own);
            const uint32_t lo_o = __shfl_sync(kFull, lo, (int)own), tb_o = __shfl_sync(kFull, tb, (int)own);
            const uint32_t t = __shfl_sync(kFull, m.t, (int)own);
            bool pass = h < total;
            uint32_t c = 0;
            if (pass) {
                c = table->cand[lo_o + (h - (end - cnt_o))];
                pass = (c >> 12) < tb_o;   // not shorter in bytes: not a candidate
                c &= 0xFFFu;
            }
            uint32_t code = c;
            if (GO) {
                // FlagDiff over the QC vectors: zero when the unmasked QuickCheck
                // passes too (processTask), else the masked pass (processTaskMasked).
                const uint32_t p0 = __shfl_sync(kFull, tp0, (int)own), p1 = __shfl_sync(kFull, tp1, (int)own);
                if (pass) {
                    const uint32_t* row = reinterpret_cast<const uint32_t*>(cfp4) + (size_t)c * 64;
                    if (((p0 ^ __ldg(row + 3)) | (p1 ^ __ldg(row + 11))) & (kPMask * kB1)) {
                        pass = dead != 0;
                        code = c | kSurvMasked;
                    }
                }
                nqc += pass;
                nmid += pass;
                const bool masked = (code & kSurvMasked) != 0;
                const uint32_t start = end - cnt_o;   // the match's first candidate
                const uint32_t at = count.step(pass, masked, start <= h0 ? 0u : start - h0, start < h0, lane);
                bool early = pass && at < block;
                go_late(pass && !early, Surv{t, code}, at, surv, ord, cap, cnt, lane);
                if (FILTER) {
                    const uint32_t hash_o = __shfl_sync(kFull, hash, (int)own), regs_o = __shfl_sync(kFull, regs, (int)own);
                    const bool filter_o = __shfl_sync(kFull, (int)filter, (int)own) != 0;
                    if (early && filter_o && !(c_sweep[c_tab[c] & 0xFFu] & ~regs_o) &&
                        lines[extra_bits(regs_o) * kNumInsns + c] != hash_o) {
                        early = false;
                        nrej++;
                    }
                }
                stage_push(early, Surv{t, code}, stage, nstage, first, cap, &cnt->v[0][0].n, lane);
                continue;
            } else {
                const uint32_t weight = pass ? mult[c] : 0u;   // pairs this record stands for
                nmid += weight;
                if (FILTER) {
                    const uint32_t hash_o = __shfl_sync(kFull, hash, (int)own), regs_o = __shfl_sync(kFull, regs, (int)own);
                    const bool filter_o = __shfl_sync(kFull, (int)filter, (int)own) != 0;
                    if (pass && filter_o && !(c_sweep[c_tab[c] & 0xFFu] & ~regs_o) &&
                        lines[extra_bits(regs_o) * kNumInsns + c] != hash_o) {
                        pass = false;
                        nrej += weight;
                    }
                }
            }
            stage_push(pass, Surv{t, code}, stage, nstage, surv, cap, &cnt->surv, lane);
        }
    }
    if (GO) stage_flush(stage, nstage, first, cap, &cnt->v[0][0].n, lane);
    else stage_flush(stage, nstage, surv, cap, &cnt->surv, lane);
    for (int o = 16; o; o >>= 1) {
        nqc += __shfl_down_sync(kFull, nqc, o);
        nmid += __shfl_down_sync(kFull, nmid, o);
        nrej += __shfl_down_sync(kFull, nrej, o);
    }
    if (lane == 0) {
        if (nqc) atomicAdd(&cnt->qc, nqc);
        if (nmid) atomicAdd(&cnt->mid, nmid);
        if (nrej) atomicAdd(&cnt->probe_rejects, nrej);
        if (GO && nrej) atomicAdd(&cnt->round_rejects, nrej);
    }
}

// ---- Length-2 candidates: an exact join over all 2,863^2 sequences ----
//
// Per dead-flags mask, every length-2 sequence (CUDA index c0 * 2863 + c1)
// gets the key of its 8 masked QuickCheck outputs; the (key, entry) table is
// radix-sorted on the device once and cached.  A target's QuickCheck hits
// among the 8.2 M candidates are then exactly the candidates with its key
// that re-pass the 8 vectors -- found by one warp-wide search per target.
// The sequences enter the (stable) sort in Go order, so those of one key stay
// in Go order.  An entry holds the index, the pruner's answer and the sizes.
constexpr uint32_t kEntryIndex = 0x7FFFFFu, kEntryPruned = 1u << 23;
__device__ __forceinline__ uint32_t entry_bytes_cuda(uint32_t e) { return 2u + ((e >> 24) & 3u); }
__device__ __forceinline__ uint32_t entry_bytes_go(uint32_t e) { return 2u + ((e >> 26) & 3u); }

// Keys of all length-2 sequences in Go order, thread per sequence.
__global__ void k_cand2_keys(uint32_t dead, uint64_t salt, uint64_t* __restrict__ keys, uint32_t* __restrict__ idx) {
    const uint64_t loose = cmp_mask(dead);
    const uint32_t n = (uint32_t)kNumInsns * (uint32_t)kNumInsns;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t c0 = c_goidx[r / kNumInsns], c1 = c_goidx[r % kNumInsns];
        const uint16_t seq[2] = {c_tab[c0], c_tab[c1]};
        uint64_t x = 0;
        for (int v = 0; v < 8; v++) {
            St s = unpack(c_vec[v]);
            exec(s, seq[0]);
            exec(s, seq[1]);
            x ^= key_term((fp_of(s) & loose) + salt, v);
        }
        keys[r] = key_final(x);
        const uint32_t bc = bytes_cuda(seq[0] & 0xFFu) + bytes_cuda(seq[1] & 0xFFu),
                       bg = bytes_go(seq[0] & 0xFFu) + bytes_go(seq[1] & 0xFFu);
        idx[r] = (c0 * kNumInsns + c1) | (should_prune(seq, 2) ? kEntryPruned : 0u) | (bc - 2) << 24 | (bg - 2) << 26;
    }
}

// X4Row of an opcode in shared memory (copied from g_x4row).
__device__ __forceinline__ X4Row load_row(const uint4 (&q)[3]) {
    const uint4 a = q[0], b = q[1], c = q[2];
    return X4Row{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
}

// After the sort: P after the QuickCheck vectors of every entry (pw, for
// FlagDiff); whether two different sets of outputs share a key (info[0]: the
// table is then built again with another salt, so that one candidate of a
// range decides QuickCheck for all); the longest range of one key (info[1]).
// Sorted by a hash, neighbours share no opcode: the per-opcode switch runs up
// to 30 arms for a warp, and every entry was run a second time for its
// successor's comparison.  The table-driven executor has one course for all
// lanes, and a warp takes 31 entries behind one that it runs for comparison
// only, whose outputs the next lane gets by a shuffle: 2.5 -> 0.37 ms for a
// mask's 8.2 M entries.
constexpr int kInfoThreads = 256;
__global__ void __launch_bounds__(kInfoThreads) k_cand2_info(uint32_t dead, const uint64_t* __restrict__ keys,
                                                             const uint32_t* __restrict__ idx, uint2* __restrict__ pw,
                                                             uint32_t* __restrict__ info) {
    __shared__ uint4 s_row[NUM_OPS][3];
    __shared__ uint32_t s_st[X4S_COUNT][kInfoThreads];   // each lane's registers
    for (int i = threadIdx.x; i < (int)NUM_OPS * 3; i += kInfoThreads) (&s_row[0][0])[i] = g_x4row[i];
    __syncthreads();
    const uint32_t pm = (kPMask & ~dead & 0xFFu) * kB1;
    const uint32_t n = (uint32_t)kNumInsns * (uint32_t)kNumInsns;
    const uint32_t lane = threadIdx.x & 31u, warps = gridDim.x * (kInfoThreads / 32);
    uint32_t* st = &s_st[0][threadIdx.x];
    uint32_t longest = 0, clash = 0;
    for (uint32_t first = (blockIdx.x * (kInfoThreads / 32) + (threadIdx.x >> 5)) * 31u; first < n; first += warps * 31u) {
        // lane 0: the entry before `first` (the very first one stands in for its own)
        const uint32_t at = first + lane, i = min(at ? at - 1u : 0u, n - 1u);
        const uint32_t c = idx[i] & kEntryIndex;
        const uint64_t key = keys[i], before = __shfl_up_sync(kFull, key, 1);
        const uint32_t insn[2] = {c_tab[c / kNumInsns], c_tab[c % kNumInsns]};
        const X4Row row[2] = {load_row(s_row[insn[0] & 0xFFu]), load_row(s_row[insn[1] & 0xFFu])};
        uint32_t differ = 0, p[2];
#pragma unroll
        for (int g = 0; g < 2; g++) {
            st[X4S_A * kInfoThreads] = c_vec4[g][0]; st[X4S_X * kInfoThreads] = c_vec4[g][1]; st[X4S_Y * kInfoThreads] = c_vec4[g][2];
            st[X4S_S * kInfoThreads] = c_vec4[g][4]; st[X4S_M * kInfoThreads] = c_vec4[g][5]; st[X4S_S0 * kInfoThreads] = c_vec4[g][6];
            st[X4S_S1 * kInfoThreads] = c_vec4[g][7];
            p[g] = c_vec4[g][3];
            exec_x4r(st, kInfoThreads, p[g], row[0], insn[0]);
            exec_x4r(st, kInfoThreads, p[g], row[1], insn[1]);
#pragma unroll
            for (int f = 0; f < (int)X4S_NONE; f++) {
                const uint32_t v = st[f * kInfoThreads];
                differ |= v ^ __shfl_up_sync(kFull, v, 1);
            }
            differ |= (p[g] ^ __shfl_up_sync(kFull, p[g], 1)) & pm;
        }
        if (lane == 0 || at > n) continue;
        pw[i] = make_uint2(p[0] & (kPMask * kB1), p[1] & (kPMask * kB1));
        if (i > 0 && before == key) {
            clash |= differ;
        } else {   // first of its range: the range's end by doubling and halving
            uint32_t step = 1;
            while (i + step < n && keys[i + step] == key) step <<= 1;
            uint32_t lo = i + (step >> 1), hi = min(i + step, n);   // keys[lo] == key; keys[hi] is another or past the end
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (keys[mid] == key) lo = mid; else hi = mid;
            }
            longest = max(longest, hi - i);
        }
    }
    if (__any_sync(kFull, clash != 0) && lane == 0) info[0] = 1u;
    longest = __reduce_max_sync(kFull, longest);
    if (lane == 0) atomicMax(info + 1, longest);
}

// Equal ranges are very uneven (a flags-only target under mask 0xFF matches
// hundreds of thousands of flags-only candidates), so a range longer than
// kJoinChunk is cut into work items that every warp drains.
constexpr uint32_t kJoinChunk = 1024;

struct JoinItem {   // candidates [lo, hi) of one target's equal range
    uint32_t t, lo, hi, exact;
    uint32_t seq;      // items of the same range before it (they lie next to each other)
    uint32_t n0, n1;   // Go semantics: its survivors of each pass
    uint32_t pad;
};

struct Cand2View {     // the sorted table of one mask
    const uint64_t* keys;
    const uint32_t* idx;
    const uint2* pw;
    uint64_t salt;
};

struct Join2Args {
    const uint64_t* tfp;
    const uint8_t* tmeta;
    uint32_t nt;
    Cand2View loose;         // the run mask's table
    Cand2View exact;         // the unmasked table (Go semantics, unmasked pass only)
    uint32_t nsorted;
    uint32_t dead;
    uint32_t stages;
    const uint32_t* best;    // Go semantics: settled passes
    Surv* surv;
    uint64_t cap;
    JoinItem* items;
    uint64_t item_cap;
    Counters* cnt;
    Surv* first;             // Go semantics: the first round's list (see k_expand)
    uint32_t* ord;
    uint32_t block;
};

// CUDA semantics: QC + MidCheck of targets x all length-2 candidates through
// the sorted table.  Lane v executes the candidate on vector v.  The byte
// filter and the pruner are applied per candidate in the equal range.
__device__ __forceinline__ void join2_range(const Join2Args& a, uint32_t t, uint32_t lo, uint32_t hi, uint64_t tv,
                                            Surv* stage, int& nstage, unsigned long long& nqc,
                                            unsigned long long& nmid, int lane) {
    const uint64_t loose = cmp_mask(a.dead);
    const uint32_t tb = a.tmeta[t] & 15u;
    for (uint32_t base = lo; base < hi; base += 32) {
        const uint32_t i = base + (uint32_t)lane;
        const uint32_t mine = i < hi ? a.loose.idx[i] : kEntryPruned;
        // shorter, and not pruned
        unsigned run = __ballot_sync(kFull, !(mine & kEntryPruned) && entry_bytes_cuda(mine) < tb);
        for (; run; run &= run - 1) {
            const uint32_t c = __shfl_sync(kFull, mine, __ffs(run) - 1) & kEntryIndex;
            St s = unpack(c_vec[lane]);
            exec(s, c_tab[c / kNumInsns]);
            exec(s, c_tab[c % kNumInsns]);
            const unsigned eq = __ballot_sync(kFull, ((tv ^ fp_of(s)) & loose) == 0);
            if ((eq & 0xFFu) != 0xFFu) continue;          // hash collision: QuickCheck fails
            nqc += lane == 0;
            const bool mid = !(a.stages & M6502_CHECK_MID) || eq == kFull;
            nmid += mid && lane == 0;
            stage_push(mid && lane == 0, Surv{t, c | kSurvLen2}, stage, nstage, a.surv, a.cap, &a.cnt->surv, lane);
        }
    }
}

__device__ __forceinline__ void join_counts(Counters* cnt, unsigned long long nqc, unsigned long long nmid) {
    for (int o = 16; o; o >>= 1) {
        nqc += __shfl_down_sync(kFull, nqc, o);
        nmid += __shfl_down_sync(kFull, nmid, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (nqc) atomicAdd(&cnt->qc, nqc);
        if (nmid) atomicAdd(&cnt->mid, nmid);
    }
}

// The range [lo, hi) of a target's key in a table.
__device__ __forceinline__ void key_range(const Cand2View& tab, uint32_t n, uint64_t key, uint32_t& lo, uint32_t& hi, int lane) {
    lo = warp_lower_bound(tab.keys, n, key, lane);
    hi = key == ~0ull ? n : warp_lower_bound(tab.keys, n, key + 1, lane);
}

// Cuts a long range into items.
__device__ __forceinline__ void push_items(const Join2Args& a, uint32_t t, uint32_t lo, uint32_t hi, bool exact, int lane) {
    const uint32_t nitems = (hi - lo + kJoinChunk - 1) / kJoinChunk;
    unsigned long long b = 0;
    if (lane == 0) b = atomicAdd(&a.cnt->join_items, (unsigned long long)nitems);
    b = __shfl_sync(kFull, b, 0);
    for (uint32_t j = lane; j < nitems; j += 32)
        if (b + j < a.item_cap)
            a.items[b + j] = JoinItem{t, lo + j * kJoinChunk, min(hi, lo + (j + 1) * kJoinChunk), exact ? 1u : 0u, j, 0, 0, 0};
}

__global__ void __launch_bounds__(256) k_qc_join2(Join2Args a) {
    __shared__ Surv s_stage[kWarpsPerBlock][kStage];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Surv* stage = s_stage[w];
    int nstage = 0;
    unsigned long long nqc = 0, nmid = 0;
    for (uint32_t t = blockIdx.x * kWarpsPerBlock + w; t < a.nt; t += gridDim.x * kWarpsPerBlock) {
        const uint64_t tv = a.tfp[(uint64_t)t * 32 + lane];
        uint32_t lo, hi;
        key_range(a.loose, a.nsorted, warp_key(tv, cmp_mask(a.dead), a.loose.salt, lane), lo, hi, lane);
        if (hi - lo <= kJoinChunk) join2_range(a, t, lo, hi, tv, stage, nstage, nqc, nmid, lane);
        else push_items(a, t, lo, hi, false, lane);
    }
    stage_flush(stage, nstage, a.surv, a.cap, &a.cnt->surv, lane);
    join_counts(a.cnt, nqc, nmid);
}

// The chunks of the long equal ranges, a warp per chunk.
__global__ void __launch_bounds__(256) k_qc_join2_items(Join2Args a) {
    __shared__ Surv s_stage[kWarpsPerBlock][kStage];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Surv* stage = s_stage[w];
    int nstage = 0;
    unsigned long long nqc = 0, nmid = 0;
    const uint64_t n = min((uint64_t)a.cnt->join_items, a.item_cap);
    for (uint64_t q = (uint64_t)blockIdx.x * kWarpsPerBlock + w; q < n; q += (uint64_t)gridDim.x * kWarpsPerBlock) {
        const JoinItem it = a.items[q];
        join2_range(a, it.t, it.lo, it.hi, a.tfp[(uint64_t)it.t * 32 + lane], stage, nstage, nqc, nmid, lane);
    }
    stage_flush(stage, nstage, a.surv, a.cap, &a.cnt->surv, lane);
    join_counts(a.cnt, nqc, nmid);
}

// Go semantics: QuickCheck of targets x all length-2 candidates.  No
// MidCheck, and the candidates of a range have one set of masked outputs (the
// table is built so), so one of them decides for all; what is left per
// candidate is its entry (pruned, size) and its FlagDiff from the tabulated P
// words: a lane each, where a warp per candidate ran it on the vectors before
// (4,096 length-3 targets, mask 0xC3: 2.36 ms, now 0.14).
// `best` ([2][nt], the length-1 winners) skips the passes a target has already
// settled (the worker stops at the first candidate length that finds one,
// worker.go:122-176).  Candidates come in Go order; a long range's items are
// counted first (k_go_join2_count), so that each knows the ordinals before it.
struct GoRange {
    bool need_u, need_m, use_exact;
    uint32_t tb, p0, p1;   // Go byte size; P after the QuickCheck vectors
};

__device__ __forceinline__ GoRange go_range(const Join2Args& a, uint32_t t, uint64_t tv, int lane) {
    GoRange r;
    r.need_u = a.best[t] == 0xFFFFFFFFu;
    r.need_m = a.dead != 0 && a.best[(uint64_t)a.nt + t] == 0xFFFFFFFFu;
    // Only the unmasked pass open: its candidates are the exact-key range of
    // the unmasked table, a subset of the masked key's range.
    r.use_exact = !r.need_m;
    r.tb = a.tmeta[t] >> 4;
    const uint32_t p = (uint32_t)(tv >> 24) & 0xFFu;
    r.p0 = __reduce_or_sync(kFull, lane < 4 ? p << (8 * lane) : 0u);
    r.p1 = __reduce_or_sync(kFull, lane >= 4 && lane < 8 ? p << (8 * (lane - 4)) : 0u);
    return r;
}

// One step of 32 candidates from `base`: whether this lane's is a survivor
// of an open pass, which, and its index.
__device__ __forceinline__ bool go_candidate(const Join2Args& a, const GoRange& r, uint32_t i, uint32_t hi, bool& masked,
                                             uint32_t& c) {
    masked = false;
    if (i >= hi) return false;
    const uint32_t e = r.use_exact ? a.exact.idx[i] : a.loose.idx[i];
    c = e & kEntryIndex;
    if ((e & kEntryPruned) || entry_bytes_go(e) >= r.tb) return false;
    if (!r.use_exact) {
        const uint2 p = a.loose.pw[i];
        masked = (((p.x ^ r.p0) | (p.y ^ r.p1)) & (kPMask * kB1)) != 0;   // FlagDiff != 0: processTaskMasked
    }
    return masked ? r.need_m : r.need_u;
}

__device__ __forceinline__ void go_scan(const Join2Args& a, const GoRange& r, uint32_t t, uint32_t lo, uint32_t hi,
                                        uint32_t n0, uint32_t n1, Surv* stage, int& nstage, unsigned long long& nqc, int lane) {
    GoCount count{n0, n1};
    for (uint32_t base = lo; base < hi; base += 32) {
        bool masked;
        uint32_t c = 0;
        const bool take = go_candidate(a, r, base + lane, hi, masked, c);
        nqc += take;
        const uint32_t at = count.step(take, masked, 0, true, lane);
        const Surv rec{t, c | kSurvLen2 | (masked ? kSurvMasked : 0u)};
        go_late(take && at >= a.block, rec, at, a.surv, a.ord, a.cap, a.cnt, lane);
        stage_push(take && at < a.block, rec, stage, nstage, a.first, a.cap, &a.cnt->v[1][0].n, lane);
    }
}

__global__ void __launch_bounds__(256) k_go_join2(Join2Args a) {
    __shared__ Surv s_stage[kWarpsPerBlock][kStage];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Surv* stage = s_stage[w];
    int nstage = 0;
    unsigned long long nqc = 0;
    for (uint32_t t = blockIdx.x * kWarpsPerBlock + w; t < a.nt; t += gridDim.x * kWarpsPerBlock) {
        const uint64_t tv = a.tfp[(uint64_t)t * 32 + lane];
        const GoRange r = go_range(a, t, tv, lane);
        if (!r.need_u && !r.need_m) continue;
        const Cand2View& tab = r.use_exact ? a.exact : a.loose;
        const uint64_t km = r.use_exact ? cmp_mask(0) : cmp_mask(a.dead);
        uint32_t lo, hi;
        key_range(tab, a.nsorted, warp_key(tv, km, tab.salt, lane), lo, hi, lane);
        if (lo == hi) continue;
        const uint32_t c = tab.idx[lo] & kEntryIndex;   // the range's QuickCheck
        St s = unpack(c_vec[lane]);
        exec(s, c_tab[c / kNumInsns]);
        exec(s, c_tab[c % kNumInsns]);
        if ((__ballot_sync(kFull, ((tv ^ fp_of(s)) & km) == 0) & 0xFFu) != 0xFFu) continue;
        if (hi - lo <= kJoinChunk) go_scan(a, r, t, lo, hi, 0, 0, stage, nstage, nqc, lane);
        else push_items(a, t, lo, hi, r.use_exact, lane);
    }
    stage_flush(stage, nstage, a.first, a.cap, &a.cnt->v[1][0].n, lane);
    join_counts(a.cnt, nqc, nqc);
}

__global__ void __launch_bounds__(256) k_go_join2_count(Join2Args a) {
    const int lane = threadIdx.x & 31;
    const uint64_t n = min((uint64_t)a.cnt->join_items, a.item_cap);
    for (uint64_t q = (uint64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); q < n; q += (uint64_t)gridDim.x * kWarpsPerBlock) {
        const JoinItem it = a.items[q];
        const GoRange r = go_range(a, it.t, a.tfp[(uint64_t)it.t * 32 + lane], lane);
        uint32_t n0 = 0, n1 = 0;
        for (uint32_t base = it.lo; base < it.hi; base += 32) {
            bool masked;
            uint32_t c;
            const bool take = go_candidate(a, r, base + lane, it.hi, masked, c);
            n0 += __popc(__ballot_sync(kFull, take && !masked));
            n1 += __popc(__ballot_sync(kFull, take && masked));
        }
        if (lane == 0) { a.items[q].n0 = n0; a.items[q].n1 = n1; }
    }
}

__global__ void __launch_bounds__(256) k_go_join2_items(Join2Args a) {
    __shared__ Surv s_stage[kWarpsPerBlock][kStage];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Surv* stage = s_stage[w];
    int nstage = 0;
    unsigned long long nqc = 0;
    const uint64_t n = min((uint64_t)a.cnt->join_items, a.item_cap);
    for (uint64_t q = (uint64_t)blockIdx.x * kWarpsPerBlock + w; q < n; q += (uint64_t)gridDim.x * kWarpsPerBlock) {
        const JoinItem it = a.items[q];
        const GoRange r = go_range(a, it.t, a.tfp[(uint64_t)it.t * 32 + lane], lane);
        uint32_t n0 = 0, n1 = 0;   // survivors of the items before it
        for (uint32_t j = lane; j < it.seq; j += 32) { n0 += a.items[q - 1 - j].n0; n1 += a.items[q - 1 - j].n1; }
        n0 = __reduce_add_sync(kFull, n0);
        n1 = __reduce_add_sync(kFull, n1);
        go_scan(a, r, it.t, it.lo, it.hi, n0, n1, stage, nstage, nqc, lane);
    }
    stage_flush(stage, nstage, a.first, a.cap, &a.cnt->v[1][0].n, lane);
    join_counts(a.cnt, nqc, nqc);
}

// First ticket of a warp of a persistent grid: its own number, counted across
// the blocks first, so that few pairs spread over the SMs.  Later tickets come
// from a counter that starts behind those.  A launch with few pairs or none, as
// in most rounds past the first, then costs neither an atomic per warp on one
// address nor the tables of idle blocks (empty launches took 6.1 us in k_small
// and 8.2 in k_exhaustive): one target 280 -> 227 us, 4,096 length-3 targets
// 914 -> 832.  Not for k_exh_items, whose items outnumber its warps where they
// count (0.6 % of the count at mask 0xFF slower): its idle blocks only leave.
__device__ __forceinline__ unsigned long long first_ticket(unsigned long long batch) {
    return ((unsigned long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * batch;
}
__device__ __forceinline__ unsigned long long later_ticket(unsigned long long* ctr, unsigned long long batch,
                                                           unsigned long long n) {
    const unsigned long long taken = (unsigned long long)gridDim.x * kWarpsPerBlock * batch;
    return taken >= n ? n : taken + atomicAdd(ctr, batch);
}

// Exhaustive check, one pair per warp (persistent, device ticket).
// MINB: resident 256-thread blocks per SM the register cap is set for (4:
// 64 registers, 3: 80, 2: 128); the autotuner picks the variant.
template <class Src, int MINB = 4>
__global__ void __launch_bounds__(256, MINB) k_exhaustive(Src src, const unsigned long long* n_pairs_ptr,
                                                        uint64_t n_cap, ExhArgs a) {
    __shared__ uint16_t s_t[kWarpsPerBlock][kMaxSeq], s_c[kWarpsPerBlock][kMaxSeq];
    __shared__ alignas(16) uint16_t s_dep[NUM_OPS][16];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t n = min((uint64_t)*n_pairs_ptr, n_cap);
    if (blockIdx.x >= n) return;   // no warp of this block has a pair
    for (int i = threadIdx.x; i < (int)NUM_OPS * 2; i += blockDim.x) reinterpret_cast<uint4*>(&s_dep[0][0])[i] = g_dep16[i];
    __syncthreads();
    unsigned long long nstates = 0, probe_rej = 0;
    __shared__ TargetCache s_tc[kWarpsPerBlock];   // the warp's last target: probe outputs, composition
    TargetCache& tc = s_tc[threadIdx.x >> 5];
    if ((threadIdx.x & 31) == 0) { tc.probe_id = kNoTarget; tc.flow_id = kNoTarget; }
    __syncwarp();
    unsigned long long next = 0, lim = 0;   // this warp's batch of tickets
    // Pairs per ticket: the knob's, but no more than leaves every warp one (few
    // large pairs in the hands of one warp: 185 us for the 1,000 that k_small
    // leaves of a pass of 2 M length-2 targets, one at a time 43).
    const unsigned long long share = n / ((uint64_t)gridDim.x * kWarpsPerBlock);
    const unsigned long long tbatch = max(1ull, min(share, (unsigned long long)(a.ticket_batch ? a.ticket_batch : kTicketBatch)));
    const uint64_t chunk_min = a.chunk_log2 ? (1ull << a.chunk_log2) : kChunk;
    // Lane 0 claims the following batch while the warp works on the current
    // one, so the atomic's latency is hidden behind a batch of pairs.
    unsigned long long ahead = 0;
    if (lane == 0) ahead = first_ticket(tbatch);
    for (;;) {
        if (next >= lim) {
            next = __shfl_sync(kFull, ahead, 0);
            lim = next + tbatch;
            if (lane == 0 && next < n) ahead = later_ticket(&a.v->exh_ticket, tbatch, n);
        }
        const unsigned long long q = next++;
        if (q >= n) break;
        const unsigned long long p = a.order ? (unsigned long long)a.order[q] : q;
        PairView pv;
        pv.t = s_t[w]; pv.c = s_c[w];
        src.load(p, s_t[w], s_c[w], pv.tn, pv.cn, pv.dead, lane);
        const uint64_t tid = src.target_id(p);
        __syncwarp();
        {
            uint32_t sw_t = 0, sw_c = 0;
            for (int i = 0; i < pv.tn; i++) sw_t |= c_sweep[pv.t[i] & 0xFFu];
            for (int i = 0; i < pv.cn; i++) sw_c |= c_sweep[pv.c[i] & 0xFFu];
            const uint32_t sw = sw_t | sw_c;   // swept extra registers
            const bool prep = a.sweep == M6502_SWEEP_REFERENCE && __popc(sw) >= 3;
            if (!probe_pair(pv, sw_t, sw_c, prep, tid, p, tc, lane)) {
                if (lane == 0) { a.fail[p] = 1u; probe_rej += src.weight(p); }
                __syncwarp();
                continue;
            }
        }
        Flow fl = dataflow_cached(pv, lane, s_dep, tid, tc);
        const bool rep = a.sweep == M6502_SWEEP_REFERENCE && fl.k >= 3;
        LaneGroups lg;
        if (a.brute) {   // one group: the whole product space, every output
            lg.active = 0; lg.my = 0; lg.maxm = 1u; lg.mybits = 0;
        } else {
            lg = lane_groups(fl, pv.dead, rep, lane);
        }
        const uint32_t brute_bits = cone_bits(fl.swept, rep);
        const bool too_big = a.brute ? brute_bits > kMaxConeBits
                                     : __any_sync(kFull, ((lg.maxm >> lane) & 1u) && lg.mybits > kMaxConeBits);
        if (too_big) {
            if (lane == 0) a.fail[p] = 3u;   // undecided: sweep beyond the cap
            __syncwarp();
            continue;
        }
        if (a.defer_bits && !a.brute &&
            __any_sync(kFull, ((lg.maxm >> lane) & 1u) && lg.mybits > a.defer_bits)) {
            if (lane == 0) a.fail[p] = 4u;   // deferred: a cone above this round's budget
            __syncwarp();
            continue;
        }
        bool ok = true;
        uint32_t big = 0;   // groups (by output lane) left for the work queue
        for (uint32_t rem = lg.maxm; rem && ok;) {
            int o; uint32_t bits, cone; uint64_t mask;
            if (a.brute) { o = 0; bits = brute_bits; cone = fl.swept; mask = cmp_mask(pv.dead); }
            else next_group(lg, rem, lane, o, bits, cone, mask);
            rem &= ~(1u << o);
            const uint64_t total = 1ull << bits;
            const uint64_t end = total <= kSmallSweep ? total : kProbe;
            ok = sweep_cone(pv, cone, fl.swept, rep, mask, 0, end, nullptr, &nstates, lane);
            if (ok && end < total) big |= 1u << o;
        }
        if (ok && big) {
            for (uint32_t rem = big; rem;) {
                int o; uint32_t bits, cone; uint64_t mask;
                if (a.brute) { o = 0; bits = brute_bits; cone = fl.swept; mask = cmp_mask(pv.dead); }
                else next_group(lg, rem, lane, o, bits, cone, mask);
                rem &= ~(1u << o);
                const uint64_t total = 1ull << bits;
                const uint64_t chunk = max(chunk_min, (total + kMaxItemsPerCone - 1) / kMaxItemsPerCone);
                const uint64_t nitems = (total - kProbe + chunk - 1) / chunk;
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(&a.v->items, (unsigned long long)nitems);
                base = __shfl_sync(kFull, base, 0);
                for (uint64_t j = lane; j < nitems; j += 32) {
                    if (base + j >= a.item_cap) break;
                    Item it;
                    it.pair = (uint32_t)p; it.cone = (uint16_t)cone; it.rep = rep ? 1 : 0; it.pad = 0;
                    it.outmask = mask;
                    it.start = kProbe + j * chunk;
                    it.count = min(chunk, total - it.start);
                    a.items[base + j] = it;
                }
            }
        }
        if (lane == 0) a.fail[p] = ok ? 0u : 1u;
        __syncwarp();
    }
    if (lane == 0 && nstates) atomicAdd(&a.cnt->states, nstates);
    if (lane == 0 && probe_rej) atomicAdd(&a.cnt->probe_rejects, probe_rej);
}

// ExhaustiveCheck of the pairs whose compared outputs depend on at most nine
// bits of the swept input, a lane per pair, ahead of k_exhaustive.
//
// The union U of the cones of all compared outputs comes from walking the
// sequences backwards (a set of locations in, the set it depends on out).
// With at most 9 bits, U is one swept register or none, and the carry or
// not: the lane runs target and candidate on every value of it, eight states
// (two packed words) at a time, inputs outside U at the first value of their
// range, and compares every output.  That is exact: U contains each output's
// cone, and the states lie in the sweep domain.  Of the pairs of the full
// length-2 enumeration that the line filter leaves, 99.6 % are decided here;
// the others are listed for k_exhaustive, in which a warp spends about 1,500
// instructions per pair (cone analysis by shuffles, ticket, staging) on 64
// packed words of states.  The line at 9 bits: a lane takes 64 dispatches per
// instruction for 512 states; one more register would make it 16,384.
// Several lanes share a pair (a warp while that fills the chip, else eight:
// lanes whose pairs differ in opcode diverge.  When the line was drawn, four,
// eight, sixteen lanes gave 7.77, 7.19, 7.54 ms for the count at 0xFF, 495, 460,
// 453 us for 20,011 checked pairs, and this enumeration alike).  The same enumeration:
// 0.56 ms for 1.1 M pairs; k_exhaustive took 2.63 ms for 1.36 M.
constexpr int kSmallLanesLog2 = 3;   // lanes per pair once the pairs alone fill the chip: 2^3
__device__ __forceinline__ uint32_t backward(uint32_t locs, uint32_t op, const uint16_t (*dep)[16]) {
    const uint32_t wr = c_wr[op];
    uint32_t r = locs & ~wr;
    for (uint32_t o = locs & wr; o; o &= o - 1) r |= dep[op][__ffs(o) - 1];
    return r;
}

template <class Src, bool LINE>
__global__ void __launch_bounds__(256) k_small(Src src, const unsigned long long* n_pairs_ptr, uint64_t n_cap,
                                               ExhArgs a, uint32_t* __restrict__ order) {
    __shared__ uint16_t s_ins[Src::kMaxT + Src::kMaxC][256];
    __shared__ alignas(16) uint16_t s_dep[NUM_OPS][16];
    const int lane = threadIdx.x & 31;
    const uint64_t n = min((uint64_t)*n_pairs_ptr, n_cap);
    if (blockIdx.x >= n) return;   // no warp of this block has a pair
    for (int i = threadIdx.x; i < (int)NUM_OPS * 2; i += blockDim.x) reinterpret_cast<uint4*>(&s_dep[0][0])[i] = g_dep16[i];
    __syncthreads();
    // Lanes per pair (log2): a warp while that fills the chip, then fewer.
    int g = 5;
    for (uint64_t warps = (uint64_t)gridDim.x * kWarpsPerBlock; g > kSmallLanesLog2 && n > warps; g--) warps <<= 1;
    const uint32_t sub = (uint32_t)lane & ((1u << g) - 1u), lead = (uint32_t)lane - sub;
    const uint32_t group = (g == 5 ? kFull : (1u << (1 << g)) - 1u) << lead;
    // A ticket is up to 16 steps of the warp: with one each, a million pairs
    // wait for 130,000 atomics on one counter.
    const uint32_t per = 32u >> g;
    const uint64_t steps = n / ((uint64_t)gridDim.x * kWarpsPerBlock * per * 4);
    const uint64_t batch = (uint64_t)per * (steps < 1 ? 1 : steps > 16 ? 16 : steps);
    // the pair's sequences: one column of the staging array for its lanes
    uint16_t *st = &s_ins[0][(threadIdx.x & ~31u) + lead], *sc = st + Src::kMaxT * 256;
    unsigned long long nstates = 0, next = 0;
    if (lane == 0) next = first_ticket(batch);
    uint64_t first = 0, upto = 0;
    for (;; first += per) {
        if (first >= upto) {
            first = __shfl_sync(kFull, next, 0);
            if (first >= n) break;
            upto = first + batch;
            if (lane == 0) next = later_ticket(&a.v->small_ticket, batch, n);
        }
        const uint64_t p = first + (uint32_t)(lane >> g);
        int tn = 0, cn = 0;
        uint32_t dead = 0, swx = 0, written = 0;
        if (p < n && sub == 0) src.load_lane(p, st, sc, 256, tn, cn, dead);
        const uint32_t head = __shfl_sync(kFull, (uint32_t)tn | (uint32_t)cn << 8 | dead << 16, (int)lead);
        tn = (int)(head & 0xFFu);
        cn = (int)((head >> 8) & 0xFFu);
        dead = head >> 16;
        __syncwarp();
        for (int i = 0; i < tn; i++) { const uint32_t op = st[i * 256] & 0xFFu; swx |= c_sweep[op]; written |= c_wr[op]; }
        for (int i = 0; i < cn; i++) { const uint32_t op = sc[i * 256] & 0xFFu; swx |= c_sweep[op]; written |= c_wr[op]; }
        const uint32_t live = written & ~(((dead & 0x0Fu) << L_C) | ((dead >> 6) << L_V));
        uint32_t ut = live, uc = live;
        for (int i = tn - 1; i >= 0; i--) ut = backward(ut, st[i * 256] & 0xFFu, s_dep);
        for (int i = cn - 1; i >= 0; i--) uc = backward(uc, sc[i * 256] & 0xFFu, s_dep);
        const uint32_t u = (ut | uc) & (swx | LB(L_A) | LB(L_C)), reg = u & ~LB(L_C);
        const bool rep = a.sweep == M6502_SWEEP_REFERENCE && __popc(swx) >= 3;
        const bool small = p < n && cone_bits(u, rep) <= 9;
        // LINE: wider pairs meet the line states first (of all their registers;
        // not under the reduced sweep), and most that are wrong end here: 4,096
        // length-3 targets 1,165 -> 917 us, length-2 Go enumeration 4.72 -> 4.22
        // ms.  Not for survivors that the line filter has seen (5 % slower at
        // 0xFF, nothing to find).
        const bool wide = p < n && !small, line = LINE && wide && !rep;
        const uint32_t take = line ? swx | LB(L_A) : reg;   // registers that vary
        auto mask = [&](uint32_t l) { return (take & LB(l)) ? 0xFFFFFFFFu : 0u; };
        const uint32_t ma = mask(L_A), mx = mask(L_X), my = mask(L_Y), ms = mask(L_S), mm = mask(L_M), m0 = mask(L_S0),
                       m1 = mask(L_S1);
        const uint32_t bs = (swx & LB(L_S)) ? 0u : 0xFDu * kB1;   // S at its first value
        const uint32_t pm = (kPMask & ~dead & 0xFFu) * kB1;
        const bool rreg = rep && !(reg & LB(L_A));
        const uint32_t words = line ? 64u : reg == 0 ? 1u : rreg ? 8u : 64u;   // packed words of the register's values
        const uint32_t total = line ? words : words << ((u & LB(L_C)) ? 1 : 0);
        bool open = (small && live) || line, differ = false;   // no live output is written: equal
        for (uint32_t q = 2 * sub; __any_sync(kFull, open); q += 2u << g) {
            uint32_t d = 0;
            if (open && q < total) {
                St t[2], c[2];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const uint32_t j = min(q + k, total - 1), i0 = (j & (words - 1)) * 4;
                    uint32_t v = i0 * kB1 + 0x03020100u;
                    if (rreg) v = c_rep[i0] | (c_rep[i0 + 1] << 8) | (c_rep[i0 + 2] << 16) | (c_rep[i0 + 3] << 24);
                    St in{v & ma, v & mx, v & my, j >= words ? kB1 : 0u, (v & ms) | bs, v & mm, v & m0, v & m1};
                    if (line) {
                        const uint32_t* w = c_line[j];
                        in = St{w[0], w[1] & mx, w[2] & my, w[3], (w[4] & ms) | bs, w[5] & mm, w[6] & m0, w[7] & m1};
                    }
                    t[k] = c[k] = in;
                }
                for (int i = 0; i < tn; i++) exec_x4n(t, st[i * 256]);
                for (int i = 0; i < cn; i++) exec_x4n(c, sc[i * 256]);
#pragma unroll
                for (int k = 0; k < 2; k++)
                    d |= (t[k].a ^ c[k].a) | (t[k].x ^ c[k].x) | (t[k].y ^ c[k].y) | ((t[k].p ^ c[k].p) & pm) |
                         (t[k].s ^ c[k].s) | (t[k].m ^ c[k].m) | (t[k].s0 ^ c[k].s0) | (t[k].s1 ^ c[k].s1);
                nstates += 4 * min(2u, total - q);
            }
            const unsigned bad = __ballot_sync(kFull, d != 0) & group;
            differ = differ || bad;
            open = open && !differ && q - 2 * sub + (2u << g) < total;   // the same for all lanes of the pair
        }
        if (p < n && sub == 0 && (small || differ)) a.fail[p] = !differ ? 0u : small ? 1u : kFailLine;
        const unsigned left = __ballot_sync(kFull, wide && !differ && sub == 0);
        if (left) {
            unsigned long long b = 0;
            if (lane == 0) b = atomicAdd(&a.v->small_left, (unsigned long long)__popc(left));
            b = __shfl_sync(kFull, b, 0) + __popc(left & ((1u << lane) - 1u));
            if (((left >> lane) & 1u) && b < n_cap) order[b] = (uint32_t)p;
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) nstates += __shfl_down_sync(kFull, nstates, o);
    if (lane == 0 && nstates) atomicAdd(&a.cnt->states, nstates);
}

template <class Src>
__global__ void __launch_bounds__(256) k_exh_items(Src src, ExhArgs a) {
    __shared__ uint16_t s_t[kWarpsPerBlock][kMaxSeq], s_c[kWarpsPerBlock][kMaxSeq];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t n = min((uint64_t)a.v->items, a.item_cap);
    unsigned long long nstates = 0;
    if (blockIdx.x >= n) return;   // the block's warps would find nothing
    for (;;) {
        unsigned long long q = 0;
        if (lane == 0) q = atomicAdd(&a.v->item_ticket, 1ull);
        q = __shfl_sync(kFull, q, 0);
        if (q >= n) break;
        const Item it = a.items[q];
        volatile uint32_t* flag = a.fail + it.pair;
        uint32_t fv = lane == 0 ? *flag : 0u;
        if (__shfl_sync(kFull, fv, 0)) continue;
        PairView pv;
        pv.t = s_t[w]; pv.c = s_c[w];
        src.load(it.pair, s_t[w], s_c[w], pv.tn, pv.cn, pv.dead, lane);
        __syncwarp();
        uint32_t swept = LB(L_A) | LB(L_C);
        for (int i = 0; i < pv.tn; i++) swept |= c_sweep[pv.t[i] & 0xFFu];
        for (int i = 0; i < pv.cn; i++) swept |= c_sweep[pv.c[i] & 0xFFu];
        const bool ok = sweep_cone(pv, it.cone, swept, it.rep != 0, it.outmask, it.start, it.start + it.count, flag,
                                   &nstates, lane);
        if (!ok && lane == 0) *flag = 1u;
        __syncwarp();
    }
    if (lane == 0 && nstates) atomicAdd(&a.cnt->states, nstates);
}

// Algorithmic work of one passing pair under the fixed measurement
// convention: every state of the product sweep (2^(9+8k), or 512 x 32^k for
// the reduced sweep) costs 10 ops per executed instruction + 3 per compare.
__device__ __forceinline__ unsigned long long algo_ops(const uint16_t* t, uint32_t tn, const uint16_t* c,
                                                       uint32_t cn, uint32_t sweep_mode) {
    uint32_t sw = 0;
    for (uint32_t i = 0; i < tn; i++) sw |= c_sweep[t[i] & 0xFFu];
    for (uint32_t i = 0; i < cn; i++) sw |= c_sweep[c[i] & 0xFFu];
    uint32_t k = (uint32_t)__popc(sw);
    uint32_t bits = 9 + k * ((sweep_mode == M6502_SWEEP_REFERENCE && k >= 3) ? 5u : 8u);
    return (1ull << bits) * (unsigned long long)(10 * (tn + cn) + 3);
}

__device__ __forceinline__ void count_failed(Counters* cnt, unsigned long long n) {
    if ((uint32_t)n) atomicAdd(&cnt->undecided, n & 0xFFFFFFFFull);
    if (n >> 32) atomicAdd(&cnt->probe_rejects, n >> 32);
}

// CUDA semantics: every pair of a passing record is a rule; its target is
// ids[t], or tbase + t (the pass-local index made global) without ids.  The
// rules of a record that stands for several candidates are written by the
// whole warp, one member per lane.
__global__ void k_emit_all(const Surv* __restrict__ surv, const unsigned long long* n_ptr, uint64_t n_cap,
                           const uint32_t* __restrict__ fail, const uint64_t* __restrict__ ids, uint64_t tbase,
                           uint32_t run_dead, m6502_rule* __restrict__ rules, uint64_t rcap,
                           unsigned long long* rule_ctr, Counters* cnt, int check_exh,
                           const uint16_t* __restrict__ targets, uint32_t tlen, uint32_t sweep_mode,
                           const CandGroups* __restrict__ groups) {
    const uint64_t n = min((uint64_t)*n_ptr, n_cap);
    const int lane = threadIdx.x & 31;
    const uint16_t* mult = groups ? groups->mult : nullptr;
    unsigned long long npass = 0, algo = 0, nund = 0;   // nund: undecided, and rejected by the line states << 32
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t p = base + threadIdx.x;
        const uint32_t f = p < n && check_exh ? fail[p] : 0u;
        bool pass = p < n && f == 0;
        const Surv s = p < n ? surv[p] : Surv{0, 0};
        const uint32_t w = p < n ? surv_weight(s.c, mult) : 0u;
        nund += f == 3u ? w : f == kFailLine ? (unsigned long long)w << 32 : 0u;   // counted, not rules
        m6502_rule r;
        memset(&r, 0, sizeof r);
        const uint32_t idx = s.c & 0x7FFFFFu;
        if (pass) {
            r.target = ids ? ids[s.t] : tbase + s.t;
            r.dead_flags = (uint8_t)run_dead;
            if (s.c & kSurvLen2) { r.cand_len = 2; r.cand[0] = c_tab[idx / kNumInsns]; r.cand[1] = c_tab[idx % kNumInsns]; }
            else { r.cand_len = 1; r.cand[0] = c_tab[idx]; }
            npass += w;
            if (check_exh) algo += w * algo_ops(targets + (uint64_t)s.t * tlen, tlen, r.cand, r.cand_len, sweep_mode);
        }
        const unsigned vote = __ballot_sync(kFull, pass);
        if (!vote) continue;
        uint32_t at = pass ? w : 0u;   // inclusive running count of the warp's rules
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(kFull, at, o);
            at += lane >= o ? x : 0u;
        }
        unsigned long long b = 0;
        if (lane == 31) b = atomicAdd(rule_ctr, (unsigned long long)at);
        b = __shfl_sync(kFull, b, 31);
        if (rcap == 0) continue;       // counted only
        const unsigned long long mine = b + at - (pass ? w : 0u);
        if (pass && w == 1 && mine < rcap) rules[mine] = r;
        for (unsigned many = __ballot_sync(kFull, pass && w > 1); many; many &= many - 1) {
            const int l = __ffs(many) - 1;
            const uint32_t mw = __shfl_sync(kFull, w, l), c = __shfl_sync(kFull, idx, l);
            const unsigned long long m0 = __shfl_sync(kFull, mine, l);
            m6502_rule q;
            memset(&q, 0, sizeof q);
            q.target = __shfl_sync(kFull, (unsigned long long)r.target, l);
            q.dead_flags = (uint8_t)run_dead;
            q.cand_len = 1;
            for (uint32_t j = lane; j < mw; j += 32) {
                q.cand[0] = c_tab[groups->member[groups->first[c] + j]];
                if (m0 + j < rcap) rules[m0 + j] = q;
            }
        }
    }
    for (int o = 16; o; o >>= 1) {
        npass += __shfl_down_sync(kFull, npass, o);
        algo += __shfl_down_sync(kFull, algo, o);
        nund += __shfl_down_sync(kFull, nund, o);
    }
    if (lane == 0 && npass) atomicAdd(&cnt->exh_pass, npass);
    if (lane == 0 && algo) atomicAdd(&cnt->algo, algo);
    if (lane == 0 && nund) count_failed(cnt, nund);
}

// Go-order rank of a survivor's candidate; length-2 candidates (bit 28)
// come after every length-1 candidate (worker.go:122: lengths ascending).
__device__ __forceinline__ uint32_t go_rank_of(uint32_t code) {
    const uint32_t idx = code & 0x7FFFFFu;
    if (code & kSurvLen2) return (1u << 28) | (c_gorank[idx / kNumInsns] * kNumInsns + c_gorank[idx % kNumInsns]);
    return c_gorank[idx];
}

// Go semantics: first passing candidate per target and pass, in Go order
// (shorter candidates first, then Go enumeration order).
__global__ void k_go_select(const Surv* __restrict__ surv, const unsigned long long* n_ptr, uint64_t n_cap,
                            const uint32_t* __restrict__ fail, uint32_t nt, uint32_t* __restrict__ best,
                            Counters* cnt, const uint16_t* __restrict__ targets, uint32_t tlen,
                            uint32_t sweep_mode) {
    const uint64_t n = min((uint64_t)*n_ptr, n_cap);
    unsigned long long npass = 0, algo = 0, nund = 0;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (uint64_t)gridDim.x * blockDim.x) {
        if (const uint32_t f = fail[p]) {   // undecided pairs count as not passing
            nund += f == 3u ? 1ull : f == kFailLine ? 1ull << 32 : 0ull;
            continue;
        }
        npass++;
        Surv s = surv[p];
        const uint32_t idx = s.c & 0x7FFFFFu, key = go_rank_of(s.c);
        uint64_t pass = (s.c & kSurvMasked) ? 1 : 0;
        atomicMin(&best[pass * nt + s.t], key);
        uint16_t cand[2];
        uint32_t cn = (s.c & kSurvLen2) ? 2u : 1u;
        if (cn == 2) { cand[0] = c_tab[idx / kNumInsns]; cand[1] = c_tab[idx % kNumInsns]; }
        else cand[0] = c_tab[idx];
        algo += algo_ops(targets + (uint64_t)s.t * tlen, tlen, cand, cn, sweep_mode);
    }
    for (int o = 16; o; o >>= 1) {   // one atomic per warp: one per thread took 250 us of a 2 M target pass
        npass += __shfl_down_sync(kFull, npass, o);
        algo += __shfl_down_sync(kFull, algo, o);
        nund += __shfl_down_sync(kFull, nund, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (npass) atomicAdd(&cnt->exh_pass, npass);
        if (algo) atomicAdd(&cnt->algo, algo);
        if (nund) count_failed(cnt, nund);
    }
}

__global__ void k_go_emit(const uint32_t* __restrict__ best, uint32_t nt, const uint16_t* __restrict__ targets,
                          uint32_t tlen, const uint64_t* __restrict__ ids, uint64_t tbase,
                          m6502_rule* __restrict__ rules, uint64_t rcap, Counters* cnt) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
        for (int pass = 0; pass < 2; pass++) {
            uint32_t key = best[(uint64_t)pass * nt + t];
            if (key == 0xFFFFFFFFu) continue;
            m6502_rule r;
            memset(&r, 0, sizeof r);
            r.target = ids ? ids[t] : tbase + t;
            if (key >> 28) {
                uint32_t rk = key & 0x0FFFFFFFu;
                r.cand_len = 2; r.cand[0] = c_gotab[rk / kNumInsns]; r.cand[1] = c_gotab[rk % kNumInsns];
            } else {
                r.cand_len = 1; r.cand[0] = c_gotab[key];
            }
            if (pass == 1) {   // FlagDiff over the QC vectors (verifier.go:591-604)
                uint32_t fd = 0;
                for (int v = 0; v < 8; v++) {
                    St a = unpack(c_vec[v]), b = a;
                    for (uint32_t i = 0; i < tlen; i++) exec(a, targets[(uint64_t)t * tlen + i]);
                    for (int i = 0; i < r.cand_len; i++) exec(b, r.cand[i]);
                    fd |= (a.p ^ b.p) & kPMask;
                }
                r.dead_flags = (uint8_t)fd;
            }
            unsigned long long idx = atomicAdd(&cnt->rules, 1ull);
            if (idx < rcap) rules[idx] = r;
        }
    }
}

// ---- Go semantics: verification in Go order, in rounds ----
//
// The Go worker stops at the first candidate (in Go order) that passes
// ExhaustiveCheck (worker.go:125-173).  Every survivor has an ordinal within
// its (target, pass) in Go order; round r verifies, for every (target, pass)
// not yet settled, the next block of its survivors (block sizes 64, 512,
// 4096, ...), and the smallest passing rank of a block settles it.  Only the
// blocks up to the first pass are swept.  The joins meet the candidates in Go
// order and number them as they go (GoCount); the scan's survivors are sorted.

// Sort key of a scanned survivor: target << 30 | masked pass << 29 | go_rank_of.
// Entries from the survivor count up to the capacity get `pad`, which sorts
// after every real key.
__global__ void k_go_keys(const Surv* __restrict__ surv, const unsigned long long* n_ptr, uint64_t cap, uint64_t pad,
                          uint64_t* __restrict__ keys) {
    const uint64_t n = min((uint64_t)*n_ptr, cap);
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < cap; p += (uint64_t)gridDim.x * blockDim.x) {
        if (p >= n) { keys[p] = pad; continue; }
        const Surv s = surv[p];
        keys[p] = ((uint64_t)s.t << 30) | ((uint64_t)((s.c & kSurvMasked) ? 1u : 0u) << 29) | go_rank_of(s.c);
    }
}

// The sorted survivors, rebuilt from their keys, with their ordinals.
__global__ void k_go_ord(const uint64_t* __restrict__ keys, const unsigned long long* n_ptr, uint64_t cap,
                         Surv* __restrict__ surv, uint32_t* __restrict__ ord, Counters* __restrict__ cnt) {
    const uint64_t n = min((uint64_t)*n_ptr, cap);
    unsigned long long mx = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i], g = k >> 29;
        uint64_t lo = 0, hi = i;   // first index of the group
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if ((keys[mid] >> 29) < g) lo = mid + 1; else hi = mid;
        }
        surv[i] = Surv{(uint32_t)(k >> 30), c_goidx[(uint32_t)k & 0x1FFFFFFFu] | ((g & 1u) ? kSurvMasked : 0u)};
        ord[i] = (uint32_t)(i - lo);
        mx = max(mx, (unsigned long long)(i - lo));
    }
    for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_down_sync(kFull, mx, o));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(&cnt->max_ord, mx);
}

// The survivors of one round: ordinals [lo, hi) of what is still open.  A
// round whose first ordinal lies past the largest one finds nothing.
__global__ void k_go_round(const Surv* __restrict__ surv, const uint32_t* __restrict__ ord,
                           const unsigned long long* n_ptr, uint64_t cap, uint32_t lo, uint32_t hi,
                           const uint32_t* __restrict__ best, uint32_t nt, Surv* __restrict__ out,
                           const Counters* __restrict__ cnt, VerifyCounters* __restrict__ v) {
    if ((unsigned long long)lo > cnt->max_ord) return;
    const uint64_t n = min((uint64_t)*n_ptr, cap);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t o = ord[i];
        if (o < lo || o >= hi) continue;
        const Surv s = surv[i];
        const uint32_t kind = (s.c & kSurvMasked) ? 1u : 0u;
        if (best[(uint64_t)kind * nt + s.t] != 0xFFFFFFFFu) continue;   // settled by an earlier round
        out[atomicAdd(&v->n, 1ull)] = s;
    }
}

// Before the length-2 phase resets the survivor counter.
__global__ void k_mark_phase(Counters* cnt) { cnt->surv1 = cnt->surv; }

// Pairwise QC / MidCheck / FlagDiff: warp per pair, lane = vector.
__global__ void __launch_bounds__(256) k_pair_vectors(CsrSource src, uint64_t n, uint8_t* __restrict__ out,
                                                       uint8_t* __restrict__ fdiff) {
    __shared__ uint16_t s_t[kWarpsPerBlock][kMaxSeq], s_c[kWarpsPerBlock][kMaxSeq];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint64_t p = (uint64_t)blockIdx.x * kWarpsPerBlock + w; p < n; p += (uint64_t)gridDim.x * kWarpsPerBlock) {
        int tn, cn;
        uint32_t dead;
        src.load(p, s_t[w], s_c[w], tn, cn, dead, lane);
        __syncwarp();
        St a = unpack(c_vec[lane]), b = a;
        for (int i = 0; i < tn; i++) exec(a, s_t[w][i]);
        for (int i = 0; i < cn; i++) exec(b, s_c[w][i]);
        uint64_t x = pack(a) ^ pack(b);
        bool eq = (x & cmp_mask(dead)) == 0;
        unsigned ev = __ballot_sync(kFull, eq);
        bool nonp = (x & 0xFFFFFFFF00FFFFFFull) == 0;
        unsigned nv = __ballot_sync(kFull, nonp);
        uint32_t pd = (lane < 8) ? ((uint32_t)(x >> 24) & kPMask) : 0u;
        for (int o = 16; o; o >>= 1) pd |= __shfl_xor_sync(kFull, pd, o);
        if (lane == 0) {
            uint8_t r = 0;
            if ((ev & 0xFFu) == 0xFFu) r |= 1;
            if (ev == kFull) r |= 2;
            out[p] = r;
            if (fdiff) fdiff[p] = (uint8_t)(((nv & 0xFFu) == 0xFFu) ? pd : 0u);
        }
        __syncwarp();
    }
}

// The pairs' verdict bits: the vector checks asked for (already in out, when
// vec is not 0) and ExhaustiveCheck's verdict.
__global__ void k_pair_verdicts(uint64_t n, uint32_t vec, const uint32_t* __restrict__ fail, uint8_t* __restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t r = vec ? out[i] & vec : 0u;
        if (fail) r |= fail[i] == 0 ? 4u : fail[i] == 3 ? 8u : 0u;   // 3: undecided
        out[i] = (uint8_t)r;
    }
}

// Runs sequence i on packed input state in[i] (thread per sequence).
__global__ void k_exec_batch(CsrSeqs src, uint64_t n, const uint64_t* __restrict__ in, uint64_t* __restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        St s = unpack(in[i]);
        for (uint32_t k = src.off[i]; k < src.off[i + 1]; k++) exec(s, src.ins[k]);
        out[i] = pack(s);
    }
}

// Sets *bad when an instruction word's opcode is outside the table (the
// search's input check for targets in device memory).
__global__ void k_check_ops(const uint16_t* __restrict__ ins, uint64_t n, uint32_t* __restrict__ bad) {
    bool b = false;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        b |= (ins[i] & 0xFFu) >= (uint32_t)NUM_OPS;
    if (__any_sync(kFull, b) && (threadIdx.x & 31) == 0) *bad = 1u;
}

// Pruned target enumeration: ids in [id0, id1) of the length-L space,
// compacted into targets/ids (order unspecified).
__global__ void k_enum_targets(uint64_t id0, uint64_t id1, uint32_t len, uint16_t* __restrict__ targets,
                               uint64_t* __restrict__ ids, uint64_t cap, unsigned long long* count) {
    const int lane = threadIdx.x & 31;
    for (uint64_t base = id0 + (uint64_t)blockIdx.x * blockDim.x; base < id1; base += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t id = base + threadIdx.x;
        uint16_t s[3] = {0, 0, 0};
        bool keep = false;
        if (id < id1) {
            uint64_t r = id;
            for (int k = (int)len - 1; k >= 0; k--) { s[k] = c_tab[r % kNumInsns]; r /= kNumInsns; }
            keep = !should_prune(s, (int)len);
        }
        unsigned vote = __ballot_sync(kFull, keep);
        if (!vote) continue;
        int leader = __ffs(vote) - 1;
        unsigned long long b = 0;
        if (lane == leader) b = atomicAdd(count, (unsigned long long)__popc(vote));
        b = __shfl_sync(kFull, b, leader);
        if (keep) {
            unsigned long long idx = b + __popc(vote & ((1u << lane) - 1u));
            if (idx < cap) {
                for (uint32_t k = 0; k < len; k++) targets[idx * len + k] = s[k];
                ids[idx] = id;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Fixed-scratch variant of the exhaustive check (m6502_exhaustive_static)
// ---------------------------------------------------------------------------
// For callers that cannot allocate device memory, the scratch of this one
// variant -- a ticket counter and one fail flag per pair -- lives in a fixed
// array compiled into the library.  Every GPU that loads the library holds
// it (a little over 4 MiB) until the process exits.  All calls share it, so
// calls that overlap on the GPU race; each call clears the part that must
// start at zero.
constexpr uint64_t kStaticMaxPairs = M6502_STATIC_MAX_PAIRS;
constexpr uint32_t kStaticMaxConeBits = 28;   // in-warp sweeps only: at most 2^28 states per cone

struct StaticScratch {
    Counters cnt;
    uint32_t fail[kStaticMaxPairs];
};

static __device__ __align__(256) unsigned char g_static_scratch[sizeof(StaticScratch)];

// CSR pairs in caller-owned device memory.  The inputs were never seen by
// the host, so lengths and opcodes are validated here; an invalid pair is
// reported instead of evaluated.
struct StaticCsrSource {
    const uint16_t* t_ins;
    const uint32_t* t_off;
    const uint16_t* c_ins;
    const uint32_t* c_off;
    uint32_t dead_;
    __device__ bool load(uint64_t p, uint16_t* st, uint16_t* sc, int& tn, int& cn, uint32_t& dead,
                         int lane) const {
        uint32_t t0 = t_off[p], t1 = t_off[p + 1], c0 = c_off[p], c1 = c_off[p + 1];
        dead = dead_;
        if (t1 <= t0 || c1 <= c0 || t1 - t0 > (uint32_t)kMaxSeq || c1 - c0 > (uint32_t)kMaxSeq) return false;
        tn = (int)(t1 - t0);
        cn = (int)(c1 - c0);
        bool ok = true;
        if (lane < tn) { st[lane] = t_ins[t0 + lane]; ok = (st[lane] & 0xFFu) < NUM_OPS; }
        if (lane < cn) { sc[lane] = c_ins[c0 + lane]; ok = ok && (sc[lane] & 0xFFu) < NUM_OPS; }
        return __all_sync(kFull, ok);
    }
};

// One pair per warp, every cone swept in-warp (no work-item queue, so the
// only scratch is the ticket and the fail flags).  fail: 0 equivalent,
// 1 not equivalent, 2 invalid pair, 3 undecided (a cone beyond 2^28 states).
__global__ void __launch_bounds__(256) k_exhaustive_static(StaticCsrSource src, uint64_t n, uint32_t sweep,
                                                            StaticScratch* scr) {
    __shared__ uint16_t s_t[kWarpsPerBlock][kMaxSeq], s_c[kWarpsPerBlock][kMaxSeq];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long nstates = 0;
    for (;;) {
        unsigned long long p = 0;
        if (lane == 0) p = atomicAdd(&scr->cnt.v[0][0].exh_ticket, 1ull);
        p = __shfl_sync(kFull, p, 0);
        if (p >= n) break;
        PairView pv;
        pv.t = s_t[w]; pv.c = s_c[w];
        pv.tn = pv.cn = 0;
        bool valid = src.load(p, s_t[w], s_c[w], pv.tn, pv.cn, pv.dead, lane);
        __syncwarp();
        if (!valid) {
            if (lane == 0) scr->fail[p] = 2u;
            continue;
        }
        Flow fl = dataflow(pv, lane);
        const bool rep = sweep == M6502_SWEEP_REFERENCE && fl.k >= 3;
        Groups g = make_groups(fl, pv.dead, rep, false, lane);
        bool too_big = false;
        for (int i = 0; i < g.n; i++) too_big = too_big || g.bits[i] > kStaticMaxConeBits;
        if (too_big) {
            if (lane == 0) scr->fail[p] = 3u;   // undecided: one warp cannot sweep it in bounded time
            __syncwarp();
            continue;
        }
        bool ok = true;
        for (int i = 0; i < g.n && ok; i++) {
            Fields f = make_fields(g.cone[i], fl.swept, rep);
            ok = sweep_states<1>(pv, f, g.mask[i], 0, 1ull << g.bits[i], nullptr, &nstates, lane);
        }
        if (lane == 0) scr->fail[p] = ok ? 0u : 1u;
        __syncwarp();
    }
}

__global__ void k_static_verdicts(const StaticScratch* scr, uint64_t n, uint8_t* __restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t f = scr->fail[i];
        out[i] = f == 0 ? 1 : (f == 1 ? 0 : (f == 3 ? 0xFE : 0xFF));
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
};

}  // namespace

struct m6502_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t sev[6] = {};   // stage boundaries of one pass
    cudaEvent_t sev2[6] = {};  // stage boundaries of the length-2 candidate phase
    cudaEvent_t aev[6 * kMaxAsyncPasses] = {};   // stage boundaries of the queued passes
    struct SearchGraph {       // the queued passes of the last search, recorded one by one
        std::vector<cudaGraphExec_t> exec;
        std::vector<uint64_t> key;   // everything the recorded launches depend on
        bool broken = false;         // recording failed once: launch directly from then on
        std::string why;             // the error that stopped recording
    } graph;
    struct PassGraph {         // one recorded pass of the pass-by-pass path (Go semantics,
        cudaGraphExec_t exec = nullptr;   // length-2 candidates, enumeration)
        std::vector<uint64_t> key;
        uint64_t stamp = 0;
    };
    PassGraph pass_graphs[8];
    uint64_t pass_graph_clock = 0;
    DevBuf cnt_slots;          // Counters of the queued passes
    DevBuf tall;               // host targets of a queued search, copied to the device pass by pass
    DevBuf opflag;             // k_check_ops result
    cudaStream_t copy = nullptr;                  // host targets of the next pass, beside the kernels of this one
    cudaEvent_t cev[kMaxAsyncPasses] = {};        // its copies
    DevBuf pairs_io;                              // m6502_check_pairs: inputs, then results, in one block each way
    void* h_io = nullptr;                         // page-locked side of it
    size_t h_io_bytes = 0;
    std::string err;
    bool failed = false;                          // this call reported an error (see Call)
    std::mutex mu;
    int sms = 148;
    int exh_blocks = 0, exh_item_blocks = 0, qc_blocks = 0, fp_blocks = 0, small_blocks = 0;
    int exh_occ[5] = {};       // resident blocks per SM of k_exhaustive<SurvSource, MINB>, by MINB
    m6502_tune tune{4, 4, 11, 1, {0, 0, 0, 0}};   // scheduling knobs (m6502_tune_set / m6502_autotune)
    uint64_t pass_targets = 1ull << 21;
    bool ready = false;
    DevBuf cfp1, cmeta1, targets, ids, tfp, tmeta, surv, fail, items, rules, cnt, best, pins, poffs,
        enum_count;
    std::vector<m6502_rule> staging;
    DevBuf cfp4;                      // packed outputs of the length-1 candidates: [2863][8 groups of 4 vectors][8 fields]
    std::vector<uint32_t> h_cfp4;     // host copy
    std::vector<uint8_t> h_cmeta;
    std::vector<uint16_t> h_tab;      // instructions, CUDA order (host copy)
    std::vector<uint32_t> h_gorank;   // Go-order rank of each
    uint32_t join_longest[256] = {};  // most candidates of one entry of the Go-semantics table
    DevBuf go_keys, go_keys2, go_ord, go_round, go_sort_tmp;   // Go-order verification rounds
    DevBuf jitems;                                             // chunks of long length-2 equal ranges
    DevBuf order;                                              // k_small: the pairs it left
    DevBuf match;                                              // k_qc_join: the targets that match
    JoinTable* join_tab[2][256] = {};             // by semantics and dead-flags mask
    CandGroups* join_groups[256] = {};            // of the CUDA-semantics tables
    uint32_t* join_lines[256] = {};               // line hashes of the candidates, [64 register sets][2863]
    bool join_built[2][256] = {};                 // tables and groups are filled, or their copies are on the stream
    bool lines_built[256] = {};
    std::vector<void*> table_blocks;              // the memory of these tables (see table_mem)
    size_t table_used = 0;                        // of the last block
    struct Cand2Table {            // sorted (key, entry) of all length-2 sequences for one mask
        uint32_t dead = 0xFFFFFFFFu;
        uint32_t longest = 0;      // longest range of one key
        uint64_t salt = 0;
        DevBuf keys, idx, pw;
        uint64_t stamp = 0;
    } cand2[4];                    // least recently used mask is rebuilt
    uint64_t cand2_clock = 0;
    DevBuf c2_keys_in, c2_idx_in, c2_sort_tmp;
    DevBuf st_tins, st_toffs, st_tout, st_tbytes, st_chains, st_entries, st_vidx, st_proven, st_cnt, st_pidx,
        st_mex, st_probs, st_traj, st_row;
    DevBuf st_keys, st_keys2, st_vals2, st_rep, st_ord, st_verdict, st_vlist, st_vpos, st_sort_tmp, st_vphase,
        st_pphase, st_live, st_rounds, st_proven_was;
};

namespace {

int set_err(m6502_ctx* ctx, int code, const std::string& msg) {
    ctx->err = msg;
    ctx->failed = ctx->failed || code != M6502_OK;
    return code;
}

// A call into the context: holds its lock, and when the call failed ends what
// it queued before it returns.  Copies from and to the caller's memory (which
// the device reads and writes by itself where it is page-locked) do not
// outlive the call, the next one does not overwrite buffers that kernels still
// read, and its launch checks do not meet this call's error.
struct Call {
    m6502_ctx* ctx;
    std::lock_guard<std::mutex> lk;
    explicit Call(m6502_ctx* c) : ctx(c), lk(c->mu) { ctx->failed = false; }
    ~Call() {
        if (!ctx->failed) return;
        cudaStreamSynchronize(ctx->copy);
        cudaStreamSynchronize(ctx->stream);
        cudaGetLastError();
    }
};

#define CK(call)                                                                            \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess)                                                              \
            return set_err(ctx, e_ == cudaErrorMemoryAllocation ? M6502_E_NOMEM : M6502_E_CUDA, \
                           std::string(#call) + ": " + cudaGetErrorString(e_));             \
    } while (0)

#define CKL(what)                                                                           \
    do {                                                                                    \
        cudaError_t e_ = cudaGetLastError();                                                \
        if (e_ != cudaSuccess)                                                              \
            return set_err(ctx, M6502_E_CUDA, std::string("launch ") + what + ": " +        \
                                                  cudaGetErrorString(e_));                  \
    } while (0)

int ensure(m6502_ctx* ctx, DevBuf& b, size_t bytes) {
    if (b.bytes >= bytes && b.p) return M6502_OK;
    if (b.p) { cudaFree(b.p); b.p = nullptr; b.bytes = 0; }
    size_t want = std::max<size_t>(bytes, 256);
    CK(cudaMalloc(&b.p, want));
    b.bytes = want;
    return M6502_OK;
}

#define TRY(x)                      \
    do {                            \
        int rc_ = (x);              \
        if (rc_ != M6502_OK) return rc_; \
    } while (0)

// ExhaustiveCheck over survivors, up to the work items, with the context's
// knobs: ticket batch and work-item size in the arguments, the register-cap
// variant and its persistent grid (SMs x resident blocks).  Brute force
// sweeps every pair's whole product in k_exhaustive.
// `filtered`: the pairs come through the line filter.
int launch_exh(m6502_ctx* ctx, const SurvSource& src, const unsigned long long* n_ptr, uint64_t cap, ExhArgs ea,
               bool filtered = false) {
    ea.ticket_batch = ctx->tune.ticket_batch;
    ea.chunk_log2 = ctx->tune.chunk_log2;
    if (!ea.brute) {
        if (filtered)
            k_small<SurvSource, false><<<ctx->small_blocks, 256, 0, ctx->stream>>>(src, n_ptr, cap, ea, (uint32_t*)ctx->order.p);
        else
            k_small<SurvSource, true><<<ctx->small_blocks, 256, 0, ctx->stream>>>(src, n_ptr, cap, ea, (uint32_t*)ctx->order.p);
        CKL("k_small");
        ea.order = (const uint32_t*)ctx->order.p;
        n_ptr = &ea.v->small_left;
    }
    const int minb = (int)ctx->tune.exh_minb;
    const unsigned grid = (unsigned)(ctx->sms * ctx->exh_occ[minb >= 2 && minb <= 4 ? minb : 4]);
    if (minb == 2)
        k_exhaustive<SurvSource, 2><<<grid, 256, 0, ctx->stream>>>(src, n_ptr, cap, ea);
    else if (minb == 3)
        k_exhaustive<SurvSource, 3><<<grid, 256, 0, ctx->stream>>>(src, n_ptr, cap, ea);
    else
        k_exhaustive<SurvSource, 4><<<grid, 256, 0, ctx->stream>>>(src, n_ptr, cap, ea);
    CKL("k_exhaustive");
    return M6502_OK;
}

// ExhaustiveCheck of n pairs from another source, work items included; n is
// the value at n_ptr, at most cap.
template <class Src>
int launch_verify(m6502_ctx* ctx, const Src& src, const unsigned long long* n_ptr, uint64_t cap, ExhArgs ea) {
    // A block per pair while that leaves blocks idle, then every resident one: a
    // thread per pair as the size filled half the chip at 20,011 pairs and one
    // SM at 48 (335 -> 278 and 135 -> 116 us, with the tickets above).
    const uint64_t blocks = std::max<uint64_t>(cap, 1);
    if (!ea.brute) {
        k_small<Src, true><<<(unsigned)std::min<uint64_t>(ctx->small_blocks, blocks), 256, 0, ctx->stream>>>(
            src, n_ptr, cap, ea, (uint32_t*)ctx->order.p);
        CKL("k_small");
        ea.order = (const uint32_t*)ctx->order.p;
        n_ptr = &ea.v->small_left;
    }
    k_exhaustive<Src><<<(unsigned)std::min<uint64_t>(ctx->exh_blocks, blocks), 256, 0, ctx->stream>>>(src, n_ptr, cap, ea);
    CKL("k_exhaustive");
    k_exh_items<Src><<<ctx->exh_item_blocks, 256, 0, ctx->stream>>>(src, ea);
    CKL("k_exh_items");
    return M6502_OK;
}

const uint16_t* join_mult(const m6502_ctx* ctx, uint32_t dead) {
    const CandGroups* g = ctx->join_groups[dead];
    return g ? g->mult : nullptr;
}

// The length-1 QuickCheck join.  A warp takes as many targets as fill the
// resident warps, up to a lane each: small searches spread over all SMs.
int launch_join1(m6502_ctx* ctx, const uint16_t* d_t, uint32_t tlen, uint64_t nt, const m6502_search_cfg& cfg,
                 uint64_t scap, Counters* cnt, const uint32_t* bad = nullptr) {
    const bool go = cfg.semantics == M6502_SEM_GO;
    const uint32_t stages = cfg.stages ? cfg.stages : M6502_CHECK_ALL, dead = cfg.dead_flags;
    // the line filter is part of ExhaustiveCheck; brute force does without
    const bool exh = (stages & M6502_CHECK_EXH) != 0, filter = exh && cfg.exh_mode != M6502_EXH_BRUTE;
    const uint64_t warps = (uint64_t)ctx->sms * 4 * kWarpsPerBlock;   // 4 resident blocks per SM
    const uint32_t chunk = (uint32_t)std::min<uint64_t>(32, (nt + warps - 1) / warps);
    const uint64_t blocks = (nt + (uint64_t)chunk * kWarpsPerBlock - 1) / ((uint64_t)chunk * kWarpsPerBlock);
    const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)ctx->sms * 4, blocks));
    const JoinTable* tab = ctx->join_tab[go][dead];
    const uint4* cfp4 = (const uint4*)ctx->cfp4.p;
    Surv* match = (Surv*)ctx->match.p;
    if (go)
        k_qc_join<true><<<grid, 256, 0, ctx->stream>>>(d_t, tlen, (uint32_t)nt, chunk, cfp4, tab, dead, stages, match, cnt, bad);
    else
        k_qc_join<false><<<grid, 256, 0, ctx->stream>>>(d_t, tlen, (uint32_t)nt, chunk, cfp4, tab, dead, stages, match, cnt, bad);
    CKL("k_qc_join");
    const uint16_t* mult = go ? nullptr : join_mult(ctx, dead);
    const uint32_t* lines = ctx->join_lines[dead];
    const uint32_t egrid = (uint32_t)std::min<uint64_t>((uint64_t)ctx->sms * 4, (nt + kWarpsPerBlock - 1) / kWarpsPerBlock);
    auto expand = [&](auto kernel) {
        kernel<<<egrid, 256, 0, ctx->stream>>>(match, d_t, tlen, cfp4, tab, dead, cfg.sweep, mult, lines, (Surv*)ctx->surv.p,
                                               scap, cnt, (Surv*)ctx->go_round.p, (uint32_t*)ctx->go_ord.p,
                                               exh ? kGoBlock : 0u);
    };
    if (go && filter) expand(k_expand<true, true>);
    else if (go) expand(k_expand<true, false>);
    else if (filter) expand(k_expand<false, true>);
    else expand(k_expand<false, false>);
    CKL("k_expand");
    return M6502_OK;
}

// Items of survivor pairs, with the work-item size of the knobs (the items
// were cut by launch_exh with the same size).
int launch_items(m6502_ctx* ctx, const SurvSource& src, ExhArgs ea) {
    ea.ticket_batch = ctx->tune.ticket_batch;
    ea.chunk_log2 = ctx->tune.chunk_log2;
    k_exh_items<SurvSource><<<ctx->exh_item_blocks, 256, 0, ctx->stream>>>(src, ea);
    CKL("k_exh_items");
    return M6502_OK;
}

// Field f (byte f of a packed state) of four states, one per byte.
uint32_t pack4(const uint64_t* states, int f) {
    uint32_t w = 0;
    for (int k = 0; k < 4; k++) w |= (uint32_t)((states[k] >> (8 * f)) & 0xFFu) << (8 * k);
    return w;
}

int init_ctx(m6502_ctx* ctx) {
    if (ctx->ready) return M6502_OK;
    CK(cudaSetDevice(ctx->device));
    uint64_t vec[32];
    for (int v = 0; v < 32; v++) {
        uint64_t x = 0;
        for (int b = 0; b < 8; b++) x |= (uint64_t)kVectors[v][b] << (8 * b);
        vec[v] = x;
    }
    uint16_t dep[NUM_OPS][NUM_LOCS], wr[NUM_OPS], sw[NUM_OPS];
    for (uint32_t op = 0; op < NUM_OPS; op++) {
        wr[op] = (uint16_t)op_deps(op, dep[op]);
        sw[op] = (uint16_t)sweep_locs_of_reads(op_reads(op));
    }
    static uint16_t tab[kNumInsns], gotab[kNumInsns];
    static uint32_t gorank[kNumInsns];
    host_tables(tab, gotab, gorank);
    uint32_t rep[32];
    for (int i = 0; i < 32; i++) rep[i] = kRepValues[i];
    uint32_t vec4[8][8];
    for (int g = 0; g < 8; g++)
        for (int f = 0; f < 8; f++) vec4[g][f] = pack4(vec + 4 * g, f);
    CK(cudaMemcpyToSymbolAsync(c_vec, vec, sizeof vec, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_vec4, vec4, sizeof vec4, 0, cudaMemcpyHostToDevice, ctx->stream));
    // Line states: A = i, the other registers a permutation of it each, the
    // carry the parity of i.
    uint32_t line[64][8];
    for (int j = 0; j < 64; j++) {
        uint64_t st[4];
        for (int k = 0; k < 4; k++) {
            const uint32_t i = (uint32_t)(4 * j + k);
            const uint32_t f[8] = {i, 5 * i + 59, 13 * i + 113, (uint32_t)__builtin_parity(i),
                                   29 * i + 7, 77 * i + 196, 141 * i + 45, 203 * i + 150};
            st[k] = 0;
            for (int b = 0; b < 8; b++) st[k] |= (uint64_t)(f[b] & 0xFFu) << (8 * b);
        }
        for (int f = 0; f < 8; f++) line[j][f] = pack4(st, f);
    }
    CK(cudaMemcpyToSymbolAsync(c_line, line, sizeof line, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_dep, dep, sizeof dep, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_wr, wr, sizeof wr, 0, cudaMemcpyHostToDevice, ctx->stream));
    uint16_t dep16[NUM_OPS][16] = {};
    for (uint32_t op = 0; op < NUM_OPS; op++)
        for (uint32_t l = 0; l < NUM_LOCS; l++) dep16[op][l] = dep[op][l];
    CK(cudaMemcpyToSymbolAsync(g_dep16, dep16, sizeof dep16, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_sweep, sw, sizeof sw, 0, cudaMemcpyHostToDevice, ctx->stream));
    uint32_t x4[NUM_OPS];
    for (uint32_t op = 0; op < NUM_OPS; op++) x4[op] = x4_desc(op);
    CK(cudaMemcpyToSymbolAsync(c_x4d, x4, sizeof x4, 0, cudaMemcpyHostToDevice, ctx->stream));
    X4Row rows[NUM_OPS];
    static_assert(sizeof(X4Row) == 3 * sizeof(uint4), "three words of 16 bytes");
    for (uint32_t op = 0; op < NUM_OPS; op++) rows[op] = x4_row(op);
    CK(cudaMemcpyToSymbolAsync(g_x4row, rows, sizeof rows, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_tab, tab, sizeof tab, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_gotab, gotab, sizeof gotab, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_gorank, gorank, sizeof gorank, 0, cudaMemcpyHostToDevice, ctx->stream));
    static uint16_t goidx[kNumInsns];
    for (int i = 0; i < kNumInsns; i++) goidx[gorank[i]] = (uint16_t)i;
    CK(cudaMemcpyToSymbolAsync(c_goidx, goidx, sizeof goidx, 0, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyToSymbolAsync(c_rep, rep, sizeof rep, 0, cudaMemcpyHostToDevice, ctx->stream));

    int occ = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_exhaustive<SurvSource>, 256, 0));
    ctx->exh_blocks = ctx->sms * std::max(occ, 1);
    ctx->exh_occ[4] = std::max(occ, 1);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_exhaustive<SurvSource, 3>, 256, 0));
    ctx->exh_occ[3] = std::max(occ, 1);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_exhaustive<SurvSource, 2>, 256, 0));
    ctx->exh_occ[2] = std::max(occ, 1);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_small<SurvSource, true>, 256, 0));
    ctx->small_blocks = ctx->sms * std::max(occ, 1);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_exh_items<SurvSource>, 256, 0));
    ctx->exh_item_blocks = ctx->sms * std::max(occ, 1);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_qc1<false>, 256, 0));
    ctx->qc_blocks = ctx->sms * std::max(occ, 1);
    ctx->fp_blocks = ctx->sms * 8;

    // length-1 candidate fingerprints and metadata
    TRY(ensure(ctx, ctx->cfp1, sizeof(uint64_t) * 32 * kNumInsns));
    TRY(ensure(ctx, ctx->cmeta1, kNumInsns));
    DevBuf tmp;
    TRY(ensure(ctx, tmp, sizeof(uint64_t) * 32 * kNumInsns));
    k_fingerprint<CandSeqs><<<ctx->fp_blocks, 256, 0, ctx->stream>>>(CandSeqs{1}, kNumInsns,
                                                                     (uint64_t*)tmp.p, nullptr);
    CKL("k_fingerprint(candidates)");
    std::vector<uint64_t> h(32 * (size_t)kNumInsns), tr(32 * (size_t)kNumInsns);
    CK(cudaMemcpyAsync(h.data(), tmp.p, h.size() * 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    cudaFree(tmp.p);
    for (int c = 0; c < kNumInsns; c++)
        for (int v = 0; v < 32; v++) tr[(size_t)v * kNumInsns + c] = h[(size_t)c * 32 + v];
    std::vector<uint8_t> meta(kNumInsns);
    for (int c = 0; c < kNumInsns; c++) {
        uint32_t op = tab[c] & 0xFF;
        uint16_t one = tab[c];
        meta[c] = (uint8_t)(bytes_cuda(op) | (bytes_go(op) << 2) | (should_prune(&one, 1) ? 0x10 : 0));
    }
    ctx->h_cfp4.resize((size_t)kNumInsns * 64);
    for (int c = 0; c < kNumInsns; c++)
        for (int g = 0; g < 8; g++)
            for (int f = 0; f < 8; f++) ctx->h_cfp4[(size_t)c * 64 + 8 * g + f] = pack4(&h[(size_t)c * 32 + 4 * g], f);
    TRY(ensure(ctx, ctx->cfp4, ctx->h_cfp4.size() * sizeof(uint32_t)));
    CK(cudaMemcpyAsync(ctx->cfp4.p, ctx->h_cfp4.data(), ctx->h_cfp4.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                       ctx->stream));
    ctx->h_cmeta = meta;
    ctx->h_tab.assign(tab, tab + kNumInsns);
    ctx->h_gorank.assign(gorank, gorank + kNumInsns);
    CK(cudaMemcpyAsync(ctx->cfp1.p, tr.data(), tr.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->cmeta1.p, meta.data(), meta.size(), cudaMemcpyHostToDevice, ctx->stream));
    TRY(ensure(ctx, ctx->cnt, sizeof(Counters)));
    CK(cudaStreamSynchronize(ctx->stream));
    ctx->ready = true;
    return M6502_OK;
}

// The group of a length-1 candidate under a dead-flags mask (see CandGroups),
// or -1 when it is alone in its group.  An instruction that writes only dead
// flags is the identity on every compared output; two of them stand for each
// other when the pairs they form also sweep the same registers (op_reads) and
// pass the same byte filter.  Then the verdict of (target, candidate) is the
// same for both: the same outputs, cones, domain and values.
int cand_group(uint32_t op, uint32_t dead) {
    uint16_t dep[NUM_LOCS];
    const uint32_t written = op_deps(op, dep);
    for (uint32_t l = 0; l < NUM_LOCS; l++)
        if ((written & LB(l)) && !(flag_bit(l) & dead)) return -1;   // a live output changes
    return (int)(sweep_locs_of_reads(op_reads(op)) << 4 | bytes_cuda(op));
}

// Memory for the tables of a mask, which live as long as the context: pieces
// of 8 MB blocks (a mask of both semantics takes 0.87 MB; an allocation of its
// own for each piece took 0.3 ms on every second or third new mask).
constexpr size_t kTableBlock = 8u << 20;
template <class T>
int table_mem(m6502_ctx* ctx, size_t n, T** out) {
    if (*out) return M6502_OK;   // kept from a call that failed later on
    const size_t bytes = (n * sizeof(T) + 255) & ~(size_t)255;
    if (ctx->table_blocks.empty() || ctx->table_used + bytes > kTableBlock) {
        void* p = nullptr;
        CK(cudaMalloc(&p, kTableBlock));
        ctx->table_blocks.push_back(p);
        ctx->table_used = 0;
    }
    *out = reinterpret_cast<T*>((char*)ctx->table_blocks.back() + ctx->table_used);
    ctx->table_used += bytes;
    return M6502_OK;
}

// JoinTable of the non-pruned length-1 candidates for one dead-flags mask,
// built once per mask.  CUDA semantics:
// one entry per group of candidates; Go semantics: every candidate (its
// passes and ranks tell the members of a group apart).
// It is part of a mask's first search: candidates go to the directory's buckets
// in enumeration order and are compared with the first members of the
// subclasses there (a vector of words per candidate and one sort over all of
// them took 0.7 ms).
int join_table(m6502_ctx* ctx, uint32_t dead, bool go) {
    if (ctx->join_built[go][dead]) return M6502_OK;
    if (!ctx->lines_built[dead]) {   // on the device meanwhile
        TRY(table_mem(ctx, (size_t)64 * kNumInsns, &ctx->join_lines[dead]));
        k_line_hash<<<(64 * kNumInsns + 255) / 256, 256, 0, ctx->stream>>>(dead, ctx->join_lines[dead]);
        CKL("k_line_hash");
        ctx->lines_built[dead] = true;
    }
    // A candidate's outputs, the dead flags masked: two groups of 8 packed words
    // (A X Y P S M S0 S1) of QuickCheck, then six of MidCheck, which Go semantics
    // does not have.
    const uint32_t pm = (kPMask & ~dead & 0xFFu) * kB1, all = 0xFFFFFFFFu;
    const uint32_t mask[8] = {all, all, all, pm, all, all, all, all};
    auto same = [&](uint32_t a, uint32_t b, int g0, int g1) {
        const uint32_t *x = &ctx->h_cfp4[(size_t)a * 64], *y = &ctx->h_cfp4[(size_t)b * 64];
        uint32_t d = 0;
        for (int g = g0; g < g1 && !d; g++)
            for (int k = 0; k < 8; k++) d |= (x[8 * g + k] ^ y[8 * g + k]) & mask[k];
        return d == 0;
    };
    // The candidates that go into the table, in enumeration order (CUDA or Go),
    // and the groups.
    int group[NUM_OPS];
    for (uint32_t op = 0; op < NUM_OPS; op++) group[op] = go ? -1 : cand_group(op, dead);
    CandGroups gr;
    std::memset(&gr, 0, sizeof gr);
    uint16_t lead[kNumInsns], order[kNumInsns];   // the candidate that stands for this one; the candidates in order
    for (uint32_t c = 0; c < (uint32_t)kNumInsns; c++) order[go ? ctx->h_gorank[c] : c] = (uint16_t)c;
    std::map<int, uint16_t> lead_of;   // by group
    struct Entry {
        uint64_t key;
        uint16_t cand, next;           // next member of its subclass
    };
    constexpr uint32_t kBuckets = 1u << kDirBits;
    constexpr uint16_t kNone = 0xFFFFu;
    std::vector<Entry> in, v;
    std::vector<uint16_t> at(kBuckets + 1), fill;   // first place of each bucket's entries
    in.reserve(kNumInsns);
    for (uint16_t c : order) {
        lead[c] = kNone;
        if (ctx->h_cmeta[c] & 0x10) continue;
        const int g = group[ctx->h_tab[c] & 0xFFu];
        lead[c] = g < 0 ? c : lead_of.emplace(g, c).first->second;
        gr.mult[lead[c]]++;
        if (lead[c] != c) continue;
        uint32_t qc[16];
        for (int w = 0; w < 16; w++) qc[w] = ctx->h_cfp4[(size_t)c * 64 + w] & mask[w % 8];
        in.push_back({join_key(qc), c, kNone});
        at[(in.back().key >> (64 - kDirBits)) + 1]++;
    }
    for (uint32_t b = 0; b < kBuckets; b++) at[b + 1] = (uint16_t)(at[b + 1] + at[b]);
    v.resize(in.size());
    fill = at;
    for (const Entry& e : in) v[fill[e.key >> (64 - kDirBits)]++] = e;
    // Bucket by bucket: the subclasses in the order of their first members, those
    // of one entry next to each other.
    std::vector<JoinTable> tab(1);
    JoinTable& t = tab[0];
    std::memset(&t, 0, sizeof t);
    struct Sub {
        uint16_t head, tail;           // places in v
        bool entry;                    // the first of its entry
    };
    std::vector<Sub> subs;
    uint32_t nu = 0, nj = 0, nc = 0;
    for (uint32_t b = 0; b < kBuckets; b++) {
        t.dir[b] = (uint16_t)nu;
        subs.clear();
        for (uint16_t i = at[b]; i < at[b + 1]; i++) {
            size_t place = 0;          // behind the subclasses of its entry
            bool member = false;
            for (size_t s = 0; s < subs.size() && !member; s++) {
                const Entry& e = v[subs[s].head];
                if (e.key != v[i].key || !same(e.cand, v[i].cand, 0, 2)) continue;
                place = s + 1;
                if (!go && !same(e.cand, v[i].cand, 2, 8)) continue;
                v[subs[s].tail].next = i;
                subs[s].tail = i;
                member = true;
            }
            if (!member) subs.insert(place ? subs.begin() + (long)place : subs.end(), Sub{i, i, place == 0});
        }
        for (const Sub& s : subs) {
            if (s.entry) {
                t.key[nu] = v[s.head].key;
                t.sub[nu++] = (uint16_t)nj;
            }
            t.start[nj++] = (uint16_t)nc;
            for (uint16_t i = s.head; i != kNone; i = v[i].next) {
                const uint32_t op = ctx->h_tab[v[i].cand] & 0xFFu;
                t.cand[nc++] = (uint16_t)(v[i].cand | (go ? bytes_go(op) : bytes_cuda(op)) << 12);
            }
        }
    }
    t.dir[kBuckets] = (uint16_t)nu;
    t.sub[nu] = (uint16_t)nj;
    t.start[nj] = (uint16_t)nc;
    for (uint32_t u = 0; go && u < nu; u++)
        ctx->join_longest[dead] = std::max<uint32_t>(ctx->join_longest[dead], t.start[t.sub[u + 1]] - t.start[t.sub[u]]);
    // The copies go on the stream of the kernels that read them.
    if (!go) {
        uint16_t next = 0, place[kNumInsns];
        for (int c = 0; c < kNumInsns; c++) {
            if (!gr.mult[c]) continue;
            gr.first[c] = place[c] = next;
            next = (uint16_t)(next + gr.mult[c]);
        }
        for (int c = 0; c < kNumInsns; c++)
            if (lead[c] != kNone) gr.member[place[lead[c]]++] = (uint16_t)c;
        for (uint32_t u = 0; u < nu; u++)
            for (uint32_t i = t.start[t.sub[u]]; i < t.start[t.sub[u + 1]]; i++)
                for (uint32_t b = t.cand[i] >> 12; b <= 2; b++) t.weight[u][b - 1] += gr.mult[t.cand[i] & 0xFFFu];
        TRY(table_mem(ctx, 1, &ctx->join_groups[dead]));
        CK(cudaMemcpyAsync(ctx->join_groups[dead], &gr, sizeof gr, cudaMemcpyHostToDevice, ctx->stream));
    }
    TRY(table_mem(ctx, 1, &ctx->join_tab[go][dead]));
    CK(cudaMemcpyAsync(ctx->join_tab[go][dead], &t, sizeof t, cudaMemcpyHostToDevice, ctx->stream));
    ctx->join_built[go][dead] = true;
    return M6502_OK;
}

// The sorted length-2 candidate table for one dead-flags mask (cached).
int cand2_table(m6502_ctx* ctx, uint32_t dead, m6502_ctx::Cand2Table** out) {
    const uint32_t n = (uint32_t)kNumInsns * (uint32_t)kNumInsns;
    m6502_ctx::Cand2Table* slot = nullptr;
    for (auto& t : ctx->cand2)
        if (t.dead == dead) slot = &t;
    if (!slot) {
        slot = &ctx->cand2[0];
        for (auto& t : ctx->cand2)
            if (t.stamp < slot->stamp) slot = &t;
        slot->dead = 0xFFFFFFFFu;
        TRY(ensure(ctx, slot->keys, (size_t)n * 8));
        TRY(ensure(ctx, slot->idx, (size_t)n * 4));
        TRY(ensure(ctx, ctx->c2_keys_in, (size_t)n * 8));
        TRY(ensure(ctx, ctx->c2_idx_in, (size_t)n * 4));
        size_t tb = 0;
        CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                           (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)n, 0, 64, ctx->stream));
        TRY(ensure(ctx, ctx->c2_sort_tmp, tb));
        TRY(ensure(ctx, slot->pw, (size_t)n * sizeof(uint2)));
        TRY(ensure(ctx, ctx->opflag, 2 * sizeof(uint32_t)));
        uint32_t info[2] = {1, 0};
        for (int attempt = 0; info[0]; attempt++) {   // two sets of outputs with one 64-bit key: another salt
            if (attempt == 8) return set_err(ctx, M6502_E_CUDA, "no salt separates the length-2 candidates");
            slot->salt = 0x9E3779B97F4A7C15ull * (uint64_t)attempt;
            k_cand2_keys<<<ctx->sms * 8, 256, 0, ctx->stream>>>(dead, slot->salt, (uint64_t*)ctx->c2_keys_in.p,
                                                                (uint32_t*)ctx->c2_idx_in.p);
            CKL("k_cand2_keys");
            tb = ctx->c2_sort_tmp.bytes;
            CK(cub::DeviceRadixSort::SortPairs(ctx->c2_sort_tmp.p, tb, (const uint64_t*)ctx->c2_keys_in.p,
                                               (uint64_t*)slot->keys.p, (const uint32_t*)ctx->c2_idx_in.p,
                                               (uint32_t*)slot->idx.p, (int)n, 0, 64, ctx->stream));
            CK(cudaMemsetAsync(ctx->opflag.p, 0, 2 * sizeof(uint32_t), ctx->stream));
            k_cand2_info<<<ctx->sms * 8, kInfoThreads, 0, ctx->stream>>>(dead, (const uint64_t*)slot->keys.p,
                                                                (const uint32_t*)slot->idx.p, (uint2*)slot->pw.p,
                                                                (uint32_t*)ctx->opflag.p);
            CKL("k_cand2_info");
            CK(cudaMemcpyAsync(info, ctx->opflag.p, sizeof info, cudaMemcpyDeviceToHost, ctx->stream));
            CK(cudaStreamSynchronize(ctx->stream));
        }
        slot->longest = info[1];
        slot->dead = dead;
    }
    slot->stamp = ++ctx->cand2_clock;
    *out = slot;
    return M6502_OK;
}

// Where a search's rules go: the caller's buffer while they fit, then the
// context's staging vector (m6502_fetch_rules).
struct RuleSink {
    m6502_rule* out;
    uint64_t cap, n;   // room, rules written
};

// `n` device rules to the sink, on the stream (not synchronised).
int deliver(m6502_ctx* ctx, RuleSink& sink, const m6502_rule* rules, uint64_t n) {
    const uint64_t k = sink.out ? std::min(n, sink.cap - sink.n) : 0;
    if (k)
        CK(cudaMemcpyAsync(sink.out + sink.n, rules, k * sizeof(m6502_rule), cudaMemcpyDeviceToHost, ctx->stream));
    sink.n += k;
    if (k < n) {
        const size_t old = ctx->staging.size();
        ctx->staging.resize(old + (n - k));
        CK(cudaMemcpyAsync(ctx->staging.data() + old, rules + k, (n - k) * sizeof(m6502_rule), cudaMemcpyDeviceToHost,
                           ctx->stream));
    }
    return M6502_OK;
}

// One device pass: nt targets (device pointer) of length tlen.  Hands its
// rules to the sink (target index = base + local, or ids[local]).
int run_pass(m6502_ctx* ctx, const m6502_search_cfg& cfg, const uint16_t* d_targets, uint64_t nt,
             uint32_t tlen, const uint64_t* d_ids, uint64_t base, RuleSink& sink, m6502_stats* st) {
    const bool go = cfg.semantics == M6502_SEM_GO;
    const uint32_t stages = cfg.stages ? cfg.stages : M6502_CHECK_ALL;
    const uint32_t dead = cfg.dead_flags;
    if ((cfg.flags & M6502_QC_SCAN) || cfg.max_cand_len >= 2) {   // stored target fingerprints
        TRY(ensure(ctx, ctx->tfp, nt * 32 * sizeof(uint64_t)));
        TRY(ensure(ctx, ctx->tmeta, nt));
    }
    uint64_t scap = std::max<uint64_t>(ctx->surv.bytes / sizeof(Surv), nt * 4 + 4096);
    uint64_t icap = std::max<uint64_t>(ctx->items.bytes / sizeof(Item), 1u << 16);
    uint64_t rcap = std::max<uint64_t>(ctx->rules.bytes / sizeof(m6502_rule), nt / 2 + 4096);
    uint64_t jcap = std::max<uint64_t>(ctx->jitems.bytes / sizeof(JoinItem), 1u << 16);
    m6502_ctx::Cand2Table *c2 = nullptr, *c2e = nullptr;   // sorted length-2 candidate keys (cached per mask)
    if (cfg.max_cand_len >= 2) {
        if (go && dead) TRY(cand2_table(ctx, 0, &c2e));   // unmasked table for targets with only that pass open
        TRY(cand2_table(ctx, dead, &c2));
        if (!c2e) c2e = c2;
    }
    const bool scan = (cfg.flags & M6502_QC_SCAN) != 0;
    const bool count_only = (cfg.flags & M6502_COUNT_ONLY) != 0;
    const bool exh = (stages & M6502_CHECK_EXH) != 0;
    const bool rounds = go && exh;   // Go semantics: verify in Go order, stop at the first pass
    const bool phase2 = cfg.max_cand_len >= 2;
    if (!scan) TRY(join_table(ctx, dead, go));
    // the scan's survivors are single candidates; the join's may stand for a group
    const CandGroups* groups = scan || go ? nullptr : ctx->join_groups[dead];
    const uint16_t* mult = groups ? groups->mult : nullptr;
    for (int attempt = 0; attempt < 6; attempt++) {
        // Every buffer the pass uses is allocated here, so that the launches
        // below can be recorded as one CUDA graph and replayed.
        TRY(ensure(ctx, ctx->surv, scap * sizeof(Surv)));
        TRY(ensure(ctx, ctx->fail, scap * sizeof(uint32_t)));
        TRY(ensure(ctx, ctx->order, scap * sizeof(uint32_t)));
        if (!scan) TRY(ensure(ctx, ctx->match, nt * sizeof(Surv)));
        TRY(ensure(ctx, ctx->items, icap * sizeof(Item)));
        TRY(ensure(ctx, ctx->rules, rcap * sizeof(m6502_rule)));
        if (go) {
            TRY(ensure(ctx, ctx->best, 2 * nt * sizeof(uint32_t)));
            TRY(ensure(ctx, ctx->go_ord, scap * 4));
            TRY(ensure(ctx, ctx->go_round, scap * sizeof(Surv)));
        }
        int end_bit = 30;   // Go-order sort keys: target << 30 | pass << 29 | rank
        while (end_bit < 63 && (nt >> (end_bit - 30)) != 0) end_bit++;
        if (rounds && scan) {
            TRY(ensure(ctx, ctx->go_keys, scap * 8));
            TRY(ensure(ctx, ctx->go_keys2, scap * 8));
            size_t tb = 0;
            CK(cub::DeviceRadixSort::SortKeys(nullptr, tb, (const uint64_t*)nullptr, (uint64_t*)nullptr, (int)scap, 0,
                                              end_bit, ctx->stream));
            TRY(ensure(ctx, ctx->go_sort_tmp, tb));
        }
        if (phase2) TRY(ensure(ctx, ctx->jitems, jcap * sizeof(JoinItem)));
        const uint64_t rlim = count_only ? 0 : rcap;   // emit kernels count past rlim without writing
        Counters* cnt = (Counters*)ctx->cnt.p;
        bool capturing = false;
        // Stage events: inside a capture they must be external record nodes.
        auto rec = [&](cudaEvent_t e) -> cudaError_t {
            return capturing ? cudaEventRecordWithFlags(e, ctx->stream, cudaEventRecordExternal)
                             : cudaEventRecord(e, ctx->stream);
        };
        // All launches of one pass, with no host read-back in between.
        auto enqueue = [&]() -> int {
        CK(cudaMemsetAsync(cnt, 0, sizeof(Counters), ctx->stream));
        CK(rec(ctx->sev[0]));
        if (scan || cfg.max_cand_len >= 2) {   // the join computes its targets' outputs itself
            k_fingerprint<FixedSeqs><<<ctx->fp_blocks, 256, 0, ctx->stream>>>(
                FixedSeqs{d_targets, tlen}, nt, (uint64_t*)ctx->tfp.p, (uint8_t*)ctx->tmeta.p);
            CKL("k_fingerprint(targets)");
        }
        CK(rec(ctx->sev[1]));
        uint32_t qgrid = (uint32_t)std::min<uint64_t>(ctx->qc_blocks, (nt + kQcTile - 1) / kQcTile);
        if (!scan) {
            TRY(launch_join1(ctx, d_targets, tlen, nt, cfg, scap, cnt));
        } else if (go)
            k_qc1<true><<<qgrid, 256, 0, ctx->stream>>>((uint64_t*)ctx->tfp.p, (uint8_t*)ctx->tmeta.p,
                                                        (uint32_t)nt, (uint64_t*)ctx->cfp1.p,
                                                        (uint8_t*)ctx->cmeta1.p, dead, stages,
                                                        (Surv*)ctx->surv.p, scap, cnt, nullptr);
        else
            k_qc1<false><<<qgrid, 256, 0, ctx->stream>>>((uint64_t*)ctx->tfp.p, (uint8_t*)ctx->tmeta.p,
                                                         (uint32_t)nt, (uint64_t*)ctx->cfp1.p,
                                                         (uint8_t*)ctx->cmeta1.p, dead, stages,
                                                         (Surv*)ctx->surv.p, scap, cnt, nullptr);
        CKL("k_qc1");
        CK(rec(ctx->sev[2]));
        SurvSource src{(const Surv*)ctx->surv.p, d_targets, tlen, dead, go ? 1 : 0, mult};
        ExhArgs ea{(uint32_t*)ctx->fail.p, (Item*)ctx->items.p, icap, cnt, &cnt->v[0][0], cfg.sweep,
                   cfg.exh_mode == M6502_EXH_BRUTE};
        // Go-order verification rounds of a phase, queued with no read-back: the
        // first round's list is in ctx->go_round and the later survivors in
        // ctx->surv with their ordinals (after a scan: all of them in ctx->surv,
        // to be sorted, over the buffer's whole capacity; entries past the
        // device's count get a key that sorts last).  Every round that a range of
        // `bound` candidates could need is launched.  On return `best` holds the
        // first passing candidate per target and pass.
        auto go_rounds = [&](int phase, uint64_t bound) -> int {
            const bool sorted = scan && phase == 0;
            if (sorted) {
                const uint64_t pad = (1ull << end_bit) - 1;   // above every real key (target < nt)
                k_go_keys<<<ctx->sms * 8, 256, 0, ctx->stream>>>((const Surv*)ctx->surv.p, &cnt->surv, scap, pad,
                                                                 (uint64_t*)ctx->go_keys.p);
                CKL("k_go_keys");
                size_t tb = ctx->go_sort_tmp.bytes;
                CK(cub::DeviceRadixSort::SortKeys(ctx->go_sort_tmp.p, tb, (const uint64_t*)ctx->go_keys.p,
                                                  (uint64_t*)ctx->go_keys2.p, (int)scap, 0, end_bit, ctx->stream));
                k_go_ord<<<ctx->sms * 8, 256, 0, ctx->stream>>>((const uint64_t*)ctx->go_keys2.p, &cnt->surv, scap,
                                                                (Surv*)ctx->surv.p, (uint32_t*)ctx->go_ord.p, cnt);
                CKL("k_go_ord");
            }
            SurvSource rs{(const Surv*)ctx->go_round.p, d_targets, tlen, dead, 1, nullptr};
            int r = 0;
            for (uint64_t lo = 0, blk = kGoBlock; lo < bound; lo += blk, blk *= 8, r++) {
                VerifyCounters* v = &cnt->v[phase][r];
                if (r > 0 || sorted) {
                    k_go_round<<<ctx->sms * 8, 256, 0, ctx->stream>>>(
                        (const Surv*)ctx->surv.p, (const uint32_t*)ctx->go_ord.p, &cnt->surv, scap, (uint32_t)lo,
                        (uint32_t)(lo + blk), (const uint32_t*)ctx->best.p, (uint32_t)nt, (Surv*)ctx->go_round.p, cnt, v);
                    CKL("k_go_round");
                }
                ExhArgs ra{(uint32_t*)ctx->fail.p, (Item*)ctx->items.p, icap, cnt, v, cfg.sweep,
                           cfg.exh_mode == M6502_EXH_BRUTE};
                TRY(launch_exh(ctx, rs, &v->n, scap, ra));
                TRY(launch_items(ctx, rs, ra));
                k_go_select<<<ctx->sms * 8, 256, 0, ctx->stream>>>((const Surv*)ctx->go_round.p, &v->n, scap,
                                                                   (const uint32_t*)ctx->fail.p, (uint32_t)nt,
                                                                   (uint32_t*)ctx->best.p, cnt, d_targets, tlen,
                                                                   cfg.sweep);
                CKL("k_go_select");
            }
            return M6502_OK;
        };
        if (go) CK(cudaMemsetAsync(ctx->best.p, 0xFF, 2 * nt * sizeof(uint32_t), ctx->stream));
        if (exh && !rounds) TRY(launch_exh(ctx, src, &cnt->surv, scap, ea, !scan));
        if (rounds) TRY(go_rounds(0, scan ? (uint64_t)kNumInsns : ctx->join_longest[dead]));
        CK(rec(ctx->sev[3]));
        if (exh && !rounds) TRY(launch_items(ctx, src, ea));
        CK(rec(ctx->sev[4]));
        // Passing survivors -> Go winners (best) or rules (CUDA semantics).
        auto select_or_emit = [&]() -> int {
            if (rounds) return M6502_OK;   // the rounds selected already
            if (go) {
                if (!exh) CK(cudaMemsetAsync(ctx->fail.p, 0, scap * sizeof(uint32_t), ctx->stream));
                k_go_select<<<ctx->sms * 8, 256, 0, ctx->stream>>>((const Surv*)ctx->surv.p, &cnt->surv, scap,
                                                                   (const uint32_t*)ctx->fail.p, (uint32_t)nt,
                                                                   (uint32_t*)ctx->best.p, cnt, d_targets, tlen,
                                                                   cfg.sweep);
                CKL("k_go_select");
            } else {
                k_emit_all<<<ctx->sms * 8, 256, 0, ctx->stream>>>((const Surv*)ctx->surv.p, &cnt->surv, scap,
                                                                  (const uint32_t*)ctx->fail.p, d_ids, base, dead,
                                                                  (m6502_rule*)ctx->rules.p, rlim, &cnt->rules, cnt,
                                                                  exh ? 1 : 0, d_targets, tlen, cfg.sweep, groups);
                CKL("k_emit_all");
            }
            return M6502_OK;
        };
        TRY(select_or_emit());
        CK(rec(ctx->sev[5]));
        if (phase2) {
            // Length-2 candidates (worker.go:122: candidate lengths 1..max).  The
            // phase-1 counts are kept on the device; buffer overflows of either
            // phase are checked once, after the pass.
            k_mark_phase<<<1, 1, 0, ctx->stream>>>(cnt);
            CKL("k_mark_phase");
            CK(cudaMemsetAsync(&cnt->surv, 0, kPhaseCounters * sizeof(unsigned long long), ctx->stream));
            CK(rec(ctx->sev2[0]));
            const uint32_t jgrid2 =
                (uint32_t)std::min<uint64_t>((uint64_t)ctx->sms * 8, (nt + kWarpsPerBlock - 1) / kWarpsPerBlock);
            const uint32_t n2 = (uint32_t)kNumInsns * (uint32_t)kNumInsns;
            auto view = [](const m6502_ctx::Cand2Table* t) {
                return Cand2View{(const uint64_t*)t->keys.p, (const uint32_t*)t->idx.p, (const uint2*)t->pw.p, t->salt};
            };
            Join2Args ja{(const uint64_t*)ctx->tfp.p, (const uint8_t*)ctx->tmeta.p, (uint32_t)nt, view(c2), view(c2e), n2,
                         dead, stages, go ? (const uint32_t*)ctx->best.p : nullptr, (Surv*)ctx->surv.p, scap,
                         (JoinItem*)ctx->jitems.p, jcap, cnt, (Surv*)ctx->go_round.p, (uint32_t*)ctx->go_ord.p,
                         rounds ? kGoBlock : 0u};
            if (go) {
                k_go_join2<<<jgrid2, 256, 0, ctx->stream>>>(ja);
                k_go_join2_count<<<ctx->sms * 8, 256, 0, ctx->stream>>>(ja);
                k_go_join2_items<<<ctx->sms * 8, 256, 0, ctx->stream>>>(ja);
            } else {
                k_qc_join2<<<jgrid2, 256, 0, ctx->stream>>>(ja);
                k_qc_join2_items<<<ctx->sms * 8, 256, 0, ctx->stream>>>(ja);
            }
            CKL("k_qc_join2");
            CK(rec(ctx->sev2[1]));
            ExhArgs ea2 = ea;
            ea2.v = &cnt->v[1][0];
            if (exh && !rounds) TRY(launch_exh(ctx, src, &cnt->surv, scap, ea2));
            if (rounds) TRY(go_rounds(1, std::max(c2->longest, c2e->longest)));
            CK(rec(ctx->sev2[2]));
            if (exh && !rounds) TRY(launch_items(ctx, src, ea2));
            CK(rec(ctx->sev2[3]));
            TRY(select_or_emit());
            CK(rec(ctx->sev2[4]));
        }
        if (!phase2) CK(rec(ctx->sev2[4]));
        if (go) {
            k_go_emit<<<ctx->sms * 8, 256, 0, ctx->stream>>>((const uint32_t*)ctx->best.p, (uint32_t)nt,
                                                             d_targets, tlen, d_ids, base,
                                                             (m6502_rule*)ctx->rules.p, rlim, cnt);
            CKL("k_go_emit");
        }
        CK(rec(ctx->sev2[5]));
        return M6502_OK;
        };   // enqueue
        // One recorded graph per pass configuration (a few kept); an identical
        // later pass replays it.
        bool launched = false;
        if (!(cfg.flags & M6502_NO_GRAPH) && !ctx->graph.broken) {
            const std::vector<uint64_t> key = {
                (uint64_t)(uintptr_t)d_targets, nt, tlen, (uint64_t)(uintptr_t)d_ids, base, cfg.semantics, cfg.sweep,
                cfg.exh_mode, stages, cfg.flags, dead, cfg.max_cand_len, scap, icap, rcap, jcap,
                (uint64_t)(uintptr_t)ctx->surv.p, (uint64_t)(uintptr_t)ctx->fail.p, (uint64_t)(uintptr_t)ctx->items.p,
                (uint64_t)(uintptr_t)ctx->order.p, (uint64_t)(uintptr_t)ctx->match.p,
                (uint64_t)(uintptr_t)ctx->rules.p, (uint64_t)(uintptr_t)ctx->cnt.p, (uint64_t)(uintptr_t)ctx->best.p,
                (uint64_t)(uintptr_t)ctx->tfp.p, (uint64_t)(uintptr_t)ctx->tmeta.p,
                (uint64_t)(uintptr_t)ctx->go_keys.p, (uint64_t)(uintptr_t)ctx->go_keys2.p,
                (uint64_t)(uintptr_t)ctx->go_ord.p, (uint64_t)(uintptr_t)ctx->go_round.p,
                (uint64_t)(uintptr_t)ctx->go_sort_tmp.p, ctx->go_sort_tmp.bytes, (uint64_t)(uintptr_t)ctx->jitems.p,
                (uint64_t)(uintptr_t)ctx->join_tab[go][dead], c2 ? (uint64_t)(uintptr_t)c2->keys.p : 0,
                c2e ? (uint64_t)(uintptr_t)c2e->keys.p : 0, ctx->tune.exh_minb, ctx->tune.ticket_batch,
                ctx->tune.chunk_log2};
            m6502_ctx::PassGraph* pg = nullptr;
            for (m6502_ctx::PassGraph& g : ctx->pass_graphs)
                if (g.exec && g.key == key) pg = &g;
            if (!pg) {   // record: the least recently used slot is replaced
                pg = &ctx->pass_graphs[0];
                for (m6502_ctx::PassGraph& g : ctx->pass_graphs)
                    if (g.stamp < pg->stamp) pg = &g;
                if (pg->exec) { cudaGraphExecDestroy(pg->exec); pg->exec = nullptr; }
                cudaGraph_t g = nullptr;
                bool ok = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
                if (ok) {
                    capturing = true;
                    const int rc = enqueue();
                    capturing = false;
                    ok = cudaStreamEndCapture(ctx->stream, &g) == cudaSuccess && rc == M6502_OK && g;
                    ok = ok && cudaGraphInstantiate(&pg->exec, g, 0) == cudaSuccess;
                    if (g) cudaGraphDestroy(g);
                }
                if (!ok) {
                    pg->exec = nullptr;
                    ctx->graph.broken = true;
                    ctx->graph.why = cudaGetErrorString(cudaGetLastError());   // clears the launch error
                    set_err(ctx, M6502_OK, "CUDA graph recording failed (" + ctx->graph.why +
                                               "); passes are launched directly");
                } else {
                    pg->key = key;
                }
            } else if (st) {
                st->graph_replays = 1;
            }
            if (pg->exec) {
                pg->stamp = ++ctx->pass_graph_clock;
                CK(cudaGraphLaunch(pg->exec, ctx->stream));
                launched = true;
            }
        }
        if (!launched) TRY(enqueue());
        Counters hc;
        bool redo = false;
        CK(cudaMemcpyAsync(&hc, cnt, sizeof hc, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        uint64_t surv_need = std::max<uint64_t>(hc.surv1, phase2 ? 0 : hc.surv), items_need = 0, listed = 0, items = 0;
        bool first_over = false;
        for (int ph = 0; ph < 2; ph++) {
            if (ph == 1) {
                // A first phase that overflowed leaves targets open that it would
                // have settled: what the second phase then asked for says nothing.
                first_over = surv_need > scap;
                if (first_over) break;
                if (phase2) surv_need = std::max<uint64_t>(surv_need, hc.surv);
            }
            for (const VerifyCounters& v : hc.v[ph]) {
                surv_need = std::max<uint64_t>(surv_need, v.n);
                items_need = std::max<uint64_t>(items_need, v.items);
                listed += v.n;
                items += v.items;
            }
        }
        if (surv_need > scap) { scap = surv_need + surv_need / 4 + 1024; redo = true; }
        if (items_need > icap) { icap = items_need + items_need / 4 + 1024; redo = true; }
        if (hc.rules > rlim && !count_only) { rcap = hc.rules + hc.rules / 4 + 1024; redo = true; }
        if (!first_over && hc.join_items > jcap) { jcap = hc.join_items + hc.join_items / 4 + 1024; redo = true; }
        if (redo) continue;
        if (!count_only) TRY(deliver(ctx, sink, (const m6502_rule*)ctx->rules.p, hc.rules));
        CK(cudaStreamSynchronize(ctx->stream));
        if (st) {
            st->targets += nt;
            st->pairs += nt * ((uint64_t)kNumInsns + (phase2 ? (uint64_t)kNumInsns * kNumInsns : 0u));
            st->qc_hits += hc.qc;
            st->mid_hits += hc.mid;
            st->exh_checked += !exh ? 0 : rounds ? listed + hc.round_rejects : hc.mid;
            st->exh_passed += hc.exh_pass;
            st->rules += hc.rules;
            st->exh_states += hc.states;
            st->exh_items += items;
            st->exh_algo_ops += hc.algo;
            st->exh_probe_rejects += hc.probe_rejects;
            st->exh_undecided += hc.undecided;
            float ms[5];
            for (int i = 0; i < 5; i++) cudaEventElapsedTime(&ms[i], ctx->sev[i], ctx->sev[i + 1]);
            st->ms_fingerprint += ms[0];
            st->ms_qc += ms[1];
            st->ms_exhaustive += ms[2];
            st->ms_exh_items += ms[3];
            st->ms_emit += ms[4];
            cudaEventElapsedTime(&ms[4], ctx->sev2[4], ctx->sev2[5]);
            st->ms_emit += ms[4];
            if (phase2) {
                for (int i = 0; i < 4; i++) cudaEventElapsedTime(&ms[i], ctx->sev2[i], ctx->sev2[i + 1]);
                st->ms_qc += ms[0];
                st->ms_exhaustive += ms[1];
                st->ms_exh_items += ms[2];
                st->ms_emit += ms[3];
            }
            st->passes += 1;
        }
        return M6502_OK;
    }
    return set_err(ctx, M6502_E_NOMEM, "device buffers kept overflowing");
}

// CUDA semantics with length-1 candidates: every pass of a search is
// queued on the stream with no host round trip in between.  Each pass has
// its own counters (survivors, work items) and stage events; all passes
// append their rules to one device buffer through one counter, with the
// global target index.  One synchronisation at the end reads every pass's
// counters; if any buffer overflowed, the whole search is re-run with larger
// buffers (nothing is dropped).  Returns M6502_E_INVAL when the search does
// not fit this path, or for an opcode outside the table: every pass checks its
// targets first, and from the first bad one on the join finds nothing.
// `targets` is in device memory; with `host` set it is filled from there pass
// by pass on a second stream, so that the copies (pageable memory: 30 MB of
// length-2 targets take longer than their search) run beside the kernels.
int search_async(m6502_ctx* ctx, const m6502_search_cfg& cfg, const uint16_t* targets, const uint16_t* host, uint64_t n,
                 uint32_t tlen, m6502_stats* st, RuleSink& sink) {
    const uint64_t P = ctx->pass_targets;
    const uint64_t npass = (n + P - 1) / P;
    if (npass == 0 || npass > (uint64_t)kMaxAsyncPasses) return set_err(ctx, M6502_E_INVAL, "too many passes");
    const uint32_t stages = cfg.stages ? cfg.stages : M6502_CHECK_ALL;
    const uint32_t dead = cfg.dead_flags;
    const bool exh = (stages & M6502_CHECK_EXH) != 0;
    const bool scan = (cfg.flags & M6502_QC_SCAN) != 0;
    const bool count_only = (cfg.flags & M6502_COUNT_ONLY) != 0;
    const uint64_t pmax = std::min(P, n);
    uint64_t scap = std::max<uint64_t>(ctx->surv.bytes / sizeof(Surv), pmax * 4 + 4096);
    uint64_t icap = std::max<uint64_t>(ctx->items.bytes / sizeof(Item), 1u << 16);
    uint64_t rcap = std::max<uint64_t>(ctx->rules.bytes / sizeof(m6502_rule), n / 2 + 4096);
    if (scan) {
        TRY(ensure(ctx, ctx->tfp, pmax * 32 * sizeof(uint64_t)));
        TRY(ensure(ctx, ctx->tmeta, pmax));
    }
    if (!scan) TRY(join_table(ctx, dead, false));
    const CandGroups* groups = scan ? nullptr : ctx->join_groups[dead];
    TRY(ensure(ctx, ctx->cnt_slots, npass * sizeof(Counters)));
    Counters* slots = (Counters*)ctx->cnt_slots.p;
    TRY(ensure(ctx, ctx->opflag, 2 * sizeof(uint32_t)));
    uint32_t* bad = (uint32_t*)ctx->opflag.p;
    for (int attempt = 0; attempt < 6; attempt++) {
        TRY(ensure(ctx, ctx->surv, scap * sizeof(Surv)));
        TRY(ensure(ctx, ctx->fail, scap * sizeof(uint32_t)));
        TRY(ensure(ctx, ctx->order, scap * sizeof(uint32_t)));
        if (!scan) TRY(ensure(ctx, ctx->match, pmax * sizeof(Surv)));
        TRY(ensure(ctx, ctx->items, icap * sizeof(Item)));
        TRY(ensure(ctx, ctx->rules, rcap * sizeof(m6502_rule)));
        // All passes, queued with no host round trip, recorded once as a CUDA
        // graph and replayed by identical later calls.
        bool capturing = false;
        // Stage events: inside a capture they must be external record nodes
        // (a plain record there only orders streams and records nothing).
        auto rec = [&](cudaEvent_t e) -> cudaError_t {
            return capturing ? cudaEventRecordWithFlags(e, ctx->stream, cudaEventRecordExternal)
                             : cudaEventRecord(e, ctx->stream);
        };
        // Pass p; the first also clears every pass's counters.
        auto enqueue = [&](uint64_t p) -> int {
            if (p == 0) {
                CK(cudaMemsetAsync(slots, 0, npass * sizeof(Counters), ctx->stream));
                CK(cudaMemsetAsync(bad, 0, sizeof(uint32_t), ctx->stream));
            }
            {
                const uint64_t b = p * P, nt = std::min(P, n - b);
                const uint16_t* d_t = targets + b * tlen;
                Counters* cnt = slots + p;
                cudaEvent_t* ev = ctx->aev + 6 * p;
                const uint32_t cgrid = (uint32_t)std::min<uint64_t>((nt * tlen + 255) / 256, (uint64_t)ctx->sms * 16);
                k_check_ops<<<cgrid, 256, 0, ctx->stream>>>(d_t, nt * tlen, bad);
                CKL("k_check_ops");
                CK(rec(ev[0]));
                if (scan) {
                    k_fingerprint<FixedSeqs><<<ctx->fp_blocks, 256, 0, ctx->stream>>>(
                        FixedSeqs{d_t, tlen}, nt, (uint64_t*)ctx->tfp.p, (uint8_t*)ctx->tmeta.p);
                    CKL("k_fingerprint(targets)");
                }
                CK(rec(ev[1]));
                if (scan) {
                    const uint32_t qgrid = (uint32_t)std::min<uint64_t>(ctx->qc_blocks, (nt + kQcTile - 1) / kQcTile);
                    k_qc1<false><<<qgrid, 256, 0, ctx->stream>>>((uint64_t*)ctx->tfp.p, (uint8_t*)ctx->tmeta.p,
                                                                 (uint32_t)nt, (uint64_t*)ctx->cfp1.p,
                                                                 (uint8_t*)ctx->cmeta1.p, dead, stages,
                                                                 (Surv*)ctx->surv.p, scap, cnt, bad);
                    CKL("k_qc1");
                } else {
                    TRY(launch_join1(ctx, d_t, tlen, nt, cfg, scap, cnt, bad));
                }
                CK(rec(ev[2]));
                SurvSource src{(const Surv*)ctx->surv.p, d_t, tlen, dead, 0, groups ? groups->mult : nullptr};
                ExhArgs ea{(uint32_t*)ctx->fail.p, (Item*)ctx->items.p, icap, cnt, &cnt->v[0][0], cfg.sweep,
                           cfg.exh_mode == M6502_EXH_BRUTE};
                if (exh) TRY(launch_exh(ctx, src, &cnt->surv, scap, ea, !scan));
                CK(rec(ev[3]));
                if (exh) TRY(launch_items(ctx, src, ea));
                CK(rec(ev[4]));
                k_emit_all<<<ctx->sms * 8, 256, 0, ctx->stream>>>((const Surv*)ctx->surv.p, &cnt->surv, scap,
                                                                  (const uint32_t*)ctx->fail.p, nullptr, b, dead,
                                                                  (m6502_rule*)ctx->rules.p, count_only ? 0 : rcap,
                                                                  &slots[0].rules, cnt, exh ? 1 : 0, d_t, tlen,
                                                                  cfg.sweep, groups);
                CKL("k_emit_all");
                CK(rec(ev[5]));
            }
            return M6502_OK;
        };
        const bool use_graph = !(cfg.flags & M6502_NO_GRAPH) && !ctx->graph.broken;
        bool replayed = false;
        if (use_graph) {
            const std::vector<uint64_t> key = {
                (uint64_t)(uintptr_t)targets, n, tlen, cfg.semantics, cfg.sweep, cfg.exh_mode, stages,
                cfg.flags, dead, scap, icap, rcap, P, (uint64_t)(uintptr_t)ctx->surv.p,
                (uint64_t)(uintptr_t)ctx->fail.p, (uint64_t)(uintptr_t)ctx->items.p, (uint64_t)(uintptr_t)ctx->order.p,
                (uint64_t)(uintptr_t)ctx->match.p,
                (uint64_t)(uintptr_t)ctx->rules.p, (uint64_t)(uintptr_t)ctx->cnt_slots.p,
                (uint64_t)(uintptr_t)ctx->tfp.p, (uint64_t)(uintptr_t)ctx->tmeta.p, (uint64_t)(uintptr_t)ctx->opflag.p,
                (uint64_t)(uintptr_t)ctx->join_tab[0][dead], ctx->tune.exh_minb, ctx->tune.ticket_batch,
                ctx->tune.chunk_log2};
            replayed = ctx->graph.exec.size() == npass && ctx->graph.key == key;
            if (!replayed) {
                for (cudaGraphExec_t e : ctx->graph.exec) cudaGraphExecDestroy(e);
                ctx->graph.exec.clear();
                // Record; if recording or instantiation fails, this context stops
                // using graphs and the passes are launched directly below.
                bool ok = true;
                for (uint64_t p = 0; p < npass && ok; p++) {
                    cudaGraph_t g = nullptr;
                    cudaGraphExec_t e = nullptr;
                    ok = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
                    if (ok) {
                        capturing = true;
                        const int rc = enqueue(p);
                        capturing = false;
                        ok = cudaStreamEndCapture(ctx->stream, &g) == cudaSuccess && rc == M6502_OK && g;
                        ok = ok && cudaGraphInstantiate(&e, g, 0) == cudaSuccess;
                        if (g) cudaGraphDestroy(g);
                    }
                    if (ok) ctx->graph.exec.push_back(e);
                }
                if (!ok) {
                    for (cudaGraphExec_t e : ctx->graph.exec) cudaGraphExecDestroy(e);
                    ctx->graph.exec.clear();
                    ctx->graph.broken = true;
                    ctx->graph.why = cudaGetErrorString(cudaGetLastError());   // clears the launch error
                    set_err(ctx, M6502_OK, "CUDA graph recording failed (" + ctx->graph.why +
                                               "); passes are launched directly");
                } else {
                    ctx->graph.key = key;
                }
            }
        }
        for (uint64_t p = 0; p < npass; p++) {
            if (host && attempt == 0) {
                const uint64_t b = p * P, nt = std::min(P, n - b);
                // a single pass has nothing to run beside: its copy goes on the same stream
                const cudaStream_t cs = npass > 1 ? ctx->copy : ctx->stream;
                // not before what was on the context's stream when the call began: the caller's
                // own work there may write the targets
                if (npass > 1 && p == 0) CK(cudaStreamWaitEvent(ctx->copy, ctx->ev0, 0));
                CK(cudaMemcpyAsync((void*)(targets + b * tlen), host + b * tlen, nt * tlen * sizeof(uint16_t),
                                   cudaMemcpyHostToDevice, cs));
                if (npass > 1) {
                    CK(cudaEventRecord(ctx->cev[p], ctx->copy));
                    CK(cudaStreamWaitEvent(ctx->stream, ctx->cev[p], 0));
                }
            }
            if (use_graph && !ctx->graph.broken) CK(cudaGraphLaunch(ctx->graph.exec[p], ctx->stream));
            else TRY(enqueue(p));
        }
        std::vector<Counters> hc(npass);
        uint32_t any_bad = 0;
        CK(cudaMemcpyAsync(hc.data(), slots, npass * sizeof(Counters), cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaMemcpyAsync(&any_bad, bad, sizeof any_bad, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        if (any_bad) return set_err(ctx, M6502_E_INVAL, "opcode out of range");
        bool redo = false;
        for (const Counters& c : hc) {
            if (c.surv > scap) { scap = std::max<uint64_t>(scap, c.surv + c.surv / 4 + 1024); redo = true; }
            const uint64_t items = c.v[0][0].items;
            if (items > icap) { icap = std::max<uint64_t>(icap, items + items / 4 + 1024); redo = true; }
        }
        const uint64_t nrules = hc[0].rules;
        if (nrules > rcap && !count_only) { rcap = nrules + nrules / 4 + 1024; redo = true; }
        if (redo) continue;
        if (!count_only) TRY(deliver(ctx, sink, (const m6502_rule*)ctx->rules.p, nrules));
        CK(cudaStreamSynchronize(ctx->stream));
        if (st) {
            for (uint64_t p = 0; p < npass; p++) {
                const Counters& c = hc[p];
                const uint64_t nt = std::min(P, n - p * P);
                st->targets += nt;
                st->pairs += nt * (uint64_t)kNumInsns;
                st->qc_hits += c.qc;
                st->mid_hits += c.mid;
                st->exh_checked += exh ? c.mid : 0;   // every MidCheck survivor, the filtered ones included
                st->exh_passed += c.exh_pass;
                st->exh_states += c.states;
                st->exh_items += c.v[0][0].items;
                st->exh_algo_ops += c.algo;
                st->exh_probe_rejects += c.probe_rejects;
                st->exh_undecided += c.undecided;
                float ms[5];
                for (int i = 0; i < 5; i++) cudaEventElapsedTime(&ms[i], ctx->aev[6 * p + i], ctx->aev[6 * p + i + 1]);
                st->ms_fingerprint += ms[0];
                st->ms_qc += ms[1];
                st->ms_exhaustive += ms[2];
                st->ms_exh_items += ms[3];
                st->ms_emit += ms[4];
                st->passes += 1;
            }
            st->rules += nrules;
            st->graph_replays = replayed ? 1u : 0u;
        }
        return M6502_OK;
    }
    return set_err(ctx, M6502_E_NOMEM, "device buffers kept overflowing");
}

int check_cfg(m6502_ctx* ctx, const m6502_search_cfg* cfg) {
    if (!cfg) return set_err(ctx, M6502_E_INVAL, "cfg is NULL");
    if (cfg->semantics > M6502_SEM_GO) return set_err(ctx, M6502_E_INVAL, "bad semantics");
    if (cfg->sweep > M6502_SWEEP_FULL) return set_err(ctx, M6502_E_INVAL, "bad sweep");
    if (cfg->exh_mode > M6502_EXH_BRUTE) return set_err(ctx, M6502_E_INVAL, "bad exh_mode");
    if (cfg->max_cand_len > 2)
        return set_err(ctx, M6502_E_INVAL, "max_cand_len > 2: the length-3 candidate space (2.3e10) has no join table");
    return M6502_OK;
}

// Nothing is staged any more: a large block goes back, others stay for the next
// search.  The C library may return a freed block of this size to the system,
// which depends on what else the process allocated, and clearing fresh pages
// then doubles the call (1.29 M rules, 20 MB: 5.5 ms with the block kept, 11 to
// 12.8 where it went back).
constexpr size_t kStagingKept = 64u << 20;
void staging_done(m6502_ctx* ctx) {
    if (ctx->staging.capacity() * sizeof(m6502_rule) > kStagingKept) ctx->staging.shrink_to_fit();
}

// Hands staged rules to the caller; what does not fit stays staged for the
// next m6502_fetch_rules.
int finish(m6502_ctx* ctx, m6502_rule* out, uint64_t cap, uint64_t* n_out) {
    const uint64_t n = ctx->staging.size();
    if (n_out) *n_out = n;
    const uint64_t k = out ? std::min(n, cap) : 0;
    if (k) std::memcpy(out, ctx->staging.data(), k * sizeof(m6502_rule));
    ctx->staging.erase(ctx->staging.begin(), ctx->staging.begin() + (long)k);
    if (n > k) return set_err(ctx, M6502_E_OVERFLOW, "rule buffer too small: the rest stays staged");
    staging_done(ctx);
    return M6502_OK;
}

// The end of a search: its rules are in the caller's buffer, the rest staged.
int finish_search(m6502_ctx* ctx, const RuleSink& sink, uint64_t* n_out) {
    const uint64_t rest = ctx->staging.size();
    if (n_out) *n_out = sink.n + rest;
    if (rest) return set_err(ctx, M6502_E_OVERFLOW, "rule buffer too small: the rest stays staged");
    staging_done(ctx);
    return M6502_OK;
}

bool valid_seq(const uint16_t* s, uint64_t n) {   // no early exit: the loop vectorises
    uint32_t bad = 0;
    for (uint64_t i = 0; i < n; i++) bad |= (uint32_t)((s[i] & 0xFFu) >= (uint32_t)NUM_OPS);
    return bad == 0;
}

// The opcode check of n instruction words already in device memory: one
// pass over them and a 4-byte read-back.
int check_ops_device(m6502_ctx* ctx, const uint16_t* d_ins, uint64_t n) {
    if (n == 0) return M6502_OK;
    TRY(ensure(ctx, ctx->opflag, sizeof(uint32_t)));
    CK(cudaMemsetAsync(ctx->opflag.p, 0, sizeof(uint32_t), ctx->stream));
    const uint32_t grid = (uint32_t)std::min<uint64_t>((n + 255) / 256, (uint64_t)ctx->sms * 16);
    k_check_ops<<<grid, 256, 0, ctx->stream>>>(d_ins, n, (uint32_t*)ctx->opflag.p);
    CKL("k_check_ops");
    uint32_t bad = 0;
    CK(cudaMemcpyAsync(&bad, ctx->opflag.p, sizeof bad, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return bad ? set_err(ctx, M6502_E_INVAL, "opcode out of range") : M6502_OK;
}

}  // namespace

// ---- tuning knobs and their cache file ----
bool tune_valid(const m6502_tune& t) {
    return t.exh_minb >= 2 && t.exh_minb <= 4 && t.ticket_batch >= 1 && t.ticket_batch <= 32 &&
           t.chunk_log2 >= 9 && t.chunk_log2 <= 16 && t.join_probe <= 1;
}

std::string device_tag(const m6502_ctx* ctx) {
    cudaDeviceProp prop;
    std::string name = "unknown";
    if (cudaGetDeviceProperties(&prop, ctx->device) == cudaSuccess) name = prop.name;
    for (char& c : name)
        if (!std::isalnum((unsigned char)c)) c = '_';
    return name + "-sm" + std::to_string(ctx->sms);
}

// $M6502_TUNE_CACHE, else $XDG_CACHE_HOME/m6502/ or ~/.cache/m6502/ plus a
// file per device; "" when none of these is set.
std::string tune_cache_path(const m6502_ctx* ctx) {
    if (const char* e = std::getenv("M6502_TUNE_CACHE")) return e;
    std::string dir;
    if (const char* x = std::getenv("XDG_CACHE_HOME")) dir = std::string(x) + "/m6502";
    else if (const char* h = std::getenv("HOME")) dir = std::string(h) + "/.cache/m6502";
    else return "";
    return dir + "/tune-" + device_tag(ctx) + ".txt";
}

const char* kTuneVersion = "m6502-b200 1.0 (sm_100a) tune 1";

// Reads a cache written by tune_save for this device; false when the file is
// missing, for another device or library, or out of range.
bool tune_load(const m6502_ctx* ctx, const std::string& path, m6502_tune* out) {
    FILE* f = std::fopen(path.c_str(), "r");
    if (!f) return false;
    char line[256];
    m6502_tune t{};
    std::string device, version;
    int seen = 0;
    while (std::fgets(line, sizeof line, f)) {
        std::string l(line);
        while (!l.empty() && (l.back() == '\n' || l.back() == '\r')) l.pop_back();
        const size_t eq = l.find('=');
        if (l.empty() || l[0] == '#' || eq == std::string::npos) continue;
        const std::string k = l.substr(0, eq), v = l.substr(eq + 1);
        const uint32_t u = (uint32_t)std::strtoul(v.c_str(), nullptr, 10);
        if (k == "device") device = v;
        else if (k == "version") version = v;
        else if (k == "exh_minb") { t.exh_minb = u; seen |= 1; }
        else if (k == "ticket_batch") { t.ticket_batch = u; seen |= 2; }
        else if (k == "chunk_log2") { t.chunk_log2 = u; seen |= 4; }
        else if (k == "join_probe") { t.join_probe = u; seen |= 8; }
    }
    std::fclose(f);
    if (seen != 15 || device != device_tag(ctx) || version != kTuneVersion || !tune_valid(t)) return false;
    *out = t;
    return true;
}

void tune_save(const m6502_ctx* ctx, const std::string& path, const m6502_tune& t, double ms,
               const std::vector<std::pair<m6502_tune, double>>& tried) {
    const size_t slash = path.rfind('/');
    if (slash != std::string::npos && slash > 0) {   // create the directory chain
        for (size_t p = path.find('/', 1); p != std::string::npos && p <= slash; p = path.find('/', p + 1))
            mkdir(path.substr(0, p).c_str(), 0755);
    }
    const std::string tmp = path + ".tmp" + std::to_string((long)getpid());
    FILE* f = std::fopen(tmp.c_str(), "w");
    if (!f) return;
    std::fprintf(f, "# m6502 tuning cache (m6502_autotune)\ndevice=%s\nversion=%s\n", device_tag(ctx).c_str(),
                 kTuneVersion);
    std::fprintf(f, "exh_minb=%u\nticket_batch=%u\nchunk_log2=%u\njoin_probe=%u\nms=%.4f\n", t.exh_minb,
                 t.ticket_batch, t.chunk_log2, t.join_probe, ms);
    for (const auto& tr : tried)   // every configuration timed, in order
        std::fprintf(f, "# tried exh_minb=%u ticket_batch=%u chunk_log2=%u join_probe=%u ms=%.4f\n",
                     tr.first.exh_minb, tr.first.ticket_batch, tr.first.chunk_log2, tr.first.join_probe, tr.second);
    std::fclose(f);
    std::rename(tmp.c_str(), path.c_str());   // readers see the old file or the whole new one
}

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

const char* m6502_version(void) { return "m6502-b200 1.0 (sm_100a)"; }

}  // extern "C"

int m6502_ctx_device(const m6502_ctx* ctx) { return ctx ? ctx->device : 0; }

extern "C" {

int m6502_create(m6502_ctx** out, const m6502_opts* opts) {
    if (!out) return M6502_E_INVAL;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return M6502_E_NODEV;
    m6502_ctx* ctx = new m6502_ctx();
    if (opts) {
        ctx->device = opts->device;
        if (opts->targets_per_pass) ctx->pass_targets = opts->targets_per_pass;
    }
    if (ctx->device < 0 || ctx->device >= ndev) { delete ctx; return M6502_E_INVAL; }
    if (cudaSetDevice(ctx->device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&ctx->ev0) != cudaSuccess || cudaEventCreate(&ctx->ev1) != cudaSuccess) {
        delete ctx;
        return M6502_E_CUDA;
    }
    bool ev_ok = true;
    for (cudaEvent_t& e : ctx->sev) ev_ok = ev_ok && cudaEventCreate(&e) == cudaSuccess;
    for (cudaEvent_t& e : ctx->sev2) ev_ok = ev_ok && cudaEventCreate(&e) == cudaSuccess;
    for (cudaEvent_t& e : ctx->aev) ev_ok = ev_ok && cudaEventCreate(&e) == cudaSuccess;
    for (cudaEvent_t& e : ctx->cev) ev_ok = ev_ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    ev_ok = ev_ok && cudaStreamCreateWithFlags(&ctx->copy, cudaStreamNonBlocking) == cudaSuccess;
    if (!ev_ok) {
        delete ctx;
        return M6502_E_CUDA;
    }
    cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, ctx->device);
    int rc = init_ctx(ctx);
    if (rc != M6502_OK) {
        fprintf(stderr, "m6502_create: %s\n", ctx->err.c_str());
        m6502_destroy(ctx);
        return rc;
    }
    {   // knobs an earlier m6502_autotune chose for this device
        const std::string path = tune_cache_path(ctx);
        m6502_tune t;
        if (!path.empty() && tune_load(ctx, path, &t)) ctx->tune = t;
    }
    *out = ctx;
    return M6502_OK;
}

void m6502_destroy(m6502_ctx* ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    for (void* p : ctx->table_blocks) cudaFree(p);
    DevBuf* bufs[] = {&ctx->cfp4, &ctx->cfp1, &ctx->cmeta1, &ctx->targets, &ctx->ids, &ctx->tfp, &ctx->tmeta,
                      &ctx->surv, &ctx->fail, &ctx->items, &ctx->rules, &ctx->cnt, &ctx->best,
                      &ctx->pins, &ctx->poffs,
                      &ctx->enum_count, &ctx->st_tins, &ctx->st_toffs, &ctx->st_tout, &ctx->st_tbytes,
                      &ctx->st_chains, &ctx->st_entries, &ctx->st_vidx, &ctx->st_proven, &ctx->st_cnt,
                      &ctx->st_pidx, &ctx->st_mex, &ctx->st_probs, &ctx->st_traj, &ctx->st_row, &ctx->st_keys,
                      &ctx->st_keys2, &ctx->st_vals2, &ctx->st_rep, &ctx->st_ord, &ctx->st_verdict,
                      &ctx->st_vlist, &ctx->st_vpos, &ctx->st_sort_tmp, &ctx->c2_keys_in, &ctx->c2_idx_in,
                      &ctx->c2_sort_tmp, &ctx->go_keys, &ctx->go_keys2, &ctx->go_ord, &ctx->go_round,
                      &ctx->go_sort_tmp, &ctx->jitems, &ctx->cnt_slots, &ctx->st_vphase, &ctx->st_pphase,
                      &ctx->st_live, &ctx->st_rounds, &ctx->st_proven_was,
                      &ctx->tall, &ctx->opflag, &ctx->order, &ctx->match, &ctx->pairs_io};
    for (DevBuf* b : bufs) if (b->p) cudaFree(b->p);
    for (cudaEvent_t e : ctx->sev) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : ctx->sev2) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : ctx->aev) if (e) cudaEventDestroy(e);
    for (cudaGraphExec_t e : ctx->graph.exec) cudaGraphExecDestroy(e);
    for (cudaEvent_t e : ctx->cev) if (e) cudaEventDestroy(e);
    if (ctx->copy) cudaStreamDestroy(ctx->copy);
    if (ctx->h_io) cudaFreeHost(ctx->h_io);
    for (m6502_ctx::PassGraph& g : ctx->pass_graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    for (auto& t : ctx->cand2) {
        if (t.keys.p) cudaFree(t.keys.p);
        if (t.idx.p) cudaFree(t.idx.p);
        if (t.pw.p) cudaFree(t.pw.p);
    }
    if (ctx->ev0) cudaEventDestroy(ctx->ev0);
    if (ctx->ev1) cudaEventDestroy(ctx->ev1);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

const char* m6502_last_error(const m6502_ctx* ctx) { return ctx ? ctx->err.c_str() : "no context"; }

void* m6502_stream(m6502_ctx* ctx) { return ctx ? (void*)ctx->stream : nullptr; }

int m6502_check_pairs(m6502_ctx* ctx, uint64_t n, const uint16_t* t_insns, const uint32_t* t_offs,
                      const uint16_t* c_insns, const uint32_t* c_offs, uint8_t dead_flags,
                      uint32_t checks, uint32_t sweep, uint32_t exh_mode, uint8_t* out,
                      uint8_t* flagdiff) {
    if (!ctx) return M6502_E_INVAL;
    Call call(ctx);
    if (n == 0) return M6502_OK;
    if (!t_insns || !t_offs || !c_insns || !c_offs || !out) return set_err(ctx, M6502_E_INVAL, "NULL buffer");
    if (sweep > M6502_SWEEP_FULL || exh_mode > M6502_EXH_BRUTE) return set_err(ctx, M6502_E_INVAL, "bad sweep mode");
    for (uint64_t i = 0; i < n; i++) {
        uint32_t tl = t_offs[i + 1] - t_offs[i], cl = c_offs[i + 1] - c_offs[i];
        if (t_offs[i + 1] < t_offs[i] || c_offs[i + 1] < c_offs[i] || tl < 1 || tl > kMaxSeq || cl < 1 || cl > kMaxSeq)
            return set_err(ctx, M6502_E_INVAL, "sequence length must be 1..16");
    }
    if (!valid_seq(t_insns + t_offs[0], t_offs[n] - t_offs[0]) || !valid_seq(c_insns + c_offs[0], c_offs[n] - c_offs[0]))
        return set_err(ctx, M6502_E_INVAL, "opcode out of range");
    CK(cudaSetDevice(ctx->device));
    // One block on the device: verdicts, FlagDiffs and counters (copied back),
    // counters, offsets and instructions (copied in).  Up to kPairsStaged bytes
    // each way go through page-locked memory in one copy; more go from and to
    // the caller's buffers.
    const bool exh = (checks & M6502_CHECK_EXH) != 0, vectors = (checks & 3u) || flagdiff;
    const size_t tin = t_offs[n], cin = c_offs[n];
    auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    const size_t o_fd = n, o_cnt = up16(2 * n), o_to = up16(o_cnt + sizeof(Counters)), o_co = o_to + up16((n + 1) * 4),
                 o_ti = o_co + up16((n + 1) * 4), o_ci = o_ti + up16(tin * 2), total = o_ci + up16(cin * 2);
    const bool staged = total <= kPairsStaged;
    TRY(ensure(ctx, ctx->pairs_io, total));
    TRY(ensure(ctx, ctx->fail, n * 4));
    TRY(ensure(ctx, ctx->order, n * 4));
    if (staged && ctx->h_io_bytes < total) {
        if (ctx->h_io) cudaFreeHost(ctx->h_io);
        ctx->h_io = nullptr;
        ctx->h_io_bytes = 0;
        CK(cudaHostAlloc(&ctx->h_io, total, cudaHostAllocDefault));
        ctx->h_io_bytes = total;
    }
    uint8_t* d = (uint8_t*)ctx->pairs_io.p;
    uint8_t* h = (uint8_t*)ctx->h_io;
    Counters hc;
    std::memset(&hc, 0, sizeof hc);
    hc.surv = n;
    const struct { size_t at, bytes; const void* from; } parts[] = {
        {o_cnt, sizeof hc, &hc}, {o_to, (n + 1) * 4, t_offs}, {o_co, (n + 1) * 4, c_offs}, {o_ti, tin * 2, t_insns},
        {o_ci, cin * 2, c_insns}};
    for (const auto& p : parts) {
        if (staged) std::memcpy(h + p.at, p.from, p.bytes);
        else CK(cudaMemcpyAsync(d + p.at, p.from, p.bytes, cudaMemcpyHostToDevice, ctx->stream));
    }
    if (staged) CK(cudaMemcpyAsync(d + o_cnt, h + o_cnt, total - o_cnt, cudaMemcpyHostToDevice, ctx->stream));
    CsrSource src{(const uint16_t*)(d + o_ti), (const uint32_t*)(d + o_to), (const uint16_t*)(d + o_ci),
                  (const uint32_t*)(d + o_co), dead_flags};
    Counters* cnt = (Counters*)(d + o_cnt);
    if (vectors) {
        const uint32_t grid = (uint32_t)std::min<uint64_t>((n + kWarpsPerBlock - 1) / kWarpsPerBlock, (uint64_t)ctx->sms * 16);
        k_pair_vectors<<<grid, 256, 0, ctx->stream>>>(src, n, d, d + o_fd);
        CKL("k_pair_vectors");
    }
    uint64_t icap = std::max<uint64_t>(ctx->items.bytes / sizeof(Item), 1u << 16);
    for (int attempt = 0;; attempt++) {
        if (exh) {
            TRY(ensure(ctx, ctx->items, icap * sizeof(Item)));
            ExhArgs ea{(uint32_t*)ctx->fail.p, (Item*)ctx->items.p, icap, cnt, &cnt->v[0][0], sweep,
                       exh_mode == M6502_EXH_BRUTE};
            TRY(launch_verify(ctx, src, &cnt->surv, n, ea));
        }
        k_pair_verdicts<<<(uint32_t)std::min<uint64_t>((n + 255) / 256, (uint64_t)ctx->sms * 8), 256, 0, ctx->stream>>>(
            n, vectors ? checks & 3u : 0u, exh ? (const uint32_t*)ctx->fail.p : nullptr, d);
        CKL("k_pair_verdicts");
        CK(cudaMemcpyAsync(staged ? (void*)(h + o_cnt) : (void*)&hc, cnt, sizeof hc, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaMemcpyAsync(staged ? h : out, d, n, cudaMemcpyDeviceToHost, ctx->stream));
        if (flagdiff) CK(cudaMemcpyAsync(staged ? h + o_fd : flagdiff, d + o_fd, n, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        if (staged) std::memcpy(&hc, h + o_cnt, sizeof hc);
        const uint64_t items = hc.v[0][0].items;
        if (items <= icap) break;
        if (attempt >= 4) return set_err(ctx, M6502_E_NOMEM, "work-item queue kept overflowing");
        icap = items + items / 4 + 1024;
        std::memset(&hc, 0, sizeof hc);
        hc.surv = n;
        CK(cudaMemcpyAsync(cnt, &hc, sizeof hc, cudaMemcpyHostToDevice, ctx->stream));
    }
    if (staged) {
        std::memcpy(out, h, n);
        if (flagdiff) std::memcpy(flagdiff, h + o_fd, n);
    }
    return M6502_OK;
}

int m6502_fingerprint(m6502_ctx* ctx, uint64_t n, const uint16_t* insns, const uint32_t* offs, uint8_t* out) {
    if (!ctx) return M6502_E_INVAL;
    Call call(ctx);
    if (n == 0) return M6502_OK;
    if (!insns || !offs || !out) return set_err(ctx, M6502_E_INVAL, "NULL buffer");
    for (uint64_t i = 0; i < n; i++) {
        uint32_t l = offs[i + 1] - offs[i];
        if (offs[i + 1] < offs[i] || l > kMaxSeq) return set_err(ctx, M6502_E_INVAL, "sequence length must be 0..16");
    }
    if (!valid_seq(insns + offs[0], offs[n] - offs[0])) return set_err(ctx, M6502_E_INVAL, "opcode out of range");
    CK(cudaSetDevice(ctx->device));
    TRY(ensure(ctx, ctx->pins, (size_t)offs[n] * 2 + 2));
    TRY(ensure(ctx, ctx->poffs, (n + 1) * 4));
    TRY(ensure(ctx, ctx->tfp, n * 32 * 8));
    CK(cudaMemcpyAsync(ctx->pins.p, insns, (size_t)offs[n] * 2, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->poffs.p, offs, (n + 1) * 4, cudaMemcpyHostToDevice, ctx->stream));
    k_fingerprint<CsrSeqs><<<ctx->fp_blocks, 256, 0, ctx->stream>>>(
        CsrSeqs{(const uint16_t*)ctx->pins.p, (const uint32_t*)ctx->poffs.p}, n, (uint64_t*)ctx->tfp.p, nullptr);
    CKL("k_fingerprint");
    std::vector<uint64_t> h(n * 32);
    CK(cudaMemcpyAsync(h.data(), ctx->tfp.p, n * 32 * 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    for (uint64_t i = 0; i < n; i++)
        for (int v = 0; v < 8; v++)
            for (int b = 0; b < 8; b++) out[i * 64 + v * 8 + b] = (uint8_t)(h[i * 32 + v] >> (8 * b));
    return M6502_OK;
}

int m6502_exec_batch(m6502_ctx* ctx, uint64_t n, const uint16_t* insns, const uint32_t* offs,
                     const uint64_t* states_in, uint64_t* states_out) {
    if (!ctx) return M6502_E_INVAL;
    Call call(ctx);
    if (n == 0) return M6502_OK;
    if (!insns || !offs || !states_in || !states_out) return set_err(ctx, M6502_E_INVAL, "NULL buffer");
    for (uint64_t i = 0; i < n; i++)
        if (offs[i + 1] < offs[i]) return set_err(ctx, M6502_E_INVAL, "offsets must not decrease");
    if (!valid_seq(insns + offs[0], offs[n] - offs[0])) return set_err(ctx, M6502_E_INVAL, "opcode out of range");
    CK(cudaSetDevice(ctx->device));
    TRY(ensure(ctx, ctx->pins, (size_t)offs[n] * 2 + 2));
    TRY(ensure(ctx, ctx->poffs, (n + 1) * 4));
    TRY(ensure(ctx, ctx->tfp, n * 16));
    uint64_t* d_in = (uint64_t*)ctx->tfp.p;
    uint64_t* d_out = d_in + n;
    CK(cudaMemcpyAsync(ctx->pins.p, insns, (size_t)offs[n] * 2, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->poffs.p, offs, (n + 1) * 4, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(d_in, states_in, n * 8, cudaMemcpyHostToDevice, ctx->stream));
    uint32_t grid = (uint32_t)std::min<uint64_t>((n + 255) / 256, (uint64_t)ctx->sms * 16);
    k_exec_batch<<<grid, 256, 0, ctx->stream>>>(CsrSeqs{(const uint16_t*)ctx->pins.p, (const uint32_t*)ctx->poffs.p},
                                                n, d_in, d_out);
    CKL("k_exec_batch");
    CK(cudaMemcpyAsync(states_out, d_out, n * 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return M6502_OK;
}

int m6502_fetch_rules(m6502_ctx* ctx, m6502_rule* out, uint64_t cap, uint64_t* n_out) {
    if (!ctx) return M6502_E_INVAL;
    Call call(ctx);
    if (cap && !out) return set_err(ctx, M6502_E_INVAL, "NULL out");
    return finish(ctx, out, cap, n_out);
}

int m6502_search(m6502_ctx* ctx, const m6502_search_cfg* cfg, const uint16_t* targets, uint64_t n,
                 uint32_t tlen, m6502_rule* out, uint64_t cap, uint64_t* n_out, m6502_stats* stats) {
    if (!ctx) return M6502_E_INVAL;
    Call call(ctx);
    TRY(check_cfg(ctx, cfg));
    if (tlen < 1 || tlen > 3) return set_err(ctx, M6502_E_INVAL, "target length must be 1..3");
    if (n > 0xFFFFFFFFull) return set_err(ctx, M6502_E_INVAL, "too many targets for one call");
    if (n && !targets) return set_err(ctx, M6502_E_INVAL, "NULL targets");
    const bool on_dev = (cfg->flags & M6502_TARGETS_ON_DEVICE) != 0;
    const bool async_ok = cfg->semantics == M6502_SEM_CUDA && cfg->max_cand_len <= 1 &&
                          n <= (uint64_t)kMaxAsyncPasses * ctx->pass_targets;
    // Opcodes are checked on the host only for host targets searched pass
    // by pass; queued searches check them on the device, in every pass.
    if (!on_dev && !async_ok && !valid_seq(targets, n * tlen))
        return set_err(ctx, M6502_E_INVAL, "opcode out of range");
    CK(cudaSetDevice(ctx->device));
    m6502_stats st;
    std::memset(&st, 0, sizeof st);
    ctx->staging.clear();
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    RuleSink sink{out, cap, 0};
    // A queued search of host targets copies them to the device pass by pass
    // and runs as a device-resident one (CUDA graphs included).
    const uint16_t* q_targets = targets;
    if (async_ok && n && !on_dev) {
        TRY(ensure(ctx, ctx->tall, n * tlen * sizeof(uint16_t)));
        q_targets = (const uint16_t*)ctx->tall.p;
    }
    if (on_dev && !async_ok) TRY(check_ops_device(ctx, q_targets, n * tlen));
    for (uint64_t b = async_ok ? n : 0; b < n; b += ctx->pass_targets) {   // passes one by one otherwise
        uint64_t nt = std::min<uint64_t>(ctx->pass_targets, n - b);
        const uint16_t* d_t;
        if (on_dev) {
            d_t = targets + b * tlen;
        } else {
            TRY(ensure(ctx, ctx->targets, nt * tlen * 2));
            CK(cudaMemcpyAsync(ctx->targets.p, targets + b * tlen, nt * tlen * 2, cudaMemcpyHostToDevice, ctx->stream));
            d_t = (const uint16_t*)ctx->targets.p;
        }
        TRY(run_pass(ctx, *cfg, d_t, nt, tlen, nullptr, b, sink, &st));
    }
    if (async_ok && n) {
        TRY(search_async(ctx, *cfg, q_targets, on_dev ? nullptr : targets, n, tlen, &st, sink));
    }
    CK(cudaEventRecord(ctx->ev1, ctx->stream));
    CK(cudaEventSynchronize(ctx->ev1));
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    st.ms_device = ms;
    if (stats) *stats = st;
    if (cfg->flags & M6502_COUNT_ONLY) {
        if (n_out) *n_out = st.rules;
        return M6502_OK;
    }
    return finish_search(ctx, sink, n_out);
}

int m6502_enumerate(m6502_ctx* ctx, const m6502_search_cfg* cfg, uint32_t tlen, uint32_t first,
                    uint32_t last, m6502_rule* out, uint64_t cap, uint64_t* n_out, m6502_stats* stats) {
    if (!ctx) return M6502_E_INVAL;
    Call call(ctx);
    TRY(check_cfg(ctx, cfg));
    if (tlen < 2 || tlen > 3) return set_err(ctx, M6502_E_INVAL, "enumeration length must be 2 or 3");
    if (last > (uint32_t)kNumInsns) last = kNumInsns;
    if (first > last) return set_err(ctx, M6502_E_INVAL, "first > last");
    CK(cudaSetDevice(ctx->device));
    m6502_stats st;
    std::memset(&st, 0, sizeof st);
    ctx->staging.clear();
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    RuleSink sink{out, cap, 0};
    const uint64_t per_first = tlen == 2 ? (uint64_t)kNumInsns : (uint64_t)kNumInsns * kNumInsns;
    // first-op slices sized so one slice holds at most ~pass_targets ids
    const uint64_t ops_per_slice = std::max<uint64_t>(1, ctx->pass_targets / per_first);
    TRY(ensure(ctx, ctx->enum_count, sizeof(unsigned long long)));
    for (uint64_t f = first; f < last; f += ops_per_slice) {
        uint64_t f1 = std::min<uint64_t>(last, f + ops_per_slice);
        uint64_t id0 = f * per_first, id1 = f1 * per_first, span = id1 - id0;
        TRY(ensure(ctx, ctx->targets, span * tlen * 2));
        TRY(ensure(ctx, ctx->ids, span * 8));
        CK(cudaMemsetAsync(ctx->enum_count.p, 0, sizeof(unsigned long long), ctx->stream));
        uint32_t grid = (uint32_t)std::min<uint64_t>((span + 255) / 256, (uint64_t)ctx->sms * 16);
        k_enum_targets<<<grid, 256, 0, ctx->stream>>>(id0, id1, tlen, (uint16_t*)ctx->targets.p,
                                                       (uint64_t*)ctx->ids.p, span,
                                                       (unsigned long long*)ctx->enum_count.p);
        CKL("k_enum_targets");
        unsigned long long nt = 0;
        CK(cudaMemcpyAsync(&nt, ctx->enum_count.p, sizeof nt, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        for (uint64_t b = 0; b < nt; b += ctx->pass_targets) {
            uint64_t m = std::min<uint64_t>(ctx->pass_targets, nt - b);
            TRY(run_pass(ctx, *cfg, (const uint16_t*)ctx->targets.p + b * tlen, m, tlen,
                         (const uint64_t*)ctx->ids.p + b, 0, sink, &st));
        }
    }
    CK(cudaEventRecord(ctx->ev1, ctx->stream));
    CK(cudaEventSynchronize(ctx->ev1));
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    st.ms_device = ms;
    if (stats) *stats = st;
    if (cfg->flags & M6502_COUNT_ONLY) {
        if (n_out) *n_out = st.rules;
        return M6502_OK;
    }
    return finish_search(ctx, sink, n_out);
}

int m6502_tune_get(m6502_ctx* ctx, m6502_tune* out) {
    if (!ctx || !out) return M6502_E_INVAL;
    Call call(ctx);
    *out = ctx->tune;
    return M6502_OK;
}

int m6502_tune_set(m6502_ctx* ctx, const m6502_tune* t) {
    if (!ctx || !t) return M6502_E_INVAL;
    Call call(ctx);
    if (!tune_valid(*t)) return set_err(ctx, M6502_E_INVAL, "tuning knob out of range");
    ctx->tune = *t;
    return M6502_OK;
}

int m6502_autotune(m6502_ctx* ctx, const char* cache_path, uint32_t flags, m6502_tune* chosen, double* ms_out) {
    if (!ctx) return M6502_E_INVAL;
    std::string path = cache_path ? std::string(cache_path) : tune_cache_path(ctx);
    if (ms_out) *ms_out = 0.0;
    if (!(flags & M6502_TUNE_FORCE)) {
        m6502_tune t;
        if (!path.empty() && tune_load(ctx, path, &t)) {
            TRY(m6502_tune_set(ctx, &t));
            if (chosen) *chosen = t;
            return M6502_OK;
        }
    }
    // Calibration workload: every pruned length-2 target, enumerated on the device.
    DevBuf tg, ids, count;
    const uint64_t span = (uint64_t)kNumInsns * kNumInsns;
    unsigned long long nt = 0;
    {
        Call call(ctx);
        CK(cudaSetDevice(ctx->device));
        TRY(ensure(ctx, tg, span * 2 * sizeof(uint16_t)));
        TRY(ensure(ctx, ids, span * sizeof(uint64_t)));
        TRY(ensure(ctx, count, sizeof(unsigned long long)));
        CK(cudaMemsetAsync(count.p, 0, sizeof(unsigned long long), ctx->stream));
        const uint32_t grid = (uint32_t)std::min<uint64_t>((span + 255) / 256, (uint64_t)ctx->sms * 16);
        k_enum_targets<<<grid, 256, 0, ctx->stream>>>(0, span, 2, (uint16_t*)tg.p, (uint64_t*)ids.p, span,
                                                       (unsigned long long*)count.p);
        CKL("k_enum_targets");
        CK(cudaMemcpyAsync(&nt, count.p, sizeof nt, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        cudaFree(ids.p);
        cudaFree(count.p);
        ids.p = count.p = nullptr;
    }
    m6502_search_cfg cfg{};
    cfg.semantics = M6502_SEM_CUDA;
    cfg.sweep = M6502_SWEEP_FULL;
    cfg.exh_mode = M6502_EXH_CONES;
    cfg.max_cand_len = 1;
    cfg.flags = M6502_TARGETS_ON_DEVICE | M6502_COUNT_ONLY;
    std::vector<std::pair<m6502_tune, double>> tried;
    // median of three timed runs after one untimed run (which records the graph)
    auto measure = [&](const m6502_tune& t, double* ms) -> int {
        TRY(m6502_tune_set(ctx, &t));
        double v[3];
        for (int r = -1; r < 3; r++) {
            m6502_stats st;
            uint64_t n = 0;
            TRY(m6502_search(ctx, &cfg, (const uint16_t*)tg.p, nt, 2, nullptr, 0, &n, &st));
            if (r >= 0) v[r] = st.ms_device;
        }
        std::sort(v, v + 3);
        *ms = v[1];
        tried.emplace_back(t, v[1]);
        return M6502_OK;
    };
    m6502_tune best = ctx->tune;
    best.exh_minb = 4; best.ticket_batch = 4; best.chunk_log2 = 11; best.join_probe = 1;   // join_probe: no effect
    double best_ms = 0;
    int rc = measure(best, &best_ms);
    // Coordinate descent: each knob in turn over its candidates, the others held.
    const uint32_t minb_v[] = {2, 3, 4}, tb_v[] = {2, 4, 8, 16}, ck_v[] = {10, 11, 12, 13};
    using Field = uint32_t m6502_tune::*;
    struct Knob { Field f; const uint32_t* v; int n; };
    const Knob knobs[] = {{&m6502_tune::exh_minb, minb_v, 3},
                          {&m6502_tune::ticket_batch, tb_v, 4}, {&m6502_tune::chunk_log2, ck_v, 4}};
    for (const Knob& k : knobs) {
        if (rc != M6502_OK) break;
        const m6502_tune base = best;
        for (int i = 0; i < k.n && rc == M6502_OK; i++) {
            if (base.*k.f == k.v[i]) continue;
            m6502_tune t = base;
            t.*k.f = k.v[i];
            double ms = 0;
            rc = measure(t, &ms);
            if (rc == M6502_OK && ms < best_ms) { best = t; best_ms = ms; }
        }
    }
    cudaFree(tg.p);
    tg.p = nullptr;
    TRY(rc);
    TRY(m6502_tune_set(ctx, &best));
    if (!path.empty()) tune_save(ctx, path, best, best_ms, tried);   // a cache that cannot be written is not an error
    if (chosen) *chosen = best;
    if (ms_out) *ms_out = best_ms;
    return M6502_OK;
}


}  // extern "C"

namespace {

// Per-device set-up of the fixed-scratch entry point: constant tables and
// the device address of g_static_scratch (in host code the array's name is
// only a stand-in, never a device address).
struct StaticDevice {
    bool ready = false;
    StaticScratch* scratch = nullptr;
    int blocks = 0;
};
constexpr int kStaticMaxDevices = 64;
StaticDevice g_static_dev[kStaticMaxDevices];
std::mutex g_static_mu;

int static_setup(int dev, StaticDevice** out) {
    std::lock_guard<std::mutex> lk(g_static_mu);
    StaticDevice& d = g_static_dev[dev];
    if (!d.ready) {
        uint64_t vec[32];
        for (int v = 0; v < 32; v++) {
            uint64_t x = 0;
            for (int b = 0; b < 8; b++) x |= (uint64_t)kVectors[v][b] << (8 * b);
            vec[v] = x;
        }
        uint16_t dep[NUM_OPS][NUM_LOCS], wr[NUM_OPS], sw[NUM_OPS];
        for (uint32_t op = 0; op < NUM_OPS; op++) {
            wr[op] = (uint16_t)op_deps(op, dep[op]);
            sw[op] = (uint16_t)sweep_locs_of_reads(op_reads(op));
        }
        uint32_t rep[32], x4[NUM_OPS];
        for (int i = 0; i < 32; i++) rep[i] = kRepValues[i];
        for (uint32_t op = 0; op < NUM_OPS; op++) x4[op] = x4_desc(op);
        if (cudaMemcpyToSymbol(c_vec, vec, sizeof vec) != cudaSuccess ||
            cudaMemcpyToSymbol(c_dep, dep, sizeof dep) != cudaSuccess ||
            cudaMemcpyToSymbol(c_wr, wr, sizeof wr) != cudaSuccess ||
            cudaMemcpyToSymbol(c_sweep, sw, sizeof sw) != cudaSuccess ||
            cudaMemcpyToSymbol(c_x4d, x4, sizeof x4) != cudaSuccess ||
            cudaMemcpyToSymbol(c_rep, rep, sizeof rep) != cudaSuccess ||
            cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess)   // the caller's stream does not wait for that one
            return M6502_E_CUDA;
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_static_scratch) != cudaSuccess || !ptr) return M6502_E_CUDA;
        int sms = 0, occ = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_exhaustive_static, 256, 0) != cudaSuccess)
            return M6502_E_CUDA;
        d.scratch = (StaticScratch*)ptr;
        d.blocks = sms * std::max(occ, 1);
        d.ready = true;
    }
    *out = &d;
    return M6502_OK;
}

}  // namespace

extern "C" {

int m6502_exhaustive_static(uint64_t n, const uint16_t* t_insns, const uint32_t* t_offs,
                            const uint16_t* c_insns, const uint32_t* c_offs, uint8_t dead_flags,
                            uint32_t sweep, uint8_t* out, void* stream) {
    if (n > kStaticMaxPairs) return M6502_E_TOOBIG;
    if (sweep > M6502_SWEEP_FULL) return M6502_E_INVAL;
    if (n == 0) return M6502_OK;
    if (!t_insns || !t_offs || !c_insns || !c_offs || !out) return M6502_E_INVAL;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return M6502_E_NODEV;
    if (dev < 0 || dev >= kStaticMaxDevices) return M6502_E_INVAL;
    StaticDevice* d = nullptr;
    int rc = static_setup(dev, &d);
    if (rc != M6502_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(&d->scratch->cnt, 0, sizeof(Counters), st) != cudaSuccess) return M6502_E_CUDA;
    StaticCsrSource src{t_insns, t_offs, c_insns, c_offs, dead_flags};
    uint64_t grid = std::min<uint64_t>((uint64_t)d->blocks, (n + kWarpsPerBlock - 1) / kWarpsPerBlock);
    k_exhaustive_static<<<(uint32_t)grid, 256, 0, st>>>(src, n, sweep, d->scratch);
    if (cudaGetLastError() != cudaSuccess) return M6502_E_CUDA;
    uint64_t vgrid = std::min<uint64_t>((n + 255) / 256, 4096);
    k_static_verdicts<<<(uint32_t)vgrid, 256, 0, st>>>(d->scratch, n, out);
    if (cudaGetLastError() != cudaSuccess) return M6502_E_CUDA;
    return M6502_OK;
}

}  // extern "C"

#include "stoke.cuh"
