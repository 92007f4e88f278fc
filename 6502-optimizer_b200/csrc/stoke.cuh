// stoke.cuh -- batched STOKE (stochastic superoptimisation) on B200.
// Included at the end of engine.cu (one translation unit: it shares the
// constant tables and the exhaustive kernels).
//
// The reference runs one goroutine per MCMC chain (pkg/stoke/search.go:88-163):
// mutate (mutator.go:30-115), cost on the test vectors (cost.go:32-81),
// Metropolis accept with T *= decay (mcmc.go:51-81), and ExhaustiveCheck of
// every shorter zero-mismatch best (search.go:102-155).  Here eight lanes run
// one chain: they draw the same random numbers (one splitmix64 state per
// chain), each evaluates the candidate on four of the test vectors, and the
// cost is a reduction over them.  Chains run in
// epochs of S steps; after each epoch the shorter zero-cost bests found during
// it are checked on all 32 vectors and proved by the exhaustive kernels, and
// the chains of proven targets restart (the reference's NewChain) or stop.

namespace {

struct StokeChain {
    uint16_t cur[kMaxSeq];
    uint16_t best[kMaxSeq];
    uint64_t rng;
    uint64_t step;          // steps this chain has run (all restarts)
    uint64_t since;         // steps since the last (re)start
    float temp;
    int32_t cost, best_cost;
    uint32_t target;
    uint32_t accepted;
    uint32_t diff;          // MidCheck vectors on which the current candidate differs
    uint8_t len, best_len, status, pad;   // status: 0 (re)start, 1 running, 2 stopped
};

struct StokeEntry {        // a shorter zero-cost best awaiting proof
    uint32_t chain, target;
    uint64_t step;
    uint16_t ins[kMaxSeq];
    uint8_t len, dead_flags, pad[6];
};

struct StokeCounters {
    unsigned long long entries, vec_ok, proofs, undecided, accepted, traj;
    unsigned long long reps;      // distinct (target, candidate) pairs among the vec_ok entries
    unsigned long long max_ord;   // largest per-target ordinal of a distinct pair
    unsigned long long round_n;   // pairs verified in the current round
    unsigned long long verified;  // pairs verified this epoch (all rounds)
    unsigned long long ex_rows;   // chains given a row of the learned proposal this epoch
    unsigned long long live;      // chains still searching this epoch
};

constexpr uint32_t kVerifyBatch = 8;   // distinct candidates per target per round under stop_on_proof
constexpr uint32_t kStokeDeferBits = 24;   // first verification phase: cones of at most 2^24 states

// Sort key of an entry: target, length, then a 33-bit hash of the
// instructions, so that identical (target, candidate) pairs are adjacent and
// shorter candidates of a target come first.
__device__ __forceinline__ uint64_t entry_key(const StokeEntry& e) {
    uint64_t h = 0x5EED;
    for (int i = 0; i < e.len; i++) h = key_mix(h ^ ((uint64_t)e.ins[i] + (uint64_t)(i + 1) * 0x9E3779B97F4A7C15ull));
    return ((uint64_t)e.target << 38) | ((uint64_t)(e.len & 31u) << 33) | (h >> 31);
}

__device__ __forceinline__ bool same_candidate(const StokeEntry& a, const StokeEntry& b) {
    if (a.target != b.target || a.len != b.len) return false;
    for (int i = 0; i < a.len; i++)
        if (a.ins[i] != b.ins[i]) return false;
    return true;
}

struct StokeTargets {
    const uint16_t* ins;
    const uint32_t* off;
    const uint64_t* out;    // [target][32] outputs on the test vectors (P & PMask)
    const uint8_t* bytes;   // Go byte size of each target
};

struct StokeParams {
    uint32_t cost_mode;     // M6502_COST_*
    uint32_t dead;
    uint32_t max_len;       // 0: max(len + 2, 10)
    uint32_t chains_per_target;
    uint32_t steps;         // steps of this epoch
    uint64_t seed;
    float decay;            // per-step temperature factor
    float t_start;
    const float* cdf;       // PROPOSAL_MIXED: 330 cumulative probabilities (3 heads) per row
    const uint32_t* row;    // per chain: its row of cdf, or kNoRow (uniform moves only)
    float learned_frac;
    m6502_mlp_example* traj;   // improving moves as labelled examples (optional)
    uint64_t traj_cap;
};

constexpr uint64_t kSmStep = 0x9E3779B97F4A7C15ull;
__device__ __forceinline__ uint64_t sm_mix(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t sm_next(uint64_t& x) { return sm_mix(x += kSmStep); }
// Uniform integer in [0, n) from the top half of a draw: high half of a
// 32x32 product (bias < n / 2^32).
__device__ __forceinline__ uint32_t below(uint32_t top, uint32_t n) { return __umulhi(top, n); }
__device__ __forceinline__ float unit(uint32_t top) { return (float)(top >> 8) * (1.0f / 16777216.0f); }
__device__ __forceinline__ uint32_t sm_below(uint64_t& x, uint32_t n) { return below((uint32_t)(sm_next(x) >> 32), n); }
__device__ __forceinline__ float sm_unit(uint64_t& x) { return unit((uint32_t)(sm_next(x) >> 32)); }

// Index drawn from one head of a chain's cumulative distribution (entries
// [a, b) of the chain's row in shared memory hold running sums): the first
// entry above a uniform point of the head's range (the last one if rounding
// leaves none).
__device__ __forceinline__ int cdf_sample(const float* cdf, int a, int b, uint64_t& rng) {
    const float base = a > 0 ? cdf[a - 1] : 0.0f;
    const float r = base + sm_unit(rng) * (cdf[b - 1] - base);
    int lo = a, hi = b - 1;   // the answer lies in [lo, hi]
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cdf[mid] > r) hi = mid; else lo = mid + 1;
    }
    return lo - a;
}

constexpr uint32_t kNoRow = 0xFFFFFFFFu;

// The model's input for every chain still searching: target, current
// candidate and its vector mismatch mask (a chain about to (re)start uses
// the target itself).  Chains of proved targets under stop_on_proof get no
// row, nor do the chains that keep the uniform proposal (the first
// `uniform8` of every 8 chains of a target); the others get consecutive
// rows (row[ci]), so the forward pass runs over the live model-driven
// chains only.
__global__ void k_stoke_examples(const StokeChain* __restrict__ chains, uint32_t n_chains, uint32_t cpt,
                                 StokeTargets tg, const uint32_t* __restrict__ proven, uint32_t stop_on_proof,
                                 uint32_t uniform8, m6502_mlp_example* __restrict__ ex, uint32_t* __restrict__ row,
                                 StokeCounters* __restrict__ sc) {
    const int lane = threadIdx.x & 31;
    for (uint32_t ci = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); ci < n_chains;
         ci += gridDim.x * kWarpsPerBlock) {
        const StokeChain& ch = chains[ci];
        const uint32_t t = ci / cpt, t0 = tg.off[t], tlen = tg.off[t + 1] - t0;
        if (ch.status == 2 || (stop_on_proof && proven[t]) || ((ci % cpt) & 7u) < uniform8) {
            if (lane == 0) row[ci] = kNoRow;
            continue;
        }
        unsigned long long r = 0;
        if (lane == 0) r = atomicAdd(&sc->ex_rows, 1ull);
        r = __shfl_sync(kFull, r, 0);
        if (lane == 0) row[ci] = (uint32_t)r;
        const bool fresh = ch.status != 1;
        m6502_mlp_example& x = ex[r];
        if (lane < 8) x.target[lane] = lane < (int)tlen ? tg.ins[t0 + lane] : 0;
        if (lane < 16) x.cand[lane] = fresh ? (lane < (int)tlen ? tg.ins[t0 + lane] : 0) : ch.cur[lane];
        if (lane == 0) {
            x.diff = fresh ? 0u : ch.diff;
            x.tlen = (uint8_t)min(tlen, 8u);
            x.clen = fresh ? (uint8_t)tlen : ch.len;
            x.pos = x.op = x.imm = 0;
            x.weight = 0;
        }
    }
}

// Softmax outputs -> running sums per head (in place), one thread per chain.
__global__ void k_cdf(float* __restrict__ p, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float* r = p + (size_t)i * 330;
        const int cut[4] = {0, 16, 74, 330};
        for (int h = 0; h < 3; h++) {
            float s = 0.0f;
            for (int k = cut[h]; k < cut[h + 1]; k++) { s += r[k]; r[k] = s; }
        }
    }
}

// The chains still searching, listed (their order does not matter: a chain's
// course depends on its own state alone); chains of proved targets stop.
__global__ void k_stoke_live(StokeChain* __restrict__ chains, uint32_t n_chains, uint32_t cpt,
                             const uint32_t* __restrict__ proven, uint32_t stop_on_proof, uint32_t* __restrict__ list,
                             StokeCounters* __restrict__ sc) {
    for (uint32_t base = blockIdx.x * blockDim.x; base < n_chains; base += gridDim.x * blockDim.x) {
        const uint32_t ci = base + threadIdx.x;
        bool live = ci < n_chains && chains[ci].status != 2;
        if (live && stop_on_proof && proven[ci / cpt]) {
            chains[ci].status = 2;
            live = false;
        }
        const unsigned vote = __ballot_sync(kFull, live);
        const int lane = threadIdx.x & 31;
        unsigned long long b = 0;
        if (lane == 0 && vote) b = atomicAdd(&sc->live, (unsigned long long)__popc(vote));
        b = __shfl_sync(kFull, b, 0) + __popc(vote & ((1u << lane) - 1u));
        if (live) list[b] = ci;
    }
}

// One epoch of the listed chains: eight lanes per chain, up to four chains per
// warp.  Lane `sub` of a chain runs the candidate on vectors 4 sub .. 4 sub +
// 3, packed in one word per register; the chain's random numbers are drawn by
// all its lanes alike.  Cost of a candidate: COST_REF: 1000 x mismatching QC
// vectors + bytes + cycles / 100 (cost.go:32-81); COST_HAMMING: differing
// output bits over the 32 vectors + bytes + cycles / 100.
// Bound by issue and by each chain's serial steps.  A warp per chain paid the
// random numbers, the mutation and the acceptance (two thirds of its
// instructions) for one chain; here up to four chains pay them together,
// written without branches on the kind of move and with the table-driven
// executor (four opcodes in a warp: one course instead of four arms of the
// switch; 21.3 -> 20.1 ms for the whole run).  A warp's steps are a serial
// chain at seven cycles per instruction, so few chains spread over more warps
// first (kEpochWarps: three per scheduler; 20.1 ms, with four 20.7, six 23.4),
// and only listed chains get a warp: the ones of a proved target lie together
// and left some SMs idle, others twice as busy.
// 256 targets x 128 chains x 4,000 steps: all epochs 20.3 -> 11.4 ms.
constexpr int kEpochChains = 8;               // chains per block of 64 threads, at most
constexpr uint32_t kEpochWarps = 148 * 4 * 3;
__global__ void __launch_bounds__(64) k_stoke_epoch(StokeChain* __restrict__ chains, const uint32_t* __restrict__ list,
                                                      StokeTargets tg, StokeParams prm,
                                                      StokeEntry* __restrict__ entries, uint64_t ecap,
                                                      StokeCounters* __restrict__ sc) {
    __shared__ uint16_t s_seq[kEpochChains][3][kMaxSeq];   // two candidates in turn, the best
    __shared__ float s_cdf[kEpochChains][330];             // the chain's learned distributions, staged once
    __shared__ uint8_t s_size[64];                         // bytes | cycles << 4 by opcode
    __shared__ uint4 s_row[NUM_OPS][3];                    // X4Row by opcode
    __shared__ uint32_t s_st[X4S_COUNT][64];               // each lane's registers
    for (int i = threadIdx.x; i < (int)NUM_OPS * 3; i += 64) (&s_row[0][0])[i] = g_x4row[i];
    if (threadIdx.x < 64)
        s_size[threadIdx.x] = (uint8_t)(bytes_go(threadIdx.x) | cycles(threadIdx.x) << 4);
    __syncthreads();
    const int lane = threadIdx.x & 31, sub = lane & 7, g = threadIdx.x >> 3, shift = lane & 24;
    const unsigned gmask = 0xFFu << shift;   // the chain's lanes
    const uint32_t live = (uint32_t)sc->live;
    const uint32_t per = min(4u, (live + kEpochWarps - 1) / kEpochWarps);   // chains per warp
    const uint32_t li = (blockIdx.x * 2u + (threadIdx.x >> 5)) * per + (uint32_t)(lane >> 3);
    const bool on = (uint32_t)(lane >> 3) < per && li < live;
    if (!__any_sync(kFull, on)) return;
    const uint32_t ci = list[on ? li : 0];
    StokeChain& ch = chains[ci];
    const uint32_t t = ci / prm.chains_per_target, status = ch.status;
    const uint32_t t0 = tg.off[t], tlen = tg.off[t + 1] - t0;
    const uint32_t tbytes = tg.bytes[t];
    const uint32_t pm = (kPMask & ~prm.dead & 0xFFu) * kB1;
    const int max_len = (int)(prm.max_len ? prm.max_len : max(tlen + 2u, 10u));
    uint16_t *cur = s_seq[g][0], *cand = s_seq[g][1], *best = s_seq[g][2];
    const int p0 = sub, p1 = sub + 8;   // the two positions this lane moves
    // this lane's four vectors and the target's outputs on them
    const uint32_t* vw = c_vec4[sub];
    const St vin{vw[0], vw[1], vw[2], vw[3], vw[4], vw[5], vw[6], vw[7]};
    St want{0, 0, 0, 0, 0, 0, 0, 0};
    for (int k = 0; k < 4; k++) {
        const St o = unpack(tg.out[(uint64_t)t * 32 + 4 * sub + k]);
        want.a |= o.a << (8 * k); want.x |= o.x << (8 * k); want.y |= o.y << (8 * k); want.p |= o.p << (8 * k);
        want.s |= o.s << (8 * k); want.m |= o.m << (8 * k); want.s0 |= o.s0 << (8 * k); want.s1 |= o.s1 << (8 * k);
    }
    // Cost of seq[0..n): every lane of the chain gets it; `zero`: no vector
    // differs; `vm`: the vectors that do.  All chains of the warp call it together.
    auto cost_of = [&](const uint16_t* seq, int n, bool& zero, uint32_t& vm, uint32_t& size) -> int32_t {
        uint32_t* st = &s_st[0][threadIdx.x];
        st[X4S_A * 64] = vin.a; st[X4S_X * 64] = vin.x; st[X4S_Y * 64] = vin.y; st[X4S_S * 64] = vin.s;
        st[X4S_M * 64] = vin.m; st[X4S_S0 * 64] = vin.s0; st[X4S_S1 * 64] = vin.s1;
        uint32_t p = vin.p, insn = seq[0];
        X4Row row = load_row(s_row[min(insn & 0xFFu, NUM_OPS - 1u)]);
        uint32_t operand = x4_operand(row, insn);
        for (int i = 0; i < n; i++) {
            const uint32_t next = seq[min(i + 1, kMaxSeq - 1)];   // it, its row and operand in flight while this one runs
            const X4Row next_row = load_row(s_row[min(next & 0xFFu, NUM_OPS - 1u)]);
            const uint32_t next_operand = x4_operand(next_row, next);
            exec_x4o(st, 64, p, row, operand);
            row = next_row;
            operand = next_operand;
        }
        const St s{st[X4S_A * 64], st[X4S_X * 64], st[X4S_Y * 64], p, st[X4S_S * 64], st[X4S_M * 64], st[X4S_S0 * 64],
                   st[X4S_S1 * 64]};
        const uint32_t da = s.a ^ want.a, dx = s.x ^ want.x, dy = s.y ^ want.y, dp = (s.p ^ want.p) & pm, ds = s.s ^ want.s,
                       dm = s.m ^ want.m, d0 = s.s0 ^ want.s0, d1 = s.s1 ^ want.s1;
        const uint32_t differ = ~x4_zero(da | dx | dy | dp | ds | dm | d0 | d1) & kH;   // 0x80 in the bytes that do
        uint32_t v = ((differ >> 7) * 0x10204080u) >> 28;                               // their four bits, gathered
        v <<= 4 * sub;
        const uint32_t h = (uint32_t)(__popc(da) + __popc(dx) + __popc(dy) + __popc(dp) + __popc(ds) + __popc(dm) +
                                      __popc(d0) + __popc(d1));
        const uint32_t z0 = p0 < n ? s_size[seq[p0] & 63u] : 0u, z1 = p1 < n ? s_size[seq[p1] & 63u] : 0u;
        uint32_t sum = h | ((z0 & 15u) + (z1 & 15u)) << 12 | ((z0 >> 4) + (z1 >> 4)) << 20;   // no field overflows in 8 lanes
        for (int o = 1; o < 8; o <<= 1) {
            sum += __shfl_xor_sync(kFull, sum, o);
            v |= __shfl_xor_sync(kFull, v, o);
        }
        vm = v;
        size = (sum >> 12) & 0xFFu;
        const int32_t base = (int32_t)(size + (sum >> 20) / 100u);
        if (prm.cost_mode == M6502_COST_REF) {
            zero = (v & 0xFFu) == 0;
            return 1000 * __popc(v & 0xFFu) + base;
        }
        zero = (sum & 0xFFFu) == 0;
        return (int32_t)(sum & 0xFFFu) + base;
    };
    int len = 0, best_len = 0;
    int32_t cost = 0, best_cost = 0;
    float temp = 0.0f;
    uint64_t rng = 0, step = ch.step, since = ch.since;
    uint32_t accepted = 0, diff = 0, size = 0;
    bool zero = false;
    const uint32_t crow = on && prm.cdf ? prm.row[ci] : kNoRow;
    const float* cdf = nullptr;
    if (crow != kNoRow) {
        const float* r = prm.cdf + (size_t)crow * 330;
        for (int i = sub; i < 330; i += 8) s_cdf[g][i] = r[i];
        cdf = s_cdf[g];
    }
    const bool fresh = on && status == 0;   // NewChain (mcmc.go:28-49): start from the target
    for (int p = p0; p < kMaxSeq; p += 8) {
        const uint16_t c = fresh ? (p < (int)tlen ? tg.ins[t0 + p] : (uint16_t)0) : ch.cur[p];
        cur[p] = c;
        cand[p] = 0;
        best[p] = fresh ? c : ch.best[p];
    }
    __syncwarp();
    {
        const int32_t c0 = cost_of(cur, fresh ? (int)tlen : 0, zero, diff, size);
        if (fresh) {
            len = best_len = (int)tlen;
            rng = prm.seed + (uint64_t)ci * 0x9E3779B97F4A7C15ull + step;
            temp = prm.t_start;
            since = 0;
            cost = best_cost = c0;
        } else if (on) {
            len = ch.len; best_len = ch.best_len;
            cost = ch.cost; best_cost = ch.best_cost;
            temp = ch.temp; rng = ch.rng;
            diff = ch.diff;
        }
    }
    for (uint32_t it = 0; it < prm.steps; it++, step++, since++) {
        // Mutate (mutator.go:30-44): replace 40%, swap 20%, delete 20%,
        // insert 10%, change immediate 10%.
        // The generator's next values do not depend on each other: the five
        // that a step can use are computed side by side.
        uint32_t z[5];
#pragma unroll
        for (int k = 0; k < 5; k++) z[k] = (uint32_t)(sm_mix(rng + (uint64_t)(k + 1) * kSmStep) >> 32);
        const uint32_t r = below(z[0], 100);
        uint32_t unit_z;   // the value the acceptance draws if it needs one
        int kind = r < 40 ? 0 : r < 60 ? 1 : r < 80 ? 2 : r < 90 ? 3 : 4;
        if (kind == 3 && len >= max_len) kind = 0;              // InsertInstruction falls back
        uint32_t immpos = 0;                                    // positions with an operand
        if (__any_sync(kFull, kind == 4)) {
            const unsigned b0 = __ballot_sync(kFull, p0 < len && has_imm(cur[p0] & 0xFFu));
            const unsigned b1 = __ballot_sync(kFull, p1 < len && has_imm(cur[p1] & 0xFFu));
            immpos = ((b0 >> shift) & 0xFFu) | ((b1 >> shift) & 0xFFu) << 8;
            if (kind == 4 && !immpos) kind = 0;                 // ChangeImmediate falls back
        }
        int pos = 0;
        uint32_t op = 0, imm = 0;
        const bool fresh_insn = kind == 0 || kind == 3;
        bool learned = false;
        if (cdf && fresh_insn) learned = unit(z[1]) < prm.learned_frac;
        if (learned) {   // position, opcode, operand from the model's distributions
            rng += 2 * kSmStep;
            const int lim = kind == 0 ? len : len + 1;
            pos = cdf_sample(cdf, 0, 16, rng);
            if (pos >= lim) pos = (int)sm_below(rng, (uint32_t)lim);
            op = (uint32_t)cdf_sample(cdf, 16, 74, rng);
            imm = has_imm(op) ? (uint32_t)cdf_sample(cdf, 74, 330, rng) : 0u;
            unit_z = (uint32_t)(sm_mix(rng + kSmStep) >> 32);
        } else {         // uniform: position, then opcode over the 58, then operand (mutator.go:108-115), as far as the move has them
            if (cdf && fresh_insn) {   // one value went to the choice above
                rng += kSmStep;
                z[1] = z[2]; z[2] = z[3]; z[3] = z[4];
                z[4] = (uint32_t)(sm_mix(rng + 5 * kSmStep) >> 32);
            }
            const uint32_t places = kind == 4 ? (uint32_t)__popc(immpos) : (uint32_t)(kind == 3 ? len + 1 : kind == 1 ? len - 1 : len);
            const bool placed = kind == 1 || kind == 2 ? len > 1 : true;
            uint32_t used = 1;
            if (placed) { pos = (int)below(z[1], places); used = 2; }
            if (fresh_insn) { op = below(z[2], NUM_OPS); used = 3; }
            if (kind == 4) {
                uint32_t m = immpos;
                for (int q = 0; q < pos; q++) m &= m - 1;
                pos = __ffs(m) - 1;
                op = cur[pos] & 0xFFu;
            }
            unit_z = used == 1 ? z[1] : used == 2 ? z[2] : z[3];
            if ((fresh_insn || kind == 4) && has_imm(op)) {
                imm = below(unit_z, 256);
                unit_z = used == 2 ? z[3] : z[4];
                used++;
            }
            rng += used * kSmStep;
        }
        const uint16_t ins = (uint16_t)(op | imm << 8);
        const bool moved = kind == 1 ? len >= 2 : kind == 2 ? len > 1 : true;
        const int nlen = kind == 3 ? len + 1 : kind == 2 && moved ? len - 1 : len;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int p = k ? p1 : p0;
            int q = p;   // the position the instruction comes from
            if (kind == 1 && moved) q = p == pos ? p + 1 : p == pos + 1 ? p - 1 : p;
            if (kind == 2 && moved) q = p < pos ? p : p + 1;
            if (kind == 3) q = p <= pos ? p : p - 1;
            uint16_t v = q < kMaxSeq ? cur[q] : (uint16_t)0;
            if ((kind == 0 || kind >= 3) && p == pos) v = ins;
            cand[p] = v;
        }
        __syncwarp();
        uint32_t ndiff;
        const int32_t ncost = cost_of(cand, on ? nlen : 0, zero, ndiff, size);
        // Metropolis accept (mcmc.go:51-81)
        const int32_t delta = ncost - cost;
        bool acc = delta <= 0;
        if (!acc && temp > 0.0f) {
            rng += kSmStep;
            acc = unit(unit_z) < __expf(-(float)delta / temp);
        }
        acc = acc && on;
        if (acc && prm.traj && delta < 0 && (kind == 0 || kind == 3)) {   // an improving move: training example
            unsigned long long e = 0;
            if (sub == 0) e = atomicAdd(&sc->traj, 1ull);
            e = __shfl_sync(gmask, e, shift);
            if (e < prm.traj_cap) {
                m6502_mlp_example& x = prm.traj[e];
                x.target[sub] = sub < (int)tlen ? tg.ins[t0 + sub] : 0;
                x.cand[p0] = p0 < len ? cur[p0] : 0;
                x.cand[p1] = p1 < len ? cur[p1] : 0;
                if (sub == 0) {
                    x.diff = diff; x.tlen = (uint8_t)min(tlen, 8u); x.clen = (uint8_t)len;
                    x.pos = (uint8_t)pos; x.op = (uint8_t)(ins & 0xFFu); x.imm = (uint8_t)(ins >> 8);
                    x.weight = 1;
                }
            }
        }
        if (acc) {
            uint16_t* tmp = cur; cur = cand; cand = tmp;
            diff = ndiff;
            len = nlen;
            cost = ncost;
            accepted++;
            if (ncost < best_cost) {
                best[p0] = cur[p0];
                best[p1] = cur[p1];
                best_len = len;
                best_cost = ncost;
                // verification trigger (search.go:101): zero mismatches and shorter
                if (zero && size < tbytes) {
                    unsigned long long e = 0;
                    if (sub == 0) e = atomicAdd(&sc->entries, 1ull);
                    e = __shfl_sync(gmask, e, shift);
                    if (e < ecap) {
                        entries[e].ins[p0] = cur[p0];
                        entries[e].ins[p1] = cur[p1];
                        if (sub == 0) {
                            entries[e].chain = ci; entries[e].target = t; entries[e].step = step;
                            entries[e].len = (uint8_t)best_len; entries[e].dead_flags = 0;
                        }
                    }
                }
            }
        }
        temp *= prm.decay;
        __syncwarp();
    }
    if (!on) return;
    ch.cur[p0] = cur[p0]; ch.cur[p1] = cur[p1];
    ch.best[p0] = best[p0]; ch.best[p1] = best[p1];
    if (sub == 0) {
        ch.len = (uint8_t)len; ch.best_len = (uint8_t)best_len;
        ch.cost = cost; ch.best_cost = best_cost;
        ch.temp = temp; ch.rng = rng; ch.step = step; ch.since = since;
        ch.target = t; ch.status = 1; ch.diff = diff;
        ch.accepted += accepted;
        atomicAdd(&sc->accepted, (unsigned long long)accepted);
    }
}

// All 32 test vectors of each entry (a shorter zero-cost best): entries
// that agree on every vector go on to ExhaustiveCheck (their indices are
// compacted into vidx, with their sort keys); FlagDiff over the QC vectors is
// recorded for masked runs.
__global__ void k_stoke_vectors(StokeEntry* __restrict__ entries, uint64_t ecap, StokeTargets tg, uint32_t dead,
                                uint32_t* __restrict__ vidx, uint64_t* __restrict__ keys,
                                StokeCounters* __restrict__ sc) {
    const int lane = threadIdx.x & 31;
    const uint64_t n = min((uint64_t)sc->entries, ecap);
    const uint64_t mask = cmp_mask(dead);
    for (uint64_t e = (uint64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); e < n;
         e += (uint64_t)gridDim.x * kWarpsPerBlock) {
        StokeEntry& en = entries[e];
        St s = unpack(c_vec[lane]);
        for (int i = 0; i < en.len; i++) exec(s, en.ins[i]);
        const uint64_t x = fp_of(s) ^ tg.out[(uint64_t)en.target * 32 + lane];
        const bool ok = __all_sync(kFull, (x & mask) == 0);
        uint32_t fd = lane < 8 ? ((uint32_t)(x >> 24) & kPMask) : 0u;
        fd = __reduce_or_sync(kFull, fd);
        if (lane == 0) {
            en.dead_flags = (uint8_t)(dead ? fd : 0u);   // FlagDiff (verifier.go:591-604)
            if (ok) {
                const unsigned long long k = atomicAdd(&sc->vec_ok, 1ull);
                vidx[k] = (uint32_t)e;
                keys[k] = entry_key(en);
            }
        }
    }
}

// Pairs (target, entry) of the entries that passed all vectors.
struct StokeSource {
    static constexpr int kMaxT = kMaxSeq, kMaxC = kMaxSeq;
    const StokeEntry* entries;
    const uint32_t* vidx;
    StokeTargets tg;
    uint32_t dead_;
    __device__ void load(uint64_t p, uint16_t* st, uint16_t* sc, int& tn, int& cn, uint32_t& dead,
                         int lane) const {
        const StokeEntry& e = entries[vidx[p]];
        const uint32_t t0 = tg.off[e.target];
        tn = (int)(tg.off[e.target + 1] - t0);
        cn = e.len;
        if (lane < tn) st[lane] = tg.ins[t0 + lane];
        if (lane < cn) sc[lane] = e.ins[lane];
        dead = dead_;
    }
    __device__ void load_lane(uint64_t p, uint16_t* st, uint16_t* sc, int ld, int& tn, int& cn, uint32_t& dead) const {
        const StokeEntry& e = entries[vidx[p]];
        const uint32_t t0 = tg.off[e.target];
        tn = (int)(tg.off[e.target + 1] - t0);
        cn = e.len;
        for (int i = 0; i < tn; i++) st[i * ld] = tg.ins[t0 + i];
        for (int i = 0; i < cn; i++) sc[i * ld] = e.ins[i];
        dead = dead_;
    }
    __device__ uint64_t target_id(uint64_t) const { return kNoTarget; }   // candidates may be empty
    __device__ uint32_t weight(uint64_t) const { return 1u; }
};

// Over the vec_ok entries sorted by key (one CTA, chunks of 1,024): rep[i] =
// sorted position of the first entry with the same (target, candidate) --
// the one that is verified for all of them -- and ord[i] = the ordinal of
// that distinct candidate within its target (0 for the shortest).
__global__ void __launch_bounds__(1024) k_stoke_dedupe(const uint64_t* __restrict__ keys,
                                                       const uint32_t* __restrict__ vals,
                                                       const StokeEntry* __restrict__ entries,
                                                       uint32_t* __restrict__ rep, uint32_t* __restrict__ ord,
                                                       StokeCounters* __restrict__ sc) {
    using Scan = cub::BlockScan<uint32_t, 1024>;
    using Reduce = cub::BlockReduce<uint32_t, 1024>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ typename Reduce::TempStorage rtmp;
    __shared__ uint32_t carry[3];   // running count of distinct pairs, last rep position, count at target start
    const uint32_t n = (uint32_t)sc->vec_ok;
    if (threadIdx.x == 0) carry[0] = carry[1] = carry[2] = 0;
    __syncthreads();
    uint32_t max_ord = 0;
    for (uint32_t base = 0; base < n; base += 1024) {
        const uint32_t i = base + threadIdx.x;
        const bool valid = i < n;
        bool is_rep = false, tstart = false;
        if (valid) {
            if (i == 0) is_rep = tstart = true;
            else {
                const uint64_t k = keys[i], kp = keys[i - 1];
                tstart = (k >> 38) != (kp >> 38);
                is_rep = tstart || k != kp || !same_candidate(entries[vals[i]], entries[vals[i - 1]]);
            }
        }
        uint32_t r, rp, rs;
        Scan(tmp).InclusiveSum(is_rep ? 1u : 0u, r);
        __syncthreads();
        r += carry[0];
        Scan(tmp).InclusiveScan(is_rep ? i : 0u, rp, cub::Max());
        __syncthreads();
        rp = max(rp, carry[1]);
        Scan(tmp).InclusiveScan(tstart ? r : 0u, rs, cub::Max());
        __syncthreads();
        rs = max(rs, carry[2]);
        if (valid) {
            rep[i] = rp;
            ord[i] = r - rs;
            max_ord = max(max_ord, r - rs);
        }
        __syncthreads();
        if (threadIdx.x == 1023) { carry[0] = r; carry[1] = rp; carry[2] = rs; }
        __syncthreads();
    }
    const uint32_t m = Reduce(rtmp).Reduce(max_ord, cub::Max());
    if (threadIdx.x == 0) { sc->reps = carry[0]; sc->max_ord = m; }
}

// One verification round: the distinct pairs whose per-target ordinal lies
// in [lo, hi) -- or, with deferred_only, the pairs an earlier round deferred
// -- skipping targets already proved when stop_on_proof is set.
__global__ void k_stoke_select(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                               const uint32_t* __restrict__ rep, const uint32_t* __restrict__ ord, uint32_t lo,
                               uint32_t hi, uint32_t stop_on_proof, const uint32_t* __restrict__ proven,
                               const uint32_t* __restrict__ verdict, uint32_t deferred_only,
                               uint32_t* __restrict__ vlist, uint32_t* __restrict__ vpos,
                               StokeCounters* __restrict__ sc) {
    const uint32_t n = (uint32_t)sc->vec_ok;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (rep[i] != i) continue;
        if (deferred_only ? verdict[i] != 4u : (ord[i] < lo || ord[i] >= hi)) continue;
        if (stop_on_proof && proven[(uint32_t)(keys[i] >> 38)]) continue;
        const unsigned long long p = atomicAdd(&sc->round_n, 1ull);
        vlist[p] = vals[i];
        vpos[p] = i;
    }
}

// Verdicts of a round -> the sorted positions of the verified pairs; proved
// targets are marked.
__global__ void k_stoke_verdicts(const uint32_t* __restrict__ fail, const uint32_t* __restrict__ vpos,
                                 const uint64_t* __restrict__ keys, uint32_t* __restrict__ verdict,
                                 uint8_t* __restrict__ vphase, uint32_t phase, uint32_t* __restrict__ proven,
                                 StokeCounters* __restrict__ sc) {
    const uint32_t n = (uint32_t)sc->round_n;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t i = vpos[p];
        verdict[i] = fail[p];
        vphase[i] = (uint8_t)phase;
        if (fail[p] == 0) proven[(uint32_t)(keys[i] >> 38)] = 1;
        if (fail[p] == 3) atomicAdd(&sc->undecided, 1ull);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->verified += n;   // deferred pairs count again when swept
}

// Every vec_ok entry whose distinct pair was proved becomes a proof (as in
// the reference, each chain's verified best is one result); its chain
// restarts (search.go:151-154).
__global__ void k_stoke_collect(const uint32_t* __restrict__ vals, const uint32_t* __restrict__ rep,
                                const uint32_t* __restrict__ verdict, const uint8_t* __restrict__ vphase,
                                const StokeEntry* __restrict__ entries, StokeCounters* __restrict__ sc,
                                StokeChain* __restrict__ chains, uint32_t* __restrict__ proof_idx,
                                uint8_t* __restrict__ proof_phase, uint64_t pcap) {
    const uint32_t n = (uint32_t)sc->vec_ok;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (verdict[rep[i]] != 0) continue;
        const uint32_t e = vals[i];
        const unsigned long long k = atomicAdd(&sc->proofs, 1ull);
        if (k < pcap) { proof_idx[k] = e; proof_phase[k] = vphase[rep[i]]; }
        chains[entries[e].chain].status = 0;
    }
}

}  // namespace

extern "C" {

int m6502_stoke_run(m6502_ctx* ctx, const m6502_stoke_cfg* cfg, const uint16_t* t_insns, const uint32_t* t_offs,
                    uint32_t n_targets, m6502_stoke_result* results, m6502_stoke_proof* proofs, uint64_t cap,
                    uint64_t* n_proofs, m6502_stoke_stats* stats) {
    if (!ctx) return M6502_E_INVAL;
    Call call(ctx);
    if (!cfg || !t_insns || !t_offs || (n_targets && !results)) return set_err(ctx, M6502_E_INVAL, "NULL argument");
    if (cfg->cost > M6502_COST_HAMMING || cfg->sweep > M6502_SWEEP_FULL || cfg->max_len > (uint32_t)kMaxSeq)
        return set_err(ctx, M6502_E_INVAL, "bad STOKE configuration");
    if (cfg->proposal > M6502_PROPOSAL_MIXED || (cfg->proposal == M6502_PROPOSAL_MIXED && !cfg->model))
        return set_err(ctx, M6502_E_INVAL, "PROPOSAL_MIXED needs a model");
    for (uint32_t t = 0; t < n_targets; t++) {
        uint32_t l = t_offs[t + 1] - t_offs[t];
        if (t_offs[t + 1] < t_offs[t] || l < 1 || l > (uint32_t)kMaxSeq - 2)
            return set_err(ctx, M6502_E_INVAL, "STOKE targets must have 1..14 instructions");
    }
    if (!valid_seq(t_insns + t_offs[0], t_offs[n_targets] - t_offs[0])) return set_err(ctx, M6502_E_INVAL, "opcode out of range");
    if (n_proofs) *n_proofs = 0;
    if (n_targets == 0) return M6502_OK;
    CK(cudaSetDevice(ctx->device));
    const uint32_t cpt = cfg->chains_per_target ? cfg->chains_per_target : 128;
    const uint64_t n_chains64 = (uint64_t)cpt * n_targets;
    if (n_chains64 > (1ull << 26)) return set_err(ctx, M6502_E_INVAL, "too many chains");
    const uint32_t n_chains = (uint32_t)n_chains64;
    const uint64_t steps = cfg->steps ? cfg->steps : 1000000ull;
    const uint32_t spe = cfg->steps_per_epoch ? cfg->steps_per_epoch : 1000u;
    const size_t tin = t_offs[n_targets];
    // targets and their vector outputs
    TRY(ensure(ctx, ctx->st_tins, tin * 2 + 2));
    TRY(ensure(ctx, ctx->st_toffs, ((size_t)n_targets + 1) * 4));
    TRY(ensure(ctx, ctx->st_tout, (size_t)n_targets * 32 * 8));
    TRY(ensure(ctx, ctx->st_tbytes, n_targets));
    std::vector<uint8_t> tb(n_targets);
    for (uint32_t t = 0; t < n_targets; t++) {
        uint32_t b = 0;
        for (uint32_t i = t_offs[t]; i < t_offs[t + 1]; i++) b += bytes_go(t_insns[i] & 0xFFu);
        tb[t] = (uint8_t)std::min(b, 255u);
    }
    CK(cudaMemcpyAsync(ctx->st_tins.p, t_insns, tin * 2, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->st_toffs.p, t_offs, ((size_t)n_targets + 1) * 4, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->st_tbytes.p, tb.data(), n_targets, cudaMemcpyHostToDevice, ctx->stream));
    k_fingerprint<CsrSeqs><<<ctx->fp_blocks, 256, 0, ctx->stream>>>(
        CsrSeqs{(const uint16_t*)ctx->st_tins.p, (const uint32_t*)ctx->st_toffs.p}, n_targets,
        (uint64_t*)ctx->st_tout.p, nullptr);
    CKL("k_fingerprint(stoke targets)");
    // chains, entries, proofs
    const uint64_t ecap = (uint64_t)n_chains * 16 + 1024;   // <= 16 shorter bests per chain and epoch
    TRY(ensure(ctx, ctx->st_chains, (size_t)n_chains * sizeof(StokeChain)));
    TRY(ensure(ctx, ctx->st_entries, ecap * sizeof(StokeEntry)));
    TRY(ensure(ctx, ctx->st_vidx, ecap * 4));
    TRY(ensure(ctx, ctx->fail, ecap * 4));
    TRY(ensure(ctx, ctx->order, ecap * 4));
    TRY(ensure(ctx, ctx->st_proven, (size_t)n_targets * 4));
    TRY(ensure(ctx, ctx->st_live, (size_t)n_chains * 4));
    TRY(ensure(ctx, ctx->st_proven_was, (size_t)n_targets * 4));
    TRY(ensure(ctx, ctx->st_cnt, sizeof(StokeCounters)));
    TRY(ensure(ctx, ctx->st_pidx, ecap * 4));
    TRY(ensure(ctx, ctx->st_keys, ecap * 8));
    TRY(ensure(ctx, ctx->st_keys2, ecap * 8));
    TRY(ensure(ctx, ctx->st_vals2, ecap * 4));
    TRY(ensure(ctx, ctx->st_rep, ecap * 4));
    TRY(ensure(ctx, ctx->st_ord, ecap * 4));
    TRY(ensure(ctx, ctx->st_verdict, ecap * 4));
    TRY(ensure(ctx, ctx->st_vlist, ecap * 4));
    TRY(ensure(ctx, ctx->st_vpos, ecap * 4));
    TRY(ensure(ctx, ctx->st_vphase, ecap));
    TRY(ensure(ctx, ctx->st_pphase, ecap));
    size_t sort_bytes = 0;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                       (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)ecap, 0, 64, ctx->stream));
    TRY(ensure(ctx, ctx->st_sort_tmp, sort_bytes + 256));
    CK(cudaMemsetAsync(ctx->st_chains.p, 0, (size_t)n_chains * sizeof(StokeChain), ctx->stream));
    CK(cudaMemsetAsync(ctx->st_proven.p, 0, (size_t)n_targets * 4, ctx->stream));
    StokeTargets tg{(const uint16_t*)ctx->st_tins.p, (const uint32_t*)ctx->st_toffs.p,
                    (const uint64_t*)ctx->st_tout.p, (const uint8_t*)ctx->st_tbytes.p};
    StokeParams prm;
    prm.cost_mode = cfg->cost;
    prm.dead = cfg->dead_flags;
    prm.max_len = cfg->max_len;
    prm.chains_per_target = cpt;
    prm.seed = cfg->seed;
    prm.cdf = nullptr;
    prm.row = nullptr;
    prm.learned_frac = cfg->learned_frac > 0 ? cfg->learned_frac : 0.5f;
    prm.traj = nullptr;
    prm.traj_cap = 0;
    const bool mixed = cfg->proposal == M6502_PROPOSAL_MIXED;
    if (mixed) {
        TRY(ensure(ctx, ctx->st_mex, (size_t)n_chains * sizeof(m6502_mlp_example)));
        TRY(ensure(ctx, ctx->st_probs, (size_t)n_chains * 330 * sizeof(float)));
        TRY(ensure(ctx, ctx->st_row, (size_t)n_chains * sizeof(uint32_t)));
    }
    uint64_t traj_total = 0;
    if (cfg->trajectories && cfg->traj_cap) {
        prm.traj_cap = std::min<uint64_t>(cfg->traj_cap, 1u << 20);
        TRY(ensure(ctx, ctx->st_traj, prm.traj_cap * sizeof(m6502_mlp_example)));
        prm.traj = (m6502_mlp_example*)ctx->st_traj.p;
    }
    if (cfg->cost == M6502_COST_REF) {
        prm.t_start = 1.0f;
        prm.decay = (float)(cfg->decay > 0.0 && cfg->decay < 1.0 ? cfg->decay : 0.9999);
    } else {
        double t0 = cfg->t_start > 0 ? cfg->t_start : 1.0, t1 = cfg->t_end > 0 ? cfg->t_end : 0.1;
        prm.t_start = (float)t0;
        prm.decay = (float)std::pow(t1 / t0, 1.0 / (double)steps);
    }
    std::vector<StokeEntry> h_entries;
    std::vector<m6502_stoke_proof> found;
    std::vector<double> first_ms(n_targets, -1.0);
    std::vector<uint64_t> first_step(n_targets, 0), first_epoch(n_targets, 0);
    m6502_stoke_stats st;
    std::memset(&st, 0, sizeof st);
    StokeCounters* sc = (StokeCounters*)ctx->st_cnt.p;
    Counters* cnt = (Counters*)ctx->cnt.p;
    uint64_t icap = std::max<uint64_t>(ctx->items.bytes / sizeof(Item), 1u << 16);
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    float ms_chains = 0, ms_verify = 0;
    uint32_t proven_targets = 0;
    uint32_t epoch_len = cfg->first_epoch ? std::min(cfg->first_epoch, spe) : spe;
    for (uint64_t done = 0; done < steps;) {
        // The first epoch runs uniform moves only: a target the first random
        // moves rewrite costs no forward pass; from the second epoch on the
        // model is refreshed for the chains still searching.
        const bool use_model = mixed && done > 0;
        const uint32_t e_steps = (uint32_t)std::min<uint64_t>(epoch_len, steps - done);
        epoch_len = (uint32_t)std::min<uint64_t>((uint64_t)epoch_len * 2, spe);
        prm.steps = e_steps;
        CK(cudaMemsetAsync(sc, 0, sizeof(StokeCounters), ctx->stream));
        CK(cudaEventRecord(ctx->sev[0], ctx->stream));
        prm.cdf = nullptr;
        if (use_model) {   // refresh the learned proposal of the chains still searching
            k_stoke_examples<<<(n_chains + kWarpsPerBlock - 1) / kWarpsPerBlock, 256, 0, ctx->stream>>>(
                (const StokeChain*)ctx->st_chains.p, n_chains, cpt, tg, (const uint32_t*)ctx->st_proven.p,
                cfg->stop_on_proof, std::min<uint32_t>(cfg->uniform_chains, 8u), (m6502_mlp_example*)ctx->st_mex.p,
                (uint32_t*)ctx->st_row.p, sc);
            CKL("k_stoke_examples");
            unsigned long long rows = 0;
            CK(cudaMemcpyAsync(&rows, &sc->ex_rows, sizeof rows, cudaMemcpyDeviceToHost, ctx->stream));
            CK(cudaStreamSynchronize(ctx->stream));
            if (rows) {
                int mrc = m6502_mlp_forward_device(cfg->model, (const m6502_mlp_example*)ctx->st_mex.p, rows,
                                                   (float*)ctx->st_probs.p, ctx->stream);
                if (mrc != M6502_OK) return set_err(ctx, mrc, "learned proposal forward pass failed");
                k_cdf<<<(uint32_t)((rows + 255) / 256), 256, 0, ctx->stream>>>((float*)ctx->st_probs.p,
                                                                             (uint32_t)rows);
                CKL("k_cdf");
                prm.cdf = (const float*)ctx->st_probs.p;
                prm.row = (const uint32_t*)ctx->st_row.p;
            }
        }
        k_stoke_live<<<std::min<uint32_t>((n_chains + 255) / 256, (uint32_t)ctx->sms * 8), 256, 0, ctx->stream>>>(
            (StokeChain*)ctx->st_chains.p, n_chains, cpt, (const uint32_t*)ctx->st_proven.p, cfg->stop_on_proof,
            (uint32_t*)ctx->st_live.p, sc);
        CKL("k_stoke_live");
        const uint32_t eblocks = std::max<uint32_t>(std::min<uint32_t>(kEpochWarps, n_chains) / 2 + 1,
                                                    (n_chains + kEpochChains - 1) / kEpochChains);
        k_stoke_epoch<<<eblocks, 64, 0, ctx->stream>>>((StokeChain*)ctx->st_chains.p, (const uint32_t*)ctx->st_live.p, tg, prm, (StokeEntry*)ctx->st_entries.p, ecap, sc);
        CKL("k_stoke_epoch");
        CK(cudaEventRecord(ctx->sev[1], ctx->stream));
        k_stoke_vectors<<<ctx->sms * 8, 256, 0, ctx->stream>>>((StokeEntry*)ctx->st_entries.p, ecap, tg,
                                                               cfg->dead_flags, (uint32_t*)ctx->st_vidx.p,
                                                               (uint64_t*)ctx->st_keys.p, sc);
        CKL("k_stoke_vectors");
        // Identical (target, candidate) pairs are verified once: sort by key,
        // pick one representative per pair, number the distinct candidates of
        // each target.
        StokeCounters hv;
        CK(cudaMemcpyAsync(&hv, sc, sizeof hv, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        const uint32_t n_ok = (uint32_t)hv.vec_ok;
        uint32_t max_ord = 0;
        if (n_ok) {
            size_t sort_bytes = ctx->st_sort_tmp.bytes;
            CK(cub::DeviceRadixSort::SortPairs(ctx->st_sort_tmp.p, sort_bytes, (const uint64_t*)ctx->st_keys.p,
                                               (uint64_t*)ctx->st_keys2.p, (const uint32_t*)ctx->st_vidx.p,
                                               (uint32_t*)ctx->st_vals2.p, (int)n_ok, 0, 64, ctx->stream));
            k_stoke_dedupe<<<1, 1024, 0, ctx->stream>>>((const uint64_t*)ctx->st_keys2.p,
                                                        (const uint32_t*)ctx->st_vals2.p,
                                                        (const StokeEntry*)ctx->st_entries.p, (uint32_t*)ctx->st_rep.p,
                                                        (uint32_t*)ctx->st_ord.p, sc);
            CKL("k_stoke_dedupe");
            CK(cudaMemcpyAsync(&hv, sc, sizeof hv, cudaMemcpyDeviceToHost, ctx->stream));
            CK(cudaStreamSynchronize(ctx->stream));
            max_ord = (uint32_t)hv.max_ord;
        }
        // Phase 0: rounds of at most kVerifyBatch distinct candidates per
        // target under stop_on_proof (a target proved in one round is skipped
        // in the next; a single round of all of them otherwise), sweeping only
        // pairs whose cones stay within 2^kStokeDeferBits states.  Phase 1:
        // the deferred pairs of targets still unproved.  Proofs of phase 0 are
        // timed at its end, so one expensive pair does not delay the rest.
        StokeSource src{(const StokeEntry*)ctx->st_entries.p, (const uint32_t*)ctx->st_vlist.p, tg, cfg->dead_flags};
        // The rounds of an epoch are queued with no read-back in between, each
        // with its own counters; the host looks at their work items once, and
        // only if a round's did not fit is the epoch's verification run again
        // with a larger queue, from the targets proved before it.
        const uint32_t n_rounds = !n_ok ? 0u : cfg->stop_on_proof ? max_ord / kVerifyBatch + 1u : 1u;
        auto verify_round = [&](uint32_t lo, uint32_t hi, uint32_t phase, VerifyCounters* v) -> int {
            CK(cudaMemsetAsync(&sc->round_n, 0, sizeof(unsigned long long), ctx->stream));
            k_stoke_select<<<ctx->sms * 4, 256, 0, ctx->stream>>>(
                (const uint64_t*)ctx->st_keys2.p, (const uint32_t*)ctx->st_vals2.p, (const uint32_t*)ctx->st_rep.p,
                (const uint32_t*)ctx->st_ord.p, lo, hi, cfg->stop_on_proof, (const uint32_t*)ctx->st_proven.p,
                (const uint32_t*)ctx->st_verdict.p, phase, (uint32_t*)ctx->st_vlist.p, (uint32_t*)ctx->st_vpos.p,
                sc);
            CKL("k_stoke_select");
            ExhArgs ea{(uint32_t*)ctx->fail.p, (Item*)ctx->items.p, icap, cnt, v, cfg->sweep, 0,
                       phase == 0 ? kStokeDeferBits : 0u};
            TRY(launch_verify(ctx, src, &sc->round_n, ecap, ea));
            k_stoke_verdicts<<<ctx->sms * 4, 256, 0, ctx->stream>>>(
                (const uint32_t*)ctx->fail.p, (const uint32_t*)ctx->st_vpos.p, (const uint64_t*)ctx->st_keys2.p,
                (uint32_t*)ctx->st_verdict.p, (uint8_t*)ctx->st_vphase.p, phase, (uint32_t*)ctx->st_proven.p, sc);
            CKL("k_stoke_verdicts");
            return M6502_OK;
        };
        for (int attempt = 0;; attempt++) {
            if (n_rounds) {
                TRY(ensure(ctx, ctx->items, icap * sizeof(Item)));
                TRY(ensure(ctx, ctx->st_rounds, ((size_t)n_rounds + 1) * sizeof(VerifyCounters)));
                CK(cudaMemsetAsync(cnt, 0, sizeof(Counters), ctx->stream));
                CK(cudaMemsetAsync(ctx->st_rounds.p, 0, ((size_t)n_rounds + 1) * sizeof(VerifyCounters), ctx->stream));
                CK(cudaMemsetAsync(ctx->st_verdict.p, 0xFF, (size_t)n_ok * 4, ctx->stream));
                CK(cudaMemcpyAsync(ctx->st_proven_was.p, ctx->st_proven.p, (size_t)n_targets * 4, cudaMemcpyDeviceToDevice,
                                   ctx->stream));
            }
            VerifyCounters* v = (VerifyCounters*)ctx->st_rounds.p;
            for (uint32_t r = 0; r < n_rounds; r++)
                TRY(verify_round(r * (cfg->stop_on_proof ? kVerifyBatch : 0u),
                                 cfg->stop_on_proof ? (r + 1) * kVerifyBatch : 0xFFFFFFFFu, 0, v + r));
            CK(cudaEventRecord(ctx->sev[3], ctx->stream));   // phase-0 proofs are complete here
            if (!n_rounds) break;
            TRY(verify_round(0, 0, 1, v + n_rounds));
            std::vector<VerifyCounters> hr((size_t)n_rounds + 1);
            CK(cudaMemcpyAsync(hr.data(), ctx->st_rounds.p, hr.size() * sizeof(VerifyCounters), cudaMemcpyDeviceToHost,
                               ctx->stream));
            CK(cudaStreamSynchronize(ctx->stream));
            uint64_t items = 0;
            for (const VerifyCounters& c : hr) items = std::max<uint64_t>(items, c.items);
            if (items <= icap) break;
            if (attempt >= 4) return set_err(ctx, M6502_E_NOMEM, "work-item queue kept overflowing");
            icap = items + items / 4 + 1024;
            CK(cudaMemcpyAsync(ctx->st_proven.p, ctx->st_proven_was.p, (size_t)n_targets * 4, cudaMemcpyDeviceToDevice,
                               ctx->stream));
            CK(cudaMemsetAsync(&sc->undecided, 0, sizeof(unsigned long long), ctx->stream));
            CK(cudaMemsetAsync(&sc->verified, 0, sizeof(unsigned long long), ctx->stream));
        }
        if (n_ok) {
            k_stoke_collect<<<ctx->sms * 4, 256, 0, ctx->stream>>>(
                (const uint32_t*)ctx->st_vals2.p, (const uint32_t*)ctx->st_rep.p, (const uint32_t*)ctx->st_verdict.p,
                (const uint8_t*)ctx->st_vphase.p, (const StokeEntry*)ctx->st_entries.p, sc,
                (StokeChain*)ctx->st_chains.p, (uint32_t*)ctx->st_pidx.p, (uint8_t*)ctx->st_pphase.p, ecap);
            CKL("k_stoke_collect");
        }
        CK(cudaEventRecord(ctx->sev[2], ctx->stream));
        StokeCounters hc;
        CK(cudaMemcpyAsync(&hc, sc, sizeof hc, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        float e_ms = 0, a = 0, b = 0;
        cudaEventElapsedTime(&e_ms, ctx->ev0, ctx->sev[2]);
        cudaEventElapsedTime(&a, ctx->sev[0], ctx->sev[1]);
        cudaEventElapsedTime(&b, ctx->sev[1], ctx->sev[2]);
        ms_chains += a;
        ms_verify += b;
        done += e_steps;
        st.epochs++;
        st.steps += (uint64_t)e_steps * n_chains;   // chains that stopped still count their slot
        st.accepted += hc.accepted;
        st.candidates += std::min<uint64_t>(hc.entries, ecap);
        st.undecided += hc.undecided;
        st.verified += hc.verified;
        if (hc.entries > ecap) return set_err(ctx, M6502_E_NOMEM, "STOKE entry buffer overflowed");
        if (prm.traj && hc.traj) {   // improving moves of this epoch -> the caller's buffer
            const uint64_t have = std::min<uint64_t>(hc.traj, prm.traj_cap);
            const uint64_t room = traj_total < cfg->traj_cap ? cfg->traj_cap - traj_total : 0;
            const uint64_t take = std::min(have, room);
            if (take)
                CK(cudaMemcpyAsync(cfg->trajectories + traj_total, prm.traj, take * sizeof(m6502_mlp_example),
                                   cudaMemcpyDeviceToHost, ctx->stream));
            traj_total += hc.traj;
        }
        if (hc.proofs) {
            std::vector<uint32_t> pidx(hc.proofs);
            std::vector<uint8_t> pph(hc.proofs);
            h_entries.resize(std::min<uint64_t>(hc.entries, ecap));
            CK(cudaMemcpyAsync(pidx.data(), ctx->st_pidx.p, pidx.size() * 4, cudaMemcpyDeviceToHost, ctx->stream));
            CK(cudaMemcpyAsync(pph.data(), ctx->st_pphase.p, pph.size(), cudaMemcpyDeviceToHost, ctx->stream));
            CK(cudaMemcpyAsync(h_entries.data(), ctx->st_entries.p, h_entries.size() * sizeof(StokeEntry),
                               cudaMemcpyDeviceToHost, ctx->stream));
            CK(cudaStreamSynchronize(ctx->stream));
            float a_ms = 0;   // end of verification phase 0
            cudaEventElapsedTime(&a_ms, ctx->ev0, ctx->sev[3]);
            std::vector<uint32_t> order(pidx.size());
            for (size_t k = 0; k < order.size(); k++) order[k] = (uint32_t)k;
            // deterministic order within the epoch: target, step, chain
            std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
                const StokeEntry &x = h_entries[pidx[a]], &y = h_entries[pidx[b]];
                if (x.target != y.target) return x.target < y.target;
                if (x.step != y.step) return x.step < y.step;
                return x.chain < y.chain;
            });
            for (uint32_t k : order) {
                const StokeEntry& en = h_entries[pidx[k]];
                const double pms = pph[k] ? e_ms : a_ms;
                m6502_stoke_proof pr;
                std::memset(&pr, 0, sizeof pr);
                pr.target = en.target; pr.chain = en.chain; pr.step = en.step; pr.ms = pms;
                pr.cand_len = en.len; pr.dead_flags = en.dead_flags;
                std::memcpy(pr.cand, en.ins, sizeof pr.cand);
                found.push_back(pr);
                const uint32_t t = en.target;
                if (first_ms[t] < 0) {
                    first_ms[t] = pms;
                    first_step[t] = en.step;
                    first_epoch[t] = st.epochs;
                    proven_targets++;
                } else if (first_epoch[t] == st.epochs &&
                           (pms < first_ms[t] || (pms == first_ms[t] && en.step < first_step[t]))) {
                    first_ms[t] = pms;
                    first_step[t] = en.step;
                }
            }
            st.proofs += hc.proofs;
        }
        if (cfg->stop_on_proof && proven_targets == n_targets) break;
    }
    CK(cudaEventRecord(ctx->ev1, ctx->stream));
    CK(cudaEventSynchronize(ctx->ev1));
    float total = 0;
    cudaEventElapsedTime(&total, ctx->ev0, ctx->ev1);
    st.ms_device = total;
    st.ms_chains = ms_chains;
    st.ms_verify = ms_verify;
    st.targets_proven = proven_targets;
    // per-target summary: first proof, and the best proof (most Go bytes, then cycles saved)
    for (uint32_t t = 0; t < n_targets; t++) {
        m6502_stoke_result& r = results[t];
        std::memset(&r, 0, sizeof r);
        r.first_proof_ms = first_ms[t];
        r.first_proof_step = first_step[t];
    }
    for (const m6502_stoke_proof& pr : found) {
        m6502_stoke_result& r = results[pr.target];
        const uint16_t* ts = t_insns + t_offs[pr.target];
        int tn = (int)(t_offs[pr.target + 1] - t_offs[pr.target]);
        int bs = 0, cs = 0;
        for (int i = 0; i < tn; i++) { bs += (int)bytes_go(ts[i] & 0xFFu); cs += (int)cycles(ts[i] & 0xFFu); }
        for (int i = 0; i < pr.cand_len; i++) { bs -= (int)bytes_go(pr.cand[i] & 0xFFu); cs -= (int)cycles(pr.cand[i] & 0xFFu); }
        if (r.proofs == 0 || bs > r.bytes_saved || (bs == r.bytes_saved && cs > r.cycles_saved)) {
            r.best_len = pr.cand_len;
            std::memcpy(r.best, pr.cand, sizeof r.best);
            r.bytes_saved = (int16_t)bs;
            r.cycles_saved = (int16_t)cs;
            r.dead_flags = pr.dead_flags;
        }
        r.proofs++;
    }
    CK(cudaStreamSynchronize(ctx->stream));
    if (cfg->traj_count) *cfg->traj_count = traj_total;
    if (stats) *stats = st;
    if (n_proofs) *n_proofs = found.size();
    if (proofs && cap) std::memcpy(proofs, found.data(), std::min<uint64_t>(cap, found.size()) * sizeof(m6502_stoke_proof));
    if (found.size() > cap) return set_err(ctx, M6502_E_OVERFLOW, "proof buffer too small");
    return M6502_OK;
}

}  // extern "C"
