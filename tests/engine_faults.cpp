// The engine's host side when a CUDA call fails, against the runtime of
// fake_cuda.h.  For every call of a search, an enumeration and a pair check:
// that call fails once; the entry point then returns with nothing queued that
// could touch the caller's memory or its own, and the same call repeated
// finds its tables whole.  Also, without a failure: kernels run after the
// copies of the tables they read, and host targets are read after the work
// that was on the engine's stream before the search.  Built and run by
// tests/test_engine_faults.py.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <vector>

#include "fake_cuda.h"
#include "m6502.h"

// The network lives in another object; no search here uses a model.
int m6502_mlp_forward_device(m6502_mlp*, const m6502_mlp_example*, unsigned long, float*, cudaStream_t) { return M6502_E_INVAL; }

static long bad = 0;
static void expect(bool ok, const char* what, const char* where, long k) {
    if (!ok && bad++ < 20) std::printf("%s: %s (failing call %ld)\n", where, what, k);
}

constexpr size_t kTableBytes = 59000, kGroupBytes = 17000;   // of a JoinTable, of CandGroups
static std::vector<char> want_table, want_groups;
static bool learn, wrong;
static std::set<const void*> hashed;      // line tables that k_line_hash has filled
static uint16_t want_target;              // what every pass's first target starts with; 0: not checked

static void hook(const std::string& name, void** a) {
    auto table = [](const void* p, size_t n, std::vector<char>& want) {
        if (learn) want.assign((const char*)p, (const char*)p + n);
        else if (std::memcmp(p, want.data(), n)) wrong = true;
    };
    if (name.find("11k_line_hash") != std::string::npos) hashed.insert(*(const void**)a[1]);
    if (name.find("9k_qc_joinI") != std::string::npos) {
        table(*(const void**)a[5], kTableBytes, want_table);
        if (want_target && **(const uint16_t**)a[0] != want_target) wrong = true;
    }
    if (name.find("8k_expandI") != std::string::npos) {
        if (const void* mult = *(const void**)a[7]) table(mult, kGroupBytes, want_groups);
        if (!hashed.count(*(const void**)a[8])) wrong = true;
    }
}

struct Scenario {
    const char* name;
    int kind;   // 0 search, 1 enumerate, 2 pair check
    uint32_t semantics, cand, flags;
    uint64_t per_pass, n;
};

struct Buffers {
    std::vector<uint16_t> t;
    std::vector<uint32_t> offs;
    std::vector<m6502_rule> rules;
    std::vector<uint8_t> out, fd;
    explicit Buffers(uint64_t n) : t(2 * n, 0x051A), offs(n + 1), rules(64), out(n), fd(n) {   // LDA #5
        for (uint64_t i = 0; i <= n; i++) offs[i] = (uint32_t)(2 * i);
        fake::page_lock(t.data(), t.size() * 2);
        fake::page_lock(offs.data(), offs.size() * 4);
        fake::page_lock(rules.data(), rules.size() * sizeof(m6502_rule));
        fake::page_lock(out.data(), out.size());
        fake::page_lock(fd.data(), fd.size());
    }
    ~Buffers() { fake::page_unlock_all(); }
    bool busy() const {
        return fake::pending(t.data(), t.size() * 2) || fake::pending(offs.data(), offs.size() * 4) ||
               fake::pending(rules.data(), rules.size() * sizeof(m6502_rule)) || fake::pending(out.data(), out.size()) ||
               fake::pending(fd.data(), fd.size());
    }
};

static int call(m6502_ctx* ctx, const Scenario& s, Buffers& b) {
    uint64_t n = 0;
    if (s.kind == 2)
        return m6502_check_pairs(ctx, s.n, b.t.data(), b.offs.data(), b.t.data(), b.offs.data(), 0, M6502_CHECK_ALL,
                                 M6502_SWEEP_REFERENCE, M6502_EXH_CONES, b.out.data(), b.fd.data());
    m6502_search_cfg cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cfg.semantics = s.semantics;
    cfg.max_cand_len = s.cand;
    cfg.flags = s.flags;
    cfg.dead_flags = 0x41;
    if (s.kind == 1) return m6502_enumerate(ctx, &cfg, 2, 3, 5, b.rules.data(), b.rules.size(), &n, nullptr);
    return m6502_search(ctx, &cfg, b.t.data(), s.n, 2, b.rules.data(), b.rules.size(), &n, nullptr);
}

static m6502_ctx* create(const Scenario& s) {
    m6502_ctx* ctx = nullptr;
    m6502_opts o;
    std::memset(&o, 0, sizeof o);
    o.targets_per_pass = s.per_pass;
    hashed.clear();
    if (m6502_create(&ctx, &o) != M6502_OK) { std::printf("no context\n"); std::exit(2); }
    return ctx;
}

// The caller's own work on the engine's stream writes the targets: they are
// read after it.
static void read_in_order(const Scenario& s, Buffers& b) {
    m6502_ctx* ctx = create(s);
    fake::main_stream = (cudaStream_t)m6502_stream(ctx);
    std::vector<uint16_t>* t = &b.t;
    fake::enqueue(fake::main_stream, [t] { for (uint16_t& w : *t) w = 0x061A; });
    want_target = 0x061A;
    wrong = false;
    expect(call(ctx, s, b) == M6502_OK, "fails", s.name, 0);
    expect(!wrong, "targets were read before the stream's earlier work", s.name, 0);
    want_target = 0;
    fake::main_stream = nullptr;
    m6502_destroy(ctx);
}

// New masks share blocks of memory: an allocation for each of a mask's tables
// takes longer than building them.
static int masks() {
    Scenario s{"new masks", 0, M6502_SEM_CUDA, 1, 0, 0, 20};
    Buffers b(s.n);
    m6502_ctx* ctx = create(s);
    expect(call(ctx, s, b) == M6502_OK, "fails", s.name, 0);
    const long before = fake::mallocs;
    for (uint32_t mask = 0; mask < 64; mask++) {
        m6502_search_cfg cfg;
        std::memset(&cfg, 0, sizeof cfg);
        cfg.semantics = mask & 1 ? M6502_SEM_GO : M6502_SEM_CUDA;
        cfg.max_cand_len = 1;
        cfg.dead_flags = (uint8_t)mask;
        uint64_t n = 0;
        expect(m6502_search(ctx, &cfg, b.t.data(), s.n, 2, b.rules.data(), b.rules.size(), &n, nullptr) == M6502_OK, "fails", s.name, mask);
    }
    expect(fake::mallocs - before <= 16, "more than a block of memory for every four masks", s.name, 0);
    m6502_destroy(ctx);
    std::printf("%ld allocations, %ld failures\n", fake::mallocs - before, bad);
    return bad ? 1 : 0;
}

int main(int argc, char** argv) {
    const std::string mode = argc > 1 ? argv[1] : "";   // tables, errors, order or masks
    if (mode == "masks") return masks();
    const bool errors = mode == "errors";
    const Scenario all[] = {
        {"search", 0, M6502_SEM_CUDA, 1, 0, 0, 20},
        {"search in three passes", 0, M6502_SEM_CUDA, 1, 0, 8, 20},
        {"search without graphs", 0, M6502_SEM_CUDA, 1, M6502_NO_GRAPH, 8, 20},
        {"Go search", 0, M6502_SEM_GO, 1, 0, 0, 20},
        {"Go search in three passes", 0, M6502_SEM_GO, 1, 0, 8, 20},
        {"Go search, length 2", 0, M6502_SEM_GO, 2, 0, 0, 20},
        {"enumeration", 1, M6502_SEM_CUDA, 1, 0, 0, 20},
        {"pair check", 2, 0, 0, 0, 0, 20},
        {"large pair check", 2, 0, 0, 0, 0, 4u << 20},
    };
    fake::on_kernel = hook;
    for (const Scenario& s : all) {
        if (s.kind == 2 && !errors) continue;
        if (mode == "order" && (s.kind || s.semantics != M6502_SEM_CUDA)) continue;
        Buffers b(s.n);
        // What the tables hold, from a call that everything before it has ended for.
        learn = true;
        m6502_ctx* ctx = create(s);
        expect(call(ctx, s, b) == M6502_OK, "fails", s.name, 0);
        fake::drain();
        expect(call(ctx, s, b) == M6502_OK, "fails when repeated", s.name, 0);
        m6502_destroy(ctx);
        learn = wrong = false;
        if (mode == "order") {
            read_in_order(s, b);
            continue;
        }
        // A first call without a failure.
        ctx = create(s);
        fake::calls = 0;
        expect(call(ctx, s, b) == M6502_OK, "fails", s.name, 0);
        const long n = fake::calls;
        if (!errors) expect(!wrong, "a kernel ran before its tables were there", s.name, 0);
        m6502_destroy(ctx);
        for (long k = 1; k <= n; k++) {
            ctx = create(s);
            fake::calls = 0;
            fake::fail_at = k;
            const int rc = call(ctx, s, b);
            fake::fail_at = 0;
            if (errors) {
                expect(!b.busy(), "work on the caller's memory is still queued after the call", s.name, k);
                expect(!fake::queued(), "work is still queued after the call", s.name, k);
                expect(call(ctx, s, b) == M6502_OK, rc ? "fails when repeated after an error" : "fails when repeated", s.name, k);
            } else {
                wrong = false;
                call(ctx, s, b);
                expect(call(ctx, s, b) == M6502_OK, "fails when repeated twice", s.name, k);
                expect(!wrong, "a repeated call met a table that was never filled", s.name, k);
            }
            m6502_destroy(ctx);
            cudaGetLastError();
        }
    }
    std::printf("%ld failures\n", bad);
    return bad ? 1 : 0;
}
