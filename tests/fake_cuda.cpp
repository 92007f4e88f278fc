// See fake_cuda.h.
#include "fake_cuda.h"

#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <vector>

struct CUevent_st { cudaStream_t stream; unsigned long long upto; };
struct Op {
    std::function<void()> run;
    const char* lo[2] = {nullptr, nullptr};   // host or device ranges it touches
    size_t bytes = 0;
};
struct CUstream_st {
    std::deque<Op> q;
    unsigned long long done = 0, issued = 0;   // operations run, enqueued
    std::vector<Op>* capture = nullptr;
};
struct CUgraph_st { std::vector<Op> ops; };
struct CUgraphExec_st { std::vector<Op> ops; };

namespace fake {
long calls = 0, fail_at = 0, mallocs = 0;
cudaError_t fail_code = cudaErrorUnknown;
cudaStream_t main_stream = nullptr;
std::function<void(const std::string&, void**)> on_kernel;

// What a host-to-device cudaMemcpy leaves behind: the copy to the device may
// still be under way when it returns, and no other stream waits for it.
CUstream_st legacy;
std::vector<cudaStream_t>& streams() { static std::vector<cudaStream_t> v{&legacy}; return v; }
std::map<const void*, std::string>& names() { static std::map<const void*, std::string> m; return m; }
cudaError_t last = cudaSuccess;

bool fails() { return ++calls == fail_at; }

void run_upto(cudaStream_t s, unsigned long long upto) {
    while (s->done < upto && !s->q.empty()) {
        Op op = std::move(s->q.front());
        s->q.pop_front();
        s->done++;
        if (op.run) op.run();
    }
}
void push(cudaStream_t s, Op op) {
    if (!s) s = &legacy;
    if (s->capture) { s->capture->push_back(std::move(op)); return; }
    const bool now = main_stream && s != main_stream && s != &legacy;
    s->q.push_back(std::move(op));
    s->issued++;
    if (now) run_upto(s, s->issued);
}
void enqueue(cudaStream_t s, std::function<void()> f) { Op o; o.run = std::move(f); push(s, std::move(o)); }
bool pending(const void* p, size_t bytes) {
    for (cudaStream_t s : streams())
        for (const Op& o : s->q)
            for (const char* lo : o.lo)
                if (lo && lo < (const char*)p + bytes && (const char*)p < lo + o.bytes) return true;
    return false;
}
size_t queued() {
    size_t n = 0;
    for (cudaStream_t s : streams()) n += s == &legacy ? 0 : s->q.size();
    return n;
}
void drain() { for (cudaStream_t s : streams()) run_upto(s, s->issued); }
std::vector<std::pair<const char*, size_t>> locked;
void page_lock(const void* p, size_t n) { locked.emplace_back((const char*)p, n); }
void page_unlock_all() { locked.clear(); }
std::map<const char*, size_t> host_blocks;   // cudaHostAlloc
bool page_locked(const void* p) {
    const char* c = (const char*)p;
    for (auto& r : locked) if (c >= r.first && c < r.first + r.second) return true;
    for (auto& r : host_blocks) if (c >= r.first && c < r.first + r.second) return true;
    return false;
}
Op copy_op(void* d, const void* s, size_t n) {
    Op o;
    o.run = [=] { if (n) std::memmove(d, s, n); };
    o.lo[0] = (const char*)d; o.lo[1] = (const char*)s; o.bytes = n;
    return o;
}
}  // namespace fake
using namespace fake;

#define FAILS() do { if (fails()) { last = fail_code; return fail_code; } } while (0)

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { FAILS(); return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10
       : a == cudaDevAttrComputeCapabilityMinor ? 0 : a == cudaDevAttrMaxGridDimX ? 0x7FFFFFFF : 49152;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof *p); std::strcpy(p->name, "fake"); return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof *a); a->ptxVersion = a->binaryVersion = 100; a->maxThreadsPerBlock = 1024; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 4; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "injected"; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }

cudaError_t cudaMalloc(void** p, size_t n) { FAILS(); mallocs++; *p = std::calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaFree(void* p) { drain(); std::free(p); return cudaSuccess; }   // waits for the device
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { FAILS(); *p = std::calloc(1, n); host_blocks[(const char*)*p] = n; return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { drain(); host_blocks.erase((const char*)p); std::free(p); return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = new CUstream_st(); streams().push_back(*s); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    run_upto(s, s->issued);
    auto& v = streams();
    for (size_t i = 0; i < v.size(); i++) if (v[i] == s) { v.erase(v.begin() + (long)i); break; }
    delete s;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    FAILS();
    if (!s || s == cudaStreamLegacy) s = &legacy;
    run_upto(s, s->issued);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { FAILS(); drain(); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = new CUevent_st{nullptr, 0}; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    FAILS();
    if (!s->capture) { e->stream = s; e->upto = s->issued; }
    return cudaSuccess;
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned) { return cudaEventRecord(e, s); }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { FAILS(); if (e->stream) run_upto(e->stream, e->upto); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    FAILS();
    cudaStream_t other = e->stream;
    const unsigned long long upto = e->upto;
    if (other) enqueue(s, [=] { run_upto(other, upto); });
    return cudaSuccess;
}

cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    FAILS();
    if (k == cudaMemcpyHostToDevice && !page_locked(s)) {
        auto held = std::make_shared<std::vector<char>>((const char*)s, (const char*)s + n);
        Op o = copy_op(d, d, n);
        o.run = [=] { std::memcpy(d, held->data(), held->size()); };
        push(st, std::move(o));
    } else if (k == cudaMemcpyDeviceToHost && !page_locked(d)) {
        run_upto(st, st->issued);
        std::memcpy(d, s, n);
    } else {
        push(st, copy_op(d, s, n));
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
    FAILS();
    if (k == cudaMemcpyHostToDevice) {   // the source has been read; the device side may come later
        auto held = std::make_shared<std::vector<char>>((const char*)s, (const char*)s + n);
        enqueue(&legacy, [=] { std::memcpy(d, held->data(), n); });
    } else {
        run_upto(&legacy, legacy.issued);
        std::memmove(d, s, n);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { FAILS(); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) { FAILS(); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char any[1 << 16]; *p = any; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s) {
    FAILS();
    Op o;
    o.run = [=] { std::memset(d, v, n); };
    o.lo[0] = (const char*)d; o.bytes = n;
    push(s, std::move(o));
    return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { FAILS(); s->capture = new std::vector<Op>(); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    *g = new CUgraph_st{std::move(*s->capture)};
    delete s->capture;
    s->capture = nullptr;
    FAILS();
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) { FAILS(); *e = new CUgraphExec_st{g->ops}; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete e; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { FAILS(); for (const Op& o : e->ops) push(s, o); return cudaSuccess; }

// ---- launches ----
static dim3 g_grid, g_block;
static size_t g_shared;
static cudaStream_t g_stream;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sh, void* s) { g_grid = g; g_block = b; g_shared = sh; g_stream = (cudaStream_t)s; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sh, void* s) { *g = g_grid; *b = g_block; *sh = g_shared; *(cudaStream_t*)s = g_stream; return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h = nullptr; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) { names()[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t s) {
    FAILS();
    const std::string name = names()[f];
    const bool look = name.find("9k_qc_joinI") != std::string::npos || name.find("8k_expandI") != std::string::npos ||
                      name.find("11k_line_hash") != std::string::npos;
    std::vector<unsigned long long> held;
    if (look) {   // parameters of at most 8 bytes each, as many as the hooks read
        const int n = name.find("11k_line_hash") != std::string::npos ? 2 : 9;
        const int four = name.find("11k_line_hash") != std::string::npos ? 0x1
                       : name.find("9k_qc_joinI") != std::string::npos ? 0xCE : 0x64;   // 32-bit parameters, by position
        for (int i = 0; i < n; i++) {
            unsigned long long v = 0;
            std::memcpy(&v, args[i], (four >> i) & 1 ? 4 : 8);
            held.push_back(v);
        }
    }
    enqueue(s, [=] {
        if (!look || !on_kernel) return;
        std::vector<unsigned long long> h = held;
        std::vector<void*> p;
        for (auto& x : h) p.push_back(&x);
        on_kernel(name, p.data());
    });
    return cudaSuccess;
}
}
