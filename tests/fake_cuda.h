// A CUDA runtime for tests on the host, linked with the engine's object file
// in place of the real one: device memory is host memory, kernels do nothing
// but what a hook does for them.  Work on a stream waits in a queue until
// something needs it done, so that a missing wait shows: a kernel that runs
// before the copy it reads, a copy still queued when the call returned.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <functional>
#include <string>

namespace fake {
// The call numbered `fail_at` (1, 2, ...; 0: none) of those that can fail
// returns `fail_code`; `calls` counts them.
extern long calls, fail_at;
extern cudaError_t fail_code;
extern long mallocs;                   // of device memory
// Copies to the device on any other stream than `main_stream` start at once,
// as far as their stream's earlier waits allow (null: every queue is lazy).
extern cudaStream_t main_stream;
// Called when a kernel runs; `args` are copies of its parameters.
extern std::function<void(const std::string& name, void** args)> on_kernel;
// A caller's buffer from page-locked memory: copies from and to it run on the
// device's time.  Those of pageable memory read it, or have written it, when
// the call that queues them returns.
void page_lock(const void* p, size_t bytes);
void page_unlock_all();
// Work still queued on any stream that touches [p, p + bytes).
bool pending(const void* p, size_t bytes);
size_t queued();                       // operations queued on all streams
void enqueue(cudaStream_t s, std::function<void()> f);   // as a caller's own work on a stream
void drain();                          // runs everything
}  // namespace fake
