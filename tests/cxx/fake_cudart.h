// Controls of the stand-in CUDA runtime (fake_cudart.cpp): device memory is host
// memory, launches are recorded and do nothing, and a call can be told to fail.
#pragma once

#include <cstddef>
#include <string>
#include <vector>

namespace fake {

// the n-th allocation / host-to-device copy / graph instantiation from now on fails
// (1: the next; 0: none); with `and_after` every later one too
void fail_malloc(int n, bool and_after = false);
void fail_upload(int n);
void fail_instantiate(int n, bool and_after = false);
// launches on non-blocking streams, eager or of graphs, while a copy from pageable
// memory or a memset on the null stream may not have arrived (no stream waits for it)
int early_launches();
int stream_waits();      // cudaStreamSynchronize calls so far
int graph_launches();    // graph launches so far
int mallocs();           // device allocations asked for so far
size_t live_bytes();     // device memory held
bool is_device(const void *p);
void *device_only(size_t bytes);  // a device pointer that the host cannot touch

struct Launch {
    std::string name;
    const void *stream;
    unsigned blocks;
    std::vector<const void *> ptr;  // the arguments named by watch(), as pointers
    bool early;                     // one of them was still in flight on
                                    // the null stream: a copy from pageable memory
                                    // returns before it has arrived, a memset before it
                                    // has run, and streams made non-blocking wait for
                                    // neither
};
// record argument `arg` (a pointer) of kernels whose name contains `kernel`
void watch(const char *kernel, int arg);
std::vector<Launch> take_launches();
// the largest dynamic shared memory that a kernel was ever allowed, and the last
struct SmemLimit {
    int last = 0, most = 0;
};
SmemLimit smem_limit(const char *kernel);

}  // namespace fake
