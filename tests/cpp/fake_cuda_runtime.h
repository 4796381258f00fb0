// A CUDA runtime made of host code, for tests of the library's memory, copy and timing code without a GPU: two devices, streams
// whose work is done only when somebody waits for it, events, and the errors the real calls answer with.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <functional>
#include <string>
#include <vector>

namespace fake {

struct Copy {
    void* dst;
    const void* src;
    size_t bytes;
};

extern size_t device_limit;            // bytes a device has; cudaMalloc beyond them fails
extern size_t pinned_limit;
extern size_t device_in_use, pinned_in_use;
extern int events_alive;
extern int elapsed_reads;              // calls of cudaEventElapsedTime
extern int failing_records;            // this many cudaEventRecord calls fail
extern std::vector<std::string> log;   // what was done, in order

// Copies enqueued that nothing has waited for yet and that touch [p, p + bytes).
bool in_flight(const void* p, size_t bytes);
bool is_device_memory(const void* p);

} // namespace fake

#define CHECK(x)                                                                          \
    do {                                                                                  \
        if (!(x)) {                                                                       \
            std::fprintf(stderr, "%s:%d: %s does not hold\n", __FILE__, __LINE__, #x);    \
            std::exit(1);                                                                 \
        }                                                                                 \
    } while (0)
