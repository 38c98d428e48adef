// Stand-in for the CUDA runtime with host memory as device memory: see alloc_main.cpp.
#pragma once

#include <cstddef>
#include <cstdint>
#include <string>

namespace fake {
extern int allocs;         // allocations so far
extern int fail_at;        // the allocation that fails (0: none)
extern int bad;            // complaints so far
extern std::string where;  // named by each complaint
void complain(const char* what);
size_t blocks();  // allocations not freed
// Whether p points to at least `bytes` of one live block; complains if not.
bool live(const void* p, int64_t bytes, const char* what);
// A caller's device array, live as long as this object.
struct Device {
    const void* p;
    Device(const void* p, size_t bytes);
    ~Device();
};
}  // namespace fake
