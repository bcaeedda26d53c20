// Preloaded in front of libcigpu.so: device allocations of chosen sizes fail on the host,
// as the allocator reports a device without memory (std::bad_alloc), without asking it.
#include <dlfcn.h>

#include <cstddef>
#include <new>

static size_t fail_bytes = 0;
static int fail_times = 0;  // -1: every time

extern "C" void alloc_fail_set(size_t bytes, int times) {
    fail_bytes = bytes;
    fail_times = times;
}

namespace cigpu {
void *dev_alloc(size_t bytes) {
    static const auto real = reinterpret_cast<void *(*)(size_t)>(dlsym(RTLD_NEXT, "_ZN5cigpu9dev_allocEm"));
    if (bytes == fail_bytes && fail_times != 0) {
        if (fail_times > 0) --fail_times;
        throw std::bad_alloc();
    }
    return real(bytes);
}
}  // namespace cigpu
