// SmemLimit (ciflow_gb300/csrc/smem_limit.cuh) against a fake CUDA runtime of several
// devices: prints one line per check that fails.
#include "../../ciflow_gb300/csrc/smem_limit.cuh"

#include <cstdio>
#include <map>

static int device = 0, calls = 0, failures = 0;
static bool fail_next = false;
static std::map<int, int> limit;  // of each device

extern "C" cudaError_t cudaGetDevice(int *d) {
    *d = device;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int value) {
    ++calls;
    if (fail_next) {
        fail_next = false;
        return cudaErrorInvalidValue;
    }
    limit[device] = value;
    return cudaSuccess;
}

static void kernel() {}

static void check(bool ok, const char *what) {
    if (!ok) std::printf("failed: %s\n", what), ++failures;
}

int main() {
    static cigpu::SmemLimit l;
    for (int round = 0; round < 2; ++round)
        for (device = 0; device < 70; device += 23) check(l.raise(kernel, 1000) == cudaSuccess && limit[device] == 1000, "device");
    check(calls == 3 + 2, "once per device, at every call past the 64th");
    device = 5;
    fail_next = true;
    check(l.raise(kernel, 1000) == cudaErrorInvalidValue, "a failure is reported");
    check(l.raise(kernel, 1000) == cudaSuccess && limit[5] == 1000, "and not remembered");
    return failures;
}
