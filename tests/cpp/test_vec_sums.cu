// The FP32 sums of the mixed solver's basis kernels on terms whose plain FP32 sum loses
// the small ones: 1 and 2^-24 at random places. Prints "name error" per sum, the error
// relative to the sum (the exact values are multiples of 2^-24 below 2^29).
#include "../../ciflow_gb300/csrc/lanczos.cu"

#include <cstdint>
#include <cstdio>
#include <vector>

using namespace cigpu;

static uint32_t rng = 12345;
static bool coin() {
    rng = rng * 1664525u + 1013904223u;
    return (rng >> 28) < 5;
}

static void report(const char *name, double got, double want) { std::printf("%s %.3e\n", name, std::fabs(got - want) / want); }

// Terms of `n` elements, one in `every` not zero: sqrt(term) for squares.
static double fill(std::vector<float> &v, int64_t n, int every, bool root) {
    v.assign((size_t)n, 0.f);
    double sum = 0;
    for (int64_t i = 0; i < n; i += every) {
        const bool one = coin();
        v[(size_t)i] = one ? 1.f : root ? 0x1p-12f : 0x1p-24f;
        sum += one ? 1.0 : 0x1p-24;
    }
    return sum;
}

static void dots(int64_t n, int nvec) {
    cudaStream_t s = nullptr;
    VecOps ops(s, n);
    std::vector<float> v, ones((size_t)n, 1.f);
    std::vector<double> want;
    DevBuf<float> V((size_t)(nvec + 2) * n), w((size_t)n);
    for (int i = 0; i < nvec + 2; ++i) {
        want.push_back(fill(v, n, 4, false));  // one element of each 16-byte load
        CIGPU_CUDA(cudaMemcpy(V.p + (size_t)i * n, v.data(), sizeof(float) * n, cudaMemcpyHostToDevice));
    }
    CIGPU_CUDA(cudaMemcpy(w.p, ones.data(), sizeof(float) * n, cudaMemcpyHostToDevice));
    ops.dots<float, float, float>(V.p, n, nvec, w.p, n, 0, -1, V.p + (size_t)nvec * n, 2, w.p);
    const double *h = ops.fetch(nvec + 2);
    double worst = 0, of = 1;
    for (int i = 0; i < nvec + 2; ++i)
        if (std::fabs(h[i] - want[i]) / want[i] >= worst) worst = std::fabs(h[i] - want[i]) / want[i], of = want[i];
    report("dots", of * (1.0 + worst), of);
}

static void couple(int64_t n) {
    std::vector<float> v, ones((size_t)n, 1.f);
    DevBuf<float> V((size_t)2 * n), x((size_t)n);
    DevBuf<double> h(8);
    const double want = fill(v, n, 1, false);
    CIGPU_CUDA(cudaMemcpy(V.p + n, v.data(), sizeof(float) * n, cudaMemcpyHostToDevice));
    CIGPU_CUDA(cudaMemcpy(x.p, ones.data(), sizeof(float) * n, cudaMemcpyHostToDevice));
    if (!cluster_ok(k_dav_couple, kDavThreads, 0)) return report("couple", 1, 1);
    ClusterLaunch(kDavThreads, 0, nullptr)(k_dav_couple, n, V.p, 0, x.p, x.p, x.p, h.p);
    double got[3];
    CIGPU_CUDA(cudaMemcpy(got, h.p, sizeof(got), cudaMemcpyDeviceToHost));
    for (double g : got) report("couple", g, want);
}

// The first direction from a residual r, orthogonal to slot 0 (zero here): ||r||^2 and the
// direction's norm.
static void step(int64_t n) {
    std::vector<float> r, ones((size_t)n, 1.f);
    DevBuf<float> V((size_t)2 * n), r32((size_t)n), c32((size_t)n), diag((size_t)n);
    DevBuf<double> out(2), dmin(1);
    const double want = fill(r, n, 1, true), one = 1.0;
    CIGPU_CUDA(cudaMemset(V.p, 0, V.bytes()));
    CIGPU_CUDA(cudaMemset(c32.p, 0, c32.bytes()));
    CIGPU_CUDA(cudaMemcpy(r32.p, r.data(), sizeof(float) * n, cudaMemcpyHostToDevice));
    CIGPU_CUDA(cudaMemcpy(diag.p, ones.data(), sizeof(float) * n, cudaMemcpyHostToDevice));
    CIGPU_CUDA(cudaMemcpy(dmin.p, &one, sizeof(one), cudaMemcpyHostToDevice));
    if (!cluster_ok(k_dav_step, kDavThreads, dav_smem(n, 30))) return report("step", 1, 1);
    ClusterLaunch(kDavThreads, dav_smem(n, 30), nullptr)(k_dav_step, n, V.p, V.p, 0, false, DavCoef{}, 1.0, 0.0, 0.0, dmin.p,
                                                         r32.p, c32.p, diag.p, out.p, out.p + 1);
    double got[2];
    CIGPU_CUDA(cudaMemcpy(got, out.p, sizeof(got), cudaMemcpyDeviceToHost));
    for (double g : got) report("step", g, want);
}

int main() {
    try {
        dots(853776, 15);
        dots(1000000, 3);
        couple(16384);
        step(16384);
    } catch (const CudaError &e) {
        std::printf("cuda %s: %s\n", e.what, cudaGetErrorString(e.err));
        return 1;
    }
    return 0;
}
