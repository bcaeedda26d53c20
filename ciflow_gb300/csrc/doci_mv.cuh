// Matrix-free DOCI matvec (doci_mv.cu).
#pragma once

#include "build.cuh"
#include "checked.cuh"

namespace cigpu {

struct DociMv {
    int L, n;                  // orbitals, electron pairs (n <= 32)
    int64_t D;                 // pair strings (rows)
    const uint64_t *strings;   // [D], colex order
    unsigned long long *err = nullptr;  // checked build: the error word
};

// The pair space split by orbitals: `s` low and L - s high ones. The strings with one
// set of high pairs are a block of consecutive ranks, C(s, m) of them for m low pairs,
// in the order of their low strings. The plan depends on (L, n) only.
constexpr int kSplitMaxLow = 12;
struct DociSector {  // the blocks with nh high and m low pairs
    int nh, m;
    int group[2];                     // blocks of one thread block (FP32, FP64 product)
    uint32_t first_task[2];           // thread blocks before this sector
    uint32_t nhigh, high0;            // high strings, and the first one's place in hbits / hbase
    uint32_t nlow, nminus, nplus;     // C(s, m), C(s, m - 1), C(s, m + 1)
    uint32_t ll0, minus0, plus0;      // offsets into the low tables
    uint32_t low0;                    // the sector's first low string in lowbits
    uint32_t n1, one0, n2, two0;      // C(s - 1, m - 1), C(s - 2, m - 1) and offsets into one / two
};
struct DociSplitView {
    int L, n, s, nsec;
    uint32_t tasks[2];
    const uint64_t *hbits;            // high strings (bit 0 = orbital s), sector by sector, colex
    const uint32_t *hbase;            // rank of each block's first string
    const uint32_t *binom;            // [64][kSplitBinomRow]: C(p, k) mod 2^32
    // per low string l of m pairs, entry-major ([entry][C(s, m)]):
    const uint32_t *ll;               // pair hops inside: target rank | (j * s + k) << 10
    const uint16_t *lminus, *lplus;   // a pair taken out of / put into orbital j: rank | j << 10
    // per orbital j (pair j < k), list-major: the low strings l that hold j (j, not k) and
    // their targets without j (with k in its place): l | target << 16
    const uint32_t *one, *two;
    const uint16_t *lowbits;          // the low strings, sector by sector
    unsigned long long *err;
    int64_t D;
    DociSector sec[kSplitMaxLow + 1];
};
constexpr int kSplitBinomRow = 34;
struct DociSplit {
    DociSplitView view{};
    size_t smem[2] = {0, 0};          // the product's shared memory, FP32 and FP64
    DevBuf<uint64_t> tables;          // all of the view's, in one block
    uint32_t nlowbits = 0;
    explicit operator bool() const { return view.s > 0; }
};
// Makes the plan where the split product is the faster one (plan.view.s stays 0 elsewhere);
// its tables are complete when the work queued on s is.
void doci_split_make(int L, int n, int64_t D, DociSplit &plan, cudaStream_t s);

// K_jk = (jk|jk) for j != k, zero where |v| <= 1e-14 (and on the diagonal): the
// pair-hop values, FP64 and (K32 may be null) FP32 (L*L each, device).
void doci_pair_table_launch(int L, const double *eri, double *K64, float *K32, cudaStream_t s);
// Entries of v with |v| > 1e-14 (synchronises s).
int64_t count_nonzero(const double *v, int64_t n, cudaStream_t s);
// y = H x: FP64 (K64, FP64 diag/x/y) and FP32 (K32, FP32 diag/x/y, FP32 accumulation).
void doci_mv64(const DociMv &p, const DociSplit &split, const double *K, const double *diag, const double *x,
               double *y, cudaStream_t s);
void doci_mv32(const DociMv &p, const DociSplit &split, const float *K, const float *diag, const float *x, float *y,
               cudaStream_t s);

}  // namespace cigpu
