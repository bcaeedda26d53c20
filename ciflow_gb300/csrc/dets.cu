// Determinant-list CI: FCI_File and CI_Big (cigpu_build_dets), and the
// Permutator_File reader (cigpu_dets_read).
//
// The reference builds a CI matrix over an arbitrary list of determinants read
// from a text file (FCI_File::construct_CI_matrix, CIMethod.cpp:890-914): every
// pair (i, j >= i) of the list goes through get_ham_element (CIMethod.cpp:459-487),
// which classifies the pair by the popcounts of up1^up2 and down1^down2 and
// evaluates the Slater-Condon rule (diagonal, one_diff_orbital, two_diff_orbitals;
// CIMethod.cpp:329-457). CI_Big (CIMethod.cpp:591-609, 928-1144) keeps part of the
// matrix and recomputes the rest in every matvec.
//
// Here the list lives on the device as records of 2W 64-bit words (up string, then
// down string; W = 1 for L <= 64, W = 2 for L <= 128). Every row is tested
// against every column (popcount of the XORs, <= 2 excitations; k_dets_scan), and the
// elements are evaluated with the reference's summation order, so the values are
// bit-identical to the reference's. The full symmetric matrix is built row by row with
// its columns ascending, so no transpose is needed and the upper triangle is the
// reference CRS. Storage:
//   CIGPU_DETS_CRS      the CRS (FP64, or FP32 hi/lo for the mixed method);
//   CIGPU_DETS_ONTHEFLY nothing but the list: every FP64 matvec rescans all pairs
//                       and applies the elements as it computes them (CI_Big with
//                       no stored part), y_i summed in a fixed order per row.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <memory>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "crs.cuh"
#include "spmv.cuh"

namespace cigpu {

namespace {

constexpr int kDetWarps = 8;   // rows per block (one warp each)
constexpr int kDetTile = 256;  // determinants per shared-memory tile
enum DetMode : int { kDetCount = 0, kDetFill64 = 1, kDetFill32 = 2 };

struct DetParams {
    int L, nup, ndown;
    uint32_t one = 1;  // see mark()
    int64_t n;
    // rows the pass visits (count / fill: the stored rows; matvec: all n) and the
    // stored block: count / fill take columns below `block` (n for a whole CRS); the
    // matvec takes the pairs outside the block (row i < block: columns >= block)
    int64_t nrows = 0, block = 0;
    int group = 32;        // rows of a warp in the count and fill passes (32, fewer in short lists)
    const uint64_t *dets;  // [n][2W]
    const double *eri;     // chemist (pq|rs), L^4
    const double *h;       // L^2
    const double *diag;    // [n]
    // count pass
    uint32_t *row_count, *upper_off;
    uint32_t *seg_count;  // [nrows][kSegs] kept elements per column segment (the fill reads them)
    uint32_t *masks = nullptr;    // [row groups][words][32] connected columns (k_dets_pairs)
    uint32_t *dropped = nullptr;  // set by a fill that met an element of 1e-14 or less
    // fill pass
    const int64_t *row_ptr;
    uint32_t *col;
    double *val64;
    float *val32, *val32lo;
};

__device__ __forceinline__ double Tm(const DetParams &p, int i, int j) { return p.h[i * p.L + j]; }
// physics <ij|kl> = chemist (ik|jl)
__device__ __forceinline__ double Vm(const DetParams &p, int i, int j, int k, int l) {
    const int64_t L = p.L;
    return p.eri[((i * L + k) * L + j) * L + l];
}

// Set bits of `up` in [min(o0,o1), max(o0,o1)) (get_nstacked, CIMethod.cpp:382-396).
template <int W>
__device__ __forceinline__ int nstacked(int o0, int o1, const uint64_t *up) {
    const int lo = min(o0, o1), hi = max(o0, o1);
    int n = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const int b0 = max(lo - 64 * w, 0), b1 = min(hi - 64 * w, 64);
        if (b1 <= b0) continue;
        uint64_t m = b1 == 64 ? ~(uint64_t)0 : (((uint64_t)1 << b1) - 1);
        m &= ~(((uint64_t)1 << b0) - 1);
        n += __popcll(up[w] & m);
    }
    return n;
}

// Orbitals of s in ascending order (get_orbs); at most `cap` of them.
template <int W>
__device__ __forceinline__ int orbitals(const uint64_t *s, int *o, int cap) {
    int n = 0;
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t x = s[w]; x && n < cap; x &= x - 1) o[n++] = 64 * w + __ffsll((long long)x) - 1;
    return n;
}

// -e when odd, on the sign bit (exact, and off GB300's slow FP64 pipe)
__device__ __forceinline__ double negate_if(double e, int odd) {
    return __longlong_as_double(__double_as_longlong(e) ^ ((long long)odd << 63));
}

// |v| > 1e-14 (SparseMatrix_CRS::PushToRow's drop threshold) as an integer compare of
// the magnitude bits; the values are finite (the integrals are validated)
__device__ __forceinline__ bool keep_value(double v) {
    return ((unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull) > 0x3D06849B86A12B9Bull;
}

// Lowest set orbital of x (cleared from x); x is a register array (constant indices).
template <int W>
__device__ __forceinline__ int pop_lowest(uint64_t *x) {
    int o = -1;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        if (o < 0 && x[w]) {
            o = 64 * w + __ffsll((long long)x[w]) - 1;
            x[w] &= x[w] - 1;
        }
    }
    return o;
}

template <int W>
__device__ __forceinline__ bool has_bit(const uint64_t *s, int o) {
    return (s[o >> 6] >> (o & 63)) & 1;
}

// get_diag_cont_one_bitstring (CIMethod.cpp:329-342): sum of T, then of the pair terms
template <int W>
__device__ double diag_one(const DetParams &p, const uint64_t *s) {
    int o[128];
    const int n = orbitals<W>(s, o, 128);
    double sum = 0;
    for (int k = 0; k < n; ++k) sum += Tm(p, o[k], o[k]);
    for (int k = 0; k + 1 < n; ++k)
        for (int l = k + 1; l < n; ++l) sum += Vm(p, o[k], o[l], o[k], o[l]) - Vm(p, o[k], o[l], o[l], o[k]);
    return sum;
}

// CIMethod::diagonal (CIMethod.cpp:398-407): (up part + down part) + the up-down part
template <int W>
__device__ double diagonal(const DetParams &p, const uint64_t *up, const uint64_t *dn) {
    double tot = diag_one<W>(p, up);
    tot += diag_one<W>(p, dn);
    double mix = 0;
#pragma unroll
    for (int wu = 0; wu < W; ++wu)
        for (uint64_t xu = up[wu]; xu; xu &= xu - 1) {
            const int a = 64 * wu + __ffsll((long long)xu) - 1;
#pragma unroll
            for (int wd = 0; wd < W; ++wd)
                for (uint64_t xd = dn[wd]; xd; xd &= xd - 1) {
                    const int b = 64 * wd + __ffsll((long long)xd) - 1;
                    mix += Vm(p, a, b, a, b);
                }
        }
    tot += mix;
    return tot;
}

// one_diff_orbital (CIMethod.cpp:409-427); `other` is the opposite-spin string
template <int W>
__device__ __forceinline__ double one_diff(const DetParams &p, const uint64_t *s1, const uint64_t *s2, const uint64_t *other) {
    uint64_t x[W], c[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
        x[w] = s1[w] ^ s2[w];
        c[w] = s1[w] & s2[w];
    }
    const int o0 = pop_lowest<W>(x), o1 = pop_lowest<W>(x);
    double e = Tm(p, o0, o1);
    // four terms' loads in flight, the terms added in order
    const int64_t L = p.L, at = (int64_t)o0 * L * L * L + (int64_t)o1 * L * L, ax = (int64_t)o0 * L * L * L + o1;
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t y = c[w]; y;) {
            double t[4], u[4];
            int n = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (y) {
                    const int z = 64 * w + __ffsll((long long)y) - 1;
                    y &= y - 1;
                    t[k] = __ldg(p.eri + at + z * L + z);       // <o0 z|o1 z>
                    u[k] = __ldg(p.eri + ax + (z * L + z) * L);  // <o0 z|z o1>
                    n = k + 1;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < n) e += t[k] - u[k];
        }
    const int diff = nstacked<W>(o0, o1, c);
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t y = other[w]; y;) {
            double t[4];
            int n = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (y) {
                    const int z = 64 * w + __ffsll((long long)y) - 1;
                    y &= y - 1;
                    t[k] = __ldg(p.eri + at + z * L + z);
                    n = k + 1;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < n) e += t[k];
        }
    return negate_if(e, diff & 1);
}

// arrange_order (CIMethod.cpp:353-380) for four ascending orbitals of which two are
// occupied in s1: (a0, a1) those of s1, (b0, b1) the others, each pair ascending.
// Written with register selects (no indexed local arrays).
template <int W>
__device__ __forceinline__ void arrange4(const int *o, const uint64_t *s1, int &a0, int &a1, int &b0, int &b1) {
    int na = 0, nb = 0;
    a0 = a1 = b0 = b1 = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (has_bit<W>(s1, o[k])) {
            if (na == 0) a0 = o[k]; else a1 = o[k];
            ++na;
        } else {
            if (nb == 0) b0 = o[k]; else b1 = o[k];
            ++nb;
        }
    }
}

// two_diff_orbitals(s1, s2) (CIMethod.cpp:429-442): same-spin double
template <int W>
__device__ __forceinline__ double two_diff_same(const DetParams &p, const uint64_t *s1, const uint64_t *s2) {
    uint64_t x[W], c[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
        x[w] = s1[w] ^ s2[w];
        c[w] = s1[w] & s2[w];
    }
    int o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = pop_lowest<W>(x);
    int a0, a1, b0, b1;
    arrange4<W>(o, s1, a0, a1, b0, b1);
    const int diff = nstacked<W>(a0, a1, c) + nstacked<W>(b0, b1, c);
    double e = Vm(p, a0, a1, b0, b1) - Vm(p, a0, a1, b1, b0);
    return negate_if(e, diff & 1);
}

// two_diff_orbitals(u1, u2, d1, d2) (CIMethod.cpp:444-457): alpha-beta double
template <int W>
__device__ __forceinline__ double two_diff_ab(const DetParams &p, const uint64_t *u1, const uint64_t *u2, const uint64_t *d1,
                              const uint64_t *d2) {
    uint64_t xu[W], cu[W], xd[W], cd[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
        xu[w] = u1[w] ^ u2[w];
        cu[w] = u1[w] & u2[w];
        xd[w] = d1[w] ^ d2[w];
        cd[w] = d1[w] & d2[w];
    }
    // arrange_order with two orbitals: the one occupied in the first string first
    int a0 = pop_lowest<W>(xu), a1 = pop_lowest<W>(xu);
    if (!has_bit<W>(u1, a0)) {
        const int t = a0;
        a0 = a1;
        a1 = t;
    }
    int b0 = pop_lowest<W>(xd), b1 = pop_lowest<W>(xd);
    if (!has_bit<W>(d1, b0)) {
        const int t = b0;
        b0 = b1;
        b1 = t;
    }
    const int diff = nstacked<W>(a0, a1, cu) + nstacked<W>(b0, b1, cd);
    double e = Vm(p, a0, b0, a1, b1);
    return negate_if(e, diff & 1);
}

// The same elements for strings of one word U (uint32_t to 32 orbitals, uint64_t to
// 64): the excitation's orbitals from the words themselves (a lowest or highest set
// bit each) and the phase from one popcount, the parity of both strings' electrons
// between the orbitals. The integrals and the order of the additions are those above.
__device__ __forceinline__ int low_bit(uint32_t x) { return __ffs((int)x) - 1; }
__device__ __forceinline__ int low_bit(uint64_t x) { return __ffsll((long long)x) - 1; }
__device__ __forceinline__ int high_bit(uint32_t x) { return 31 - __clz((int)x); }
__device__ __forceinline__ int high_bit(uint64_t x) { return 63 - __clzll((long long)x); }
__device__ __forceinline__ int bits(uint32_t x) { return __popc(x); }
__device__ __forceinline__ int bits(uint64_t x) { return __popcll(x); }

// The orbitals from the lower of two single bits up to, not including, the other.
template <typename U>
__device__ __forceinline__ U between(U a, U b) {
    return (a - 1) ^ (b - 1);
}

template <typename U>
__device__ __forceinline__ double word_double_ab(const DetParams &p, U u1, U u2, U d1, U d2) {
    const U xu = u1 ^ u2, xd = d1 ^ d2;
    const U a0 = xu & u1, a1 = xu & u2, b0 = xd & d1, b1 = xd & d2;
    const int odd = bits((U)((u1 & u2 & between(a0, a1)) ^ (d1 & d2 & between(b0, b1)))) & 1;
    const uint32_t L = (uint32_t)p.L;  // L^4 <= 2^24
    const double e = __ldg(p.eri + (((uint32_t)low_bit(a0) * L + (uint32_t)low_bit(a1)) * L + (uint32_t)low_bit(b0)) * L +
                           (uint32_t)low_bit(b1));
    return negate_if(e, odd);
}

template <typename U>
__device__ __forceinline__ double word_double_same(const DetParams &p, U s1, U s2) {
    const U x = s1 ^ s2, a = x & s1, b = x & s2;
    const U alo = a & (0 - a), blo = b & (0 - b);
    const int odd = bits((U)(s1 & s2 & (between(alo, (U)(a ^ alo)) ^ between(blo, (U)(b ^ blo))))) & 1;
    const uint32_t L = (uint32_t)p.L, a0 = low_bit(a), a1 = high_bit(a), b0 = low_bit(b), b1 = high_bit(b);
    const double e = __ldg(p.eri + ((a0 * L + b0) * L + a1) * L + b1) - __ldg(p.eri + ((a0 * L + b1) * L + a1) * L + b0);
    return negate_if(e, odd);
}

template <typename U>
__device__ __forceinline__ double word_single(const DetParams &p, U s1, U s2, U other) {
    const U x = s1 ^ s2, c = s1 & s2;
    const U lo = x & (0 - x);
    const uint32_t L = (uint32_t)p.L, o0 = low_bit(x), o1 = high_bit(x);
    double e = __ldg(p.h + o0 * L + o1);
    const double *ez = p.eri + (o0 * L + o1) * L * L, *ex = p.eri + o0 * L * L * L + o1;
    for (U y = c; y;) {  // four terms' loads in flight, the terms added in order
        double t[4], u[4];
        int n = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (y) {
                const uint32_t z = low_bit(y);
                y &= y - 1;
                t[k] = __ldg(ez + z * (L + 1));        // <o0 z|o1 z>
                u[k] = __ldg(ex + z * (L + 1) * L);    // <o0 z|z o1>
                n = k + 1;
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < n) e += t[k] - u[k];
    }
    for (U y = other; y;) {
        double t[4];
        int n = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (y) {
                const uint32_t z = low_bit(y);
                y &= y - 1;
                t[k] = __ldg(ez + z * (L + 1));
                n = k + 1;
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < n) e += t[k];
    }
    return negate_if(e, bits((U)(c & between(lo, (U)(x ^ lo)))) & 1);
}

template <int W>
__global__ void k_dets_diag(DetParams p, double *diag) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < p.n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t *d = p.dets + i * 2 * W;
        diag[i] = diagonal<W>(p, d, d + W);
    }
}

// ---------------------------------------------------------------------------
// The pair scan of the build and of the matvec without a stored matrix.
//
// A block owns kScanRows rows, one per lane of every warp; its warps split the
// columns. A warp stages 32 columns and every lane tests its row against each of
// them, so a column is one broadcast shared-memory read and 32 pairs are a few
// integer instructions: the 32-bit words of the two determinants' XOR (each word
// rotated by its own amount) are OR-ed together and the pair passes when at most 4
// bits are set. The OR never has more bits than the words together, so no connected
// pair fails; the few others that pass are dropped below. What bounds it is POPC,
// 16 lanes per clock and SM: one of them per pair here (a popcount per word before).
//
// The pairs that pass, a few in a hundred, go to the warp's queue in shared memory
// and are evaluated 32 at a time on full warps: doubles first, then the singles, a
// chain of FP64 additions that costs the warp the same with one lane as with all
// of them. Evaluated where they were found, one lane or two of a warp at work, they
// were the time of the pass. (L=32 8a8b CISD list, 52,705 determinants, list to
// CRS and one product: 23.4 -> 4.6 ms; matvec without a stored matrix of a random 70%
// of the L=28 7a7b CISD list, 21,500 determinants: 4.53 -> 0.49 ms.)
//
// The queue holds a row's columns in ascending order (words in order, a row's bits
// in order), so the fill writes each row's kept elements in order at the row's start
// plus the counts of the segments before it.
constexpr int kScanRows = 32;
constexpr int kSegs = 64;  // column segments of the count and fill passes
constexpr int kQueue = 256;                 // a word of 8 rows fits whatever passes
constexpr int kQueueColBits = 27;           // queue entry: row << 27 | column - the queue's first column
constexpr uint32_t kQueueColMask = (1u << kQueueColBits) - 1u;

// 32-bit words a determinant is tested with: 2 (L <= 32), 4 (L <= 64) or 8.
template <int W, int NW>
__device__ __forceinline__ void scan_key(const uint64_t *rec, uint32_t *k) {
    if constexpr (NW == 2) {
        k[0] = (uint32_t)rec[0];
        k[1] = __funnelshift_l((uint32_t)rec[1], (uint32_t)rec[1], 16);
    } else {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const uint32_t v = (uint32_t)(rec[w >> 1] >> (32 * (w & 1)));
            k[w] = __funnelshift_l(v, v, w * (32 / NW));
        }
    }
}

// m += bit where x has at most 4 bits set. The multiply-add (one = 1, not known to
// the compiler) keeps the add off the ALU pipe, which the XORs and compares fill.
__device__ __forceinline__ void mark(uint32_t &m, uint32_t x, uint32_t bit, uint32_t one) {
    asm("{\n\t.reg .pred q;\n\tsetp.le.u32 q, %1, 4;\n\t@q mad.lo.u32 %0, %2, %3, %0;\n\t}"
        : "+r"(m)
        : "r"((uint32_t)__popc(x)), "r"(one), "r"(bit));
}

// Where a segment's kept elements of the lane's row begin: the row's start and the counts of
// the segments before it, the warp summing a row at a time (a lane's own 63 counts lie 256
// bytes from its neighbour's).
__device__ __forceinline__ int64_t segment_start(const DetParams &p, int64_t r0, int seg) {
    const int lane = threadIdx.x & 31;
    const int64_t i = r0 + lane;
    const int rows = (int)min((int64_t)p.group, p.nrows - r0);
    int64_t at = lane < rows ? p.row_ptr[i] : 0;
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
        const uint32_t *c = p.seg_count + (r0 + r) * kSegs;
        const uint32_t sum = __reduce_add_sync(0xffffffffu, (lane < seg ? c[lane] : 0u) + (lane + 32 < seg ? c[lane + 32] : 0u));
        if (lane == r) at += sum;
    }
    return at;
}

// Shared memory of one warp.
template <int W, int NW>
struct ScanWarp {
    alignas(16) uint32_t key[32 * NW];  // the staged columns
    double val[kQueue];
    uint32_t at[kQueue];
    uint16_t single[kQueue];  // queue positions of the singles
    uint32_t run[kScanRows], low[kScanRows];  // kept elements so far; those below the diagonal
};

template <int W>
struct ScanRow {
    uint64_t s[kScanRows][2 * W];
};

// The fill's output of one queue entry's value, lanes in queue order. `live` lanes hold an
// entry: row, column j, value v.
template <int MODE, int W, int NW>
__device__ __forceinline__ void scan_emit(const DetParams &p, ScanWarp<W, NW> &q, const int64_t *rowpos, bool live, int row,
                                          int64_t j, double v) {
    const int lane = threadIdx.x & 31;
    const bool keep = live && keep_value(v);
    const unsigned kb = __ballot_sync(0xffffffffu, keep);
    if (kb == 0) return;
    // the kept entries of this lane's row
    const unsigned same = __match_any_sync(0xffffffffu, live ? row : 32 + lane) & kb;
    if (keep) {
        const int before = __popc(same & ((1u << lane) - 1u));
        const int64_t pos = rowpos[row] + q.run[row] + before;
        p.col[pos] = (uint32_t)j;
        if (MODE == kDetFill64) {
            p.val64[pos] = v;
        } else {
            split_fp32(v, p.val32[pos], p.val32lo[pos]);
        }
    }
    __syncwarp();
    if (keep && (same >> lane) == 1u) q.run[row] += __popc(same);  // the row's last kept lane
    __syncwarp();
}

// The element of a connected pair, row's determinant (ui, di) against list entry j; 0 for
// a pair that is not connected. A single is left to single_of.
template <int W, typename U>
__device__ __forceinline__ double pair_of(const DetParams &p, const uint64_t *ui, int64_t i, int64_t j, bool &single) {
    const uint64_t *di = ui + W;
    double v = 0;
    if constexpr (W == 1) {
        const ulonglong2 rj = __ldg(reinterpret_cast<const ulonglong2 *>(p.dets) + j);
        const U u1 = (U)ui[0], d1 = (U)di[0], u2 = (U)rj.x, d2 = (U)rj.y;
        const int nu = bits((U)(u1 ^ u2)), nd = bits((U)(d1 ^ d2));
        if (nu + nd == 2) {
            single = true;
        } else if (nu == 2 && nd == 2) {
            v = word_double_ab<U>(p, u1, u2, d1, d2);
        } else if (nu + nd == 4) {
            v = word_double_same<U>(p, nu ? u1 : d1, nu ? u2 : d2);
        } else if (nu + nd == 0) {
            v = p.diag[i];  // the row itself, or a repeat of its determinant in the list
        }
    } else {
        uint64_t uj[W], dj[W];
        int nu = 0, nd = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uj[w] = __ldg(p.dets + j * 2 * W + w);
            dj[w] = __ldg(p.dets + j * 2 * W + W + w);
            nu += __popcll(ui[w] ^ uj[w]);
            nd += __popcll(di[w] ^ dj[w]);
        }
        if (nu + nd == 0) {
            v = p.diag[i];
        } else if (nu + nd == 2) {
            single = true;
        } else if (nu == 2 && nd == 2) {
            v = two_diff_ab<W>(p, ui, uj, di, dj);
        } else if (nu + nd == 4) {
            uint64_t a[W], b[W];
#pragma unroll
            for (int w = 0; w < W; ++w) {
                a[w] = nu ? ui[w] : di[w];
                b[w] = nu ? uj[w] : dj[w];
            }
            v = two_diff_same<W>(p, a, b);
        }
    }
    return v;
}

template <int W, typename U>
__device__ __forceinline__ double single_of(const DetParams &p, const uint64_t *ui, int64_t j) {
    const uint64_t *di = ui + W;
    if constexpr (W == 1) {
        const ulonglong2 rj = __ldg(reinterpret_cast<const ulonglong2 *>(p.dets) + j);
        const U u1 = (U)ui[0], d1 = (U)di[0], u2 = (U)rj.x, d2 = (U)rj.y;
        const bool up = u1 != u2;
        return word_single<U>(p, up ? u1 : d1, up ? u2 : d2, up ? d1 : u1);
    } else {
        uint64_t a[W], b[W], o[W];
        bool up = false;
#pragma unroll
        for (int w = 0; w < W; ++w) up = up || ui[w] != __ldg(p.dets + j * 2 * W + w);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            a[w] = up ? ui[w] : di[w];
            b[w] = __ldg(p.dets + j * 2 * W + (up ? 0 : W) + w);
            o[w] = up ? di[w] : ui[w];
        }
        return one_diff<W>(p, a, b, o);
    }
}

// Evaluates and outputs the queue's n entries (columns from `first`).
template <int MODE, int W, int NW>
__device__ __noinline__ void scan_flush(const DetParams &p, ScanWarp<W, NW> &q, const ScanRow<W> &rows,
                                        const int64_t *rowpos, int64_t r0, int n, int64_t first) {
    using U = std::conditional_t<NW == 2, uint32_t, uint64_t>;
    const int lane = threadIdx.x & 31;
    auto put = [&](int k, int row, int64_t j, double v) {
        if (MODE != kDetCount) {
            q.val[k] = v;
        } else if (keep_value(v)) {
            atomicAdd(&q.run[row], 1u);  // integer counts: any order
            if (j < r0 + row) atomicAdd(&q.low[row], 1u);
        }
    };
    __syncwarp();
    int ns = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        bool single = false;
        if (k < n) {
            const uint32_t e = q.at[k];
            const int row = (int)(e >> kQueueColBits);
            const int64_t j = first + (e & kQueueColMask);
            const double v = pair_of<W, U>(p, rows.s[row], r0 + row, j, single);
            if (!single) put(k, row, j, v);
        }
        const unsigned sb = __ballot_sync(0xffffffffu, single);
        if (single) q.single[ns + __popc(sb & ((1u << lane) - 1u))] = (uint16_t)k;
        ns += __popc(sb);
    }
    __syncwarp();
    for (int k0 = 0; k0 < ns; k0 += 32) {
        if (k0 + lane < ns) {
            const int k = q.single[k0 + lane];
            const uint32_t e = q.at[k];
            const int row = (int)(e >> kQueueColBits);
            const int64_t j = first + (e & kQueueColMask);
            put(k, row, j, single_of<W, U>(p, rows.s[row], j));
        }
    }
    __syncwarp();
    if (MODE != kDetCount) {
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + lane;
            const bool live = k < n;
            const uint32_t e = live ? q.at[k] : 0u;
            scan_emit<MODE, W, NW>(p, q, rowpos, live, (int)(e >> kQueueColBits), first + (e & kQueueColMask),
                                   live ? q.val[k] : 0.0);
        }
    }
    __syncwarp();
}

// The lane's row (words rk) against the 32 staged columns: bit c set where the pair may
// be connected.
template <int NW>
__device__ __forceinline__ uint32_t scan_word(const uint32_t *key, const uint32_t *rk, uint32_t one) {
    uint32_t m = 0;
#pragma unroll
    for (int c = 0; c < 32; c += (NW == 2 ? 2 : 1)) {
        if constexpr (NW == 2) {
            const uint4 k = *reinterpret_cast<const uint4 *>(key + c * NW);
            mark(m, (k.x ^ rk[0]) | (k.y ^ rk[1]), 1u << c, one);
            mark(m, (k.z ^ rk[0]) | (k.w ^ rk[1]), 2u << c, one);
        } else {
            uint32_t o = 0;
#pragma unroll
            for (int w = 0; w < NW; w += 4) {
                const uint4 k = *reinterpret_cast<const uint4 *>(key + c * NW + w);
                o |= (k.x ^ rk[w]) | (k.y ^ rk[w + 1]);
                o |= (k.z ^ rk[w + 2]) | (k.w ^ rk[w + 3]);
            }
            mark(m, o, 1u << c, one);
        }
    }
    return m;
}

// The bits of m whose pairs are connected (at most four spin orbitals differ).
template <int NW>
__device__ __forceinline__ uint32_t connected(const uint32_t *key, const uint32_t *rk, uint32_t m) {
    uint32_t x = 0;
    for (; m; m &= m - 1) {
        const int c = __ffs((int)m) - 1;
        int d = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) d += __popc(key[c * NW + w] ^ rk[w]);
        if (d <= 4) x |= 1u << c;
    }
    return x;
}

// One-warp blocks, one per 32 rows and segment of the columns (grid: row groups x kSegs),
// so that a segment dense in connected pairs holds up no other (the L=32 list's build:
// 15.7 ms with the segments as the warps of one block, which then wait for the densest;
// 9.2 ms with 16 one-warp blocks of them, 4.6 with 64 and the single-word element
// functions).
template <int W, int NW, int MODE>
__global__ void __launch_bounds__(32, 32) k_dets_scan(const DetParams p) {
    __shared__ ScanWarp<W, NW> q;
    __shared__ ScanRow<W> rows;
    __shared__ int64_t rowpos[kScanRows];
    const int lane = threadIdx.x;
    const int64_t group = blockIdx.x / kSegs;
    const int seg = (int)(blockIdx.x - group * kSegs);
    const int64_t r0 = group * p.group;
    const int64_t i = r0 + lane;
    const bool active = lane < p.group && i < p.nrows;
    uint64_t rec[2 * W];
#pragma unroll
    for (int w = 0; w < 2 * W; ++w) rec[w] = active ? p.dets[i * 2 * W + w] : 0;
    uint32_t rk[NW];
    scan_key<W, NW>(rec, rk);
#pragma unroll
    for (int w = 0; w < 2 * W; ++w) rows.s[lane][w] = rec[w];
    q.run[lane] = q.low[lane] = 0;
    const int64_t words = (p.block + 31) / 32, w0 = words * seg / kSegs, w1 = words * (seg + 1) / kSegs;
    if (w0 == w1) {  // a short list has fewer words than segments
        if (MODE == kDetCount && active) p.seg_count[i * kSegs + seg] = 0;
        return;
    }
    if (MODE == kDetFill64 || MODE == kDetFill32) rowpos[lane] = segment_start(p, r0, seg);
    __syncwarp();
    const uint32_t one = p.one;
    int qn = 0;
    int64_t first = 0;
    uint64_t next[2 * W];
    auto load = [&](int64_t word) {
        const int64_t j = word * 32 + lane;
#pragma unroll
        for (int w = 0; w < 2 * W; ++w) next[w] = (word < w1 && j < p.block) ? __ldg(p.dets + j * 2 * W + w) : 0;
    };
    load(w0);
    for (int64_t word = w0; word < w1; ++word) {
        const int64_t base = word * 32;
        uint32_t ck[NW];
        scan_key<W, NW>(next, ck);
#pragma unroll
        for (int w = 0; w < NW; ++w) q.key[lane * NW + w] = ck[w];
        __syncwarp();
        load(word + 1);
        uint32_t m = scan_word<NW>(q.key, rk, one);
        __syncwarp();  // the staged columns are read; the next word's may be written
        if (p.block - base < 32) m &= (1u << (int)(p.block - base)) - 1u;
        if (!active) m = 0;
        if (!__any_sync(0xffffffffu, m)) continue;
        int off = __popc(m);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, off, o);
            if (lane >= o) off += u;
        }
        const int total = __shfl_sync(0xffffffffu, off, 31);
        off -= __popc(m);
        if (qn > 0 && (qn + total > kQueue || base - first > (int64_t)(kQueueColMask - 32))) {
            scan_flush<MODE, W, NW>(p, q, rows, rowpos, r0, qn, first);
            qn = 0;
        }
        if (qn == 0) first = base;
        const uint32_t tag = ((uint32_t)lane << kQueueColBits) | (uint32_t)(base - first);
        if (total <= kQueue) {
            for (int k = qn + off; m; m &= m - 1) q.at[k++] = tag + (uint32_t)(__ffs((int)m) - 1);
            qn += total;
        } else {  // a dense word: eight rows at a time fill the queue at most
            for (int g = 0; g < 4; ++g) {
                const int g0 = __shfl_sync(0xffffffffu, off, 8 * g);
                const int g1 = g < 3 ? __shfl_sync(0xffffffffu, off, (8 * g + 8) & 31) : total;
                if ((lane >> 3) == g)
                    for (int k = off - g0; m; m &= m - 1) q.at[k++] = tag + (uint32_t)(__ffs((int)m) - 1);
                if (g1 > g0) scan_flush<MODE, W, NW>(p, q, rows, rowpos, r0, g1 - g0, first);
            }
        }
    }
    if (qn > 0) scan_flush<MODE, W, NW>(p, q, rows, rowpos, r0, qn, first);
    if constexpr (MODE == kDetCount) {
        if (active) {
            p.seg_count[i * kSegs + seg] = q.run[lane];
            if (q.run[lane]) atomicAdd(p.row_count + i, q.run[lane]);  // integer sums: any order
            if (q.low[lane]) atomicAdd(p.upper_off + i, q.low[lane]);
        }
    }
}

// ---------------------------------------------------------------------------
// The build where no integral is dropped (every |(pq|rs)| > 1e-14: molecules without
// symmetry, rotated orbitals). The row structure is then the connected pairs, so the
// count pass evaluates nothing: it scans, tests the pairs that pass exactly in place and,
// while they fit kMaskBytes and the device's memory, leaves the 32-column masks (n^2 / 8
// bytes) for the fill. The fill reads the masks (or scans again), and every element's place follows from its row's
// count as it is queued, so doubles and singles are written as they are evaluated. An
// element that vanishes all the same (a difference of equal integrals) is counted, and
// the build starts again with the passes above, which evaluate twice. L=32 8a8b CISD
// list, list to CRS and one product: 4.64 -> 3.22 ms.
constexpr size_t kMaskBytes = size_t(1) << 30;
// Lists shorter than this evaluate twice all the same: a wait for the count of vanished
// elements, and the masks' passes, cost as much as their few elements (60 determinants 125
// against 121 us, 442 136 and 132, 1,000 151 and 149).
constexpr int64_t kShortList = 1000;

template <int W, int NW>
struct FillWarp {
    alignas(16) uint32_t key[32 * NW];
    uint32_t at[kQueue], pos[kQueue];  // queue entry; its place in the row
    uint16_t single[kQueue];
    int64_t rowpos[kScanRows];
    ScanRow<W> rows;
};

template <int MODE, int W, int NW>
__device__ __noinline__ void fill_flush(const DetParams &p, FillWarp<W, NW> &q, int64_t r0, int n, int64_t first) {
    using U = std::conditional_t<NW == 2, uint32_t, uint64_t>;
    const int lane = threadIdx.x & 31;
    bool dropped = false;
    auto put = [&](int k, int row, int64_t j, double v) {
        const int64_t pos = q.rowpos[row] + q.pos[k];
        p.col[pos] = (uint32_t)j;
        if (MODE == kDetFill64) {
            p.val64[pos] = v;
        } else {
            split_fp32(v, p.val32[pos], p.val32lo[pos]);
        }
        dropped = dropped || !keep_value(v);
    };
    __syncwarp();
    int ns = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        bool single = false;
        if (k < n) {
            const uint32_t e = q.at[k];
            const int row = (int)(e >> kQueueColBits);
            const int64_t j = first + (e & kQueueColMask);
            const double v = pair_of<W, U>(p, q.rows.s[row], r0 + row, j, single);
            if (!single) put(k, row, j, v);
        }
        const unsigned sb = __ballot_sync(0xffffffffu, single);
        if (single) q.single[ns + __popc(sb & ((1u << lane) - 1u))] = (uint16_t)k;
        ns += __popc(sb);
    }
    __syncwarp();
    for (int k0 = 0; k0 < ns; k0 += 32) {
        if (k0 + lane < ns) {
            const int k = q.single[k0 + lane];
            const uint32_t e = q.at[k];
            const int row = (int)(e >> kQueueColBits);
            const int64_t j = first + (e & kQueueColMask);
            put(k, row, j, single_of<W, U>(p, q.rows.s[row], j));
        }
    }
    if (__any_sync(0xffffffffu, dropped) && lane == 0) *p.dropped = 1u;  // any writer's 1
    __syncwarp();
}

// One-warp blocks, 32 rows x a segment of the columns, as the passes above. MASKS: the
// count leaves the masks, the fill reads them ([row group][word][32 rows]).
template <int W, int NW, int MODE, bool MASKS>
__global__ void __launch_bounds__(32, 32) k_dets_pairs(const DetParams p) {
    __shared__ FillWarp<W, NW> q;
    const int lane = threadIdx.x;
    const int64_t group = blockIdx.x / kSegs, r0 = group * p.group, i = r0 + lane;
    const int seg = (int)(blockIdx.x - group * kSegs);
    const bool active = lane < p.group && i < p.nrows;
    uint64_t rec[2 * W];
#pragma unroll
    for (int w = 0; w < 2 * W; ++w) q.rows.s[lane][w] = rec[w] = active ? p.dets[i * 2 * W + w] : 0;
    uint32_t rk[NW];
    scan_key<W, NW>(rec, rk);
    const int64_t words = (p.block + 31) / 32, w0 = words * seg / kSegs, w1 = words * (seg + 1) / kSegs;
    uint32_t run = 0, low = 0;
    if (w0 == w1) {  // a short list has fewer words than segments
        if (MODE == kDetCount && active) p.seg_count[i * kSegs + seg] = 0;
        return;
    }
    if (MODE != kDetCount) q.rowpos[lane] = segment_start(p, r0, seg);
    __syncwarp();
    const uint32_t one = p.one;
    uint32_t *masks = p.masks + group * words * 32 + lane;
    int qn = 0;
    int64_t first = 0;
    constexpr bool kScan = MODE == kDetCount || !MASKS;
    uint64_t next[2 * W];
    uint32_t ahead = 0;
    auto load = [&](int64_t word) {
        if constexpr (kScan) {
            const int64_t j = word * 32 + lane;
#pragma unroll
            for (int w = 0; w < 2 * W; ++w) next[w] = (word < w1 && j < p.block) ? __ldg(p.dets + j * 2 * W + w) : 0;
        } else {
            ahead = word < w1 ? __ldcs(masks + word * 32) : 0u;
        }
    };
    load(w0);
    for (int64_t word = w0; word < w1; ++word) {
        const int64_t base = word * 32;
        uint32_t m;
        if constexpr (kScan) {
            uint32_t ck[NW];
            scan_key<W, NW>(next, ck);
#pragma unroll
            for (int w = 0; w < NW; ++w) q.key[lane * NW + w] = ck[w];
            __syncwarp();
            load(word + 1);
            m = scan_word<NW>(q.key, rk, one);
            if (p.block - base < 32) m &= (1u << (int)(p.block - base)) - 1u;
            m = connected<NW>(q.key, rk, active ? m : 0u);
            __syncwarp();  // the staged columns are read; the next word's may be written
        } else {
            m = ahead;
            load(word + 1);
        }
        if constexpr (MODE == kDetCount) {
            run += __popc(m);
            low += __popc(base + 32 <= i ? m : base < i ? m & ((1u << (int)(i - base)) - 1u) : 0u);
            if (MASKS) masks[word * 32] = m;
        } else {
            if (!__any_sync(0xffffffffu, m)) continue;
            const int mine = __popc(m);
            int off = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, off, o);
                if (lane >= o) off += u;
            }
            const int total = __shfl_sync(0xffffffffu, off, 31);
            off -= mine;
            if (qn > 0 && (qn + total > kQueue || base - first > (int64_t)(kQueueColMask - 32))) {
                fill_flush<MODE, W, NW>(p, q, r0, qn, first);
                qn = 0;
            }
            if (qn == 0) first = base;
            const uint32_t tag = ((uint32_t)lane << kQueueColBits) | (uint32_t)(base - first);
            auto push = [&](int k) {
                for (; m; m &= m - 1, ++k) {
                    q.at[k] = tag + (uint32_t)(__ffs((int)m) - 1);
                    q.pos[k] = run++;
                }
            };
            if (total <= kQueue) {
                push(qn + off);
                qn += total;
            } else {  // a dense word: eight rows at a time fill the queue at most
                for (int g = 0; g < 4; ++g) {
                    const int g0 = __shfl_sync(0xffffffffu, off, 8 * g);
                    const int g1 = g < 3 ? __shfl_sync(0xffffffffu, off, (8 * g + 8) & 31) : total;
                    if ((lane >> 3) == g) push(off - g0);
                    if (g1 > g0) fill_flush<MODE, W, NW>(p, q, r0, g1 - g0, first);
                }
            }
        }
    }
    if constexpr (MODE == kDetCount) {
        if (active) {
            p.seg_count[i * kSegs + seg] = run;
            if (run) atomicAdd(p.row_count + i, run);  // integer sums: any order
            if (low) atomicAdd(p.upper_off + i, low);
        }
    } else if (qn > 0) {
        fill_flush<MODE, W, NW>(p, q, r0, qn, first);
    }
}

// ---------------------------------------------------------------------------
// The matvec without a stored matrix: y_i = sum_j H_ij x_j, every element recomputed. A
// block owns 32 rows; its warps take every kMvWarps-th word of the columns, which spreads
// dense stretches over them, and meet once at the end. A warp keeps the masks of up to
// kMvSpan words and queues their pairs row by row, so that after the evaluation every
// lane adds its own row's products, one after the other: about as many FP64 additions for
// the warp as the longest row has elements in the queue. (Words queued one by one, the
// lanes of a row finding each other for each 32 entries: 600 instructions per 32
// elements, 0.49 ms for the L=28 list; now
// 0.48.)
//
// RANGED: a list with a stored block (CI_Big with a kept part) leaves out the block's
// pairs. CL: the blocks (a cluster) that share 32 rows' columns. Two where one would leave
// the SMs fewer than four, three of which an SM holds at a time. One | two, alone and among
// other products: 6,189 rows of L=24 254 | 138 and 100 | 76 us, 16,471 of L=24 956 | 536
// alone, 12,290 of L=28 453 | 262 and 182 | 173, 21,507 853 | 613 and 492 | 505, 52,705 of
// L=32 2.89 | 3.43 ms; four or eight were slower among others everywhere.
constexpr int kMvWarps = 8;
constexpr int kMvSpan = 16;

template <int W, int NW>
struct MatvecWarp {
    alignas(16) uint32_t key[32 * NW];
    double val[kQueue], xv[kQueue];
    uint32_t mask[kMvSpan][32];
    int64_t base[kMvSpan];
    uint16_t at[kQueue], single[kQueue];  // row << 9 | word << 5 | column; queue positions of the singles
};

// Rows of the matvec's groups of 32, in runs of 2^shift consecutive ones from as many places
// of the list: in a list ordered by excitation the best connected rows stand together, and
// a block with 32 of them (a CISD list's reference and first singles) ends long after the
// others. Whole runs keep the words that many of a group's rows meet. Rows of one word in
// runs of 16, of two in runs of 8 (their elements take longer), in order from 8 groups
// per SM, where other groups fill the wait. Alone and among other products, runs | in
// order: L=70 4a4b, 6,100 rows 302 and 172 | 517 and 180 us, 14,000 822 and 728 | 1,067
// and 773 (the matvec of a warp per row and element it replaced: 368 and 1,268 alone);
// L=24 6a6b, 16,471 513 and 394 | 540 and 398; L=28 7a7b, 21,500 885 and 480 | 1,159 and
// 500; L=32 8a8b, 35,000 1,485 and 1,134 | 2,211 and 1,273, 52,705 3,071 and 2,629 | 2,898
// and 2,504. Lists in no order take the same time either way, but for where the group of
// their best connected row stands in the grid.
// The rows of the stored block make groups of their own, which skip its columns; its last
// ones, short of a group, go with the rest.
struct MvRows {
    int64_t inside, outside;  // groups of the stored block's rows, and of the others
    int shift;
    // the place in the list of a group's row `lane`: n or more where there is none
    __device__ int64_t place(int64_t group, int lane) const {
        const bool in = group < inside;
        const int64_t groups = in ? inside : outside, g = in ? group : group - inside;
        const int64_t i = (((lane >> shift) * groups + g) << shift) + (lane & ((1 << shift) - 1));
        return in ? i : inside * kScanRows + i;
    }
};

// Evaluates the queued words (n pairs in all, `mine` of the lane's row) and adds them.
template <int W, int NW>
__device__ __noinline__ double matvec_flush(const DetParams &p, MatvecWarp<W, NW> &q, const ScanRow<W> &rows,
                                            const int64_t *at, int span, int n, int mine, const double *__restrict__ x, double acc) {
    using U = std::conditional_t<NW == 2, uint32_t, uint64_t>;
    const int lane = threadIdx.x & 31;
    int start = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, start, o);
        if (lane >= o) start += u;
    }
    start -= mine;
    for (int s = 0, k = start; s < span; ++s)
        for (uint32_t m = q.mask[s][lane]; m; m &= m - 1)
            q.at[k++] = (uint16_t)(lane << 9 | s << 5 | (__ffs((int)m) - 1));
    __syncwarp();
    auto place = [&](int k, int &row, int64_t &j) {
        const int e = q.at[k];
        row = e >> 9;
        j = q.base[(e >> 5) & 15] + (e & 31);
    };
    int ns = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        bool single = false;
        if (k < n) {
            int row;
            int64_t j;
            place(k, row, j);
            const double xj = __ldg(x + j);
            const double v = pair_of<W, U>(p, rows.s[row], at[row], j, single);
            if (!single) q.val[k] = v;
            q.xv[k] = xj;
        }
        const unsigned sb = __ballot_sync(0xffffffffu, single);
        if (single) q.single[ns + __popc(sb & ((1u << lane) - 1u))] = (uint16_t)k;
        ns += __popc(sb);
    }
    __syncwarp();
    for (int k0 = 0; k0 < ns; k0 += 32) {
        if (k0 + lane < ns) {
            const int k = q.single[k0 + lane];
            int row;
            int64_t j;
            place(k, row, j);
            q.val[k] = single_of<W, U>(p, rows.s[row], j);
        }
    }
    __syncwarp();
    for (int k = start; k < start + mine; ++k) {
        const double v = q.val[k];
        if (keep_value(v)) acc = fma(v, q.xv[k], acc);
    }
    __syncwarp();
    return acc;
}

template <int W, int NW, bool RANGED, int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(32 * kMvWarps, 3)
    k_dets_matvec(const DetParams p, const MvRows map, const double *__restrict__ x, double *__restrict__ y) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ ScanRow<W> rows;
    __shared__ int64_t at[kScanRows];  // the rows' places in the list
    __shared__ double part[kMvWarps][kScanRows];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % CL;  // of the rows' blocks
    MatvecWarp<W, NW> &q = reinterpret_cast<MatvecWarp<W, NW> *>(smem)[warp];
    const int64_t group = blockIdx.x / CL;
    const int64_t i = map.place(group, lane);
    const bool active = i < p.n;
    uint64_t rec[2 * W];
#pragma unroll
    for (int w = 0; w < 2 * W; ++w) rec[w] = active ? p.dets[i * 2 * W + w] : 0;
    uint32_t rk[NW];
    scan_key<W, NW>(rec, rk);
    if (warp == 0) {
        at[lane] = i;
#pragma unroll
        for (int w = 0; w < 2 * W; ++w) rows.s[lane][w] = rec[w];
    }
    __syncthreads();
    const int64_t c_lo = (RANGED && group < map.inside) ? p.block : 0;  // the stored rows' pairs outside the block
    const int64_t words = (p.n - c_lo + 31) / 32;
    const uint32_t one = p.one;
    uint64_t next[2 * W];
    auto load = [&](int64_t word) {
        const int64_t j = c_lo + word * 32 + lane;
#pragma unroll
        for (int w = 0; w < 2 * W; ++w) next[w] = (word < words && j < p.n) ? __ldg(p.dets + j * 2 * W + w) : 0;
    };
    int span = 0, n = 0, mine = 0;
    double acc = 0;
    auto flush = [&] {
        acc = matvec_flush<W, NW>(p, q, rows, at, span, n, mine, x, acc);
        span = n = mine = 0;
    };
    auto add = [&](int64_t base, uint32_t m, int total) {
        q.mask[span][lane] = m;
        if (lane == 0) q.base[span] = base;
        ++span;
        n += total;
        mine += __popc(m);
    };
    load(rank * kMvWarps + warp);
    for (int64_t word = rank * kMvWarps + warp; word < words; word += CL * kMvWarps) {
        const int64_t base = c_lo + word * 32;
        uint32_t ck[NW];
        scan_key<W, NW>(next, ck);
#pragma unroll
        for (int w = 0; w < NW; ++w) q.key[lane * NW + w] = ck[w];
        __syncwarp();
        load(word + CL * kMvWarps);
        uint32_t m = scan_word<NW>(q.key, rk, one);
        if (p.n - base < 32) m &= (1u << (int)(p.n - base)) - 1u;
        if (!active) m = 0;
        if (RANGED && i < p.block && base < p.block)
            m = p.block - base >= 32 ? 0u : m & ~((1u << (int)(p.block - base)) - 1u);
        m = connected<NW>(q.key, rk, m);
        const int total = __reduce_add_sync(0xffffffffu, __popc(m));  // the staged columns are read
        if (total == 0) continue;
        if (span == kMvSpan || n + total > kQueue) flush();
        if (total <= kQueue) {
            add(base, m, total);
            continue;
        }
        for (int g = 0; g < 4; ++g) {  // a dense word: eight rows at a time fill the queue at most
            const uint32_t mg = (lane >> 3) == g ? m : 0u;
            add(base, mg, __reduce_add_sync(0xffffffffu, __popc(mg)));
            flush();
        }
    }
    if (n > 0) flush();
    part[warp][lane] = acc;
    auto cluster = cooperative_groups::this_cluster();
    cluster.sync();
    if (rank == 0 && warp == 0 && active) {
        double a = 0;
        for (int b = 0; b < CL; ++b) {
            const double *sums = cluster.map_shared_rank(&part[0][0], b);
            for (int w = 0; w < kMvWarps; ++w) a += sums[w * kScanRows + lane];
        }
        // rows of the stored block add to the stored block's product, already in y
        y[i] = ((RANGED && i < p.block) ? y[i] : 0.0) + a;
    }
    cluster.sync();  // the sums are read
}

// The same for short lists: a warp owns one row and its lanes test 32 columns at a time, so
// that a few thousand rows make enough warps; the pairs found are queued and evaluated 32
// at a time, and every 32nd of them is added by one lane. Half the pairs per instruction of
// the kernel above, whose 32 rows to a warp leave a short list's blocks too few. Alone,
// and among other products, this | that: 1,577 rows of L=36 44 | 126 and 17 | 46 us; 5,665
// of L=20 133 | 280 and 107 | 123; 6,189 of L=24 236 | 138 and 129 | 76; 12,290 of L=28
// 623 | 262 and 400 | 173; longer strings the same (ordered lists, one right after another):
// 6,100 rows of L=60 195 | 220, 8,000 290 | 286, of L=70 (two words) 3,000 141 | 129, 6,100
// 335 | 296, 10,000 683 | 548.
constexpr int64_t kMvShort = 6000;

template <int W>
struct RowQueue {
    double val[kQueue];
    uint32_t at[kQueue];  // columns
    uint16_t single[kQueue];
};

template <int W, int NW>
__device__ __noinline__ double row_flush(const DetParams &p, RowQueue<W> &q, const uint64_t *row, int64_t i, int n,
                                         const double *__restrict__ x, double acc) {
    using U = std::conditional_t<NW == 2, uint32_t, uint64_t>;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    int ns = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        bool single = false;
        if (k < n) {
            const double v = pair_of<W, U>(p, row, i, q.at[k], single);
            if (!single) q.val[k] = v;
        }
        const unsigned sb = __ballot_sync(0xffffffffu, single);
        if (single) q.single[ns + __popc(sb & ((1u << lane) - 1u))] = (uint16_t)k;
        ns += __popc(sb);
    }
    __syncwarp();
    for (int k0 = 0; k0 < ns; k0 += 32)
        if (k0 + lane < ns) {
            const int k = q.single[k0 + lane];
            q.val[k] = single_of<W, U>(p, row, q.at[k]);
        }
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
        const double v = q.val[k];
        if (keep_value(v)) acc = fma(v, __ldg(x + q.at[k]), acc);
    }
    __syncwarp();
    return acc;
}

template <int W, int NW, bool RANGED>
__global__ void __launch_bounds__(32 * kMvWarps) k_dets_matvec_rows(const DetParams p, const double *__restrict__ x,
                                                                    double *__restrict__ y) {
    __shared__ RowQueue<W> queues[kMvWarps];
    __shared__ uint64_t rows[kMvWarps][2 * W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * kMvWarps + warp;
    if (i >= p.n) return;
    RowQueue<W> &q = queues[warp];
    uint64_t ri[2 * W];
#pragma unroll
    for (int w = 0; w < 2 * W; ++w) ri[w] = __ldg(p.dets + i * 2 * W + w);
    if (lane < 2 * W) rows[warp][lane] = __ldg(p.dets + i * 2 * W + lane);
    const int64_t c_lo = (RANGED && i < p.block) ? p.block : 0;  // a stored row's pairs outside the block
    int n = 0;
    double acc = 0;
    for (int64_t base = c_lo; base < p.n; base += 32) {
        const int64_t j = base + lane;
        int d = 0;
#pragma unroll
        for (int w = 0; w < 2 * W; ++w) {
            const uint64_t v = (j < p.n ? __ldg(p.dets + j * 2 * W + w) : ~ri[w]) ^ ri[w];
            d += NW == 2 ? __popc((uint32_t)v) : __popcll(v);
        }
        const unsigned m = __ballot_sync(0xffffffffu, d <= 4);  // past the list: every bit differs
        if (m == 0) continue;
        if (n + 32 > kQueue) {
            acc = row_flush<W, NW>(p, q, rows[warp], i, n, x, acc);
            n = 0;
        }
        if (d <= 4) q.at[n + __popc(m & ((1u << lane) - 1u))] = (uint32_t)j;
        n += __popc(m);
    }
    if (n > 0) acc = row_flush<W, NW>(p, q, rows[warp], i, n, x, acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    // rows of the stored block add to the stored block's product, already in y
    if (lane == 0) y[i] = ((RANGED && i < p.block) ? y[i] : 0.0) + acc;
}

__global__ void k_sum_u32(const uint32_t *a, int64_t n, unsigned long long *out) {
    unsigned long long s = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s += a[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);  // integer sum: exact in any order
}

int rows_grid(int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + kDetWarps - 1) / kDetWarps, (int64_t)sm_count() * 16));
}

// Rows of a warp in the build's passes. A short list has few words of columns and few
// groups of 32 rows, each a long queue of connected pairs on one warp; fewer rows make more
// warps. List to CRS in us, 32 | 16 | 8 | 4 rows: 60 determinants of L=8 150 | 137 | 128 | 125,
// 442 of L=10 170 | 145 | 137 | 136, 1,486 of L=14 190 | 169 | 164 | 168, 5,000 of L=20 322 |
// 292 | 298 | 335, 8,000 of L=24 444 | 413 | 435 | 537 and, with vanishing integrals, 632 | 535 |
// 530 | 649.
int build_group(int64_t n) { return n < kShortList ? 4 : n < 10000 ? 8 : 32; }

unsigned segment_blocks(const DetParams &p) {
    const int64_t blocks = (p.nrows + p.group - 1) / p.group * kSegs;
    if (blocks > (int64_t)INT32_MAX) throw std::invalid_argument("determinant list too long");
    return (unsigned)blocks;
}

// f with the words of 64 and of 32 bits a determinant of the list takes.
template <typename F>
void by_words(const DetParams &p, int W, F &&f) {
    if (W == 2)
        f(std::integral_constant<int, 2>{}, std::integral_constant<int, 8>{});
    else if (p.L > 32)
        f(std::integral_constant<int, 1>{}, std::integral_constant<int, 4>{});
    else
        f(std::integral_constant<int, 1>{}, std::integral_constant<int, 2>{});
}

template <int MODE>
void rows(const DetParams &p, int W, cudaStream_t s) {
    by_words(p, W, [&](auto w, auto nw) { k_dets_scan<w(), nw(), MODE><<<segment_blocks(p), 32, 0, s>>>(p); });
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
}

template <int MODE>
void pairs(const DetParams &p, int W, cudaStream_t s) {
    by_words(p, W, [&](auto w, auto nw) {
        if (p.masks)
            k_dets_pairs<w(), nw(), MODE, true><<<segment_blocks(p), 32, 0, s>>>(p);
        else
            k_dets_pairs<w(), nw(), MODE, false><<<segment_blocks(p), 32, 0, s>>>(p);
    });
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
}

void matvec(const DetParams &p, int W, const double *x, double *y, cudaStream_t s) {
    const bool ranged = p.block > 0 && p.block < p.n;  // a partly stored list
    by_words(p, W, [&](auto w, auto nw) {
        if (p.n < kMvShort) {
            const unsigned blocks = (unsigned)((p.n + kMvWarps - 1) / kMvWarps);
            if (ranged)
                k_dets_matvec_rows<w(), nw(), true><<<blocks, 32 * kMvWarps, 0, s>>>(p, x, y);
            else
                k_dets_matvec_rows<w(), nw(), false><<<blocks, 32 * kMvWarps, 0, s>>>(p, x, y);
            return;
        }
        MvRows map;
        map.inside = ranged ? p.block / kScanRows : 0;
        map.outside = (p.n - map.inside * kScanRows + kScanRows - 1) / kScanRows;
        const unsigned groups = (unsigned)(map.inside + map.outside);
        map.shift = groups >= 8 * (unsigned)sm_count() ? 5 : w() == 2 ? 3 : 4;
        constexpr int smem = (int)sizeof(MatvecWarp<w(), nw()>) * kMvWarps;
        auto go = [&](auto kern, unsigned blocks) {
            // the same value at every call: concurrent callers never lower it
            CIGPU_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            kern<<<blocks, 32 * kMvWarps, smem, s>>>(p, map, x, y);
        };
        const bool two = groups < 4 * (unsigned)sm_count();
        if (ranged && two)
            go(k_dets_matvec<w(), nw(), true, 2>, 2 * groups);
        else if (ranged)
            go(k_dets_matvec<w(), nw(), true, 1>, groups);
        else if (two)
            go(k_dets_matvec<w(), nw(), false, 2>, 2 * groups);
        else
            go(k_dets_matvec<w(), nw(), false, 1>, groups);
    });
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
}

DetParams params_of(const cigpu_crs &c) {
    DetParams p{};
    p.L = c.L;
    p.nup = c.nup;
    p.ndown = c.ndown;
    p.n = c.dim;
    p.dets = c.dets.p;
    p.eri = c.ham->d_eri.p;
    p.h = c.ham->d_h.p;
    p.diag = c.diag.p;
    p.nrows = c.dim;
    p.block = c.onthefly ? c.det_block : c.dim;
    return p;
}

// one line of a determinant file: "<up bits>|<down bits>", most significant orbital first
bool parse_line(const std::string &line, int words, uint64_t *up, uint64_t *down, int *nbits) {
    const size_t bar = line.find('|');
    if (bar == std::string::npos) return false;
    auto parse = [&](const std::string &s, uint64_t *out) {
        for (int w = 0; w < words; ++w) out[w] = 0;
        int bit = 0;
        for (size_t k = s.size(); k-- > 0;) {
            const char ch = s[k];
            if (ch == '0' || ch == '1') {
                if (bit >= 64 * words) return -1;
                if (ch == '1') out[bit >> 6] |= (uint64_t)1 << (bit & 63);
                ++bit;
            } else if (ch != ' ' && ch != '\t' && ch != '\r') {
                return -1;
            }
        }
        return bit;
    };
    const int a = parse(line.substr(0, bar), up), b = parse(line.substr(bar + 1), down);
    if (a <= 0 || b <= 0) return false;
    *nbits = std::max(a, b);
    return true;
}

// ---------------------------------------------------------------------------
// RDMs of a list's state (DensFILE::construct_CI_one_dens / construct_CI_two_dens,
// CIDens.cpp:1468-1529): every pair i <= j contributes c_i c_j through the
// reference's fill rules (fill_density_matrix_one / fill_density_matrix,
// CIDens.cpp:676-896) into the symmetric (min, max) storage of CIDens. The sums are
// accumulated as 64-bit fixed-point integers (value * 2^60, rounded to nearest) with
// integer atomics: integer addition is associative, so the result does not depend on
// the order the warps reach an element (bit-identical runs), and two's-complement
// wrap-around keeps every final sum exact while it lies within +-8 (RDM elements lie
// within +-1). Each contribution is rounded by at most 2^-61.
struct RdmAcc {
    unsigned long long *one, *aa, *ab, *bb;
    int L, np;
    bool two;
};

__device__ __forceinline__ void acc_add(unsigned long long *at, double v) {
    atomicAdd(at, (unsigned long long)__double2ll_rn(v * 0x1p60));
}
__device__ __forceinline__ void rdm_add_one(const RdmAcc &R, int spin, int o1, int o2, double v) {
    const int a = min(o1, o2), b = max(o1, o2);
    acc_add(R.one + ((int64_t)spin * R.L + a) * R.L + b, v);
}
// add_two_rdm (CIDens.cpp:227-256)
__device__ __forceinline__ void rdm_add_two(const RdmAcc &R, int spin, int o1, int o2, int o3, int o4, double v) {
    const int L = R.L;
    if (spin == 1) {
        const int64_t A = (int64_t)o1 * L + o2, B = (int64_t)o3 * L + o4;
        acc_add(R.ab + min(A, B) * (int64_t)L * L + max(A, B), v);
        return;
    }
    if (o1 == o2 || o3 == o4) return;
    int odd = 0;
    if (o1 > o2) {
        const int t = o1;
        o1 = o2;
        o2 = t;
        odd ^= 1;
    }
    if (o3 > o4) {
        const int t = o3;
        o3 = o4;
        o4 = t;
        odd ^= 1;
    }
    const int64_t A = o1 * L + o2 - (o1 + 1) * (o1 + 2) / 2, B = o3 * L + o4 - (o3 + 1) * (o3 + 2) / 2;
    acc_add((spin == 0 ? R.aa : R.bb) + min(A, B) * R.np + max(A, B), negate_if(v, odd));
}

// fill_one_dense (CIDens.cpp:676-754) for strings b1 -> b2 differing in one orbital;
// `same` is the other spin's string. alpha: the moved electron is alpha.
template <int W>
__device__ void fill_single(const RdmAcc &R, const uint64_t *b1, const uint64_t *b2, const uint64_t *same, double contr,
                            bool alpha) {
    uint64_t x[W], c[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
        x[w] = b1[w] ^ b2[w];
        c[w] = b1[w] & b2[w];
    }
    const int o0 = pop_lowest<W>(x), o1 = pop_lowest<W>(x);
    contr = negate_if(contr, nstacked<W>(o0, o1, c) & 1);
    rdm_add_one(R, alpha ? 0 : 1, o0, o1, contr);
    if (!R.two) return;
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t y = c[w]; y; y &= y - 1) {
            const int z = 64 * w + __ffsll((long long)y) - 1;
            rdm_add_two(R, alpha ? 0 : 2, o0, z, o1, z, contr);
        }
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t y = same[w]; y; y &= y - 1) {
            const int z = 64 * w + __ffsll((long long)y) - 1;
            if (alpha)
                rdm_add_two(R, 1, o0, z, o1, z, contr);
            else
                rdm_add_two(R, 1, z, o0, z, o1, contr);
        }
}

// fill_two_dense (CIDens.cpp:756-779): a same-spin double
template <int W>
__device__ void fill_double_same(const RdmAcc &R, const uint64_t *s1, const uint64_t *s2, double contr, int spin) {
    uint64_t x[W], c[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
        x[w] = s1[w] ^ s2[w];
        c[w] = s1[w] & s2[w];
    }
    int o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = pop_lowest<W>(x);
    int a0, a1, b0, b1;
    arrange4<W>(o, s1, a0, a1, b0, b1);
    const int diff = nstacked<W>(a0, a1, c) + nstacked<W>(b0, b1, c);
    rdm_add_two(R, spin, a0, a1, b0, b1, negate_if(contr, diff & 1));
}

// fill_two_dense_upanddown (CIDens.cpp:781-806): an alpha-beta double
template <int W>
__device__ void fill_double_ab(const RdmAcc &R, const uint64_t *u1, const uint64_t *u2, const uint64_t *d1,
                               const uint64_t *d2, double contr) {
    uint64_t xu[W], cu[W], xd[W], cd[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
        xu[w] = u1[w] ^ u2[w];
        cu[w] = u1[w] & u2[w];
        xd[w] = d1[w] ^ d2[w];
        cd[w] = d1[w] & d2[w];
    }
    int a0 = pop_lowest<W>(xu), a1 = pop_lowest<W>(xu);
    if (!has_bit<W>(u1, a0)) {
        const int t = a0;
        a0 = a1;
        a1 = t;
    }
    int b0 = pop_lowest<W>(xd), b1 = pop_lowest<W>(xd);
    if (!has_bit<W>(d1, b0)) {
        const int t = b0;
        b0 = b1;
        b1 = t;
    }
    const int diff = nstacked<W>(a0, a1, cu) + nstacked<W>(b0, b1, cd);
    rdm_add_two(R, 1, a0, b0, a1, b1, negate_if(contr, diff & 1));
}

// fill_diagonal (CIDens.cpp:808-853)
template <int W>
__device__ void fill_diag(const RdmAcc &R, const uint64_t *up, const uint64_t *dn, double contr) {
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t y = up[w]; y; y &= y - 1) rdm_add_one(R, 0, 64 * w + __ffsll((long long)y) - 1, 64 * w + __ffsll((long long)y) - 1, contr);
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t y = dn[w]; y; y &= y - 1) rdm_add_one(R, 1, 64 * w + __ffsll((long long)y) - 1, 64 * w + __ffsll((long long)y) - 1, contr);
    if (!R.two) return;
    for (int spin = 0; spin < 2; ++spin) {
        const uint64_t *s = spin == 0 ? up : dn;
#pragma unroll
        for (int w = 0; w < W; ++w)
            for (uint64_t y = s[w]; y; y &= y - 1) {
                const int i = 64 * w + __ffsll((long long)y) - 1;
                // partners j > i
#pragma unroll
                for (int w2 = 0; w2 < W; ++w2) {
                    uint64_t y2 = s[w2];
                    if (w2 == w) y2 &= y & (y - 1);  // bits above i in the same word
                    else if (w2 < w) y2 = 0;
                    for (; y2; y2 &= y2 - 1) {
                        const int j = 64 * w2 + __ffsll((long long)y2) - 1;
                        rdm_add_two(R, spin == 0 ? 0 : 2, i, j, i, j, contr);
                    }
                }
            }
    }
#pragma unroll
    for (int w = 0; w < W; ++w)
        for (uint64_t y = up[w]; y; y &= y - 1) {
            const int i = 64 * w + __ffsll((long long)y) - 1;
#pragma unroll
            for (int w2 = 0; w2 < W; ++w2)
                for (uint64_t y2 = dn[w2]; y2; y2 &= y2 - 1) {
                    const int j = 64 * w2 + __ffsll((long long)y2) - 1;
                    rdm_add_two(R, 1, i, j, i, j, contr);
                }
        }
}

template <int W>
__global__ void __launch_bounds__(32 * kDetWarps) k_dets_rdm(DetParams p, const double *__restrict__ c, RdmAcc R) {
    __shared__ uint64_t tile[kDetTile * 2 * W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int64_t r0 = (int64_t)blockIdx.x * kDetWarps; r0 < p.n; r0 += (int64_t)gridDim.x * kDetWarps) {
        const int64_t i = r0 + warp;
        const bool active = i < p.n;
        uint64_t ui[W], di[W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            ui[w] = active ? p.dets[i * 2 * W + w] : 0;
            di[w] = active ? p.dets[i * 2 * W + W + w] : 0;
        }
        const double ci = active ? c[i] : 0.0;
        // columns j >= i: tiles from the one holding i
        for (int64_t base = (r0 / kDetTile) * kDetTile; base < p.n; base += kDetTile) {
            const int tn = (int)(p.n - base < kDetTile ? p.n - base : kDetTile);
            __syncthreads();
            for (int t = threadIdx.x; t < tn * 2 * W; t += blockDim.x) tile[t] = p.dets[base * 2 * W + t];
            __syncthreads();
            if (!active) continue;
            for (int jj = lane; jj < tn; jj += 32) {
                const int64_t j = base + jj;
                if (j < i) continue;
                const uint64_t *uj = tile + jj * 2 * W, *dj = uj + W;
                int nu = 0, nd = 0;
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    nu += __popcll(ui[w] ^ uj[w]);
                    nd += __popcll(di[w] ^ dj[w]);
                }
                if (nu + nd > 4) continue;
                const double contr = ci * c[j];
                // fill_density_matrix_one / fill_density_matrix (CIDens.cpp:855-896)
                if (nu == 0 && nd == 0) fill_diag<W>(R, ui, di, contr);
                else if (nu == 2 && nd == 0) fill_single<W>(R, ui, uj, di, contr, true);
                else if (nu == 0 && nd == 2) fill_single<W>(R, di, dj, ui, contr, false);
                else if (R.two && nu == 4 && nd == 0) fill_double_same<W>(R, ui, uj, contr, 0);
                else if (R.two && nu == 0 && nd == 4) fill_double_same<W>(R, di, dj, contr, 2);
                else if (R.two && nu == 2 && nd == 2) fill_double_ab<W>(R, ui, uj, di, dj, contr);
            }
        }
    }
}

// Expands the (min, max) fixed-point storage into the full symmetric output arrays.
__global__ void k_rdm_expand(RdmAcc R, double *rdm1, double *aa, double *ab, double *bb) {
    const int L = R.L, np = R.np;
    const int64_t L2 = (int64_t)L * L, n1 = 2 * L2, n2 = (int64_t)np * np, n3 = L2 * L2;
    const int64_t total = n1 + (R.two ? 2 * n2 + n3 : 0);
    auto val = [](unsigned long long q) { return (double)(long long)q * 0x1p-60; };
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        if (t < n1) {
            const int64_t s = t / L2, ij = t - s * L2;
            const int i = (int)(ij / L), j = (int)(ij - (int64_t)i * L);
            rdm1[t] = val(R.one[(s * L + min(i, j)) * L + max(i, j)]);
        } else if (t < n1 + 2 * n2) {
            const int64_t u = t - n1, which = u / n2, ij = u - which * n2;
            const int64_t i = ij / np, j = ij - i * np;
            const unsigned long long *X = which == 0 ? R.aa : R.bb;
            (which == 0 ? aa : bb)[ij] = val(X[min(i, j) * np + max(i, j)]);
        } else {
            const int64_t ij = t - n1 - 2 * n2, i = ij / L2, j = ij - i * L2;
            ab[ij] = val(R.ab[min(i, j) * L2 + max(i, j)]);
        }
    }
}

}  // namespace

void dets_rdm(cigpu_crs &c, const double *c_dev, double *rdm1, double *aa, double *ab, double *bb, cudaStream_t s) {
    const int L = c.L, np = L * (L - 1) / 2;
    const int64_t L2 = (int64_t)L * L, n1 = 2 * L2, n2 = (int64_t)np * np, n3 = L2 * L2;
    const bool two = aa && ab && bb;
    DevBuf<unsigned long long> acc(n1 + (two ? 2 * n2 + n3 : 0));
    CIGPU_CUDA(cudaMemsetAsync(acc.p, 0, acc.bytes(), s));
    RdmAcc R{acc.p, two ? acc.p + n1 : nullptr, two ? acc.p + n1 + 2 * n2 : nullptr, two ? acc.p + n1 + n2 : nullptr,
             L, np, two};
    DetParams p = params_of(c);
    if (c.det_words == 1)
        k_dets_rdm<1><<<rows_grid(c.dim), 32 * kDetWarps, 0, s>>>(p, c_dev, R);
    else
        k_dets_rdm<2><<<rows_grid(c.dim), 32 * kDetWarps, 0, s>>>(p, c_dev, R);
    CIGPU_CUDA(cudaGetLastError());
    DevBuf<double> out(n1 + (two ? 2 * n2 + n3 : 0));
    double *o1 = out.p, *oaa = two ? out.p + n1 : nullptr, *obb = two ? out.p + n1 + n2 : nullptr,
           *oab = two ? out.p + n1 + 2 * n2 : nullptr;
    const int64_t total = (int64_t)out.n;
    k_rdm_expand<<<(int)std::min<int64_t>((total + 255) / 256, (int64_t)sm_count() * 8), 256, 0, s>>>(R, o1, oaa, oab, obb);
    CIGPU_CUDA(cudaGetLastError());
    count_launch(2);
    if (rdm1) CIGPU_CUDA(cudaMemcpyAsync(rdm1, o1, sizeof(double) * n1, cudaMemcpyDeviceToHost, s));
    if (two) {
        CIGPU_CUDA(cudaMemcpyAsync(aa, oaa, sizeof(double) * n2, cudaMemcpyDeviceToHost, s));
        CIGPU_CUDA(cudaMemcpyAsync(bb, obb, sizeof(double) * n2, cudaMemcpyDeviceToHost, s));
        CIGPU_CUDA(cudaMemcpyAsync(ab, oab, sizeof(double) * n3, cudaMemcpyDeviceToHost, s));
    }
    CIGPU_CUDA(cudaStreamSynchronize(s));
}

void dets_mv64(cigpu_crs &c, const double *x, double *y, cudaStream_t s) {
    DetParams p = params_of(c);
    // the stored leading block first (rows and columns below det_block), then every
    // pair outside it recomputed (CI_Big::mvprod, CIMethod.cpp:943-984)
    if (c.det_block > 0) spmv_f64(c.det_block, c.nnz_full, c.row_ptr.p, c.col.p, c.val64.p, x, y, s);
    if (c.det_block < c.dim) matvec(p, c.det_words, x, y, s);  // nothing outside a whole-list block
}

}  // namespace cigpu

using namespace cigpu;

extern "C" {

int cigpu_dets_read(const char *path, int words, int64_t capacity, uint64_t *up, uint64_t *down, int64_t *ndet,
                    int *max_orbitals) {
    if (!path || !ndet || (words != 1 && words != 2) || capacity < 0) return CIGPU_EINVAL;
    std::ifstream f(path);
    if (!f.is_open()) return CIGPU_ENOTFOUND;
    std::string line;
    int64_t n = 0;
    int maxb = 0;
    uint64_t u[2], d[2];
    while (std::getline(f, line)) {
        if (line.find('#') != std::string::npos) continue;  // Permutator_File::read_file skips comment lines
        if (line.find_first_not_of(" \t\r") == std::string::npos) continue;
        int nb = 0;
        if (!parse_line(line, words, u, d, &nb)) return CIGPU_EINVAL;
        maxb = std::max(maxb, nb);
        if (up && down && n < capacity) {
            for (int w = 0; w < words; ++w) {
                up[n * words + w] = u[w];
                down[n * words + w] = d[w];
            }
        }
        ++n;
    }
    *ndet = n;
    if (max_orbitals) *max_orbitals = maxb;
    return (up && down && n > capacity) ? CIGPU_ENOMEM : CIGPU_OK;
}

}  // extern "C"

namespace cigpu {
namespace {

// keep: the leading determinants whose block of the matrix is stored (all of them
// for CRS storage; 0 for CI_Big without a stored part)
int build_dets(cigpu_ham *ham, int64_t ndet, int words, const uint64_t *up, const uint64_t *down, int storage,
               int precision, int64_t keep, cigpu_stream stream, cigpu_crs **out) {
    if (!ham || !up || !down || !out) return CIGPU_EINVAL;
    *out = nullptr;
    if (ndet < 1 || ndet > (int64_t)UINT32_MAX || (words != 1 && words != 2)) return CIGPU_EINVAL;
    if (storage != CIGPU_DETS_CRS && storage != CIGPU_DETS_ONTHEFLY) return CIGPU_EINVAL;
    if (precision != CIGPU_FP64 && precision != CIGPU_MIXED) return CIGPU_EINVAL;
    if (storage == CIGPU_DETS_ONTHEFLY && precision != CIGPU_FP64) return CIGPU_ENOTSUP;
    if (keep < 0 || keep > ndet) return CIGPU_EINVAL;
    const int W = ham->L <= 64 ? 1 : 2;
    if (words < W) return CIGPU_EINVAL;
    // every determinant: nup / ndown electrons inside the L orbitals (the reference
    // takes the counts from the Hamiltonian and assumes them)
    std::vector<uint64_t> rec((size_t)ndet * 2 * W, 0);
    for (int64_t i = 0; i < ndet; ++i) {
        int cu = 0, cd = 0;
        for (int w = 0; w < words; ++w) {
            const uint64_t u = up[i * words + w], d = down[i * words + w];
            const int lo = 64 * w;
            const uint64_t valid = ham->L - lo >= 64 ? ~(uint64_t)0 : (ham->L - lo <= 0 ? 0 : (((uint64_t)1 << (ham->L - lo)) - 1));
            if ((u & ~valid) || (d & ~valid)) return CIGPU_EINVAL;
            cu += __builtin_popcountll(u);
            cd += __builtin_popcountll(d);
            if (w < W) {
                rec[(size_t)i * 2 * W + w] = u;
                rec[(size_t)i * 2 * W + W + w] = d;
            }
        }
        if (cu != ham->nup || cd != ham->ndown) return CIGPU_EINVAL;
    }
    CIGPU_TRY
    std::unique_ptr<cigpu_crs> c(new cigpu_crs);
    c->ham = ham;
    c->method = CIGPU_DETS;
    c->precision = precision;
    c->L = ham->L;
    c->nup = ham->nup;
    c->ndown = ham->ndown;
    c->dim = ndet;
    c->det_words = W;
    c->onthefly = storage == CIGPU_DETS_ONTHEFLY;
    c->det_block = c->onthefly ? keep : ndet;
    CIGPU_CUDA(cudaGetDevice(&c->device));
    if (stream) {
        c->stream = static_cast<cudaStream_t>(stream);
    } else {
        CIGPU_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
        c->own_stream = true;
    }
    cudaStream_t s = c->stream;
    StreamScope scope(s);
    const auto t0 = std::chrono::steady_clock::now();
    c->dets.alloc(rec.size());
    CIGPU_CUDA(cudaMemcpyAsync(c->dets.p, rec.data(), rec.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
    c->diag.alloc(ndet);
    DetParams p = params_of(*c);
    {
        const int g = (int)std::max<int64_t>(1, std::min<int64_t>((ndet + 255) / 256, (int64_t)sm_count() * 8));
        if (W == 1)
            k_dets_diag<1><<<g, 256, 0, s>>>(p, c->diag.p);
        else
            k_dets_diag<2><<<g, 256, 0, s>>>(p, c->diag.p);
        CIGPU_CUDA(cudaGetLastError());
        count_launch();
    }
    if (c->det_block > 0) {
        // the stored rows: the whole matrix (CRS storage) or the leading block of CI_Big
        const int64_t nb = c->det_block;
        p.nrows = nb;
        p.block = nb;
        p.group = build_group(nb);
        // the sums that start at zero in one block: elements below the diagonal (64 bits),
        // vanished elements, each row's count
        DevBuf<uint32_t> sums((size_t)nb + 4), segs((size_t)nb * kSegs);
        unsigned long long *const lower = reinterpret_cast<unsigned long long *>(sums.p);
        uint32_t *const dropped = sums.p + 2, *const count = sums.p + 4;
        c->upper_off.alloc(nb);
        c->row_ptr.alloc(nb + 1);
        p.row_count = count;
        p.dropped = dropped;
        p.upper_off = c->upper_off.p;
        p.seg_count = segs.p;
        p.row_ptr = c->row_ptr.p;
        // structure: the row structure is the connected pairs (see k_dets_pairs)
        auto passes = [&](bool structure) {
            DevBuf<uint32_t> masks;
            const size_t words = (size_t)((nb + 31) / 32), groups = (size_t)((nb + p.group - 1) / p.group);
            if (structure && groups * words * 32 * sizeof(uint32_t) <= kMaskBytes) {
                try {
                    masks.alloc(groups * words * 32);
                } catch (const std::bad_alloc &) {  // the fill scans again
                }
            }
            p.masks = masks.p;
            CIGPU_CUDA(cudaMemsetAsync(sums.p, 0, sums.bytes(), s));
            CIGPU_CUDA(cudaMemsetAsync(c->upper_off.p, 0, c->upper_off.bytes(), s));
            if (structure)
                pairs<kDetCount>(p, W, s);
            else
                rows<kDetCount>(p, W, s);
            exclusive_scan_u32(count, c->row_ptr.p, nb, s);
            k_sum_u32<<<(int)std::min<int64_t>((nb + 255) / 256, 1024), 256, 0, s>>>(c->upper_off.p, nb, lower);
            CIGPU_CUDA(cudaGetLastError());
            count_launch();
            int64_t nnz = 0;
            unsigned long long nlow = 0;
            CIGPU_CUDA(cudaMemcpyAsync(&nnz, c->row_ptr.p + nb, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
            CIGPU_CUDA(cudaMemcpyAsync(&nlow, lower, sizeof(nlow), cudaMemcpyDeviceToHost, s));
            CIGPU_CUDA(cudaStreamSynchronize(s));
            c->nnz_full = nnz;
            c->nnz_upper = nnz - (int64_t)nlow;
            const auto storage = [&] {
                const size_t n = (size_t)std::max<int64_t>(nnz, 1);
                c->col.alloc(n);
                if (precision == CIGPU_FP64) {
                    c->val64.alloc(n);
                } else {
                    c->val32.alloc(n);
                    c->val32lo.alloc(n);
                }
            };
            try {
                storage();
            } catch (const std::bad_alloc &) {  // without the masks' memory held beside it
                if (!masks.p) throw;
                masks.release();
                p.masks = nullptr;
                storage();
            }
            p.col = c->col.p;
            p.val64 = c->val64.p;
            p.val32 = c->val32.p;
            p.val32lo = c->val32lo.p;
            if (structure && precision == CIGPU_FP64)
                pairs<kDetFill64>(p, W, s);
            else if (structure)
                pairs<kDetFill32>(p, W, s);
            else if (precision == CIGPU_FP64)
                rows<kDetFill64>(p, W, s);
            else
                rows<kDetFill32>(p, W, s);
            if (!structure) return true;
            uint32_t d = 0;
            CIGPU_CUDA(cudaMemcpyAsync(&d, dropped, sizeof(d), cudaMemcpyDeviceToHost, s));
            CIGPU_CUDA(cudaStreamSynchronize(s));
            return d == 0;
        };
        if (ham->eri_zero || nb < kShortList || !passes(true)) passes(false);
    }
    CIGPU_CUDA(cudaStreamSynchronize(s));
    c->build_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    *out = c.release();
    return CIGPU_OK;
    CIGPU_CATCH
}

}  // namespace
}  // namespace cigpu

extern "C" {

int cigpu_build_dets(cigpu_ham *ham, int64_t ndet, int words, const uint64_t *up, const uint64_t *down, int storage,
                     int precision, cigpu_stream stream, cigpu_crs **out) {
    return build_dets(ham, ndet, words, up, down, storage, precision, storage == CIGPU_DETS_CRS ? ndet : 0, stream,
                      out);
}

int cigpu_build_dets_partial(cigpu_ham *ham, int64_t ndet, int words, const uint64_t *up, const uint64_t *down,
                             int64_t keep, cigpu_stream stream, cigpu_crs **out) {
    return build_dets(ham, ndet, words, up, down, CIGPU_DETS_ONTHEFLY, CIGPU_FP64, keep, stream, out);
}

}  // extern "C"
