// Matrix-free DOCI matvec: y = H x over the seniority-zero pair space without a
// stored matrix. k_doci_mv, the general kernel, forms every hop's rank; larger spaces
// take k_doci_split (below).
//
// Replaces SparseMatrix_CRS_Sym::mvprod (SparseMatrix_CRS.cpp:700-723) on the DOCI
// matrix of DOCI::construct_CI_matrix (CIMethod.cpp:611-660). Every off-diagonal
// element of that matrix is a pair hop: row I (pair string S) couples to
// J = S - j + k (j occupied, k empty) with the value K_jk = <jj|kk> = (jk|jk),
// which depends on the two orbitals only (the phase of a pair hop is even), and
// elements with |K_jk| <= 1e-14 are not stored. So a row is generated from its
// string, the L x L table K (shared memory) and the string's rank prefixes:
//
//   y_I = H_II x_I + sum_{j in S, k not in S} K_jk x_J.
//
// The rank of J costs O(1). With p_1 < ... < p_n the occupied orbitals of S and
// rank(S) = sum_m C(p_m, m) (colex, CIMethod.cpp:689-747), j = p_{a+1} and b the
// number of occupied orbitals below k:
//   k > j:  rank(J) = I - C(j, a+1) + (P_b - P_{a+1}) + C(k, b),
//           P_m = sum_{i <= m} (C(p_i, i-1) - C(p_i, i))
//   k < j:  rank(J) = I - C(j, a+1) + C(k, b+1) + (Q_a - Q_b),
//           Q_m = sum_{i <= m} (C(p_i, i+1) - C(p_i, i))
// (the electrons between j and k shift one place), evaluated modulo 2^32: the
// result is a rank below 2^32, so the wrap cancels.
//
// A group of 8-32 lanes per row (about 16 hops per lane). The group writes the
// row's occupied / empty orbital lists and the prefixes (a scan over the group) to
// shared memory, then takes the n (L - n) hops in rounds of up to 8 per lane:
// ranks first, then the round's gathers of x together (L2-resident: 2.7 M FP32
// entries are 10.8 MB at L=24), then one multiply-add each, all lanes on the same
// instruction stream (an FP64
// multiply-add issued for part of a warp would occupy GB300's FP64 pipe for the
// whole warp). The group's sums meet in a fixed shuffle tree and the diagonal term
// is added last, so the order is fixed (bit-reproducible run to run).
//
// Bytes per matvec: the pair strings (8 per row), the diagonal and x read once, y
// written once; the hop gathers hit x in L2. The matrix the CRS form streams
// (145 elements per row at L=24, 12 bytes each in FP64) is not stored at all.
#include "doci_mv.cuh"

#include <algorithm>

namespace cigpu {

namespace {

constexpr int kMvThreads = 256;
constexpr int kMvWarps = kMvThreads / 32;
constexpr int kBW = 34;  // binomial table row: C(nn, kk) for kk <= 33 (n <= 32)

struct RowScratch {
    uint8_t occ[32];
    uint8_t emp[64];
    uint32_t P[33], Q[33];
};

// Hops a lane takes per round: their ranks are formed first and their x gathers
// issued together, so each lane keeps up to kHopBatch L2 loads in flight.
constexpr int kHopBatch = 8;

// G lanes per row, 32 / G rows per warp. Every row of a space has the same n (L - n)
// hops, so the rounds are the same for every group of the warp: no lane runs a
// round that is empty for it except in the last one. Fewer lanes per row mean
// fewer steps in the lanes' final sum (on GB300's FP64 pipe a shuffle-add of the
// FP64 form costs as much as a round of hops).
template <typename T, int G>
__global__ void __launch_bounds__(kMvThreads) k_doci_mv(const DociMv p, const T *__restrict__ K,
                                                        const T *__restrict__ diag, const T *__restrict__ x,
                                                        T *__restrict__ y) {
    constexpr int R = 32 / G;  // rows per warp
    constexpr int kChunk = 32 / G;  // prefix entries per lane (n <= 32)
    __shared__ uint32_t binom[64 * kBW];  // C(nn, kk) mod 2^32
    __shared__ RowScratch rs[kMvWarps][R];
    extern __shared__ __align__(16) unsigned char smem[];
    T *Ks = reinterpret_cast<T *>(smem);  // K[j * L + k]
    const int L = p.L, n = p.n, nv = L - n;
    for (int i = threadIdx.x; i < 64 * kBW; i += blockDim.x) {
        const int nn = i / kBW, kk = i % kBW;
        binom[i] = (nn <= L && kk <= n + 1) ? (uint32_t)d_binom(nn, kk) : 0u;
    }
    for (int i = threadIdx.x; i < L * L; i += blockDim.x) Ks[i] = K[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = lane / G, gl = lane % G;
    RowScratch &w = rs[warp][grp];
    const int nh = n * nv;
    // h / nv as umulhi(h, ceil(2^32 / nv)): exact for h < 4096 and nv < 64 (nh <= 992)
    const uint32_t inv_nv = nv > 0 ? (uint32_t)((0x100000000ull + nv - 1) / nv) : 0u;
    const int64_t rows_per_pass = (int64_t)gridDim.x * kMvWarps * R;
    for (int64_t r0 = ((int64_t)blockIdx.x * kMvWarps + warp) * R; r0 < p.D; r0 += rows_per_pass) {
        const int64_t r = r0 + grp;
        const bool live = r < p.D;
        const uint64_t s = live ? __ldg(p.strings + r) : 0;
        // occupied / empty lists
        if (live)
            for (int i = gl; i < L; i += G) {
                const int below = __popcll(s & ((((uint64_t)1) << i) - 1));
                if ((s >> i) & 1)
                    w.occ[below] = (uint8_t)i;
                else
                    w.emp[i - below] = (uint8_t)i;
            }
        __syncwarp();
        // rank prefixes over the occupied orbitals: lane gl owns indices
        // gl * kChunk .. gl * kChunk + kChunk - 1 (0-based m holds p_{m+1})
        uint32_t dP[kChunk], dQ[kChunk], sP = 0, sQ = 0;
#pragma unroll
        for (int c = 0; c < kChunk; ++c) {
            const int m = gl * kChunk + c;
            uint32_t a = 0, b = 0;
            if (live && m < n) {
                const int pm = w.occ[m];
                a = binom[pm * kBW + m] - binom[pm * kBW + m + 1];
                b = binom[pm * kBW + m + 2] - binom[pm * kBW + m + 1];
            }
            sP += a;
            sQ += b;
            dP[c] = sP;
            dQ[c] = sQ;
        }
        uint32_t eP = sP, eQ = sQ;  // inclusive scan of the chunk sums over the group
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const uint32_t uP = __shfl_up_sync(0xffffffffu, eP, o, G), uQ = __shfl_up_sync(0xffffffffu, eQ, o, G);
            if (gl >= o) {
                eP += uP;
                eQ += uQ;
            }
        }
        if (live) {
#pragma unroll
            for (int c = 0; c < kChunk; ++c) {
                const int m = gl * kChunk + c;
                if (m < n) {
                    w.P[m + 1] = eP - sP + dP[c];
                    w.Q[m + 1] = eQ - sQ + dQ[c];
                }
            }
            if (gl == 0) w.P[0] = w.Q[0] = 0;
        }
        __syncwarp();
        const uint32_t I = (uint32_t)r;
        T acc = 0;
        for (int h0 = 0; h0 < nh; h0 += G * kHopBatch) {
            const int nu = min(kHopBatch, (nh - h0 + G - 1) / G);  // the same for every group
            uint32_t J[kHopBatch];
            T kv[kHopBatch];
#pragma unroll
            for (int u = 0; u < kHopBatch; ++u) {
                if (u < nu) {
                    const int h = h0 + G * u + gl;
                    J[u] = 0xFFFFFFFFu;
                    kv[u] = 0;
                    if (live && h < nh) {
                        const int a = (int)__umulhi((uint32_t)h, inv_nv), bi = h - a * nv;
                        const int j = w.occ[a], k = w.emp[bi];
                        const int b = __popcll(s & ((((uint64_t)1) << k) - 1));
                        uint32_t t = I - binom[j * kBW + a + 1];
                        if (k > j)
                            t += w.P[b] - w.P[a + 1] + binom[k * kBW + b];
                        else
                            t += binom[k * kBW + b + 1] + w.Q[a] - w.Q[b];
                        J[u] = t;
                        kv[u] = Ks[j * L + k];
                    }
                }
            }
            T xv[kHopBatch];
#pragma unroll
            for (int u = 0; u < kHopBatch; ++u)
                if (u < nu) {
                    // 0xFFFFFFFF marks a lane without a hop this round; any other rank
                    // outside the space is a violation (skipped in every build)
                    bool ok = index_ok(J[u], (uint64_t)p.D);
                    if (J[u] != 0xFFFFFFFFu) ok = CIGPU_CHECK(p.err, ok, kCheckHopRank, J[u]) && ok;
                    xv[u] = ok ? __ldg(x + J[u]) : (T)0;
                }
#pragma unroll
            for (int u = 0; u < kHopBatch; ++u)
                if (u < nu) acc += kv[u] * xv[u];
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, G);
        if (live && gl == 0) y[r] = acc + __ldg(diag + r) * __ldg(x + r);
        __syncwarp();  // the scratch is rewritten by the next rows
    }
}

// ---------------------------------------------------------------------------
// The product by low and high orbitals (larger spaces).
//
// With the orbitals split into s low and L - s high ones, the strings of one high
// part h are a block of consecutive ranks, ordered by their low part l: x is a ragged
// matrix x(h, l). A pair hop between two high orbitals moves to another block at the
// same l, one between two low ones stays in the block, and one between a low and a
// high orbital takes l to a string of one pair less or more. So nothing of a hop's
// rank depends on the row as a whole:
//   * high - high: the lanes of a warp (consecutive l) read consecutive x of another
//     block; its start and K_jk are the same for all of them;
//   * low - low: the target in the block and the orbital pair come from a table over
//     l alone;
//   * low - high: the blocks h + k and h - k are staged in shared memory once and
//     gathered from there, with the target from a table over l and K from the row of
//     k (consecutive words over j: no bank conflict).
// A hop is two or three shared-memory reads and a multiply-add where the general
// kernel forms a rank (two popcounts' worth of lookups and selects, ~110 issue slots
// per 32 hops). What bounds it: in FP32 the shared-memory gathers, in FP64 the FP64
// pipe. Among other products: L=24, 12 pairs (2,704,156 rows, 144 hops): FP32 1,072 -> 203
// us, FP64 1.69 -> 0.74 ms (the FP64 pipe's share 0.62); L=20, 8 pairs (125,970): 54 -> 23
// us and 81 -> 39 us.
//
// A thread block takes `group` consecutive high strings of one sector (number of high
// pairs); a thread takes whole rows, in eight running sums (two per kind of hop) that
// meet in a fixed order.
// Threads per block (and rows it aims at): 256 in FP32, 512 in FP64, whose staged
// blocks leave room for two thread blocks per SM (L=24: 843 us with 256, 751 with 512;
// FP32 227 and 348 in the same measurement).
template <typename T>
__host__ __device__ constexpr int split_threads() {
    return sizeof(T) == 4 ? 256 : 512;
}
constexpr size_t kSplitMaxSmem = 112 * 1024;  // two FP64 blocks per SM
// The split product serves spaces of at least kSplitMinRows rows whose blocks hold at
// least kSplitMinBlock strings on average. Below, a block's preparation (neighbour
// starts, staging) shows: L=16 8 pairs, 12,870 rows, FP32 13.5 us against 11.5 of the
// general kernel, L=17 8 pairs, 24,310 rows, 14.5 against 20.6. Few pairs (or holes) in
// many orbitals make blocks of a string or two: L=40 4 pairs (3.8 a block) 77.9 against
// 63.7 us, L=30 26 pairs (6.8) 37.9 against 35.0, L=30 5 pairs (11.3) 51.4 against 74.9.
constexpr int64_t kSplitMinRows = 20000;
constexpr int64_t kSplitMinBlock = 10;

// Bytes of shared memory of one thread block (the kernel carves it in this order).
template <typename T>
__host__ __device__ inline size_t split_smem(int s, int Lh, const DociSector &c) {
    const size_t g = c.group[sizeof(T) == 8], nv = Lh - c.nh, nhh = (size_t)c.nh * nv;
    size_t b = sizeof(T) * ((size_t)s * s + g * (c.nlow + nv * c.nminus + c.nh * c.nplus + (size_t)Lh * s + nhh));
    b = (b + 7) & ~(size_t)7;
    return b + 8 * g + 4 * g * (nhh + 1 + Lh);
}

template <typename T>
__global__ void __launch_bounds__(split_threads<T>()) k_doci_split(const DociSplitView p, const T *__restrict__ K,
                                                              const T *__restrict__ diag, const T *__restrict__ x,
                                                              T *__restrict__ y) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NT = split_threads<T>(), kType = sizeof(T) == 8;
    const int s = p.s, Lh = p.L - p.s, L = p.L;
    int q = 0;
    while (q + 1 < p.nsec && blockIdx.x >= p.sec[q + 1].first_task[kType]) ++q;
    const DociSector &c = p.sec[q];
    const int nh = c.nh, nv = Lh - nh, m = c.m, nhh = nh * nv;
    const int nlow = (int)c.nlow, nminus = (int)c.nminus, nplus = (int)c.nplus;
    const int gmax = c.group[kType];
    const uint32_t h0 = (blockIdx.x - c.first_task[kType]) * (uint32_t)gmax;
    const int g = (int)min((uint32_t)gmax, c.nhigh - h0);
    T *Kll = reinterpret_cast<T *>(smem);          // [s * s]
    T *own = Kll + s * s;                          // [g][nlow]
    T *up = own + (size_t)gmax * nlow;             // [g][nv][nminus]: the blocks h + k
    T *dn = up + (size_t)gmax * nv * nminus;       // [g][nh][nplus]: the blocks h - k
    T *Kup = dn + (size_t)gmax * nh * nplus;       // [g][nv][s]: K of the staged blocks' k
    T *Kdn = Kup + (size_t)gmax * nv * s;          // [g][nh][s]
    T *Khh = Kdn + (size_t)gmax * nh * s;          // [g][nhh]
    uint64_t *hb = reinterpret_cast<uint64_t *>((reinterpret_cast<uintptr_t>(Khh + (size_t)gmax * nhh) + 7) & ~(uintptr_t)7);
    uint32_t *hhb = reinterpret_cast<uint32_t *>(hb + gmax);  // [g][nhh]: starts of the high-high targets
    uint32_t *rb = hhb + (size_t)gmax * nhh;                  // [g][1 + Lh]: starts of the block, h + k, h - k
    const int t = threadIdx.x;
    for (int i = t; i < g; i += NT) {
        hb[i] = __ldg(p.hbits + c.high0 + h0 + i);
        rb[i * (1 + Lh)] = __ldg(p.hbase + c.high0 + h0 + i);
    }
    for (int i = t; i < s * s; i += NT) Kll[i] = __ldg(K + (i / s) * L + i % s);
    __syncthreads();
    // start of the block with high string b and mm low pairs: the high pairs' part of
    // the rank
    auto start_of = [&](uint64_t b, int mm) {
        uint32_t r = 0;
        for (int k = mm + 1; b; b &= b - 1, ++k) r += __ldg(p.binom + (s + __ffsll((long long)b) - 1) * kSplitBinomRow + k);
        return r;
    };
    // the i-th set bit of b
    auto nth = [](uint64_t b, int i) {
        for (; i > 0; --i) b &= b - 1;
        return __ffsll((long long)b) - 1;
    };
    const uint64_t full = (((uint64_t)1) << Lh) - 1;
    for (int e = t; e < g * Lh; e += NT) {  // the low-high neighbours: nv of h + k, nh of h - k
        const int i = e / Lh, r = e - i * Lh;
        const bool add = r < nv;
        const int k = add ? nth(full & ~hb[i], r) : nth(hb[i], r - nv);
        const bool any = add ? m > 0 : m < s;
        rb[i * (1 + Lh) + 1 + r] = any ? start_of(hb[i] ^ ((uint64_t)1 << k), add ? m - 1 : m + 1) : 0u;
        T *Kr = add ? Kup + ((size_t)i * nv + r) * s : Kdn + ((size_t)i * nh + r - nv) * s;
        for (int j = 0; j < s; ++j) Kr[j] = __ldg(K + (s + k) * L + j);
    }
    for (int e = t; e < g * nhh; e += NT) {
        const int i = e / nhh, r = e - i * nhh, a = r / nv;
        const int j = nth(hb[i], a), k = nth(full & ~hb[i], r - a * nv);
        hhb[e] = start_of(hb[i] ^ ((uint64_t)1 << j) ^ ((uint64_t)1 << k), m);
        Khh[e] = __ldg(K + (s + j) * L + s + k);
    }
    __syncthreads();
    auto stage = [&](T *dst, const uint32_t *starts, int rows, int per, int len) {
        // rows = g * per blocks of len entries; row r starts at starts[(r / per) * (1 + Lh) + r % per]
        const int warp = t >> 5, lane = t & 31;
        if (len < 32) {
            for (int e = t; e < rows * len; e += NT) {
                const int r = e / len;
                const uint32_t at = starts[(r / per) * (1 + Lh) + r % per] + (uint32_t)(e - r * len);
                dst[e] = CIGPU_CHECK(p.err, index_ok(at, (uint64_t)p.D), kCheckHopRank, at) ? __ldg(x + at) : (T)0;
            }
            return;
        }
        for (int r = warp; r < rows; r += NT / 32) {
            const uint32_t b = starts[(r / per) * (1 + Lh) + r % per];
            for (int l = lane; l < len; l += 32) {
                const uint32_t at = b + (uint32_t)l;
                dst[(size_t)r * len + l] =
                    CIGPU_CHECK(p.err, index_ok(at, (uint64_t)p.D), kCheckHopRank, at) ? __ldg(x + at) : (T)0;
            }
        }
    };
    stage(own, rb, g, 1, nlow);
    if (m > 0 && nv > 0) stage(up, rb + 1, g * nv, nv, nminus);
    if (m < s && nh > 0) stage(dn, rb + 1 + nv, g * nh, nh, nplus);
    __syncthreads();
    const uint32_t *ll = p.ll + c.ll0;
    const uint16_t *lm = p.lminus + c.minus0, *lp = p.lplus + c.plus0;
    const int nll = m * (s - m);
    for (int it = t; it < g * nlow; it += NT) {
        const int i = it / nlow, l = it - i * nlow;
        const T *ow = own + (size_t)i * nlow;
        T a0 = 0, a1 = 0, b0 = 0, b1 = 0, c0 = 0, c1 = 0, d0 = 0, d1 = 0;
        {
            const uint32_t *hs = hhb + (size_t)i * nhh;
            const T *hk = Khh + (size_t)i * nhh;
            int e = 0;
            for (; e + 4 <= nhh; e += 4) {  // four loads in flight
                T v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t at = hs[e + u] + (uint32_t)l;
                    v[u] = CIGPU_CHECK(p.err, index_ok(at, (uint64_t)p.D), kCheckHopRank, at) ? __ldg(x + at) : (T)0;
                }
                a0 += hk[e] * v[0];
                a1 += hk[e + 1] * v[1];
                a0 += hk[e + 2] * v[2];
                a1 += hk[e + 3] * v[3];
            }
            for (; e < nhh; ++e) {
                const uint32_t at = hs[e] + (uint32_t)l;
                a0 += hk[e] * (CIGPU_CHECK(p.err, index_ok(at, (uint64_t)p.D), kCheckHopRank, at) ? __ldg(x + at) : (T)0);
            }
        }
        {
            int e = 0;
            for (; e + 4 <= nll; e += 4) {
                uint32_t w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) w[u] = __ldg(ll + (size_t)(e + u) * nlow + l);
                b0 += Kll[w[0] >> 10] * ow[w[0] & 1023u];
                b1 += Kll[w[1] >> 10] * ow[w[1] & 1023u];
                b0 += Kll[w[2] >> 10] * ow[w[2] & 1023u];
                b1 += Kll[w[3] >> 10] * ow[w[3] & 1023u];
            }
            for (; e < nll; ++e) {
                const uint32_t w = __ldg(ll + (size_t)e * nlow + l);
                b0 += Kll[w >> 10] * ow[w & 1023u];
            }
        }
        if (nv > 0)
            for (int e = 0; e < m; ++e) {
                const uint32_t w = __ldg(lm + (size_t)e * nlow + l);
                const T *xr = up + (size_t)i * nv * nminus + (w & 1023u), *kr = Kup + (size_t)i * nv * s + (w >> 10);
                int r = 0;
                for (; r + 2 <= nv; r += 2) {
                    c0 += kr[0] * xr[0];
                    c1 += kr[s] * xr[nminus];
                    kr += 2 * s;
                    xr += 2 * nminus;
                }
                if (r < nv) c0 += kr[0] * xr[0];
            }
        if (nh > 0)
            for (int e = 0; e < s - m; ++e) {
                const uint32_t w = __ldg(lp + (size_t)e * nlow + l);
                const T *xr = dn + (size_t)i * nh * nplus + (w & 1023u), *kr = Kdn + (size_t)i * nh * s + (w >> 10);
                int r = 0;
                for (; r + 2 <= nh; r += 2) {
                    d0 += kr[0] * xr[0];
                    d1 += kr[s] * xr[nplus];
                    kr += 2 * s;
                    xr += 2 * nplus;
                }
                if (r < nh) d0 += kr[0] * xr[0];
            }
        const uint32_t row = rb[i * (1 + Lh)] + (uint32_t)l;
        y[row] = ((a0 + a1) + (b0 + b1)) + ((c0 + c1) + (d0 + d1)) + __ldg(diag + row) * ow[l];
    }
}

// The plan's tables, one launch on the build's stream and no wait: with a copy of the
// binomials from the host, two launches that read them from memory and a wait, the plan was
// a third of a small space's build (L=18 9 pairs, mixed build 107 us without it, 144 so, 116
// now).
__device__ __forceinline__ uint32_t low_rank(uint32_t b, const uint32_t *binom) {
    uint32_t r = 0;
    for (int k = 1; b; b &= b - 1, ++k) r += binom[(__ffs((int)b) - 1) * kSplitBinomRow + k];
    return r;
}

// b without bit j, the bits above it one place down.
__device__ __forceinline__ uint32_t squeeze(uint32_t b, int j) {
    const uint32_t low = (1u << j) - 1u;
    return (b & low) | ((b >> 1) & ~low);
}

struct SplitBinom {
    uint32_t c[64 * kSplitBinomRow];  // C(p, k) mod 2^32, 0 past the space's orbitals and pairs
};
struct SplitTables {  // what the launch writes, in DociSplit's block
    uint64_t *hbits;
    uint32_t *hbase, *binom, *ll, *one, *two;
    uint16_t *lminus, *lplus, *lowbits;
};

constexpr int kSplitThreads = 256;
constexpr int kSplitLowBlocks = 16, kSplitHighBlocks = 32;  // per sector

// Blocks of sector blockIdx.y: a thread per low string (by m pairs) and orbital, or per high
// string.
__global__ void __launch_bounds__(kSplitThreads)
    k_split_tables(const __grid_constant__ DociSplitView p, const __grid_constant__ SplitBinom table, const SplitTables out) {
    __shared__ uint32_t binom[64 * kSplitBinomRow];
    __shared__ uint16_t rank[1 << kSplitMaxLow];  // of every low string among those of its size
    const DociSector &c = p.sec[blockIdx.y];
    const int s = p.s, m = c.m;
    const bool low = blockIdx.x < kSplitLowBlocks;
    const int used = (low ? s + 1 : p.L + 1) * kSplitBinomRow;
    for (int i = threadIdx.x; i < used; i += kSplitThreads) binom[i] = table.c[i];
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < 64 * kSplitBinomRow; i += kSplitThreads) out.binom[i] = table.c[i];
    __syncthreads();
    if (!low) {  // high strings and block starts
        const int Lh = p.L - s;
        for (uint32_t i = (blockIdx.x - kSplitLowBlocks) * kSplitThreads + threadIdx.x; i < c.nhigh;
             i += (gridDim.x - kSplitLowBlocks) * kSplitThreads) {
            uint64_t b = 0;
            uint32_t rest = i, r = 0;
            for (int k = c.nh, o = Lh - 1; k > 0; --o)
                if (binom[o * kSplitBinomRow + k] <= rest) {
                    rest -= binom[o * kSplitBinomRow + k];
                    b |= (uint64_t)1 << o;
                    r += binom[(s + o) * kSplitBinomRow + m + k];
                    --k;
                }
            out.hbits[c.high0 + i] = b;
            out.hbase[c.high0 + i] = r;
        }
        return;
    }
    for (int b = threadIdx.x; b < (1 << s); b += kSplitThreads) rank[b] = (uint16_t)low_rank((uint32_t)b, binom);
    __syncthreads();
    const uint32_t all = (1u << s) - 1u;
    for (uint32_t it = blockIdx.x * kSplitThreads + threadIdx.x; it < c.nlow * (uint32_t)s; it += kSplitLowBlocks * kSplitThreads) {
        const int j = (int)(it / c.nlow);
        const uint32_t l = it - (uint32_t)j * c.nlow;
        uint32_t b = 0, rest = l;  // the low string of rank l
        for (int k = m, o = s - 1; k > 0; --o)
            if (binom[o * kSplitBinomRow + k] <= rest) {
                rest -= binom[o * kSplitBinomRow + k];
                b |= 1u << o;
                --k;
            }
        if (j == 0) out.lowbits[c.low0 + l] = (uint16_t)b;
        // entries run down the orbitals: those of the orbitals above j come first
        const uint32_t above = all & ~((2u << j) - 1u), bj = b ^ (1u << j), at = rank[bj];
        const uint32_t held = __popc(b & above), empty = __popc(~b & above);
        if (!((b >> j) & 1u)) {
            out.lplus[c.plus0 + empty * c.nlow + l] = (uint16_t)(at | ((uint32_t)j << 10));
            continue;
        }
        out.lminus[c.minus0 + held * c.nlow + l] = (uint16_t)(at | ((uint32_t)j << 10));
        out.one[c.one0 + (uint32_t)j * c.n1 + rank[squeeze(bj, j)]] = l | (at << 16);
        uint32_t e = held * (uint32_t)(s - m);
        for (int k = s - 1; k >= 0; --k) {
            if ((b >> k) & 1u) continue;
            const uint32_t to = rank[bj ^ (1u << k)];
            out.ll[c.ll0 + e++ * c.nlow + l] = to | ((uint32_t)(j * s + k) << 10);
            if (k > j) {  // pair (j, k): row-major, j < k
                const uint32_t q = (uint32_t)(j * s - j * (j + 1) / 2 + k - j - 1);
                out.two[c.two0 + q * c.n2 + rank[squeeze(squeeze(bj, k), j)]] = l | (to << 16);
            }
        }
    }
}

template <typename T>
void launch_split(const DociSplit &sp, const T *K, const T *diag, const T *x, T *y, cudaStream_t s) {
    static SmemLimit limit;
    CIGPU_CUDA(limit.raise(k_doci_split<T>, kSplitMaxSmem));
    constexpr int kType = sizeof(T) == 8;
    DociSplitView v = sp.view;
    v.err = check_word_device();
    k_doci_split<T><<<v.tasks[kType], split_threads<T>(), sp.smem[kType], s>>>(v, K, diag, x, y);
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
}

// K_jk = (jk|jk) (chemist), zero where |v| <= 1e-14 and on the diagonal; FP64, and FP32
// where K32 is given.
__global__ void k_doci_pair_table(int L, const double *__restrict__ eri, double *__restrict__ K64,
                                  float *__restrict__ K32) {
    const int L1 = L;
    const int64_t L2 = (int64_t)L * L, L3 = L2 * L;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < L * L; t += gridDim.x * blockDim.x) {
        const int j = t / L, k = t % L;
        const int lo = j < k ? j : k, hi = j < k ? k : j;
        double v = (j == k) ? 0.0 : eri[lo * L3 + hi * L2 + lo * L1 + hi];
        if (!(v > kZero || v < -kZero)) v = 0.0;
        K64[t] = v;
        if (K32) K32[t] = (float)v;
    }
}

__global__ void k_count_nonzero(const double *__restrict__ v, int64_t n, unsigned long long *__restrict__ out) {
    unsigned long long c = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        c += (v[i] > kZero || v[i] < -kZero) ? 1 : 0;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

template <typename T, int G>
void launch_mv_g(const DociMv &p0, const T *K, const T *diag, const T *x, T *y, cudaStream_t s) {
    DociMv p = p0;
    p.err = check_word_device();
    const size_t sm = sizeof(T) * (size_t)p.L * p.L;
    static SmemLimit limit;  // L = 63: 31 KB of FP64 K
    CIGPU_CUDA(limit.raise(k_doci_mv<T, G>, 64 * 1024));
    constexpr int rows_per_block = kMvWarps * (32 / G);
    const int64_t blocks = std::min<int64_t>((p.D + rows_per_block - 1) / rows_per_block, (int64_t)sm_count() * 8);
    k_doci_mv<T, G><<<(unsigned)std::max<int64_t>(blocks, 1), kMvThreads, sm, s>>>(p, K, diag, x, y);
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
}

// Lanes per row from the hop count: about 16 hops per lane (at least 8 lanes).
template <typename T>
void launch_mv(const DociMv &p, const T *K, const T *diag, const T *x, T *y, cudaStream_t s) {
    const int nh = p.n * (p.L - p.n);
    if (nh > 384)
        launch_mv_g<T, 32>(p, K, diag, x, y, s);
    else if (nh > 192)
        launch_mv_g<T, 16>(p, K, diag, x, y, s);
    else
        launch_mv_g<T, 8>(p, K, diag, x, y, s);
}

}  // namespace

void doci_pair_table_launch(int L, const double *eri, double *K64, float *K32, cudaStream_t s) {
    k_doci_pair_table<<<(L * L + 255) / 256, 256, 0, s>>>(L, eri, K64, K32);
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
}

int64_t count_nonzero(const double *v, int64_t n, cudaStream_t s) {
    DevBuf<unsigned long long> out(1);
    CIGPU_CUDA(cudaMemsetAsync(out.p, 0, sizeof(unsigned long long), s));
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, (int64_t)sm_count() * 8);
    k_count_nonzero<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, s>>>(v, n, out.p);
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
    unsigned long long h = 0;
    CIGPU_CUDA(cudaMemcpyAsync(&h, out.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    CIGPU_CUDA(cudaStreamSynchronize(s));
    return (int64_t)h;
}

void doci_split_make(int L, int n, int64_t D, DociSplit &sp, cudaStream_t st) {
    sp.view = DociSplitView{};
    if (n < 1 || n >= L || D < kSplitMinRows) return;
    DociSplitView v{};
    v.L = L;
    v.n = n;
    v.D = D;
    uint32_t nll = 0, nmi = 0, npl = 0, nhi = 0, nlo = 0, none = 0, ntwo = 0;
    for (int s = std::min(kSplitMaxLow, (L + 1) / 2); s >= 4; --s) {
        const int Lh = L - s;
        size_t bytes[2] = {0, 0};
        uint64_t tasks[2] = {0, 0};
        nll = nmi = npl = nhi = nlo = none = ntwo = 0;
        v.nsec = 0;
        for (int m = std::max(0, n - Lh); m <= std::min(s, n); ++m) {
            DociSector c{};
            c.m = m;
            c.nh = n - m;
            c.nhigh = (uint32_t)d_binom(Lh, c.nh);
            c.nlow = (uint32_t)d_binom(s, m);
            c.nminus = m > 0 ? (uint32_t)d_binom(s, m - 1) : 0u;
            c.nplus = m < s ? (uint32_t)d_binom(s, m + 1) : 0u;
            for (int k = 0; k < 2; ++k) {
                const auto need = [&] { return k ? split_smem<double>(s, Lh, c) : split_smem<float>(s, Lh, c); };
                const uint32_t want = (uint32_t)(k ? split_threads<double>() : split_threads<float>()) / c.nlow;
                c.group[k] = (int)std::min({std::max(want, 1u), c.nhigh, 64u});
                while (c.group[k] > 1 && need() > kSplitMaxSmem / (k ? 1 : 2)) --c.group[k];
                c.first_task[k] = (uint32_t)tasks[k];
                tasks[k] += (c.nhigh + c.group[k] - 1) / c.group[k];
                bytes[k] = std::max(bytes[k], need());
            }
            c.high0 = nhi;
            c.ll0 = nll;
            c.minus0 = nmi;
            c.plus0 = npl;
            c.low0 = nlo;
            c.n1 = m > 0 ? (uint32_t)d_binom(s - 1, m - 1) : 0u;
            c.n2 = m > 0 && m < s ? (uint32_t)d_binom(s - 2, m - 1) : 0u;
            c.one0 = none;
            c.two0 = ntwo;
            nhi += c.nhigh;
            nlo += c.nlow;
            none += (uint32_t)s * c.n1;
            ntwo += (uint32_t)(s * (s - 1) / 2) * c.n2;
            nll += (uint32_t)(m * (s - m)) * c.nlow;
            nmi += (uint32_t)m * c.nlow;
            npl += (uint32_t)(s - m) * c.nlow;
            v.sec[v.nsec++] = c;
        }
        if (std::max(bytes[0], bytes[1]) <= kSplitMaxSmem && std::max(tasks[0], tasks[1]) <= (uint64_t)INT32_MAX) {
            v.s = s;
            for (int k = 0; k < 2; ++k) {
                v.tasks[k] = (uint32_t)tasks[k];
                sp.smem[k] = bytes[k];
            }
            break;
        }
    }
    if (v.s == 0 || (int64_t)nhi * kSplitMinBlock > D) return;
    SplitBinom table{};  // Pascal's triangle; p <= L and k <= n + 1 are read
    for (int p = 0; p <= L; ++p)
        for (int k = 0; k <= std::min(n + 1, p); ++k)
            table.c[p * kSplitBinomRow + k] =
                k == 0 ? 1u : table.c[(p - 1) * kSplitBinomRow + k - 1] + table.c[(p - 1) * kSplitBinomRow + k];
    // one block: an allocation and its release cost a build a microsecond or two each
    size_t words = 0;
    const auto place = [&](size_t n, size_t size) {  // each on 256 bytes, as an allocation
        const size_t at = words;
        words += (n * size + 255) / 256 * 32;
        return at;
    };
    const size_t at[] = {place(nhi, 8), place(nhi, 4),  place((size_t)64 * kSplitBinomRow, 4), place(nll, 4), place(none, 4),
                         place(ntwo, 4), place(nmi, 2), place(npl, 2), place(nlo, 2)};
    sp.tables.alloc(words);
    const auto u32 = [&](int i) { return reinterpret_cast<uint32_t *>(sp.tables.p + at[i]); };
    const auto u16 = [&](int i) { return reinterpret_cast<uint16_t *>(sp.tables.p + at[i]); };
    const SplitTables out{sp.tables.p + at[0], u32(1), u32(2), u32(3), u32(4), u32(5), u16(6), u16(7), u16(8)};
    sp.nlowbits = nlo;
    v.hbits = out.hbits;
    v.hbase = out.hbase;
    v.binom = out.binom;
    v.ll = out.ll;
    v.one = out.one;
    v.two = out.two;
    v.lminus = out.lminus;
    v.lplus = out.lplus;
    v.lowbits = out.lowbits;
    k_split_tables<<<dim3(kSplitLowBlocks + kSplitHighBlocks, v.nsec), kSplitThreads, 0, st>>>(v, table, out);
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
    sp.view = v;
}

void doci_mv64(const DociMv &p, const DociSplit &split, const double *K, const double *diag, const double *x,
               double *y, cudaStream_t s) {
    if (split)
        launch_split<double>(split, K, diag, x, y, s);
    else
        launch_mv<double>(p, K, diag, x, y, s);
}

void doci_mv32(const DociMv &p, const DociSplit &split, const float *K, const float *diag, const float *x, float *y,
               cudaStream_t s) {
    if (split)
        launch_split<float>(split, K, diag, x, y, s);
    else
        launch_mv<float>(p, K, diag, x, y, s);
}

}  // namespace cigpu
