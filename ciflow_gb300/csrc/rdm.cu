// 1- and 2-RDMs of a CI vector on the device.
//
// Replaces CIDens::construct_density with DensFCI / DensDOCI (CIDens.cpp:323-334,
// 1073-1224, 1530-1631). The reference loops over all determinant pairs and
// classifies each by popcount (O(dim^2)); here only connected pairs contribute. FCI sums
// have a fixed order (no atomics); DOCI sums are fixed-point integers collected by
// integer atomics, the same in any order. Both are bit-reproducible.
//
// FCI. Write C[Ia][Ib] for the CI vector. Every contribution of fill_density_matrix
// (CIDens.cpp:676-881) with a pair (I, J), I <= J in row order, is one of
//   * alpha pair (Ia, Ja >= Ia, same Ib): diagonal, single or alpha-alpha double. The
//     same-spin elements only need the string-pair densities
//        D[Ia,Ja] = sum_b C[Ia][b] C[Ja][b];
//   * beta pair (Ib, Jb > Ib, same Ia): the mirror image with C transposed;
//   * Gamma_ab[(ar,br),(ac,bc)], a product of an alpha and a beta excitation or
//     occupation.
// Step 1 computes the pair densities (a warp per eight string pairs). Step 2 sums, for
// each same-spin RDM element, a host-built list of (density, +/-1) terms -- the list
// encodes the reference's orbital ordering and antisymmetry signs (add_one_rdm /
// add_two_rdm, CIDens.cpp:227-292). Step 3, the alpha-beta block: for each alpha
// excitation (ar < ac) the string sums
//        g_x[Ib] = sum_(Ia -> Ja) s_a C[Ia][Ib] C[Ja][x(Ib)]
// over its string pairs, x the identity or one of Ib's single excitations, one thread
// per Ib with 36 or 12 of its sums in registers; then the sums of s_b g_x[Ib] over the Ib that
// belong to each (br, bc). The identity's sums, over the Ib that hold z, are the
// elements with beta occupation z; the mirror pass (identity only) gives those with
// alpha occupation.
//
// DOCI (DensDOCI, CIDens.cpp:1073-1224): the sums of c_I^2 n_j n_k and of the pair-hop
// products c_I c_J, on larger spaces as dot products of the blocks of strings with one
// set of high pairs (k_doci_rdm_split, a thread block per block of strings), else by a
// thread per orbital pair j <= k over a slice of the pair strings (k_doci_rdm).
//
// Storage follows CIDens: the 1-RDM and each 2-RDM block are symmetric pair
// matrices (Vector2d, matrix.cpp:674-690), accumulated on (min, max) and mirrored.
//
// Determinant lists (DensFILE) are handled in dets.cu: a pair scan with 64-bit
// fixed-point integer atomics (order-independent sums, also bit-reproducible).
#include <algorithm>
#include <memory>
#include <mutex>
#include <stdexcept>

#include "checked.cuh"
#include "crs.cuh"

namespace cigpu {
namespace {

constexpr int kRdmThreads = 256;

inline int pidx(int p, int q, int L) { return p * L + q - (p + 1) * (p + 2) / 2; }

// C(n, k) for n, k < 64 (strings of up to 63 orbitals), filled once.
struct BinomTable {
    int64_t c[64][65];
    BinomTable() {
        for (int n = 0; n < 64; ++n)
            for (int k = 0; k <= 64; ++k) c[n][k] = d_binom(n, k);
    }
};

uint32_t hrank(uint64_t s) {
    static const BinomTable bt;
    int64_t r = 0;
    int m = 0;
    while (s) {
        ++m;
        r += bt.c[__builtin_ctzll(s)][m];
        s &= s - 1;
    }
    return (uint32_t)r;
}

int hnstacked(int a, int b, uint64_t common) {
    const int lo = std::min(a, b), hi = std::max(a, b);
    int c = 0;
    for (int i = lo + 1; i < hi; ++i) c += (int)((common >> i) & 1);
    return c;
}

// One spin's pair list and its RDM terms.
struct PairPlan {
    std::vector<uint32_t> I, J;  // pairs: [self..., singles..., doubles...]
};

struct Plan {
    int L, np;
    int64_t Da, Db;
    PairPlan a, b;
    size_t off_ga, off_gb, off_g0, off_g2, nslots;
    // density layout: [Da | Db]
    size_t off_da, off_db, ndens;
    struct Term {
        uint32_t slot, dens;
        int8_t coef;
    };
    std::vector<Term> terms;  // in generation order; grouped by slot (stably) afterwards
};

// String pairs of each excitation of one spin: list pidx(r, c), r < c, holds the pairs
// (I, J = I - r + c) with their signs; with `diag`, list np + u the strings (I, I)
// holding orbital u.
struct ExcitationLists {
    std::vector<uint32_t> ptr;
    std::vector<uint64_t> pair;  // I | J << 32
    std::vector<int8_t> sign;
};

// The members of each sum over strings: place x * D + I in the string sums, the sign in
// bit 31.
struct SumLists {
    std::vector<uint32_t> ptr, at;
};

void add_term(Plan &P, size_t slot, size_t dens, int coef) {
    P.terms.push_back({(uint32_t)slot, (uint32_t)dens, (int8_t)coef});
}

// Slot of a symmetric pair matrix entry (min, max) of dimension dimx at offset off.
size_t sym_slot(size_t off, size_t dimx, size_t A, size_t B) {
    return off + std::min(A, B) * dimx + std::max(A, B);
}

// add_two_rdm for a same-spin block (CIDens.cpp:240-255): sorts both pairs with sign flips.
void add_two_same(Plan &P, size_t off, int o1, int o2, int o3, int o4, size_t dens, int coef) {
    if (o1 == o2 || o3 == o4) return;
    if (o1 > o2) { std::swap(o1, o2); coef = -coef; }
    if (o3 > o4) { std::swap(o3, o4); coef = -coef; }
    add_term(P, sym_slot(off, P.np, pidx(o1, o2, P.L), pidx(o3, o4, P.L)), dens, coef);
}

// Pairs and terms of one spin. `alpha` selects which 1-RDM / same-spin block.
void plan_spin(Plan &P, const SpinTables &t, bool alpha) {
    const int L = P.L, n = t.n;
    PairPlan &pp = alpha ? P.a : P.b;
    const int64_t D = t.D;
    // self pairs
    for (int64_t I = 0; I < D; ++I) {
        pp.I.push_back((uint32_t)I);
        pp.J.push_back((uint32_t)I);
    }
    // upper singles
    struct Single { uint32_t I, J; int lo, hi, sign; uint64_t common; };
    std::vector<Single> singles;
    for (int64_t I = 0; I < D; ++I) {
        const uint64_t s = t.strings[I];
        for (int j = 0; j < L; ++j) {
            if (!((s >> j) & 1)) continue;
            for (int l = j + 1; l < L; ++l) {
                if ((s >> l) & 1) continue;
                const uint64_t u = s ^ ((uint64_t)1 << j) ^ ((uint64_t)1 << l);
                const uint32_t J = hrank(u);  // > I since l > j
                singles.push_back({(uint32_t)I, J, j, l, (hnstacked(j, l, s & u) & 1) ? -1 : 1, s & u});
            }
        }
    }
    for (auto &x : singles) {
        pp.I.push_back(x.I);
        pp.J.push_back(x.J);
    }
    // upper same-spin doubles
    struct Dbl { uint32_t I, J; int o[4]; int sign; };
    std::vector<Dbl> dbls;
    for (int64_t I = 0; I < D; ++I) {
        const uint64_t s = t.strings[I];
        for (int j1 = 0; j1 < L; ++j1) {
            if (!((s >> j1) & 1)) continue;
            for (int j2 = j1 + 1; j2 < L; ++j2) {
                if (!((s >> j2) & 1)) continue;
                for (int l1 = 0; l1 < L; ++l1) {
                    if ((s >> l1) & 1) continue;
                    for (int l2 = l1 + 1; l2 < L; ++l2) {
                        if ((s >> l2) & 1) continue;
                        const uint64_t u = s ^ ((uint64_t)1 << j1) ^ ((uint64_t)1 << j2) ^ ((uint64_t)1 << l1) ^
                                           ((uint64_t)1 << l2);
                        const uint32_t J = hrank(u);
                        if (J <= (uint32_t)I) continue;
                        // fill_two_dense (CIDens.cpp:756-779): row orbitals first, ascending
                        const uint64_t c = s & u;
                        const int diff = hnstacked(j1, j2, c) + hnstacked(l1, l2, c);
                        dbls.push_back({(uint32_t)I, J, {j1, j2, l1, l2}, (diff & 1) ? -1 : 1});
                    }
                }
            }
        }
    }
    for (auto &x : dbls) {
        pp.I.push_back(x.I);
        pp.J.push_back(x.J);
    }
    (void)n;
    // terms
    const size_t d0 = alpha ? P.off_da : P.off_db;
    const size_t g1 = alpha ? P.off_ga : P.off_gb;
    const size_t gs = alpha ? P.off_g0 : P.off_g2;
    for (int64_t I = 0; I < D; ++I) {  // self pairs (fill_diagonal, CIDens.cpp:808-853)
        const uint64_t s = t.strings[I];
        int o[64], k = 0;
        for (int b = 0; b < L; ++b)
            if ((s >> b) & 1) o[k++] = b;
        for (int i = 0; i < k; ++i) add_term(P, sym_slot(g1, L, o[i], o[i]), d0 + I, 1);
        for (int i = 0; i < k; ++i)
            for (int j = i + 1; j < k; ++j) add_two_same(P, gs, o[i], o[j], o[i], o[j], d0 + I, 1);
    }
    for (size_t q = 0; q < singles.size(); ++q) {  // fill_one_dense (CIDens.cpp:676-754)
        const Single &x = singles[q];
        const size_t pi = (size_t)D + q;
        add_term(P, sym_slot(g1, L, x.lo, x.hi), d0 + pi, x.sign);
        for (int z = 0; z < L; ++z)
            if ((x.common >> z) & 1) add_two_same(P, gs, x.lo, z, x.hi, z, d0 + pi, x.sign);
    }
    for (size_t q = 0; q < dbls.size(); ++q) {
        const Dbl &x = dbls[q];
        const size_t pi = (size_t)D + singles.size() + q;
        add_two_same(P, gs, x.o[0], x.o[1], x.o[2], x.o[3], d0 + pi, x.sign);
    }
}

ExcitationLists excitation_lists(const SpinTables &t, bool diag) {
    const int L = t.L, np = L * (L - 1) / 2, nl = np + (diag ? L : 0);
    ExcitationLists e;
    e.ptr.assign((size_t)nl + 1, 0);
    auto each = [&](auto &&f) {  // f(list, I, J, odd) in the order of the strings
        for (int64_t I = 0; I < t.D; ++I) {
            for (int x = 0; x < t.ns; ++x) {
                const uint32_t w = t.s_info[(size_t)I * t.ns + x];
                const int r = (w >> 12) & 63, c = (w >> 18) & 63;
                if (r < c) f(pidx(r, c, L), I, t.s_target[(size_t)I * t.ns + x], (w >> 24) & 1u);
            }
            if (diag)
                for (int m = 0; m < t.n; ++m) f(np + t.occ[(size_t)I * t.n + m], I, (uint32_t)I, 0u);
        }
    };
    each([&](int q, int64_t, uint32_t, uint32_t) { ++e.ptr[(size_t)q + 1]; });
    for (int q = 0; q < nl; ++q) e.ptr[(size_t)q + 1] += e.ptr[q];
    e.pair.resize(e.ptr[nl]);
    e.sign.resize(e.ptr[nl]);
    std::vector<uint32_t> fill(e.ptr.begin(), e.ptr.end() - 1);
    each([&](int q, int64_t I, uint32_t J, uint32_t odd) {
        e.pair[fill[q]] = (uint64_t)I | ((uint64_t)J << 32);
        e.sign[fill[q]++] = odd ? -1 : 1;
    });
    return e;
}

// The sums (r, c), r != c, over the single excitations r -> c of one spin's strings
// (singles), and the sums over the strings that hold z, list z * L + z (or z without
// singles) of the identity's place.
SumLists sum_lists(const SpinTables &t, bool singles) {
    const int L = t.L, nl = singles ? L * L : L;
    const uint32_t D = (uint32_t)t.D, ident = singles ? (uint32_t)t.ns * D : 0u;
    SumLists e;
    e.ptr.assign((size_t)nl + 1, 0);
    auto each = [&](auto &&f) {
        for (int64_t I = 0; I < t.D; ++I) {
            if (singles)
                for (int x = 0; x < t.ns; ++x) {
                    const uint32_t w = t.s_info[(size_t)I * t.ns + x];
                    f((int)((w >> 12) & 63) * L + (int)((w >> 18) & 63), (uint32_t)x * D + (uint32_t)I, (w >> 24) & 1u);
                }
            for (int m = 0; m < t.n; ++m) {
                const int z = t.occ[(size_t)I * t.n + m];
                f(singles ? z * L + z : z, ident + (uint32_t)I, 0u);
            }
        }
    };
    each([&](int q, uint32_t, uint32_t) { ++e.ptr[(size_t)q + 1]; });
    for (int q = 0; q < nl; ++q) e.ptr[(size_t)q + 1] += e.ptr[q];
    e.at.resize(e.ptr[nl]);
    std::vector<uint32_t> fill(e.ptr.begin(), e.ptr.end() - 1);
    each([&](int q, uint32_t at, uint32_t odd) { e.at[fill[q]++] = at | (odd << 31); });
    return e;
}

// ---------------------------------------------------------------------------
// Step 1: pair densities. C is D1 x D2 row-major. A warp takes eight pairs, which
// mostly share their first string (the lists run over it): nine coalesced loads feed
// eight multiply-adds, and the eight sums meet in one exchange of halves. Bound by the
// FP64 pipe (2 lanes per clock and SM): 112 M multiply-adds per spin at L=12 6a6b,
// 0.18 ms at its rate, 0.20 measured (1.23 ms when the same kernel also formed the
// densities weighted by the other spin's occupations, 12 of 32 lanes at work).
constexpr int kPairBatch = 8;

__global__ void __launch_bounds__(kRdmThreads) k_pair_dens(const double *__restrict__ C, int64_t D2,
                                                           const uint32_t *__restrict__ pI,
                                                           const uint32_t *__restrict__ pJ, int64_t npairs,
                                                           double *__restrict__ dens, int64_t D1,
                                                           unsigned long long *err) {
    const int lane = threadIdx.x & 31;
    const int64_t wid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t p0 = wid * kPairBatch; p0 < npairs; p0 += nw * kPairBatch) {
        const double *ri[kPairBatch], *rj[kPairBatch];
        bool same = true;
#pragma unroll
        for (int k = 0; k < kPairBatch; ++k) {
            const int64_t p = p0 + k < npairs ? p0 + k : npairs - 1;  // a short last batch repeats its last pair
            uint32_t I = pI[p], J = pJ[p];
            if (!CIGPU_CHECK(err, index_ok(I, (uint64_t)D1) && index_ok(J, (uint64_t)D1), kCheckRdmPair, p)) I = J = 0;
            ri[k] = C + (int64_t)I * D2;
            rj[k] = C + (int64_t)J * D2;
            same = same && ri[k] == ri[0];
        }
        double acc[kPairBatch];
#pragma unroll
        for (int k = 0; k < kPairBatch; ++k) acc[k] = 0;
        if (same) {
            for (int64_t b = lane; b < D2; b += 32) {
                const double v = ri[0][b];
#pragma unroll
                for (int k = 0; k < kPairBatch; ++k) acc[k] += v * rj[k][b];
            }
        } else {
            for (int64_t b = lane; b < D2; b += 32) {
#pragma unroll
                for (int k = 0; k < kPairBatch; ++k) acc[k] += ri[k][b] * rj[k][b];
            }
        }
        // halves exchanged: after three steps lane l holds a quarter warp's sum of pair l / 4
#pragma unroll
        for (int h = 4, o = 16; h > 0; h >>= 1, o >>= 1) {
            const bool hi = lane & o;
#pragma unroll
            for (int k = 0; k < h; ++k) {
                const double give = hi ? acc[k] : acc[k + h];
                const double keep = hi ? acc[k + h] : acc[k];
                acc[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        double a = acc[0];
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        if ((lane & 3) == 0 && p0 + (lane >> 2) < npairs) dens[p0 + (lane >> 2)] = a;
    }
}

// Step 2: per-slot sums of +/- densities, a warp per slot (lanes over the terms, then the
// warp tree: a fixed order). A thread per slot took 79 us for the 243,000 terms of L=12
// 6a6b, the longest lists one after the other: 60 us more per call.
__global__ void k_slot_gather(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ idx,
                              const int8_t *__restrict__ coef, const double *__restrict__ dens, int64_t nslots,
                              double *__restrict__ acc, int64_t ndens, unsigned long long *err) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s < nslots; s += nw) {
        double v = 0;
        for (uint32_t e = ptr[s] + lane; e < ptr[s + 1]; e += 32) {
            const uint32_t k = idx[e];
            if (!CIGPU_CHECK(err, index_ok(k, (uint64_t)ndens), kCheckRdmTerm, e)) continue;
            v += __longlong_as_double(__double_as_longlong(dens[k]) ^ ((long long)(coef[e] < 0) << 63));
        }
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) acc[s] = v;
    }
}

// Step 3: string sums. For each string pair (I, J) of list q (C's first string) the
// block stages row J and every thread, on its own second string S, adds
// s C[I][S] C[J][x(S)] to the sums of kAbX of S's single excitations x, and (first
// chunk) to the identity's. The sums stay in registers over the list's pairs and are
// stored once, G[q - q0][x][S] (x = ns: the identity). A multiply-add per term and its
// gather from shared memory: bound by the FP64 pipe, 0.57 G multiply-adds at L=12 6a6b,
// 0.90 ms at its rate. (One thread per (br, bc) walking lists of string pairs, the
// sign a second FP64 product, on 264 blocks of 160 threads: 4.36 ms. Now 1.25.)
constexpr int kAbThreads = 128;
// Excitations per thread: 36 where the strings alone make three blocks per SM (L=12 6a6b:
// each row staged once, 1.25 against 1.39 ms), else 12, whose chunks make up to three
// times as many blocks (L=10 5a5b would have 110).
constexpr int kAbWide = 36, kAbNarrow = 12;

__device__ __forceinline__ void copy8_async(double *dst, const double *src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src));
}

template <int kAbX>
__global__ void __launch_bounds__(kAbThreads) k_string_sums(const double *__restrict__ C, int64_t D2,
                                                            const uint32_t *__restrict__ target, int ns,
                                                            const uint32_t *__restrict__ ptr,
                                                            const uint64_t *__restrict__ pair,
                                                            const int8_t *__restrict__ sign, int q0,
                                                            double *__restrict__ G, int64_t D1,
                                                            unsigned long long *err) {
    extern __shared__ double rows[];  // [2][D2]
    const int q = q0 + blockIdx.z, x0 = blockIdx.y * kAbX, nx = min(kAbX, ns - x0);
    const uint32_t e0 = ptr[q], e1 = ptr[q + 1];
    const int64_t S = blockIdx.x * (int64_t)kAbThreads + threadIdx.x;
    const bool act = S < D2;
    uint32_t at[kAbX];
#pragma unroll
    for (int x = 0; x < kAbX; ++x) {
        at[x] = 0;
        if (act && x < nx) {
            at[x] = __ldg(target + S * ns + x0 + x);
            if (!CIGPU_CHECK(err, index_ok(at[x], (uint64_t)D2), kCheckRdmExcit, S)) at[x] = 0;
        }
    }
    double acc[kAbX], ident = 0;
#pragma unroll
    for (int x = 0; x < kAbX; ++x) acc[x] = 0;
    auto pair_of = [&](uint32_t e, uint32_t &I, uint32_t &J) {
        const uint64_t pr = __ldg(pair + e);
        I = (uint32_t)pr;
        J = (uint32_t)(pr >> 32);
        if (!CIGPU_CHECK(err, index_ok(I, (uint64_t)D1) && index_ok(J, (uint64_t)D1), kCheckRdmPair, e)) I = J = 0;
    };
    auto stage = [&](uint32_t e, double *dst) {
        uint32_t I, J;
        pair_of(e, I, J);
        const double *src = C + (int64_t)J * D2;
        for (int64_t b = threadIdx.x; b < D2; b += kAbThreads) copy8_async(dst + b, src + b);
        asm volatile("cp.async.commit_group;");
    };
    if (e0 < e1) stage(e0, rows);
    for (uint32_t e = e0; e < e1; ++e) {
        const double *row = rows + ((e - e0) & 1) * D2;
        uint32_t I, J;
        pair_of(e, I, J);
        double v = act ? C[(int64_t)I * D2 + S] : 0.0;
        v = __longlong_as_double(__double_as_longlong(v) ^ ((long long)(__ldg(sign + e) < 0) << 63));
        asm volatile("cp.async.wait_group 0;");
        __syncthreads();  // this pair's row is staged; the other buffer is read
        if (e + 1 < e1) stage(e + 1, rows + ((e + 1 - e0) & 1) * D2);
        if (act) {
            if (x0 == 0) ident += v * row[S];
#pragma unroll
            for (int x = 0; x < kAbX; ++x)
                if (x < nx) acc[x] += v * row[at[x]];
        }
    }
    if (!act) return;
    double *g = G + (int64_t)blockIdx.z * (ns + 1) * D2 + S;
#pragma unroll
    for (int x = 0; x < kAbX; ++x)
        if (x < nx) g[(int64_t)(x0 + x) * D2] = acc[x];
    if (x0 == 0) g[(int64_t)ns * D2] = ident;
}

// The identity's string sums alone (no staging: row J is read at S itself).
__global__ void __launch_bounds__(kAbThreads) k_string_sums_ident(const double *__restrict__ C, int64_t D2,
                                                                  const uint32_t *__restrict__ ptr,
                                                                  const uint64_t *__restrict__ pair,
                                                                  const int8_t *__restrict__ sign, int q0,
                                                                  double *__restrict__ G, int64_t D1,
                                                                  unsigned long long *err) {
    const int q = q0 + blockIdx.z;
    const uint32_t e0 = ptr[q], e1 = ptr[q + 1];
    const int64_t S = blockIdx.x * (int64_t)kAbThreads + threadIdx.x;
    if (S >= D2) return;
    constexpr int U = 8;  // pairs in flight
    double acc = 0;
    for (uint32_t e = e0; e < e1; e += U) {
        double a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            a[u] = b[u] = 0.0;
            if (e + u < e1) {
                const uint64_t pr = __ldg(pair + e + u);
                uint32_t I = (uint32_t)pr, J = (uint32_t)(pr >> 32);
                if (!CIGPU_CHECK(err, index_ok(I, (uint64_t)D1) && index_ok(J, (uint64_t)D1), kCheckRdmPair, e)) I = J = 0;
                a[u] = C[(int64_t)I * D2 + S];
                b[u] = C[(int64_t)J * D2 + S];
                a[u] = __longlong_as_double(__double_as_longlong(a[u]) ^ ((long long)(__ldg(sign + e + u) < 0) << 63));
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) acc += a[u] * b[u];
    }
    G[(int64_t)blockIdx.z * D2 + S] = acc;
}

// out[q][t] = the signed sum of list t over the string sums of q, one warp each.
__global__ void k_sum_strings(const double *__restrict__ G, int64_t per_q, const uint32_t *__restrict__ ptr,
                              const uint32_t *__restrict__ at, int nt, int nq, double *__restrict__ out,
                              unsigned long long *err) {
    const int lane = threadIdx.x & 31;
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (w >= (int64_t)nq * nt) return;
    const int64_t q = w / nt;
    const int t = (int)(w - q * nt);
    const double *g = G + q * per_q;
    double v = 0;
    for (uint32_t e = ptr[t] + lane; e < ptr[t + 1]; e += 32) {
        const uint32_t k = at[e];
        if (!CIGPU_CHECK(err, index_ok(k & 0x7FFFFFFFu, (uint64_t)per_q), kCheckRdmTerm, e)) continue;
        const double x = g[k & 0x7FFFFFFFu];
        v += __longlong_as_double(__double_as_longlong(x) ^ ((long long)(k >> 31) << 63));
    }
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) out[w] = v;
}

// Assemble the outputs, mirrored: the same-spin sums, and Gamma_ab's upper triangle
// from t1[(ar < ac)][br, bc], t2[(br < bc)][z] (alpha occupation z) and, after the np
// rows of t2, t2[np + u][z] (beta occupation u, alpha occupation z).
__global__ void k_rdm_assemble(const double *__restrict__ acc, const double *__restrict__ t1,
                               const double *__restrict__ t2, int L, int np, size_t off_ga, size_t off_gb,
                               size_t off_g0, size_t off_g2, double *__restrict__ rdm1, double *__restrict__ aa,
                               double *__restrict__ ab, double *__restrict__ bb) {
    const int64_t L2 = (int64_t)L * L;
    const int64_t n1 = 2 * L2, n2 = (int64_t)np * np, n3 = L2 * L2;
    const int64_t total = n1 + 2 * n2 + n3;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < n1) {
            const int s = (int)(i / L2), a = (int)((i % L2) / L), b = (int)(i % L);
            rdm1[i] = acc[(s == 0 ? off_ga : off_gb) + (size_t)min(a, b) * L + max(a, b)];
        } else if (i < n1 + 2 * n2) {
            const int64_t j = i - n1;
            const int blk = (int)(j / n2);
            const int A = (int)((j % n2) / np), B = (int)(j % np);
            const double v = acc[(blk == 0 ? off_g0 : off_g2) + (size_t)min(A, B) * np + max(A, B)];
            (blk == 0 ? aa : bb)[j % n2] = v;
        } else {
            const int64_t j = i - n1 - 2 * n2;
            const int64_t A = j / L2, B = j % L2;
            const int64_t lo = min(A, B), hi = max(A, B);
            const int ar = (int)(lo / L), ac = (int)(hi / L), br = (int)(lo % L), bc = (int)(hi % L);
            double v;
            if (ar < ac)
                v = t1[(int64_t)(ar * L + ac - (ar + 1) * (ar + 2) / 2) * L2 + br * L + bc];
            else if (br < bc)
                v = t2[(int64_t)(br * L + bc - (br + 1) * (br + 2) / 2) * L + ar];
            else
                v = t2[(int64_t)(np + br) * L + ar];
            ab[j] = v;
        }
    }
}

__global__ void k_transpose(const double *__restrict__ a, int64_t rows, int64_t cols, double *__restrict__ t) {
    __shared__ double tile[32][33];
    const int64_t r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y)
        if (r0 + i < rows && c0 + threadIdx.x < cols) tile[i][threadIdx.x] = a[(r0 + i) * cols + c0 + threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y)
        if (c0 + i < cols && r0 + threadIdx.x < rows) t[(c0 + i) * rows + r0 + threadIdx.x] = tile[threadIdx.x][i];
}

// ---------------------------------------------------------------------------
// DOCI: thread (j,k) of an L*L block accumulates, over the block's pair strings,
//   A_jk = sum c_I^2 n_j n_k   and   B_jk = sum_{j in I, k not in I, k > j} c_I c_J,
// J = I - j + k. The block stages kDociChunk strings at a time in shared memory
// (one coalesced load of strings and c) with each string's rank prefix, so every
// pair-hop rank costs O(1): with p_1 < ... < p_n the occupied orbitals and
// rank(S) = sum_m C(p_m, m), moving the electron at j = p_{a+1} to the empty
// k > j (b electrons below k, j included) shifts p_{a+2..b} down one place:
//   rank(J) = I - C(j, a+1) + (P_b - P_{a+1}) + C(k, b),
//   P_m = sum_{i <= m} (C(p_i, i-1) - C(p_i, i)),
// evaluated modulo 2^32 (the result is a rank below 2^32, so the wrap cancels).
//
// The sums are 64-bit fixed-point integers (value * 2^60) on the integer pipe: a
// thread's FP64 add would occupy GB300's FP64 pipe (2 lanes per clock per SM) for
// the whole warp even when one lane of it needs the add, and most lanes of a warp
// skip a given string. Each coefficient becomes c * 2^62 (rounded to nearest, from
// its bit fields, |c| <= 1 for a normalised state), a product is the rounded high
// half of the 128-bit product (scale 2^60), and integer addition is associative, so
// the sums do not depend on order; each term is rounded by at most 2^-61 and every
// sum lies within +-1.
constexpr int kDociChunk = 128;
constexpr int kDociMaxL = 32;
constexpr int kRdmBatch = 8;  // pair hops gathered per round (loads in flight per thread)

// c * 2^62 rounded to nearest (|c| <= 1), from the IEEE-754 fields on the integer pipe.
__device__ __forceinline__ long long fx62(double c) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(c);
    const int e = (int)((u >> 52) & 0x7FF);
    if (e == 0) return 0;  // zero (and subnormals, below 2^-1022)
    const unsigned long long m = (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    const int sh = e - 1013;  // c * 2^62 = m * 2^(e - 1023 - 52 + 62)
    unsigned long long r;
    if (sh >= 0)
        r = sh <= 10 ? (m << sh) : 0x4000000000000000ull;  // |c| <= 1 keeps sh <= 10
    else if (sh > -64)
        r = (m + (1ull << (-sh - 1))) >> (-sh);
    else
        r = 0;
    return (u >> 63) ? -(long long)r : (long long)r;
}

// (a * b) / 2^64 rounded to nearest: a, b at scale 2^62 give a product at 2^60.
__device__ __forceinline__ long long fxmul(long long a, long long b) {
    const long long hi = __mul64hi(a, b);
    const unsigned long long lo = (unsigned long long)a * (unsigned long long)b;
    return hi + (long long)(lo >> 63);
}

// A fixed-point value as two signed 32-bit digits, hi 2^32 + lo: the four products of a
// multiplication are then signed 32 x 32 -> 64 bit, with no corrections.
__device__ __forceinline__ long long fxdigits(long long a) {
    const uint32_t lo = (uint32_t)a, hi = (uint32_t)((unsigned long long)a >> 32) + (lo >> 31);
    return (long long)((unsigned long long)hi << 32 | lo);
}

// sum += fxmul(a, b) of two values in digits: of a b = hh 2^64 + mid 2^32 + ll, rounded to
// nearest at 2^64, the low half of ll changes nothing.
__device__ __forceinline__ void fxadd(long long &sum, long long a, long long b) {
    const int ah = (int)(a >> 32), al = (int)a, bh = (int)(b >> 32), bl = (int)b;
    const long long ll = (long long)al * bl;  // within +-2^62
    long long mid = (long long)((uint32_t)(ll >> 32) + 0x80000000u);
    mid += (long long)ah * bl;
    mid += (long long)al * bh;
    sum += (long long)ah * bh;
    sum += mid >> 32;
}

__device__ __forceinline__ void add_to(long long *at, long long v) {
    atomicAdd(reinterpret_cast<unsigned long long *>(at), (unsigned long long)v);
}

__global__ void k_doci_rdm(const double *__restrict__ c, const uint64_t *__restrict__ strings, int64_t D, int L,
                           int n, long long *__restrict__ sums, unsigned long long *err) {
    __shared__ uint32_t binom[(kDociMaxL + 1) * (kDociMaxL + 2)];  // C(nn, kk), nn <= L, kk <= n + 1
    __shared__ uint64_t ss[kDociChunk];
    __shared__ long long cs[kDociChunk], cs2[kDociChunk];  // c_I * 2^62, c_I^2 * 2^60
    __shared__ uint32_t pre[kDociChunk][kDociMaxL + 1];
    constexpr int BW = kDociMaxL + 2;
    for (int i = threadIdx.x; i < (kDociMaxL + 1) * BW; i += blockDim.x) {
        const int nn = i / BW, kk = i % BW;
        binom[i] = (nn <= L && kk <= n + 1) ? (uint32_t)d_binom(nn, kk) : 0u;
    }
    // thread t owns the pair (j, k), j <= k, of the upper triangle in row-major
    // order (A is symmetric, B is summed for j < k only)
    const int t = threadIdx.x;
    const bool work = t < L * (L + 1) / 2;
    int j = 0, k = 0;
    if (work) {
        int rem = t;
        while (rem >= L - j) {
            rem -= L - j;
            ++j;
        }
        k = j + rem;
    }
    const bool hop = work && k > j;
    const uint64_t below_j = work ? (((uint64_t)1 << j) - 1) : 0, below_k = work ? (((uint64_t)1 << k) - 1) : 0;
    long long A = 0, B = 0;
    for (int64_t base = (int64_t)blockIdx.x * kDociChunk; base < D; base += (int64_t)gridDim.x * kDociChunk) {
        __syncthreads();  // the previous chunk is consumed (and the table is ready)
        const int cnt = (D - base) < kDociChunk ? (int)(D - base) : kDociChunk;
        for (int q = t; q < cnt; q += blockDim.x) {  // blocks of fewer than kDociChunk threads loop
            const uint64_t st = strings[base + q];
            const long long cf = fx62(c[base + q]);
            ss[q] = st;
            cs[q] = cf;
            cs2[q] = fxmul(cf, cf);
            uint32_t P = 0;
            pre[q][0] = 0;
            int m = 0;
            for (uint64_t x = st; x; x &= x - 1) {
                ++m;
                const int pm = __ffsll((long long)x) - 1;
                P += binom[pm * BW + m - 1] - binom[pm * BW + m];
                pre[q][m] = P;
            }
        }
        __syncthreads();
        if (work) {
            // kRdmBatch strings per round: ranks first, then their gathers of c
            // together, so several L2 loads are in flight per thread
            for (int i0 = 0; i0 < cnt; i0 += kRdmBatch) {
                uint32_t rr[kRdmBatch];
#pragma unroll
                for (int u = 0; u < kRdmBatch; ++u) {
                    const int i = i0 + u;
                    rr[u] = 0xFFFFFFFFu;
                    if (i < cnt) {
                        const uint64_t st = ss[i];
                        const bool nj = (st >> j) & 1, nk = (st >> k) & 1;
                        if (nj && nk) A += cs2[i];
                        if (hop && nj && !nk) {
                            const int a = __popcll(st & below_j), b = __popcll(st & below_k);
                            rr[u] = (uint32_t)(base + i) - binom[j * BW + a + 1] + pre[i][b] - pre[i][a + 1] +
                                    binom[k * BW + b];
                            if (!CIGPU_CHECK(err, index_ok(rr[u], (uint64_t)D), kCheckHopRank, rr[u])) rr[u] = 0xFFFFFFFFu;
                        }
                    }
                }
                double cv[kRdmBatch];
#pragma unroll
                for (int u = 0; u < kRdmBatch; ++u) cv[u] = rr[u] < (uint64_t)D ? __ldg(c + rr[u]) : 0.0;
#pragma unroll
                for (int u = 0; u < kRdmBatch; ++u)
                    if (rr[u] < (uint64_t)D) B += fxmul(cs[i0 + u], fx62(cv[u]));
            }
        }
    }
    // added at (j, k), j <= k, of the [2][L][L] sums (zero before the launch; the lower
    // triangle is not written and not read): integer sums, the same in any order. A
    // finishing kernel that summed 608 blocks' partials, a thread per element, took 181 us.
    if (work) {
        add_to(sums + j * L + k, A);
        add_to(sums + L * L + j * L + k, B);
    }
}

// ---------------------------------------------------------------------------
// The same sums by low and high orbitals (larger spaces; see the split product in
// doci_mv.cu for the blocks). A pair hop's two coefficients lie in blocks whose starts
// are shared by all of a block's strings, so the sums are dot products of blocks:
//   * j, k high: the block h with the block h - j + k, string by string;
//   * j, k low: inside the block, over the list of the strings that hold j and not k;
//   * j low, k high: the block h with the staged block h + k, over the list of the
//     strings that hold j.
// Every lane of a warp has a product to add (a thread per orbital pair found one in
// four strings to act on, and formed a rank for each), and A needs only the blocks'
// sums of squares, per block and per low string. The products and sums are the
// fixed-point integers above, so the result is the same bit for bit in any order:
// integer atomics collect them. Bound by instruction issue (49 for 32
// products, ALU 41%) and the barriers around the staging (three blocks per SM: 65 KB of
// shared memory each at L=24). L=24,
// 12 pairs: 3.80 -> 0.74 ms per cigpu_rdm with a sum at a time for every warp, 0.66 with
// four and in digits, 0.65 without the block's own matrices of sums (the kernel 490 -> 418
// us; the vector's way from host memory is 150).
constexpr int kSplitRdmThreads = 256;  // 384: L=24 0.63, L=27 19 pairs 1.47 against 1.36 ms; 512: 0.68, 1.80
constexpr int kSplitRdmWarps = kSplitRdmThreads / 32;
// Spaces whose blocks hold at least this many strings on average take it: a block of
// strings costs a thread block some microseconds whatever its length (L=27, 19 pairs, 76
// strings a block: 3.72 -> 1.36 ms per call; L=19, 12 pairs, 98: 280 -> 121 us; L=30, 24
// pairs, 19 strings: 1.44 ms against 2.43 when the split took 2.42 and 134 in those; L=30, 5
// pairs, 11: 0.49 against 0.83).
constexpr int64_t kSplitRdmBlock = 40;
constexpr size_t kSplitRdmMaxSmem = 200 * 1024;

__global__ void k_fix62(const double *__restrict__ c, int64_t n, long long *__restrict__ f) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        f[i] = fxdigits(fx62(c[i]));
}

__device__ __forceinline__ long long warp_sum(long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The sums over the warp of four values per lane, by exchange of halves: lane's is that of
// a[lane >> 3].
__device__ __forceinline__ long long sum_four(const long long (&a)[4], int lane) {
    const bool h = lane & 16, q = lane & 8;
    const long long b0 = (h ? a[2] : a[0]) + __shfl_xor_sync(0xffffffffu, h ? a[0] : a[2], 16);
    const long long b1 = (h ? a[3] : a[1]) + __shfl_xor_sync(0xffffffffu, h ? a[1] : a[3], 16);
    long long v = (q ? b1 : b0) + __shfl_xor_sync(0xffffffffu, q ? b0 : b1, 8);
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A thread block per block of strings (several to one thread block left its last ones, and
// the sectors of short blocks, to run alone: 0.90 ms per call at L=24 with a few, 0.74 with one).
// sums: [2][L][L] (A, then B; j <= k), low: [lowbits] sums of squares per low string.
__global__ void __launch_bounds__(kSplitRdmThreads, 4) k_doci_rdm_split(const DociSplitView p,
                                                                     const long long *__restrict__ cf,
                                                                     long long *__restrict__ sums,
                                                                     long long *__restrict__ low) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int L = p.L, s = p.s, Lh = L - s, t = threadIdx.x, warp = t >> 5, lane = t & 31;
    long long *area = reinterpret_cast<long long *>(smem);
    // a block of strings has one sum for an element of either: added to memory as it is formed
    long long *sA = sums, *sB = sums + L * L;
    auto start_of = [&](uint64_t b, int mm) {
        uint32_t r = 0;
        for (int k = mm + 1; b; b &= b - 1, ++k) r += __ldg(p.binom + (s + __ffsll((long long)b) - 1) * kSplitBinomRow + k);
        return r;
    };
    auto nth = [](uint64_t b, int i) {
        for (; i > 0; --i) b &= b - 1;
        return __ffsll((long long)b) - 1;
    };
    auto load = [&](uint32_t at) {
        return CIGPU_CHECK(p.err, index_ok(at, (uint64_t)p.D), kCheckHopRank, at) ? __ldg(cf + at) : 0ll;
    };
    const uint64_t full = (((uint64_t)1) << Lh) - 1;
    const int np = s * (s - 1) / 2;
    uint32_t h = blockIdx.x;
    int q = 0;
    for (; q + 1 < p.nsec && h >= p.sec[q].nhigh; ++q) h -= p.sec[q].nhigh;
    const DociSector &c = p.sec[q];
    const int nh = c.nh, nv = Lh - nh, m = c.m, nhh = nh * nv;
    const int nlow = (int)c.nlow, nminus = (int)c.nminus, n1 = (int)c.n1, n2 = (int)c.n2;
    long long *own = area, *sq = own + nlow, *up = sq + nlow;  // [nlow], [nlow], [nv][nminus]
    uint32_t *hhb = reinterpret_cast<uint32_t *>(up + (size_t)nv * nminus);  // [nhh]
    uint32_t *hhe = hhb + nhh;                                                // [nhh]
    uint32_t *upb = hhe + nhh;                                                // [nv]
    const uint32_t *one = p.one + c.one0, *two = p.two + c.two0;
    const uint64_t hb = __ldg(p.hbits + c.high0 + h);
    const uint32_t base = __ldg(p.hbase + c.high0 + h);
    __shared__ int nhop, job;
    if (t == 0) nhop = job = 0;
    __syncthreads();
    for (int e = t; e < nhh; e += kSplitRdmThreads) {
        const int a = e / nv, j = nth(hb, a), k = nth(full & ~hb, e - a * nv);
        if (k < j) continue;  // summed from the other side
        const int at = atomicAdd(&nhop, 1);  // in any order
        hhb[at] = start_of(hb ^ ((uint64_t)1 << j) ^ ((uint64_t)1 << k), m);
        hhe[at] = (uint32_t)(j * L + k);
    }
    if (m > 0)
        for (int r = t; r < nv; r += kSplitRdmThreads)
            upb[r] = start_of(hb | ((uint64_t)1 << nth(full & ~hb, r)), m - 1);
    for (int l = t; l < nlow; l += kSplitRdmThreads) {
        const long long v = load(base + (uint32_t)l);
        long long v2 = 0;
        fxadd(v2, v, v);
        own[l] = v;
        sq[l] = v2;
        add_to(low + c.low0 + l, v2);
    }
    __syncthreads();
    if (m > 0)
        for (int r = warp; r < nv; r += kSplitRdmWarps)
            for (int l = lane; l < nminus; l += 32) up[(size_t)r * nminus + l] = load(upb[r] + (uint32_t)l);
    __syncthreads();  // the blocks h + k are staged
    // Four sums at a time, the next four for whichever warp is free, the longest first: one
    // sum at a time, its reduction, its place and its atomic cost as much as its products.
    const int hops = (nhop + 3) / 4, mixed = m > 0 ? (nv * s + 3) / 4 : 0, pairs = n2 > 0 ? (np + 3) / 4 : 0;
    const int squares = m > 0 && nh > 0 ? s : 0, jobs = hops + mixed + pairs + squares + (nh > 0);
    for (;;) {
        int g = lane == 0 ? atomicAdd(&job, 1) : 0;
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= jobs) break;
        long long a[4] = {0, 0, 0, 0};
        const int mine = lane >> 3;  // of the four, after the reduction
        const bool writes = (lane & 7) == 0;
        if (g < hops) {  // high - high
            uint32_t b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) b[u] = hhb[min(4 * g + u, nhop - 1)];
            for (int l = lane; l < nlow; l += 32) {
                const long long v = own[l];
#pragma unroll
                for (int u = 0; u < 4; ++u) fxadd(a[u], v, load(b[u] + (uint32_t)l));
            }
            const long long sum = sum_four(a, lane);
            const int e = 4 * g + mine;
            if (writes && e < nhop) add_to(sB + (hhe[e] / L + s) * L + s + hhe[e] % L, sum);
            continue;
        }
        g -= hops;
        if (g < mixed) {  // low - high
            const uint32_t *w[4];
            const long long *row[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = min(4 * g + u, nv * s - 1), r = e / s;
                w[u] = one + (size_t)(e - r * s) * n1;
                row[u] = up + (size_t)r * nminus;
            }
            for (int x = lane; x < n1; x += 32) {
                uint32_t v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = __ldg(w[u] + x);
#pragma unroll
                for (int u = 0; u < 4; ++u) fxadd(a[u], own[v[u] & 0xFFFFu], row[u][v[u] >> 16]);
            }
            const long long sum = sum_four(a, lane);
            const int e = 4 * g + mine, r = e / s;
            if (writes && e < nv * s) add_to(sB + (e - r * s) * L + s + nth(full & ~hb, r), sum);
            continue;
        }
        g -= mixed;
        if (g < pairs) {  // low - low: pairs (j, k), row-major, j < k
            const uint32_t *w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) w[u] = two + (size_t)min(4 * g + u, np - 1) * n2;
            for (int x = lane; x < n2; x += 32) {
                uint32_t v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = __ldg(w[u] + x);
#pragma unroll
                for (int u = 0; u < 4; ++u) fxadd(a[u], own[v[u] & 0xFFFFu], own[v[u] >> 16]);
            }
            const long long sum = sum_four(a, lane);
            int e = 4 * g + mine, j = 0;
            if (writes && e < np) {
                for (; e >= s - 1 - j; ++j) e -= s - 1 - j;
                add_to(sB + j * L + j + 1 + e, sum);
            }
            continue;
        }
        g -= pairs;
        long long v = 0;
        if (g < squares) {  // squares of the block's strings that hold g
            for (int x = lane; x < n1; x += 32) v += sq[__ldg(one + (size_t)g * n1 + x) & 0xFFFFu];
            v = warp_sum(v);
            for (int i = lane; i < nh; i += 32) add_to(sA + g * L + s + nth(hb, i), v);
        } else {  // squares of the block
            for (int l = lane; l < nlow; l += 32) v += sq[l];
            v = warp_sum(v);
            for (int e = lane; e < nh * nh; e += 32) {
                const int i = e / nh, k = e - i * nh;
                if (k >= i) add_to(sA + (s + nth(hb, i)) * L + s + nth(hb, k), v);
            }
        }
    }
}

// A of two low orbitals (block.x = j * s + k, j <= k): the sums of squares of the low
// strings that hold both.
__global__ void k_doci_rdm_low(const DociSplitView p, uint32_t n, const long long *__restrict__ low,
                               long long *__restrict__ sums) {
    const int j = blockIdx.x / p.s, k = blockIdx.x - j * p.s;
    if (k < j) return;
    const uint32_t both = (1u << j) | (1u << k);
    long long a = 0;
    for (uint32_t l = threadIdx.x; l < n; l += blockDim.x)
        if ((p.lowbits[l] & both) == both) a += low[l];
    a = warp_sum(a);
    if ((threadIdx.x & 31) == 0 && a != 0) add_to(sums + j * p.L + k, a);
}

// Blocks of strings of the plan.
uint32_t split_blocks(const DociSplitView &v) {
    uint32_t n = 0;
    for (int q = 0; q < v.nsec; ++q) n += v.sec[q].nhigh;
    return n;
}

size_t split_rdm_smem(const DociSplitView &v) {
    size_t most = 0;
    for (int q = 0; q < v.nsec; ++q) {
        const DociSector &c = v.sec[q];
        const size_t nv = v.L - v.s - c.nh;
        most = std::max(most, 8 * (2 * (size_t)c.nlow + nv * c.nminus) + 4 * (2 * c.nh * nv + nv));
    }
    return most;
}

__global__ void k_doci_rdm_finish(const long long *__restrict__ sums, int L, int np, double *__restrict__ rdm1,
                                  double *__restrict__ aa, double *__restrict__ ab, double *__restrict__ bb) {
    const int L2 = L * L;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L2) return;
    const int j = t / L, k = t % L;
    const int tu = j <= k ? t : k * L + j;  // the sums hold j <= k
    const double A = (double)sums[tu] * 0x1p-60, B = (double)sums[L2 + tu] * 0x1p-60;  // fixed point, 2^60
    // 1-RDM (both spins): gamma_jj = A_jj
    if (j == k) {
        rdm1[j * L + j] = A;
        rdm1[L2 + j * L + j] = A;
    }
    // Gamma_ab(jk,jk) = A_jk; Gamma_ab(jj,kk) = Gamma_ab(kk,jj) = B_jk (j < k)
    ab[(int64_t)(j * L + k) * L2 + j * L + k] = A;
    if (j < k) {
        ab[(int64_t)(j * L + j) * L2 + k * L + k] = B;
        ab[(int64_t)(k * L + k) * L2 + j * L + j] = B;
        const int P = j * L + k - (j + 1) * (j + 2) / 2;
        aa[(int64_t)P * np + P] = A;
        bb[(int64_t)P * np + P] = A;
    }
}

// The two L x L matrices a DOCI state's RDMs reduce to, in CIDens element terms:
//   Pm[j][k] = get_two_rdm(1, j, j, k, k)   (pair hop B_jk; A_jj on the diagonal)
//   Dm[j][k] = get_two_rdm(0, j, k, j, k)   (A_jk; zero on the diagonal)
__global__ void k_doci_pairs_finish(const long long *__restrict__ sums, int L, double *__restrict__ Pm,
                                    double *__restrict__ Dm) {
    const int L2 = L * L;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L2) return;
    const int j = t / L, k = t % L;
    const int tu = j <= k ? t : k * L + j;  // the sums hold j <= k (B: j < k)
    const double A = (double)sums[tu] * 0x1p-60, B = (double)sums[L2 + tu] * 0x1p-60;  // fixed point, 2^60
    Pm[t] = j == k ? A : B;
    Dm[t] = j == k ? 0.0 : A;
}

template <typename T>
DevBuf<T> upload(const std::vector<T> &v, cudaStream_t s) {
    DevBuf<T> d(std::max<size_t>(v.size(), 1));
    if (!v.empty()) CIGPU_CUDA(cudaMemcpyAsync(d.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    return d;
}

}  // namespace

// The device copy of an FCI CRS's RDM plan: the string-pair lists, the per-element
// term lists and the alpha-beta excitation lists. It depends on the string tables
// only, so it is made on the first RDM call of a CRS and kept with it.
struct FciRdmPlan {
    int64_t npa = 0, npb = 0;
    size_t ndens = 0, nslots = 0;
    size_t off_da = 0, off_db = 0;
    size_t off_ga = 0, off_gb = 0, off_g0 = 0, off_g2 = 0;
    DevBuf<uint32_t> aI, aJ, bI, bJ;          // string pairs per spin
    DevBuf<uint32_t> dptr, didx;              // terms of every same-spin RDM element (CSR)
    DevBuf<int8_t> dcf;
    DevBuf<uint32_t> ap, bp;                  // alpha excitations ar < ac; beta ones and occupations
    DevBuf<uint64_t> apair, bpair;
    DevBuf<int8_t> asign, bsign;
    DevBuf<uint32_t> btp, bta, atp, ata;      // sums over beta strings by (br, bc), over alpha strings by z
};

// The split plan of a DOCI matrix, made on the first call (the mixed builds have it);
// null where the space is not split.
const DociSplit *doci_split_of(cigpu_crs &c, cudaStream_t s) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (!c.split_tried) {
        doci_split_make(c.L, c.nup, c.dim, c.split, s);
        CIGPU_CUDA(cudaStreamSynchronize(s));  // for callers on other streams
        c.split_tried = true;
    }
    return c.split && (int64_t)split_blocks(c.split.view) * kSplitRdmBlock <= c.dim &&
                   split_rdm_smem(c.split.view) <= kSplitRdmMaxSmem
               ? &c.split
               : nullptr;
}

// Adds the fixed-point sums A, B ([2][L][L], j <= k, zero before) of device vector c:
// by the general kernel, and through the split plan.
void doci_rdm_sums(const cigpu_crs &c, const double *c_dev, long long *sums, unsigned long long *err, cudaStream_t s) {
    const int th = ((c.L * (c.L + 1) / 2 + 31) / 32) * 32;  // one thread per pair j <= k
    const int64_t chunks = (c.dim + kDociChunk - 1) / kDociChunk;
    k_doci_rdm<<<(int)std::min<int64_t>(chunks, (int64_t)sm_count() * 4), th, 0, s>>>(c_dev, c.strings.p, c.dim, c.L, c.nup,
                                                                                      sums, err);
    count_launch();
}

void doci_rdm_split(const DociSplit &sp, const double *c_dev, long long *sums, cudaStream_t s) {
    static SmemLimit limit;
    CIGPU_CUDA(limit.raise(k_doci_rdm_split, kSplitRdmMaxSmem));
    DociSplitView v = sp.view;
    v.err = check_word_device();
    DevBuf<long long> fixed((size_t)v.D), low(sp.nlowbits);
    CIGPU_CUDA(cudaMemsetAsync(low.p, 0, low.bytes(), s));
    k_fix62<<<sm_count() * 8, 256, 0, s>>>(c_dev, v.D, fixed.p);
    k_doci_rdm_split<<<split_blocks(v), kSplitRdmThreads, split_rdm_smem(v), s>>>(v, fixed.p, sums, low.p);
    k_doci_rdm_low<<<v.s * v.s, 256, 0, s>>>(v, sp.nlowbits, low.p, sums);
    CIGPU_CUDA(cudaGetLastError());
    count_launch(3);
}

std::shared_ptr<FciRdmPlan> make_fci_rdm_plan(cigpu_crs &c, cudaStream_t s) {
    const int L = c.L, np = L * (L - 1) / 2;
    const int64_t L2 = (int64_t)L * L;
    const int64_t n2 = (int64_t)np * np;
    const SpinTables &ta = c.ta;
    const SpinTables &tb = (c.ndown == c.nup) ? c.ta : c.tb;
    Plan P;
    P.L = L;
    P.np = np;
    P.Da = ta.D;
    P.Db = tb.D;
    P.off_ga = 0;
    P.off_gb = L2;
    P.off_g0 = 2 * L2;
    P.off_g2 = P.off_g0 + n2;
    P.nslots = P.off_g2 + n2;
    // pair counts first (densities layout needs them)
    auto count_pairs = [&](const SpinTables &t) {
        size_t n = (size_t)t.D;
        for (int64_t I = 0; I < t.D; ++I) {
            for (int q = 0; q < t.ns; ++q) n += t.s_target[(size_t)I * t.ns + q] > (uint32_t)I;
            for (int q = 0; q < t.nd; ++q) n += t.d_target[(size_t)I * t.nd + q] > (uint32_t)I;
        }
        return n;
    };
    const size_t npa = count_pairs(ta), npb = count_pairs(tb);
    P.off_da = 0;
    P.off_db = npa;
    P.ndens = npa + npb;
    plan_spin(P, ta, true);
    plan_spin(P, tb, false);
    if (P.a.I.size() != npa || P.b.I.size() != npb) throw std::runtime_error("rdm plan: pair count mismatch");
    // CSR of the slot terms: a stable counting sort keeps each slot's generation order
    std::vector<uint32_t> ptr(P.nslots + 1, 0), idx(P.terms.size());
    std::vector<int8_t> cf(P.terms.size());
    for (const auto &t : P.terms) ++ptr[t.slot + 1];
    for (size_t q = 0; q < P.nslots; ++q) ptr[q + 1] += ptr[q];
    {
        std::vector<uint32_t> fill(ptr.begin(), ptr.end() - 1);
        for (const auto &t : P.terms) {
            const uint32_t at = fill[t.slot]++;
            idx[at] = t.dens;
            cf[at] = t.coef;
        }
    }
    auto R = std::make_shared<FciRdmPlan>();
    R->npa = (int64_t)npa;
    R->npb = (int64_t)npb;
    R->ndens = P.ndens;
    R->nslots = P.nslots;
    R->off_da = P.off_da;
    R->off_db = P.off_db;
    R->off_ga = P.off_ga;
    R->off_gb = P.off_gb;
    R->off_g0 = P.off_g0;
    R->off_g2 = P.off_g2;
    const ExcitationLists ea = excitation_lists(ta, false), eb = excitation_lists(tb, true);
    const SumLists sb = sum_lists(tb, true), sa = sum_lists(ta, false);
    R->aI = upload(P.a.I, s);
    R->aJ = upload(P.a.J, s);
    R->bI = upload(P.b.I, s);
    R->bJ = upload(P.b.J, s);
    R->dptr = upload(ptr, s);
    R->didx = upload(idx, s);
    R->dcf = upload(cf, s);
    R->ap = upload(ea.ptr, s);
    R->apair = upload(ea.pair, s);
    R->asign = upload(ea.sign, s);
    R->bp = upload(eb.ptr, s);
    R->bpair = upload(eb.pair, s);
    R->bsign = upload(eb.sign, s);
    R->btp = upload(sb.ptr, s);
    R->bta = upload(sb.at, s);
    R->atp = upload(sa.ptr, s);
    R->ata = upload(sa.at, s);
    CIGPU_CUDA(cudaStreamSynchronize(s));  // the host vectors go out of scope
    return R;
}

// Matrices of at most this many bytes (10 orbitals) leave the device in one copy: on small
// spaces the four copies to the caller's pageable memory are a good part of the call (L=6
// 3a3b 114 -> 89 us).
constexpr size_t kOneCopyBytes = 128 * 1024;

void crs_rdm(cigpu_crs &c, const double *c_dev, double *rdm1, double *aa, double *ab, double *bb, cudaStream_t s) {
    if (c.method == CIGPU_DETS) {
        dets_rdm(c, c_dev, rdm1, aa, ab, bb, s);
        return;
    }
    const int L = c.L, np = L * (L - 1) / 2;
    const int64_t L2 = (int64_t)L * L;
    const int64_t n1 = 2 * L2, n2 = (int64_t)np * np, n3 = L2 * L2;
    DevBuf<double> out(n1 + 2 * n2 + n3);
    double *o1 = out.p, *oaa = out.p + n1, *obb = out.p + n1 + n2, *oab = out.p + n1 + 2 * n2;
    Trace tr("rdm", s);
    if (c.method == CIGPU_DOCI) {
        if (L * L > 1024) throw std::invalid_argument("DOCI RDM needs L <= 32");
        CIGPU_CUDA(cudaMemsetAsync(out.p, 0, sizeof(double) * out.n, s));
        DevBuf<long long> sums((size_t)2 * L2);
        CIGPU_CUDA(cudaMemsetAsync(sums.p, 0, sums.bytes(), s));
        if (const DociSplit *sp = doci_split_of(c, s))
            doci_rdm_split(*sp, c_dev, sums.p, s);
        else
            doci_rdm_sums(c, c_dev, sums.p, check_word_device(), s);
        k_doci_rdm_finish<<<(int)((L2 + 255) / 256), 256, 0, s>>>(sums.p, L, np, o1, oaa, oab, obb);
        CIGPU_CUDA(cudaGetLastError());
        count_launch();
        CIGPU_CUDA(cudaStreamSynchronize(s));
        tr.mark("doci kernels");
    } else {
        if (L > 32) throw std::invalid_argument("FCI RDM needs L <= 32");
        if (!c.rdm_plan) {
            c.rdm_plan = make_fci_rdm_plan(c, s);
            tr.mark("host plan");
        }
        const FciRdmPlan &R = *c.rdm_plan;
        const SpinTables &ta = c.ta;
        const SpinTables &tb = (c.ndown == c.nup) ? c.ta : c.tb;
        // C^T for the beta densities
        DevBuf<double> Ct((size_t)c.dim);
        {
            dim3 grid((unsigned)((tb.D + 31) / 32), (unsigned)((ta.D + 31) / 32));
            k_transpose<<<grid, dim3(32, 8), 0, s>>>(c_dev, ta.D, tb.D, Ct.p);
            count_launch();
        }
        const size_t sm = sizeof(double) * 2 * (size_t)tb.D;
        if (np > 0 && sm > 200 * 1024) throw std::invalid_argument("FCI RDM: beta string space too large");
        DevBuf<double> dens(R.ndens);
        const int G = sm_count() * 8;
        unsigned long long *ew = check_word_device();
        const auto pair_grid = [](int64_t n) {  // a batch of pairs per warp
            constexpr int64_t per = kPairBatch * (kRdmThreads / 32);
            return (unsigned)std::min<int64_t>((n + per - 1) / per, INT32_MAX);
        };
        k_pair_dens<<<pair_grid(R.npa), kRdmThreads, 0, s>>>(c_dev, tb.D, R.aI.p, R.aJ.p, R.npa, dens.p + R.off_da, ta.D, ew);
        k_pair_dens<<<pair_grid(R.npb), kRdmThreads, 0, s>>>(Ct.p, ta.D, R.bI.p, R.bJ.p, R.npb, dens.p + R.off_db, tb.D, ew);
        count_launch(2);
        tr.mark("pair densities");
        DevBuf<double> acc(R.nslots);
        k_slot_gather<<<G, kRdmThreads, 0, s>>>(R.dptr.p, R.didx.p, R.dcf.p, dens.p, (int64_t)R.nslots, acc.p,
                                                (int64_t)R.ndens, ew);
        count_launch();
        tr.mark("slot sums");
        // the alpha-beta block: string sums of a batch of excitations (at most
        // kAbBatchBytes of them), then the sums over the strings
        constexpr size_t kAbBatchBytes = size_t(64) << 20;
        DevBuf<double> t1((size_t)std::max(np, 1) * L2), t2((size_t)(np + L) * L);
        auto batches = [&](int nq, size_t per_q, auto &&f) {
            const int most = (int)std::min<size_t>({(size_t)std::max(nq, 1), 65535,
                                                    std::max<size_t>(1, kAbBatchBytes / (per_q * sizeof(double)))});
            DevBuf<double> g((size_t)most * per_q);
            for (int q0 = 0; q0 < nq; q0 += most) f(g.p, q0, std::min(most, nq - q0));
        };
        const int nsb = tb.ns;
        batches(np, (size_t)(nsb + 1) * tb.D, [&](double *g, int q0, int nq) {
            const int64_t per = (int64_t)(nsb + 1) * tb.D;
            const unsigned tiles = (unsigned)((tb.D + kAbThreads - 1) / kAbThreads);
            auto go = [&](auto kern, int x) {
                // one fixed limit: concurrent callers (server workers) never lower it
                CIGPU_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
                kern<<<dim3(tiles, (unsigned)std::max(1, (nsb + x - 1) / x), (unsigned)nq), kAbThreads, sm, s>>>(
                    c_dev, tb.D, c.fp.b.s_target, nsb, R.ap.p, R.apair.p, R.asign.p, q0, g, ta.D, ew);
            };
            if ((int64_t)tiles * nq >= 3 * (int64_t)sm_count())
                go(k_string_sums<kAbWide>, kAbWide);
            else
                go(k_string_sums<kAbNarrow>, kAbNarrow);
            k_sum_strings<<<(unsigned)((nq * L2 + 3) / 4), 128, 0, s>>>(g, per, R.btp.p, R.bta.p, (int)L2, nq,
                                                                        t1.p + (int64_t)q0 * L2, ew);
            count_launch(2);
        });
        tr.mark("alpha-beta doubles");
        batches(np + L, (size_t)ta.D, [&](double *g, int q0, int nq) {
            const dim3 grid((unsigned)((ta.D + kAbThreads - 1) / kAbThreads), 1, (unsigned)nq);
            k_string_sums_ident<<<grid, kAbThreads, 0, s>>>(Ct.p, ta.D, R.bp.p, R.bpair.p, R.bsign.p, q0, g, tb.D, ew);
            k_sum_strings<<<(unsigned)((nq * L + 3) / 4), 128, 0, s>>>(g, ta.D, R.atp.p, R.ata.p, L, nq,
                                                                       t2.p + (int64_t)q0 * L, ew);
            count_launch(2);
        });
        tr.mark("alpha occupations");
        k_rdm_assemble<<<G, kRdmThreads, 0, s>>>(acc.p, t1.p, t2.p, L, np, R.off_ga, R.off_gb, R.off_g0, R.off_g2, o1, oaa,
                                                 oab, obb);
        CIGPU_CUDA(cudaGetLastError());
        count_launch();
        CIGPU_CUDA(cudaStreamSynchronize(s));
    }
    if (out.bytes() <= kOneCopyBytes) {
        std::vector<double> host(out.n);
        CIGPU_CUDA(cudaMemcpyAsync(host.data(), out.p, out.bytes(), cudaMemcpyDeviceToHost, s));
        CIGPU_CUDA(cudaStreamSynchronize(s));
        const double *h = host.data();
        if (rdm1) std::copy(h, h + n1, rdm1);
        if (aa) std::copy(h + n1, h + n1 + n2, aa);
        if (bb) std::copy(h + n1 + n2, h + n1 + 2 * n2, bb);
        if (ab) std::copy(h + n1 + 2 * n2, h + out.n, ab);
    } else {
        if (rdm1) CIGPU_CUDA(cudaMemcpyAsync(rdm1, o1, sizeof(double) * n1, cudaMemcpyDeviceToHost, s));
        if (aa) CIGPU_CUDA(cudaMemcpyAsync(aa, oaa, sizeof(double) * n2, cudaMemcpyDeviceToHost, s));
        if (bb) CIGPU_CUDA(cudaMemcpyAsync(bb, obb, sizeof(double) * n2, cudaMemcpyDeviceToHost, s));
        if (ab) CIGPU_CUDA(cudaMemcpyAsync(ab, oab, sizeof(double) * n3, cudaMemcpyDeviceToHost, s));
        CIGPU_CUDA(cudaStreamSynchronize(s));
    }
    tr.mark("assemble + copy out");
}

int doci_pair_partials() { return 1; }

void doci_pair_matrices(cigpu_crs &c, const double *c_dev, double *partial, double *Pm, double *Dm, cudaStream_t s) {
    if (c.method != CIGPU_DOCI || c.L > 32) throw std::invalid_argument("DOCI pair matrices need a DOCI CRS, L <= 32");
    const int L = c.L;
    long long *sums = reinterpret_cast<long long *>(partial);
    CIGPU_CUDA(cudaMemsetAsync(sums, 0, sizeof(long long) * 2 * L * L, s));
    doci_rdm_sums(c, c_dev, sums, check_word_device(), s);
    k_doci_pairs_finish<<<(L * L + 255) / 256, 256, 0, s>>>(sums, L, Pm, Dm);
    CIGPU_CUDA(cudaGetLastError());
    count_launch();
}

}  // namespace cigpu

// ---------------------------------------------------------------------------
// DOCI RDMs without any device allocation (cigpu_rdm_doci_noalloc).
//
// Some callers cannot allocate device memory at the point where they need the
// RDMs: a host framework that hands out all device memory from its own fixed
// pool and forbids cudaMalloc on its request path, or a latency-bound loop where
// the implicit device synchronisation of cudaMalloc/cudaFree would stall work
// queued by others. For them the sums of the DOCI RDM kernel live in a fixed
// array inside this library instead of in allocated scratch.
//
// The array below is file-scope device memory: every GPU that loads the library
// holds it (16 KiB) until the process exits. Host code must not take its name as
// a device address; the address is looked up once per device with
// cudaGetSymbolAddress (on the first call on that device, which should therefore
// come before any stream capture) and kept for the life of the process, so it
// does not survive a cudaDeviceReset of that device. The call runs on the current
// device, which must be the one the CRS was built on (CIGPU_EINVAL otherwise).
// Every call shares the array and leaves its contents behind: calls that overlap
// on the GPU race on it.
namespace cigpu {
namespace {

constexpr int kNoAllocSums = 2 * kDociMaxL * kDociMaxL;  // 16 KiB: [2][L][L], L <= 32

static __device__ __align__(256) long long g_doci_rdm_scratch[kNoAllocSums];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
long long *g_scratch_addr[kMaxDevices] = {nullptr};

// Device address of the scratch array on the current device (set up once per device).
cudaError_t scratch_address(long long **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_doci_rdm_scratch);
        if (e != cudaSuccess) return e;
        g_scratch_addr[dev] = static_cast<long long *>(p);
    }
    *out = g_scratch_addr[dev];
    return cudaSuccess;
}

}  // namespace
}  // namespace cigpu

extern "C" int cigpu_rdm_doci_noalloc(cigpu_crs *crs, const double *c, double *rdm1, double *rdm2_aa,
                                      double *rdm2_ab, double *rdm2_bb, cigpu_stream stream) {
    using namespace cigpu;
    if (!crs || !c || !rdm1 || !rdm2_aa || !rdm2_ab || !rdm2_bb) return CIGPU_EINVAL;
    if (crs->method != CIGPU_DOCI) return CIGPU_EINVAL;
    const int L = crs->L, np = L * (L - 1) / 2;
    const int64_t L2 = (int64_t)L * L;
    // one thread per orbital pair (j, k), and 2 L^2 sums must fit
    if (L2 > 1024) return CIGPU_ENOTSUP;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return CIGPU_ECUDA;
    if (dev != crs->device) return CIGPU_EINVAL;  // the matrix and the scratch must share a device
    long long *sums = nullptr;
    cudaError_t e = scratch_address(&sums);
    if (e != cudaSuccess) {
        std::fprintf(stderr, "cigpu: scratch address lookup failed: %s\n", cudaGetErrorString(e));
        return CIGPU_ECUDA;
    }
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : crs->stream;
    // the finishing kernel only writes the nonzero DOCI entries: clear the outputs
    if (cudaMemsetAsync(rdm1, 0, sizeof(double) * 2 * L2, s) != cudaSuccess ||
        cudaMemsetAsync(rdm2_aa, 0, sizeof(double) * np * np, s) != cudaSuccess ||
        cudaMemsetAsync(rdm2_bb, 0, sizeof(double) * np * np, s) != cudaSuccess ||
        cudaMemsetAsync(rdm2_ab, 0, sizeof(double) * L2 * L2, s) != cudaSuccess)
        return CIGPU_ECUDA;
    if (cudaMemsetAsync(sums, 0, sizeof(long long) * 2 * L2, s) != cudaSuccess) return CIGPU_ECUDA;
    doci_rdm_sums(*crs, c, sums, nullptr, s);  // no error word: allocates nothing
    k_doci_rdm_finish<<<(int)((L2 + 255) / 256), 256, 0, s>>>(sums, L, np, rdm1, rdm2_aa, rdm2_ab, rdm2_bb);
    if (cudaGetLastError() != cudaSuccess) return CIGPU_ECUDA;
    count_launch();
    return CIGPU_OK;
}
