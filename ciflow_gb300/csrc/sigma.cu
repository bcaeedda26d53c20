// FP32 product of the mixed method for FCI: a direct-CI sigma vector, the same-spin
// part from the strings' own matrices and the opposite-spin part factorised.
//
// With E^s_pq = a+_ps a_qs for spin s and real orbitals,
//   H = T^a + T^b + sum_pqrs (pq|rs) E^a_pq E^b_rs,
// T^s the one- and two-electron part of one spin (a sparse matrix over its strings: the
// diagonal, singles and doubles of the string tables), and a factorisation
// (pq|rs) = sum_k s_k F^k_pq F^k_rs with symmetric F^k (a pivoted Cholesky factor of the
// pair matrix, s_k = 1; eigenpairs with their signs when the integrals are indefinite)
// gives
//   y = T^a x + x T^b + sum_k A^a_k (s_k A^b_k x),   A^s_k = sum_pq F^k_pq E^s_pq.
// Only beta excitations form z_k = A^b_k x and only alpha ones act on it: half the
// factor work of squaring A_k = A^a_k + A^b_k (the form before: 72 excitations x 16
// factors twice per row at L=12 6a6b, now 36 twice and 522 same-spin elements).
//
// The alpha excitations are applied in two steps, so that the R factors of a row are
// read once and not once per excitation: a row J forms, for each of its alpha
// excitations (J -> I by pq), the one number
//   w = sign sum_k s_k F^k_pq z_k(J)
// into W[I][e'] (e' the excitation of I that leads back to J), and a row I then adds its
// n_a (L - n_a) numbers, a contiguous read. Gathering the factors instead moved 64 bytes
// per excitation through L2 (2 x 3.9 GB per product), which bound the product.
//
// One product is three launches:
//   k_sigma_pad    x padded to whole tiles and transposed;
//   k_sigma_parts  two kinds of block: pairs of blocks form W on 64 x 64 string tiles
//                  (opposite_tile), others u = x T^b on the transposed vectors
//                  (same_rows);
//   k_sigma_sum    y = T^a x + u + the sums of W.
// L=12 6a6b, rank 16: 308 -> 193 us per product (k_sigma_parts 145, k_sigma_sum 60); L=10 5a5b: the stored
// values 38.5, the operator 15.9 us.
//
// This replaces only the mixed method's FP32 correction products: the operator
// equals the reference Hamiltonian up to FP32 rounding and the factorisation's
// truncation (a remaining pair diagonal below 1e-10 of the largest), while the FP64 anchor
// products and residuals keep using the stored matrix, whose elements are the
// reference's bit for bit; the residual the solver reports is that exact one.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "checked.cuh"
#include "sigma.cuh"
#include "small_eigh.h"

namespace cigpu {

namespace {

namespace cg = cooperative_groups;

constexpr int kTile = kSigmaTile;
constexpr int kC = kSigmaChunk;
constexpr int kPanel = 32;     // columns of a same-spin block
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kHalf = kC / 2;  // factors of a pass that one block of a pair forms
constexpr int kZk = kTile * (kTile + 1);  // one factor of the staged tile

// ---- packed FP32 pairs ----
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ float signed_by(float v, uint32_t odd) {
    return __uint_as_float(__float_as_uint(v) ^ (odd << 31));
}

// ---- string tables of the operator ----
// Rows of T^s: {self, diagonal}, singles, doubles, padding {self, 0}; `ne` per string.
__global__ void k_sigma_rows(const SpinDev t, int ne, uint2 *__restrict__ rows, unsigned long long *err) {
    const int64_t total = t.D * ne;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t S = i / ne;
        const int e = (int)(i - S * ne);
        uint32_t J = (uint32_t)S;
        float v = 0.f;
        if (e == 0) {
            v = (float)t.diag[S];
        } else if (e <= t.ns) {
            const int64_t at = S * t.ns + e - 1;
            J = t.s_target[at];
            v = signed_by((float)t.s_part[at], (t.s_info[at] >> 24) & 1u);
        } else if (e <= t.ns + t.nd) {
            const int64_t at = S * t.nd + e - 1 - t.ns;
            J = t.d_target[at];
            v = (float)t.d_val[at];
        }
        if (!CIGPU_CHECK(err, index_ok(J, (uint64_t)t.D), kCheckColumn, J)) {
            J = (uint32_t)S;
            v = 0.f;
        }
        rows[i] = make_uint2(J, __float_as_uint(v));
    }
    (void)err;
}

// W row that excitation e of string J feeds: target I, place of the excitation that
// leads back (I's occupied orbital ascending, then its empty one; see the tables).
__global__ void k_sigma_back(const SpinDev t, int L, uint32_t *__restrict__ w) {
    const int64_t total = t.D * t.ns;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t I = t.s_target[i], info = t.s_info[i];
        const int j = (info >> 12) & 63, l = (info >> 18) & 63;  // J holds j, I holds l in its place
        int at_l = 0, below_j = 0;
        for (int m = 0; m < t.n; ++m) {
            const int o = t.occ[(int64_t)I * t.n + m];
            at_l += o < l;
            below_j += o < j;
        }
        w[i] = I * (uint32_t)t.ns + (uint32_t)(at_l * (L - t.n) + j - below_j);
    }
}

// Single excitations as the opposite-spin tiles read them: {target, pair << 1 | odd},
// pair = lo * L + hi; with `back`, the W row in place of the target.
__global__ void k_sigma_singles(const SpinDev t, int L, const uint32_t *__restrict__ back, uint2 *__restrict__ out,
                                unsigned long long *err) {
    const int64_t total = t.D * t.ns;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t w = t.s_info[i];
        uint32_t J = back ? back[i] : t.s_target[i];
        if (!CIGPU_CHECK(err, index_ok(J, (uint64_t)(back ? total : t.D)), kCheckColumn, J)) J = 0;
        out[i] = make_uint2(J, (((w & 63u) * (uint32_t)L + ((w >> 6) & 63u)) << 1) | ((w >> 24) & 1u));
    }
    (void)err;
}

struct SigmaArgs {
    int L, R, nsa, nsb;
    int64_t Da, Db, Pa, Pb;
    const uint2 *sa, *sb;             // single excitations: alpha {W row, pair}, beta {target, pair}
    const float *F, *G, *ga, *fb;     // as in SigmaOp
    const uint2 *rows;                // the beta strings' same-spin rows
    int ne;
    int tiles, panels, chunks, per;   // opposite tiles; same-spin panels and row chunks
    int slabs, slab_r;                // sets of W and yd, each of slab_r factors (see sigma_slabs)
    int panel_rows;                   // rows of xT a same-spin block holds in shared memory (0: none)
    const float *xT;
    float *W, *yd, *uT;
};

// x [Da][Db] into xp [Da][Pb] (zero past Db) and xT [Db][Pa] (zero past Da).
__global__ void k_sigma_pad(const float *__restrict__ x, int64_t Da, int64_t Db, int64_t Pa, int64_t Pb,
                            float *__restrict__ xp, float *__restrict__ xT) {
    constexpr int kSide = 32;
    __shared__ float tile[kSide][kSide + 1];
    const int64_t r0 = (int64_t)blockIdx.y * kSide, c0 = (int64_t)blockIdx.x * kSide;
    for (int i = threadIdx.y; i < kSide; i += blockDim.y) {
        const int64_t r = r0 + i, c = c0 + threadIdx.x;
        const float v = r < Da && c < Db ? x[r * Db + c] : 0.f;
        tile[i][threadIdx.x] = v;
        if (r < Da) xp[r * Pb + c] = v;
    }
    __syncthreads();
    for (int i = threadIdx.y; i < kSide; i += blockDim.y) {
        const int64_t c = c0 + i, r = r0 + threadIdx.x;
        if (c < Db) xT[c * Pa + r] = tile[threadIdx.x][i];
    }
}

// Dynamic shared memory of an opposite-spin tile.
size_t opposite_smem(int L) { return sizeof(float) * ((size_t)L * L * (kHalf + kC) + (size_t)kHalf * kZk); }

// W and yd of a 64 alpha x 64 beta tile, by the two blocks of a cluster. Passes of 16
// factors: block h forms z_k for its eight of them -- a warp takes a beta string, its
// lanes the tile's alpha strings, two each, so the excitation and with it F is the same
// for the warp -- into its shared memory; after the cluster's barrier it takes half the
// alpha strings, a warp each with its lanes on the beta strings, two each, reads all 16
// z_k of its rows (half of them from the other block's shared memory) and forms w, the
// pair and with it s_k F the same for the warp again. A coefficient read from shared
// memory costs the 128 bytes per clock of its way back to the registers even when all
// lanes read one address, and that bounds the tile: with two rows per lane it serves
// two multiply-adds. The excitations' descriptors
// are read a step ahead (without, their latency cost 20 of 165 us).
__device__ __forceinline__ void opposite_tile(const SigmaArgs &a, float *sm) {
    auto cluster = cg::this_cluster();
    const int half = (int)cluster.block_rank();
    const int L2 = a.L * a.L, nsa = a.nsa, nsb = a.nsb;
    float *Fs = sm, *Gs = Fs + L2 * kHalf;  // [L2][8] of this block's factors, [L2][16]
    float *z = Gs + L2 * kC;                // [8][kTile alpha][kTile + 1 beta]
    const int slab = (int)(blockIdx.x / 2) / a.tiles, tile = (int)(blockIdx.x / 2) - slab * a.tiles;
    const int c_begin = slab * a.slab_r, c_end = min(a.R, c_begin + a.slab_r);
    float *W = a.W + (int64_t)slab * a.Da * nsa * a.Pb, *yd = a.yd + (int64_t)slab * a.Da * a.Pb;
    const int64_t tb = (int64_t)(tile % (int)(a.Pb / kTile)) * kTile, ta = (int64_t)(tile / (int)(a.Pb / kTile)) * kTile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = c_begin; c < c_end; c += kC) {
        if (c > c_begin) cluster.sync();  // both blocks are done with the factors and z
        const float4 *F4 = reinterpret_cast<const float4 *>(a.F) + (size_t)(c / kC) * L2 * (kC / 4);
        const float4 *G4 = reinterpret_cast<const float4 *>(a.G) + (size_t)(c / kC) * L2 * (kC / 4);
        for (int i = threadIdx.x; i < L2 * (kHalf / 4); i += kThreads)
            reinterpret_cast<float4 *>(Fs)[i] = __ldg(F4 + (i / 2) * (kC / 4) + half * 2 + (i & 1));
        for (int i = threadIdx.x; i < L2 * (kC / 4); i += kThreads) reinterpret_cast<float4 *>(Gs)[i] = __ldg(G4 + i);
        __syncthreads();
        const int k0 = c + half * kHalf;
        for (int cl = warp; cl < kTile; cl += kWarps) {
            const int64_t Ib = tb + cl;
            uint64_t acc[2][kHalf / 2];
            if (Ib < a.Db) {
                const float *xc = a.xT + ta + lane;  // rows of Pa, zero past Da
                const float x0 = __ldg(xc + Ib * a.Pa), x1 = __ldg(xc + Ib * a.Pa + 32);
#pragma unroll
                for (int k = 0; k < kHalf / 2; ++k) {
                    const float f0 = __ldg(a.fb + (int64_t)(k0 + 2 * k) * a.Db + Ib),
                                f1 = __ldg(a.fb + (int64_t)(k0 + 2 * k + 1) * a.Db + Ib);
                    acc[0][k] = pack2(x0 * f0, x0 * f1);
                    acc[1][k] = pack2(x1 * f0, x1 * f1);
                }
                const uint2 *ex = a.sb + Ib * nsb;
                uint2 w[4];  // the next four excitations
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (u < nsb) w[u] = __ldg(ex + u);
                for (int e = 0; e < nsb; e += 4) {  // eight loads of x in flight
                    uint2 v[4];
                    float u0[4], u1[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = w[u];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (e + 4 + u < nsb) w[u] = __ldg(ex + e + 4 + u);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (e + u < nsb) {
                            u0[u] = signed_by(__ldg(xc + (int64_t)v[u].x * a.Pa), v[u].y & 1u);
                            u1[u] = signed_by(__ldg(xc + (int64_t)v[u].x * a.Pa + 32), v[u].y & 1u);
                        }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (e + u < nsb) {
                            const uint64_t p0 = pack2(u0[u], u0[u]), p1 = pack2(u1[u], u1[u]);
                            const ulonglong2 *f = reinterpret_cast<const ulonglong2 *>(Fs + (v[u].y >> 1) * kHalf);
#pragma unroll
                            for (int k = 0; k < kHalf / 4; ++k) {
                                const ulonglong2 f2 = f[k];
                                acc[0][2 * k] = fma2(f2.x, p0, acc[0][2 * k]);
                                acc[1][2 * k] = fma2(f2.x, p1, acc[1][2 * k]);
                                acc[0][2 * k + 1] = fma2(f2.y, p0, acc[0][2 * k + 1]);
                                acc[1][2 * k + 1] = fma2(f2.y, p1, acc[1][2 * k + 1]);
                            }
                        }
                }
            } else {
#pragma unroll
                for (int k = 0; k < kHalf / 2; ++k) acc[0][k] = acc[1][k] = 0;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float *zc = z + (lane + 32 * h) * (kTile + 1) + cl;
#pragma unroll
                for (int k = 0; k < kHalf / 2; ++k) {
                    float lo, hi;
                    unpack2(acc[h][k], lo, hi);
                    zc[2 * k * kZk] = lo;
                    zc[(2 * k + 1) * kZk] = hi;
                }
            }
        }
        cluster.sync();
        const float *z0 = cluster.map_shared_rank(z, 0), *z1 = cluster.map_shared_rank(z, 1);
        for (int r = half * (kTile / 2) + warp; r < (half + 1) * (kTile / 2); r += kWarps) {
            const int64_t Ia = ta + r;
            if (Ia >= a.Da) continue;
            uint64_t zz[2][kC / 2];
            float d[2] = {0.f, 0.f};
#pragma unroll
            for (int k = 0; k < kC / 2; ++k) {
                const float *zr = (k < kHalf / 2 ? z0 + 2 * k * kZk : z1 + (2 * k - kHalf) * kZk) + r * (kTile + 1) + lane;
                const float g0 = __ldg(a.ga + (int64_t)(c + 2 * k) * a.Da + Ia), g1 = __ldg(a.ga + (int64_t)(c + 2 * k + 1) * a.Da + Ia);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float lo = zr[32 * h], hi = zr[kZk + 32 * h];
                    zz[h][k] = pack2(lo, hi);
                    d[h] += g0 * lo + g1 * hi;
                }
            }
            float *ydr = yd + Ia * a.Pb + tb + lane;
#pragma unroll
            for (int h = 0; h < 2; ++h) ydr[32 * h] = c == c_begin ? d[h] : ydr[32 * h] + d[h];
            const uint2 *ex = a.sa + Ia * nsa;
            float *Wc = W + tb + lane;
            uint2 w[2];  // the next two excitations
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (u < nsa) w[u] = __ldg(ex + u);
            for (int e = 0; e < nsa; e += 2) {
                uint2 v[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) v[u] = w[u];
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (e + 2 + u < nsa) w[u] = __ldg(ex + e + 2 + u);
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    if (e + u < nsa) {
                        const ulonglong2 *g = reinterpret_cast<const ulonglong2 *>(Gs + (v[u].y >> 1) * kC);
                        uint64_t s[2][2] = {{0, 0}, {0, 0}};
#pragma unroll
                        for (int k = 0; k < kC / 4; ++k) {
                            const ulonglong2 g2 = g[k];
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                s[h][0] = fma2(g2.x, zz[h][2 * k], s[h][0]);
                                s[h][1] = fma2(g2.y, zz[h][2 * k + 1], s[h][1]);
                            }
                        }
                        float *at = Wc + (int64_t)v[u].x * a.Pb;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float p0, p1, p2, p3;
                            unpack2(s[h][0], p0, p1);
                            unpack2(s[h][1], p2, p3);
                            const float x = signed_by((p0 + p1) + (p2 + p3), v[u].y & 1u);
                            at[32 * h] = c == c_begin ? x : at[32 * h] + x;
                        }
                    }
            }
        }
    }
    cluster.sync();  // the other block may still be reading this one's z
}

// Same-spin rows. A warp takes four rows of T, a group of 8 lanes each, and 32
// consecutive columns of the other spin, 16 bytes a lane: an element is half a broadcast
// 16-byte shared-memory read, one 16-byte read of X and four multiply-adds. Bound by the
// 128 bytes per clock that come back from L1 or shared memory.
constexpr int kSameE = 16;                // elements staged per warp and row
constexpr int kSameRow = 2 * kSameE + 4;  // words: rows of a warp's four on different banks

__device__ __forceinline__ void fma4(float4 &a, float s, const float4 x) {
    a.x += s * x.x;
    a.y += s * x.y;
    a.z += s * x.z;
    a.w += s * x.w;
}

// sum_e value_e X[target_e] over the elements [eb, ee), multiples of 8, of row S of the
// lane's group (rows of ne elements); Xc: X at the lane's columns, rows P apart (in shared
// or global memory); st: the warp's staging area.
template <bool SHARED>
__device__ __forceinline__ float4 same_row(const uint2 *__restrict__ rows, int ne, int eb, int ee, int64_t S,
                                           const float *Xc, int64_t P, uint32_t *st) {
    const int lane = threadIdx.x & 31, g = lane >> 3, l = lane & 7;
    const uint32_t *mine = st + g * kSameRow;
    float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
    // each lane brings two elements of its group's row, one step ahead
    const uint4 *src = reinterpret_cast<const uint4 *>(rows + S * ne + eb) + l;
    uint4 next = eb + 2 * l < ee ? __ldg(src) : make_uint4(0u, 0u, 0u, 0u);
    for (int e0 = eb; e0 < ee; e0 += kSameE) {
        __syncwarp();
        const int n = min(kSameE, ee - e0);  // a multiple of 8
        *reinterpret_cast<uint4 *>(st + g * kSameRow + 4 * l) = next;
        __syncwarp();
        src += kSameE / 2;
        if (e0 + kSameE + 2 * l < ee) next = __ldg(src);
        for (int e = 0; e < n; e += 8) {
            uint4 d[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) d[u] = *reinterpret_cast<const uint4 *>(mine + 2 * e + 4 * u);
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if constexpr (SHARED) {
                    v[2 * u] = *reinterpret_cast<const float4 *>(Xc + d[u].x * (uint32_t)P);
                    v[2 * u + 1] = *reinterpret_cast<const float4 *>(Xc + d[u].z * (uint32_t)P);
                } else {
                    v[2 * u] = __ldg(reinterpret_cast<const float4 *>(Xc + (int64_t)d[u].x * P));
                    v[2 * u + 1] = __ldg(reinterpret_cast<const float4 *>(Xc + (int64_t)d[u].z * P));
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                fma4(a0, __uint_as_float(d[u].y), v[2 * u]);
                fma4(a1, __uint_as_float(d[u].w), v[2 * u + 1]);
            }
        }
    }
    return make_float4(a0.x + a1.x, a0.y + a1.y, a0.z + a1.z, a0.w + a1.w);
}

// uT rows of one panel (32 alpha columns) and one chunk of beta strings. Where the
// panel fits, xT's 32 columns are copied to shared memory first.
__device__ __forceinline__ void same_rows(const SigmaArgs &a, int block, float *sm) {
    __shared__ __align__(16) uint32_t stage[kWarps][4 * kSameRow];
    const int panel = block / a.chunks, chunk = block - panel * a.chunks;
    if (panel >= a.panels) return;  // the odd block of the last cluster
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 3, l = lane & 7;
    const int64_t col = (int64_t)panel * kPanel;
    if (a.panel_rows > 0) {
        for (int i = threadIdx.x; i < (int)a.Db * (kPanel / 4); i += kThreads)
            reinterpret_cast<float4 *>(sm)[i] =
                __ldg(reinterpret_cast<const float4 *>(a.xT + (int64_t)(i >> 3) * a.Pa + col) + (i & 7));
        __syncthreads();
    }
    const int64_t groups = (a.Db + 3) / 4, g1 = min(groups, (int64_t)(chunk + 1) * a.per);
    for (int64_t q = (int64_t)chunk * a.per + warp; q < g1; q += kWarps) {
        const int64_t S = min(4 * q + g, a.Db - 1);  // rows past the last repeat it, and are not written
        const float4 r = a.panel_rows > 0 ? same_row<true>(a.rows, a.ne, 0, a.ne, S, sm + 4 * l, kPanel, stage[warp])
                                          : same_row<false>(a.rows, a.ne, 0, a.ne, S, a.xT + col + 4 * l, a.Pa, stage[warp]);
        if (4 * q + g < a.Db) *reinterpret_cast<float4 *>(a.uT + S * a.Pa + col + 4 * l) = r;
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) k_sigma_parts(const SigmaArgs a) {
    extern __shared__ __align__(16) float sm[];
    const int opposite = 2 * a.tiles * a.slabs;
    if ((int)blockIdx.x < opposite)
        opposite_tile(a, sm);
    else
        same_rows(a, (int)blockIdx.x - opposite, sm);
}

// y(Ia, Ib) = (T^a x) + yd + the sum of W's rows of Ia + uT(Ib, Ia), 32 beta columns per
// panel (blockIdx.y), alpha strings in chunks (blockIdx.x) of `per` groups of four. SPLIT:
// chunks of at most half as many groups as a block has warps give each group two warps,
// which take half of its elements and of its numbers each: such a block is one chain of
// gathers per warp, and half of it is half the time (L=20 4a1b, 792 elements a row: the
// product among others 101 -> 78 us with it).
template <bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
    k_sigma_sum(const SigmaArgs a, const uint2 *__restrict__ rows, int ne, int per, const float *__restrict__ xp,
                float *__restrict__ y) {
    __shared__ __align__(16) uint32_t stage[kWarps][4 * kSameRow];
    __shared__ float4 second[SPLIT ? kWarps / 2 : 1][32];
    constexpr int kGroups = SPLIT ? kWarps / 2 : kWarps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 3, l = lane & 7;
    const int part = SPLIT ? warp / kGroups : 0;
    const int eb = part ? ne / 16 * 8 : 0, ee = SPLIT && !part ? ne / 16 * 8 : ne;
    const int wb = part ? a.nsa / 2 : 0, we = SPLIT && !part ? a.nsa / 2 : a.nsa;
    const int64_t P = a.Pb, col = (int64_t)blockIdx.y * kPanel + 4 * l;
    const int64_t groups = (a.Da + 3) / 4, g1 = min(groups, (int64_t)(blockIdx.x + 1) * per);
    for (int64_t q = (int64_t)blockIdx.x * per + warp % kGroups; SPLIT || q < g1; q += kGroups) {
        const bool live = !SPLIT || q < g1;
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        if (live) {
            const int64_t S = min(4 * q + g, a.Da - 1);
            const float4 r = same_row<false>(rows, ne, eb, ee, S, xp + col, P, stage[warp]);
            float4 b0 = make_float4(0.f, 0.f, 0.f, 0.f), b1 = b0;
            for (int slab = 0; slab < a.slabs; ++slab) {
                const float *w = a.W + ((int64_t)slab * a.Da + S) * a.nsa * P + col;
                if (!part) fma4(b0, 1.f, __ldg(reinterpret_cast<const float4 *>(a.yd + ((int64_t)slab * a.Da + S) * P + col)));
                int e = wb;
                for (; e + 8 <= we; e += 8) {  // read once: streamed past L1
                    float4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = __ldcs(reinterpret_cast<const float4 *>(w + (int64_t)(e + u) * P));
#pragma unroll
                    for (int u = 0; u < 8; u += 2) {
                        fma4(b0, 1.f, v[u]);
                        fma4(b1, 1.f, v[u + 1]);
                    }
                }
                for (; e < we; ++e) fma4(b0, 1.f, __ldcs(reinterpret_cast<const float4 *>(w + (int64_t)e * P)));
            }
            c[0] = r.x + (b0.x + b1.x);
            c[1] = r.y + (b0.y + b1.y);
            c[2] = r.z + (b0.z + b1.z);
            c[3] = r.w + (b0.w + b1.w);
        }
        if constexpr (SPLIT) {
            if (part) second[warp % kGroups][lane] = make_float4(c[0], c[1], c[2], c[3]);
            __syncthreads();
            if (part) return;
            const float4 v = second[warp][lane];
            c[0] += v.x;
            c[1] += v.y;
            c[2] += v.z;
            c[3] += v.w;
        }
        if (live) {
            const int64_t S = min(4 * q + g, a.Da - 1);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (4 * q + g < a.Da && col + u < a.Db)
                    y[S * a.Db + col + u] = c[u] + __ldg(a.uT + (col + u) * a.Pa + S);
        }
        if (SPLIT) return;  // one group per pair of warps
    }
}

// Row chunks of the same-spin panels: blocks of 512 threads, one per SM, each on one panel
// of 32 columns (118 KB of x at L=12: it stays in L1 or shared memory); the number of
// chunks that leaves the fewest row groups on the busiest SM. One panel (few strings of
// the other spin) takes a chunk for every SM: L=20 4a1b, 1,212 row groups in at most 64
// chunks left 88 SMs idle and its warps a second round (k_sigma_sum 113 us, the product 155;
// with a chunk for every SM 101).
int same_chunks(int64_t groups, int64_t panels) {
    const int64_t sms = sm_count();
    int best = 1;
    int64_t cost = INT64_MAX;
    for (int c = 1; c <= sms && (c - 1) * 8 < groups; ++c) {
        const int64_t per = (groups + c - 1) / c, rounds = (panels * c + sms - 1) / sms;
        if (per * rounds + 2 * rounds < cost) {  // a block's start and end: about two row groups
            cost = per * rounds + 2 * rounds;
            best = c;
        }
    }
    return best;
}

// Sets of W: a grid of fewer pairs of blocks than SMs runs passes of 16 factors side by
// side, each set's sums in its own W, and k_sigma_sum adds the sets (one after the other
// a pass costs such a grid about 25 us whatever the space: L=10 5a5b, 16 tiles, rank 60:
// 124 -> 50 us).
int sigma_slabs(int64_t tiles, int R, int64_t sms) {
    const int64_t passes = R / kC, most = std::max<int64_t>(1, std::min<int64_t>(passes, sms / (2 * tiles)));
    const int64_t per = (passes + most - 1) / most;
    return (int)((passes + per - 1) / per);  // no set without a pass
}

constexpr size_t kSigmaMaxSmem = 200 * 1024;
constexpr size_t kSigmaMaxPanel = 192 * 1024;  // a same-spin panel held in shared memory
// A grid of fewer 32 x 32 string tiles than SMs.
bool sigma_small_grid(const SpinTables &ta, const SpinTables &tb) {
    return ((ta.D + 31) / 32) * ((tb.D + 31) / 32) < sm_count();
}

// Whether the operator is the faster product, alone on the GPU. Its time (us): 22 for the
// launches and the same-spin part, and for every pass of 16 factors and wave of blocks 5
// and 0.43 per single excitation of a row (fitted to 27.5 to 43 us a pass at 52 to 88
// excitations). The stored values come at about 5.5 TB/s, rows padded to whole tiles of
// beta strings; on small grids at about 3.3 TB/s of the rows' own. Measured, operator |
// stored, among others:
//   L=15 3a3b (207,025 rows) padded rank 112 272 | 311 us, 128 308 | 311; L=16 4a2b (218,400)
//   96 252 | 299, 128 326 | 299; L=20 3a2b (216,600) 64 198 | 398, 128 364 | 398; L=12 6a6b 32
//   316 | 1,800;
//   small grids: L=10 4a4b (44,100) 16 42 | 38, 64 47 | 39; L=10 5a4b (52,920) 16 43 | 64, 64
//   49 | 64; L=12 3a3b (48,400) 16 45 | 48, 80 78 | 48; L=11 4a3b (54,450) 32 45 | 66, 80 74 |
//   66; L=12 5a2b (52,272) 32 53 | 74, 80 108 | 74; L=11 4a4b (108,900) 80 107 | 125; L=13
//   5a2b (100,386) 96 213 | 139; L=9 4a4b (15,876) 16 37 | 16.
// With other solves beside, where only the work counts, any grid takes it (L=10 4a4b 12 | 28
// us, L=9 4a4b 11 | 7).
bool sigma_pays(const SpinTables &ta, const SpinTables &tb, int R) {
    const auto pad = [](int64_t d) { return (d + kTile - 1) / kTile * kTile; };
    const int64_t tiles = pad(ta.D) / kTile * (pad(tb.D) / kTile), sms = sm_count();
    const int64_t slabs = sigma_slabs(tiles, R, sms), passes = (R / kC + slabs - 1) / slabs;
    const int64_t waves = (2 * tiles * slabs + sms - 1) / sms;
    const double op = 22.0 + (double)(waves * passes) * (5.0 + 0.43 * (ta.ns + tb.ns));
    const bool small = sigma_small_grid(ta, tb);
    const double width = 1.0 + ta.ns + tb.ns + ta.nd + tb.nd + (double)ta.ns * tb.ns;
    const double bytes = 4.0 * (double)ta.D * (double)(small ? tb.D : pad(tb.D)) * width;
    return op <= bytes / (small ? 3.3e6 : 5.5e6);
}

}  // namespace

size_t sigma_bytes(int L, int na, int nb, int R) {
    auto dim = [&](int n) { return d_binom(L, n); };
    auto pad = [](int64_t d) { return (d + kTile - 1) / kTile * kTile; };
    auto rows = [&](int n) {  // same-spin rows and the excitation places
        return dim(n) * (8 * (1 + 2 * (int64_t)n * (L - n) + d_binom(n, 2) * d_binom(L - n, 2) + 8));
    };
    const int64_t Da = dim(na), Db = dim(nb), slabs = sigma_slabs(pad(Da) / kTile * (pad(Db) / kTile), R, 152);
    return (size_t)(rows(na) + rows(nb)) +
           sizeof(float) * ((size_t)Da * (slabs * (na * (L - na) + 1) + 1) * pad(Db) + 2 * (size_t)Db * pad(Da) + (size_t)(Da + Db) * R +
                            2 * (size_t)L * L * R);
}

bool sigma_prepare(SigmaOp &op, int L, const double *h, const double *eri, const SpinTables &ta,
                   const SpinTables &tb, const FciParams &p, bool any_grid, cudaStream_t s) {
    op.R = 0;
    if (!sigma_applies(L) || ta.D < 1 || tb.D < 1) return false;
    // the padded ranks the space takes: none, and the factorisation need not begin
    int most = kSigmaMaxRank;
    while (!any_grid && most > 0 && !sigma_pays(ta, tb, most)) most -= kC;
    if (most == 0) return false;
    const int L2 = L * L;
    const size_t N = (size_t)L2;
    // The factors, in the space of orbital pairs p >= q: with c = 1 on the diagonal
    // pairs and sqrt 2 off it, V[P][Q] = c_P c_Q (pq|rs) is the two-electron part in
    // the operators (E_pq + E_qp) / c_P. A pivoted incomplete Cholesky factor of V
    // (two-electron integrals are positive semidefinite as a pair matrix) stops
    // when the largest remaining diagonal falls below 1e-10 of the largest; an
    // indefinite V takes its eigenpairs instead. A factor v gives the symmetric
    // F_pq = F_qp = v_P / c_P.
    const int P = L * (L + 1) / 2;
    std::vector<int> pp(P), pq_(P);
    std::vector<double> cP(P);
    for (int p = 0, i = 0; p < L; ++p)
        for (int q = 0; q <= p; ++q, ++i) {
            pp[i] = p;
            pq_[i] = q;
            cP[i] = p == q ? 1.0 : std::sqrt(2.0);
        }
    const size_t L1 = L, L3 = N * L1;
    auto eri_at = [&](int p, int q, int r, int t) { return eri[p * L3 + q * N + r * L1 + t]; };
    std::vector<double> V((size_t)P * P);
    for (int i = 0; i < P; ++i)
        for (int j = 0; j < P; ++j) V[(size_t)i * P + j] = cP[i] * cP[j] * eri_at(pp[i], pq_[i], pp[j], pq_[j]);
    std::vector<std::vector<double>> vecs;  // factors in the pair space
    std::vector<double> sgn;
    {
        std::vector<double> d(P);
        double d0 = 0;
        for (int i = 0; i < P; ++i) d0 = std::max(d0, d[i] = V[(size_t)i * P + i]);
        bool psd = true;
        while ((int)vecs.size() < P && d0 > 0) {
            int k = 0;
            for (int i = 1; i < P; ++i)
                if (d[i] > d[k]) k = i;
            if (d[k] <= 1e-10 * d0) break;
            std::vector<double> l(P);
            for (int i = 0; i < P; ++i) {
                double v = V[(size_t)i * P + k];
                for (const auto &u : vecs) v -= u[i] * u[k];
                l[i] = v;
            }
            const double r = std::sqrt(d[k]);
            for (int i = 0; i < P; ++i) {
                l[i] /= r;
                d[i] -= l[i] * l[i];
                if (d[i] < -1e-8 * d0) psd = false;
            }
            vecs.push_back(std::move(l));
            sgn.push_back(1.0);
            if ((int)vecs.size() > most) return false;  // so many positive pivots: the rank is no lower
            if (!psd) break;
        }
        if (!psd) {  // indefinite: eigenpairs of the pair matrix
            vecs.clear();
            sgn.clear();
            std::vector<double> A = V, w, z;
            symmetric_eigh(P, A, w, z);
            double wmax = 0;
            for (double v : w) wmax = std::max(wmax, std::fabs(v));
            for (int k = 0; k < P; ++k)
                if (std::fabs(w[k]) > 1e-10 * wmax) {
                    std::vector<double> l(P);
                    const double sc = std::sqrt(std::fabs(w[k]));
                    for (int i = 0; i < P; ++i) l[i] = sc * z[(size_t)i * P + k];
                    vecs.push_back(std::move(l));
                    sgn.push_back(w[k] < 0 ? -1.0 : 1.0);
                }
        }
    }
    const int rank = (int)vecs.size();
    const int R = std::max(kSigmaChunk, (rank + kSigmaChunk - 1) / kSigmaChunk * kSigmaChunk);
    if (R > most || opposite_smem(L) > kSigmaMaxSmem || ta.D * std::max(ta.ns, 1) > (int64_t)UINT32_MAX)
        return false;
    // [R / 16][L^2][16]
    std::vector<float> F(N * R, 0.f), G(N * R, 0.f);
    auto place = [&](size_t pq, int k) { return ((size_t)(k / kC) * N + pq) * kC + k % kC; };
    for (int j = 0; j < rank; ++j)
        for (int i = 0; i < P; ++i) {
            const double f = vecs[j][i] / cP[i];
            const size_t a = place((size_t)pp[i] * L + pq_[i], j), b = place((size_t)pq_[i] * L + pp[i], j);
            F[a] = F[b] = (float)f;
            G[a] = G[b] = (float)(sgn[j] * f);
        }
    // per-string diagonal sums over occupied orbitals, factor-major
    auto diag_sums = [&](const SpinTables &t, const std::vector<float> &X, std::vector<float> &xs) {
        xs.assign((size_t)R * t.D, 0.f);
        for (int j = 0; j < R; ++j)
            for (int64_t S = 0; S < t.D; ++S) {
                double v = 0;
                for (int m = 0; m < t.n; ++m) v += X[place((size_t)t.occ[(size_t)S * t.n + m] * (L + 1), j)];
                xs[(size_t)j * t.D + S] = (float)v;
            }
    };
    std::vector<float> ga, fb;
    diag_sums(ta, G, ga);
    diag_sums(tb, F, fb);
    auto up = [&](DevBuf<float> &buf, const std::vector<float> &v) {
        buf.alloc(v.size());
        if (!v.empty()) CIGPU_CUDA(cudaMemcpyAsync(buf.p, v.data(), v.size() * sizeof(float), cudaMemcpyHostToDevice, s));
    };
    up(op.F, F);
    up(op.G, G);
    up(op.ga, ga);
    up(op.fb, fb);
    op.L = L;
    op.rank = rank;
    op.Da = ta.D;
    op.Db = tb.D;
    op.Pa = (ta.D + kTile - 1) / kTile * kTile;
    op.Pb = (tb.D + kTile - 1) / kTile * kTile;
    op.nea = (p.a.nfull + 7) / 8 * 8;
    op.neb = (p.b.nfull + 7) / 8 * 8;
    op.ea.alloc((size_t)op.Da * op.nea);
    op.eb.alloc((size_t)op.Db * op.neb);
    op.sa.alloc(std::max<size_t>((size_t)op.Da * ta.ns, 1));
    op.sb.alloc(std::max<size_t>((size_t)op.Db * tb.ns, 1));
    const int g = sm_count() * 8;
    unsigned long long *ew = check_word_device();
    k_sigma_rows<<<g, 256, 0, s>>>(p.a, op.nea, op.ea.p, ew);
    k_sigma_rows<<<g, 256, 0, s>>>(p.b, op.neb, op.eb.p, ew);
    count_launch(2);
    if (ta.ns > 0) {
        DevBuf<uint32_t> back((size_t)op.Da * ta.ns);
        k_sigma_back<<<g, 256, 0, s>>>(p.a, L, back.p);
        k_sigma_singles<<<g, 256, 0, s>>>(p.a, L, back.p, op.sa.p, ew);
        count_launch(2);
    }
    if (tb.ns > 0) {
        k_sigma_singles<<<g, 256, 0, s>>>(p.b, L, nullptr, op.sb.p, ew);
        count_launch();
    }
    CIGPU_CUDA(cudaGetLastError());
    op.xp.alloc((size_t)op.Da * op.Pb);
    op.xT.alloc((size_t)op.Db * op.Pa);
    op.uT.alloc((size_t)op.Db * op.Pa);
    op.slabs = sigma_slabs((op.Pa / kTile) * (op.Pb / kTile), R, sm_count());
    op.yd.alloc((size_t)op.slabs * op.Da * op.Pb);
    op.W.alloc(std::max<size_t>((size_t)op.slabs * op.Da * ta.ns * op.Pb, 1));
    op.R = R;
    return true;
}

void sigma_mv32(SigmaOp &op, const FciParams &p, const float *x, float *y, cudaStream_t s) {
    static SmemLimit limit;
    CIGPU_CUDA(limit.raise(k_sigma_parts, kSigmaMaxSmem));
    SigmaArgs a{};
    a.L = op.L;
    a.R = op.R;
    a.nsa = p.a.ns;
    a.nsb = p.b.ns;
    a.Da = op.Da;
    a.Db = op.Db;
    a.Pa = op.Pa;
    a.Pb = op.Pb;
    a.sa = op.sa.p;
    a.sb = op.sb.p;
    a.F = op.F.p;
    a.G = op.G.p;
    a.ga = op.ga.p;
    a.fb = op.fb.p;
    a.rows = op.eb.p;
    a.ne = op.neb;
    a.tiles = (int)((op.Pa / kTile) * (op.Pb / kTile));
    a.panels = (int)((op.Da + kPanel - 1) / kPanel);
    a.slabs = op.slabs;
    a.slab_r = (op.R / kC + op.slabs - 1) / op.slabs * kC;
    const int64_t gb = (op.Db + 3) / 4, ga = (op.Da + 3) / 4;
    a.chunks = same_chunks(gb, a.panels);
    a.per = (int)((gb + a.chunks - 1) / a.chunks);
    const size_t panel = sizeof(float) * kPanel * (size_t)op.Db;
    a.panel_rows = panel <= kSigmaMaxPanel ? (int)op.Db : 0;
    a.xT = op.xT.p;
    a.W = op.W.p;
    a.yd = op.yd.p;
    a.uT = op.uT.p;
    const size_t smem = std::max(opposite_smem(op.L), a.panel_rows ? panel : 0);
    const int64_t blocks = 2 * (int64_t)a.tiles * a.slabs + ((int64_t)a.panels * a.chunks + 1) / 2 * 2;
    k_sigma_pad<<<dim3((unsigned)(op.Pb / 32), (unsigned)(op.Pa / 32)), dim3(32, 8), 0, s>>>(x, op.Da, op.Db, op.Pa, op.Pb,
                                                                                             op.xp.p, op.xT.p);
    k_sigma_parts<<<(unsigned)blocks, kThreads, smem, s>>>(a);
    const int pb = (int)((op.Db + kPanel - 1) / kPanel), c = same_chunks(ga, pb);
    const int per = (int)((ga + c - 1) / c);
    const auto sum = 2 * per <= kWarps ? k_sigma_sum<true> : k_sigma_sum<false>;
    sum<<<dim3((unsigned)c, (unsigned)pb), kThreads, 0, s>>>(a, op.ea.p, op.nea, per, op.xp.p, y);
    CIGPU_CUDA(cudaGetLastError());
    count_launch(3);
}

}  // namespace cigpu
