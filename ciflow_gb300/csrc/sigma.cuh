// FP32 product of the mixed method for FCI from a factorised two-electron part
// (sigma.cu): a direct-CI sigma vector in place of the stored-matrix product.
#pragma once

#include "build.cuh"

namespace cigpu {

constexpr int kSigmaTile = 64;       // strings per tile side
constexpr int kSigmaChunk = 16;      // factors per pass (the rank is padded to a multiple)
constexpr int kSigmaMaxRank = 128;   // padded rank limit
constexpr int kSigmaMaxL = 24;       // orbitals limit (the factorisation is an L^2 x L^2 eigenproblem on the host)

struct SigmaOp {
    int L = 0;
    int rank = 0;  // factors kept
    int R = 0;     // rank padded to a multiple of kSigmaChunk; 0: the operator is not in use
    int64_t Da = 0, Db = 0, Pa = 0, Pb = 0;  // strings of each spin, and padded to kSigmaTile
    int slabs = 1;                           // sets of W and yd
    int nea = 0, neb = 0;                    // same-spin elements per string (padded to 8)
    DevBuf<float> F, G;                  // [R/16][L*L][16]: factors F^k and s_k F^k
    DevBuf<float> ga, fb;                // per-string diagonal sums of G (alpha), F (beta): [R][Da], [R][Db]
    DevBuf<uint2> ea, eb;                // same-spin rows: [D][ne] {target, value}
    DevBuf<uint2> sa, sb;                // single excitations {W row | target, pair << 1 | odd}: [D][ns]
    DevBuf<float> xp, xT, uT, W, yd;     // work: x padded, x transposed, the beta part, W, its diagonal part
};

// Whether a space of L orbitals can use the operator (before the rank is known).
inline bool sigma_applies(int L) { return L >= 1 && L <= kSigmaMaxL; }

// Factorises (pq|rs) = sum_k s_k F^k_pq F^k_rs (a pivoted Cholesky factor of the
// pair matrix to 1e-10 of its largest diagonal; eigenpairs when it is indefinite),
// forms the per-string tables (p: the string tables on the device) and allocates the
// work buffers. False (op.R = 0) when the space does not qualify (too many orbitals, or a
// rank past kSigmaMaxRank or, unless any_grid, past the one to which the operator is faster
// than the stored values).
bool sigma_prepare(SigmaOp &op, int L, const double *h, const double *eri, const SpinTables &ta,
                   const SpinTables &tb, const FciParams &p, bool any_grid, cudaStream_t s);

// Device bytes of the operator's tables and work buffers at the padded rank R.
size_t sigma_bytes(int L, int na, int nb, int R);

// y = H x in FP32 (x, y: [Da][Db] device vectors).
void sigma_mv32(SigmaOp &op, const FciParams &p, const float *x, float *y, cudaStream_t s);

}  // namespace cigpu
