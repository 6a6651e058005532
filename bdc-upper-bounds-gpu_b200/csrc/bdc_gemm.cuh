// bdc_gemm.cuh -- FP64 tiled matrix products for the factored engine.
//
// C(m, n) = alpha * sum_k A(m, k) B(k, n) (+ C).  Element (r, c) of an operand
// lives at ptr[r * ld + c] or, transposed, ptr[c * ld + r].  The kernels are in
// bdc_mma.cuh (FP64 mma.sync tiles).  All launches are "grouped": one launch
// runs a list of products (GemmDesc) and CTA i finds its product through a
// prefix table of tile counts.
#pragma once

#include "bdc_common.cuh"

namespace bdc {

struct Operand {
    const void* ptr = nullptr;
    int64_t ld = 0;
    int trans = 0;  // 0: (r,c) at ptr[r*ld+c]; 1: at ptr[c*ld+r]
};

struct GemmDesc {
    Operand A;        // M x K
    Operand B;        // K x N
    double* C;        // element (m,n) at C[m*ldc_m + n*ldc_n]
    int64_t ldc_m, ldc_n;
    int M, N, K;
    double alpha;
    int accumulate;   // C += alpha AB instead of C = alpha AB
    int tiles_m, tiles_n;  // filled by the planner
    int tile_begin;        // first CTA of this product in its launch
};

// The BA epilogue of the D-side product G = LA * RB (see bdc_factored.cu).
struct BaEpilogue {
    int n;                       // string length; x = m * H2 + col
    int n2;
    const double* __restrict__ hx;  // h(x) at representatives
    double* Lt;                  // log of the unnormalised iterate (in place)
    double* Pw;                  // |O(x)| * exp(Lt - shift) (in place)
    double inv_c;
    double* part;                // per-CTA partials [ctas][8]: max D, sum |O| e, max logW, sum |O| p D, zero flag
    const DevState* st;
    double* Dout;                // optional: D(x) at every representative (dense layout)
    double eta;                  // step of the exponentiated-gradient update: ln p' = ln p + eta D - ln Z
                                 // (1 is the BA update)
    int row0;                    // global x_hi of the product's row 0 (a shard of the rows; 0 on one GPU)
};

// what the epilogue's update needs beside the element itself
struct BaConst {
    double shift, lnz, inv_z, inv_c, eta;
    uint32_t mask, odd, row0;
};
__device__ __forceinline__ BaConst ba_const(const BaEpilogue& ep, const DevState* st) {
    BaConst k;
    k.shift = st->shift;
    k.lnz = st->log_z;
    k.inv_z = exp(-k.lnz);
    k.inv_c = ep.inv_c;
    k.eta = ep.eta;
    k.mask = low_mask(ep.n2);
    k.odd = (uint32_t)ep.n & 1u;
    k.row0 = (uint32_t)ep.row0;
    return k;
}

// a thread's share of the update's statistics
struct BaStats {
    double mD = -1.7976931348623157e308, sE = 0.0, mL = -1.7976931348623157e308, sR = 0.0, zero = 0.0;
};

// the update of one representative (orbit o) whose G value is g: lt, pw are
// replaced, D is returned.  An entry that is exactly 0 in the caller's
// distribution (lt is NaN) takes ln p = 0, as the reference's
// apply_log_kernel leaves ln 0 at 0 (backend/BAA.cu:573-580); later iterates
// keep exact logarithms.
__device__ __forceinline__ double ba_update(double g, double h, double o, double& lt, double& pw, const BaConst& k,
                                            BaStats& s) {
    const double D = h - g * k.inv_c;
    const bool zero_in = (lt != lt);
    const double lw = (zero_in ? 0.0 : lt - k.lnz) + k.eta * D - k.shift;
    const double e = exp(lw);
    s.sR = fma(pw * k.inv_z, D, s.sR);
    lt = lw;
    pw = o * e;
    s.mD = D > s.mD ? D : s.mD;  // (a comparison and a select: fmax costs twice that)
    s.mL = lw > s.mL ? lw : s.mL;
    s.sE = fma(o, e, s.sE);
    if (zero_in) s.zero = 1.0;
    return D;
}

}  // namespace bdc
