// bdc_direct.cuh -- one BA iteration of a small problem straight from its
// channel matrix.
//
// The products and transforms of the factored iteration are seven dependent
// launches whose work, for a small problem, is far below a launch.  Where
// C(n,k) < 2^16 the matrix folded over the output orbits,
//     T[x][r] = sum_{y in O(r)} N(x, y)     (representative x, output representative r),
// fits 16-bit integers (sum_y N(x, y) = C(n,k)), and where it also stays in L2
// an iteration is two passes over it:
//     q(r) = sum_x |O(x)| e(x) T[x][r] / (|O(r)| C Z),   D(x) = h(x) - sum_r T[x][r] ln q(r) / C,
// with the update between them.  One launch does D, the update and the next
// iteration's q from one read of a row; every CTA first adds the shares that
// the launch before left.  A problem of one CTA runs any number of iterations
// in one launch.
// (The reference evaluates every pair anew: backend/BAA.cu:429-530, 590-639.)
#pragma once

#include <cfloat>

#include "bdc_common.cuh"

namespace bdc {

// the state after an update whose statistics are mD = max D, sE = sum |O| e,
// mL = max (logW - shift), sR = sum |O| p D, zero = an input was exactly 0
__device__ __forceinline__ void fac_finish(double mD, double sE, double mL, double sR, double zero, double a,
                                           double eta, DevState* st) {
    st->zero_p = (zero != 0.0);
    if (!(sE > 0.0) || !isfinite(sE) || mL > 600.0 || mL < -600.0) {
        st->error = 1;          // kErrShift: e over/underflowed; re-scale from Lt, then finish
        st->max_logw = mL;      // relative to shift; k_fac_rescale subtracts it
        st->max_d = mD;
        st->rate = sR;
        return;
    }
    // Lt holds ln p + eta D - shift, so ln p' - ln p = eta D - shift - ln Z
    const double lnz = log(sE);
    const double ln2 = 0.69314718055994530942;
    const double mx = st->zero_p ? INFINITY : (eta * mD - st->shift - lnz) / ln2;
    st->max_d = mD;
    st->rate = sR;
    st->best_ub = fmin(st->best_ub, mD);
    st->best_rate = fmax(st->best_rate, sR);
    st->lse = st->shift + lnz;
    st->mx = mx;
    st->max_logw = mL + st->shift;
    st->log_z = lnz;
    // next shift: the largest new ln p plus eta times the current bound on D
    st->shift = (mL - lnz) + eta * mD;
    st->zero_p = 0;
    st->iter += 1;
    st->done = !(mx >= a);
}

constexpr int kDirectThreads = 512;
constexpr int kDirectWarps = kDirectThreads / 32;

// What several CTAs hand from one launch to the next: their shares of q and
// of the update's statistics, and the state before those are applied.  Every
// CTA of the next launch adds all shares itself (in the same order), so that
// no CTA waits for another inside a launch.
struct DirectSlot {
    double* part;     // [grid][NYp] shares of q
    double* stat;     // [grid][8] shares of the update's statistics
    DevState* state;
};

struct DirectPlan {
    const uint16_t* T;      // [R][NYp], zero past NY
    const uint32_t* reps;   // ascending
    int64_t R;
    int NY, NYp;            // output representatives, padded to 8
    const double* members;  // [NYp] |O(r)|, 1 past NY
    DirectSlot slot[2];
    double *Lt, *Pw;
    const double* hx;
    double inv_c;
    int n, n2;
};

// an exact small integer as a double by one FP64 addition (2^52 + v - 2^52);
// the conversion unit has a quarter of that rate
__device__ __forceinline__ double direct_f64(uint32_t v) {
    return __hiloint2double(0x43300000, (int)v) - 4503599627370496.0;
}

__device__ __forceinline__ double direct_lnq(double sum, double members, double inv_c, double inv_z) {
    const double q = sum * inv_c * inv_z / members;
    return q != 0.0 ? log(q) : 0.0;  // the reference's ln 0 = 0 (backend/BAA.cu:573-580)
}

// a reduction of the statistics' shares v of one warp: 0 max D, 1 sum |O| e,
// 2 max logW, 3 sum |O| p D, 4 the zero flag
__device__ __forceinline__ double direct_stat(int which, double v) {
    const bool sum = which == 1 || which == 3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xFFFFFFFFu, v, o);
        v = sum ? v + t : fmax(v, t);
    }
    return v;
}
__device__ __forceinline__ double direct_stat0(int which) { return which == 1 || which == 3 ? 0.0 : -DBL_MAX; }

// the statistics in slot S applied to the state st (in shared memory)
__device__ __forceinline__ void direct_finish(const DirectSlot& S, int grid, double a, double eta, double (&sred)[5],
                                              DevState* st) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 5) {
        double v = direct_stat0(warp);
        for (int b = lane; b < grid; b += 32) {
            const double t = S.stat[(size_t)b * 8 + warp];
            v = (warp == 1 || warp == 3) ? v + t : fmax(v, t);
        }
        v = direct_stat(warp, v);
        if (lane == 0) sred[warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) fac_finish(sred[0], sred[1], sred[2], sred[3], sred[4], a, eta, st);
    __syncthreads();
}

// One CTA, after the last launch of a chain: the state from slot S
__global__ void __launch_bounds__(160) k_direct_finish(DirectSlot S, int grid, double a, double eta, DevState* out) {
    __shared__ double sred[5];
    __shared__ DevState st;
    if (threadIdx.x == 0) st = *S.state;
    __syncthreads();
    if (!st.done && !st.error) direct_finish(S, grid, a, eta, sred, &st);
    if (threadIdx.x == 0) *out = st;
}

// What a launch does: kDirectQ: the shares of q of the current iterate;
// kDirectD: ln q from the shares of the launch before, D, the update and its
// statistics; both: the next iterate's shares as well.
enum { kDirectQ = 1, kDirectD = 2 };

// LPX lanes share a representative (8 M output representatives each, in
// 16-byte pieces), 32 / LPX groups a warp; a group takes U representatives at
// a time, so that U rows are in flight and U exponentials run in U lanes.
// SOLO: one CTA runs `iters` iterations, starting from its own q.  Else one
// launch of a chain: `slot` is what it reads (kDirectD) and the other slot
// what it writes; the first launch (kDirectQ alone) takes the state from st.
template <int LPX, int M, bool SOLO>
__global__ void __launch_bounds__(kDirectThreads)
k_direct(DirectPlan P, int what, int slot, int iters, double a, double eta, double* __restrict__ Dout, DevState* st) {
    constexpr int U = M > 1 ? (LPX >= 2 ? 2 : 1) : (LPX >= 4 ? 4 : LPX), XPW = 32 / LPX, W = 8 * M;
    extern __shared__ __align__(16) double red[];  // [kDirectWarps][LPX * W], at least 512 pairs
    __shared__ __align__(16) double slnq[LPX * W];
    __shared__ double sred[5][kDirectWarps], fin[5];
    __shared__ DevState S;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool first = !(what & kDirectD);
    const DirectSlot in = slot ? P.slot[1] : P.slot[0];
    const DirectSlot to = (first || slot) ? P.slot[0] : P.slot[1];
    if (tid == 0) S = (SOLO || first) ? *st : *in.state;
    for (int y = tid; y < LPX * W; y += kDirectThreads) slnq[y] = 0.0;
    __syncthreads();
    const int sub = lane % LPX, grp = lane / LPX;
    const int pieces = P.NYp / 8;  // 16-byte pieces of a row
    const int64_t step = (int64_t)gridDim.x * kDirectWarps * XPW * U;
    const int64_t i0 = (((int64_t)blockIdx.x * kDirectWarps + warp) * XPW + grp) * U;
    // sums of q over shares [y] in v (this thread's y = tid) -> slnq
    // (entries 2e, 2e + 1 of the pieces that the lanes of a group read together
    // lie side by side: at their place in the row, 64 bytes apart, a read took 4
    // or 8 passes)
    auto to_lnq = [&](double sum) {
        const int m = (tid >> 3) / LPX, lane8 = (tid >> 3) % LPX, e = tid & 7;
        if (tid < P.NYp)
            slnq[((m * 4 + (e >> 1)) * LPX + lane8) * 2 + (e & 1)] =
                direct_lnq(sum, P.members[tid], P.inv_c, exp(-S.log_z));
    };
    if (SOLO) {
        if (S.done || S.error) return;
    } else {
        if (!first && !S.done && !S.error && iters > 0) direct_finish(in, gridDim.x, a, eta, fin, &S);
        if (blockIdx.x == 0 && tid == 0) *to.state = S;
        if (S.done || S.error) return;
        if (!first) {
            // thread (c, g): outputs 2c, 2c + 1 of the CTAs g, g + ng, ...
            const int nc = P.NYp / 2, ng = kDirectThreads / nc, c = tid % nc, g = tid / nc;
            double2 s = make_double2(0.0, 0.0);
            if (g < ng) {
                const double2* p = reinterpret_cast<const double2*>(in.part) + c;
                int b = g;
                for (; b + 7 * ng < (int)gridDim.x; b += 8 * ng) {
                    double2 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = p[(size_t)(b + u * ng) * nc];
#pragma unroll
                    for (int u = 0; u < 8; ++u) s.x += v[u].x, s.y += v[u].y;
                }
                for (; b < (int)gridDim.x; b += ng) {
                    const double2 v = p[(size_t)b * nc];
                    s.x += v.x;
                    s.y += v.y;
                }
            }
            reinterpret_cast<double2*>(red)[tid] = s;
            __syncthreads();
            double sum = 0.0;
            if (tid < P.NYp)
                for (int v = 0; v < ng; ++v) sum += red[(v * nc) * 2 + tid];
            to_lnq(sum);
            __syncthreads();
        }
    }
    // one CTA: a q pass, then per iteration D, the update and the next q
    for (int it = SOLO ? -1 : 0; it < (SOLO ? iters : 1); ++it) {
        const bool do_d = SOLO ? it >= 0 : !first;
        const bool do_q = SOLO ? it + 1 < iters : (what & kDirectQ) != 0;
        const double shift = S.shift, lnz = S.log_z;
        const double inv_z = exp(-lnz);
        double acc[W];
#pragma unroll
        for (int j = 0; j < W; ++j) acc[j] = 0.0;
        double mD = -DBL_MAX, sE = 0.0, mL = -DBL_MAX, sR = 0.0, zero = 0.0;
        // positions and state of the next step are loaded before this step's
        // sums (the position must arrive before the state can be asked for),
        // and short rows too (long ones would not fit in registers)
        uint4 nrow[U][M];
        uint32_t nx = 0, nxd = 0;
        double npw = 0.0, nlt = 0.0, nhx = 0.0;
        const int ul = sub % U;  // this lane's representative among the U of its group
        auto fetch_rows = [&](int64_t ib) {
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const int pc = m * LPX + sub;
                    nrow[u][m] = (ib + u < P.R && pc < pieces)
                                     ? __ldg(reinterpret_cast<const uint4*>(P.T + (ib + u) * P.NYp) + pc)
                                     : make_uint4(0u, 0u, 0u, 0u);
                }
        };
        // the longest rows of the next step on their way to L1 (k = 9, 10; shorter
        // ones lose more to the instructions than they gain)
        auto touch_rows = [&](int64_t ib) {
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const int pc = m * LPX + sub;
                    if (ib + u < P.R && pc < pieces)
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const uint4*>(P.T + (ib + u) * P.NYp) + pc));
                }
        };
        auto fetch_rep = [&](int64_t ib) { nx = ib + ul < P.R ? __ldg(P.reps + ib + ul) : 0u; };
        auto fetch_state = [&](int64_t ib) {
            nxd = (nx & ~low_mask(P.n2)) | reverse_bits(nx & low_mask(P.n2), P.n2);
            if (ib + ul < P.R) {
                npw = P.Pw[nxd];
                if (do_d) {
                    nlt = P.Lt[nxd];
                    nhx = __ldg(P.hx + nxd);
                }
            }
        };
        if (M == 1) fetch_rows(i0);
        fetch_rep(i0);
        fetch_state(i0);
        for (int64_t ib = i0; __any_sync(0xFFFFFFFFu, ib < P.R); ib += step) {
            if (M > 1) fetch_rows(ib);
            uint4 row[U][M];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int m = 0; m < M; ++m) row[u][m] = nrow[u][m];
            const uint32_t x = nx, xd = nxd;
            const bool live = ib + ul < P.R;
            const double pw = live ? npw : 0.0, lt = nlt, hx = nhx;
            if (M == 1) fetch_rows(ib + step);
            else if (LPX >= 8) touch_rows(ib + step);
            fetch_rep(ib + step);
            double wq = pw;
            if (do_d) {
                double d[U];
#pragma unroll
                for (int u = 0; u < U; ++u) d[u] = 0.0;
#pragma unroll
                for (int m = 0; m < M; ++m)
#pragma unroll
                    for (int e2 = 0; e2 < 4; ++e2) {
                        const double2 l = *reinterpret_cast<const double2*>(slnq + ((m * 4 + e2) * LPX + sub) * 2);
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const uint32_t p = e2 == 0 ? row[u][m].x : e2 == 1 ? row[u][m].y : e2 == 2 ? row[u][m].z : row[u][m].w;
                            d[u] = fma(direct_f64(p & 0xFFFFu), l.x, d[u]);
                            d[u] = fma(direct_f64(p >> 16), l.y, d[u]);
                        }
                    }
                // the group's sums: lane sub ends with that of representative sub % U
                double g;
                if constexpr (U == 4) {
                    const bool b0 = sub & 1, b1 = sub & 2;
                    const double k0 = b0 ? d[1] : d[0], s0 = b0 ? d[0] : d[1];
                    const double k1 = b0 ? d[3] : d[2], s1 = b0 ? d[2] : d[3];
                    const double t0 = k0 + __shfl_xor_sync(0xFFFFFFFFu, s0, 1);
                    const double t1 = k1 + __shfl_xor_sync(0xFFFFFFFFu, s1, 1);
                    g = (b1 ? t1 : t0) + __shfl_xor_sync(0xFFFFFFFFu, b1 ? t0 : t1, 2);
                } else if constexpr (U == 2) {
                    const bool b0 = sub & 1;
                    g = (b0 ? d[1] : d[0]) + __shfl_xor_sync(0xFFFFFFFFu, b0 ? d[0] : d[1], 1);
                } else {
                    g = d[0];
                }
#pragma unroll
                for (int o = U; o < LPX; o <<= 1) g += __shfl_xor_sync(0xFFFFFFFFu, g, o);
                fetch_state(ib + step);
                const double D = hx - g * P.inv_c;
                // an entry that is exactly 0 in the caller's distribution (Lt
                // holds NaN) takes ln p = 0 (backend/BAA.cu:573-580)
                const bool zero_in = (lt != lt);
                const double lw = (zero_in ? 0.0 : lt - lnz) + eta * D - shift;
                const double o = (double)orbit_size(x, P.n), e = exp(lw);
                wq = live ? o * e : 0.0;
                if (live && sub < U) {
                    P.Lt[xd] = lw;
                    P.Pw[xd] = wq;
                    if (Dout) Dout[xd] = D;
                    mD = fmax(mD, D);
                    mL = fmax(mL, lw);
                    sE = fma(o, e, sE);
                    sR = fma(pw * inv_z, D, sR);
                    if (zero_in) zero = 1.0;
                }
            } else {
                fetch_state(ib + step);
            }
            if (do_q) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double w = U == 1 ? wq : __shfl_sync(0xFFFFFFFFu, wq, u, LPX);
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const uint32_t p[4] = {row[u][m].x, row[u][m].y, row[u][m].z, row[u][m].w};
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            acc[m * 8 + e] =
                                fma(direct_f64((p[e >> 1] >> (16 * (e & 1))) & 0xFFFFu), w, acc[m * 8 + e]);
                    }
                }
            }
        }
        // this CTA's shares
        if (do_q) {
#pragma unroll
            for (int j = 0; j < W; ++j) {
#pragma unroll
                for (int o = LPX; o < 32; o <<= 1) acc[j] += __shfl_xor_sync(0xFFFFFFFFu, acc[j], o);
                if (grp == 0) red[warp * (LPX * W) + ((j / 8) * LPX + sub) * 8 + (j & 7)] = acc[j];
            }
        }
        if (do_d) {
            const double v[5] = {mD, sE, mL, sR, zero};
#pragma unroll
            for (int w = 0; w < 5; ++w) {
                const double r = direct_stat(w, v[w]);
                if (lane == 0) sred[w][warp] = r;
            }
        }
        __syncthreads();
        if (do_d && warp < 5) {
            const double r = direct_stat(warp, lane < kDirectWarps ? sred[warp][lane] : direct_stat0(warp));
            if (lane == 0) {
                if (SOLO) fin[warp] = r;
                else to.stat[(size_t)blockIdx.x * 8 + warp] = r;
            }
        }
        double sum = 0.0;
        if (do_q && tid < P.NYp) {
#pragma unroll
            for (int v = 0; v < kDirectWarps; ++v) sum += red[v * (LPX * W) + tid];
            if (!SOLO) to.part[(size_t)blockIdx.x * P.NYp + tid] = sum;
        }
        if (SOLO) {
            __syncthreads();
            if (do_d && tid == 0) fac_finish(fin[0], fin[1], fin[2], fin[3], fin[4], a, eta, &S);
            __syncthreads();
            if (do_d && (S.done || S.error)) break;
            if (do_q) to_lnq(sum);
            __syncthreads();
        }
    }
    if (SOLO && tid == 0) *st = S;
}

constexpr int direct_smem(int lpx, int m) {
    const int b = kDirectWarps * lpx * 8 * m * (int)sizeof(double), pairs = kDirectThreads * 2 * (int)sizeof(double);
    return b > pairs ? b : pairs;
}

// T[x][r] from the half tables: a thread per entry
__global__ void k_direct_table(Split sp, HalfTables A, HalfTables B, const uint32_t* __restrict__ reps, int64_t R,
                               const uint32_t* __restrict__ yreps, int NY, int NYp, uint16_t* __restrict__ T) {
    const int64_t total = R * NYp;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / NYp;
        const int j = (int)(e % NYp);
        uint32_t s = 0;
        if (j < NY) {
            const uint32_t x = reps[i], y = yreps[j], ry = reverse_bits(y, sp.k), cy = complement_bits(y, sp.k),
                           ry2 = reverse_bits(cy, sp.k);
            s = split_count(sp, A, B, x, y);
            if (ry != y) s += split_count(sp, A, B, x, ry);
            if (cy != y && cy != ry) s += split_count(sp, A, B, x, cy);
            if (ry2 != y && ry2 != ry && ry2 != cy) s += split_count(sp, A, B, x, ry2);
        }
        T[e] = (uint16_t)s;
    }
}

}  // namespace bdc
