// bdc_mma.cuh -- FP64 matrix products on the FP64 tensor-core path of sm_100
// (mma.sync.aligned.m8n8k4 .f64: 256 multiply-adds per warp instruction, the
// same peak as FP64 FMA on the CUDA cores but with 1/8 of the issue slots and
// operands read once per fragment).
//
// C(m, n) = sum_k A(m, k) B(k, n) over a "grouped" list of products
// (GemmDesc, bdc_gemm.cuh): CTA i runs tile i of the product whose
// tile_begin <= i.  A split of the contraction is expressed by several
// descriptors with offset operands and separate outputs.
//
// Tile: BM x BN x 16, 256 threads = WM x WN warps, warp tile (8 MT) x (8 NT).
// Global -> registers -> shared memory (k-major, rows padded by 4 doubles so
// that both the transposing stores and the fragment loads are 2 wavefronts per
// warp access), double buffered; the next k-slice is fetched into registers
// while the tensor cores work on the current one.
//
// Fragment layout of m8n8k4 .f64 (g = lane / 4, t = lane % 4):
//   A: a = A[g][t]   B: b = B[t][g]   C/D: c[i] = C[g][2t + i], i = 0, 1
#pragma once

#include "bdc_gemm.cuh"

namespace bdc {

__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ double opnd_load(const Operand& o, int64_t r, int64_t c) {
    const int64_t idx = o.trans ? c * o.ld + r : r * o.ld + c;
    return __ldg((const double*)o.ptr + idx);
}

template <int BM, int BN, int WM, int WN>
struct MmaCfg {
    static constexpr int BK = 16;
    static constexpr int MT = BM / (8 * WM);
    static constexpr int NT = BN / (8 * WN);
    static constexpr int PA = BM + 4;  // padded row of the k-major A tile
    static constexpr int PB = BN + 4;
    static constexpr int A_PER = BK * BM / 256;
    static constexpr int B_PER = BK * BN / 256;
    static_assert(WM * WN == 8, "256 threads");
    static_assert(MT >= 1 && NT >= 1, "warp tile");
    static_assert((BK * BM) % 256 == 0 && (BK * BN) % 256 == 0, "loader");
};

// Loads one k-slice of A (BM x 16) and B (16 x BN) into registers.  Threads
// walk the operand's contiguous direction so that global reads coalesce.
template <int BM, int BN, int WM, int WN>
struct MmaLoader {
    using C = MmaCfg<BM, BN, WM, WN>;
    double ra[C::A_PER], rb[C::B_PER];

    __device__ __forceinline__ void load(const Operand& A, const Operand& B, int M, int N, int K, int m0, int n0,
                                         int k0, bool a_rows, bool b_cols) {
        const int tid = threadIdx.x;
#pragma unroll
        for (int i = 0; i < C::A_PER; ++i) {
            const int e = tid + i * 256;
            const int kk = a_rows ? e / BM : e % C::BK;
            const int mm = a_rows ? e % BM : e / C::BK;
            const int m = m0 + mm, k = k0 + kk;
            ra[i] = (m < M && k < K) ? opnd_load(A, m, k) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < C::B_PER; ++i) {
            const int e = tid + i * 256;
            const int kk = b_cols ? e / BN : e % C::BK;
            const int nn = b_cols ? e % BN : e / C::BK;
            const int n = n0 + nn, k = k0 + kk;
            rb[i] = (n < N && k < K) ? opnd_load(B, k, n) : 0.0;
        }
    }

    __device__ __forceinline__ void store(double* As, double* Bs, bool a_rows, bool b_cols) {
        const int tid = threadIdx.x;
#pragma unroll
        for (int i = 0; i < C::A_PER; ++i) {
            const int e = tid + i * 256;
            const int kk = a_rows ? e / BM : e % C::BK;
            const int mm = a_rows ? e % BM : e / C::BK;
            As[kk * C::PA + mm] = ra[i];
        }
#pragma unroll
        for (int i = 0; i < C::B_PER; ++i) {
            const int e = tid + i * 256;
            const int kk = b_cols ? e / BN : e % C::BK;
            const int nn = b_cols ? e % BN : e / C::BK;
            Bs[kk * C::PB + nn] = rb[i];
        }
    }
};

// The main loop: acc[MT][NT][2] += A_tile * B_tile over the whole contraction.
template <int BM, int BN, int WM, int WN>
__device__ __forceinline__ void mma_mainloop(const GemmDesc& d, int m0, int n0, double* smem,
                                             double (&acc)[MmaCfg<BM, BN, WM, WN>::MT][MmaCfg<BM, BN, WM, WN>::NT][2]) {
    using C = MmaCfg<BM, BN, WM, WN>;
    const Operand A = d.A, B = d.B;
    const int M = d.M, N = d.N, K = d.K;
    const bool a_rows = A.trans != 0;   // A(m,k) contiguous along m
    const bool b_cols = B.trans == 0;   // B(k,n) contiguous along n
    double* As[2] = {smem, smem + C::BK * C::PA};
    double* Bs[2] = {smem + 2 * C::BK * C::PA, smem + 2 * C::BK * C::PA + C::BK * C::PB};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int wm0 = (warp / WN) * (8 * C::MT), wn0 = (warp % WN) * (8 * C::NT);
#pragma unroll
    for (int i = 0; i < C::MT; ++i)
#pragma unroll
        for (int j = 0; j < C::NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

    MmaLoader<BM, BN, WM, WN> ld;
    const int nk = (K + C::BK - 1) / C::BK;
    ld.load(A, B, M, N, K, m0, n0, 0, a_rows, b_cols);
    ld.store(As[0], Bs[0], a_rows, b_cols);
    __syncthreads();
    for (int s = 0; s < nk; ++s) {
        const int cur = s & 1;
        if (s + 1 < nk) ld.load(A, B, M, N, K, m0, n0, (s + 1) * C::BK, a_rows, b_cols);
        const double* as = As[cur];
        const double* bs = Bs[cur];
#pragma unroll
        for (int kq = 0; kq < C::BK / 4; ++kq) {
            double a[C::MT], b[C::NT];
#pragma unroll
            for (int i = 0; i < C::MT; ++i) a[i] = as[(kq * 4 + t) * C::PA + wm0 + i * 8 + g];
#pragma unroll
            for (int j = 0; j < C::NT; ++j) b[j] = bs[(kq * 4 + t) * C::PB + wn0 + j * 8 + g];
#pragma unroll
            for (int i = 0; i < C::MT; ++i)
#pragma unroll
                for (int j = 0; j < C::NT; ++j) mma_f64(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
        if (s + 1 < nk) ld.store(As[cur ^ 1], Bs[cur ^ 1], a_rows, b_cols);
        __syncthreads();
    }
}

template <int BM, int BN, int WM, int WN>
constexpr int mma_smem_bytes() {
    return (int)sizeof(double) * 2 * MmaCfg<BM, BN, WM, WN>::BK * (MmaCfg<BM, BN, WM, WN>::PA + MmaCfg<BM, BN, WM, WN>::PB);
}

}  // namespace bdc

namespace bdc {

// ---------------------------------------------------------------------------
// Multi-stage variant for FP64 operands: tiles move global -> shared memory by
// cp.async (16-byte pieces, zero-filled past the operand's edge), STAGES deep,
// so that several k-slices are in flight without staging registers.  Each
// operand keeps its global orientation in shared memory:
//   AK: A k-major [BK][BM+4] (A contiguous along m) or m-major [BM][BK+4]
//   BKM: B k-major [BK][BN+4] (B contiguous along n) or n-major [BN][BK+4]
// Requirements (checked by the host): both operands FP64, 16-byte aligned
// bases, even leading dimensions and even contraction offsets.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

template <int BM, int BN, bool AK, bool BKM>
struct CpCfg {
    static constexpr int BK = 16;
    static constexpr int PK = BK + 4;
    static constexpr int A_ELEMS = AK ? BK * (BM + 4) : BM * PK;
    static constexpr int B_ELEMS = BKM ? BK * (BN + 4) : BN * PK;
    static constexpr int STAGE = A_ELEMS + B_ELEMS;
};

template <int BM, int BN, int WM, int WN, bool AK, bool BKM, int STAGES>
constexpr int mma_cp_smem_bytes() {
    return (int)sizeof(double) * STAGES * CpCfg<BM, BN, AK, BKM>::STAGE;
}

// One operand's copies of a thread.  KROW: the tile's rows run along the
// contraction (16 of them, DIM contiguous entries each), else along the
// operand's own dimension (DIM rows of 16).  A thread's pieces of 16 bytes lie
// a fixed number of rows apart, so that a slice costs an addition and a copy
// per piece; the addresses and bounds are worked out once per tile (recomputed
// for every piece, they were a third of the products' instructions).
template <int DIM, bool KROW>
struct CpOperand {
    static constexpr int PITCH = KROW ? DIM + 4 : 20;
    static constexpr int PER_ROW = KROW ? DIM / 2 : 8;   // pieces of a row
    static constexpr int ROWS = KROW ? 16 : DIM;
    static constexpr int STEP = 256 / PER_ROW;            // rows between a thread's pieces
    static constexpr int N = (ROWS * PER_ROW + 255) / 256;
    static constexpr bool GUARD = ROWS * PER_ROW < 256;   // not every thread has a piece
    const char* base;  // any valid address, for copies of no bytes
    const char* g;     // the first piece in the next slice
    int64_t row_step, k_step;
    int row, col, s, edge;  // edge: bytes (KROW) or rows (else) inside the operand's dimension
    __device__ __forceinline__ void init(const Operand& o, int at, int lim) {
        const double* p = (const double*)o.ptr;
        base = (const char*)p;
        row = threadIdx.x / PER_ROW;
        col = (threadIdx.x % PER_ROW) * 2;
        s = row * PITCH + col;
        row_step = (int64_t)STEP * o.ld * 8;
        if (KROW) {
            const int c = at + col;
            edge = c + 1 < lim ? 16 : (c < lim ? 8 : 0);
            g = (const char*)(p + (int64_t)row * o.ld + c);
            k_step = 16 * o.ld * 8;
        } else {
            edge = lim - at;
            g = (const char*)(p + (int64_t)(at + row) * o.ld + col);
            k_step = 16 * 8;
        }
    }
    // the slice [k0, k0 + 16) of K into one stage; slices come in order
    __device__ __forceinline__ void load(int k0, int K, double* stage) {
        if (!GUARD || row < ROWS) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                int bytes;
                if (KROW) {
                    bytes = k0 + row + i * STEP < K ? edge : 0;
                } else {
                    const int left = K - k0 - col;
                    bytes = row + i * STEP < edge ? (left >= 2 ? 16 : (left == 1 ? 8 : 0)) : 0;
                }
                cp_async16(stage + s + i * STEP * PITCH, bytes ? g + i * row_step : base, bytes);
            }
        }
        g += k_step;
    }
};

template <int BM, int BN, bool AK, bool BKM>
struct CpLoader {
    CpOperand<BM, AK> a;
    CpOperand<BN, BKM> b;
    int K;
    __device__ __forceinline__ void init(const GemmDesc& d, int m0, int n0) {
        a.init(d.A, m0, d.M);
        b.init(d.B, n0, d.N);
        K = d.K;
    }
    __device__ __forceinline__ void load(int k0, double* stage) {
        a.load(k0, K, stage);
        b.load(k0, K, stage + CpCfg<BM, BN, AK, BKM>::A_ELEMS);
    }
};

// The k loop of one tile; returns with every copy landed and the shared memory
// free.
template <int BM, int BN, int WM, int WN, bool AK, bool BKM, int STAGES>
__device__ __forceinline__ void mma_mainloop_cp(const GemmDesc& d, int m0, int n0, double* smem,
                                            double (&acc)[MmaCfg<BM, BN, WM, WN>::MT][MmaCfg<BM, BN, WM, WN>::NT][2]) {
    using M_ = MmaCfg<BM, BN, WM, WN>;
    using C = CpCfg<BM, BN, AK, BKM>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int wm0 = (warp / WN) * (8 * M_::MT), wn0 = (warp % WN) * (8 * M_::NT);
#pragma unroll
    for (int i = 0; i < M_::MT; ++i)
#pragma unroll
        for (int j = 0; j < M_::NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    CpLoader<BM, BN, AK, BKM> ld;
    ld.init(d, m0, n0);
    const int nk = (d.K + C::BK - 1) / C::BK;
#pragma unroll
    for (int st = 0; st < STAGES - 1; ++st) {
        if (st < nk) ld.load(st * C::BK, smem + st * C::STAGE);
        cp_async_commit();
    }
    int cur = 0, nxt = STAGES - 1;  // stages of this slice and of the one to fetch
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        {
            const int nx = kt + STAGES - 1;
            if (nx < nk) ld.load(nx * C::BK, smem + nxt * C::STAGE);
            cp_async_commit();
            nxt = nxt + 1 == STAGES ? 0 : nxt + 1;
        }
        const double* as = smem + cur * C::STAGE;
        cur = cur + 1 == STAGES ? 0 : cur + 1;
        const double* bs = as + C::A_ELEMS;
#pragma unroll
        for (int kq = 0; kq < C::BK / 4; ++kq) {
            double a[M_::MT], b[M_::NT];
            const int kr = kq * 4 + t;
#pragma unroll
            for (int i = 0; i < M_::MT; ++i) {
                const int m = wm0 + i * 8 + g;
                a[i] = AK ? as[kr * (BM + 4) + m] : as[m * C::PK + kr];
            }
#pragma unroll
            for (int j = 0; j < M_::NT; ++j) {
                const int n = wn0 + j * 8 + g;
                b[j] = BKM ? bs[kr * (BN + 4) + n] : bs[n * C::PK + kr];
            }
#pragma unroll
            for (int i = 0; i < M_::MT; ++i)
#pragma unroll
                for (int j = 0; j < M_::NT; ++j) mma_f64(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
}

}  // namespace bdc
