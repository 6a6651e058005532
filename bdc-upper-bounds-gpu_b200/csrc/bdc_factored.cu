// bdc_factored.cu -- the factored engine: one BA iteration as FP64 matrix
// products over the half tables, with the BA update fused into the largest one.
//
// Reference path replaced (Pintz45/BDC-Upper-Bounds-GPU): the iteration of
// backend/BAA.cu:590-639 (q pass 429-485, D pass 487-530, normalisation
// 590-639, max deviation 916-946).  The reference evaluates N(x,y) pair by
// pair through the split identity (total_transitions, BAA.cu:340-395):
//     N(x, y) = sum_j A_j[x_hi][y_hi] * B_{k-j}[x_lo][y_lo],
// A_j = cache_{n1,j}, B_m = cache_{n2,m}.  For a fixed j this is a Kronecker
// product, so with the iterate laid out as a 2^{n1} x 2^{n2} matrix P:
//   q side:  Q_j = A_j^T P B_{k-j}                (the 2^j x 2^{k-j} block of q)
//   D side:  G   = sum_j A_j Lq_j B_{k-j}^T,  D(x) = h(x) - G(x) / C(n,k)
// with Lq_j = ln q reshaped to 2^j x 2^{k-j} and h(x) = sum_y W ln W (from
// the count path, once per handle).  Each term uses the cheaper association:
// "L" terms (2^j <= 2^{k-j}) contract x_hi first, "R" terms contract x_lo
// first.  Every representative is <= its complement, so its top bit is 0 and
// only the rows x_hi < H1/2 of the iterate and of G exist.  Per iteration:
//   1. U = AL^T Pw, V = Pw BR            (Pw = |O(x)| p(x) at representatives,
//                                          0 elsewhere; AL, BR: tables of the
//                                          words of length a and b, below)
//   2. the word transforms of U and V -> shares of acc[y]; fold the orbits -> ln q
//   3. the word transforms of ln q -> ML, NR
//   4. G = [AL | NR] [ML ; BR^T] with the BA update as epilogue: D, logW,
//      exp(logW - shift), the new iterate (in place) and block partials of
//      max D, sum |O| e, max logW, sum |O| p D
//   5. one-block finalize: ln Z, mx, upper bound, stop test, next shift.
// The contraction of 1 and 4 runs over the words of one length per half, a =
// floor(k/2) characters of x_hi and b = k - 1 - a of x_lo (2^a + 2^b of them):
// occurrences of shorter words are fixed combinations of those of length a
// (bdc_words.cuh).  With the words of every length up to a and b it had twice
// the length (190 instead of 96 at n = 24, k = 12).
// The products run on the FP64 tensor-core path (bdc_mma.cuh).  Counts are
// exact integers < 2^16 widened to FP64; all sums are FP64.  The tile shape
// and split of the large products are picked at set-up by timing candidates.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <initializer_list>
#include <map>
#include <string>
#include <type_traits>
#include <vector>

#include <cstring>

#include "bdc_direct.cuh"
#include "bdc_engine.cuh"
#include "bdc_gemm.cuh"
#include "bdc_mma.cuh"
#include "bdc_ozaki.cuh"
#include "bdc_words.cuh"

namespace bdc {

constexpr int kErrShift = 1;  // DevState::error: exp shift out of range, re-scale

// tile configurations of the FP64 tensor-core products (BM x BN, warps WM x WN)
enum MmaConfig {
    CFG_128x64 = 1, CFG_64x128, CFG_64x64, CFG_128x16, CFG_16x128, CFG_128x32, CFG_64x32, CFG_32x128,
    CFG_32x64, CFG_COUNT  // (the numbers stand in tune files)
};
static const int kCfgBM[CFG_COUNT] = {0, 128, 64, 64, 128, 16, 128, 64, 32, 32};
static const int kCfgBN[CFG_COUNT] = {0, 64, 128, 64, 16, 128, 32, 32, 128, 64};

struct Launch {
    GemmDesc* d = nullptr;   // device descriptors
    int* map = nullptr;      // CTA -> descriptor index
    int n = 0, tiles = 0, cfg = CFG_64x64;
    int layout = -1;         // -1: register-staged mainloop; else the cp.async one (see k_mma_store)
};

}  // namespace bdc

struct FactoredState {
    int H1 = 0, H2 = 0, KL = 0, KR = 0, Kp = 0;  // KL = 2^a, KR = 2^b words, Kp = KL + KR padded
    int H1h = 0;              // rows held: x_hi in [row0, row0 + H1h) (all x_hi < H1 / 2 on one GPU)
    int row0 = 0;             // first row held (a shard of the rows over several GPUs; 0 on one GPU)
    int64_t i0 = 0, Rl = 0;   // the representatives in those rows: [i0, i0 + Rl) of the ascending list
    int64_t* d_rowstart = nullptr;  // [H1h + 1]: held row r's representatives are [i0 + rowstart[r], i0 + rowstart[r + 1])
    double* rpart = nullptr;        // [2 H1h]: per-row partials of the load
    int rows_smem = 0;              // dynamic shared memory of the row kernels
    double* Pw = nullptr;     // [2^{n-1}]  |O(x)| e(x) at representatives, 0 elsewhere
    double* Lt = nullptr;     // [2^{n-1}]  ln e(x) (p = e / Z)
    double* hx = nullptr;     // [2^{n-1}]  h(x) at representatives
    uint16_t* Bp = nullptr;   // low-half tables, row c = table row rev(c) (dense column order)
    double* Ddense = nullptr; // [2^{n-1}] D(x) of a map with D output (allocated on first use)
    double* dout = nullptr;   // where the G epilogue writes D (nullptr: nowhere)
    double eta = 1.0;         // step of the update in the G epilogue (1: the BA map)
    std::vector<int> colmax;  // per dense column: largest x_hi of a representative, -1 if none
    double* LA = nullptr;     // [H1h][Kp]  = [AL | NR]
    double* RB = nullptr;     // [Kp][H2]  = [ML ; BR^T]
    double* ulpart = nullptr; // [S1][KL][H2]   split slices of U
    double* vrpart = nullptr; // [S2][KR][H1h]  split slices of V, word-major
    int S1 = 1, S2 = 1;
    uint8_t* d_ns[2] = {};    // slices of each 16 columns of U, of each 16 rows of V
    // the word transforms (bdc_words.cuh)
    bdc::WordPlan plan;
    bdc::WordPlan* d_plan = nullptr;
    int words_smem = 0, words_r = 0;  // words_r: characters of the longest slice
    void* d_wtab[2] = {};     // each side's weights, terms and their ranges
    double* qparts = nullptr; // [plan.parts][2^k]  shares of acc[y] of the transforms' CTAs
    double* qacc = nullptr;   // [2^k]     a shard's sums
    int* d_mids = nullptr;    // the fold's middles, one per CTA
    int n_mids = 0;
    double* lnq_full = nullptr;  // [2^k]
    // small problems: the iteration straight from the folded matrix (bdc_direct.cuh)
    bool direct = false;
    bool products = false;    // the products are set up (beside the direct form: see kBesideBytes)
    bdc::DirectPlan dp{};
    int d_lpx = 0, d_m = 1, d_grid = 0;  // d_grid: the most CTAs, which the slots have room for
    int beside = 1;                      // instances that run at the same time (a batch)
    double* d_members = nullptr;
    double* epart = nullptr;  // [ctas][8]
    double* spart = nullptr;  // [kStatRows][8]
    int ctas_g = 0;
    bdc::OzakiG* oz = nullptr;  // G on the int8 tensor cores (when set up and chosen)
    bool use_oz = false;
    bdc::Launch ul, vr, g;
    int launches_per_iter = 0;
    // V runs on a branch beside U
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    // a captured chunk of kGraphIters iterations for the threshold graph_a
    cudaGraphExec_t graph = nullptr;
    double graph_a = 0.0;
    // accelerated loop: the normalised log iterate x_t and the graph of
    // kAccSteps steps
    double* snap0 = nullptr;
    cudaGraphExec_t cycle = nullptr;
    double cycle_eta = 0.0;
    // captured single BA maps (factored_map), by their vectors
    struct MapGraph {
        const double* pin = nullptr;
        double* pout = nullptr;
        double* dout = nullptr;
        cudaGraphExec_t exec = nullptr;
    };
    MapGraph maps[4];
    int maps_next = 0;
};

namespace bdc {

__device__ __forceinline__ bool gated(const DevState* st) { return st && (st->done || st->error); }

enum Stage { ST_QBIG = 0, ST_QSMALL, ST_FOLD, ST_DSMALL, ST_G, ST_FIN, ST_COUNT };
static cudaError_t enqueue_stage(bdc_handle* H, int stage, double a);

// Dense layout of the iterate: row x_hi, column rev(x_lo) (the low half
// bit-reversed).  A representative x satisfies x <= rev(x) and x <=
// rev(comp(x)), so x_hi is at most a bound that rises and then falls along
// the columns; whole tiles of the dense matrices then hold no
// representative and are skipped.  The map is its own inverse.
__host__ __device__ __forceinline__ uint32_t fac_pos(uint32_t x, int n2) {
    const uint32_t m = low_mask(n2);
    return (x & ~m) | reverse_bits(x & m, n2);
}

// the index of representative x in a dense buffer that holds the rows
// x_hi >= row0 (a shard of the rows; row0 = 0 on one GPU)
__host__ __device__ __forceinline__ uint32_t fac_loc(uint32_t x, int n, int row0) {
    return fac_pos(x, n >> 1) - ((uint32_t)row0 << (n >> 1));
}

// Kernels that touch every representative walk the dense arrays in memory
// order and test the position (dense_is_rep), coalesced, instead of the
// ascending list (whose positions are bit-reversed in a row).

// ------------------------------------------------ products: plain store
// LAYOUT < 0: register-staged mainloop (any operand kind); otherwise the
// cp.async mainloop with A k-major when bit 0 is set and B k-major when bit 1
// is set (FP64 operands only)
template <int BM, int BN, int WM, int WN, int LAYOUT>
__global__ void __launch_bounds__(256) k_mma_store(const GemmDesc* __restrict__ descs, const int* __restrict__ map,
                                                   const DevState* st) {
    using C = MmaCfg<BM, BN, WM, WN>;
    if (gated(st)) return;
    extern __shared__ __align__(16) double smem[];
    const GemmDesc& d = descs[map[blockIdx.x]];
    const int t = blockIdx.x - d.tile_begin;
    const int m0 = (t / d.tiles_n) * BM, n0 = (t % d.tiles_n) * BN;
    double acc[C::MT][C::NT][2];
    if constexpr (LAYOUT < 0) mma_mainloop<BM, BN, WM, WN>(d, m0, n0, smem, acc);
    else mma_mainloop_cp<BM, BN, WM, WN, (LAYOUT & 1) != 0, (LAYOUT & 2) != 0, 3>(d, m0, n0, smem, acc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int wm0 = (warp / WN) * (8 * C::MT), wn0 = (warp % WN) * (8 * C::NT);
#pragma unroll
    for (int i = 0; i < C::MT; ++i) {
        const int m = m0 + wm0 + i * 8 + g;
        if (m >= d.M) continue;
#pragma unroll
        for (int j = 0; j < C::NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int n = n0 + wn0 + j * 8 + 2 * tq + h;
                if (n >= d.N) continue;
                double* c = d.C + (int64_t)m * d.ldc_m + (int64_t)n * d.ldc_n;
                const double v = d.alpha * acc[i][j][h];
                *c = d.accumulate ? *c + v : v;
            }
    }
}

// ------------------------------------------- the G product + BA update
// rows are x_hi, columns x_lo, x = (x_hi << n2) | x_lo; only representatives
// are updated; block partials [max D, sum |O| e, max (logW - shift),
// sum |O| p D, input-zero flag] go to ep.part[blockIdx.x * 8 + 0..4].
// CTA b takes tile tiles[b] of those that hold representatives.  The sums
// leave the fragments through shared memory (the mainloop's, at a pitch of 8
// extra doubles: 16-byte stores of a fragment's pair without conflicts), so
// that the update runs a row at a time with 16-byte loads and stores of two
// adjacent columns: on the fragments themselves every access touched twice
// the sectors and the orbit tests and addresses were 2/3 of 210 instructions
// an element.  84 -> 67 us at 24/12 (135 MB of device memory: 21 us).
constexpr int g_stages(int bm, int bn, int, int) { return bm * bn <= 4096 ? 2 : 3; }
template <int BM, int BN, int WM, int WN, bool WITH_D>
__global__ void __launch_bounds__(256, (BM * BN <= 4096) ? 4 : 2) k_mma_ba(const GemmDesc* __restrict__ descs, const int* __restrict__ tiles,
                                                   BaEpilogue ep, const DevState* st) {
    using C = MmaCfg<BM, BN, WM, WN>;
    constexpr int LD = BN + 8;
    if (gated(st)) return;
    extern __shared__ __align__(16) double smem[];
    const GemmDesc& d = descs[0];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int wm0 = (warp / WN) * (8 * C::MT), wn0 = (warp % WN) * (8 * C::NT);
    const int t = tiles[blockIdx.x];
    const int m0 = (t / d.tiles_n) * BM, n0 = (t % d.tiles_n) * BN;
    const int M = d.M, N = d.N;
    // the state of the tile on its way to L2 while the products run
    constexpr int LINES = BM * BN / 16;  // 128-byte lines of one array
    for (int q = threadIdx.x; q < LINES; q += 256) {
        const int m = m0 + q / (BN / 16), n = n0 + (q % (BN / 16)) * 16;
        if (m < M && n < N && dense_is_rep((uint32_t)m + (uint32_t)ep.row0, (uint32_t)n + 8, low_mask(ep.n2), 0u)) {
            const size_t at = ((size_t)m << ep.n2) + n;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(ep.hx + at));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(ep.Pw + at));
            if (!WITH_D || ep.Lt) asm volatile("prefetch.global.L2 [%0];" ::"l"(ep.Lt + at));
        }
    }
    {
        double acc[C::MT][C::NT][2];
        mma_mainloop_cp<BM, BN, WM, WN, false, true, g_stages(BM, BN, 0, 0)>(d, m0, n0, smem, acc);
        static_assert(BM * LD * (int)sizeof(double) <= mma_cp_smem_bytes<BM, BN, WM, WN, false, true, g_stages(BM, BN, 0, 0)>(), "tile");
#pragma unroll
        for (int i = 0; i < C::MT; ++i)
#pragma unroll
            for (int j = 0; j < C::NT; ++j)
                *reinterpret_cast<double2*>(smem + (wm0 + i * 8 + g) * LD + wn0 + j * 8 + 2 * tq) =
                    make_double2(acc[i][j][0], acc[i][j][1]);
    }
    const BaConst kc = ba_const(ep, st);
    BaStats bs;
    __syncthreads();
    constexpr int SEG = BN / 64, ROWS = BM * SEG;  // 64-column segments of rows, one per warp at a time
#pragma unroll 1
    for (int q0 = warp; q0 < ROWS; q0 += 16) {
        double2 hv[2], lv[2], pv[2];
        bool r0[2], r1[2];
        uint32_t xd[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + 8 * u, m = m0 + q / SEG, n = n0 + (q % SEG) * 64 + 2 * lane;
            const bool in = q < ROWS && m < M && n < N;
            const uint32_t r = (uint32_t)m + kc.row0;
            r0[u] = in && dense_is_rep(r, (uint32_t)n, kc.mask, kc.odd);
            r1[u] = in && dense_is_rep(r, (uint32_t)n + 1, kc.mask, kc.odd);
            xd[u] = ((uint32_t)m << ep.n2) | (uint32_t)n;
            if (r0[u] || r1[u]) {
                hv[u] = __ldg(reinterpret_cast<const double2*>(ep.hx + xd[u]));
                pv[u] = *reinterpret_cast<const double2*>(ep.Pw + xd[u]);
                if (!WITH_D || ep.Lt) lv[u] = *reinterpret_cast<const double2*>(ep.Lt + xd[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (!(r0[u] || r1[u])) continue;
            const int q = q0 + 8 * u;
            const uint32_t r = (uint32_t)(m0 + q / SEG) + kc.row0, n = xd[u] & kc.mask;
            const double2 gv = *reinterpret_cast<const double2*>(smem + (q / SEG) * LD + (q % SEG) * 64 + 2 * lane);
            if (WITH_D && !ep.Lt) {  // an evaluation: no update
                const double d0 = hv[u].x - gv.x * kc.inv_c, d1 = hv[u].y - gv.y * kc.inv_c;
                if (r0[u]) {
                    bs.mD = fmax(bs.mD, d0);
                    bs.sR = fma(pv[u].x * kc.inv_z, d0, bs.sR);
                    if (ep.Dout) ep.Dout[xd[u]] = d0;
                }
                if (r1[u]) {
                    bs.mD = fmax(bs.mD, d1);
                    bs.sR = fma(pv[u].y * kc.inv_z, d1, bs.sR);
                    if (ep.Dout) ep.Dout[xd[u] + 1] = d1;
                }
                continue;
            }
            if (r0[u]) {
                const double D = ba_update(gv.x, hv[u].x, dense_orbit(r, n, kc.mask, kc.odd), lv[u].x, pv[u].x, kc, bs);
                if (WITH_D) ep.Dout[xd[u]] = D;
            }
            if (r1[u]) {
                const double D = ba_update(gv.y, hv[u].y, dense_orbit(r, n + 1, kc.mask, kc.odd), lv[u].y, pv[u].y, kc, bs);
                if (WITH_D) ep.Dout[xd[u] + 1] = D;
            }
            *reinterpret_cast<double2*>(ep.Lt + xd[u]) = lv[u];
            *reinterpret_cast<double2*>(ep.Pw + xd[u]) = pv[u];
        }
    }
    double mD = bs.mD, sE = bs.sE, mL = bs.mL, sR = bs.sR, zero = bs.zero;
    __shared__ double red[5][8];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        mD = fmax(mD, __shfl_xor_sync(0xFFFFFFFFu, mD, off));
        mL = fmax(mL, __shfl_xor_sync(0xFFFFFFFFu, mL, off));
        sE += __shfl_xor_sync(0xFFFFFFFFu, sE, off);
        sR += __shfl_xor_sync(0xFFFFFFFFu, sR, off);
        zero = fmax(zero, __shfl_xor_sync(0xFFFFFFFFu, zero, off));
    }
    if (lane == 0) {
        red[0][warp] = mD;
        red[1][warp] = sE;
        red[2][warp] = mL;
        red[3][warp] = sR;
        red[4][warp] = zero;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a0 = red[0][0], a1 = red[1][0], a2 = red[2][0], a3 = red[3][0], a4 = red[4][0];
        for (int w = 1; w < 8; ++w) {
            a0 = fmax(a0, red[0][w]);
            a1 += red[1][w];
            a2 = fmax(a2, red[2][w]);
            a3 += red[3][w];
            a4 = fmax(a4, red[4][w]);
        }
        double* p = ep.part + (size_t)blockIdx.x * 8;
        p[0] = a0;
        p[1] = a1;
        p[2] = a2;
        p[3] = a3;
        p[4] = a4;
    }
}

#define BDC_CFG_ARGS_128x64 128, 64, 4, 2
#define BDC_CFG_ARGS_64x128 64, 128, 2, 4
#define BDC_CFG_ARGS_64x64 64, 64, 2, 4
#define BDC_CFG_ARGS_128x16 128, 16, 8, 1
#define BDC_CFG_ARGS_16x128 16, 128, 1, 8
#define BDC_CFG_ARGS_128x32 128, 32, 4, 2
#define BDC_CFG_ARGS_64x32 64, 32, 4, 2
#define BDC_CFG_ARGS_32x128 32, 128, 2, 4
#define BDC_CFG_ARGS_32x64 32, 64, 2, 4

static int cfg_smem(int cfg, int layout = -1) {
#define CASE_(C, ARGS)                                                                          \
    case C:                                                                                     \
        switch (layout) {                                                                       \
            case 0: return mma_cp_smem_bytes<ARGS, false, false, 3>();                          \
            case 1: return mma_cp_smem_bytes<ARGS, true, false, 3>();                           \
            case 2: return mma_cp_smem_bytes<ARGS, false, true, g_stages(ARGS)>();                           \
            case 3: return mma_cp_smem_bytes<ARGS, true, true, 3>();                            \
            default: return mma_smem_bytes<ARGS>();                                             \
        }
    switch (cfg) {
        CASE_(CFG_128x64, BDC_CFG_ARGS_128x64)
        CASE_(CFG_64x128, BDC_CFG_ARGS_64x128)
        CASE_(CFG_64x64, BDC_CFG_ARGS_64x64)
        CASE_(CFG_128x16, BDC_CFG_ARGS_128x16)
        CASE_(CFG_16x128, BDC_CFG_ARGS_16x128)
        CASE_(CFG_128x32, BDC_CFG_ARGS_128x32)
        CASE_(CFG_64x32, BDC_CFG_ARGS_64x32)
        CASE_(CFG_32x128, BDC_CFG_ARGS_32x128)
        CASE_(CFG_32x64, BDC_CFG_ARGS_32x64)
    }
#undef CASE_
    return 0;
}

// the cp.async mainloop is instantiated for the layouts the products use:
// 3 (U: both k-major), 0 (V and the solver's A B^T: both contraction-major);
// the register-staged one for 64x64 tiles (the solver's odd leading dimensions)
static bool cp_instantiated(int layout) { return layout == 0 || layout == 3; }

static cudaError_t set_smem_attrs() {
    static bool done = false;
    if (done) return cudaSuccess;
#define SET_K(KERNEL, BYTES)                                                                     \
    {                                                                                            \
        cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES); \
        if (e != cudaSuccess) return e;                                                          \
    }
#define SET_STORE(ARGS)                                                                          \
    SET_K((k_mma_store<ARGS, -1>), (mma_smem_bytes<ARGS>()))
#define SET_STORE_CP(ARGS)                                                                       \
    SET_K((k_mma_store<ARGS, 0>), (mma_cp_smem_bytes<ARGS, false, false, 3>()))                 \
    SET_K((k_mma_store<ARGS, 3>), (mma_cp_smem_bytes<ARGS, true, true, 3>()))
#define SET_BA(ARGS)                                                                             \
    SET_K((k_mma_ba<ARGS, false>), (mma_cp_smem_bytes<ARGS, false, true, g_stages(ARGS)>()))                  \
    SET_K((k_mma_ba<ARGS, true>), (mma_cp_smem_bytes<ARGS, false, true, g_stages(ARGS)>()))
    SET_STORE(BDC_CFG_ARGS_64x64)
    SET_STORE_CP(BDC_CFG_ARGS_128x64)
    SET_STORE_CP(BDC_CFG_ARGS_64x128)
    SET_STORE_CP(BDC_CFG_ARGS_64x64)
    SET_STORE_CP(BDC_CFG_ARGS_128x16)
    SET_STORE_CP(BDC_CFG_ARGS_16x128)
    SET_STORE_CP(BDC_CFG_ARGS_128x32)
    SET_STORE_CP(BDC_CFG_ARGS_64x32)
    SET_STORE_CP(BDC_CFG_ARGS_32x128)
    SET_STORE_CP(BDC_CFG_ARGS_32x64)
    SET_BA(BDC_CFG_ARGS_128x64)
    SET_BA(BDC_CFG_ARGS_64x128)
    SET_BA(BDC_CFG_ARGS_64x64)
#undef SET_BA
#undef SET_STORE_CP
#undef SET_STORE
#undef SET_K
    done = true;
    return cudaSuccess;
}

static cudaError_t launch_store(const Launch& L, cudaStream_t s, const DevState* st) {
    if (L.n == 0 || L.tiles == 0) return cudaSuccess;
    const int lay = cp_instantiated(L.layout) ? L.layout : -1;
    if (lay < 0 && L.cfg != CFG_64x64) return cudaErrorInvalidValue;
    const int sm = cfg_smem(L.cfg, lay);
#define GO_(NAME)                                                                                           \
    case CFG_##NAME:                                                                                        \
        if (lay == 0) k_mma_store<BDC_CFG_ARGS_##NAME, 0><<<L.tiles, 256, sm, s>>>(L.d, L.map, st);         \
        else if (lay == 3) k_mma_store<BDC_CFG_ARGS_##NAME, 3><<<L.tiles, 256, sm, s>>>(L.d, L.map, st);    \
        break;
    if (lay < 0) {
        k_mma_store<BDC_CFG_ARGS_64x64, -1><<<L.tiles, 256, sm, s>>>(L.d, L.map, st);
        return cudaGetLastError();
    }
    switch (L.cfg) {
        GO_(128x64)
        GO_(64x128)
        GO_(64x64)
        GO_(128x16)
        GO_(16x128)
        GO_(128x32)
        GO_(64x32)
        GO_(32x128)
        GO_(32x64)
        default: return cudaErrorInvalidValue;
    }
#undef GO_
    return cudaGetLastError();
}

// G: A = [A_L | N_R] contiguous along the contraction, B = [M_L ; B_R^T]
// contiguous along the output columns: the cp.async mainloop with layout 2
static cudaError_t launch_ba(const Launch& L, const BaEpilogue& ep, cudaStream_t s, const DevState* st) {
    if (L.layout != 2) return cudaErrorInvalidValue;
    const bool wd = ep.Dout != nullptr || !ep.Lt;
    const int sm = cfg_smem(L.cfg, 2);
#define GO_(NAME)                                                                                \
    case CFG_##NAME:                                                                             \
        if (wd) k_mma_ba<BDC_CFG_ARGS_##NAME, true><<<L.tiles, 256, sm, s>>>(L.d, L.map, ep, st); \
        else k_mma_ba<BDC_CFG_ARGS_##NAME, false><<<L.tiles, 256, sm, s>>>(L.d, L.map, ep, st);   \
        break;
    switch (L.cfg) {
        GO_(128x64)
        GO_(64x128)
        GO_(64x64)
        default: return cudaErrorInvalidValue;
    }
#undef GO_
    return cudaGetLastError();
}

// ------------------------------------------------------------ small kernels
// the statistics of rows part[b * 8 ..] added up by 256 threads, valid in thread 0
__device__ __forceinline__ void stat_reduce(const double* __restrict__ part, int b0, int b1, double (&v)[5]) {
    __shared__ double red[5][8];
    v[0] = v[2] = -DBL_MAX;
    v[1] = v[3] = v[4] = 0.0;
#pragma unroll 4
    for (int b = b0 + (int)threadIdx.x; b < b1; b += 256) {
        const double* p = part + (size_t)b * 8;
        v[0] = fmax(v[0], p[0]);
        v[1] += p[1];
        v[2] = fmax(v[2], p[2]);
        v[3] += p[3];
        v[4] = fmax(v[4], p[4]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int w = 0; w < 5; ++w) {
            const double t = __shfl_xor_sync(0xFFFFFFFFu, v[w], o);
            v[w] = (w == 1 || w == 3) ? v[w] + t : fmax(v[w], t);
        }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int w = 0; w < 5; ++w) red[w][threadIdx.x >> 5] = v[w];
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int u = 1; u < 8; ++u)
#pragma unroll
        for (int w = 0; w < 5; ++w) v[w] = (w == 1 || w == 3) ? v[w] + red[w][u] : fmax(v[w], red[w][u]);
}

// many partials (large n) first come down to kStatRows rows: one CTA alone
// took 36 us for the 16,512 of 28/13
constexpr int kStatRows = 128, kStatMany = 4096;
__global__ void __launch_bounds__(256) k_fac_stats(const double* __restrict__ part, int nb, double* __restrict__ out,
                                                   const DevState* st) {
    if (gated(st)) return;
    double v[5];
    const int n = (nb + kStatRows - 1) / kStatRows;
    stat_reduce(part, blockIdx.x * n, min(nb, (int)(blockIdx.x + 1) * n), v);
    if (threadIdx.x == 0)
#pragma unroll
        for (int w = 0; w < 5; ++w) out[blockIdx.x * 8 + w] = v[w];
}

__global__ void __launch_bounds__(256)
k_fac_finalize(const double* __restrict__ part, int nb, double a, double eta, DevState* st) {
    if (gated(st)) return;
    double v[5];
    stat_reduce(part, 0, nb, v);
    if (threadIdx.x == 0) fac_finish(v[0], v[1], v[2], v[3], v[4], a, eta, st);
}

// re-scale after an exp over/underflow: Lt -= s, Pw = |O| exp(Lt), sum
__global__ void __launch_bounds__(256)
k_fac_rescale(const uint32_t* __restrict__ reps, int64_t R, int n, int row0, double* Lt, double* Pw,
              double* part, DevState* st, int on_shift_error) {
    if (on_shift_error && st->error != kErrShift) return;  // queued unconditionally in a captured map
    const double s = st->max_logw;  // max of Lt after the failed epilogue
    double sum = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < R; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t x = reps[i], xd = fac_loc(x, n, row0);
        const double l = Lt[xd] - s;
        const double o = (double)orbit_size(x, n);
        Lt[xd] = l;
        const double e = exp(l);
        Pw[xd] = o * e;
        sum = fma(o, e, sum);
    }
    __shared__ double red[256];
    red[threadIdx.x] = sum;
    __syncthreads();
    for (int t = 128; t > 0; t >>= 1) {
        if (threadIdx.x < t) red[threadIdx.x] += red[threadIdx.x + t];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_fac_rescale_finish(const double* part, int nb, double a, DevState* st, int on_shift_error) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (on_shift_error && st->error != kErrShift) return;
    double sE = 0.0;
    for (int b = 0; b < nb; ++b) sE += part[b];
    // Lt now holds logW - (shift + s) with maximum 0
    const double shift_eff = st->shift + st->max_logw;
    const double lnz = log(sE);
    const double ln2 = 0.69314718055994530942;
    const double mx = st->zero_p ? INFINITY : (st->max_d - shift_eff - lnz) / ln2;
    st->best_ub = fmin(st->best_ub, st->max_d);
    st->best_rate = fmax(st->best_rate, st->rate);
    st->lse = shift_eff + lnz;
    st->mx = mx;
    st->max_logw = shift_eff;
    st->log_z = lnz;
    st->shift = -lnz + st->max_d;
    st->zero_p = 0;
    st->error = 0;
    st->iter += 1;
    st->done = !(mx >= a);
}

// one warp
__global__ void k_fac_load_finish(const double* part, int nb, int k, DevState* st) {
    if (blockIdx.x != 0) return;
    const double mx = warp_parts<true>(part, nb, 2);
    const double z = warp_parts<true>(part + 1, nb, 2);
    if (threadIdx.x != 0) return;
    st->log_z = 0.0;
    st->shift = mx + (double)k * 0.69314718055994530942;  // first guess; re-scaled if off
    st->zero_p = (z != 0.0);
}

// ---- per-representative vectors <-> dense rows, one CTA per held row.
// The representatives of row x_hi are a contiguous run of the ascending list
// in ascending x_lo, while the dense row stores column rev(x_lo): the CTA
// ranks the row's representatives by a block scan of the flags in x_lo order
// and moves the run through shared memory, so that both sides are read and
// written in memory order.  Shared memory: the run (8 bytes per column) and
// the ranks (2 bytes per column, 0xFFFF where no representative).
constexpr uint16_t kNoRank = 0xFFFF;

__host__ __device__ constexpr int rows_smem_bytes(int n2) { return (8 + 2) << n2; }

// ranks of the representatives of row xh in x_lo order into rk; returns their
// number (every thread)
__device__ __forceinline__ int row_ranks(uint32_t xh, int n, int n2, uint16_t* rk) {
    __shared__ int wsum[8];
    const int H2 = 1 << n2, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = H2 >= 256 ? H2 / 256 : 1;  // consecutive x_lo per thread
    const int lo0 = tid * C;
    int cnt = 0;
    for (int j = 0; j < C && lo0 + j < H2; ++j) cnt += is_rep((xh << n2) | (uint32_t)(lo0 + j), n) ? 1 : 0;
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int base = incl - cnt, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) base += wsum[w];
        total += wsum[w];
    }
    for (int j = 0; j < C && lo0 + j < H2; ++j) {
        const bool rep = is_rep((xh << n2) | (uint32_t)(lo0 + j), n);
        rk[lo0 + j] = rep ? (uint16_t)base : kNoRank;
        base += rep ? 1 : 0;
    }
    __syncthreads();
    return total;
}

// p -> (Pw, Lt) on the held rows, per-row partials [max ln p, zero flag]
// (k_fac_load's per-element rules)
__global__ void __launch_bounds__(256) k_fac_load_rows(const int64_t* __restrict__ rs, int n, int row0,
                                                       const double* __restrict__ p, double* __restrict__ Pw,
                                                       double* __restrict__ Lt, double* __restrict__ part,
                                                       int strict_zero) {
    extern __shared__ double rsm[];
    const int n2 = n >> 1, H2 = 1 << n2, r = blockIdx.x;
    uint16_t* rk = reinterpret_cast<uint16_t*>(rsm + H2);
    const uint32_t xh = (uint32_t)(row0 + r);
    const int cnt = row_ranks(xh, n, n2, rk);
    const int64_t b0 = rs[r];
    for (int j = threadIdx.x; j < cnt; j += 256) rsm[j] = p[b0 + j];
    __syncthreads();
    double mx = -DBL_MAX;
    int zero = 0;
    double* pw = Pw + ((int64_t)r << n2);
    double* lt = Lt + ((int64_t)r << n2);
    for (int c = threadIdx.x; c < H2; c += 256) {
        const uint32_t xl = reverse_bits((uint32_t)c, n2);
        const uint16_t k = rk[xl];
        if (k == kNoRank) continue;
        const double v = rsm[k];
        pw[c] = (double)orbit_size((xh << n2) | xl, n) * v;
        if (strict_zero) {
            lt[c] = (v > 0.0) ? log(v) : -INFINITY;
            if (v > 0.0) mx = fmax(mx, log(v));
            continue;
        }
        const double l = (v != 0.0) ? log(v) : 0.0;
        lt[c] = (v != 0.0) ? l : __longlong_as_double(0x7ff8000000000000ll);
        mx = fmax(mx, l);
        if (v == 0.0) zero = 1;
    }
    __shared__ double red[8];
    __shared__ int zr[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmax(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        zero |= __shfl_xor_sync(0xFFFFFFFFu, zero, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = mx;
        zr[threadIdx.x >> 5] = zero;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            red[0] = fmax(red[0], red[w]);
            zr[0] |= zr[w];
        }
        part[2 * r] = red[0];
        part[2 * r + 1] = (double)zr[0];
    }
}

// MODE 0: p = Pw / (|O| Z) (k_fac_store's rule); MODE 1: out = dense (a
// gather of D); MODE 2: dense = v (a scatter of h), on the held rows
template <int MODE>
__global__ void __launch_bounds__(256) k_fac_rows(const int64_t* __restrict__ rs, int n, int row0,
                                                  const double* __restrict__ src, double* __restrict__ dst,
                                                  const DevState* st) {
    extern __shared__ double rsm[];
    const int n2 = n >> 1, H2 = 1 << n2, r = blockIdx.x;
    uint16_t* rk = reinterpret_cast<uint16_t*>(rsm + H2);
    const uint32_t xh = (uint32_t)(row0 + r);
    const int cnt = row_ranks(xh, n, n2, rk);
    const int64_t b0 = rs[r];
    const double inv_z = (MODE == 0) ? exp(-st->log_z) : 1.0;
    if (MODE == 2) {
        for (int j = threadIdx.x; j < cnt; j += 256) rsm[j] = src[b0 + j];
        __syncthreads();
        double* d = dst + ((int64_t)r << n2);
        for (int c = threadIdx.x; c < H2; c += 256) {
            const uint16_t k = rk[reverse_bits((uint32_t)c, n2)];
            if (k != kNoRank) d[c] = rsm[k];
        }
        return;
    }
    const double* d = src + ((int64_t)r << n2);
    for (int c = threadIdx.x; c < H2; c += 256) {
        const uint32_t xl = reverse_bits((uint32_t)c, n2);
        const uint16_t k = rk[xl];
        if (k == kNoRank) continue;
        rsm[k] = (MODE == 0) ? d[c] * inv_z / (double)orbit_size((xh << n2) | xl, n) : d[c];
    }
    __syncthreads();
    for (int j = threadIdx.x; j < cnt; j += 256) dst[b0 + j] = rsm[j];
}

// constant parts of LA (AL columns) and RB (BR^T rows) from the bundles
__global__ void k_fill_tables(int H1, int H2, int Kp, const uint16_t* __restrict__ bhi, int strideA,
                              const uint16_t* __restrict__ blo, int strideB, const int* __restrict__ colmap,
                              int KL, int KR, double* LA, double* RB) {
    // colmap[c] for c < KL: bundle offset (of A_j) of AL column c;
    // colmap[KL + c] for c < KR: bundle offset (of B_m) of BR column c
    const int64_t nA = (int64_t)H1 * KL, nB = (int64_t)KR * H2;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nA + nB;
         e += (int64_t)gridDim.x * blockDim.x) {
        if (e < nA) {
            const int64_t xh = e / KL;
            const int c = (int)(e % KL);
            LA[xh * Kp + c] = (double)bhi[xh * strideA + colmap[c]];
        } else {
            const int64_t f = e - nA;
            const int c = (int)(f / H2);
            const int64_t xl = f % H2;
            RB[(int64_t)(KL + c) * H2 + xl] = (double)blo[xl * strideB + colmap[KL + c]];
        }
    }
}

// the low-half tables in dense-column order: row c = table row rev(c)
__global__ void k_permute_rows(const uint16_t* __restrict__ src, int64_t stride, int rows, int n2,
                               uint16_t* __restrict__ dst) {
    const int64_t total = (int64_t)rows * stride;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e / stride, w = e % stride;
        dst[e] = src[(int64_t)reverse_bits((uint32_t)c, n2) * stride + w];
    }
}

// ------------------------------------------------------------ planning
static Operand op_f64(const double* p, int64_t ld, int trans) {
    Operand o;
    o.ptr = p;
    o.ld = ld;
    o.trans = trans;
    return o;
}

static GemmDesc make_desc(Operand A, Operand B, double* C, int64_t ldc_m, int64_t ldc_n, int M, int N, int K) {
    GemmDesc d{};
    d.A = A;
    d.B = B;
    d.C = C;
    d.ldc_m = ldc_m;
    d.ldc_n = ldc_n;
    d.M = M;
    d.N = N;
    d.K = K;
    d.alpha = 1.0;
    d.accumulate = 0;
    return d;
}

// the operand restricted to contraction indices >= k0
static Operand k_offset(Operand o, bool is_a, int64_t k0) {
    if (k0 == 0) return o;
    const int64_t step = is_a ? (o.trans ? k0 * o.ld : k0) : (o.trans ? k0 : k0 * o.ld);
    o.ptr = (const double*)o.ptr + step;
    return o;
}

// S products over consecutive slices of the contraction, output s at C + s * cstride;
// slice boundaries are multiples of 16 (whole k-slices, aligned operands)
static void split_k(std::vector<GemmDesc>& out, const GemmDesc& d, int S, int64_t cstride) {
    for (int s = 0; s < S; ++s) {
        const int64_t k0 = ((int64_t)d.K * s / S) & ~(int64_t)15;
        const int64_t k1 = (s + 1 == S) ? d.K : (((int64_t)d.K * (s + 1) / S) & ~(int64_t)15);
        GemmDesc e = d;
        e.A = k_offset(d.A, true, k0);
        e.B = k_offset(d.B, false, k0);
        e.K = (int)(k1 - k0);
        e.C = d.C + s * cstride;
        out.push_back(e);
    }
}

static int assign_tiles(std::vector<GemmDesc>& v, int cfg) {
    int t = 0;
    for (auto& d : v) {
        d.tiles_m = (d.M + kCfgBM[cfg] - 1) / kCfgBM[cfg];
        d.tiles_n = (d.N + kCfgBN[cfg] - 1) / kCfgBN[cfg];
        d.tile_begin = t;
        t += d.tiles_m * d.tiles_n;
    }
    return t;
}

static void free_launch(Launch& L) {
    cudaFree(L.d);
    cudaFree(L.map);
    L.d = nullptr;
    L.map = nullptr;
}

// the cp.async layout of a list of products, or -1 when a product does not
// qualify (an odd leading dimension or a base that is not 16-byte aligned) or
// the layouts differ
static int cp_layout(const std::vector<GemmDesc>& v) {
    int lay = -2;
    for (const auto& d : v) {
        if ((d.A.ld & 1) || (d.B.ld & 1)) return -1;
        if (((uintptr_t)d.A.ptr & 15) || ((uintptr_t)d.B.ptr & 15)) return -1;
        const int l = (d.A.trans ? 1 : 0) | (d.B.trans ? 0 : 2);
        if (lay == -2) lay = l;
        else if (lay != l) return -1;
    }
    return lay < 0 ? -1 : lay;
}

static cudaError_t make_launch(Launch& L, std::vector<GemmDesc> v, int cfg) {
    free_launch(L);
    L.cfg = cfg;
    L.layout = cp_layout(v);
    L.n = (int)v.size();
    L.tiles = assign_tiles(v, cfg);
    if (v.empty()) return cudaSuccess;
    std::vector<int> map(L.tiles);
    for (int i = 0; i < (int)v.size(); ++i)
        for (int t = 0; t < v[i].tiles_m * v[i].tiles_n; ++t) map[v[i].tile_begin + t] = i;
    cudaError_t e = cudaMalloc(&L.d, sizeof(GemmDesc) * v.size());
    if (e == cudaSuccess) e = upload(L.d, v.data(), sizeof(GemmDesc) * v.size());
    if (e == cudaSuccess) e = cudaMalloc(&L.map, sizeof(int) * map.size());
    if (e == cudaSuccess) e = upload(L.map, map.data(), sizeof(int) * map.size());
    return e;
}

template <typename F>
static float time_ms(bdc_handle* H, F&& launch, cudaError_t* err = nullptr) {
    // the best of three rounds of three launches, after a warm-up launch; a
    // launch that returns an error (or leaves one) makes the time 1e30 and
    // the error is passed out through err
    cudaError_t first = cudaSuccess;
    auto run = [&] {
        if constexpr (std::is_same_v<decltype(launch()), cudaError_t>) {
            const cudaError_t e = launch();
            if (first == cudaSuccess) first = e;
        } else {
            launch();
        }
    };
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    run();
    float best = 1e30f;
    for (int round = 0; round < 3; ++round) {
        cudaEventRecord(a, H->stream);
        for (int r = 0; r < 3; ++r) run();
        cudaEventRecord(b, H->stream);
        cudaEventSynchronize(b);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, a, b);
        best = std::min(best, ms / 3.f);
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    const cudaError_t last = cudaGetLastError();
    if (first == cudaSuccess) first = last;
    if (err) *err = first;
    return first == cudaSuccess ? best : 1e30f;
}

// G with only the tiles that hold representatives (colmax: per dense column
// the largest row of a representative); CTA i runs tile map[i]
static cudaError_t make_tile_launch(Launch& L, GemmDesc d, int cfg, const std::vector<int>& colmax) {
    free_launch(L);
    L.cfg = cfg;
    L.layout = cp_layout({d});
    L.n = 1;
    const int BM = kCfgBM[cfg], BN = kCfgBN[cfg];
    d.tiles_m = (d.M + BM - 1) / BM;
    d.tiles_n = (d.N + BN - 1) / BN;
    d.tile_begin = 0;
    std::vector<int> ids;
    for (int tm = 0; tm < d.tiles_m; ++tm)
        for (int tn = 0; tn < d.tiles_n; ++tn) {
            int mx = -1;
            for (int c = tn * BN; c < std::min(d.N, (tn + 1) * BN); ++c) mx = std::max(mx, colmax[c]);
            if (mx >= tm * BM) ids.push_back(tm * d.tiles_n + tn);
        }
    L.tiles = (int)ids.size();
    if (ids.empty()) return cudaSuccess;
    cudaError_t e = cudaMalloc(&L.d, sizeof(GemmDesc));
    if (e == cudaSuccess) e = upload(L.d, &d, sizeof(GemmDesc));
    if (e == cudaSuccess) e = cudaMalloc(&L.map, sizeof(int) * ids.size());
    if (e == cudaSuccess) e = upload(L.map, ids.data(), sizeof(int) * ids.size());
    return e;
}

// Tuning choices pinned in a text file named by the environment variable
// BDC_TUNE_FILE (lines "n k key a b"): a choice found there is used without
// timing, new choices are appended, so that repeated runs (a profiler's, for
// instance) execute the same kernels.
struct TuneFile {
    std::string path;
    std::map<std::string, std::pair<int, int>> m;
    std::vector<std::string> fresh;
    int n = 0, k = 0;
    void load(int n_, int k_) {
        n = n_;
        k = k_;
        const char* e = getenv("BDC_TUNE_FILE");
        if (!e || !*e) return;
        path = e;
        FILE* f = fopen(path.c_str(), "r");
        if (!f) return;
        int a, b, nn, kk;
        char key[64];
        while (fscanf(f, "%d %d %63s %d %d", &nn, &kk, key, &a, &b) == 5)
            if (nn == n && kk == k) m[key] = {a, b};
        fclose(f);
    }
    bool get(const char* key, int* a, int* b) const {
        auto it = m.find(key);
        if (it == m.end()) return false;
        *a = it->second.first;
        *b = it->second.second;
        return true;
    }
    // whether every one of these choices is made already
    bool has(std::initializer_list<const char*> keys) const {
        return std::all_of(keys.begin(), keys.end(), [&](const char* key) { return m.count(key) != 0; });
    }
    void put(const char* key, int a, int b) {
        if (path.empty()) return;
        m[key] = {a, b};
        char line[128];
        snprintf(line, sizeof(line), "%d %d %s %d %d\n", n, k, key, a, b);
        fresh.push_back(line);
    }
    void save() {
        if (path.empty() || fresh.empty()) return;
        FILE* f = fopen(path.c_str(), "a");
        if (!f) return;
        for (auto& l : fresh) fputs(l.c_str(), f);
        fclose(f);
        fresh.clear();
    }
};

// chooses tile shape (from cfgs) and split of U or V by timing run(candidate),
// the product together with the transform that reads its slices; gen(cfg, S)
// lists the descriptors of a candidate (S: the split of the longest
// contraction, kfull its length), post(cfg, S) tells the transform its slices.
// preset: no timing; the first shape and the largest split, which the timing
// finds for nearly every direct problem's products (G 64x64 for all of them)
template <typename Gen, typename Post, typename Run>
static bdc_status tune_product(bdc_handle* H, TuneFile& tf, const char* key, Launch& L, Gen&& gen, Post&& post, Run&& run,
                               const std::vector<int>& cfgs, int kfull, int max_split, int kmin, const char* what,
                               int* split_out, bool preset) {
    float best = 1e30f;
    int best_cfg = cfgs[0], best_s = 1;
    bool pinned = tf.get(key, &best_cfg, &best_s);
    // (the slices' buffers hold max_split of them)
    if (pinned && (std::find(cfgs.begin(), cfgs.end(), best_cfg) == cfgs.end() || best_s < 1 || best_s > max_split)) {
        pinned = false;
        best_cfg = cfgs[0];
        best_s = 1;
    }
    if (preset && !pinned)
        while (2 * best_s <= max_split && kfull / (2 * best_s) >= kmin) best_s *= 2;
    for (int cfg : cfgs) {
        if (pinned || preset) break;
        for (int S = 1; S <= max_split; S *= 2) {
            if (S > 1 && kfull / S < kmin) break;
            std::vector<GemmDesc> v = gen(cfg, S);
            Launch T;
            BDC_CUDA_TRY(make_launch(T, v, cfg));
            if (T.tiles > 64 * H->num_sms) {
                free_launch(T);
                continue;
            }
            BDC_CUDA_TRY(post(cfg, S));
            cudaError_t e = cudaSuccess;
            const float ms = time_ms(H, [&] { return run(T); }, &e);
            free_launch(T);
            BDC_CUDA_TRY(e);
            if (ms < best) {
                best = ms;
                best_cfg = cfg;
                best_s = S;
            }
        }
    }
    if (!pinned && !preset) tf.put(key, best_cfg, best_s);
    BDC_CUDA_TRY(make_launch(L, gen(best_cfg, best_s), best_cfg));
    BDC_CUDA_TRY(post(best_cfg, best_s));
    *split_out = best_s;
    if (H->verbose)
        printf("bdc: tuned %s: tile %dx%d, split %d, %.1f us with the transform\n", what, kCfgBM[best_cfg],
               kCfgBN[best_cfg], best_s, best * 1e3f);
    return BDC_OK;
}

// slices of a block whose contraction has length kb, when one of length kfull has S
static int block_slices(int S, int kb, int kfull) {
    return std::max(1, (int)(((int64_t)S * kb + kfull - 1) / kfull));
}

// f with the transforms' kernels for slices of up to r characters
template <typename F>
static cudaError_t words_kernels(int r, F&& f) {
    if (word_threads(r) == 512) return f(k_words_q<512, 1>, k_words_d<512, 1>);
    return word_ctas(r) == 3 ? f(k_words_q<256, 3>, k_words_d<256, 3>) : f(k_words_q<256, 1>, k_words_d<256, 1>);
}

// the word transforms of both sides
static cudaError_t launch_words(bool q_side, const FactoredState* F, cudaStream_t s, const DevState* st) {
    const int g = F->plan.ctas, sm = F->words_smem, t = word_threads(F->words_r);
    return words_kernels(F->words_r, [&](auto* q, auto* d) {
        if (q_side) q<<<g, t, sm, s>>>(F->d_plan, F->qparts, st);
        else d<<<g, t, sm, s>>>(F->d_plan, F->lnq_full, st);
        return cudaGetLastError();
    });
}

// the largest transform's shared memory (k = 14), for every handle
static cudaError_t set_words_attrs(int r) {
    const int smem = word_smem(13, 12);
    return words_kernels(r, [&](auto* q, auto* d) {
        const cudaError_t e = cudaFuncSetAttribute(q, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(d, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    });
}

// N(w, v) of every word v in the `len` characters of w, by heap index
static std::vector<int> word_occurrences(int w, int len) {
    std::vector<int> occ((size_t)2 << len, 0);
    occ[1] = 1;
    for (int i = len - 1; i >= 0; --i) {  // the next character ends v or is skipped
        const int b = (w >> i) & 1;
        for (int j = len - i; j > 0; --j)
            for (int v = b; v < (1 << j); v += 2) occ[(1 << j) + v] += occ[(1 << (j - 1)) + (v >> 1)];
    }
    return occ;
}

cudaError_t dgemm_scratch_alloc(DgemmScratch& sc, int max_tiles, cudaStream_t s) {
    dgemm_scratch_free(sc);
    cudaError_t e = cudaMalloc(&sc.desc, sizeof(GemmDesc));
    if (e == cudaSuccess) e = cudaMalloc(&sc.map, sizeof(int) * (size_t)std::max(1, max_tiles));
    if (e == cudaSuccess) e = cudaMemsetAsync(sc.map, 0, sizeof(int) * (size_t)std::max(1, max_tiles), s);
    if (e == cudaSuccess) sc.tiles = max_tiles;
    return e;
}

void dgemm_scratch_free(DgemmScratch& sc) {
    cudaFree(sc.desc);
    cudaFree(sc.map);
    sc = DgemmScratch{};
}

// C (M x N, row stride ldc) = alpha A B^T (+ C when accumulate) for row-major
// A (M x K, stride lda) and B (N x K, stride ldb) on the FP64 tensor-core
// path; a helper for small dense work outside the iteration (the certified
// solver's Newton systems).  The descriptor goes to sc.desc on the same
// stream, so a call does not overwrite it under the previous call's kernel.
cudaError_t dgemm_nt(const DgemmScratch& sc, const double* A, int lda, const double* B, int ldb, double* C, int ldc,
                     int M, int N, int K, double alpha, int accumulate, cudaStream_t s) {
    static bool attrs = false;
    if (!attrs) {
        cudaError_t e = set_smem_attrs();
        if (e != cudaSuccess) return e;
        attrs = true;
    }
    std::vector<GemmDesc> v{make_desc(op_f64(A, lda, 0), op_f64(B, ldb, 1), C, ldc, 1, M, N, K)};
    v[0].alpha = alpha;
    v[0].accumulate = accumulate;
    Launch L;
    L.cfg = CFG_64x64;
    L.layout = cp_layout(v);
    L.n = 1;
    L.tiles = assign_tiles(v, CFG_64x64);
    if (L.tiles > sc.tiles || !sc.desc) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemcpyAsync(sc.desc, v.data(), sizeof(GemmDesc), cudaMemcpyHostToDevice, s);
    L.d = (GemmDesc*)sc.desc;
    L.map = sc.map;
    if (e == cudaSuccess) e = launch_store(L, s, nullptr);
    L.d = nullptr;  // owned by the scratch
    L.map = nullptr;
    return e;
}

bool factored_supports(int n, int k) {
    // needs k < n (W is not the identity), half tables that fit the uint16
    // bundles, a dense 2^{n-1} state that fits comfortably in device memory,
    // and word transforms whose vectors fit in shared memory (k <= 14)
    return k >= 1 && k < n && n >= 2 && n <= 28 && k <= 14;
}

static BaEpilogue make_epilogue(bdc_handle* H);

// ------------------------------------------------------- small problems
// The direct iteration (bdc_direct.cuh) where the folded matrix has 16-bit
// entries, at most 512 output representatives and kDirectBytes in all.  Its
// time grows with the matrix, that of the products hardly: 18/10 (37 MB) 28 us
// an iteration against 45, 22/5 (1,049,600 representatives) 76 against 61.5;
// 21/5 (526,848) takes 24 (42), 16/8 13, 17/9 16 (41).
constexpr int64_t kDirectBytes = 40ll << 20;
constexpr int64_t kDirectReps = 600000;
// one CTA runs a problem of up to this many passes over its rows, many
// iterations a launch (10/5: 3.8 us each); more CTAs share a larger one, one
// iteration a launch
constexpr int kDirectSoloPasses = 6;

static int64_t orbit_count(int len) {  // orbits of {id, rev, comp, rev comp} on `len`-bit words
    if (len == 0) return 1;
    return ((1ll << len) + (1ll << ((len + 1) / 2)) + ((len % 2 == 0) ? (1ll << (len / 2)) : 0)) / 4;
}

static bool direct_supports(const bdc_handle* H) {
    const int64_t ny = (orbit_count(H->k) + 7) / 8 * 8;
    return H->shard_world == 1 && H->k <= 10 && H->C < 65536.0 && H->R <= kDirectReps && H->R * ny * 2 <= kDirectBytes;
}

template <bool SOLO, typename F>
static cudaError_t direct_kernel(int lpx, int m, F&& f) {
    switch (m * 32 + lpx) {
        case 32 + 1: return f(k_direct<1, 1, SOLO>, direct_smem(1, 1));
        case 32 + 2: return f(k_direct<2, 1, SOLO>, direct_smem(2, 1));
        case 96 + 1: return f(k_direct<1, 3, SOLO>, direct_smem(1, 3));
        case 96 + 2: return f(k_direct<2, 3, SOLO>, direct_smem(2, 3));
        case 96 + 4: return f(k_direct<4, 3, SOLO>, direct_smem(4, 3));
        case 96 + 8: return f(k_direct<8, 3, SOLO>, direct_smem(8, 3));
        case 96 + 16: return f(k_direct<16, 3, SOLO>, direct_smem(16, 3));
        default: return cudaErrorInvalidValue;
    }
}

// In a batch the direct iteration of a large problem loses to the products: its
// time grows with the rows of all instances, which no longer fit beside one
// another, that of the products hardly.  Handles above one of these sizes hold
// both forms and a batch of more than kBesideDirect instances takes the
// products.  Measured, ms of 48 accelerated steps, products per word length /
// direct / products: 18/10 x 16 12.4 / 21.1 / 9.4, x 3 5.2 / 5.5 / 3.4, 21/5 x 4 6.3 /
// 7.3 / 5.2, 20/3 x 16 12.3 / 14.2 / 9.5, 18/9 x 8 6.8 / 7.3 / 5.3; below them
// 17/9 x 16 8.4 / 8.3 / 9.1, 16/8 x 16 8.2 / 4.8 / 7.0, 19/7 x 8 6.9 / 6.5 / 5.1.
// The second form is set up without timing its choices (18/10 7 -> 9 ms; 38 with the
// products per word length alone) and takes less memory than the folded matrix.
constexpr int64_t kBesideBytes = 12ll << 20, kBesideReps = 200000;
constexpr int kBesideDirect = 2;

static bool direct_holds_products(const bdc_handle* H) {
    return H->R > kBesideReps || H->R * ((orbit_count(H->k) + 7) / 8 * 8) * 2 > kBesideBytes;
}

static bool runs_direct(const FactoredState* F) {
    return F->direct && !(F->products && F->beside > kBesideDirect);
}

// The CTAs of a launch: alone as many as have a pass over rows to do, one an SM;
// in a batch the instances share the SMs.  Instances that each take all of them
// run one after the other, every one with the latency of a launch and all its
// CTAs adding all shares: 64 iterations of 17/9 x 16 17.7 ms so, 9.0 shared.
static int direct_grid(const bdc_handle* H) {
    return std::max(1, std::min(H->fac->d_grid, H->num_sms / H->fac->beside));
}

void factored_beside(bdc_handle* H, int instances) {
    if (H->fac) H->fac->beside = std::max(1, instances);
}

static cudaError_t launch_direct(bdc_handle* H, int grid, int what, int slot, int iters, double a) {
    FactoredState* F = H->fac;
    auto go = [&](auto* k, int smem) {
        k<<<grid, kDirectThreads, smem, H->stream>>>(F->dp, what, slot, iters, a, F->eta, F->dout, H->d_st);
        return cudaGetLastError();
    };
    return grid == 1 ? direct_kernel<true>(F->d_lpx, F->d_m, go) : direct_kernel<false>(F->d_lpx, F->d_m, go);
}

// `iters` iterations from the current state: one launch with one CTA; else
// one for the first q, one per iteration and one for the last state
static cudaError_t enqueue_direct(bdc_handle* H, double a, int iters) {
    FactoredState* F = H->fac;
    if (iters < 1) return cudaSuccess;
    const int grid = direct_grid(H);
    if (grid == 1) return launch_direct(H, grid, kDirectQ | kDirectD, 0, iters, a);
    cudaError_t e = launch_direct(H, grid, kDirectQ, 0, 0, a);
    // (iters > 0 in the kernel: the slot holds an update's statistics)
    for (int i = 0; i < iters && e == cudaSuccess; ++i)
        e = launch_direct(H, grid, i + 1 < iters ? kDirectQ | kDirectD : kDirectD, i & 1, i, a);
    if (e != cudaSuccess) return e;
    k_direct_finish<<<1, 160, 0, H->stream>>>(F->dp.slot[iters & 1], grid, a, F->eta, H->d_st);
    return cudaGetLastError();
}

static bdc_status direct_init(bdc_handle* H) {
    FactoredState* F = H->fac;
    DirectPlan& P = F->dp;
    std::vector<uint32_t> yreps;
    std::vector<double> members;
    for (uint32_t y = 0; y < (1u << H->k); ++y) {
        if (!is_rep(y, H->k)) continue;
        uint32_t img[4] = {y, reverse_bits(y, H->k), complement_bits(y, H->k), 0};
        img[3] = reverse_bits(img[2], H->k);
        std::sort(img, img + 4);
        members.push_back((double)(std::unique(img, img + 4) - img));
        yreps.push_back(y);
    }
    P.NY = (int)yreps.size();
    P.NYp = (P.NY + 7) / 8 * 8;
    members.resize(P.NYp, 1.0);
    const int pieces = P.NYp / 8;
    // lanes and pieces a lane with the fewest idle slots: k <= 4 has 1 piece,
    // k = 5 .. 10 have 2, 3, 5, 9, 17, 34
    F->d_m = pieces <= 2 ? 1 : 3;
    F->d_lpx = 1;
    while (F->d_lpx * F->d_m < pieces) F->d_lpx *= 2;
    const int per_pass = kDirectWarps * (32 / F->d_lpx) * (F->d_m == 1 ? std::min(F->d_lpx, 4) : std::min(F->d_lpx, 2));
    const int64_t passes = (H->R + per_pass - 1) / per_pass;
    F->d_grid = passes <= kDirectSoloPasses ? 1 : (int)std::min<int64_t>(passes, H->num_sms);
    P.R = H->R;
    P.reps = H->d_reps;
    P.Lt = F->Lt;
    P.Pw = F->Pw;
    P.hx = F->hx;
    P.inv_c = H->inv_c;
    P.n = H->n;
    P.n2 = H->s.n2;
    uint16_t* T = nullptr;
    uint32_t* d_y = nullptr;
    const size_t tb = (size_t)H->R * P.NYp * sizeof(uint16_t), vb = sizeof(double) * P.NYp;
    BDC_CUDA_TRY(cudaMalloc(&T, tb));
    P.T = T;
    BDC_CUDA_TRY(cudaMalloc(&F->d_members, vb));
    P.members = F->d_members;
    for (DirectSlot& S : P.slot) {
        BDC_CUDA_TRY(cudaMalloc(&S.part, vb * F->d_grid));
        BDC_CUDA_TRY(cudaMalloc(&S.stat, sizeof(double) * 8 * F->d_grid));
        BDC_CUDA_TRY(cudaMalloc(&S.state, sizeof(DevState)));
    }
    H->bytes += tb + vb * (2 * F->d_grid + 1);
    BDC_CUDA_TRY(upload(F->d_members, members.data(), vb));
    BDC_CUDA_TRY(cudaMalloc(&d_y, sizeof(uint32_t) * yreps.size()));
    BDC_CUDA_TRY(upload(d_y, yreps.data(), sizeof(uint32_t) * yreps.size()));
    k_direct_table<<<H->num_sms * 8, 256, 0, H->stream>>>(H->s, H->A, H->B, H->d_reps, H->R, d_y, P.NY, P.NYp, T);
    BDC_CUDA_TRY(cudaGetLastError());
    auto attr = [&](auto* k, int smem) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    };
    BDC_CUDA_TRY(direct_kernel<true>(F->d_lpx, F->d_m, attr));
    BDC_CUDA_TRY(direct_kernel<false>(F->d_lpx, F->d_m, attr));
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    cudaFree(d_y);
    F->direct = true;
    if (H->verbose)
        printf("bdc: direct iteration: %d output representatives, %.1f MB, %d lanes a row, %d CTAs\n", P.NY,
               tb / 1048576.0, F->d_lpx, F->d_grid);
    return BDC_OK;
}

bdc_status factored_init(bdc_handle* H) {
    BDC_CUDA_TRY(set_smem_attrs());
    FactoredState* F = new FactoredState();
    H->fac = F;
    TuneFile tf;
    tf.load(H->n, H->k);
    const Split& s = H->s;
    F->H1 = 1 << s.n1;
    F->H2 = 1 << s.n2;
    // every representative is <= its complement, so its top bit is 0 and
    // x_hi < H1 / 2: only those rows of the iterate and of G are needed
    F->H1h = F->H1 / 2;
    // the rows this handle holds: all of them on one GPU; a window of whole
    // rows, balanced by the number of representatives, for shard rank r of w
    // (representatives ascend, and x_hi = x >> n2, so a row window is one
    // contiguous range of them)
    std::vector<uint32_t> hr((size_t)H->R);
    BDC_CUDA_TRY(cudaMemcpyAsync(hr.data(), H->d_reps, sizeof(uint32_t) * hr.size(), cudaMemcpyDeviceToHost,
                                 H->stream));
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    {
        const int w = H->shard_world, r = H->shard_rank;
        if (w < 1 || r < 0 || r >= w || w > F->H1h)
            return fail(BDC_ERR_ARG, "factored engine: shard %d of %d over %d rows", r, w, F->H1h);
        auto below = [&](int row) {  // representatives with x_hi < row
            return (int64_t)(std::lower_bound(hr.begin(), hr.end(), (uint32_t)row << s.n2) - hr.begin());
        };
        auto cut = [&](int q) {  // first row of shard q
            if (q <= 0) return 0;
            if (q >= w) return F->H1h;
            const int64_t target = H->R * q / w;
            int lo = 0, hi = F->H1h;
            while (lo < hi) {
                const int mid = (lo + hi) / 2;
                if (below(mid) >= target) hi = mid;
                else lo = mid + 1;
            }
            return std::max(lo, q);  // at least one row per shard
        };
        const int c0 = std::min(cut(r), F->H1h - (w - r)), c1 = (r + 1 == w) ? F->H1h : std::min(cut(r + 1), F->H1h - (w - r - 1));
        F->row0 = c0;
        F->H1h = c1 - c0;
        F->i0 = below(c0);
        F->Rl = below(c1) - F->i0;
        // where each held row's run of representatives starts (k_fac_rows)
        std::vector<int64_t> rs((size_t)F->H1h + 1);
        for (int q = 0; q <= F->H1h; ++q) rs[(size_t)q] = below(c0 + q) - F->i0;
        BDC_CUDA_TRY(cudaMalloc(&F->d_rowstart, sizeof(int64_t) * rs.size()));
        BDC_CUDA_TRY(upload(F->d_rowstart, rs.data(), sizeof(int64_t) * rs.size()));
        BDC_CUDA_TRY(cudaMalloc(&F->rpart, sizeof(double) * 2 * (size_t)F->H1h));
        F->rows_smem = rows_smem_bytes(s.n2);
        // (a limit belongs to the process: the largest, n = 28, by every handle that needs one)
        if (F->rows_smem > 48 * 1024) {
            constexpr int rows_max = rows_smem_bytes(14);
            BDC_CUDA_TRY(cudaFuncSetAttribute(k_fac_load_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_max));
            BDC_CUDA_TRY(cudaFuncSetAttribute(k_fac_rows<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_max));
            BDC_CUDA_TRY(cudaFuncSetAttribute(k_fac_rows<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_max));
            BDC_CUDA_TRY(cudaFuncSetAttribute(k_fac_rows<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_max));
        }
    }
    // words of length a of the high half, b of the low half
    const int k = H->k, wa = k / 2, wb = k - 1 - wa;
    const int KL = 1 << wa, KR = 1 << wb;
    F->KL = KL;
    F->KR = KR;
    F->Kp = (KL + KR + 7) / 8 * 8;
    const int64_t NX = (int64_t)F->H1h * F->H2;  // the dense rows held
    const int ny = 1 << k;
    const int H1 = F->H1h, H2 = F->H2, Kp = F->Kp;  // H1: the rows kept
    const int max_split = 16;

    auto al = [&](double** p, size_t cnt) -> cudaError_t {
        H->bytes += cnt * sizeof(double);
        return cudaMalloc(p, cnt * sizeof(double) + 16);
    };
    BDC_CUDA_TRY(al(&F->Pw, NX));
    BDC_CUDA_TRY(al(&F->Lt, NX));
    BDC_CUDA_TRY(al(&F->hx, NX));
    const bool direct = direct_supports(H);
    if (direct && !direct_holds_products(H)) {
        BDC_CUDA_TRY(cudaMemsetAsync(F->hx, 0, sizeof(double) * NX, H->stream));
        BDC_CUDA_TRY(cudaMemsetAsync(F->Pw, 0, sizeof(double) * NX, H->stream));
        BDC_CUDA_TRY(cudaMemsetAsync(F->Lt, 0, sizeof(double) * NX, H->stream));
        BDC_CUDA_TRY(al(&F->epart, (size_t)H->nb_upd * 8));
        k_fac_rows<2><<<F->H1h, 256, F->rows_smem, H->stream>>>(F->d_rowstart, H->n, F->row0, H->d_h + F->i0, F->hx,
                                                                nullptr);
        BDC_CUDA_TRY(cudaGetLastError());
        return direct_init(H);
    }
    BDC_CUDA_TRY(al(&F->LA, (size_t)H1 * Kp));
    BDC_CUDA_TRY(al(&F->RB, (size_t)Kp * H2));
    BDC_CUDA_TRY(al(&F->ulpart, (size_t)max_split * H2 * KL));
    BDC_CUDA_TRY(al(&F->vrpart, (size_t)max_split * H1 * KR));
    BDC_CUDA_TRY(al(&F->lnq_full, (size_t)ny));
    BDC_CUDA_TRY(cudaMemsetAsync(F->LA, 0, sizeof(double) * H1 * Kp, H->stream));
    BDC_CUDA_TRY(cudaMemsetAsync(F->RB, 0, sizeof(double) * Kp * H2, H->stream));
    BDC_CUDA_TRY(cudaMemsetAsync(F->hx, 0, sizeof(double) * NX, H->stream));
    BDC_CUDA_TRY(cudaMemsetAsync(F->Pw, 0, sizeof(double) * NX, H->stream));
    BDC_CUDA_TRY(cudaMemsetAsync(F->Lt, 0, sizeof(double) * NX, H->stream));
    BDC_CUDA_TRY(cudaMemsetAsync(F->lnq_full, 0, sizeof(double) * ny, H->stream));

    // low-half tables in dense-column order, and the largest row of a
    // representative in each dense column (for skipping empty tiles)
    {
        const size_t cnt = (size_t)H2 * H->B.stride;
        BDC_CUDA_TRY(cudaMalloc(&F->Bp, cnt * sizeof(uint16_t) + 16));
        H->bytes += cnt * sizeof(uint16_t);
        k_permute_rows<<<H->num_sms * 8, 256, 0, H->stream>>>(H->B.rows, H->B.stride, H2, s.n2, F->Bp);
        BDC_CUDA_TRY(cudaGetLastError());
        F->colmax.assign(H2, -1);
        for (int64_t i = F->i0; i < F->i0 + F->Rl; ++i) {
            const uint32_t xd = fac_pos(hr[i], s.n2);
            const int c = (int)(xd & low_mask(s.n2)), xh = (int)(xd >> s.n2) - F->row0;
            if (xh > F->colmax[c]) F->colmax[c] = xh;
        }
    }

    // constant table columns of LA (AL) and rows of RB (BR^T)
    {
        std::vector<int> colmap(KL + KR);
        for (int c = 0; c < KL; ++c) colmap[c] = bundle_offset(wa) + c;
        for (int c = 0; c < KR; ++c) colmap[KL + c] = bundle_offset(wb) + c;
        int* d_cm = nullptr;
        BDC_CUDA_TRY(cudaMalloc(&d_cm, sizeof(int) * colmap.size()));
        BDC_CUDA_TRY(upload(d_cm, colmap.data(), sizeof(int) * colmap.size()));
        k_fill_tables<<<H->num_sms * 8, 256, 0, H->stream>>>(H1, H2, Kp, H->A.rows + (size_t)F->row0 * H->A.stride,
                                                            H->A.stride, F->Bp,
                                                            H->B.stride, d_cm, KL, KR, F->LA, F->RB);
        BDC_CUDA_TRY(cudaGetLastError());
        BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
        cudaFree(d_cm);
    }
    k_fac_rows<2><<<F->H1h, 256, F->rows_smem, H->stream>>>(F->d_rowstart, H->n, F->row0, H->d_h + F->i0, F->hx,
                                                            nullptr);
    BDC_CUDA_TRY(cudaGetLastError());

    // ---- the word transforms: one CTA per word and slice of 2^r strings of
    // the other half.  The largest r <= 12 (64 KB a tree level) that still
    // gives kWordCtas CTAs: a CTA's first and last steps do not shrink with its
    // slice, but with far fewer CTAs than SMs the rounds' latency is all there
    // is (22/11: 67 us an iteration with 96 CTAs at r = 10, 80 with 64 at 11;
    // 24/12: 165 with 96 at r = 12, 168 with 160 at 11, 190 with 320 at 10).
    // A slice fixes at most 3 characters (WordAux::occ).
    constexpr int kWordCtas = 80;
    {
        WordPlan& P = F->plan;
        P.k = k;
        const int half[2] = {s.n1, s.n2};              // characters of the words' half
        const int bits[2] = {s.n2, s.n1 - 1};          // free characters of the other half
        int rmax = 12;
        auto ctas = [&](int r) {
            return (KL << (bits[0] - std::min(bits[0], r))) + (KR << (bits[1] - std::min(bits[1], r)));
        };
        while (ctas(rmax) < kWordCtas && rmax > std::max({4, bits[0] - 3, bits[1] - 2})) --rmax;
        int cta = 0;
        for (int d = 0; d < 2; ++d) {
            WordSide& S = P.side[d];
            S.words_log = d == 0 ? wa : wb;
            S.last0 = d;  // x_hi read backwards ends in its leading 0
            S.r = std::min(bits[d], rmax);
            S.t = bits[d] - S.r;
            S.leaf0 = d == 0 ? 0 : F->row0;
            S.leaves = d == 0 ? H2 : H1;
            S.cta0 = cta;
            const int W = S.words_log;
            std::vector<double> wt((size_t)2 << (2 * W), 0.0);
            std::vector<WordTerm> terms((size_t)kWordTerms << W, WordTerm{0.0, 0, 0});
            std::vector<int> first((size_t)(kWordMaxHalf + 2) << W, 0);
            for (int w = 0; w < (1 << W); ++w) {
                // (the second side's words are consumed from their last character)
                const int path = d == 0 ? w : (int)reverse_bits((uint32_t)w, W);
                const std::vector<int> in_path = word_occurrences(path, W);
                int cnt = 0;
                for (int j = 0; j <= W; ++j) {
                    first[(size_t)w * (kWordMaxHalf + 2) + j] = cnt;
                    for (int v = 0; v < (1 << j); ++v) {
                        const int occ = in_path[(1 << j) + v];
                        if (!occ) continue;
                        const double c = (double)occ / (double)binom(half[d] - j, W - j);
                        wt[((size_t)w << (W + 1)) + (1 << j) + v] = c;
                        terms[(size_t)w * kWordTerms + cnt++] = WordTerm{c, v, 0};
                    }
                }
                for (int j = W + 1; j < kWordMaxHalf + 2; ++j) first[(size_t)w * (kWordMaxHalf + 2) + j] = cnt;
            }
            const size_t b0 = terms.size() * sizeof(WordTerm), b1 = wt.size() * sizeof(double),
                         b2 = first.size() * sizeof(int);
            BDC_CUDA_TRY(cudaMalloc(&F->d_wtab[d], b0 + b1 + b2));
            uint8_t* tab = (uint8_t*)F->d_wtab[d];
            BDC_CUDA_TRY(upload(tab, terms.data(), b0));
            BDC_CUDA_TRY(upload(tab + b0, wt.data(), b1));
            BDC_CUDA_TRY(upload(tab + b0 + b1, first.data(), b2));
            S.terms = (const WordTerm*)tab;
            S.weight = (const double*)(tab + b0);
            S.first = (const int*)(tab + b0 + b1);
            S.out = d == 0 ? F->RB : F->LA + KL;
            S.leaf_stride = d == 0 ? 1 : Kp;
            S.word_stride = d == 0 ? H2 : 1;
            S.in = d == 0 ? F->ulpart : F->vrpart;
            S.slice_stride = (int64_t)S.leaves << S.words_log;
            // (cleared by an upload like the ones that follow: a memset queued on
            // the handle's stream could land after them)
            const std::vector<uint8_t> none((size_t)(S.leaves + 15) / 16, 0);
            BDC_CUDA_TRY(cudaMalloc(&F->d_ns[d], none.size()));
            BDC_CUDA_TRY(upload(F->d_ns[d], none.data(), none.size()));
            S.ns = F->d_ns[d];
            cta += 1 << (S.words_log + S.t);
            S.part0 = P.parts;
            P.parts += word_parts(S, k);
            if (d == 0) P.parts_l = P.parts;
            F->words_smem = std::max(F->words_smem, word_smem(word_cap(S, k), S.r));
        }
        P.ctas = cta;
        F->words_r = std::max(P.side[0].r, P.side[1].r);
        BDC_CUDA_TRY(set_words_attrs(F->words_r));
        BDC_CUDA_TRY(cudaMalloc(&F->d_plan, sizeof(WordPlan)));
        BDC_CUDA_TRY(upload(F->d_plan, &P, sizeof(WordPlan)));
        BDC_CUDA_TRY(al(&F->qparts, (size_t)P.parts << k));
        // (what a CTA can have no share of stays 0: it is never written)
        BDC_CUDA_TRY(cudaMemsetAsync(F->qparts, 0, sizeof(double) * ((size_t)P.parts << k), H->stream));
        BDC_CUDA_TRY(al(&F->qacc, (size_t)ny));
        const int mb = k - 2 * fold_edge(k);
        std::vector<int> mids;
        for (int m = 0; m < (1 << mb); ++m)
            if (is_rep((uint32_t)m, mb)) mids.push_back(m);
        F->n_mids = (int)mids.size();
        BDC_CUDA_TRY(cudaMalloc(&F->d_mids, sizeof(int) * mids.size()));
        BDC_CUDA_TRY(upload(F->d_mids, mids.data(), sizeof(int) * mids.size()));
    }
    BDC_CUDA_TRY(cudaStreamCreateWithFlags(&F->side, cudaStreamNonBlocking));
    BDC_CUDA_TRY(cudaEventCreateWithFlags(&F->ev_join, cudaEventDisableTiming));
    BDC_CUDA_TRY(cudaEventCreateWithFlags(&F->ev_fork, cudaEventDisableTiming));

    // the candidates below are compared by their times: on an idle GPU the
    // first ones would run at a lower clock and from cold instruction caches
    // (the choices at 22/11 and 23/11 then differed by 15 to 30 us a run; up to
    // n = 16 the products take 6 to 10 us by any of them, and 4 ms is a third of
    // the set-up, as where only a batch takes them)
    if (H->n > 16 && !direct && !tf.has({"u", "v", "g", "oz"})) {
        cudaEvent_t e0, e1;
        BDC_CUDA_TRY(cudaEventCreate(&e0));
        BDC_CUDA_TRY(cudaEventCreate(&e1));
        cudaError_t e = cudaEventRecord(e0, H->stream);
        float ms = 0.f;
        for (int i = 0; i < 100 && ms < 4.f && e == cudaSuccess; ++i) {
            for (int j = 0; j < 16 && e == cudaSuccess; ++j) e = launch_words(true, F, H->stream, nullptr);
            if (e == cudaSuccess) e = cudaEventRecord(e1, H->stream);
            if (e == cudaSuccess) e = cudaEventSynchronize(e1);
            if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        BDC_CUDA_TRY(e);
    }

    // ---- the two products of the q side: U (KL x H2) = AL^T Pw, V (H1h x KR) = Pw BR
    // Only the rows x_hi <= colmax[c] of a dense column c hold
    // representatives: U contracts each block of columns over those rows
    // only, V each block of rows over the columns that reach it.  The split
    // of a block is proportional to its contraction; the transform reads as
    // many slices as a block has.
    {
        // per block of BN columns: the rows it contracts (0: no representative)
        auto col_rows = [&](int n0, int nb) {
            int kb = 0;
            for (int c = n0; c < n0 + nb; ++c) kb = std::max(kb, F->colmax[c] + 1);
            return kb == 0 ? 0 : std::min(H1, (kb + 15) & ~15);  // rows past the last representative are zero
        };
        // A(m = w, kk = x_hi) = LA[x_hi * Kp + w]; B(kk = x_hi, n = col) = Pw; C(w, col) -> U[w][col]
        auto gen = [&](int cfg, int S) {
            std::vector<GemmDesc> v;
            const int BN = kCfgBN[cfg];
            for (int n0 = 0; n0 < H2; n0 += BN) {
                const int nb = std::min(BN, H2 - n0), kb = col_rows(n0, nb);
                if (kb == 0) continue;
                GemmDesc d = make_desc(op_f64(F->LA, Kp, 1), op_f64(F->Pw + n0, H2, 0), F->ulpart + n0, H2, 1, KL, nb, kb);
                split_k(v, d, block_slices(S, kb, H1), (int64_t)H2 * KL);
            }
            return v;
        };
        auto post = [&](int cfg, int S) -> cudaError_t {
            std::vector<uint8_t> ns((size_t)(H2 + 15) / 16, 0);
            const int BN = kCfgBN[cfg];
            for (int c = 0; c < H2; c += 16) {
                const int n0 = c / BN * BN, kb = col_rows(n0, std::min(BN, H2 - n0));
                ns[(size_t)c / 16] = kb == 0 ? 0 : (uint8_t)block_slices(S, kb, H1);
            }
            return upload(F->d_ns[0], ns.data(), ns.size());
        };
        const std::vector<int> cfgs = KL >= 128  ? std::vector<int>{CFG_128x64, CFG_64x64, CFG_64x128}
                                      : KL == 64 ? std::vector<int>{CFG_64x64, CFG_64x128}
                                      : KL == 32 ? std::vector<int>{CFG_32x64, CFG_32x128}
                                                 : std::vector<int>{CFG_16x128};
        bdc_status rc = tune_product(H, tf, "u", F->ul, gen, post, [&](const Launch& T) {
            const cudaError_t e = launch_store(T, H->stream, nullptr);
            return e != cudaSuccess ? e : launch_words(true, F, H->stream, nullptr);
        }, cfgs, H1, max_split, 16, "U = AL^T Pw", &F->S1, direct);
        if (rc != BDC_OK) return rc;
    }
    {
        // per block of BM rows: the columns [clo, clo + kb) that reach it (kb = 0: none)
        auto row_cols = [&](int m0, int* clo_out) {
            int clo = H2, chi = -1;
            for (int c = 0; c < H2; ++c)
                if (F->colmax[c] >= m0) {
                    clo = std::min(clo, c);
                    chi = c;
                }
            if (chi < 0) return 0;
            clo &= ~15;  // whole k-slices; the columns added at either end are zero in these rows
            *clo_out = clo;
            return std::min(H2, (chi + 1 + 15) & ~15) - clo;
        };
        // A(m = x_hi, kk = col) = Pw; B(kk = col, n = w) = RB[(KL + w) * H2 + col]; C(x_hi, w) -> V[w][x_hi]
        auto gen = [&](int cfg, int S) {
            std::vector<GemmDesc> v;
            const int BM = kCfgBM[cfg];
            for (int m0 = 0; m0 < H1; m0 += BM) {
                int clo = 0;
                const int mb = std::min(BM, H1 - m0), kb = row_cols(m0, &clo);
                if (kb == 0) continue;
                const Operand A = k_offset(op_f64(F->Pw + (int64_t)m0 * H2, H2, 0), true, clo);
                const Operand B = k_offset(op_f64(F->RB + (int64_t)KL * H2, H2, 1), false, clo);
                GemmDesc d = make_desc(A, B, F->vrpart + m0, 1, H1, mb, KR, kb);
                split_k(v, d, block_slices(S, kb, H2), (int64_t)H1 * KR);
            }
            return v;
        };
        auto post = [&](int cfg, int S) -> cudaError_t {
            std::vector<uint8_t> ns((size_t)(H1 + 15) / 16, 0);
            const int BM = kCfgBM[cfg];
            for (int r = 0; r < H1; r += 16) {
                int clo = 0;
                const int kb = row_cols(r / BM * BM, &clo);
                ns[(size_t)r / 16] = kb == 0 ? 0 : (uint8_t)block_slices(S, kb, H2);
            }
            return upload(F->d_ns[1], ns.data(), ns.size());
        };
        const std::vector<int> cfgs = KR >= 64   ? std::vector<int>{CFG_64x64, CFG_128x64}
                                      : KR == 32 ? std::vector<int>{CFG_64x32, CFG_128x32}
                                                 : std::vector<int>{CFG_128x16};
        bdc_status rc = tune_product(H, tf, "v", F->vr, gen, post, [&](const Launch& T) {
            // beside U, as it runs in an iteration
            const Launch keep = F->vr;
            F->vr = T;
            cudaError_t e = enqueue_stage(H, ST_QBIG, -INFINITY);
            F->vr = keep;
            return e != cudaSuccess ? e : launch_words(true, F, H->stream, nullptr);
        }, cfgs, H2, max_split, 16, "V = Pw BR", &F->S2, direct);
        if (rc != BDC_OK) return rc;
    }

    // ---- G = LA RB with the BA epilogue; the tile shape is tuned on the
    // zero state (set_p re-initialises everything it touches)
    {
        // (128x128 tiles do not fit the two-CTAs-per-SM register budget of the
        // fused epilogue)
        const int cfgs[3] = {CFG_128x64, CFG_64x128, CFG_64x64};
        int ctas_max = 0;
        for (int c : cfgs) ctas_max = std::max(ctas_max, ((H1 + kCfgBM[c] - 1) / kCfgBM[c]) * ((H2 + kCfgBN[c] - 1) / kCfgBN[c]));
        BDC_CUDA_TRY(al(&F->epart, (size_t)std::max(ctas_max, H->nb_upd) * 8));
        BDC_CUDA_TRY(al(&F->spart, (size_t)kStatRows * 8));
        float best = 1e30f;
        int best_cfg = CFG_128x64;
        GemmDesc d = make_desc(op_f64(F->LA, Kp, 0), op_f64(F->RB, H2, 0), nullptr, 0, 0, H1, H2, Kp);
        BaEpilogue ep{};
        ep.n = H->n;
        ep.n2 = H->s.n2;
        ep.hx = F->hx;
        ep.Lt = F->Lt;
        ep.Pw = F->Pw;
        ep.inv_c = H->inv_c;
        ep.part = F->epart;
        ep.eta = 1.0;
        ep.row0 = F->row0;
        int unused = 0;
        bool pinned = tf.get("g", &best_cfg, &unused);
        if (pinned && std::find(cfgs, cfgs + 3, best_cfg) == cfgs + 3) {
            pinned = false;
            best_cfg = CFG_128x64;
        }
        const bool preset = direct && !pinned;
        if (preset) best_cfg = CFG_64x64;
        for (int c : cfgs) {
            if (pinned || preset) break;
            Launch T;
            BDC_CUDA_TRY(make_tile_launch(T, d, c, F->colmax));
            cudaError_t e = cudaSuccess;
            const float ms = time_ms(H, [&] { return launch_ba(T, ep, H->stream, H->d_st); }, &e);
            BDC_CUDA_TRY(e);
            if (ms < best) {
                best = ms;
                best_cfg = c;
            }
            free_launch(T);
        }
        if (!pinned && !preset) tf.put("g", best_cfg, 0);
        tf.save();
        BDC_CUDA_TRY(make_tile_launch(F->g, d, best_cfg, F->colmax));
        F->ctas_g = F->g.tiles;
        if (H->verbose)
            printf("bdc: tuned G: tile %dx%d, %d of %d tiles hold representatives, %d CTAs, %.1f us%s\n",
                   kCfgBM[best_cfg], kCfgBN[best_cfg], F->g.tiles,
                   ((H1 + kCfgBM[best_cfg] - 1) / kCfgBM[best_cfg]) * ((H2 + kCfgBN[best_cfg] - 1) / kCfgBN[best_cfg]),
                   F->ctas_g, pinned || preset ? 0.f : best * 1e3f, pinned ? " (pinned)" : preset ? " (preset)" : "");
        BDC_CUDA_TRY(cudaMemsetAsync(F->Pw, 0, sizeof(double) * NX, H->stream));
        BDC_CUDA_TRY(cudaMemsetAsync(F->Lt, 0, sizeof(double) * NX, H->stream));
        BDC_CUDA_TRY(cudaMemsetAsync(H->d_st, 0, sizeof(DevState), H->stream));
    }
    // G on the int8 tensor cores (bdc_ozaki.cu), with the slicing of its FP64
    // operands, where that times faster than the FP64 product chosen above;
    // BDC_G_KERNEL=dmma or ozaki forces one of the two
    {
        const char* gk = getenv("BDC_G_KERNEL");
        const bool force_fp = gk && !strcmp(gk, "dmma");
        const bool force_oz = gk && !strcmp(gk, "ozaki");
        int pick = -1, unused = 0;
        // a pinned choice (0: FP64, 8 or 16: int8 with that many epilogue
        // warps); a forced int8 G ignores a pinned FP64 one
        const bool has_pick = tf.get("oz", &pick, &unused);
        const bool pinned = has_pick && !(force_oz && pick == 0);
        if (!force_fp && !(pinned && pick == 0) && (!direct || force_oz)) {
            // an entry of ML is ln q against nonnegative weights that add up to
            // sum_j C(a, j) C(n2, k - j) / C(n1 - j, a - j); NR the same from
            // the other side
            auto weight = [&](int words, int half, int other) {
                double t = 0.0;
                for (int j = 0; j <= words; ++j)
                    t += (double)binom(words, j) * (double)binom(other, k - j) / (double)binom(half - j, words - j);
                return t;
            };
            const double cmax = std::max(1.0, std::max(weight(wa, s.n1, s.n2), weight(wb, s.n2, s.n1)));
            const OzakiInput in{F->LA, F->RB, Kp, KL, KR, H1, H2, F->colmax.data(), F->lnq_full, H->k, cmax};
            const char* why = nullptr;
            bdc_status rc = ozaki_init(H, in, &F->oz, &why);
            if (rc != BDC_OK) return rc;
            float t_fp = 0.f, t_oz[2] = {0.f, 0.f};
            if (F->oz && pinned) {
                F->oz->epi = pick == 8 ? 8 : 16;
            } else if (F->oz) {
                // both on the zeroed state (the products' cost does not depend
                // on the values); the int8 product with 16 and with 8
                // epilogue warps
                const BaEpilogue ep = make_epilogue(H);
                cudaError_t e = cudaSuccess;
                if (!force_oz) {
                    t_fp = time_ms(H, [&] { return launch_ba(F->g, ep, H->stream, H->d_st); }, &e);
                    BDC_CUDA_TRY(e);
                }
                for (int v = 0; v < 2; ++v) {
                    F->oz->epi = v == 0 ? 16 : 8;
                    t_oz[v] = time_ms(H, [&] {
                        const cudaError_t e1 = ozaki_prepare(F->oz, H->d_st, H->stream);
                        return e1 != cudaSuccess ? e1 : ozaki_product(F->oz, ep, H->d_st, H->stream);
                    }, &e);
                    BDC_CUDA_TRY(e);
                }
                F->oz->epi = t_oz[1] < t_oz[0] ? 8 : 16;
                const bool use = force_oz || std::min(t_oz[0], t_oz[1]) < t_fp;
                tf.put("oz", use ? F->oz->epi : 0, 0);
                tf.save();
                BDC_CUDA_TRY(cudaMemsetAsync(F->Pw, 0, sizeof(double) * NX, H->stream));
                BDC_CUDA_TRY(cudaMemsetAsync(F->Lt, 0, sizeof(double) * NX, H->stream));
                BDC_CUDA_TRY(cudaMemsetAsync(H->d_st, 0, sizeof(DevState), H->stream));
                if (!use) {
                    ozaki_free(F->oz);
                    F->oz = nullptr;
                }
            }
            F->use_oz = F->oz != nullptr;
            if (H->verbose) {
                if (F->use_oz)
                    printf("bdc: G on the int8 tensor cores: %d tiles of %dx%d over %d CTAs, %d epilogue warps, "
                           "%d B shared memory, ring of %d, %d FP64 tile%s%s\n", F->oz->tiles, kOzBM, kOzTN,
                           F->oz->grid, F->oz->epi, F->oz->smem, F->oz->stages, 1 + F->oz->two_tiles,
                           F->oz->two_tiles ? "s" : "", t_oz[0] > 0.f ? "" : " (pinned)");
                else
                    printf("bdc: G stays on the FP64 product: %s\n", why ? why : "timed slower");
                if (t_oz[0] > 0.f)
                    printf("bdc: G timed: FP64 %.1f us, int8 with slicing %.1f us (16 epilogue warps), %.1f us (8)\n",
                           t_fp * 1e3f, t_oz[0] * 1e3f, t_oz[1] * 1e3f);
            }
        }
    }
    // U, V; the q-side transform; fold; the D-side transform; G (plus the
    // slicing kernel on the int8 path); finalize
    F->launches_per_iter = (F->ul.n > 0) + (F->vr.n > 0) + 3 + 1 + 1 + (F->use_oz ? 1 : F->ctas_g > kStatMany ? 1 : 0);
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    F->products = true;
    return direct ? direct_init(H) : BDC_OK;
}

void factored_free(bdc_handle* H) {
    FactoredState* F = H->fac;
    if (!F) return;
    for (double* p : {F->Pw, F->Lt, F->hx, F->LA, F->RB, F->ulpart, F->vrpart, F->qparts, F->qacc, F->lnq_full,
                      F->epart, F->spart})
        cudaFree(p);
    cudaFree(F->Bp);
    cudaFree(F->Ddense);
    cudaFree(F->d_rowstart);
    cudaFree(F->rpart);
    cudaFree(F->d_plan);
    cudaFree(F->d_members);
    cudaFree((void*)F->dp.T);
    for (DirectSlot& S : F->dp.slot) {
        cudaFree(S.part);
        cudaFree(S.stat);
        cudaFree(S.state);
    }
    cudaFree(F->d_mids);
    for (auto* d : F->d_wtab) cudaFree(d);
    for (auto* d : F->d_ns) cudaFree(d);
    if (F->side) cudaStreamDestroy(F->side);
    if (F->ev_join) cudaEventDestroy(F->ev_join);
    if (F->ev_fork) cudaEventDestroy(F->ev_fork);
    if (F->graph) cudaGraphExecDestroy(F->graph);
    if (F->cycle) cudaGraphExecDestroy(F->cycle);
    for (auto& m : F->maps)
        if (m.exec) cudaGraphExecDestroy(m.exec);
    cudaFree(F->snap0);
    for (Launch* L : {&F->ul, &F->vr, &F->g}) free_launch(*L);
    ozaki_free(F->oz);
    delete F;
    H->fac = nullptr;
}

static BaEpilogue make_epilogue(bdc_handle* H) {
    FactoredState* F = H->fac;
    BaEpilogue ep;
    ep.n = H->n;
    ep.n2 = H->s.n2;
    ep.hx = F->hx;
    ep.Lt = F->Lt;
    ep.Pw = F->Pw;
    ep.inv_c = H->inv_c;
    ep.part = F->epart;
    ep.st = H->d_st;
    ep.Dout = F->dout;
    ep.eta = F->eta;
    ep.row0 = F->row0;
    return ep;
}

// the stages of one iteration (enum Stage), each gated by DevState::done / error

// acc = the sum of nparts vectors of 2^k -> ln q
static cudaError_t launch_fold(bdc_handle* H, const double* parts, int nparts, cudaStream_t s) {
    const FactoredState* F = H->fac;
    k_words_fold<<<F->n_mids, kFoldThreads, 0, s>>>(parts, nparts, H->k, H->inv_c, F->d_mids, F->lnq_full, H->d_lnq,
                                                   H->d_st);
    return cudaGetLastError();
}

static cudaError_t enqueue_stage(bdc_handle* H, int stage, double a) {
    FactoredState* F = H->fac;
    cudaStream_t s = H->stream;
    cudaError_t e = cudaSuccess;
    switch (stage) {
        case ST_QBIG: {
            // U and V are independent: V runs on a branch beside U
            if ((e = cudaEventRecord(F->ev_fork, s)) != cudaSuccess) return e;
            if ((e = cudaStreamWaitEvent(F->side, F->ev_fork, 0)) != cudaSuccess) return e;
            if ((e = launch_store(F->vr, F->side, H->d_st)) != cudaSuccess) return e;
            if ((e = cudaEventRecord(F->ev_join, F->side)) != cudaSuccess) return e;
            if ((e = launch_store(F->ul, s, H->d_st)) != cudaSuccess) return e;
            return cudaStreamWaitEvent(s, F->ev_join, 0);
        }
        case ST_QSMALL: return launch_words(true, F, s, H->d_st);
        case ST_FOLD: return launch_fold(H, F->qparts, F->plan.parts, s);
        case ST_DSMALL:
            if ((e = launch_words(false, F, s, H->d_st)) != cudaSuccess) return e;
            if (F->use_oz) return ozaki_prepare(F->oz, H->d_st, s);
            break;
        case ST_G:
            if (F->use_oz) return ozaki_product(F->oz, make_epilogue(H), H->d_st, s);
            return launch_ba(F->g, make_epilogue(H), s, H->d_st);
        case ST_FIN:
        {
            const int nb = F->use_oz ? ozaki_partials(F->oz) : F->ctas_g;
            if (nb > kStatMany) {
                k_fac_stats<<<kStatRows, 256, 0, s>>>(F->epart, nb, F->spart, H->d_st);
                k_fac_finalize<<<1, 256, 0, s>>>(F->spart, kStatRows, a, F->eta, H->d_st);
            } else {
                k_fac_finalize<<<1, 256, 0, s>>>(F->epart, nb, a, F->eta, H->d_st);
            }
            break;
        }
    }
    return cudaGetLastError();
}

static cudaError_t enqueue_iterations(bdc_handle* H, double a, int iters) {
    if (runs_direct(H->fac)) return enqueue_direct(H, a, iters);
    for (int i = 0; i < iters; ++i) {
        for (int st = 0; st < ST_COUNT; ++st) {
            cudaError_t e = enqueue_stage(H, st, a);
            if (e != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

static cudaError_t enqueue_iteration(bdc_handle* H, double a) { return enqueue_iterations(H, a, 1); }

cudaError_t factored_enqueue_iterations(bdc_handle* H, double a, int iters) { return enqueue_iterations(H, a, iters); }


// the first shift's inputs over every representative (as k_fac_load writes
// them for its own): a shard sets the same p on every rank, so each one
// derives the same shift without an exchange
__global__ void __launch_bounds__(256) k_lnp_all(const double* __restrict__ p, int64_t R, int strict_zero,
                                                 double* __restrict__ part) {
    double mx = -DBL_MAX;
    int zero = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < R; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = p[i];
        if (strict_zero) {
            if (v > 0.0) mx = fmax(mx, log(v));
            continue;
        }
        mx = fmax(mx, (v != 0.0) ? log(v) : 0.0);
        if (v == 0.0) zero = 1;
    }
    __shared__ double red[256];
    __shared__ int zr[256];
    red[threadIdx.x] = mx;
    zr[threadIdx.x] = zero;
    __syncthreads();
    for (int t = 128; t > 0; t >>= 1) {
        if (threadIdx.x < t) {
            red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + t]);
            zr[threadIdx.x] |= zr[threadIdx.x + t];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = red[0];
        part[2 * blockIdx.x + 1] = (double)zr[0];
    }
}

bdc_status factored_load_p(bdc_handle* H, int strict_zero) {
    FactoredState* F = H->fac;
    // (Pw is zero away from the representatives from set-up on: every kernel
    // writes it only there, and the load rewrites all of them)
    const int nb = H->nb_upd;
    k_fac_load_rows<<<F->H1h, 256, F->rows_smem, H->stream>>>(F->d_rowstart, H->n, F->row0, H->d_p[0] + F->i0, F->Pw,
                                                              F->Lt, F->rpart, strict_zero);
    if (H->shard_world > 1) {
        // the first shift from every rank's p, not only the held rows
        k_lnp_all<<<nb, 256, 0, H->stream>>>(H->d_p[0], H->R, strict_zero, F->epart);
        k_fac_load_finish<<<1, 32, 0, H->stream>>>(F->epart, nb, H->k, H->d_st);
    } else {
        k_fac_load_finish<<<1, 32, 0, H->stream>>>(F->rpart, F->H1h, H->k, H->d_st);
    }
    BDC_CUDA_TRY(cudaGetLastError());
    return BDC_OK;
}

// ------------------------------------------------ passes at the current p
// ln q over every y from the representatives' slots
__global__ void k_lnq_expand(int k, const double* __restrict__ lnq, double* __restrict__ lnq_full) {
    const int y = blockIdx.x * blockDim.x + threadIdx.x;
    if (y < (1 << k)) lnq_full[y] = lnq[orbit_rep((uint32_t)y, k)];
}

// sum over the block partials of sum |O| p D (the evaluation's rate)
__global__ void __launch_bounds__(256) k_eval_rate(const double* __restrict__ part, int nb, double* __restrict__ out) {
    __shared__ double red[8];
    double s = 0.0;
    for (int b = threadIdx.x; b < nb; b += 256) s += part[(size_t)b * 8 + 3];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; ++w) s += red[w];
    *out = s;
}

// whether the passes below run on this handle; a direct one has no products
// (its passes take the count path)
bool factored_has_passes(const bdc_handle* H) {
    return H->engine == BDC_ENGINE_FACTORED && !H->fac->direct && H->shard_world == 1;
}

// A device error that an earlier call returned stays with the handle until the
// next load, and the passes' kernels leave at once while it is set, so a pass
// would hand out what was there before.  Every call that can meet one copies
// the state back, so the host's copy tells.
static bdc_status refuse_after_error(const bdc_handle* H) {
    if (H->h_st->error)
        return fail(BDC_ERR_NUMERIC, "factored engine: device error %d of an earlier call", H->h_st->error);
    return BDC_OK;
}

// ln q of the current iterate into H->d_lnq (0 in the slots that are no
// representative's): the q side of an iteration.  Of the state only `done` is
// written (cleared, as the kernels skip their work while it is set).
bdc_status factored_log_q(bdc_handle* H) {
    if (bdc_status rs = refuse_after_error(H)) return rs;
    const size_t slots = (size_t)1 << (H->k >= 1 ? H->k - 1 : 0);
    BDC_CUDA_TRY(cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), H->stream));
    BDC_CUDA_TRY(cudaMemsetAsync(H->d_lnq, 0, sizeof(double) * slots, H->stream));
    for (int st : {ST_QBIG, ST_QSMALL, ST_FOLD}) BDC_CUDA_TRY(enqueue_stage(H, st, -INFINITY));
    return BDC_OK;
}

// D in dense order, allocated on first use; false where there is no memory for
// it (a gigabyte at n = 28)
bool factored_dense_d(bdc_handle* H) {
    FactoredState* F = H->fac;
    if (F->Ddense) return true;
    const size_t bytes = sizeof(double) * (size_t)F->H1h * F->H2;
    if (cudaMalloc(&F->Ddense, bytes) != cudaSuccess) {
        (void)cudaGetLastError();
        F->Ddense = nullptr;
        return false;
    }
    H->bytes += bytes;
    return true;
}

// the D side from lnq_full: G with an epilogue that leaves the state alone;
// D per representative into D_out, or nowhere (nullptr)
static bdc_status eval_d(bdc_handle* H, double* D_out) {
    FactoredState* F = H->fac;
    if (D_out && !factored_dense_d(H)) return fail(BDC_ERR_CUDA, "no device memory for D in dense order");
    BDC_CUDA_TRY(launch_words(false, F, H->stream, H->d_st));
    BaEpilogue ep = make_epilogue(H);
    ep.Lt = nullptr;
    ep.Dout = D_out ? F->Ddense : nullptr;
    BDC_CUDA_TRY(launch_ba(F->g, ep, H->stream, H->d_st));
    if (!D_out) return BDC_OK;
    k_fac_rows<1><<<F->H1h, 256, F->rows_smem, H->stream>>>(F->d_rowstart, H->n, F->row0, F->Ddense, D_out + F->i0,
                                                            H->d_st);
    BDC_CUDA_TRY(cudaGetLastError());
    return BDC_OK;
}

// D per representative for the ln q in H->d_lnq, into H->d_d
bdc_status factored_divergence(bdc_handle* H) {
    if (bdc_status rs = refuse_after_error(H)) return rs;
    FactoredState* F = H->fac;
    const int ny = 1 << H->k;
    BDC_CUDA_TRY(cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), H->stream));
    k_lnq_expand<<<(ny + 255) / 256, 256, 0, H->stream>>>(H->k, H->d_lnq, F->lnq_full);
    BDC_CUDA_TRY(cudaGetLastError());
    return eval_d(H, H->d_d);
}

// I(p;W) of the current iterate (nats) and, with D_out, D per representative:
// one forward evaluation, the state untouched
bdc_status factored_evaluate(bdc_handle* H, double* D_out, double* rate) {
    FactoredState* F = H->fac;
    bdc_status rc = factored_log_q(H);
    if (rc == BDC_OK) rc = eval_d(H, D_out);
    if (rc != BDC_OK) return rc;
    k_eval_rate<<<1, 256, 0, H->stream>>>(F->epart, F->ctas_g, H->d_scalar + 5);
    BDC_CUDA_TRY(cudaGetLastError());
    BDC_CUDA_TRY(cudaMemcpyAsync(rate, H->d_scalar + 5, sizeof(double), cudaMemcpyDeviceToHost, H->stream));
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    return BDC_OK;
}

// ----------------------------------------------- rows over several GPUs
void factored_shard_range(const bdc_handle* H, int* row0, int* rows, int64_t* i0, int64_t* i1) {
    const FactoredState* F = H->fac;
    *row0 = F->row0;
    *rows = F->H1h;
    *i0 = F->i0;
    *i1 = F->i0 + F->Rl;
}

// q side on the held rows: partial sums acc[y] = sum_{held x} |O(x)| e(x) N(x, y)
// of every term (the fold's first two phases), to the host
bdc_status factored_shard_q(bdc_handle* H, double* acc) {
    FactoredState* F = H->fac;
    cudaStream_t s = H->stream;
    BDC_CUDA_TRY(cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), s));
    BDC_CUDA_TRY(enqueue_stage(H, ST_QBIG, -INFINITY));
    BDC_CUDA_TRY(enqueue_stage(H, ST_QSMALL, -INFINITY));
    const int ny = 1 << H->k;
    k_words_acc<<<(ny + 255) / 256, 256, 0, s>>>(F->qparts, F->plan.parts_l, F->plan.parts, H->k, F->qacc);
    BDC_CUDA_TRY(cudaGetLastError());
    BDC_CUDA_TRY(cudaMemcpyAsync(acc, F->qacc, sizeof(double) * ny, cudaMemcpyDeviceToHost, s));
    BDC_CUDA_TRY(cudaStreamSynchronize(s));
    return BDC_OK;
}

// from the summed acc: ln q, the D side and G with the update on the held
// rows; part5 = this shard's [max D, sum |O| e, max logW, sum |O| p D, zero]
bdc_status factored_shard_d(bdc_handle* H, const double* acc, double* part5) {
    FactoredState* F = H->fac;
    cudaStream_t s = H->stream;
    const int ny = 1 << H->k;
    BDC_CUDA_TRY(cudaMemcpyAsync(F->qacc, acc, sizeof(double) * ny, cudaMemcpyHostToDevice, s));
    BDC_CUDA_TRY(launch_fold(H, F->qacc, 1, s));
    BDC_CUDA_TRY(enqueue_stage(H, ST_DSMALL, -INFINITY));
    BDC_CUDA_TRY(enqueue_stage(H, ST_G, -INFINITY));
    const int nb = F->use_oz ? ozaki_partials(F->oz) : F->ctas_g;
    std::vector<double> part((size_t)nb * 8);
    BDC_CUDA_TRY(cudaMemcpyAsync(part.data(), F->epart, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, s));
    BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, s));
    BDC_CUDA_TRY(cudaStreamSynchronize(s));
    if (H->h_st->error) return fail(BDC_ERR_NUMERIC, "sharded iteration: device error %d", H->h_st->error);
    double mD = -DBL_MAX, sE = 0.0, mL = -DBL_MAX, sR = 0.0, zero = 0.0;
    for (int b = 0; b < nb; ++b) {
        mD = std::max(mD, part[(size_t)b * 8 + 0]);
        sE += part[(size_t)b * 8 + 1];
        mL = std::max(mL, part[(size_t)b * 8 + 2]);
        sR += part[(size_t)b * 8 + 3];
        zero = std::max(zero, part[(size_t)b * 8 + 4]);
    }
    part5[0] = mD;
    part5[1] = sE;
    part5[2] = mL;
    part5[3] = sR;
    part5[4] = zero;
    return BDC_OK;
}

// the update's finish from the combined part5 (max, sum, max, sum, max over
// the shards): ln Z, mx, the bound, the stop test and the next shift, the
// same on every shard
bdc_status factored_shard_finish(bdc_handle* H, const double* part5, double a) {
    FactoredState* F = H->fac;
    cudaStream_t s = H->stream;
    double row[8] = {part5[0], part5[1], part5[2], part5[3], part5[4], 0.0, 0.0, 0.0};
    BDC_CUDA_TRY(cudaMemcpyAsync(F->epart, row, sizeof(row), cudaMemcpyHostToDevice, s));
    k_fac_finalize<<<1, 256, 0, s>>>(F->epart, 1, a, 1.0, H->d_st);
    BDC_CUDA_TRY(cudaGetLastError());
    BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, s));
    BDC_CUDA_TRY(cudaStreamSynchronize(s));
    if (H->h_st->error)
        return fail(BDC_ERR_NUMERIC, "sharded iteration: exp shift out of range (device error %d)", H->h_st->error);
    return BDC_OK;
}

bdc_status factored_store_p(bdc_handle* H, double* p_out) {
    FactoredState* F = H->fac;
    k_fac_rows<0><<<F->H1h, 256, F->rows_smem, H->stream>>>(F->d_rowstart, H->n, F->row0, F->Pw, p_out + F->i0,
                                                            H->d_st);
    BDC_CUDA_TRY(cudaGetLastError());
    return BDC_OK;
}


static bdc_status rescale(bdc_handle* H, double a);

// One BA map on device vectors: p_in (per representative, sum |O| p = 1; a
// zero entry stays zero) -> p_out.  The bound max_x D(x) and the rate I(p;W)
// of p_in (nats) are left in H->h_st->max_d / rate; with D_out set, D(x) of
// p_in per representative.  Leaves the handle's iterate at p_out.
// the kernels of one map, queued on H->stream: load, iteration, re-scale
// when the iteration flagged an out-of-range shift (the kernels check the
// flag themselves), D gather, store, and the state copied to the host mirror
static cudaError_t enqueue_map(bdc_handle* H, const double* p_in, double* p_out, double* D_out) {
    FactoredState* F = H->fac;
    cudaStream_t s = H->stream;
    cudaError_t e = cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    // (Pw is zero away from the representatives from set-up on: every kernel
    // writes it only there, and the load below rewrites all of them)
    const int nb = H->nb_upd;
    k_fac_load_rows<<<F->H1h, 256, F->rows_smem, s>>>(F->d_rowstart, H->n, F->row0, p_in + F->i0, F->Pw, F->Lt,
                                                      F->rpart, 1);
    k_fac_load_finish<<<1, 32, 0, s>>>(F->rpart, F->H1h, H->k, H->d_st);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    F->dout = D_out ? F->Ddense : nullptr;
    e = enqueue_iteration(H, -INFINITY);
    F->dout = nullptr;
    if (e != cudaSuccess) return e;
    k_fac_rescale<<<nb, 256, 0, s>>>(H->d_reps + F->i0, F->Rl, H->n, F->row0, F->Lt, F->Pw, F->epart, H->d_st, 1);
    k_fac_rescale_finish<<<1, 32, 0, s>>>(F->epart, nb, -INFINITY, H->d_st, 1);
    if (D_out)
        k_fac_rows<1><<<F->H1h, 256, F->rows_smem, s>>>(F->d_rowstart, H->n, F->row0, F->Ddense, D_out + F->i0, H->d_st);
    k_fac_rows<0><<<F->H1h, 256, F->rows_smem, s>>>(F->d_rowstart, H->n, F->row0, F->Pw, p_out + F->i0, H->d_st);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, s);
}

// One BA map on device vectors: p_in (per representative, sum |O| p = 1; a
// zero entry stays zero) -> p_out.  The bound max_x D(x) and the rate I(p;W)
// of p_in (nats) are left in H->h_st->max_d / rate; with D_out set, D(x) of
// p_in per representative.  The kernels of a map are captured once per
// (p_in, p_out, D_out) into a CUDA graph (the last four are kept), so a map
// costs one graph launch and one synchronisation.
bdc_status factored_map(bdc_handle* H, const double* p_in, double* p_out, double* D_out) {
    FactoredState* F = H->fac;
    const int64_t NX = (int64_t)F->H1h * F->H2;
    if (D_out && !F->Ddense) {
        BDC_CUDA_TRY(cudaMalloc(&F->Ddense, sizeof(double) * NX));
        H->bytes += sizeof(double) * NX;
    }
    cudaGraphExec_t exec = nullptr;
    for (auto& m : F->maps)
        if (m.exec && m.pin == p_in && m.pout == p_out && m.dout == D_out) exec = m.exec;
    if (!exec) {
        // captured on the handle's own stream, launched on the caller's
        cudaStream_t keep = H->stream;
        BDC_CUDA_TRY(cudaStreamSynchronize(keep));
        H->stream = H->own_stream;
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(H->own_stream, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            e = enqueue_map(H, p_in, p_out, D_out);
            const cudaError_t e2 = cudaStreamEndCapture(H->own_stream, &g);
            if (e == cudaSuccess) e = e2;
        }
        H->stream = keep;
        if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, g, 0);
        if (g) cudaGraphDestroy(g);
        BDC_CUDA_TRY(e);
        auto& slot = F->maps[F->maps_next];
        F->maps_next = (F->maps_next + 1) % 4;
        if (slot.exec) cudaGraphExecDestroy(slot.exec);
        slot.pin = p_in;
        slot.pout = p_out;
        slot.dout = D_out;
        slot.exec = exec;
    }
    BDC_CUDA_TRY(cudaGraphLaunch(exec, H->stream));
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    if (H->h_st->error) return fail(BDC_ERR_NUMERIC, "factored engine: device error %d", H->h_st->error);
    return BDC_OK;
}

bdc_status factored_recover(bdc_handle* H, double a) {
    if (H->h_st->error != kErrShift) return fail(BDC_ERR_NUMERIC, "factored engine: device error %d", H->h_st->error);
    return rescale(H, a);
}

static bdc_status rescale(bdc_handle* H, double a) {
    FactoredState* F = H->fac;
    k_fac_rescale<<<H->nb_upd, 256, 0, H->stream>>>(H->d_reps + F->i0, F->Rl, H->n, F->row0, F->Lt, F->Pw, F->epart, H->d_st, 0);
    k_fac_rescale_finish<<<1, 32, 0, H->stream>>>(F->epart, H->nb_upd, a, H->d_st, 0);
    BDC_CUDA_TRY(cudaGetLastError());
    return BDC_OK;
}

static void fill_stats(bdc_handle* H, long long it0, bdc_stats* stats) {
    if (!stats) return;
    const double ln2 = 0.69314718055994530942;
    stats->iters = H->h_st->iter - it0;
    stats->total_iters = H->h_st->iter;
    stats->mx = H->h_st->mx;
    stats->upper_bound = H->h_st->max_d / ln2;
    stats->rate = H->h_st->rate / ln2;
    stats->lse = H->h_st->lse / ln2;
    stats->best_upper_bound = H->h_st->best_ub / ln2;
    stats->best_rate = H->h_st->best_rate / ln2;
    stats->converged = H->h_st->done;
}

// kGraphIters iterations captured once (per threshold a) on the handle's own
// stream and replayed on whatever stream the handle queues on; the device
// done / error flags make iterations past convergence no-ops
constexpr int kGraphIters = 8;

static bdc_status ensure_graph(bdc_handle* H, double a) {
    FactoredState* F = H->fac;
    if (F->graph && F->graph_a == a) return BDC_OK;
    if (F->graph) {
        cudaGraphExecDestroy(F->graph);
        F->graph = nullptr;
    }
    cudaStream_t keep = H->stream;
    H->stream = H->own_stream;
    BDC_CUDA_TRY(cudaStreamSynchronize(keep));
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(H->own_stream, cudaStreamCaptureModeThreadLocal);
    e = e == cudaSuccess ? enqueue_iterations(H, a, kGraphIters) : e;
    cudaError_t e2 = cudaStreamEndCapture(H->own_stream, &g);
    H->stream = keep;
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&F->graph, g, 0);
    if (g) cudaGraphDestroy(g);
    BDC_CUDA_TRY(e);
    F->graph_a = a;
    return BDC_OK;
}

bdc_status factored_iterate(bdc_handle* H, int64_t max_iters, double a, bdc_stats* stats) {
    FactoredState* F = H->fac;
    BDC_CUDA_TRY(cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), H->stream));
    const long long it0 = H->h_st->iter;
    long long target = it0 + max_iters;
    // the host reads the state after a chunk.  With a threshold the chunks grow
    // from 1, since iterations past the stop still cost their launches (4 us each:
    // 22/1, which stops after one, 120 us from chunks of 8 on, 91 from 1); a direct
    // handle's launches past it cost 1 us.  Without one nothing ends the loop early.
    int64_t chunk = a == -INFINITY ? 256 : F->direct ? 8 : 1;
    for (int guard = 0; guard < 1000000; ++guard) {
        const long long done_iters = H->h_st->iter;
        const int64_t remaining = target - done_iters;
        if (remaining <= 0) break;
        const int64_t c = chunk < remaining ? chunk : remaining;
        // whole graphs for the bulk of the chunk, single iterations for the rest
        const bool solo = F->direct && F->d_grid == 1;  // one launch runs them all
        const int64_t ng = (c >= kGraphIters && !solo) ? c / kGraphIters : 0;
        if (ng > 0) {
            bdc_status rc = ensure_graph(H, a);
            if (rc != BDC_OK) return rc;
        }
        for (int64_t i = 0; i < ng; ++i) BDC_CUDA_TRY(cudaGraphLaunch(F->graph, H->stream));
        if (c > ng * kGraphIters) BDC_CUDA_TRY(enqueue_iterations(H, a, (int)(c - ng * kGraphIters)));
        BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
        BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
        if (H->h_st->error == kErrShift) {
            bdc_status rc = rescale(H, a);
            if (rc != BDC_OK) return rc;
            BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
            BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
        } else if (H->h_st->error) {
            return fail(BDC_ERR_NUMERIC, "factored engine: device error %d", H->h_st->error);
        }
        if (H->h_st->done) break;
        if (chunk < 256) chunk *= 2;
    }
    fill_stats(H, it0, stats);
    return BDC_OK;
}

// ------------------------------------------------------ accelerated loop
// Nesterov-accelerated exponentiated gradient on the simplex, driven by the
// adjoint of I(p;W): its gradient over the probabilities of the strings is
// dI/dp(x) = D(x) - 1, so the mirror (exponentiated-gradient) step of length
// eta is ln p' = ln y + eta D(y) - ln Z, which for eta = 1 and y = p is the
// BA update.  Per step t (all on the device, kAccSteps steps per graph):
//   y_t     = normalise(exp(x_t + beta_t (x_t - x_{t-1}))),  beta_t = t / (t + 3)
//   D(y_t), I(y_t)                 the fused forward/backward (G epilogue)
//   x_{t+1} = ln y_t + eta D(y_t) - ln Z
// with x the normalised log iterate.  Adaptive restart: when I(y_t) falls
// below I(y_{t-1}), the step is discarded, the momentum is dropped (t = 0)
// and the next point is y = x_t.  Every evaluated y gives a valid bracket
// I(y) <= C <= max_x D(x; y), tracked as best_rate / best_ub; the loop stops
// on the device when best_ub - best_rate < the requested gap.
constexpr int kAccSteps = 8;
constexpr double kAccEta = 1.5;

__device__ __forceinline__ double block_sum256(double v) {
    __shared__ double red[256];
    red[threadIdx.x] = v;
    __syncthreads();
    for (int t = 128; t > 0; t >>= 1) {
        if (threadIdx.x < t) red[threadIdx.x] += red[threadIdx.x + t];
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

__device__ __forceinline__ double block_max256(double v) {
    __shared__ double red[256];
    red[threadIdx.x] = v;
    __syncthreads();
    for (int t = 128; t > 0; t >>= 1) {
        if (threadIdx.x < t) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + t]);
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

__device__ __forceinline__ bool acc_gated(const DevState* st) { return st->error != 0 || st->done; }

// the device-side stop (the bracket of the evaluated points is below the gap)
__device__ __forceinline__ bool acc_stop(DevState* st) {
    if (st->best_ub - st->best_rate < st->ng_gap) st->done = 1;
    return st->done != 0;
}

// after the last evaluation of a launch sequence: the host reads done next
__global__ void k_acc_stop(DevState* st) {
    if (acc_gated(st) || threadIdx.x != 0) return;
    acc_stop(st);
}

// decides what the last evaluation means for the iterate: stop, accept
// (mode 1), restart (mode 2) or nothing yet (mode 0, the fresh start)
__global__ void k_acc_decide(DevState* st) {
    if (acc_gated(st) || threadIdx.x != 0) return;
    if (st->ng_mode < 0) {  // set by the host: nothing evaluated since the start
        st->ng_mode = 0;
        st->ng_t = 0;
        st->ng_prev_rate = -DBL_MAX;
        return;
    }
    if (acc_stop(st)) return;
    if (st->rate >= st->ng_prev_rate) {
        st->ng_mode = 1;
        st->ng_prev_rate = st->rate;
        st->ng_t += 1;
    } else {
        st->ng_mode = 2;
        st->ng_t = 0;
        st->ng_prev_rate = -DBL_MAX;
    }
}

// x_t (dense, at representatives), the extrapolated ln y into Lt and its
// |O| y into Pw in one pass, two columns a thread with 16-byte accesses; block
// max of ln y and block sums of |O| y.  ln y is near-normalised (y = x times a
// power of the last step), so exp needs no shift; k_acc_setz redoes the pass
// where it would.  Bound by memory: two reads and three writes of a double a
// representative.  Measured at 24/12, a whole step: 251 us with a pass for ln y,
// a pass for its exponentials and four single-block launches, 219 us now
// (155 us of it the iteration).
__global__ void __launch_bounds__(256) k_acc_extrap(int64_t pairs, int n, int row0, double* __restrict__ xa,
                                                    double* __restrict__ Lt, double* __restrict__ Pw,
                                                    double* __restrict__ part, const DevState* st) {
    if (acc_gated(st)) return;
    const int mode = st->ng_mode;
    const double lnz = st->log_z;
    const double beta = (double)st->ng_t / ((double)st->ng_t + 3.0);
    const int n2 = n >> 1;
    const uint32_t mask = low_mask(n2), odd = (uint32_t)n & 1u;
    double mx = -DBL_MAX, sum = 0.0;
    constexpr int U = 2;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j0 < pairs; j0 += U * step) {
        double2 old[U], lt[U];
        bool in[U][2];
        uint32_t r[U], c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t j = j0 + u * step;
            const uint32_t xd = 2u * (uint32_t)j;
            r[u] = (xd >> n2) + (uint32_t)row0;
            c[u] = xd & mask;
            in[u][0] = j < pairs && dense_is_rep(r[u], c[u], mask, odd);
            in[u][1] = j < pairs && dense_is_rep(r[u], c[u] + 1u, mask, odd);
            if (in[u][0] || in[u][1]) {
                old[u] = reinterpret_cast<const double2*>(xa)[j];
                if (mode == 1) lt[u] = reinterpret_cast<const double2*>(Lt)[j];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!in[u][0] && !in[u][1]) continue;
            const int64_t j = j0 + u * step;
            double nx[2], y[2], pw[2];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const double ao = v ? old[u].y : old[u].x;
                if (mode == 1) {
                    nx[v] = (v ? lt[u].y : lt[u].x) - lnz;
                    // an input at exact zero (ln p = -inf) stays there
                    y[v] = (nx[v] == -INFINITY) ? nx[v] : nx[v] + beta * (nx[v] - ao);
                } else {
                    nx[v] = y[v] = ao;
                }
                if (in[u][v]) {
                    pw[v] = dense_orbit(r[u], c[u] + v, mask, odd) * exp(y[v]);
                    mx = fmax(mx, y[v]);
                    sum += pw[v];
                }
            }
            if (in[u][0] && in[u][1]) {
                if (mode == 1) reinterpret_cast<double2*>(xa)[j] = make_double2(nx[0], nx[1]);
                reinterpret_cast<double2*>(Lt)[j] = make_double2(y[0], y[1]);
                reinterpret_cast<double2*>(Pw)[j] = make_double2(pw[0], pw[1]);
            } else {
                const int v = in[u][0] ? 0 : 1;
                if (mode == 1) xa[2 * j + v] = nx[v];
                Lt[2 * j + v] = y[v];
                Pw[2 * j + v] = pw[v];
            }
        }
    }
    mx = block_max256(mx);
    sum = block_sum256(sum);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = mx;
        part[2 * blockIdx.x + 1] = sum;
    }
}

// ln Z of y and the exp shift of the next update (max ln y - ln Z + eta * last
// bound), by the first block.  Where max ln y is so far from 0 that exp lost
// range, which a start far from the optimum brings about, the grid takes |O|
// exp(ln y - max) for all of y itself and its last block finishes: every block
// reduces the partials, so that the common case waits for nothing.  Measured at
// 22/11, 32 steps: from such a start 5.0 ms with that pass in one block, 3.3 ms
// now; 3.3 ms from an even start, before and now.
constexpr double kAccRange = 40.0;  // (a uniform start over 2^28 inputs has -19.4)
__global__ void __launch_bounds__(256) k_acc_setz(double* __restrict__ part, int nb, double eta, int64_t nx, int n,
                                                  int row0, double* __restrict__ Lt, double* __restrict__ Pw,
                                                  DevState* st) {
    if (acc_gated(st)) return;
    double mx = -DBL_MAX, sum = 0.0;
    for (int b = threadIdx.x; b < nb; b += 256) {
        mx = fmax(mx, part[2 * b]);
        sum += part[2 * b + 1];
    }
    mx = block_max256(mx);
    if (fabs(mx) <= kAccRange) {
        if (blockIdx.x != 0) return;
        sum = block_sum256(sum);
    } else {
        const int n2 = n >> 1;
        const uint32_t mask = low_mask(n2), odd = (uint32_t)n & 1u;
        sum = 0.0;
        for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < nx; i += gridDim.x * (int64_t)256) {
            const uint32_t xd = (uint32_t)i, r = (xd >> n2) + (uint32_t)row0, c = xd & mask;
            if (!dense_is_rep(r, c, mask, odd)) continue;
            const double l = Lt[xd] - mx, v = dense_orbit(r, c, mask, odd) * exp(l);
            Lt[xd] = l;
            Pw[xd] = v;
            sum += v;
        }
        sum = block_sum256(sum);
        double* shares = part + 2 * nb;  // [gridDim.x], beside the partials that others may still read
        __shared__ bool last;
        if (threadIdx.x == 0) {
            shares[blockIdx.x] = sum;
            __threadfence();
            last = atomicAdd(&st->ticket[3], 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
        sum = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) sum += __ldcg(shares + b);
        sum = block_sum256(sum);
        if (threadIdx.x == 0) st->ticket[3] = 0u;
        mx = 0.0;
    }
    if (threadIdx.x != 0) return;
    const double lnz = log(sum);
    st->log_z = lnz;
    st->shift = mx - lnz + eta * st->max_d;
}

static cudaError_t enqueue_acc_step(bdc_handle* H, double eta) {
    FactoredState* F = H->fac;
    if (!F->snap0) return cudaErrorInvalidValue;  // factored_acc_buffers first
    cudaStream_t s = H->stream;
    const int nb = H->nb_upd;
    k_acc_decide<<<1, 32, 0, s>>>(H->d_st);
    const int64_t nx = (int64_t)F->H1h << H->s.n2;  // the dense positions of the held rows
    k_acc_extrap<<<nb, 256, 0, s>>>(nx / 2, H->n, F->row0, F->snap0, F->Lt, F->Pw, F->epart, H->d_st);
    k_acc_setz<<<nb, 256, 0, s>>>(F->epart, nb, eta, nx, H->n, F->row0, F->Lt, F->Pw, H->d_st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const double keep = F->eta;
    F->eta = eta;
    e = enqueue_iteration(H, -INFINITY);
    F->eta = keep;
    return e;
}

cudaError_t factored_enqueue_acc_steps(bdc_handle* H, int steps, double eta) {
    for (int i = 0; i < steps; ++i) {
        cudaError_t e = enqueue_acc_step(H, eta);
        if (e != cudaSuccess) return e;
    }
    k_acc_stop<<<1, 32, 0, H->stream>>>(H->d_st);
    return cudaGetLastError();
}

// the loop's snapshot x_t (dense, allocated on first use)
bdc_status factored_acc_buffers(bdc_handle* H) {
    FactoredState* F = H->fac;
    if (F->snap0) return BDC_OK;
    const size_t NX = (size_t)F->H1h * F->H2;
    BDC_CUDA_TRY(cudaMalloc(&F->snap0, sizeof(double) * NX));
    H->bytes += sizeof(double) * NX;
    return BDC_OK;
}

// x_t = the current normalised log iterate; nothing evaluated yet
__global__ void __launch_bounds__(256) k_acc_init(int64_t nx, int n, int row0, const double* __restrict__ Lt,
                                                  double* __restrict__ xa, DevState* st,
                                                  double gap_nats) {
    const double lnz = st->log_z;
    const int n2 = n >> 1;
    const uint32_t mask = low_mask(n2);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nx; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t xd = (uint32_t)i;
        if (!dense_is_rep((xd >> n2) + (uint32_t)row0, xd & mask, mask, (uint32_t)n & 1u)) continue;
        xa[xd] = Lt[xd] - lnz;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->ng_mode = -1;
        st->ng_gap = gap_nats;
        st->done = 0;
    }
}

bdc_status factored_acc_start(bdc_handle* H, double gap_bits) {
    bdc_status rc = factored_acc_buffers(H);
    if (rc != BDC_OK) return rc;
    FactoredState* F = H->fac;
    k_acc_init<<<H->nb_upd, 256, 0, H->stream>>>((int64_t)F->H1h << H->s.n2, H->n, F->row0, F->Lt, F->snap0, H->d_st,
                                                 gap_bits * 0.69314718055994530942);
    BDC_CUDA_TRY(cudaGetLastError());
    return BDC_OK;
}

double factored_acc_eta() {
    const char* e = getenv("BDC_ACCEL_STEP");
    const double v = (e && *e) ? atof(e) : kAccEta;
    return (v > 0.0 && v <= 4.0) ? v : kAccEta;
}

static bdc_status ensure_cycle_graph(bdc_handle* H, double eta) {
    FactoredState* F = H->fac;
    if (F->cycle && F->cycle_eta == eta) return BDC_OK;
    // the snapshot vectors must exist before the steps are captured
    bdc_status rc = factored_acc_buffers(H);
    if (rc != BDC_OK) return rc;
    if (F->cycle) {
        cudaGraphExecDestroy(F->cycle);
        F->cycle = nullptr;
    }
    cudaStream_t keep = H->stream;
    H->stream = H->own_stream;
    BDC_CUDA_TRY(cudaStreamSynchronize(keep));
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(H->own_stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) e = factored_enqueue_acc_steps(H, kAccSteps, eta);
    cudaError_t e2 = cudaStreamEndCapture(H->own_stream, &g);
    H->stream = keep;
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&F->cycle, g, 0);
    if (g) cudaGraphDestroy(g);
    BDC_CUDA_TRY(e);
    F->cycle_eta = eta;
    return BDC_OK;
}

bdc_status factored_accelerate(bdc_handle* H, int64_t max_evals, double gap_bits, bdc_stats* stats) {
    FactoredState* F = H->fac;
    const double ln2 = 0.69314718055994530942;
    const double eta = factored_acc_eta();
    BDC_CUDA_TRY(cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), H->stream));
    BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    const long long it0 = H->h_st->iter;
    // a plain step first when the iterate still carries the caller's exact
    // zeros (ln 0 = 0 applies to the first update only)
    if (H->h_st->iter == 0 && max_evals > 0) {
        bdc_status rc = factored_iterate(H, 1, -INFINITY, nullptr);
        if (rc != BDC_OK) return rc;
    }
    bool converged = (H->h_st->best_ub - H->h_st->best_rate) / ln2 < gap_bits;
    if (!converged && H->h_st->iter - it0 < max_evals) {
        bdc_status rc = ensure_cycle_graph(H, eta);
        if (rc != BDC_OK) return rc;
        rc = factored_acc_start(H, gap_bits);
        if (rc != BDC_OK) return rc;
        int64_t chunk = 1;
        for (int guard = 0; guard < 1000000; ++guard) {
            const int64_t remaining = max_evals - (H->h_st->iter - it0);
            // whole graphs while they fit, single steps for the rest
            if (remaining <= 0) break;
            if (remaining >= kAccSteps) {
                const int64_t c = std::min<int64_t>(chunk, remaining / kAccSteps);
                for (int64_t i = 0; i < c; ++i) BDC_CUDA_TRY(cudaGraphLaunch(F->cycle, H->stream));
            } else {
                BDC_CUDA_TRY(factored_enqueue_acc_steps(H, (int)remaining, eta));
            }
            BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
            BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
            if (H->h_st->error == kErrShift) {
                // an exp shift went out of range: finish that evaluation by
                // re-scaling; the next step's decision takes it from there
                rc = rescale(H, -INFINITY);
                if (rc != BDC_OK) return rc;
                BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
                BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
            } else if (H->h_st->error) {
                return fail(BDC_ERR_NUMERIC, "accelerated loop: device error %d", H->h_st->error);
            }
            if (H->h_st->done) break;
            if (chunk < 64) chunk *= 2;
        }
        converged = (H->h_st->best_ub - H->h_st->best_rate) / ln2 < gap_bits;
    }
    BDC_CUDA_TRY(cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), H->stream));
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    fill_stats(H, it0, stats);
    if (stats) stats->converged = converged;
    return BDC_OK;
}

// a direct handle's iterations have no stages, and a chain of them reads the
// folded matrix once each: the chain is timed as a whole
static bdc_status direct_profile(bdc_handle* H, int iters, bdc_profile_t* out) {
    FactoredState* F = H->fac;
    cudaEvent_t ev[2];
    for (auto& e : ev) BDC_CUDA_TRY(cudaEventCreate(&e));
    const long long target = H->h_st->iter + iters;
    double tot = 0.0;
    while (H->h_st->iter < target) {
        BDC_CUDA_TRY(cudaEventRecord(ev[0], H->stream));
        BDC_CUDA_TRY(enqueue_iterations(H, -INFINITY, (int)(target - H->h_st->iter)));
        BDC_CUDA_TRY(cudaEventRecord(ev[1], H->stream));
        BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
        BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ev[0], ev[1]);
        tot += ms;
        if (!H->h_st->error) continue;
        // an out-of-range shift interrupted the chain: finish that iteration
        bdc_status rc = factored_recover(H, -INFINITY);
        if (rc != BDC_OK) return rc;
        BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
        BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    }
    for (auto& e : ev) cudaEventDestroy(e);
    out->ms_q = out->ms_fold = out->ms_update = 0.0;
    out->ms_iter = out->ms_d = out->ms_main = tot / iters;
    out->work_main = 4.0 * (double)H->R * (double)F->dp.NY;
    out->bytes_main = (double)H->R * (2.0 * (double)F->dp.NYp + 40.0);
    out->launches = 1;
    out->iters = iters;
    out->main_kind = 3;
    return BDC_OK;
}

bdc_status factored_profile(bdc_handle* H, int iters, bdc_profile_t* out) {
    FactoredState* F = H->fac;
    BDC_CUDA_TRY(cudaMemsetAsync(&H->d_st->done, 0, sizeof(int), H->stream));
    if (F->direct) return direct_profile(H, iters, out);
    cudaEvent_t ev[ST_COUNT + 1];
    for (auto& e : ev) BDC_CUDA_TRY(cudaEventCreate(&e));
    double acc[ST_COUNT] = {0}, tot = 0;
    for (int it = 0; it < iters; ++it) {
        BDC_CUDA_TRY(cudaEventRecord(ev[0], H->stream));
        for (int st = 0; st < ST_COUNT; ++st) {
            BDC_CUDA_TRY(enqueue_stage(H, st, -INFINITY));
            BDC_CUDA_TRY(cudaEventRecord(ev[st + 1], H->stream));
        }
        BDC_CUDA_TRY(cudaEventSynchronize(ev[ST_COUNT]));
        BDC_CUDA_TRY(cudaMemcpy(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost));
        if (H->h_st->error == kErrShift) {
            bdc_status rc = rescale(H, -INFINITY);
            if (rc != BDC_OK) return rc;
        }
        float ms;
        for (int st = 0; st < ST_COUNT; ++st) {
            cudaEventElapsedTime(&ms, ev[st], ev[st + 1]);
            acc[st] += ms;
        }
        cudaEventElapsedTime(&ms, ev[0], ev[ST_COUNT]);
        tot += ms;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    BDC_CUDA_TRY(cudaMemcpyAsync(H->h_st, H->d_st, sizeof(DevState), cudaMemcpyDeviceToHost, H->stream));
    BDC_CUDA_TRY(cudaStreamSynchronize(H->stream));
    out->ms_q = (acc[ST_QBIG] + acc[ST_QSMALL]) / iters;
    out->ms_fold = acc[ST_FOLD] / iters;
    out->ms_d = (acc[ST_DSMALL] + acc[ST_G]) / iters;
    out->ms_update = acc[ST_FIN] / iters;
    out->ms_iter = tot / iters;
    out->ms_main = acc[ST_G] / iters;
    // algorithmic work of G: one K-long dot product per representative
    out->work_main = 2.0 * (double)H->R * (double)(F->KL + F->KR);
    out->launches = F->launches_per_iter;
    out->iters = iters;
    out->main_kind = F->use_oz ? 2 : 1;
    out->bytes_main = 40.0 * (double)F->Rl;
    return BDC_OK;
}

}  // namespace bdc
