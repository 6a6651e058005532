// bdc_words.cuh -- the word transforms of the factored engine: the part of
// both passes between the large products and ln q.
//
// The products contract one half of x with words of one length only.  With a
// = floor(k/2), b = k - 1 - a, a term j <= a of the split identity (N(x, y) =
// sum_j N(x_hi, y_hi) N(x_lo, y_lo), |y_hi| = j; total_transitions,
// backend/BAA.cu:340-395) uses
//     N(x_hi, v) = sum_{|w| = a} N(x_hi, w) N(w, v) / C(n1 - j, a - j),  |v| = j
// (every occurrence of v in x_hi extends to C(n1 - j, a - j) sets of a
// positions), and a term j > a the same with the last b characters of y and
// x_lo.  So every term j <= a together is
//     sum_{|w| = a} N(x_hi, w) F_w(x_lo),
//     F_w(x_lo) = sum_z N(x_lo, z) c_w[z],
//     c_w[z] = sum_{|v| = k - |z|} N(w, v) ln q(v z) / C(n1 - |v|, a - |v|),
// a product with 2^a columns instead of one per word of every length up to a
// (2^{a+1} - 1), and F_w is a transform of ln q: consume the characters of w,
// then those of x_lo.  Consuming a character b on the left of a coefficient
// vector over words is c[z] <- c[z] + c[b z] (an occurrence of a word in b x'
// either skips the b or matches it with its first character).  The q side
// runs the transposed steps.  The terms j > a are the mirror image (words
// consumed from the right); ln q is invariant under reversal, so the same
// code serves both halves with w and x_hi read backwards.
//
// One CTA per word w and slice of the other half's strings.  Consuming w, the
// first step, needs no steps of its own: c_w[z] is a sum over the distinct
// subsequences v of w (at most 54 for 7 characters), each a run of ln q at
// stride one, and the transposed step adds a + 1 products per output y.  The
// other half is consumed four characters at a time in shared memory, the
// coefficient vectors in heap order (word z at index 2^{|z|} + value): a
// thread takes one tail z of one node (a fixed prefix), reads the 31
// coefficients c[v z], |v| <= 4, and forms the 16 children's coefficients at
// z in registers (83 additions), so a round of four characters costs 3 shared
// memory accesses per output instead of 12.
//
// Bound by the latency of the rounds (2-4 warps a scheduler, a block barrier
// between rounds), not by a pipe.  At 24/12 q 25 us, fold 8.2, D 22 us; the
// products per word length that this replaces took 46 + 19 + 50 us and let the
// large products contract 190 words instead of 96: an iteration 312 -> 155 us
// with the rest.  512 threads a CTA (22/11: 67 -> 77 us an iteration) and
// shorter trees (r = 9, 10 at 24/12: 193-228 us) were slower.
#pragma once

#include "bdc_common.cuh"

namespace bdc {

constexpr int kWordMaxHalf = 7;  // characters of a word: floor(k / 2), k <= 14
constexpr int kWordTerms = 64;   // distinct subsequences of a word (54 for 0101010)

struct WordTerm {
    double weight;
    int v, pad;
};

// One half's words and the other half's strings ("leaves")
struct WordSide {
    int words_log;      // a (or b): 2^words_log words
    int last0;          // 1: the strings carry a fixed last character 0 beside the leaf bits
    int r, t;           // leaf bits: r >= 1 in the tree, t leading ones fixed per CTA
    int leaf0, leaves;  // leaves [leaf0, leaf0 + leaves) are held
    int cta0;           // first CTA of this side
    int part0;          // its first partial q vector (word_parts of them)
    // N(w, v) / C(half length - |v|, words_log - |v|) for the words |v| <= words_log:
    // dense by heap index, and the nonzero ones by length (terms of w: [first[w][j], first[w][j + 1]))
    const double* weight;        // [2^words_log][2^{words_log + 1}]
    const struct WordTerm* terms;  // [2^words_log][kWordTerms]
    const int* first;            // [2^words_log][kWordMaxHalf + 2]
    // D side: F_w(leaf) goes to out[(leaf - leaf0) * leaf_stride + w * word_stride]
    double* out;
    int64_t leaf_stride, word_stride;
    // q side: in[s * slice_stride + w * leaves + (leaf - leaf0)] summed over
    // the slices s < ns[(leaf - leaf0) >> 4]
    const double* in;
    int64_t slice_stride;
    const uint8_t* ns;
};

struct WordPlan {
    WordSide side[2];
    int k;
    int ctas;           // CTAs of both sides
    int parts_l, parts; // partial q vectors of the first side and of both
};

// An output word y = v z takes |v| <= words_log characters from this half and z
// from the other, which has `reach` of them.  So v has at least word_least
// characters, and the other half's words at most word_cap; for k above n / 2
// that leaves few of the splits.
__host__ __device__ __forceinline__ int word_reach(const WordSide& S) { return S.r + S.t + S.last0; }
__host__ __device__ __forceinline__ int word_least(const WordSide& S, int k) {
    return k > word_reach(S) ? k - word_reach(S) : 0;
}
__host__ __device__ __forceinline__ int word_cap(const WordSide& S, int k) {
    return k - 1 < word_reach(S) ? k - 1 : word_reach(S);
}
// k = n - 1: v is all of w and z all of the other half, so a transform is a
// permutation of ln q and its transpose one of U, and the side's shares of acc
// are one vector.  The general steps, on 2^k coefficients a word, took 15/14 from
// the 44 us an iteration of the products per word length to 90; 34 so (12/11: 34,
// 37, 24; with least and cap alone 15/14 46).  Those two are what short halves
// need elsewhere: 16/14 92 -> 59, 17/14 98 -> 62 (92 and 91 per word length).
__host__ __device__ __forceinline__ bool word_whole(const WordSide& S, int k) {
    return k - S.words_log == word_reach(S);
}
__host__ __device__ __forceinline__ int word_parts(const WordSide& S, int k) {
    return word_whole(S, k) ? 1 : 1 << (S.t + S.words_log);
}

__device__ __forceinline__ int word_len(int h) { return 31 - __clz(h); }

// N(p, u) of the words u at heap indices 1 .. 15 in the c <= 3 characters p
// (bit c - 1 first), one thread per word
__device__ __forceinline__ double word_occ(int p, int c, int u) {
    const int d = word_len(u);
    int n1 = 0, n2 = 0, n3 = 0;  // occurrences of the word's first 1, 2, 3 characters
    for (int i = c - 1; i >= 0; --i) {
        const int b = (p >> i) & 1;
        if (d >= 3 && (u & 1) == b) n3 += n2;
        if (d >= 2 && ((u >> (d - 2)) & 1) == b) n2 += n1;
        if (d >= 1 && ((u >> (d - 1)) & 1) == b) n1 += 1;
    }
    return (double)(d == 0 ? 1 : d == 1 ? n1 : d == 2 ? n2 : n3);
}

// shared memory beside the two buffers: the weights (or terms) of w and N(p, u)
struct WordAux {
    WordTerm terms[kWordTerms];
    double weight[2 << kWordMaxHalf];
    __align__(16) double occ[16];
    int first[kWordMaxHalf + 2];
};

// children of a node four (Q) characters deeper, for one tail: X[v] over the
// words |v| <= Q in heap order -> out[u] for the 2^Q strings u, whose first
// character is bit 0 of the index: out[u] = sum_v N(u, v) X[v]
template <int Q>
struct WordExpand {
    static __device__ __forceinline__ void run(const double (&X)[2 << Q], double* out, int stride) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            double Y[1 << Q];
#pragma unroll
            for (int d = 0; d < Q; ++d)
#pragma unroll
                for (int v = 0; v < (1 << d); ++v) {
                    const int h = (1 << d) + v;
                    Y[h] = X[h] + X[h + ((1 + b) << d)];
                }
            WordExpand<Q - 1>::run(Y, out + b * stride, 2 * stride);
        }
    }
};
template <>
struct WordExpand<0> {
    static __device__ __forceinline__ void run(const double (&X)[2], double* out, int) { out[0] = X[1]; }
};

// the transpose: in[u] over the 2^Q strings -> X[v] = sum_u N(u, v) in[u]
template <int Q>
struct WordContract {
    static __device__ __forceinline__ void run(double (&X)[2 << Q], const double* in, int stride) {
        double Y0[1 << Q], Y1[1 << Q];
        WordContract<Q - 1>::run(Y0, in, 2 * stride);
        WordContract<Q - 1>::run(Y1, in + stride, 2 * stride);
#pragma unroll
        for (int d = 0; d <= Q; ++d)
#pragma unroll
            for (int v = 0; v < (1 << d); ++v) {
                double s = 0.0;
                if (d < Q) s = Y0[(1 << d) + v] + Y1[(1 << d) + v];
                if (d > 0) {
                    const int tail = (1 << (d - 1)) + (v & ((1 << (d - 1)) - 1));
                    s += (v >> (d - 1)) ? Y1[tail] : Y0[tail];
                }
                X[(1 << d) + v] = s;
            }
    }
};
template <>
struct WordContract<0> {
    static __device__ __forceinline__ void run(double (&X)[2], const double* in, int) { X[1] = in[0]; }
};

// shared memory of a transform CTA, in doubles: a buffer for the words of up to
// cap characters or the 2^{r+1} coefficients of a tree level, and one for a level
__host__ __device__ constexpr int word_buf(int cap, int r) { return 2 << (cap > r ? cap : r); }
__host__ __device__ constexpr int word_smem(int cap, int r) {
    return (int)sizeof(double) * (word_buf(cap, r) + (2 << r));
}

// characters per tree round, from the root: 4, 4, ..., then the rest
__host__ __device__ constexpr int word_round(int rem) { return rem < 4 ? rem : 4; }

// threads of a transform CTA whose slices have r characters, and the most items
// (nodes times tails) of a round: k_words_q takes one a thread.  From r = 9 on
// that is 2^{r-3} or the 256 nodes after eight characters, whichever is more.
__host__ __device__ constexpr int word_threads(int r) { return r <= 11 ? 256 : 512; }
// CTAs an SM that the registers are kept to: three for short slices, which leave
// room for them and meet in batches (48 accelerated steps of 13/11 x 64 23.9 ms with
// two, 21.0 with three, 14/12 x 64 26.4 and 23.3); longer ones lose more to the
// spilled registers (22/11 62.0 us an iteration with one, 64.7 with three)
__host__ __device__ constexpr int word_ctas(int r) { return r <= 8 ? 3 : 1; }
__host__ __device__ constexpr int word_items(int k, int r) {
    int most = 0;
    for (int i = 0; i < r; i += word_round(r - i)) {
        const int rem = r - i, left = rem - word_round(rem), tails = (2 << (left < k ? left : k)) - 1;
        most = (tails << i) > most ? (tails << i) : most;
    }
    return most;
}
constexpr bool word_items_fit() {
    for (int k = 1; k <= 2 * kWordMaxHalf; ++k)
        for (int r = 1; r <= 12; ++r)
            if (word_items(k, r) > word_threads(r)) return false;
    return true;
}
static_assert(word_items_fit(), "a round of the q side has more items than its CTA threads");

// one round of the D side for one item: node u after i characters, tail at
// heap index h; Lp, Lc: longest word of a parent / child node.  In the root's
// round the words of length k are ln q itself (times s0).
template <int Q>
__device__ __forceinline__ void word_expand_item(double* wsm, int src, int dst, int u, int h, int i, int Lp, int Lc, int k, const double* __restrict__ lnq,
                                                 double s0, bool root, bool leaf, double* __restrict__ out,
                                                 int64_t leaf_stride, int first, int leaf0, int leaves) {
    const int l = word_len(h), val = h - (1 << l);
    const int p = src + (root ? 0 : (u << (Lp + 1)));
    double X[2 << Q], Y[1 << Q];
#pragma unroll
    for (int d = 0; d <= Q; ++d)
#pragma unroll
        for (int v = 0; v < (1 << d); ++v) {
            const int idx = (((1 << d) + v) << l) | val;
            double x = 0.0;
            if (l + d <= Lp) x = (root && l + d == k) ? s0 * __ldg(lnq + idx - (1 << k)) : wsm[p + idx];
            X[(1 << d) + v] = x;
        }
    WordExpand<Q>::run(X, Y, 1);
#pragma unroll
    for (int v = 0; v < (1 << Q); ++v) {
        const int node = u + (v << i);
        if (leaf) {
            const int at = first + node - leaf0;
            if (at >= 0 && at < leaves) out[(int64_t)at * leaf_stride] = Y[v];
        } else {
            wsm[dst + (node << (Lc + 1)) + h] = Y[v];
        }
    }
}

// D side: ln q -> F_w over the strings of the other half
template <int T, int CTAS>
__global__ void __launch_bounds__(T, CTAS) k_words_d(const WordPlan* __restrict__ plan, const double* __restrict__ lnq,
                                               const DevState* st) {
    if (st && (st->done || st->error)) return;
    extern __shared__ __align__(16) double wsm[];
    const int side = (int)blockIdx.x >= plan->side[1].cta0 ? 1 : 0;
    const WordSide S = plan->side[side];
    const int k = plan->k, a = S.words_log, r = S.r, t = S.t, tid = threadIdx.x;
    const int id = (int)blockIdx.x - S.cta0;
    const int w = id >> t, beta = id & ((1 << t) - 1);
    const int first = beta << r;
    if (first + (1 << r) <= S.leaf0 || first >= S.leaf0 + S.leaves) return;  // no held leaf in this slice
    double* out = S.out + (int64_t)w * S.word_stride;
    if (word_whole(S, k)) {
        const double* q = lnq + ((side ? (int)reverse_bits((uint32_t)w, a) : w) << (k - a));
        for (int i = tid; i < (1 << r); i += T) {
            const int at = first + i - S.leaf0;
            if (at >= 0 && at < S.leaves)
                out[(int64_t)at * S.leaf_stride] = __ldg(q + reverse_bits((uint32_t)(first + i), k - a));
        }
        return;
    }
    const int cap = word_cap(S, k);  // longest word that can still occur
    double* c = wsm;
    double* other = wsm + word_buf(cap, r);
    const int nk = 1 << k;  // heap indices of the words shorter than k: [1, nk)
    // the last characters that are fixed in this CTA (the first of them highest)
    const int fixed = S.last0 + t;
    const int tailc = (int)reverse_bits((uint32_t)beta, t) << S.last0;
    __shared__ WordAux aux;
    for (int e = tid; e < kWordTerms; e += T) aux.terms[e] = S.terms[w * kWordTerms + e];
    if (tid < kWordMaxHalf + 2) aux.first[tid] = S.first[w * (kWordMaxHalf + 2) + tid];
    if (tid >= 32 && tid < 48) aux.occ[tid - 32] = tid > 32 ? word_occ(tailc, fixed, tid - 32) : 0.0;
    // ln q to the second buffer where it fits: from global memory each of the
    // dozen or so term steps below would wait for L2
    const bool staged = (2 << r) >= nk;
    if (staged) {
        for (int y = 2 * tid; y < nk; y += 8 * T) {
            double2 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (y + 2 * u * T < nk) v[u] = __ldg(reinterpret_cast<const double2*>(lnq + y + 2 * u * T));
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (y + 2 * u * T < nk) *reinterpret_cast<double2*>(other + y + 2 * u * T) = v[u];
        }
    }
    // c_w: zero below k - a characters ...
    for (int h = tid; h < (1 << (k - a)); h += T) c[h] = 0.0;
    __syncthreads();
    const double s0 = aux.terms[0].weight;  // |v| = 0
    // ... else the terms of w, four tails z a thread at a time
    for (int j = max(1, k - cap); j <= a; ++j) {
        const int d = k - j, n = 1 << d;
        const int e0 = aux.first[j], e1 = aux.first[j + 1];
        for (int z = tid; z < n; z += 4 * T) {
            double x[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
            for (int e = e0; e < e1; ++e) {
                const double wt = aux.terms[e].weight;
                const int at = (aux.terms[e].v << d) + z;
                if (staged) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (z + i * T < n) x[i] = fma(wt, other[at + i * T], x[i]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (z + i * T < n) x[i] = fma(wt, __ldg(lnq + at + i * T), x[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (z + i * T < n) c[n + z + i * T] = x[i];
        }
    }
    __syncthreads();
    // (buffers as offsets: pointers that change roles would be generic ones)
    const int second = word_buf(cap, r);
    int src = 0, dst = second;
    if (fixed > 0) {
        // consume the fixed last characters: c[z] <- sum_u N(p, u) c[z u] over
        // their subsequences u
        const int capr = min(k - 1, r);
        for (int h = 1 + tid; h < (2 << capr); h += T) {
            double x = c[h];
            for (int d = 1; d <= fixed; ++d) {
                const int g = h << d;  // the 2^d words z u, two at a time
                const double* p = g < (2 << cap) ? c + g : lnq + (g - nk);
                if (g >= (2 << cap) && (g < nk || g >= 2 * nk)) break;  // none that long
                const double f = g < (2 << cap) ? 1.0 : s0;
                for (int v = 0; v < (1 << d); v += 2) {
                    const double2 o = *reinterpret_cast<const double2*>(aux.occ + (1 << d) + v);
                    const double2 q = *reinterpret_cast<const double2*>(p + v);
                    x = fma(o.x * f, q.x, x);
                    x = fma(o.y * f, q.y, x);
                }
            }
            other[h] = x;
        }
        __syncthreads();
        src = second;
        dst = 0;
    }
    // the tree over the r free characters
    for (int i = 0; i < r;) {
        const int rem = r - i, q = word_round(rem);
        const int Lp = min(k, rem), Lc = min(k, rem - q);
        const bool root = i == 0, leaf = rem == q;
        const int tails = 2 << Lc;  // heap indices of a child's words, 0 unused
        for (int e = tid; e < (tails << i); e += T) {
            const int u = e >> (Lc + 1), h = e & (tails - 1);
            if (h == 0) continue;
#define BDC_ITEM_(Q_)                                                                                               \
    word_expand_item<Q_>(wsm, src, dst, u, h, i, Lp, Lc, k, lnq, s0, root, leaf, out, S.leaf_stride, first, S.leaf0, \
                         S.leaves)
            switch (q) {
                case 4: BDC_ITEM_(4); break;
                case 3: BDC_ITEM_(3); break;
                case 2: BDC_ITEM_(2); break;
                default: BDC_ITEM_(1); break;
            }
#undef BDC_ITEM_
        }
        __syncthreads();
        const int x = src;
        src = dst;
        dst = x;
        i += q;
    }
}

// one round of the q side for the item (u, h): the 2^Q children's values at
// the tail -> X[v], |v| <= Q (read by every thread before any of them writes)
template <int Q>
__device__ __forceinline__ void word_contract_load(double (&X)[32], const double* wsm, int src, int u, int h, int i,
                                                   int Lc, bool leaf) {
    double in[1 << Q];
    // (a leaf node is its one value)
#pragma unroll
    for (int v = 0; v < (1 << Q); ++v)
        in[v] = leaf ? wsm[src + u + (v << i)] : wsm[src + ((u + (v << i)) << (Lc + 1)) + h];
    double Z[2 << Q];
    WordContract<Q>::run(Z, in, 1);
#pragma unroll
    for (int h2 = 1; h2 < (2 << Q); ++h2) X[h2] = Z[h2];
}

// X[v] added to the parent's words v z, one length of v at a time (for a
// fixed length the words v z of different tails are distinct); a word whose
// tail is as long as a child's longest, or with |v| = 0, is written first here
template <int Q>
__device__ __forceinline__ void word_contract_add(const double (&X)[32], double* wsm, int dst, int u, int h, int Lp, int Lc, bool live) {
    const int l = word_len(h), val = h - (1 << l);
    const int p = dst + (u << (Lp + 1));
#pragma unroll
    for (int d = 0; d <= Q; ++d) {
        if (live && l + d <= Lp) {
#pragma unroll
            for (int v = 0; v < (1 << d); ++v) {
                const int idx = (((1 << d) + v) << l) | val;
                if (d == 0 || l == Lc) wsm[p + idx] = X[(1 << d) + v];
                else wsm[p + idx] += X[(1 << d) + v];
            }
        }
        __syncthreads();
    }
}

// q side: the products' columns U_w (summed over their split slices) -> this
// word's and slice's share of acc[y] = sum_x |O| e(x) N(x, y), a vector of 2^k
// (the second side's with y reversed).  One item of a round a thread
// (word_items).
template <int T, int CTAS>
__global__ void __launch_bounds__(T, CTAS) k_words_q(const WordPlan* __restrict__ plan, double* __restrict__ parts,
                                               const DevState* st) {
    if (st && (st->done || st->error)) return;
    extern __shared__ __align__(16) double wsm[];
    const int side = (int)blockIdx.x >= plan->side[1].cta0 ? 1 : 0;
    const WordSide S = plan->side[side];
    const int k = plan->k, a = S.words_log, r = S.r, t = S.t, tid = threadIdx.x;
    const int id = (int)blockIdx.x - S.cta0;
    const int w = id >> t, beta = id & ((1 << t) - 1);
    const int first = beta << r;
    const int nk = 1 << k;
    if (word_whole(S, k)) {
        double* q = parts + ((int64_t)S.part0 << k) + ((side ? (int)reverse_bits((uint32_t)w, a) : w) << (k - a));
        for (int i = tid; i < (1 << r); i += T) {
            const int at = first + i - S.leaf0, n = at >= 0 && at < S.leaves ? (int)S.ns[at >> 4] : 0;
            const double* p = S.in + (int64_t)w * S.leaves + at;
            double x = 0.0;
#pragma unroll 4
            for (int s = 0; s < n; ++s) x += __ldg(p + s * S.slice_stride);
            const int z = (int)reverse_bits((uint32_t)(first + i), k - a);
            q[z] = x;
            if (S.last0) q[z + 1] = 0.0;  // (the strings end in 0)
        }
        return;
    }
    double* part = parts + ((int64_t)(S.part0 + id) << k);
    if (first + (1 << r) <= S.leaf0 || first >= S.leaf0 + S.leaves) return;
    const int least = word_least(S, k), cap = word_cap(S, k);
    // the tree, deepest characters first; the rounds alternate between the
    // buffers so that the root ends in the second
    const int rounds = (r + 3) / 4;
    const int second = word_buf(cap, r);
    int dst = (rounds & 1) ? second : 0, src = (rounds & 1) ? 0 : second;
    // the leaves first: the split slices added up, 4 leaves x 4 slices of a
    // thread in flight (a slice at a time, each added slice waited for L2)
    for (int i = tid; i < (1 << r); i += 4 * T) {
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        int n[4], most = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int at = first + i + q * T - S.leaf0;
            n[q] = (i + q * T < (1 << r) && at >= 0 && at < S.leaves) ? (int)S.ns[at >> 4] : 0;
            most = max(most, n[q]);
        }
        const double* p = S.in + (int64_t)w * S.leaves + (first + i - S.leaf0);
        for (int s = 0; s < most; s += 4) {
            double v[4][4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    v[e][q] = s + e < n[q] ? __ldg(p + (s + e) * S.slice_stride + q * T) : 0.0;
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int q = 0; q < 4; ++q) x[q] += v[e][q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (i + q * T < (1 << r)) wsm[src + i + q * T] = x[q];
    }
    __syncthreads();
    for (int g = rounds - 1; g >= 0; --g) {
        const int i = 4 * g, rem = r - i, q = word_round(rem);
        const int Lp = min(k, rem), Lc = min(k, rem - q);
        const bool leaf = rem == q;
        const int tails = 2 << Lc;
        // an item per thread: node u, tail h in [1, tails)
        const int u = tid / (tails - 1), h = 1 + tid % (tails - 1);
        const bool live = u < (1 << i);
        double X[32];
#define BDC_ROUND_(Q_)                                                                  \
    if (live) word_contract_load<Q_>(X, wsm, src, u, h, i, Lc, leaf);         \
    word_contract_add<Q_>(X, wsm, dst, u, h, Lp, Lc, live);
        switch (q) {
            case 4: BDC_ROUND_(4) break;
            case 3: BDC_ROUND_(3) break;
            case 2: BDC_ROUND_(2) break;
            default: BDC_ROUND_(1) break;
        }
#undef BDC_ROUND_
        const int x = src;
        src = dst;
        dst = x;
    }
    // the root is in the second buffer
    const double* root = wsm + second;
    double* c = wsm;
    // the root's words up to length min(k, r).  The fixed last characters
    // p: a word z u takes N(p, u) t[z], up to `fixed` characters u
    const int fixed = S.last0 + t, tailc = (int)reverse_bits((uint32_t)beta, t) << S.last0;
    const int top = 2 << min(k, r);  // end of the root's heap
    __shared__ WordAux aux;
    if (tid >= 32 && tid < 48) aux.occ[tid - 32] = tid > 32 ? word_occ(tailc, fixed, tid - 32) : 0.0;
    for (int h = tid; h < (2 << a); h += T) aux.weight[h] = __ldg(S.weight + ((size_t)w << (a + 1)) + h);
    __syncthreads();
    const double* wt = aux.weight;
    // two adjacent words at even heap index h
    auto after = [&](int h) {
        double2 x = make_double2(0.0, 0.0);
        if (h < top) x = *reinterpret_cast<const double2*>(root + h);
        for (int d = 1; d <= fixed; ++d) {
            const int g = h >> d;
            if (g > 0 && g < top) {
                const double2 o = *reinterpret_cast<const double2*>(aux.occ + (1 << d) + (h & ((1 << d) - 1)));
                const double t = root[g];
                x.x = fma(o.x, t, x.x);
                x.y = fma(o.y, t, x.y);
            }
        }
        return x;
    };
    // (k - a >= 1, so the shortest words read begin at an even index)
    for (int h = (1 << (k - a)) + 2 * tid; h < (2 << cap); h += 2 * T) *reinterpret_cast<double2*>(c + h) = after(h);
    __syncthreads();
    // acc[v z] = sum over the splits of y into |v| <= a characters and the
    // rest; two adjacent y share v and their z are adjacent
    for (int y = 2 * tid; y < nk; y += 2 * T) {
        // (y begins with the `least` characters that come from w at least)
        if (least > 0 && wt[(1 << least) + (y >> (k - least))] == 0.0) continue;
        double2 x = make_double2(0.0, 0.0);
        if (least == 0) {
            const double2 z0 = after(nk + y);
            x = make_double2(wt[1] * z0.x, wt[1] * z0.y);
        }
#pragma unroll
        for (int j = 1; j <= kWordMaxHalf; ++j) {
            if (j > a) break;
            if (j < least) continue;
            const int d = k - j;
            const double w = wt[(1 << j) + (y >> d)];
            const double2 z = *reinterpret_cast<const double2*>(c + (1 << d) + (y & ((1 << d) - 1)));
            x.x = fma(w, z.x, x.x);
            x.y = fma(w, z.y, x.y);
        }
        *reinterpret_cast<double2*>(part + y) = x;
    }
}

// ------------------------------------------------------------------ q fold
// q(rep r) = sum_{y in O(r)} acc[y] / (|O(r)| C Z), ln q with the reference's
// 0 for q == 0 (backend/BAA.cu:573-580), over every y and in the rep slots.
// acc is the sum of the parts; the second side's are reversed, which the sum
// over an orbit does not see.  A CTA takes the words whose middle bits (all
// but 2 leading and 2 trailing ones) are the images of one middle m: up to 64
// words, closed under the group, in runs of four adjacent ones per part.
constexpr int kFoldThreads = 256;
__host__ __device__ constexpr int fold_edge(int k) { return k >= 4 ? 2 : (k >= 2 ? 1 : 0); }

__global__ void __launch_bounds__(kFoldThreads)
k_words_fold(const double* __restrict__ parts, int nparts, int k, double inv_c, const int* __restrict__ mids,
             double* __restrict__ lnq_full, double* __restrict__ lnq, const DevState* st) {
    if (st && (st->done || st->error)) return;
    __shared__ double sum[4][64];
    const int e = fold_edge(k), mb = k - 2 * e, m = mids[blockIdx.x];
    const int el = threadIdx.x & 63, grp = threadIdx.x >> 6;
    const int slot = el >> 4, hi = (el >> 2) & 3, lo = el & 3;
    // slot s holds the image of m under group element s: 1 reverse, 2 complement, 3 both
    uint32_t mm = (uint32_t)m;
    if (slot & 1) mm = reverse_bits(mm, mb);
    if (slot & 2) mm = complement_bits(mm, mb);
    const bool live = hi < (1 << e) && lo < (1 << e);
    const uint32_t y = live ? ((uint32_t)hi << (k - e)) | (mm << e) | (uint32_t)lo : 0u;
    double a = 0.0;
    {
        const double* p = parts + y;
        int i = grp;
        for (; i + 28 < nparts; i += 32) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = p[(size_t)(i + 4 * u) << k];
#pragma unroll
            for (int u = 0; u < 8; ++u) a += v[u];
        }
        for (; i < nparts; i += 4) a += p[(size_t)i << k];
    }
    sum[grp][el] = a;
    __syncthreads();
    if (grp != 0) return;
    sum[0][el] = (sum[0][el] + sum[1][el]) + (sum[2][el] + sum[3][el]);
    __syncwarp();
    asm volatile("bar.sync 1, 64;" ::: "memory");
    if (!live) return;
    // the orbit of y in the order of its representative: r, rev, comp, rev comp
    uint32_t img[4];
    img[0] = y;
    img[1] = reverse_bits(y, k);
    img[2] = complement_bits(y, k);
    img[3] = reverse_bits(img[2], k);
    int g0 = 0;
#pragma unroll
    for (int g = 1; g < 4; ++g)
        if (img[g] < img[g0]) g0 = g;
    auto value = [&](int g) {  // acc at the image of y under g
        const uint32_t h = img[g] >> (k - e), l = img[g] & ((1u << e) - 1u);
        return sum[0][((slot ^ g) << 4) | (h << 2) | l];
    };
    uint32_t seen[4];
    double acc = 0.0;
    int nm = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t z = img[g0 ^ j];
        bool dup = false;
        for (int q = 0; q < nm; ++q) dup |= seen[q] == z;
        if (dup) continue;
        seen[nm++] = z;
        acc += value(g0 ^ j);
    }
    const double q = acc * inv_c * exp(-st->log_z) / (double)nm;
    const double lq = (q != 0.0) ? log(q) : 0.0;
    lnq_full[y] = lq;
    if (img[g0] == y) lnq[y] = lq;  // representatives are < 2^{k-1}
}

// the raw sums acc[y] over the parts (a shard's share of q)
__global__ void k_words_acc(const double* __restrict__ parts, int parts_l, int nparts, int k,
                            double* __restrict__ acc) {
    const int y = blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= (1 << k)) return;
    const uint32_t ry = reverse_bits((uint32_t)y, k);
    double a = 0.0;
    for (int i = 0; i < parts_l; ++i) a += parts[((size_t)i << k) + y];
    for (int i = parts_l; i < nparts; ++i) a += parts[((size_t)i << k) + ry];
    acc[y] = a;
}

}  // namespace bdc
