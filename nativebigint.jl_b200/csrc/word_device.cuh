// word_device.cuh — device side of the word products (word.h): constants, the
// radix-odd steps, block transforms, leaf products, coefficients and carried
// limb sums, shared by the kernels of word_kernels.cu and powmod_chain.cu.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "word.cuh"
#include "word.h"

namespace nbg {

using wd::Tw;

struct WConst {
    uint32_t p[WPR_MAX], pinv[WPR_MAX];
    uint32_t half[WPR_MAX];          // the multiple of p nearest to 2^31
    Tw r3[WPR_MAX];                  // e(1/3)
    Tw r5[WPR_MAX][4];               // -1/4, (c1-c2)/2, f1, f2 of e(1/5) (see dft5)
    uint32_t c7[WPR_MAX][3], f7[WPR_MAX][3];  // cosine and sine halves of e(j/7) in 2^32 form
    uint32_t wt[WPR_MAX][WPR_MAX];       // words of W_i = p_0 ... p_(i-1) (i words)
    uint32_t gar[WPR_MAX][WPR_MAX];      // mixed radix: gar[i][j] = -W_j / W_i mod p_i in 2^32 form (j < i)
};
static __constant__ WConst c_w[WSETS];
// Fills the constants (host); every file that includes this copies them to its c_w.
void word_fill_const(WConst h[WSETS]);

// ---------------------------------------------------------------------------
// radix-odd steps: in and out in [0, 2p) unless said otherwise

// y_j = sum x_i e(ij/3): with w + w^2 = -1 one product suffices
template <int SET>
__device__ __forceinline__ void dft3(uint32_t* x, int st, int i, uint32_t p) {
    const uint32_t p2 = 2 * p;
    uint32_t &a = x[0], &b = x[st], &c = x[2 * st];
    const uint32_t t = wd::mulw(b - c + p2, c_w[SET].r3[i], p);
    const uint32_t y0 = wd::sub_if(wd::sub_if(a + b, p2) + c, p2);
    const uint32_t y1 = wd::sub_if(wd::sub_if(a - c + p2, p2) + t, p2);
    const uint32_t u = wd::sub_if(a - b + p2, p2);
    const uint32_t y2 = wd::sub_if(u - t + p2, p2);
    a = y0;
    b = y1;
    c = y2;
}
// cosine halves c1, c2 = -1/4 +- d: two products for the even part, four for the odd
template <int SET>
__device__ __forceinline__ void dft5(uint32_t* x, int st, int i, uint32_t p) {
    const uint32_t p2 = 2 * p;
    const Tw q = c_w[SET].r5[i][0], d = c_w[SET].r5[i][1], f1 = c_w[SET].r5[i][2], f2 = c_w[SET].r5[i][3];
    const uint32_t x0 = x[0], x1 = x[st], x2 = x[2 * st], x3 = x[3 * st], x4 = x[4 * st];
    const uint32_t s1 = wd::sub_if(x1 + x4, p2), s2 = wd::sub_if(x2 + x3, p2);
    const uint32_t d1 = x1 - x4 + p2, d2 = x2 - x3 + p2;
    const uint32_t s = wd::sub_if(s1 + s2, p2);
    const uint32_t b0 = wd::sub_if(x0 + wd::mulw(s, q, p), p2);
    const uint32_t e = wd::mulw(s1 - s2 + p2, d, p);
    const uint32_t C1 = wd::sub_if(b0 + e, p2), C2 = wd::sub_if(b0 - e + p2, p2);
    const uint32_t S1 = wd::sub_if(wd::mulw(d1, f1, p) + wd::mulw(d2, f2, p), p2);
    const uint32_t S2 = wd::sub_if(wd::mulw(d1, f2, p) - wd::mulw(d2, f1, p) + p2, p2);
    x[0] = wd::sub_if(x0 + s, p2);
    x[st] = wd::sub_if(C1 + S1, p2);
    x[4 * st] = wd::sub_if(C1 - S1 + p2, p2);
    x[2 * st] = wd::sub_if(C2 + S2, p2);
    x[3 * st] = wd::sub_if(C2 - S2 + p2, p2);
}
// even and odd parts as sums of three wide products and one reduction each
template <int SET>
__device__ __forceinline__ void dft7(uint32_t* x, int st, int i, uint32_t p) {
    const uint32_t p2 = 2 * p, pinv = c_w[SET].pinv[i];
    const uint32_t x0 = x[0];
    uint32_t s[3], d[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        s[k] = wd::sub_if(x[(k + 1) * st] + x[(6 - k) * st], p2);
        d[k] = wd::sub_if(x[(k + 1) * st] - x[(6 - k) * st] + p2, p2);
    }
    x[0] = wd::sub_if(wd::sub_if(wd::sub_if(x0 + s[0], p2) + s[1], p2) + s[2], p2);
#pragma unroll
    for (int j = 1; j <= 3; j++) {
        uint64_t ce = 0, so = 0;
#pragma unroll
        for (int k = 1; k <= 3; k++) {
            const int t = j * k % 7, a = t <= 3 ? t : 7 - t;  // cos(t) = cos(7 - t), sin(t) = -sin(7 - t)
            ce += wd::mulx(s[k - 1], c_w[SET].c7[i][a - 1]);
            so += wd::mulx(t <= 3 ? d[k - 1] : p2 - d[k - 1], c_w[SET].f7[i][a - 1]);
        }
        // each sum < 3 * 2p * p, reduced below 1.5p + p
        const uint32_t C = wd::sub_if(x0 + wd::sub_if(wd::redc(ce, p, pinv), p2), p2);
        const uint32_t S = wd::sub_if(wd::redc(so, p, pinv), p2);
        x[j * st] = wd::sub_if(C + S, p2);
        x[(7 - j) * st] = wd::sub_if(C - S + p2, p2);
    }
}

template <int ODD, int LJ, int SET = 0>
__device__ __forceinline__ void dft_odd(uint32_t* x, int i, uint32_t p) {
#pragma unroll
    for (int r = 0; r < (1 << LJ); r++) {
        if (ODD == 3) dft3<SET>(x + r, 1 << LJ, i, p);
        if (ODD == 5) dft5<SET>(x + r, 1 << LJ, i, p);
        if (ODD == 7) dft7<SET>(x + r, 1 << LJ, i, p);
    }
}

// ---------------------------------------------------------------------------
// packing

// A limb times 2^-32 modulo p, in (0, 4p) (RED: [0, 2p)): one Montgomery
// reduction, whose factor the unpack's scale constants take back.  The upper
// word goes below 3p first: with p > 2^32/6 (set 0) one subtraction does it, with
// p > 2^32/11 two (below 2^31 + p/2 after the first).  Two products with the constants
// 2^32 and 1 took 8 multiply slots instead of 3, a third of
// k_wcol_fwd's (10,000 mixed products: that pass 3.10 -> 2.89 ms).
template <bool RED, int SET = 0>
__device__ __forceinline__ uint32_t wpack(uint64_t v, int pi, uint32_t p) {
    static_assert(word_pack_ok(SET), "primes too small for the upper word's reduction");
    uint32_t hi = (uint32_t)(v >> 32);
    if (SET) hi = wd::sub_if(hi, c_w[SET].half[pi]);
    const uint32_t y = wd::redc((uint64_t)wd::sub_if(hi, 3 * p) << 32 | (uint32_t)v, p, c_w[SET].pinv[pi]);
    return RED ? wd::sub_if(y, 2 * p) : y;
}

// ---------------------------------------------------------------------------
// blocks: M = 2^LM consecutive values on M/16 threads, 16 values per thread.
// A round runs J levels on sub-blocks of 2^LL values; a thread takes 2^(4-J)
// groups of 2^J values at stride S = 2^(LL-J).  The last round always runs two
// levels on 16 consecutive values, leaving the thread four whole leaves.
// Shared memory is padded by four words in 16 and 16 in 256: the last round's
// 16 words per thread move as four 16-byte accesses, and every stride (16 at
// least before that round) is free of bank conflicts or two-way.  A group's
// values lie at compile-time offsets from its first one: its index has zeros
// in the bits that e * S occupies, so the padding of the sum is the sum of the
// paddings.

__host__ __device__ constexpr int wpad(int i) { return i + ((i >> 4) << 2) + ((i >> 8) << 4); }
__host__ __device__ constexpr int wwords(int m) { return m + m / 4 + m / 16; }  // padded words of m >= 64 values

// index of the first value of thread t's q-th group
template <int LM, int LL, int J>
__device__ __forceinline__ int wpos(int t, int q) {
    constexpr int S = 1 << (LL - J), T = 1 << (LM - 4);
    static_assert(S >= 16, "strides below the padding period");
    const int gi = t + q * T;
    return ((gi >> (LL - J)) << LL) + (gi & (S - 1));
}
template <int LM, int LL, int J, int NV>
__device__ __forceinline__ void wround_fwd(uint32_t* x, int t, const Tw* __restrict__ tab, uint32_t h0, uint32_t p) {
    constexpr int T = 1 << (LM - 4);
#pragma unroll
    for (int q = 0; q < (1 << (4 - J)); q++)
        wd::tree_fwd<J, 1, NV, 16>(x + (q << J), tab, (h0 << (LM - LL)) + (uint32_t)((t + q * T) >> (LL - J)), p);
}
template <int LM, int LL, int J>
__device__ __forceinline__ void wround_rev(uint32_t* x, int t, const Tw* __restrict__ tab, uint32_t h0, uint32_t p) {
    constexpr int T = 1 << (LM - 4);
#pragma unroll
    for (int q = 0; q < (1 << (4 - J)); q++)
        wd::tree_rev<J, 1>(x + (q << J), tab, (h0 << (LM - LL)) + (uint32_t)((t + q * T) >> (LL - J)), p);
}
template <int LM, int LL, int J>
__device__ __forceinline__ void wput(uint32_t* s, const uint32_t* x, int t) {
#pragma unroll
    for (int q = 0; q < (1 << (4 - J)); q++) {
        uint32_t* d = s + wpad(wpos<LM, LL, J>(t, q));
#pragma unroll
        for (int e = 0; e < (1 << J); e++) d[wpad(e << (LL - J))] = x[(q << J) + e];
    }
}
template <int LM, int LL, int J>
__device__ __forceinline__ void wget(const uint32_t* s, uint32_t* x, int t) {
#pragma unroll
    for (int q = 0; q < (1 << (4 - J)); q++) {
        const uint32_t* d = s + wpad(wpos<LM, LL, J>(t, q));
#pragma unroll
        for (int e = 0; e < (1 << J); e++) x[(q << J) + e] = d[wpad(e << (LL - J))];
    }
}
// the 16 consecutive values 16t .. 16t+15
__device__ __forceinline__ uint4* wrow(uint32_t* s, int t) { return reinterpret_cast<uint4*>(s + wpad(16 * t)); }
__device__ __forceinline__ void wput16(uint32_t* s, const uint32_t* x, int t) {
#pragma unroll
    for (int k = 0; k < 4; k++) wrow(s, t)[k] = make_uint4(x[4 * k], x[4 * k + 1], x[4 * k + 2], x[4 * k + 3]);
}
__device__ __forceinline__ void wget16(uint32_t* s, uint32_t* x, int t) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint4 v = wrow(s, t)[k];
        x[4 * k] = v.x;
        x[4 * k + 1] = v.y;
        x[4 * k + 2] = v.z;
        x[4 * k + 3] = v.w;
    }
}

// level splits of a block: J1, J2 (0: none), then the two leaf levels
template <int LM>
struct WSplit;
template <>
struct WSplit<12> { static constexpr int J1 = 4, J2 = 4; };
template <>
struct WSplit<11> { static constexpr int J1 = 4, J2 = 3; };
template <>
struct WSplit<10> { static constexpr int J1 = 3, J2 = 3; };
template <>
struct WSplit<9> { static constexpr int J1 = 3, J2 = 2; };
template <>
struct WSplit<8> { static constexpr int J1 = 4, J2 = 0; };
template <>
struct WSplit<7> { static constexpr int J1 = 3, J2 = 0; };
template <>
struct WSplit<6> { static constexpr int J1 = 2, J2 = 0; };

// NV blocks (the operands' values at x[16 v ..], their shared memory SM words
// apart) down to their leaves, from the first round's values: x[16 v + k] =
// value 16t + k in [0, 4p).  The operands of a product go down together: they
// share every constant load and barrier and double the independent butterflies.
template <int LM, int NV, int SM>
__device__ __forceinline__ void wblock_down(uint32_t* x, uint32_t* s, int t, const Tw* __restrict__ tab, uint32_t h0,
                                            uint32_t p, bool live) {
    constexpr int J1 = WSplit<LM>::J1, J2 = WSplit<LM>::J2;
    if (live) {
        wround_fwd<LM, LM, J1, NV>(x, t, tab, h0, p);
#pragma unroll
        for (int v = 0; v < NV; v++) wput<LM, LM, J1>(s + v * SM, x + 16 * v, t);
    }
    __syncthreads();
    if constexpr (J2 > 0) {
        if (live) {
#pragma unroll
            for (int v = 0; v < NV; v++) wget<LM, LM - J1, J2>(s + v * SM, x + 16 * v, t);
            wround_fwd<LM, LM - J1, J2, NV>(x, t, tab, h0, p);
#pragma unroll
            for (int v = 0; v < NV; v++) wput<LM, LM - J1, J2>(s + v * SM, x + 16 * v, t);
        }
        __syncthreads();
    }
    if (live) {
#pragma unroll
        for (int v = 0; v < NV; v++) wget16(s + v * SM, x + 16 * v, t);
        const uint32_t idx = (h0 << (LM - 4)) + (uint32_t)t;
#pragma unroll
        for (int q = 0; q < 4; q++) wd::tree_fwd<2, 4, NV, 16>(x + q, tab, idx, p);
    }
}

// The way back: a[0..16) = leaf values 16t .. 16t+15 in [0, 2p), out: the
// first round's values.  Safe right after wblock_down on the same `s`: each
// thread first writes the 16 words that only it read last.
template <int LM>
__device__ __forceinline__ void wblock_up(uint32_t* a, uint32_t* s, int t, const Tw* __restrict__ ti, uint32_t h0,
                                          uint32_t p, bool live) {
    constexpr int J1 = WSplit<LM>::J1, J2 = WSplit<LM>::J2;
    const uint32_t p2 = 2 * p;
    if (live) {
        const uint32_t idx = (h0 << (LM - 4)) + (uint32_t)t;
        Tw w1[1], w2[2];
        wd::load_tw<0>(ti, idx, w1);
        wd::load_tw<1>(ti, idx, w2);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            wd::bf_rev(a[e], a[e + 4], w2[0], p, p2);
            wd::bf_rev(a[e + 8], a[e + 12], w2[1], p, p2);
        }
#pragma unroll
        for (int e = 0; e < 8; e++) wd::bf_rev(a[e], a[e + 8], w1[0], p, p2);
        wput16(s, a, t);
    }
    __syncthreads();
    if constexpr (J2 > 0) {
        if (live) {
            wget<LM, LM - J1, J2>(s, a, t);
            wround_rev<LM, LM - J1, J2>(a, t, ti, h0, p);
            wput<LM, LM - J1, J2>(s, a, t);
        }
        __syncthreads();
    }
    if (live) {
        wget<LM, LM, J1>(s, a, t);
        wround_rev<LM, LM, J1>(a, t, ti, h0, p);
    }
}

// a * b mod X^4 - rho (NEG: X^4 + rho), a in [0, p), b in [0, 2p); the result
// carries a factor 2^-32 and lies in [0, 2p).  rho b_j first, so a coefficient is
// four products below 2p^2, together below 2^63, and one reduction to below 3p.
// Reducing the three upper sums first, then times rho, took three reductions more
// and 3% longer (k_wblock of 100 squares of 65536 limbs 0.324 ms against 0.316).
template <bool NEG>
__device__ __forceinline__ void wleaf(uint32_t* a, const uint32_t* b, wd::Tw rho, uint32_t p, uint32_t pinv) {
    uint32_t w[4];
#pragma unroll
    for (int k = 1; k < 4; k++) {
        w[k] = wd::mulw(b[k], rho, p);
        if (NEG) w[k] = 2 * p - w[k];
    }
    uint32_t c[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        uint64_t s = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) s += wd::mulx(a[i], i <= k ? b[k - i] : w[k + 4 - i]);
        c[k] = wd::sub_if(wd::redc(s, p, pinv), 2 * p);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) a[k] = c[k];
}

// The 16 consecutive leaf values a *= b (or a *= a), all in [0, 4p) before, [0, 2p) after.
template <int LM>
__device__ __forceinline__ void wpoint(uint32_t* a, uint32_t* b, bool sqr, int t, const Tw* __restrict__ tf, uint32_t h0,
                                       uint32_t p, uint32_t pinv) {
    const uint32_t p2 = 2 * p;
    Tw w2[2];
    wd::load_tw<1>(tf, (h0 << (LM - 4)) + (uint32_t)t, w2);
#pragma unroll
    for (int k = 0; k < 16; k++) {
        a[k] = wd::sub_if(wd::sub_if(a[k], p2), p);
        b[k] = sqr ? a[k] : wd::sub_if(b[k], p2);
    }
    wleaf<false>(a, b, w2[0], p, pinv);
    wleaf<true>(a + 4, b + 4, w2[0], p, pinv);
    wleaf<false>(a + 8, b + 8, w2[1], p, pinv);
    wleaf<true>(a + 12, b + 12, w2[1], p, pinv);
}

// ---------------------------------------------------------------------------
// unpack: coefficients and carried limbs, tiles of UNPACK_TL limbs

// The coefficient (below 2^160) whose residues (representatives below 2p,
// scaled) are r: mixed-radix digits y_i, each one sum of wide products and one
// reduction, then sum y_i W_i by columns of 32 bits.
constexpr int WCOEF = 5;  // 32-bit words of a coefficient
template <int SET>
__device__ __forceinline__ void wcoef(const uint32_t* r, const uint32_t* sc, uint32_t* v) {
    constexpr int NP = word_np(SET);
    uint32_t y[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const uint32_t p = c_w[SET].p[i];
        uint64_t s = wd::mulx(r[i], sc[i]);  // < 2p^2; the others < p_j p, p_j < 2.3p
#pragma unroll
        for (int j = 0; j < i; j++) s += wd::mulx(y[j], c_w[SET].gar[i][j]);
        // below 1.5p, 1.9p, then 3p: one or two subtractions
        y[i] = wd::sub_if(wd::redc(s, p, c_w[SET].pinv[i]), p);
        if (i > 1) y[i] = wd::sub_if(y[i], p);
    }
    uint64_t s = y[0];
#pragma unroll
    for (int k = 0; k < WCOEF; k++) {
        // at most four full products (below 2^62 each) per column: the sixth
        // digit is below 2^8, as the coefficient is below 2^153
        uint64_t col = k + 1 < NP ? wd::mulx(y[k + 1], c_w[SET].wt[k + 1][k]) : 0;
#pragma unroll
        for (int i = k + 2; i < NP; i++) col += wd::mulx(y[i], c_w[SET].wt[i][k]);
        s += col;  // s < 2^33 before
        v[k] = (uint32_t)s;
        s >>= 32;
    }
}

__device__ __forceinline__ uint32_t gp_join(uint32_t lower, uint32_t upper) {
    // bit 0 generate, bit 1 propagate; lower limbs, then upper
    return ((upper & 1u) | ((upper >> 1) & lower & 1u)) | (upper & lower & 2u);
}

// Carry-lookahead over a warp: the state of the parts up to this lane's.
__device__ __forceinline__ uint32_t warp_scan(uint32_t agg) {
    const int lane = (int)threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, agg, off);
        if (lane >= off) agg = gp_join(o, agg);
    }
    return agg;
}
// The state of the parts below this lane's, from that up to it.
__device__ __forceinline__ uint32_t warp_below(uint32_t incl) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, 1);
    return ((int)threadIdx.x & 31) ? o : 2u;
}
// The same over the threads, then over the warps: the state of the parts below this
// thread's, and the whole run's.
__device__ __forceinline__ uint32_t cta_state(uint32_t agg, uint32_t* wagg, uint32_t& total) {
    const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
    const uint32_t incl = warp_scan(agg);
    if (lane == 31) wagg[wid] = incl;
    __syncthreads();
    const uint32_t w = warp_scan(lane < nw ? wagg[lane] : 2u);
    total = __shfl_sync(0xffffffffu, w, nw - 1);
    const uint32_t below = __shfl_sync(0xffffffffu, w, wid ? wid - 1 : 0);
    return gp_join(wid ? below : 2u, warp_below(incl));
}
// The carry into this thread's part for a carry of 0 into the CTA's run.
__device__ __forceinline__ uint32_t cta_scan(uint32_t agg, uint32_t* wagg, uint32_t& total) {
    return cta_state(agg, wagg, total) & 1u;
}

__device__ __forceinline__ void add_carry(uint64_t* own, uint64_t cin) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
        own[q] += cin;
        cin = cin && own[q] == 0;
    }
}

// Limb sums of up to 4 * NT limbs, four per thread, from their coefficients'
// words lo + mid 2^64 + hi 2^128.  s_mid/s_hi entry 0 and s_c[0]: what reaches
// the first limb from below (s_c[0] may be written until the first barrier).
// own: the limbs with every carry inside the run; returns the run's state.
template <int NT>
struct LimbShared {
    uint64_t mid[NT + 1];
    uint32_t hi[NT + 1][2];
    uint32_t c[NT + 1];
    uint32_t wagg[32];
};
template <int NT>
__device__ __forceinline__ uint32_t limb_sums(LimbShared<NT>& S, int t, int nt, const uint64_t* lo, const uint64_t* mid,
                                              const uint32_t* hi, int nlimbs, uint64_t* own) {
    const bool in = t < nt;
    if (in) {
        S.mid[t + 1] = mid[3];
        S.hi[t + 1][0] = hi[2];
        S.hi[t + 1][1] = hi[3];
    }
    __syncthreads();
    // limb sums lo_i + mid_(i-1) + hi_(i-2) and their carries (0..2)
    uint32_t cy[4] = {0, 0, 0, 0};
    if (in) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint64_t m1 = q ? mid[q - 1] : S.mid[t];
            const uint32_t h2 = q > 1 ? hi[q - 2] : S.hi[t][q];
            uint64_t s = lo[q] + m1;
            uint32_t c = s < m1;
            s += h2;
            c += s < h2;
            own[q] = s;
            cy[q] = c;
        }
        S.c[t + 1] = cy[3];
    }
    __syncthreads();
    uint32_t agg = 0;
    if (in) {
        uint32_t k = S.c[t], g = 0, prop = 1;  // carry of the sum below; carry of adding it
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint64_t s = own[q] + k + g;  // k + g <= 3
            g = s < (uint64_t)(k + g);
            own[q] = s;
            k = cy[q];
            prop &= (4 * t + q < nlimbs && s == ~0ULL) ? 1u : 0u;
        }
        agg = g | (prop << 1);
    }
    uint32_t total;
    const uint64_t cin = cta_scan(agg, S.wagg, total);  // carry into the run taken as 0
    if (in) add_carry(own, cin);
    return total;
}

__device__ __forceinline__ void store_limbs(uint64_t* __restrict__ r, int64_t wt, int64_t w1, const uint64_t* own) {
    if (wt + 3 < w1) {
        ulonglong2* dst = reinterpret_cast<ulonglong2*>(r + wt);
        if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
            dst[0] = make_ulonglong2(own[0], own[1]);
            dst[1] = make_ulonglong2(own[2], own[3]);
            return;
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (wt + q < w1) r[wt + q] = own[q];
}

template <int SET>
__device__ __forceinline__ void coef_words(const uint32_t* r, const uint32_t* sc, uint64_t& lo, uint64_t& mid,
                                           uint32_t& hi) {
    uint32_t v[WCOEF];
    wcoef<SET>(r, sc, v);
    lo = v[0] | (uint64_t)v[1] << 32;
    mid = v[2] | (uint64_t)v[3] << 32;
    hi = v[4];
}

// Four consecutive coefficients; prime k's residues are x[k * stride].
template <int SET>
__device__ __forceinline__ void coef4(const uint4* __restrict__ x, int stride, const uint32_t* sc, uint64_t* lo,
                                      uint64_t* mid, uint32_t* hi) {
    constexpr int NP = word_np(SET);
    uint32_t r[4][NP];
#pragma unroll
    for (int k = 0; k < NP; k++) {
        const uint4 q = x[(size_t)k * stride];
        r[0][k] = q.x;
        r[1][k] = q.y;
        r[2][k] = q.z;
        r[3][k] = q.w;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) coef_words<SET>(r[q], sc, lo[q], mid[q], hi[q]);
}

// ---------------------------------------------------------------------------
// one-CTA products: N/16 threads per prime

template <int ODD, int LM>
struct WSmall {
    static constexpr int N = ODD << LM, M = 1 << LM, T = M / 16, TP = N / 16;
    static constexpr int NT = (WPR * TP + 31) / 32 * 32, SM = wwords(M);
    static constexpr int LT = N / 4 + 1;  // threads with limbs: r may have N + 1
    static constexpr int OPW = WPR * ODD * SM;  // words of one operand's blocks
    static constexpr size_t limb_bytes = (sizeof(LimbShared<LT>) + 15) / 16 * 16;
    static constexpr size_t bytes = limb_bytes + sizeof(uint32_t) * 2 * OPW;
};


// A thread's place: prime pi, thread u of that prime, block j, thread t of the block.
template <int ODD, int LM>
struct SmallThread {
    using W = WSmall<ODD, LM>;
    bool live;
    int pi, u, j, t;
    uint32_t p, pinv;
    const Tw *tf, *ti;  // the block's constants
    uint32_t *sp, *s;   // the prime's blocks, this thread's block
    __device__ __forceinline__ SmallThread(uint32_t* sm, const void* wtf, const void* wti, int wL) {
        const int tid = (int)threadIdx.x;
        live = tid < WPR * W::TP;
        pi = live ? tid / W::TP : 0;
        u = live ? tid - pi * W::TP : 0;
        j = u / W::T;
        t = u & (W::T - 1);
        p = c_w[0].p[pi];
        pinv = c_w[0].pinv[pi];
        const size_t toff = ((size_t)pi * ODD + j) << wL;
        tf = (const Tw*)wtf + toff;
        ti = (const Tw*)wti + toff;
        sp = sm + pi * ODD * W::SM;
        s = sp + j * W::SM;
        // the constants of every round, on their way while the limbs load: a
        // round then waits for the L1 instead of the L2
        constexpr int LINES = (1 << (LM - 2)) / 16;  // 128-byte lines per block and direction
        for (int i = tid; i < 2 * WPR * ODD * LINES; i += W::NT) {
            const int ln = i % LINES, blk = i / LINES % (WPR * ODD);
            const Tw* tb = (const Tw*)(i / (LINES * WPR * ODD) ? wti : wtf) + ((size_t)blk << wL) + 16 * ln;
            asm volatile("prefetch.global.L1 [%0];" ::"l"(tb));
        }
    }
    // The first round's values of an operand of n limbs (ODD > 1: into its
    // shared blocks spv, read back by fetch after a barrier).
    template <class LD>
    __device__ __forceinline__ void load(uint32_t* x, uint32_t* spv, int n, LD limb) const {
        constexpr int J1 = WSplit<LM>::J1;
        if (!live) return;
        if (ODD == 1) {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const int i = wpos<LM, LM, J1>(t, k >> J1) + ((k & ((1 << J1) - 1)) << (LM - J1));
                x[k] = wpack<false>(i < n ? limb(i) : 0ull, pi, p);
            }
        } else {
            for (int c = u; c < W::M; c += W::TP) {
                uint32_t y[ODD];
#pragma unroll
                for (int r = 0; r < ODD; r++) {
                    const int i = c + (r << LM);
                    y[r] = wpack<true>(i < n ? limb(i) : 0ull, pi, p);
                }
                dft_odd<ODD, 0>(y, pi, p);
#pragma unroll
                for (int r = 0; r < ODD; r++) spv[r * W::SM + wpad(c)] = y[r];
            }
        }
    }
    __device__ __forceinline__ void fetch(uint32_t* x, int op) const {
        if (ODD > 1 && live) wget<LM, LM, WSplit<LM>::J1>(s + op * W::OPW, x, t);
    }
    template <int NV>
    __device__ __forceinline__ void down(uint32_t* x) const {
        wblock_down<LM, NV, W::OPW>(x, s, t, tf, 1u, p, live);
    }
    __device__ __forceinline__ void point(uint32_t* x, bool sqr) const {
        if (live) wpoint<LM>(x, x + 16, sqr, t, tf, 1u, p, pinv);
    }
    // back to residues in the shared blocks (barrier at the end)
    __device__ __forceinline__ void up(uint32_t* a) const {
        wblock_up<LM>(a, s, t, ti, 1u, p, live);
        if (live) wput<LM, LM, WSplit<LM>::J1>(s, a, t);
        __syncthreads();
        if (ODD > 1) {
            if (live) {
                for (int c = u; c < W::M; c += W::TP) {
                    uint32_t v[ODD];
#pragma unroll
                    for (int r = 0; r < ODD; r++) v[r] = sp[r * W::SM + wpad(c)];
                    dft_odd<ODD, 0>(v, pi, p);
#pragma unroll
                    for (int r = 0; r < ODD; r++) sp[((ODD - r) % ODD) * W::SM + wpad(c)] = v[r];
                }
            }
            __syncthreads();
        }
    }
    // four coefficients of thread tid < N/4 from the shared blocks sm
    __device__ __forceinline__ static void coefs(const uint32_t* sm, const uint32_t* wsc, uint64_t* lo, uint64_t* mid,
                                                 uint32_t* hi) {
        const int tid = (int)threadIdx.x;
#pragma unroll
        for (int q = 0; q < 4; q++) lo[q] = mid[q] = 0, hi[q] = 0;
        if (4 * tid >= W::N) return;
        uint32_t sc[WPR];
#pragma unroll
        for (int k = 0; k < WPR; k++) sc[k] = wsc[k];
        const uint32_t* q0 = sm + ((4 * tid) >> LM) * W::SM + wpad((4 * tid) & (W::M - 1));  // four in one padded run
        coef4<0>(reinterpret_cast<const uint4*>(q0), ODD * W::SM / 4, sc, lo, mid, hi);
    }
};

}  // namespace nbg
