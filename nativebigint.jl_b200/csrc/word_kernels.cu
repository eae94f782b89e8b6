// word_kernels.cu — kernels of the word products (word.h): products through
// transforms modulo five 30-bit primes, one coefficient per 64-bit limb.
//
//   k_wcol_fwd  limbs -> residues, the radix-`odd` step and the first lj levels
//               of one column's R rows, in registers
//   k_wmid      long transforms: the levels between the first column pass and
//               the blocks, in registers
//   k_wblock    per block of M values: the other levels of a and b, the leaf
//               products, the levels back
//   k_wcol_rev  the first lj levels and the radix-`odd` step backwards
//   k_wunpack   five residues -> coefficient (mixed radix), carried limb sums
//   k_wcarry    carries between unpack tiles
//   k_wsmall    a whole product of at most 3072 coefficients in one CTA
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "word.cuh"
#include "word.h"

namespace nbg {

using wd::Tw;

struct WConst {
    uint32_t p[WPR], pinv[WPR];
    Tw c32[WPR], one[WPR];       // 2^32 mod p, 1
    Tw r3[WPR];                  // e(1/3)
    Tw r5[WPR][5];               // -1/4, (c1-c2)/2, f1, f2 of e(1/5) (see dft5); [4] unused
    uint32_t c7[WPR][3], f7[WPR][3];  // cosine and sine halves of e(j/7) in 2^32 form
    uint32_t wt[WPR][WPR];       // words of W_i = p_0 ... p_(i-1) (i words)
    uint32_t gar[WPR][WPR];      // mixed radix: gar[i][j] = -W_j / W_i mod p_i in 2^32 form (j < i)
};
__constant__ WConst c_w;

// ---------------------------------------------------------------------------
// host constants

static uint64_t pw(uint64_t a, uint64_t e, uint64_t p) {
    uint64_t r = 1;
    for (a %= p; e; e >>= 1, a = a * a % p)
        if (e & 1) r = r * a % p;
    return r;
}
static uint64_t inv(uint64_t a, uint64_t p) { return pw(a, p - 2, p); }
// a primitive root: p - 1 = 105 * 2^18 * c, its prime factors are 2, 3, 5, 7 and c's
static uint64_t prim_root(uint64_t p) {
    for (uint64_t g = 2;; g++) {
        bool ok = true;
        uint64_t n = p - 1;
        for (uint64_t f = 2; ok && f * f <= n; f++)
            if (n % f == 0) {
                ok = pw(g, (p - 1) / f, p) != 1;
                while (n % f == 0) n /= f;
            }
        if (ok && n > 1) ok = pw(g, (p - 1) / n, p) != 1;
        if (ok) return g;
    }
}
static uint64_t root_of(int i) {
    static const uint64_t g[WPR] = {prim_root(WPRIMES[0]), prim_root(WPRIMES[1]), prim_root(WPRIMES[2]),
                                    prim_root(WPRIMES[3]), prim_root(WPRIMES[4])};
    return g[i];
}
static Tw mk(uint64_t w, uint64_t p) { return Tw{(uint32_t)w, (uint32_t)((w << 32) / p)}; }
static uint32_t mont(uint64_t w, uint64_t p) { return (uint32_t)(((w % p) << 32) % p); }

static cudaError_t small_attributes();

cudaError_t word_init() {
    WConst h{};
    for (int i = 0; i < WPR; i++) {
        const uint64_t p = WPRIMES[i], g = root_of(i);
        h.p[i] = (uint32_t)p;
        uint32_t x = 1;
        for (int k = 0; k < 5; k++) x *= 2 - (uint32_t)p * x;  // Newton: p^-1 mod 2^32
        h.pinv[i] = x;
        h.c32[i] = mk((uint64_t(1) << 32) % p, p);
        h.one[i] = mk(1, p);
        h.r3[i] = mk(pw(g, (p - 1) / 3, p), p);
        const uint64_t h2 = inv(2, p), w5 = pw(g, (p - 1) / 5, p), w7 = pw(g, (p - 1) / 7, p);
        auto half = [&](uint64_t w, int a, int b, bool minus) {  // (w^a +- w^b) / 2
            const uint64_t x1 = pw(w, a, p), x2 = pw(w, b, p);
            return (x1 + (minus ? p - x2 : x2)) % p * h2 % p;
        };
        const uint64_t c1 = half(w5, 1, 4, false), c2 = half(w5, 2, 3, false);
        h.r5[i][0] = mk((p - inv(4, p)) % p, p);
        h.r5[i][1] = mk((c1 + p - c2) % p * h2 % p, p);
        h.r5[i][2] = mk(half(w5, 1, 4, true), p);
        h.r5[i][3] = mk(half(w5, 2, 3, true), p);
        for (int k = 0; k < 3; k++) {
            h.c7[i][k] = mont(half(w7, k + 1, 6 - k, false), p);
            h.f7[i][k] = mont(half(w7, k + 1, 6 - k, true), p);
        }
        uint64_t Wi = 1;
        for (int t = 0; t < i; t++) Wi = Wi * (WPRIMES[t] % p) % p;
        const uint64_t iw = inv(Wi, p);
        uint64_t Wj = 1;
        for (int j = 0; j < i; j++) {
            h.gar[i][j] = mont((p - Wj * iw % p) % p, p);
            Wj = Wj * (WPRIMES[j] % p) % p;
        }
        uint32_t w[WPR] = {1};
        for (int t = 0; t < i; t++) {
            uint64_t cy = 0;
            for (int k = 0; k < WPR; k++) {
                cy += (uint64_t)w[k] * WPRIMES[t];
                w[k] = (uint32_t)cy;
                cy >>= 32;
            }
        }
        for (int k = 0; k < WPR; k++) h.wt[i][k] = w[k];
    }
    cudaError_t e = small_attributes();
    return e == cudaSuccess ? cudaMemcpyToSymbol(c_w, &h, sizeof h) : e;
}

void word_scales(const WordShape& s, uint32_t out[WPR]) {
    // 2^32 (pointwise) * 2^32 (unpack's reduction) / (odd * 2^levels * W_i)
    static const struct Table {
        uint32_t v[8][WORD_MAX_LOG2][WPR];
        Table() {
            uint64_t W[WPR];
            for (int i = 0; i < WPR; i++) {
                W[i] = 1;
                for (int j = 0; j < i; j++) W[i] = W[i] * (WPRIMES[j] % WPRIMES[i]) % WPRIMES[i];
            }
            for (int odd = 1; odd < 8; odd += 2)
                for (int lev = 0; lev < WORD_MAX_LOG2; lev++)
                    for (int i = 0; i < WPR; i++) {
                        const uint64_t p = WPRIMES[i], r = (uint64_t(1) << 32) % p;
                        v[odd][lev][i] = (uint32_t)(r * r % p * inv(odd * pw(2, (uint64_t)lev, p) % p * W[i] % p, p) % p);
                    }
        }
    } t;
    for (int i = 0; i < WPR; i++) out[i] = t.v[s.odd][s.lj + s.lm - 2][i];
}

// The split of the rows above the blocks: one column pass up to 32 rows (its
// values fit a thread's registers), else the two passes whose larger row count
// is least.
static bool row_split(int odd, int lj, int& j2) {
    j2 = 0;
    const int64_t R = (int64_t)odd << lj;
    if (R <= 32) return R >= 2;
    int64_t best = INT64_MAX;
    for (int j = 2; j <= 5 && j <= lj; j++) {
        const int64_t r1 = (int64_t)odd << (lj - j), r2 = int64_t(1) << j;
        if (r1 < 2 || r1 > 32 || std::max(r1, r2) >= best) continue;
        best = std::max(r1, r2);
        j2 = j;
    }
    return best != INT64_MAX;
}

// Every supported shape, shortest first.
static const std::vector<WordShape>& shape_list() {
    static const std::vector<WordShape> list = [] {
        std::vector<WordShape> v;
        for (int odd : {1, 3, 5, 7})
            for (int k = 6; k <= WORD_MAX_LOG2; k++) {
                const int64_t N = (int64_t)odd << k;
                if (k <= 11 && WPR * N <= 16 * 1024) {
                    v.push_back(WordShape{(int32_t)N, odd, 0, 0, k, true});
                    continue;
                }
                for (int lm : {12, 10, 8, 6}) {
                    int j2;
                    if (k < lm || !row_split(odd, k - lm, j2)) continue;
                    v.push_back(WordShape{(int32_t)N, odd, k - lm, j2, lm, false});
                    break;
                }
            }
        std::sort(v.begin(), v.end(), [](const WordShape& x, const WordShape& y) { return x.N < y.N; });
        return v;
    }();
    return list;
}

bool word_shape(int64_t nconv, WordShape& s) {
    const std::vector<WordShape>& v = shape_list();
    const auto it = std::lower_bound(v.begin(), v.end(), nconv,
                                     [](const WordShape& x, int64_t n) { return x.N < n; });
    if (it == v.end()) return false;
    s = *it;
    return true;
}

// ---------------------------------------------------------------------------
// tables

size_t word_table_bytes(int odd, int L) { return sizeof(Tw) * ((size_t)WPR * odd << L); }

__device__ uint32_t pw_dev(uint32_t a, uint32_t e, uint32_t p) {
    uint64_t r = 1, b = a;
    for (; e; e >>= 1, b = b * b % p)
        if (e & 1) r = r * b % p;
    return (uint32_t)r;
}

struct WRoots {
    uint32_t g[WPR];
};
// entry h = 2^l + n of (prime i, block j): e((j + odd * bitrev_l(n)) / (odd * 2^(l+1))) and its inverse
__global__ void k_wtable(Tw* __restrict__ fwd, Tw* __restrict__ bwd, int odd, int L, WRoots g) {
    const int64_t total = (int64_t)WPR * odd << L;
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < total; x += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t h = (uint32_t)(x & ((int64_t(1) << L) - 1));
        const int ij = (int)(x >> L), i = ij / odd, j = ij - i * odd;
        const uint32_t p = c_w.p[i];
        uint32_t e = 0;
        if (h) {
            const int l = 31 - __clz(h);
            const uint32_t n = h - (1u << l);
            const uint32_t brv = l ? __brev(n) >> (32 - l) : 0;
            e = (p - 1) / ((uint32_t)odd << (l + 1)) * ((uint32_t)j + (uint32_t)odd * brv);
        }
        const uint32_t w = pw_dev(g.g[i], e, p), v = e ? pw_dev(g.g[i], p - 1 - e, p) : 1u;
        fwd[x] = Tw{w, (uint32_t)(((uint64_t)w << 32) / p)};
        bwd[x] = Tw{v, (uint32_t)(((uint64_t)v << 32) / p)};
    }
}

cudaError_t word_build_tables(int odd, int L, void* fwd, void* bwd, cudaStream_t st) {
    WRoots g;
    for (int i = 0; i < WPR; i++) g.g[i] = (uint32_t)root_of(i);
    k_wtable<<<148 * 8, 256, 0, st>>>((Tw*)fwd, (Tw*)bwd, odd, L, g);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// radix-odd steps: in and out in [0, 2p) unless said otherwise

// y_j = sum x_i e(ij/3): with w + w^2 = -1 one product suffices
__device__ __forceinline__ void dft3(uint32_t* x, int st, int i, uint32_t p) {
    const uint32_t p2 = 2 * p;
    uint32_t &a = x[0], &b = x[st], &c = x[2 * st];
    const uint32_t t = wd::mulw(b - c + p2, c_w.r3[i], p);
    const uint32_t y0 = wd::sub_if(wd::sub_if(a + b, p2) + c, p2);
    const uint32_t y1 = wd::sub_if(wd::sub_if(a - c + p2, p2) + t, p2);
    const uint32_t u = wd::sub_if(a - b + p2, p2);
    const uint32_t y2 = wd::sub_if(u - t + p2, p2);
    a = y0;
    b = y1;
    c = y2;
}
// cosine halves c1, c2 = -1/4 +- d: two products for the even part, four for the odd
__device__ __forceinline__ void dft5(uint32_t* x, int st, int i, uint32_t p) {
    const uint32_t p2 = 2 * p;
    const Tw q = c_w.r5[i][0], d = c_w.r5[i][1], f1 = c_w.r5[i][2], f2 = c_w.r5[i][3];
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
__device__ __forceinline__ void dft7(uint32_t* x, int st, int i, uint32_t p) {
    const uint32_t p2 = 2 * p, pinv = c_w.pinv[i];
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
            ce += wd::mulx(s[k - 1], c_w.c7[i][a - 1]);
            so += wd::mulx(t <= 3 ? d[k - 1] : p2 - d[k - 1], c_w.f7[i][a - 1]);
        }
        // each sum < 3 * 2p * p, reduced below 1.5p + p
        const uint32_t C = wd::sub_if(x0 + wd::sub_if(wd::redc(ce, p, pinv), p2), p2);
        const uint32_t S = wd::sub_if(wd::redc(so, p, pinv), p2);
        x[j * st] = wd::sub_if(C + S, p2);
        x[(7 - j) * st] = wd::sub_if(C - S + p2, p2);
    }
}

template <int ODD, int LJ>
__device__ __forceinline__ void dft_odd(uint32_t* x, int i, uint32_t p) {
#pragma unroll
    for (int r = 0; r < (1 << LJ); r++) {
        if (ODD == 3) dft3(x + r, 1 << LJ, i, p);
        if (ODD == 5) dft5(x + r, 1 << LJ, i, p);
        if (ODD == 7) dft7(x + r, 1 << LJ, i, p);
    }
}

// ---------------------------------------------------------------------------
// job lookup: segment of this CTA, its product and the CTA's index inside it

// A launch's products: a batch's tables, or (nseg = 0) one product by value.
struct WArgs {
    const DProd* prods;
    const WSeg* segs;
    const int32_t* plist;
    int32_t nseg;
    DProd one;
};

__device__ __forceinline__ const DProd& wjob(const WArgs& A, int& local) {
    local = (int)blockIdx.x;
    if (A.nseg == 0) return A.one;
    const WSeg* __restrict__ segs = A.segs;
    int lo = 0, hi = A.nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (segs[mid].begin <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const WSeg g = segs[lo];
    const int q = ((int)blockIdx.x - g.begin) / g.cpp;
    local = (int)blockIdx.x - g.begin - q * g.cpp;
    return A.prods[A.plist[g.first + q]];
}

constexpr int WT = 256;  // threads per CTA

// ---------------------------------------------------------------------------
// column passes: one thread holds the R rows of one column of one prime

// A limb modulo p, in [0, 4p) (RED: [0, 2p)).
template <bool RED>
__device__ __forceinline__ uint32_t wpack(uint64_t v, int pi, uint32_t p) {
    const uint32_t y = wd::mulw((uint32_t)(v >> 32), c_w.c32[pi], p) + wd::mulw((uint32_t)v, c_w.one[pi], p);
    return RED ? wd::sub_if(y, 2 * p) : y;
}

// LM: log2 of the column count when the blocks are 4096 values (row strides are
// then immediate offsets), 0: read from the product.  Rows past the operand are
// not packed, and when they are its upper half (odd = 1, a half-length operand,
// which one of two always is) the first level is a copy.
template <int ODD, int LJ, int LM>
__global__ void __launch_bounds__(WT, 4) k_wcol_fwd(const __grid_constant__ WArgs A) {
    constexpr int R = ODD << LJ;
    int local;
    const DProd& P = wjob(A, local);
    const int lm = LM ? LM : P.wlm + P.wj2;
    const int id = local * WT + (int)threadIdx.x;
    const int c = id & ((1 << lm) - 1);
    int pi = id >> lm;  // operand-major: a's primes, then b's
    const bool isb = pi >= WPR;
    if (isb) pi -= WPR;
    if (pi >= WPR || (isb && P.sqr)) return;
    const int n = (int)(isb ? P.ncb : P.nca);
    const int rows = (n + (1 << lm) - 1) >> lm;
    const uint64_t* __restrict__ src = (isb ? P.b : P.a) + c;
    uint32_t* __restrict__ dst = (isb ? P.wb : P.wa) + (size_t)pi * (size_t)P.wN + c;
    const uint32_t p = c_w.p[pi];
    const Tw* tab = (const Tw*)P.wtf + (((size_t)pi * ODD) << P.wL);
    uint32_t x[R];
    auto rowsin = [&](auto r0c, auto r1c) {
        constexpr int r0 = decltype(r0c)::value, r1 = decltype(r1c)::value;
        uint64_t v[r1 - r0];
#pragma unroll
        for (int r = r0; r < r1; r++) v[r - r0] = c + (r << lm) < n ? __ldg(src + ((size_t)r << lm)) : 0ull;
#pragma unroll
        for (int r = r0; r < r1; r++) x[r] = r < rows ? wpack<(ODD > 1)>(v[r - r0], pi, p) : 0u;
    };
    constexpr int H = R / 2;
    if (ODD == 1 && LJ > 0 && rows <= H) {
        rowsin(std::integral_constant<int, 0>{}, std::integral_constant<int, H>{});
#pragma unroll
        for (int r = 0; r < H; r++) x[r + H] = x[r];
        wd::tree_fwd<LJ, 1, 1, 0, 1>(x, tab, 1u, p);
    } else {
        if (R > 16) {  // at most half of the limbs in registers at once
            rowsin(std::integral_constant<int, 0>{}, std::integral_constant<int, H>{});
            rowsin(std::integral_constant<int, H>{}, std::integral_constant<int, R>{});
        } else {
            rowsin(std::integral_constant<int, 0>{}, std::integral_constant<int, R>{});
        }
        dft_odd<ODD, LJ>(x, pi, p);
#pragma unroll
        for (int j = 0; j < ODD; j++) wd::tree_fwd<LJ, 1>(x + (j << LJ), tab + ((size_t)j << P.wL), 1u, p);
    }
#pragma unroll
    for (int r = 0; r < R; r++) dst[(size_t)r << lm] = x[r];
}

template <int ODD, int LJ, int LM>
__global__ void __launch_bounds__(WT, LM ? 4 : 3) k_wcol_rev(const __grid_constant__ WArgs A) {
    constexpr int R = ODD << LJ;
    int local;
    const DProd& P = wjob(A, local);
    const int lm = LM ? LM : P.wlm + P.wj2;
    const int id = local * WT + (int)threadIdx.x;
    const int c = id & ((1 << lm) - 1);
    const int pi = id >> lm;
    if (pi >= WPR) return;
    uint32_t* __restrict__ dst = P.wa + (size_t)pi * (size_t)P.wN + c;
    const uint32_t p = c_w.p[pi];
    uint32_t x[R];
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = dst[(size_t)r << lm];
    const Tw* tab = (const Tw*)P.wti + (((size_t)pi * ODD) << P.wL);
#pragma unroll
    for (int j = 0; j < ODD; j++) wd::tree_rev<LJ, 1>(x + (j << LJ), tab + ((size_t)j << P.wL), 1u, p);
    dft_odd<ODD, LJ>(x, pi, p);
    // the inverse step is the forward one with output i at -i mod odd
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = r >> LJ, ri = (ODD - i) % ODD;
        dst[(size_t)((ri << LJ) + (r & ((1 << LJ) - 1))) << lm] = x[r];
    }
}

// Middle passes: the 2^J rows (2^lm apart) of one column of a segment, the
// subtree of the segment's node, above blocks of 4096.  In place; all columns of a segment share
// their constants.
template <int J, bool FWD>
__global__ void __launch_bounds__(WT) k_wmid(const __grid_constant__ WArgs A) {
    int local;
    const DProd& P = wjob(A, local);
    constexpr int lm = 12;  // more than 32 rows only stand above 4096-value blocks
    const int j1 = P.wlj - J, R1 = P.wodd << j1;
    const int id = local * WT + (int)threadIdx.x;
    const int c = id & ((1 << lm) - 1);
    int op = (id >> lm) / R1;  // operand-major, then prime
    const int seg = (id >> lm) - op * R1;
    const bool isb = op >= WPR;
    const int pi = isb ? op - WPR : op;
    if (pi >= WPR || (isb && (!FWD || P.sqr))) return;
    uint32_t* __restrict__ x0 = (isb ? P.wb : P.wa) + (size_t)pi * (size_t)P.wN + ((size_t)seg << (lm + J)) + c;
    const uint32_t p = c_w.p[pi];
    const Tw* tab = (const Tw*)(FWD ? P.wtf : P.wti) + (((size_t)pi * P.wodd + (seg >> j1)) << P.wL);
    const uint32_t node = (1u << j1) + (uint32_t)(seg & ((1 << j1) - 1));
    uint32_t x[1 << J];
#pragma unroll
    for (int r = 0; r < (1 << J); r++) x[r] = x0[(size_t)r << lm];
    if (FWD) wd::tree_fwd<J, 1>(x, tab, node, p);
    else wd::tree_rev<J, 1>(x, tab, node, p);
#pragma unroll
    for (int r = 0; r < (1 << J); r++) x0[(size_t)r << lm] = x[r];
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

// c = a * b mod X^4 - rho (rho in 2^32 form), a in [0, p), b in [0, 2p); the
// result carries a factor 2^-32 and lies in [0, 2p).  Sums of at most four
// products of 2p^2 and one of 2.5p * p stay below 2^64.
__device__ __forceinline__ void wleaf(uint32_t* a, const uint32_t* b, uint32_t rho, uint32_t p, uint32_t pinv) {
    uint32_t h[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        uint64_t s = 0;
#pragma unroll
        for (int i = k + 1; i < 4; i++) s += wd::mulx(a[i], b[k + 4 - i]);
        h[k] = wd::redc(s, p, pinv);
    }
    uint32_t c[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        uint64_t s = k < 3 ? wd::mulx(h[k], rho) : 0;
#pragma unroll
        for (int i = 0; i <= k; i++) s += wd::mulx(a[i], b[k - i]);
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
    const uint32_t r0 = 0u - w2[0].q * p, r1 = 0u - w2[1].q * p;  // w * 2^32 mod p
#pragma unroll
    for (int k = 0; k < 16; k++) {
        a[k] = wd::sub_if(wd::sub_if(a[k], p2), p);
        b[k] = sqr ? a[k] : wd::sub_if(b[k], p2);
    }
    wleaf(a, b, r0, p, pinv);
    wleaf(a + 4, b + 4, p - r0, p, pinv);
    wleaf(a + 8, b + 8, r1, p, pinv);
    wleaf(a + 12, b + 12, p - r1, p, pinv);
}

template <int LM>
__global__ void __launch_bounds__(WT, 3) k_wblock(const __grid_constant__ WArgs A) {
    constexpr int T = 1 << (LM - 4), PER = WT / T;  // threads per block, blocks per CTA
    constexpr int SM = wwords(1 << LM);
    constexpr int J1 = WSplit<LM>::J1;
    __shared__ __align__(16) uint32_t sm[PER][2][SM];
    int local;
    const DProd& P = wjob(A, local);
    const int g = (int)threadIdx.x / T, t = (int)threadIdx.x & (T - 1);
    const int R = P.wodd << P.wlj;
    const int blk = local * PER + g;  // prime-major, then block
    const bool live = blk < WPR * R;
    const int pi = live ? blk / R : 0, row = live ? blk - pi * R : 0;
    const int j = row >> P.wlj;
    const uint32_t h0 = (1u << P.wlj) + (uint32_t)(row & ((1 << P.wlj) - 1));
    const uint32_t p = c_w.p[pi], pinv = c_w.pinv[pi];
    const size_t toff = ((size_t)pi * P.wodd + j) << P.wL, xoff = (size_t)pi * (size_t)P.wN + ((size_t)row << LM);
    const Tw* tf = (const Tw*)P.wtf + toff;
    uint32_t* xa = P.wa + xoff;
    uint32_t x[32];  // a's 16 values, then b's
    auto load = [&](uint32_t* v, const uint32_t* src) {
#pragma unroll
        for (int k = 0; k < 16; k++)
            v[k] = src[wpos<LM, LM, J1>(t, k >> J1) + ((k & ((1 << J1) - 1)) << (LM - J1))];
    };
    uint32_t* const a = x;
    if (live) load(x, xa);
    if (!P.sqr) {
        if (live) load(x + 16, P.wb + xoff);
        wblock_down<LM, 2, SM>(x, sm[g][0], t, tf, h0, p, live);
    } else {
        wblock_down<LM, 1, SM>(x, sm[g][0], t, tf, h0, p, live);
    }
    if (live) wpoint<LM>(x, x + 16, P.sqr, t, tf, h0, p, pinv);
    wblock_up<LM>(x, sm[g][0], t, (const Tw*)P.wti + toff, h0, p, live);
    if (live) {
#pragma unroll
        for (int k = 0; k < 16; k++)
            xa[wpos<LM, LM, J1>(t, k >> J1) + ((k & ((1 << J1) - 1)) << (LM - J1))] = a[k];
    }
}

// ---------------------------------------------------------------------------
// unpack: coefficients and carried limbs, tiles of UNPACK_TL limbs

// The coefficient whose residues (representatives below 2p, scaled) are r:
// mixed-radix digits y_i, each one sum of wide products and one reduction, then
// sum y_i W_i by columns of 32 bits (at most four products below 2^62 each).
__device__ __forceinline__ void wcoef(const uint32_t* r, const uint32_t* sc, uint32_t* v) {
    uint32_t y[WPR];
#pragma unroll
    for (int i = 0; i < WPR; i++) {
        const uint32_t p = c_w.p[i];
        uint64_t s = wd::mulx(r[i], sc[i]);  // < 2p^2; the others < 1.3p^2 each
#pragma unroll
        for (int j = 0; j < i; j++) s += wd::mulx(y[j], c_w.gar[i][j]);
        // below 1.5p, 1.85p, 2.2p, 2.5p, 2.8p: one or two subtractions
        y[i] = wd::sub_if(wd::redc(s, p, c_w.pinv[i]), p);
        if (i > 1) y[i] = wd::sub_if(y[i], p);
    }
    uint64_t s = y[0];
#pragma unroll
    for (int k = 0; k < WPR - 1; k++) {
        uint64_t col = wd::mulx(y[k + 1], c_w.wt[k + 1][k]);
#pragma unroll
        for (int i = k + 2; i < WPR; i++) col += wd::mulx(y[i], c_w.wt[i][k]);
        // col < (4 - k) * 2^62 and s < 2^33: no overflow
        s += col;
        v[k] = (uint32_t)s;
        s >>= 32;
    }
    v[WPR - 1] = (uint32_t)s;
}

__device__ __forceinline__ uint32_t gp_join(uint32_t lower, uint32_t upper) {
    // bit 0 generate, bit 1 propagate; lower limbs, then upper
    return ((upper & 1u) | ((upper >> 1) & lower & 1u)) | (upper & lower & 2u);
}

// Limb sums of up to 4 * NT limbs, four per thread, from their coefficients'
// words lo + mid 2^64 + hi 2^128.  s_mid/s_hi entry 0 and s_c[0]: what reaches
// the first limb from below (s_c[0] may be written until the first barrier).
// own: the limbs with every carry inside the run; returns this thread's
// inclusive (generate, propagate) state of the run in the last thread.
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
    // carry-lookahead over the threads, then over the warps
    const int lane = t & 31, wid = t >> 5;
    uint32_t incl = agg;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl = gp_join(o, incl);
    }
    if (lane == 31) S.wagg[wid] = incl;
    __syncthreads();
    uint32_t wpre = lane < (int)(blockDim.x >> 5) ? S.wagg[lane] : 2u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, wpre, off);
        if (lane >= off) wpre = gp_join(o, wpre);
    }
    wpre = wid ? __shfl_sync(0xffffffffu, wpre, wid ? wid - 1 : 0) : 2u;
    uint32_t excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = 2u;
    uint64_t cin = gp_join(wpre, excl) & 1u;  // carry into the run taken as 0
    if (in) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            own[q] += cin;
            cin = cin && own[q] == 0;
        }
    }
    return gp_join(wpre, incl);
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

__device__ __forceinline__ void coef_words(const uint32_t* r, const uint32_t* sc, uint64_t& lo, uint64_t& mid,
                                           uint32_t& hi) {
    uint32_t v[WPR];
    wcoef(r, sc, v);
    lo = v[0] | (uint64_t)v[1] << 32;
    mid = v[2] | (uint64_t)v[3] << 32;
    hi = v[4];
}

// Four consecutive coefficients; prime k's residues are x[k * stride].
__device__ __forceinline__ void coef4(const uint4* __restrict__ x, int stride, const uint32_t* sc, uint64_t* lo,
                                      uint64_t* mid, uint32_t* hi) {
    uint32_t r[4][WPR];
#pragma unroll
    for (int k = 0; k < WPR; k++) {
        const uint4 q = x[(size_t)k * stride];
        r[0][k] = q.x;
        r[1][k] = q.y;
        r[2][k] = q.z;
        r[3][k] = q.w;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) coef_words(r[q], sc, lo[q], mid[q], hi[q]);
}

__global__ void __launch_bounds__(WT) k_wunpack(const __grid_constant__ WArgs A) {
    __shared__ LimbShared<WT> S;
    __shared__ uint64_t h_lo, h_mid2;  // the limb sum below the tile
    __shared__ uint32_t h_hi3;
    int tile;
    const DProd& P = wjob(A, tile);
    const int t = (int)threadIdx.x;
    const int N = P.wN;
    const uint32_t* __restrict__ x = P.wa;
    const int64_t w0 = (int64_t)tile * UNPACK_TL, w1 = min(w0 + (int64_t)UNPACK_TL, P.rn);
    uint32_t sc[WPR];
#pragma unroll
    for (int i = 0; i < WPR; i++) sc[i] = P.wsc[i];
    // the three coefficients before the tile
    if (t < 3) {
        const int64_t i = w0 - 1 - t;
        uint64_t lo = 0, mid = 0;
        uint32_t hi = 0;
        if (i >= 0 && i < N) {
            uint32_t r[WPR];
#pragma unroll
            for (int k = 0; k < WPR; k++) r[k] = x[(size_t)k * N + i];
            coef_words(r, sc, lo, mid, hi);
        }
        if (t == 0) {
            h_lo = lo;
            S.mid[0] = mid;
            S.hi[0][1] = hi;
        } else if (t == 1) {
            h_mid2 = mid;
            S.hi[0][0] = hi;
        } else {
            h_hi3 = hi;
        }
        __syncwarp(7u);
        if (t == 0) {
            uint64_t s = h_lo + h_mid2;
            uint32_t c = s < h_mid2;
            s += h_hi3;
            c += s < h_hi3;
            S.c[0] = c;
        }
    }
    const int64_t wt = w0 + 4 * t;
    uint64_t lo[4] = {0, 0, 0, 0}, mid[4] = {0, 0, 0, 0}, own[4];
    uint32_t hi[4] = {0, 0, 0, 0};
    if (wt < N) {  // N is a multiple of 4: all four or none
        coef4(reinterpret_cast<const uint4*>(x + wt), N / 4, sc, lo, mid, hi);
    }
    const uint32_t tot = limb_sums<WT>(S, t, WT, lo, mid, hi, (int)(w1 - w0), own);
    store_limbs(P.r, wt, w1, own);
    if (t == WT - 1) P.agg[tile] = tot;
}

// Carries between a product's unpack tiles: one warp per 32 tiles.  The carry
// into its first tile comes from the last lower tile that does not propagate
// (almost always the one before); a tile's carry stops at its first limb
// unless that limb is all ones, and then the warp walks the run.  Only r is
// written, each tile by one warp.
__global__ void __launch_bounds__(WT) k_wcarry(const __grid_constant__ WArgs A) {
    int local;
    const DProd& P = wjob(A, local);
    const int lane = (int)threadIdx.x & 31;
    const int64_t k0 = ((int64_t)local * (WT / 32) + (threadIdx.x >> 5)) * 32, nt = P.ntl;
    if (k0 >= nt) return;
    uint32_t cin = 0;
    for (int64_t k = k0 - 32; k >= 0; k -= 32) {
        const uint32_t a = P.agg[k + lane];
        const unsigned stop = __ballot_sync(0xffffffffu, !(a & 2u));
        if (stop) {
            cin = __shfl_sync(0xffffffffu, a, 31 - __clz(stop)) & 1u;
            break;
        }
    }
    const int64_t k = k0 + lane;
    uint32_t incl = k < nt ? P.agg[k] : 0u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl = gp_join(o, incl);
    }
    uint32_t excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = 2u;
    bool walk = false;
    if (k < nt && (gp_join(cin, excl) & 1u)) {
        uint64_t* w = P.r + k * UNPACK_TL;
        if (*w != ~0ULL) *w += 1;
        else walk = true;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, walk); m; m &= m - 1) {
        const int64_t b0 = (k0 + __ffs(m) - 1) * UNPACK_TL, b1 = min(b0 + (int64_t)UNPACK_TL, P.rn);
        for (int64_t w = b0; w < b1; w += 32) {
            const int64_t wl = w + lane;
            const uint64_t v = wl < b1 ? P.r[wl] : 0ULL;  // past the tile: stops the run
            const unsigned stop = __ballot_sync(0xffffffffu, v != ~0ULL);
            const int e = stop ? __ffs(stop) - 1 : 32;
            if (lane < e) P.r[wl] = 0;
            else if (lane == e && wl < b1) P.r[wl] = v + 1;
            if (stop) break;
        }
    }
}

// ---------------------------------------------------------------------------
// small products: one CTA does all of it, N/16 threads per prime; the
// transforms, the residues and the limbs stay on chip

template <int ODD, int LM>
struct WSmall {
    static constexpr int N = ODD << LM, M = 1 << LM, T = M / 16, TP = N / 16;
    static constexpr int NT = (WPR * TP + 31) / 32 * 32, SM = wwords(M);
    static constexpr int LT = N / 4 + 1;  // threads with limbs: r may have N + 1
    static constexpr int OPW = WPR * ODD * SM;  // words of one operand's blocks
    static constexpr size_t bytes = (sizeof(LimbShared<LT>) + 15) / 16 * 16 + sizeof(uint32_t) * 2 * OPW;
};

template <int ODD, int LM>
__global__ void __launch_bounds__(WSmall<ODD, LM>::NT, WSmall<ODD, LM>::NT > 320 ? 1 : 640 / WSmall<ODD, LM>::NT)
    k_wsmall(const __grid_constant__ WArgs A) {
    using W = WSmall<ODD, LM>;
    constexpr int J1 = WSplit<LM>::J1, N = W::N, M = W::M, SM = W::SM, TP = W::TP;
    static_assert(W::LT <= W::NT && W::NT <= 1024, "limb threads");
    extern __shared__ __align__(16) unsigned char dyn[];
    LimbShared<W::LT>& S = *reinterpret_cast<LimbShared<W::LT>*>(dyn);
    uint32_t* sm = reinterpret_cast<uint32_t*>(dyn + (sizeof(LimbShared<W::LT>) + 15) / 16 * 16);
    int local;
    const DProd& P = wjob(A, local);
    const int tid = (int)threadIdx.x;
    const bool live = tid < WPR * TP;
    const int pi = live ? tid / TP : 0, u = live ? tid - pi * TP : 0;
    const int j = u / W::T, t = u & (W::T - 1);
    const uint32_t p = c_w.p[pi], pinv = c_w.pinv[pi];
    const size_t toff = ((size_t)pi * ODD + j) << P.wL;
    const Tw *tf = (const Tw*)P.wtf + toff, *ti = (const Tw*)P.wti + toff;
    uint32_t* const sp = sm + pi * ODD * SM;  // this prime's blocks
    uint32_t* const s = sp + j * SM;
    uint32_t x[32];  // a's 16 values, then b's
    uint32_t* const a = x;
    auto load = [&](uint32_t* v, uint32_t* spv, const uint64_t* __restrict__ src, int n) {
        if (!live) return;
        if (ODD == 1) {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const int i = wpos<LM, LM, J1>(t, k >> J1) + ((k & ((1 << J1) - 1)) << (LM - J1));
                v[k] = wpack<false>(i < n ? __ldg(src + i) : 0ull, pi, p);
            }
        } else {
            for (int c = u; c < M; c += TP) {
                uint32_t y[ODD];
#pragma unroll
                for (int r = 0; r < ODD; r++) {
                    const int i = c + (r << LM);
                    y[r] = wpack<true>(i < n ? __ldg(src + i) : 0ull, pi, p);
                }
                dft_odd<ODD, 0>(y, pi, p);
#pragma unroll
                for (int r = 0; r < ODD; r++) spv[r * SM + wpad(c)] = y[r];
            }
        }
    };
    // the constants of every later round, on their way while the limbs load: a
    // round then waits for the L1 instead of the L2
    constexpr int LINES = (1 << (LM - 2)) / 16;  // 128-byte lines per block and direction
    for (int i = tid; i < 2 * WPR * ODD * LINES; i += W::NT) {
        const int ln = i % LINES, blk = i / LINES % (WPR * ODD);
        const Tw* tb = (const Tw*)(i / (LINES * WPR * ODD) ? P.wti : P.wtf) + ((size_t)blk << P.wL) + 16 * ln;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(tb));
    }
    load(x, sp, P.a, (int)P.nca);
    if (!P.sqr) load(x + 16, sp + W::OPW, P.b, (int)P.ncb);
    if (ODD > 1) {
        __syncthreads();
        if (live) wget<LM, LM, J1>(s, x, t);
        if (live && !P.sqr) wget<LM, LM, J1>(s + W::OPW, x + 16, t);
    }
    if (!P.sqr) wblock_down<LM, 2, W::OPW>(x, s, t, tf, 1u, p, live);
    else wblock_down<LM, 1, W::OPW>(x, s, t, tf, 1u, p, live);
    if (live) wpoint<LM>(x, x + 16, P.sqr, t, tf, 1u, p, pinv);
    wblock_up<LM>(a, s, t, ti, 1u, p, live);
    if (live) wput<LM, LM, J1>(s, a, t);
    __syncthreads();
    if (ODD > 1) {
        if (live) {
            for (int c = u; c < M; c += TP) {
                uint32_t v[ODD];
#pragma unroll
                for (int r = 0; r < ODD; r++) v[r] = sp[r * SM + wpad(c)];
                dft_odd<ODD, 0>(v, pi, p);
#pragma unroll
                for (int r = 0; r < ODD; r++) sp[((ODD - r) % ODD) * SM + wpad(c)] = v[r];
            }
        }
        __syncthreads();
    }
    // coefficients and limbs: thread tid < LT has four
    uint64_t lo[4] = {0, 0, 0, 0}, mid[4] = {0, 0, 0, 0}, own[4];
    uint32_t hi[4] = {0, 0, 0, 0};
    if (tid == 0) {
        S.mid[0] = 0;
        S.hi[0][0] = S.hi[0][1] = 0;
        S.c[0] = 0;
    }
    if (4 * tid < N) {
        uint32_t sc[WPR];
#pragma unroll
        for (int k = 0; k < WPR; k++) sc[k] = P.wsc[k];
        const uint32_t* q0 = sm + ((4 * tid) >> LM) * SM + wpad((4 * tid) & (M - 1));  // four in one padded run
        coef4(reinterpret_cast<const uint4*>(q0), ODD * SM / 4, sc, lo, mid, hi);
    }
    const int rn = (int)P.rn, top = min(rn, 4 * W::LT);
    limb_sums<W::LT>(S, tid, W::LT, lo, mid, hi, top, own);
    if (tid < W::LT) store_limbs(P.r, 4 * tid, top, own);
    for (int i = top + tid; i < rn; i += W::NT) P.r[i] = 0;  // limbs above the operands' magnitudes
}

// ---------------------------------------------------------------------------
// launches

int64_t word_ctas(int kind, const WordShape& s, int sqr, int64_t rn) {
    const int64_t M = int64_t(1) << s.lm, R = (int64_t)s.odd << s.lj;
    const int64_t cols = M << s.j2, mcols = (int64_t)s.N >> s.j2;
    const int64_t tiles = (rn + UNPACK_TL - 1) / UNPACK_TL;
    switch (kind) {
        case JK_WCOL_FWD: return ((sqr ? 1 : 2) * WPR * cols + WT - 1) / WT;
        case JK_WCOL_REV: return (WPR * cols + WT - 1) / WT;
        case JK_WMID_FWD: return ((sqr ? 1 : 2) * WPR * mcols + WT - 1) / WT;
        case JK_WMID_REV: return (WPR * mcols + WT - 1) / WT;
        case JK_WBLOCK: return (WPR * R * (M / 16) + WT - 1) / WT;
        case JK_WSMALL: return 1;
        case JK_WCARRY: return (tiles + WT - 1) / WT;  // 8 warps of 32 tiles
        default: return tiles;
    }
}

using WKernel = void (*)(const WArgs);
struct WLaunch {
    WKernel fn;
    int threads;
    size_t smem;
};

template <int ODD, int LM>
static WLaunch small_kernel() {
    return WLaunch{k_wsmall<ODD, LM>, WSmall<ODD, LM>::NT, WSmall<ODD, LM>::bytes};
}
template <int ODD, int LJ>
static WLaunch col_kernel(int kind, bool lm12) {
    if (kind == JK_WCOL_FWD) return WLaunch{lm12 ? k_wcol_fwd<ODD, LJ, 12> : k_wcol_fwd<ODD, LJ, 0>, WT, 0};
    return WLaunch{lm12 ? k_wcol_rev<ODD, LJ, 12> : k_wcol_rev<ODD, LJ, 0>, WT, 0};
}
template <int J>
static WLaunch mid_kernel(int kind) {
    return WLaunch{kind == JK_WMID_FWD ? k_wmid<J, true> : k_wmid<J, false>, WT, 0};
}

static WLaunch word_kernel(int kind, int variant) {
    switch (kind) {
        case JK_WUNPACK: return WLaunch{k_wunpack, WT, 0};
        case JK_WCARRY: return WLaunch{k_wcarry, WT, 0};
        case JK_WBLOCK:
            switch (variant) {
                case 12: return WLaunch{k_wblock<12>, WT, 0};
                case 10: return WLaunch{k_wblock<10>, WT, 0};
                case 8: return WLaunch{k_wblock<8>, WT, 0};
                case 6: return WLaunch{k_wblock<6>, WT, 0};
            }
            break;
        case JK_WMID_FWD:
        case JK_WMID_REV:
            switch (variant) {
                case 2: return mid_kernel<2>(kind);
                case 3: return mid_kernel<3>(kind);
                case 4: return mid_kernel<4>(kind);
                case 5: return mid_kernel<5>(kind);
            }
            break;
        case JK_WCOL_FWD:
        case JK_WCOL_REV:
            switch (variant & 0xffff) {
#define NBG_COL(O, J) \
    case (O << 8) | J: return col_kernel<O, J>(kind, variant >> 16);
                NBG_COL(1, 1) NBG_COL(1, 2) NBG_COL(1, 3) NBG_COL(1, 4) NBG_COL(1, 5)
                NBG_COL(3, 0) NBG_COL(3, 1) NBG_COL(3, 2) NBG_COL(3, 3)
                NBG_COL(5, 0) NBG_COL(5, 1) NBG_COL(5, 2)
                NBG_COL(7, 0) NBG_COL(7, 1) NBG_COL(7, 2)
#undef NBG_COL
            }
            break;
        case JK_WSMALL:
            switch (variant) {
#define NBG_SMALL(O, M) \
    case (O << 8) | M: return small_kernel<O, M>();
#define NBG_SMALLS                                                                                          \
    NBG_SMALL(1, 6) NBG_SMALL(1, 7) NBG_SMALL(1, 8) NBG_SMALL(1, 9) NBG_SMALL(1, 10) NBG_SMALL(1, 11)       \
    NBG_SMALL(3, 6) NBG_SMALL(3, 7) NBG_SMALL(3, 8) NBG_SMALL(3, 9) NBG_SMALL(3, 10) NBG_SMALL(5, 6)        \
    NBG_SMALL(5, 7) NBG_SMALL(5, 8) NBG_SMALL(5, 9) NBG_SMALL(7, 6) NBG_SMALL(7, 7) NBG_SMALL(7, 8)
                NBG_SMALLS
#undef NBG_SMALL
            }
            break;
    }
    return WLaunch{nullptr, 0, 0};
}

static cudaError_t small_attributes() {
    cudaError_t e = cudaSuccess;
#define NBG_SMALL(O, M)                                                                                     \
    if (e == cudaSuccess)                                                                                   \
        e = cudaFuncSetAttribute(k_wsmall<O, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,               \
                                 (int)WSmall<O, M>::bytes);
    NBG_SMALLS
#undef NBG_SMALL
    return e;
}

static cudaError_t launch(int kind, int variant, const WArgs& a, int64_t nctas, cudaStream_t st) {
    if (nctas <= 0) return cudaSuccess;
    const WLaunch k = word_kernel(kind, variant);
    if (!k.fn || nctas > 0x7fffffff) return cudaErrorInvalidValue;
    k.fn<<<(unsigned)nctas, k.threads, k.smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_word(int kind, int variant, const DProd* prods, const WSeg* segs, int nseg, const int32_t* plist,
                        int64_t nctas, cudaStream_t st) {
    WArgs a{};
    a.prods = prods;
    a.segs = segs;
    a.plist = plist;
    a.nseg = nseg;
    return launch(kind, variant, a, nctas, st);
}

cudaError_t launch_word_one(int kind, int variant, const DProd& P, int64_t nctas, cudaStream_t st) {
    WArgs a{};
    a.one = P;
    return launch(kind, variant, a, nctas, st);
}

}  // namespace nbg
