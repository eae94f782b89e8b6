// word_kernels.cu — kernels of the word products (word.h): products through
// transforms modulo five or six 30-bit primes, one coefficient per 64-bit limb.
//
//   k_wcol_fwd  limbs -> residues, the radix-`odd` step and the first lj levels
//               of one column's R rows, in registers
//   k_wmid      long transforms: the levels between the first column pass and
//               the blocks, in registers
//   k_wblock    per block of M values: the other levels of a and b, the leaf
//               products, the levels back
//   k_wtail     the first lj levels and the radix-`odd` step backwards, residues
//               -> coefficient (mixed radix), carried limb sums
//   k_wcarry    carries between the runs of limbs
//   k_wsmall    a whole product of at most 3072 coefficients in one CTA
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "word_device.cuh"

namespace nbg {

// ---------------------------------------------------------------------------
// host constants

static uint64_t pw(uint64_t a, uint64_t e, uint64_t p) {
    uint64_t r = 1;
    for (a %= p; e; e >>= 1, a = a * a % p)
        if (e & 1) r = r * a % p;
    return r;
}
static uint64_t inv(uint64_t a, uint64_t p) { return pw(a, p - 2, p); }
// the least primitive root of p (trial division of p - 1)
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
static uint64_t root_of(int set, int i) {
    static const struct Table {
        uint64_t g[WSETS][WPR_MAX];
        Table() {
            for (int t = 0; t < WSETS; t++)
                for (int k = 0; k < word_np(t); k++) g[t][k] = prim_root(WPRIMES[t][k]);
        }
    } t;
    return t.g[set][i];
}
static Tw mk(uint64_t w, uint64_t p) { return Tw{(uint32_t)w, (uint32_t)((w << 32) / p)}; }
static uint32_t mont(uint64_t w, uint64_t p) { return (uint32_t)(((w % p) << 32) % p); }

static cudaError_t small_attributes();

static void fill_set(int set, WConst& h) {
    h = WConst{};
    const uint32_t* P = WPRIMES[set];
    for (int i = 0; i < word_np(set); i++) {
        const uint64_t p = P[i], g = root_of(set, i);
        h.p[i] = (uint32_t)p;
        uint32_t x = 1;
        for (int k = 0; k < 5; k++) x *= 2 - (uint32_t)p * x;  // Newton: p^-1 mod 2^32
        h.pinv[i] = x;
        h.half[i] = (uint32_t)(((uint64_t(1) << 31) + p / 2) / p * p);
        if ((p - 1) % 3 == 0) h.r3[i] = mk(pw(g, (p - 1) / 3, p), p);
        if (set == 0) {  // radix 5 and 7
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
        }
        uint64_t Wi = 1;
        for (int t = 0; t < i; t++) Wi = Wi * (P[t] % p) % p;
        const uint64_t iw = inv(Wi, p);
        uint64_t Wj = 1;
        for (int j = 0; j < i; j++) {
            h.gar[i][j] = mont((p - Wj * iw % p) % p, p);
            Wj = Wj * (P[j] % p) % p;
        }
        uint32_t w[WPR_MAX] = {1};
        for (int t = 0; t < i; t++) {
            uint64_t cy = 0;
            for (int k = 0; k < WPR_MAX; k++) {
                cy += (uint64_t)w[k] * P[t];
                w[k] = (uint32_t)cy;
                cy >>= 32;
            }
        }
        for (int k = 0; k < WPR_MAX; k++) h.wt[i][k] = w[k];
    }
}

void word_fill_const(WConst h[WSETS]) {
    for (int t = 0; t < WSETS; t++) fill_set(t, h[t]);
}

cudaError_t word_init() {
    WConst h[WSETS];
    word_fill_const(h);
    cudaError_t e = small_attributes();
    return e == cudaSuccess ? cudaMemcpyToSymbol(c_w, h, sizeof h) : e;
}

void word_scales(const WordShape& s, uint32_t* out) {
    // 2^64 (the operands' packing) * 2^32 (pointwise) * 2^32 (unpack's reduction) / (odd * 2^levels * W_i)
    constexpr int LEV = 26;
    static const struct Table {
        uint32_t v[WSETS][8][LEV][WPR_MAX];
        Table() {
            for (int set = 0; set < WSETS; set++)
                for (int i = 0; i < word_np(set); i++) {
                    const uint64_t p = WPRIMES[set][i], r = (uint64_t(1) << 32) % p, r2 = r * r % p;
                    uint64_t W = 1;
                    for (int j = 0; j < i; j++) W = W * (WPRIMES[set][j] % p) % p;
                    for (int odd = 1; odd < 8; odd += 2)
                        for (int lev = 0; lev < LEV; lev++)
                            v[set][odd][lev][i] = (uint32_t)(r2 * r2 % p * inv(odd * pw(2, (uint64_t)lev, p) % p * W % p, p) % p);
                }
        }
    } t;
    for (int i = 0; i < word_np(s.set); i++) out[i] = t.v[s.set][s.odd][s.lj + s.lm - 2][i];
}

// The split of the rows above the blocks: one column pass up to 32 rows (its
// values fit a thread's registers), else the two passes whose larger row count
// is least.
static bool row_split(int odd, int lj, int& j2) {
    j2 = 0;
    const int64_t R = (int64_t)odd << lj;
    if (R <= 32) return R >= 2;
    int64_t best = INT64_MAX;
    for (int j = 3; j <= 5 && j <= lj; j++) {
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
                    v.push_back(WordShape{(int32_t)N, odd, 0, 0, k, true, 0});
                    continue;
                }
                for (int lm : {12, 10, 8}) {
                    int j2;
                    if (k < lm || !row_split(odd, k - lm, j2)) continue;
                    v.push_back(WordShape{(int32_t)N, odd, k - lm, j2, lm, false, 0});
                    break;
                }
            }
        // six primes: 32 (24) first rows, then a middle pass of up to 256
        for (int k = 22; k <= 25; k++) v.push_back(WordShape{1 << k, 1, k - 12, k - 17, 12, false, 2});
        for (int k = 21; k <= 23; k++) v.push_back(WordShape{3 << k, 3, k - 12, k - 15, 12, false, 1});
        std::sort(v.begin(), v.end(), [](const WordShape& x, const WordShape& y) { return x.N < y.N; });
        return v;
    }();
    return list;
}

bool word_shape(int64_t nconv, WordShape& s, bool coarse) {
    static const std::vector<WordShape> few = [] {
        std::vector<WordShape> v;
        for (const WordShape& x : shape_list())
            if (x.odd <= 3 || x.N > 131072) v.push_back(x);
        return v;
    }();
    const std::vector<WordShape>& v = coarse ? few : shape_list();
    const auto it = std::lower_bound(v.begin(), v.end(), nconv,
                                     [](const WordShape& x, int64_t n) { return x.N < n; });
    if (it == v.end()) return false;
    s = *it;
    return true;
}

// ---------------------------------------------------------------------------
// tables

size_t word_table_bytes(int set, int odd, int L) { return sizeof(Tw) * ((size_t)word_np(set) * odd << L); }

__device__ uint32_t pw_dev(uint32_t a, uint32_t e, uint32_t p) {
    uint64_t r = 1, b = a;
    for (; e; e >>= 1, b = b * b % p)
        if (e & 1) r = r * b % p;
    return (uint32_t)r;
}

struct WRoots {
    uint32_t g[WPR_MAX];
};
constexpr int PWB = 15;  // powers g^e through g^(e mod 2^15) and g^(2^15 (e / 2^15))
// pwt[i][0][x] = g_i^x, pwt[i][1][x] = g_i^(2^15 x), x < 2^15
__global__ void k_wpowers(uint32_t* __restrict__ pwt, int set, int np, WRoots g) {
    const int total = np << (PWB + 1);
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < total; x += gridDim.x * blockDim.x) {
        const int i = x >> (PWB + 1);
        const uint32_t e = (uint32_t)x & ((1u << PWB) - 1);
        pwt[x] = pw_dev(g.g[i], (x >> PWB) & 1 ? e << PWB : e, c_w[set].p[i]);
    }
}
// entry h = 2^l + n of (prime i, block j): e((j + odd * bitrev_l(n)) / (odd * 2^(l+1))) and its inverse
__global__ void k_wtable(Tw* __restrict__ fwd, Tw* __restrict__ bwd, const uint32_t* __restrict__ pwt, int set, int np,
                         int odd, int L) {
    const int64_t total = (int64_t)np * odd << L;
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < total; x += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t h = (uint32_t)(x & ((int64_t(1) << L) - 1));
        const int ij = (int)(x >> L), i = ij / odd, j = ij - i * odd;
        const uint32_t p = c_w[set].p[i];
        uint32_t e = 0;
        if (h) {
            const int l = 31 - __clz(h);
            const uint32_t n = h - (1u << l);
            const uint32_t brv = l ? __brev(n) >> (32 - l) : 0;
            e = (p - 1) / ((uint32_t)odd << (l + 1)) * ((uint32_t)j + (uint32_t)odd * brv);
        }
        const uint32_t* t = pwt + ((size_t)i << (PWB + 1));
        auto power = [&](uint32_t q) {
            return (uint32_t)((uint64_t)t[q & ((1u << PWB) - 1)] * t[(1u << PWB) + (q >> PWB)] % p);
        };
        const uint32_t w = power(e), v = e ? power(p - 1 - e) : 1u;
        fwd[x] = Tw{w, (uint32_t)(((uint64_t)w << 32) / p)};
        bwd[x] = Tw{v, (uint32_t)(((uint64_t)v << 32) / p)};
    }
}

cudaError_t word_build_tables(int set, int odd, int L, void* fwd, void* bwd, cudaStream_t st) {
    WRoots g{};
    for (int i = 0; i < word_np(set); i++) g.g[i] = (uint32_t)root_of(set, i);
    uint32_t* pwt = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&pwt, sizeof(uint32_t) * ((size_t)word_np(set) << (PWB + 1)), st);
    if (e != cudaSuccess) return e;
    k_wpowers<<<148 * 4, 256, 0, st>>>(pwt, set, word_np(set), g);
    k_wtable<<<148 * 8, 256, 0, st>>>((Tw*)fwd, (Tw*)bwd, pwt, set, word_np(set), odd, L);
    e = cudaGetLastError();
    const cudaError_t f = cudaFreeAsync(pwt, st);
    return e != cudaSuccess ? e : f;
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

// A kernel of a single product may be on the GPU before the one it follows has
// finished (programmatic launch): nothing that one wrote, and nothing it may
// still read, is touched before this, and what it wrote (operands, which may be
// the result before, and residues) is not read by __ldg: the read-only path wants
// data that nothing writes while this kernel is on the GPU.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A pointer whose loads stay below this point (a wait or a barrier before it): the
// compiler may take the load intrinsics for functions of the address alone.
template <class T>
__device__ __forceinline__ T* from_here(T* p) {
    asm volatile("" : "+l"(p) : : "memory");
    return p;
}
// The next kernel's CTAs may come once every CTA is here: near the end, so that
// they spread over the SMs as those empty (from the start of the kernel, the
// blocks of a 65536 x 65521-limb product piled up: 31 -> 38 us per call).
__device__ __forceinline__ void let_next() { asm volatile("griddepcontrol.launch_dependents;"); }

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

// LM: log2 of the column count when the blocks are 4096 values (row strides are
// then immediate offsets), 0: read from the product.  Rows past the operand are
// not packed, and when they are its upper half (odd = 1, a half-length operand,
// which one of two always is) the first level is a copy.  Bound by the multiply
// pipe (66% busy) and, in long batches, memory: 100 squares of 65536 limbs 0.080 ms,
// 3.9 TB/s of operands and residues.  64 registers: at 5 CTAs per SM the columns
// spill (10,000 mixed products 13.05 -> 13.28 ms).
template <int ODD, int LJ, int LM, int SET>
__global__ void __launch_bounds__(WT, 4) k_wcol_fwd(const __grid_constant__ WArgs A) {
    constexpr int R = ODD << LJ, NP = word_np(SET);
    int local;
    const DProd& P = wjob(A, local);
    wait_previous();
    const int lm = LM ? LM : P.wlm + P.wj2;
    const int id = local * WT + (int)threadIdx.x;
    const int c = id & ((1 << lm) - 1);
    int pi = id >> lm;  // operand-major: a's primes, then b's
    const bool isb = pi >= NP;
    if (isb) pi -= NP;
    if (A.nseg == 0 && id < 2 && P.ntl <= WORD_FUSED_TILES) P.agg[P.ntl + id] = 0;  // k_wtail's counts of CTAs and of carries
    if (pi >= NP || (isb && P.sqr)) return;
    const int n = (int)(isb ? P.ncb : P.nca);
    const int rows = (n + (1 << lm) - 1) >> lm;
    const uint64_t* src = from_here(isb ? P.b : P.a) + c;
    uint32_t* __restrict__ dst = (isb ? P.wb : P.wa) + (size_t)pi * (size_t)P.wN + c;
    const uint32_t p = c_w[SET].p[pi];
    const Tw* tab = (const Tw*)P.wtf + (((size_t)pi * ODD) << P.wL);
    uint32_t x[R];
    auto rowsin = [&](auto r0c, auto r1c) {
        constexpr int r0 = decltype(r0c)::value, r1 = decltype(r1c)::value;
        uint64_t v[r1 - r0];
#pragma unroll
        for (int r = r0; r < r1; r++) v[r - r0] = c + (r << lm) < n ? __ldcg(src + ((size_t)r << lm)) : 0ull;
#pragma unroll
        for (int r = r0; r < r1; r++) x[r] = r < rows ? wpack<(ODD > 1), SET>(v[r - r0], pi, p) : 0u;
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
        dft_odd<ODD, LJ, SET>(x, pi, p);
#pragma unroll
        for (int j = 0; j < ODD; j++) wd::tree_fwd<LJ, 1>(x + (j << LJ), tab + ((size_t)j << P.wL), 1u, p);
    }
#pragma unroll
    for (int r = 0; r < R; r++) dst[(size_t)r << lm] = x[r];  // no let_next: it cost the batches' passes 4%
}

// A middle pass works on segments of 2^j rows (2^12 apart: more than 32 rows only
// stand above blocks of 4096), each the subtree of a node, in place; all columns of
// a segment share their constants.  A segment's first word, constants and node:
struct MidJob {
    uint32_t* x;
    const Tw* tab;
    uint32_t node, p;
    bool live;
};
// item: (operand, prime, segment) in that order; j levels, R1 segments per prime
template <bool FWD, int SET>
__device__ __forceinline__ MidJob mid_job(const DProd& P, int item, int j) {
    constexpr int NP = word_np(SET);
    const int j1 = P.wlj - j, R1 = P.wodd << j1;
    const int op = item / R1, seg = item - op * R1;
    const bool isb = op >= NP;
    const int pi = isb ? op - NP : op;
    MidJob J;
    J.live = pi < NP && !(isb && (!FWD || P.sqr));
    if (!J.live) return J;
    J.x = (isb ? P.wb : P.wa) + (size_t)pi * (size_t)P.wN + ((size_t)seg << (12 + j));
    J.tab = (const Tw*)(FWD ? P.wtf : P.wti) + (((size_t)pi * P.wodd + (seg >> j1)) << P.wL);
    J.node = (1u << j1) + (uint32_t)(seg & ((1 << j1) - 1));
    J.p = c_w[SET].p[pi];
    return J;
}

// The 2^J rows of one column, in registers.
template <int J, bool FWD, int SET>
__global__ void __launch_bounds__(WT) k_wmid(const __grid_constant__ WArgs A) {
    constexpr int lm = 12;
    int local;
    const DProd& P = wjob(A, local);
    wait_previous();
    const int id = local * WT + (int)threadIdx.x;
    const MidJob M = mid_job<FWD, SET>(P, id >> lm, J);
    if (!M.live) return;
    uint32_t* __restrict__ x0 = M.x + (id & ((1 << lm) - 1));
    uint32_t x[1 << J];
#pragma unroll
    for (int r = 0; r < (1 << J); r++) x[r] = x0[(size_t)r << lm];
    if (FWD) wd::tree_fwd<J, 1>(x, M.tab, M.node, M.p);
    else wd::tree_rev<J, 1>(x, M.tab, M.node, M.p);
    let_next();
#pragma unroll
    for (int r = 0; r < (1 << J); r++) x0[(size_t)r << lm] = x[r];
}

// 64 to 256 rows: tiles of 2^J rows by 2^(12-J) columns (64 to 256 bytes per
// row), four levels in registers, a turn through shared memory, the other J - 4
// levels.  One pass over memory instead of two: at these lengths the register
// passes run at the memory's rate (2^24-limb square: 1.6 GB and 0.40 ms, 4.0 TB/s).
// Wider tiles (32 columns, 512 threads) took 0.43 ms.
template <int J, bool FWD, int SET>
__global__ void __launch_bounds__(WT, 4) k_wmid_sm(const __grid_constant__ WArgs A) {
    constexpr int lm = 12, CW = 1 << (12 - J), K = J - 4, NG = 1 << (4 - K);  // NG groups of 2^K values per thread
    __shared__ uint32_t s[4096 + 16 * 16];
    auto at = [](int i) { return i + ((i >> 8) << 4); };  // rows of 16 words: the two half-warps in distinct banks
    int local;
    const DProd& P = wjob(A, local);
    wait_previous();
    const MidJob M = mid_job<FWD, SET>(P, local >> J, J);  // 2^J tiles per segment
    if (!M.live) return;                                    // the whole CTA
    const int tid = (int)threadIdx.x, c = tid & (CW - 1), g = tid >> (12 - J);
    uint32_t* __restrict__ x0 = M.x + (local & ((1 << J) - 1)) * CW + c;
    uint32_t x[16];
    auto outer_io = [&](bool st) {  // rows g + e * 2^K
#pragma unroll
        for (int e = 0; e < 16; e++) {
            uint32_t* w = x0 + ((size_t)(g + (e << K)) << lm);
            if (st) *w = x[e];
            else x[e] = *w;
        }
    };
    auto inner_io = [&](bool st) {  // group q: sub-block b = g + q * (16 / NG), rows b * 2^K + e
#pragma unroll
        for (int q = 0; q < NG; q++)
#pragma unroll
            for (int e = 0; e < (1 << K); e++) {
                uint32_t* w = x0 + ((size_t)(((g + q * (16 / NG)) << K) + e) << lm);
                if (st) *w = x[(q << K) + e];
                else x[(q << K) + e] = *w;
            }
    };
    auto outer_sm = [&](bool st) {
#pragma unroll
        for (int e = 0; e < 16; e++) {
            uint32_t& w = s[at((g + (e << K)) * CW + c)];
            if (st) w = x[e];
            else x[e] = w;
        }
    };
    auto inner_sm = [&](bool st) {
#pragma unroll
        for (int q = 0; q < NG; q++)
#pragma unroll
            for (int e = 0; e < (1 << K); e++) {
                uint32_t& w = s[at((((g + q * (16 / NG)) << K) + e) * CW + c)];
                if (st) w = x[(q << K) + e];
                else x[(q << K) + e] = w;
            }
    };
    if (FWD) {
        outer_io(false);
        wd::tree_fwd<4, 1>(x, M.tab, M.node, M.p);
        outer_sm(true);
        __syncthreads();
        inner_sm(false);
#pragma unroll
        for (int q = 0; q < NG; q++)
            wd::tree_fwd<K, 1>(x + (q << K), M.tab, (M.node << 4) + (uint32_t)(g + q * (16 / NG)), M.p);
        let_next();
        inner_io(true);
    } else {
        inner_io(false);
#pragma unroll
        for (int q = 0; q < NG; q++)
            wd::tree_rev<K, 1>(x + (q << K), M.tab, (M.node << 4) + (uint32_t)(g + q * (16 / NG)), M.p);
        inner_sm(true);
        __syncthreads();
        outer_sm(false);
        wd::tree_rev<4, 1>(x, M.tab, M.node, M.p);
        let_next();
        outer_io(true);
    }
}

// ---------------------------------------------------------------------------
// blocks

template <int LM>
struct WBlockSmem {
    static constexpr int PER = WT >> (LM - 4), SM = wwords(1 << LM);  // blocks per CTA, words of one
    static constexpr int words = PER * 2 * SM;
};
template <int LM, int SET>
__device__ __forceinline__ void wblock(const DProd& P, int local, uint32_t* smw) {
    constexpr int T = 1 << (LM - 4), PER = WBlockSmem<LM>::PER, SM = WBlockSmem<LM>::SM;
    constexpr int J1 = WSplit<LM>::J1;
    uint32_t(*sm)[2][SM] = reinterpret_cast<uint32_t(*)[2][SM]>(smw);
    const int g = (int)threadIdx.x / T, t = (int)threadIdx.x & (T - 1);
    const int R = P.wodd << P.wlj;
    const int blk = local * PER + g;  // prime-major, then block
    const bool live = blk < word_np(SET) * R;
    const int pi = live ? blk / R : 0, row = live ? blk - pi * R : 0;
    const int j = row >> P.wlj;
    const uint32_t h0 = (1u << P.wlj) + (uint32_t)(row & ((1 << P.wlj) - 1));
    const uint32_t p = c_w[SET].p[pi], pinv = c_w[SET].pinv[pi];
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
    let_next();
    if (live) {
#pragma unroll
        for (int k = 0; k < 16; k++)
            xa[wpos<LM, LM, J1>(t, k >> J1) + ((k & ((1 << J1) - 1)) << (LM - J1))] = a[k];
    }
}

// Both operands' 16 values per thread share each level's constants.  Bound by the
// multiply pipe: 60% of its measured rate over 10,000 mixed products, 6.08 ms.
// 64 registers for four CTAs per SM: three (80 registers) took 6.38 ms against
// 6.12 then, two (96) 8% more than three.  One launch serves every block size of set 0.
template <int SET>
__global__ void __launch_bounds__(WT, 4) k_wblock(const __grid_constant__ WArgs A) {
    __shared__ __align__(16) uint32_t sm[WBlockSmem<12>::words];
    static_assert(WBlockSmem<10>::words <= WBlockSmem<12>::words && WBlockSmem<8>::words <= WBlockSmem<12>::words, "");
    int local;
    const DProd& P = wjob(A, local);
    wait_previous();
    if (SET || P.wlm == 12) {
        wblock<12, SET>(P, local, sm);
    } else if constexpr (SET == 0) {
        if (P.wlm == 10) wblock<10, SET>(P, local, sm);
        else wblock<8, SET>(P, local, sm);
    }
}

// ---------------------------------------------------------------------------
// carries between a product's tiles (runs of k_wtail, tiles of the FP64 unpack;
// P.tl limbs each)

// A warp's 32 tiles, one per lane (k: this lane's, a: its state, carry: whether
// one comes in).  It stops at the first limb unless that is all ones.  A tile that
// propagates is all ones and becomes zeros, unread, runs of such tiles together;
// in the others the warp finds the end of the run.  Only r is written, each tile
// by one warp.  (Reads go to L2: other CTAs of a running kernel may have written
// what is read.)  Bound by the stores; walking every tile, 32 limbs at a time, and
// looking down 32 tiles at a time took 4096-limb all-ones squares 58 us per call,
// 65536 210 and 2^22 1175, now 17, 39 and 673 (uniform limbs 15, 22, 640).
__device__ __forceinline__ void carry_fix(uint64_t* r, int64_t tl, int64_t rn, int64_t k, uint32_t a, bool carry) {
    const int lane = (int)threadIdx.x & 31;
    const int64_t kw = k - lane;
    const bool ones = carry && (a & 2u);
    bool walk = false;
    if (carry && !ones) {
        uint64_t* w = r + k * tl;
        const uint64_t v = __ldcg(w);
        if (v != ~0ULL) *w = v + 1;
        else walk = true;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, ones); m;) {
        const int s = __ffs(m) - 1, up = __ffs(~(m >> s));
        const int len = up ? up - 1 : 32;  // tiles s .. s + len - 1
        const int64_t b1 = (kw + s + len) * tl;
        for (int64_t w = (kw + s) * tl + lane; w < b1; w += 32) r[w] = 0;
        m &= len == 32 ? 0u : ~(((1u << len) - 1) << s);
    }
    for (unsigned m = __ballot_sync(0xffffffffu, walk); m; m &= m - 1) {
        const int64_t b0 = (kw + __ffs(m) - 1) * tl, b1 = min(b0 + (int64_t)tl, rn);
        bool end = false;
        for (int64_t w = b0 + lane; !end && w - lane < b1; w += 128) {
            uint64_t v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = w + 32 * q < b1 ? __ldcg(r + w + 32 * q) : 0ULL;  // past the tile: ends the run
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (end) break;
                const unsigned stop = __ballot_sync(0xffffffffu, v[q] != ~0ULL);
                const int e = stop ? __ffs(stop) - 1 : 32;
                if (lane < e) r[w + 32 * q] = 0;
                else if (lane == e && w + 32 * q < b1) r[w + 32 * q] = v[q] + 1;
                end = stop != 0;
            }
        }
    }
}

// Every carry of a product of few tiles, by one CTA.
template <int NT>
__device__ __forceinline__ void carry_all(const DProd& P, uint32_t* wagg) {
    uint64_t* const r = from_here(P.r);
    const uint32_t* const agg = from_here(P.agg);
    uint32_t cin = 0;
    for (int64_t k0 = 0; k0 < P.ntl; k0 += NT) {
        const int64_t k = k0 + (int)threadIdx.x;
        const uint32_t a = k < P.ntl ? __ldcg(agg + k) : 0u;
        __syncthreads();  // wagg's previous readers
        uint32_t total;
        const uint32_t st = cta_state(a, wagg, total);
        carry_fix(r, P.tl, P.rn, k, a, k < P.ntl && (gp_join(cin, st) & 1u));
        cin = gp_join(cin, total) & 1u;
    }
}

// The carry into tile k0: of the last lower tile that does not propagate, almost
// always among the 32 before, which every warp looks at; past those the CTA
// goes down 16 tiles per thread at a time.
__device__ __forceinline__ uint32_t carry_below(const uint32_t* agg, int64_t k0, uint32_t* found) {
    const int lane = (int)threadIdx.x & 31;
    {
        const uint32_t a = k0 > lane ? __ldcg(agg + (k0 - 1 - lane)) : 0u;
        const unsigned stop = __ballot_sync(0xffffffffu, !(a & 2u));
        if (stop) return __shfl_sync(0xffffffffu, a, __ffs(stop) - 1) & 1u;
    }
    for (int64_t top = k0 - 33; top >= 0; top -= 16 * WT) {  // the whole CTA: all warps saw the same 32
        uint32_t best = 0;  // greatest (tile, generates) that does not propagate, plus one
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int64_t i = top - (j * WT + (int)threadIdx.x);
            const uint32_t a = i >= 0 ? __ldcg(agg + i) : 2u;
            if (!(a & 2u)) best = max(best, ((uint32_t)i << 1 | (a & 1u)) + 1u);
        }
        best = __reduce_max_sync(0xffffffffu, best);
        if (threadIdx.x == 0) *found = 0;
        __syncthreads();
        if (lane == 0 && best) atomicMax(found, best);
        __syncthreads();
        best = *found;
        __syncthreads();
        if (best) return (best - 1) & 1u;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// tail: the first levels backwards, coefficients, carried limbs

// A CTA has CW adjacent columns of all R rows and every prime.  Its threads run
// the columns backwards into shared memory, then a warp (or half of one) takes
// a row's run of CW consecutive coefficients, four per lane, to limbs.  As two
// kernels the residues made one more trip through memory (40 of about 70 bytes
// per coefficient); the arithmetic of the second half hides the loads of
// another CTA's first half.  The three columns left of the tile are run too:
// their coefficients reach into its first limbs (in column 0, from the row above).
// Bound by the multiply pipe (65% busy; 100 squares of 65536 limbs: 0.178 ms).
// Several runs per CTA left a 4096-limb square four CTAs, 19 -> 27 us.
template <int ODD, int LJ, int SET>
struct WTail {
    static constexpr int R = ODD << LJ, NP = word_np(SET);
    static constexpr int RUN = word_run(R);               // limbs of a run: a lane has four
    static constexpr int CW = RUN, W = CW + 4;            // columns: one run; words of a row (4 left of the tile)
    // a warp per run up to 8 rows, then two runs each; 12 half-warps for the short runs
    static constexpr int NT = RUN == 64 ? 192 : R <= 8 ? 32 * R : 32 * ((R + 1) / 2);
    static constexpr int LANES = RUN / 4;                 // lanes of a run
    static constexpr size_t halo_bytes = ((size_t)R * 3 * 24 + 15) / 16 * 16;  // lo, mid, hi of three coefficients per row
    static constexpr size_t bytes = halo_bytes + sizeof(uint32_t) * NP * R * W;
};

// LM as in k_wcol_fwd.
template <int ODD, int LJ, int LM, int SET>
__global__ void __launch_bounds__(WTail<ODD, LJ, SET>::NT, 1024 / WTail<ODD, LJ, SET>::NT)
    k_wtail(const __grid_constant__ WArgs A) {
    using T = WTail<ODD, LJ, SET>;
    constexpr int R = T::R, NP = T::NP, W = T::W, LANES = T::LANES;
    extern __shared__ __align__(16) unsigned char dyn[];
    struct Halo {
        uint64_t lo, mid, hi;
    };
    Halo* const halo = reinterpret_cast<Halo*>(dyn);
    uint32_t* const sm = reinterpret_cast<uint32_t*>(dyn + T::halo_bytes);
    int local;
    const DProd& P = wjob(A, local);
    wait_previous();
    const int tid = (int)threadIdx.x;
    const int lm = LM ? LM : P.wlm + P.wj2, cols = 1 << lm;
    const int N = P.wN, c0 = local * T::CW;
    // columns c0 - 3 .. c0 + CW - 1 of every prime
    for (int q = tid; q < NP * (T::CW + 3); q += T::NT) {
        const int pi = q / (T::CW + 3), cc = q - pi * (T::CW + 3) - 3;
        const bool up = c0 + cc < 0;  // left of column 0: the ends of the rows above
        const uint32_t* src = from_here(P.wa) + (size_t)pi * (size_t)N + (c0 + cc + (up ? cols : 0));
        const uint32_t p = c_w[SET].p[pi];
        uint32_t x[R];
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = __ldcg(src + ((size_t)r << lm));
        const Tw* tab = (const Tw*)P.wti + (((size_t)pi * ODD) << P.wL);
#pragma unroll
        for (int j = 0; j < ODD; j++) wd::tree_rev<LJ, 1>(x + (j << LJ), tab + ((size_t)j << P.wL), 1u, p);
        dft_odd<ODD, LJ, SET>(x, pi, p);
        // the inverse step is the forward one with output i at -i mod odd
        uint32_t* d = sm + pi * R * W + 4 + cc;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int row = (((ODD - (r >> LJ)) % ODD) << LJ) + (r & ((1 << LJ) - 1));
            if (!up) d[row * W] = x[r];
            else if (row + 1 < R) d[(row + 1) * W] = x[r];
            else d[0] = 0;  // row 0 has nothing below it
        }
    }
    __syncthreads();
    uint32_t sc[NP];
#pragma unroll
    for (int k = 0; k < NP; k++) sc[k] = P.wsc[k];
    if (tid < 3 * R) {  // coefficients -1, -2, -3 of each row
        const int row = tid / 3, j = tid - 3 * row;
        uint32_t r[NP], hi;
#pragma unroll
        for (int k = 0; k < NP; k++) r[k] = sm[(k * R + row) * W + 3 - j];
        uint64_t lo, mid;
        coef_words<SET>(r, sc, lo, mid, hi);
        halo[tid] = Halo{lo, mid, hi};
    }
    __syncthreads();
    const int lane = tid & (LANES - 1);
    const int64_t rn = P.rn;
    const bool fused = A.nseg == 0 && P.ntl <= WORD_FUSED_TILES;
    for (int row = tid / LANES; row < R; row += T::NT / LANES) {
        // what reaches lane 0's first limbs: mid and hi words of the quad below and its last carry
        uint64_t in_mid = halo[3 * row].mid;
        uint32_t in_hi3 = (uint32_t)halo[3 * row].hi, in_hi2 = (uint32_t)halo[3 * row + 1].hi, in_c;
        {
            const uint64_t m = halo[3 * row + 1].mid, h = halo[3 * row + 2].hi;
            uint64_t s = halo[3 * row].lo + m;
            in_c = s < m;
            s += h;
            in_c += s < h;
        }
        uint64_t lo[4], mid[4], own[4];
        uint32_t hi[4], cy[4];
        coef4<SET>(reinterpret_cast<const uint4*>(sm + row * W + 4 + 4 * lane), R * W / 4, sc, lo, mid,
                   hi);
        auto sum = [&](int q, uint64_t m, uint32_t h) {
            uint64_t s = lo[q] + m;
            uint32_t c = s < m;
            s += h;
            c += s < h;
            own[q] = s;
            cy[q] = c;
        };
        sum(2, mid[1], hi[0]);
        sum(3, mid[2], hi[1]);
        uint64_t pm = __shfl_up_sync(0xffffffffu, mid[3], 1, LANES);
        uint32_t ph2 = __shfl_up_sync(0xffffffffu, hi[2], 1, LANES), ph3 = __shfl_up_sync(0xffffffffu, hi[3], 1, LANES);
        uint32_t pc = __shfl_up_sync(0xffffffffu, cy[3], 1, LANES);
        if (lane == 0) {
            pm = in_mid;
            ph2 = in_hi2;
            ph3 = in_hi3;
            pc = in_c;
        }
        in_mid = __shfl_sync(0xffffffffu, mid[3], LANES - 1, LANES);
        in_hi2 = __shfl_sync(0xffffffffu, hi[2], LANES - 1, LANES);
        in_hi3 = __shfl_sync(0xffffffffu, hi[3], LANES - 1, LANES);
        in_c = __shfl_sync(0xffffffffu, cy[3], LANES - 1, LANES);
        sum(0, pm, ph2);
        sum(1, mid[0], ph3);
        const int64_t wr = (int64_t)row * cols + c0, wt = wr + 4 * lane;
        uint32_t k = pc, gen = 0, prop = 1;  // carry of the sum below; carry of adding it
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint64_t s = own[q] + k + gen;  // k + gen <= 3
            gen = s < (uint64_t)(k + gen);
            own[q] = s;
            k = cy[q];
            prop &= (wt + q < rn && s == ~0ULL) ? 1u : 0u;
        }
        uint32_t incl = gen | (prop << 1);
#pragma unroll
        for (int off = 1; off < LANES; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off, LANES);
            if (lane >= off) incl = gp_join(o, incl);
        }
        const uint32_t below = __shfl_up_sync(0xffffffffu, incl, 1, LANES);
        add_carry(own, lane ? below & 1u : 0u);  // carry into the run taken as 0, added later
        store_limbs(P.r, wt, rn, own);
        if (lane == LANES - 1 && wr < rn) {
            P.agg[wr / T::RUN] = incl;
            if (fused && (incl & 1u)) atomicAdd(P.agg + P.ntl + 1, 1u);
            if (wr + T::RUN == N && rn > N) {  // limb N: the last coefficients' upper words
                P.r[N] = in_mid + in_hi2 + in_c;
                P.agg[N / T::RUN] = 0;
            }
        }
    }
    let_next();
    // limbs above the operands' magnitudes
    for (int64_t i = (int64_t)N + 1 + (int64_t)local * T::NT + tid; i < rn; i += (int64_t)(cols / T::CW) * T::NT) P.r[i] = 0;
    if (!fused) return;
    // one product of few runs: its last CTA carries between them instead of another
    // launch (in batches the fences cost 10% of the pass, so k_wcarry does it
    // there), and only if some run carries out at all (a limb sum within 3 of
    // 2^64, so hardly ever but for operands made of ones or zeros)
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        last = atomicAdd(P.agg + P.ntl, 1u) == (uint32_t)(cols / T::CW - 1);
        __threadfence();
    }
    __syncthreads();
    __shared__ uint32_t wagg[T::NT / 32];
    if (last && __ldcg(from_here(P.agg) + P.ntl + 1) != 0) carry_all<T::NT>(P, wagg);
}

// Tiles of a warp of k_wcarry: one per lane, but 2048 limbs of the FP64 passes' long
// tiles, so that many warps zero a run of them (600,000-limb all-ones square there,
// replayed: 130 us with 32 tiles each, 101 so).
__host__ __device__ constexpr int carry_per_warp(int tl) { return tl > 128 ? 2048 / tl : 32; }

// (Registers for eight CTAs per SM: a batch has a short one per product.)
__global__ void __launch_bounds__(WT, 8) k_wcarry(const __grid_constant__ WArgs A) {
    int local;
    const DProd& P = wjob(A, local);
    wait_previous();
    __shared__ uint32_t wagg[WT / 32], found;
    const int per = carry_per_warp((int)P.tl), lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
    const bool few = P.ntl <= per;  // most products of a batch: one warp has all tiles
    if (few && wid) return;
    const int64_t k0 = (int64_t)local * (WT / 32 * per), k = k0 + wid * per + lane;  // a lane's tile
    const bool in = lane < per && k < P.ntl;
    uint64_t* const r = from_here(P.r);
    const uint32_t* const agg = from_here(P.agg);
    const uint32_t a = in ? __ldcg(agg + k) : 2u;  // others pass a carry on
    if (few) {
        const uint32_t below = warp_below(warp_scan(a));
        carry_fix(r, P.tl, P.rn, k, a, in && (below & 1u));
        return;
    }
    uint32_t total;
    const uint32_t cin = carry_below(agg, k0, &found), st = cta_state(a, wagg, total);
    carry_fix(r, P.tl, P.rn, k, a, in && (gp_join(cin, st) & 1u));
}

// ---------------------------------------------------------------------------
// small products: one CTA does all of it; the transforms, the residues and the
// limbs stay on chip.  Bound by the latency of one CTA's rounds (177 x 152 limbs: 7 us
// per call in sequence, 5 of them the launch itself; FP64 passes 56 us).

template <int ODD, int LM>
__global__ void __launch_bounds__(WSmall<ODD, LM>::NT, WSmall<ODD, LM>::NT > 320 ? 1 : 640 / WSmall<ODD, LM>::NT)
    k_wsmall(const __grid_constant__ WArgs A) {
    using W = WSmall<ODD, LM>;
    static_assert(W::LT <= W::NT && W::NT <= 1024, "limb threads");
    extern __shared__ __align__(16) unsigned char dyn[];
    LimbShared<W::LT>& S = *reinterpret_cast<LimbShared<W::LT>*>(dyn);
    uint32_t* sm = reinterpret_cast<uint32_t*>(dyn + W::limb_bytes);
    int local;
    const DProd& P = wjob(A, local);
    const int tid = (int)threadIdx.x;
    const SmallThread<ODD, LM> th(sm, P.wtf, P.wti, P.wL);
    wait_previous();
    uint32_t x[32];  // a's 16 values, then b's
    // in L1 for the other primes' threads (from pinned host memory, 700 x 630 limbs
    // 36 us per call, by __ldcg 38; plain loads are not moved up: 43)
    const uint64_t *pa = from_here(P.a), *pb = from_here(P.b);
    th.load(x, th.sp, (int)P.nca, [&](int i) { return __ldca(pa + i); });
    if (!P.sqr) th.load(x + 16, th.sp + W::OPW, (int)P.ncb, [&](int i) { return __ldca(pb + i); });
    if (ODD > 1) {
        __syncthreads();
        th.fetch(x, 0);
        if (!P.sqr) th.fetch(x + 16, 1);
    }
    if (!P.sqr) th.template down<2>(x);
    else th.template down<1>(x);
    th.point(x, P.sqr);
    th.up(x);
    // coefficients and limbs: thread tid < LT has four
    uint64_t lo[4], mid[4], own[4];
    uint32_t hi[4];
    if (tid == 0) {
        S.mid[0] = 0;
        S.hi[0][0] = S.hi[0][1] = 0;
        S.c[0] = 0;
    }
    SmallThread<ODD, LM>::coefs(sm, P.wsc, lo, mid, hi);
    const int rn = (int)P.rn, top = min(rn, 4 * W::LT);
    limb_sums<W::LT>(S, tid, W::LT, lo, mid, hi, top, own);
    let_next();
    if (tid < W::LT) store_limbs(P.r, 4 * tid, top, own);
    for (int i = top + tid; i < rn; i += W::NT) P.r[i] = 0;  // limbs above the operands' magnitudes
}

// ---------------------------------------------------------------------------
// launches

int64_t word_ctas(int kind, const WordShape& s, int sqr, int64_t ntl) {
    const int64_t M = int64_t(1) << s.lm, R = (int64_t)s.odd << s.lj;
    const int64_t cols = M << s.j2, mthreads = (int64_t)s.N >> (s.j2 > 5 ? 4 : s.j2), np = word_np(s.set);
    const int R1 = s.odd << (s.lj - s.j2);
    switch (kind) {
        case JK_WCOL_FWD: return ((sqr ? 1 : 2) * np * cols + WT - 1) / WT;
        case JK_WMID_FWD: return ((sqr ? 1 : 2) * np * mthreads + WT - 1) / WT;
        case JK_WMID_REV: return (np * mthreads + WT - 1) / WT;
        case JK_WBLOCK: return (np * R * (M / 16) + WT - 1) / WT;
        case JK_WSMALL: return 1;
        case JK_WCARRY: {
            const int64_t per = WT / 32 * carry_per_warp(s.N ? word_run(R1) : UNPACK_TL);
            return (ntl + per - 1) / per;
        }
        default: return cols / word_run(R1);  // JK_WTAIL
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
template <int ODD, int LJ, int LM, int SET>
static WLaunch tail_kernel() {
    using T = WTail<ODD, LJ, SET>;
    return WLaunch{k_wtail<ODD, LJ, LM, SET>, T::NT, T::bytes};
}
template <int ODD, int LJ>
static WLaunch col_kernel(int kind, bool lm12) {
    if (lm12) return kind == JK_WCOL_FWD ? WLaunch{k_wcol_fwd<ODD, LJ, 12, 0>, WT, 0} : tail_kernel<ODD, LJ, 12, 0>();
    // no supported length has these rows above other column counts
    if constexpr ((ODD == 1 && (LJ == 1 || LJ == 5)) || (ODD == 3 && LJ == 0)) return WLaunch{nullptr, 0, 0};
    else return kind == JK_WCOL_FWD ? WLaunch{k_wcol_fwd<ODD, LJ, 0, 0>, WT, 0} : tail_kernel<ODD, LJ, 0, 0>();
}
template <int J>
static WLaunch mid_kernel(int kind) {
    return WLaunch{kind == JK_WMID_FWD ? k_wmid<J, true, 0> : k_wmid<J, false, 0>, WT, 0};
}
template <int J, int SET>
static WLaunch mid_sm_kernel(int kind) {
    return WLaunch{kind == JK_WMID_FWD ? k_wmid_sm<J, true, SET> : k_wmid_sm<J, false, SET>, WT, 0};
}

// Kernels of the six-prime sets.
template <int SET, int ODD, int LJ>
static WLaunch big_kernel(int kind, int variant) {
    switch (kind) {
        case JK_WCOL_FWD: return WLaunch{k_wcol_fwd<ODD, LJ, 0, SET>, WT, 0};
        case JK_WTAIL: return tail_kernel<ODD, LJ, 0, SET>();
        case JK_WBLOCK: return WLaunch{k_wblock<SET>, WT, 0};
        case JK_WMID_FWD:
        case JK_WMID_REV:
            if constexpr (SET == 2)  // (set 1 has 64 middle rows at least)
                if (variant == 5) return WLaunch{kind == JK_WMID_FWD ? k_wmid<5, true, SET> : k_wmid<5, false, SET>, WT, 0};
            switch (variant) {
                case 6: return mid_sm_kernel<6, SET>(kind);
                case 7: return mid_sm_kernel<7, SET>(kind);
                case 8: return mid_sm_kernel<8, SET>(kind);
            }
    }
    return WLaunch{nullptr, 0, 0};
}

static WLaunch word_kernel(int kind, int variant) {
    if (kind == JK_WCARRY) return WLaunch{k_wcarry, WT, 0};
    if (variant >> 20 == 1) return big_kernel<1, 3, 3>(kind, variant & 0xfffff);
    if (variant >> 20 == 2) return big_kernel<2, 1, 5>(kind, variant & 0xfffff);
    switch (kind) {
        case JK_WBLOCK: return WLaunch{k_wblock<0>, WT, 0};
        case JK_WCOL_FWD:
        case JK_WTAIL:  // one kernel per row count: a switch inside one kernel took 25% longer (registers)
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
        case JK_WMID_FWD:
        case JK_WMID_REV:
            switch (variant) {
                case 3: return mid_kernel<3>(kind);
                case 4: return mid_kernel<4>(kind);
                case 5: return mid_kernel<5>(kind);
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

// Raises the dynamic shared-memory limit of every kernel above the default.
static cudaError_t small_attributes() {
    cudaError_t e = cudaSuccess;
    auto raise = [&](const WLaunch& l) {
        if (e == cudaSuccess && l.fn && l.smem > 0)
            e = cudaFuncSetAttribute(l.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l.smem);
    };
#define NBG_SMALL(O, M) raise(small_kernel<O, M>());
    NBG_SMALLS
#undef NBG_SMALL
    for (int odd : {1, 3, 5, 7})
        for (int lj = 0; lj <= 5; lj++)
            for (int l12 = 0; l12 < 2; l12++) raise(word_kernel(JK_WTAIL, l12 << 16 | odd << 8 | lj));
    raise(word_kernel(JK_WTAIL, 1 << 20));
    raise(word_kernel(JK_WTAIL, 2 << 20));
    return e;
}

static cudaError_t launch(int kind, int variant, const WArgs& a, int64_t nctas, cudaStream_t st) {
    if (nctas <= 0) return cudaSuccess;
    const WLaunch k = word_kernel(kind, variant);
    if (!k.fn || nctas > 0x7fffffff) return cudaErrorInvalidValue;
    if (a.nseg == 0) {  // one product: its short kernels start while the one before drains
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)nctas);
        cfg.blockDim = dim3((unsigned)k.threads);
        cfg.dynamicSmemBytes = k.smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, k.fn, a);
    }
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
