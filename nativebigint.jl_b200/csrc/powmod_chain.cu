// powmod_chain.cu — whole Barrett power chains, one CTA per chain.
//
// A step (product x*y, q1*mu, q3*m, subtraction and corrections) is a serial
// chain of short kernels when each part is a launch: for 256-limb moduli about
// 35 us per step, most of it launch gaps, cold constants and residues going
// through global memory.  Chains are independent, so k_pm_chain runs the steps
// of one chain in one CTA: the three products are the one-CTA word product
// (word_device.cuh) with T and q2 in shared memory, the transforms of mu and m
// are made once and kept there, a squaring transforms one operand, and the
// subtraction of r2 reads it from the registers that assembled it.
// Bound by the latency of a step's serial rounds, about 12 us (64 chains of
// 256-limb moduli and 1024-bit exponents: 43 -> 15 ms on the device).
#include <cuda_runtime.h>

#include "powmod_kernels.h"
#include "word_device.cuh"

namespace nbg {

template <int ODD, int LM>
struct ChainShape {
    using W = WSmall<ODD, LM>;
    static constexpr size_t words = sizeof(uint64_t) * 4 * W::LT;           // T, q2
    static constexpr size_t spec = (sizeof(uint32_t) * W::OPW + 15) / 16 * 16;  // a kept transform
    static constexpr size_t bytes = W::limb_bytes + 2 * words + 2 * spec + sizeof(uint32_t) * 2 * W::OPW;
};

// d = x - y on four limbs per thread (limbs at or above n read as zero) across
// the CTA; returns whether the whole subtraction borrows.
__device__ __forceinline__ bool cta_sub(uint32_t* wagg, uint64_t* d, const uint64_t* x, const uint64_t* y) {
    uint32_t b = 0, eq = 1;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint64_t t = x[q] - y[q];
        const uint32_t b1 = x[q] < y[q];
        d[q] = t - b;
        eq &= t == 0 ? 1u : 0u;
        b = b1 | (t < (uint64_t)b ? 1u : 0u);
    }
    __syncthreads();  // wagg's previous readers
    uint32_t total;
    uint64_t cin = cta_scan(b | (eq << 1), wagg, total);  // all limbs equal: a borrow passes
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint64_t t = d[q];
        d[q] = t - cin;
        cin = cin && t == 0;
    }
    return total & 1u;
}

// Steps [s0, s1) of the chain blockIdx.x.  k: modulus limbs, N >= 2k; q1*mu has
// 2k + 1 coefficients: when that is N + 1 the last one wraps onto the first and
// is moved back (it is the product of the two top limbs).
template <int ODD, int LM>
__global__ void __launch_bounds__(WSmall<ODD, LM>::NT, WSmall<ODD, LM>::NT > 256 ? 1 : 2)
    k_pm_chain(const PmChains C, const uint64_t* __restrict__ mus, const void* wtf, const void* wti, int wL, WScale sc,
               int64_t s0, int64_t s1) {
    using W = WSmall<ODD, LM>;
    using CS = ChainShape<ODD, LM>;
    constexpr int LT = W::LT, N = W::N;
    extern __shared__ __align__(16) unsigned char dyn[];
    LimbShared<LT>& S = *reinterpret_cast<LimbShared<LT>*>(dyn);
    uint64_t* const T = reinterpret_cast<uint64_t*>(dyn + W::limb_bytes);
    uint64_t* const Q = T + 4 * LT;
    uint32_t* const smu = reinterpret_cast<uint32_t*>(dyn + W::limb_bytes + 2 * CS::words);
    uint32_t* const smm = smu + CS::spec / 4;
    uint32_t* const sm = smm + CS::spec / 4;
    const int c = (int)blockIdx.x, tid = (int)threadIdx.x;
    const int k = (int)C.k, lmu = k + 1;
    const int64_t steps = min(C.nsteps[c], s1);
    if (s0 >= steps) return;
    const uint64_t* __restrict__ m = C.mod + (int64_t)c * k;
    const uint64_t* __restrict__ mu = mus + (int64_t)c * (k + 2);
    uint64_t* const slots = C.slots + (int64_t)c * C.nslot * k;
    const uint8_t* __restrict__ ops = C.ops + (int64_t)c * C.max_steps * 3;
    const bool wrap = 2 * k + 1 > N;
    const SmallThread<ODD, LM> th(sm, wtf, wti, wL);
    if (tid == 0) {
        S.mid[0] = 0;
        S.hi[0][0] = S.hi[0][1] = 0;
        S.c[0] = 0;
    }
    uint32_t x[32];
    // x[0..16) = the transform of n limbs; x[16..32) of n2 more when given
    auto transform = [&](int n, auto limb) {
        th.load(x, th.sp, n, limb);
        if (ODD > 1) {
            __syncthreads();
            th.fetch(x, 0);
        }
        th.template down<1>(x);
    };
    auto keep = [&](uint32_t* spec) {
        if (th.live) wput16(spec + th.pi * ODD * W::SM + th.j * W::SM, x, th.t);
    };
    auto kept = [&](uint32_t* spec) {
        if (th.live) wget16(spec + th.pi * ODD * W::SM + th.j * W::SM, x + 16, th.t);
    };
    // the product's limbs, four per thread
    auto assemble = [&](int nlimbs, bool wrapped, uint64_t* own) {
        th.up(x);
        uint64_t lo[4], mid[4];
        uint32_t hi[4];
        SmallThread<ODD, LM>::coefs(sm, sc.v, lo, mid, hi);
        if (wrapped && (tid == 0 || 4 * tid == N)) {
            const uint64_t a = T[2 * k - 1], b = mu[k];
            const uint64_t plo = a * b, phi = __umul64hi(a, b);
            if (tid == 0) {
                const uint64_t l = lo[0], h = mid[0];
                const uint32_t b0 = l < plo;
                lo[0] = l - plo;
                mid[0] = h - phi - b0;
                hi[0] -= (h < phi) || (h - phi < (uint64_t)b0);
            } else {
                lo[0] = plo;
                mid[0] = phi;
            }
        }
        limb_sums<LT>(S, tid, LT, lo, mid, hi, nlimbs, own);
    };
    transform(lmu, [&](int i) { return mu[i]; });
    keep(smu);
    __syncthreads();  // the shared blocks are reused
    transform(k, [&](int i) { return m[i]; });
    keep(smm);
    __syncthreads();
    uint64_t own[4], r[4], y[4];
    for (int64_t s = s0; s < steps; s++) {
        const int od = ops[3 * s], oa = ops[3 * s + 1], ob = ops[3 * s + 2];
        const uint64_t* pa = slots + (int64_t)oa * k;
        uint64_t* dst = slots + (int64_t)od * k;
        if (ob == PM_COPY) {
            for (int i = tid; i < k; i += W::NT) dst[i] = pa[i];
            __syncthreads();
            continue;
        }
        // T = x * y
        if (oa == ob) {
            transform(k, [&](int i) { return pa[i]; });
        } else {
            const uint64_t* pb = slots + (int64_t)ob * k;
            th.load(x, th.sp, k, [&](int i) { return pa[i]; });
            th.load(x + 16, th.sp + W::OPW, k, [&](int i) { return pb[i]; });
            if (ODD > 1) {
                __syncthreads();
                th.fetch(x, 0);
                th.fetch(x + 16, 1);
            }
            th.template down<2>(x);
        }
        th.point(x, oa == ob);
        assemble(2 * k, false, own);
        if (tid < LT) {
#pragma unroll
            for (int q = 0; q < 4; q++) T[4 * tid + q] = own[q];
        }
        __syncthreads();
        // q2 = floor(T / B^(k-1)) * mu
        transform(k + 1, [&](int i) { return T[k - 1 + i]; });
        kept(smu);
        th.point(x, false);
        assemble(2 * k + 2, wrap, own);
        if (tid < LT) {
#pragma unroll
            for (int q = 0; q < 4; q++) Q[4 * tid + q] = own[q];
        }
        __syncthreads();
        // r2 = floor(q2 / B^(k+1)) * m, of which the low k + 1 limbs matter
        transform(lmu, [&](int i) { return Q[k + 1 + i]; });
        kept(smm);
        th.point(x, false);
        assemble(2 * k + 1, false, own);
        // r = (T - r2) mod B^(k+1), then r -= m while r >= m
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = 4 * tid + q;
            const bool in = tid < LT && i <= k;
            y[q] = in ? own[q] : 0;
            r[q] = in ? T[i] : 0;
        }
        cta_sub(S.wagg, own, r, y);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int i = 4 * tid + q;
            r[q] = i <= k ? own[q] : 0;
            y[q] = i < k ? m[i] : 0;
        }
        for (int it = 0; it < 4; it++) {
            if (cta_sub(S.wagg, own, r, y)) break;
#pragma unroll
            for (int q = 0; q < 4; q++) r[q] = own[q];
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (4 * tid + q < k) dst[4 * tid + q] = r[q];
        __syncthreads();
    }
}

struct ChainKernel {
    void (*fn)(const PmChains, const uint64_t*, const void*, const void*, int, WScale, int64_t, int64_t);
    int odd, lm, threads;
    size_t smem;
};
template <int ODD, int LM>
static constexpr ChainKernel chain() {
    static_assert(ChainShape<ODD, LM>::bytes <= 220 * 1024, "shared memory");
    return ChainKernel{k_pm_chain<ODD, LM>, ODD, LM, WSmall<ODD, LM>::NT, ChainShape<ODD, LM>::bytes};
}
static const ChainKernel CHAINS[] = {chain<1, 6>(), chain<1, 7>(), chain<3, 6>(), chain<1, 8>(),  chain<3, 7>(),
                                     chain<1, 9>(), chain<3, 8>(), chain<1, 10>(), chain<3, 9>()};

// Every modulus that fits, at any number of chains: product batches were slower
// wherever measured (ms per call, batches against chains, 512-bit exponents: 256
// limbs 1 chain 45/8, 64 60/11, 600 155/56; 400 limbs 8 50/13, 300 141/54; 512
// limbs 600 372/97; 513 limbs 8 63/19; 768 limbs 1 78/19, 148 247/38, 300 474/89).
static const ChainKernel* chain_for(int64_t k) {
    for (const ChainKernel& c : CHAINS)
        if (((int64_t)c.odd << c.lm) >= 2 * k) return &c;
    return nullptr;
}

bool pm_chain_shape(int64_t k, WordShape& s) {
    const ChainKernel* c = chain_for(k);
    if (!c) return false;
    s = WordShape{c->odd << c->lm, c->odd, 0, 0, c->lm, true, 0};
    return true;
}

cudaError_t pm_chain_init() {
    WConst h[WSETS];
    word_fill_const(h);
    cudaError_t e = cudaMemcpyToSymbol(c_w, h, sizeof h);
    for (const ChainKernel& c : CHAINS)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(c.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.smem);
    return e;
}

cudaError_t pm_launch_chain(const PmChains& C, const uint64_t* mu, const void* wtf, const void* wti, int wL,
                            const WScale& sc, int64_t s0, int64_t s1, cudaStream_t st) {
    const ChainKernel* c = chain_for(C.k);
    if (!c) return cudaErrorInvalidValue;
    c->fn<<<(unsigned)C.count, c->threads, c->smem, st>>>(C, mu, wtf, wti, wL, sc, s0, s1);
    return cudaGetLastError();
}

}  // namespace nbg
