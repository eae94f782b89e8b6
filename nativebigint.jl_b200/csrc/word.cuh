// word.cuh — arithmetic modulo 30-bit primes on 32-bit registers.
//
// Values are lazy representatives: the forward (decimation by X^L - w^2 into
// X^(L/2) -+ w) butterflies take and return [0, 4p), the reverse ones [0, 2p);
// p < 2^30 keeps 4p below 2^32.  A product with a constant w uses the
// precomputed quotient w' = floor(w * 2^32 / p): y*w - floor(y*w'/2^32)*p lies
// in [0, 2p) for every 32-bit y (one multiply-high and two low multiplies; the
// multiply-high issues at a quarter of the FP32 rate and bounds the kernels).
#pragma once
#include <cstdint>

namespace nbg {
namespace wd {

struct Tw {  // constant and its quotient floor(w * 2^32 / p)
    uint32_t w, q;
};

__device__ __forceinline__ uint32_t mulw(uint32_t y, Tw t, uint32_t p) {
    return y * t.w - __umulhi(y, t.q) * p;
}
// [0, 2c) -> [0, c)
__device__ __forceinline__ uint32_t sub_if(uint32_t x, uint32_t c) { return min(x, x - c); }

// x * 2^-32 mod p for x < 2^64, as a value in (0, x / 2^32 + p]; pinv = p^-1 mod 2^32
__device__ __forceinline__ uint32_t redc(uint64_t x, uint32_t p, uint32_t pinv) {
    const uint32_t m = (uint32_t)x * pinv;
    return (uint32_t)(x >> 32) - __umulhi(m, p) + p;
}
__device__ __forceinline__ uint64_t mulx(uint32_t a, uint32_t b) { return (uint64_t)a * b; }

// X, Y in [0, 4p) -> X + wY, X - wY in [0, 4p)
__device__ __forceinline__ void bf_fwd(uint32_t& X, uint32_t& Y, Tw t, uint32_t p, uint32_t p2) {
    const uint32_t x = sub_if(X, p2), v = mulw(Y, t, p);
    X = x + v;
    Y = x - v + p2;
}
// X, Y in [0, 2p) -> X + Y, (X - Y)w in [0, 2p)
__device__ __forceinline__ void bf_rev(uint32_t& X, uint32_t& Y, Tw t, uint32_t p, uint32_t p2) {
    const uint32_t d = X - Y + p2;
    X = sub_if(X + Y, p2);
    Y = mulw(d, t, p);
}

// 2^t consecutive table entries starting at tab[i << t] (16-byte loads from t = 1 on)
template <int T>
__device__ __forceinline__ void load_tw(const Tw* __restrict__ tab, uint32_t i, Tw* o) {
    if (T == 0) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(tab + i));
        o[0] = Tw{v.x, v.y};
    } else {
        const uint4* s = reinterpret_cast<const uint4*>(tab + ((size_t)i << T));
#pragma unroll
        for (int k = 0; k < (1 << T) / 2; k++) {
            const uint4 v = __ldg(s + k);
            o[2 * k] = Tw{v.x, v.y};
            o[2 * k + 1] = Tw{v.z, v.w};
        }
    }
}

// J levels on 2^J values x[0], x[ST], x[2 ST], ...: the subtree under node
// `idx` (heap order) of a forward table.  NV vectors, VS apart, share the constants; the first T0 levels
// are the caller's.
template <int J, int ST, int NV = 1, int VS = 0, int T0 = 0>
__device__ __forceinline__ void tree_fwd(uint32_t* x, const Tw* __restrict__ tab, uint32_t idx, uint32_t p) {
    const uint32_t p2 = 2 * p;
    auto level = [&](auto tc) {
        constexpr int t = decltype(tc)::value;
        constexpr int h = (1 << J) >> (t + 1);
        Tw w[1 << t];
        load_tw<t>(tab, idx, w);
#pragma unroll
        for (int i = 0; i < (1 << t); i++)
#pragma unroll
            for (int e = 0; e < h; e++)
#pragma unroll
                for (int v = 0; v < NV; v++)
                    bf_fwd(x[v * VS + (2 * h * i + e) * ST], x[v * VS + (2 * h * i + e + h) * ST], w[i], p, p2);
    };
    if constexpr (J > 0 && T0 < 1) level(std::integral_constant<int, 0>{});
    if constexpr (J > 1) level(std::integral_constant<int, 1>{});
    if constexpr (J > 2) level(std::integral_constant<int, 2>{});
    if constexpr (J > 3) level(std::integral_constant<int, 3>{});
    if constexpr (J > 4) level(std::integral_constant<int, 4>{});
}
template <int J, int ST>
__device__ __forceinline__ void tree_rev(uint32_t* x, const Tw* __restrict__ tab, uint32_t idx, uint32_t p) {
    const uint32_t p2 = 2 * p;
    auto level = [&](auto tc) {
        constexpr int t = decltype(tc)::value;
        constexpr int h = (1 << J) >> (t + 1);
        Tw w[1 << t];
        load_tw<t>(tab, idx, w);
#pragma unroll
        for (int i = 0; i < (1 << t); i++)
#pragma unroll
            for (int e = 0; e < h; e++) bf_rev(x[(2 * h * i + e) * ST], x[(2 * h * i + e + h) * ST], w[i], p, p2);
    };
    if constexpr (J > 4) level(std::integral_constant<int, 4>{});
    if constexpr (J > 3) level(std::integral_constant<int, 3>{});
    if constexpr (J > 2) level(std::integral_constant<int, 2>{});
    if constexpr (J > 1) level(std::integral_constant<int, 1>{});
    if constexpr (J > 0) level(std::integral_constant<int, 0>{});
}

}  // namespace wd
}  // namespace nbg
