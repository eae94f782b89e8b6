// word.h — products through transforms over five (or six) 30-bit primes ("word"
// products): every 64-bit limb is one coefficient, so packing is a reduction
// and the results are the carried sums of the convolution's coefficients.
//
// A transform of length N = odd * 2^k (odd in {1, 3, 5, 7}) works modulo
// X^N - 1: one radix-`odd` step splits it into X^(2^k) - e(j/odd) (e(t) a fixed
// primitive root's t-th turn), then each X^L - e(t) splits into
// X^(L/2) - e(t/2) and X^(L/2) + e(t/2).  Node n of level l under block j
// (level 0 is the block itself) has t = (j/odd + bitrev_l(n)) / 2^l; its
// butterfly constant e(t/2) is entry 2^l + n of block j's table, so a subtree's
// constants are contiguous per level and every size shares one table.  The
// splitting stops two levels early: the leaves are polynomials modulo
// X^4 - e(t), multiplied directly, which needs a quarter of the table.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "types.h"

namespace nbg {

// Prime sets.  Set 0 (p = 1 mod 105 * 2^18, product above 2^149) serves
// lengths odd * 2^k up to 7 * 2^19: of m + n - 1 coefficients each is below
// min(m, n) * 2^128, and min(m, n) below 2^21.  Above 3.6M
// points the coefficients need a sixth prime and the roots more twos: set 1
// (p = 1 mod 3 * 2^22) for 3 * 2^k, set 2 (p = 1 mod 2^23) for 2^k, k <= 25;
// their products exceed 2^176.
constexpr int WPR = 5;      // primes of set 0
constexpr int WPR_MAX = 6;
constexpr int WSETS = 3;
constexpr int word_np(int set) { return set ? 6 : WPR; }
constexpr uint32_t WPRIMES[WSETS][WPR_MAX] = {
    {1073479681u, 1018429441u, 908328961u, 880803841u, 825753601u, 0},
    {943718401u, 918552577u, 880803841u, 754974721u, 666894337u, 415236097u},
    {998244353u, 897581057u, 880803841u, 754974721u, 645922817u, 595591169u}};
// every residue of 32 bits reaches [0, 3p): by one subtraction of 3p in set 0,
// else by the multiple of p nearest to 2^31 and then 3p
constexpr bool word_pack_ok(int set) {
    for (int i = 0; i < word_np(set); i++) {
        const uint64_t p = WPRIMES[set][i];
        if (set ? (uint64_t(1) << 31) + p / 2 > 6 * p : (uint64_t(1) << 32) > 6 * p) return false;
    }
    return true;
}
constexpr int WORD_MAX_LOG2 = 20;               // set 0: k <= 20 (leaves at level k - 2 <= 18)

// Shape of a word product's transform: N = odd * 2^lj * M.  Blocks of M = 2^lm
// consecutive values (each one subtree) are transformed in shared memory;
// column passes above them work on the rows of one column in registers: one
// pass of odd * 2^lj rows, or, past 32 rows, a first one of odd * 2^(lj - j2)
// and a middle one of 2^j2 (from 64 rows on with a turn through shared memory).
struct WordShape {
    int32_t N = 0, odd = 0, lj = 0, j2 = 0, lm = 0;
    bool small = false;  // one CTA per product (at most 3072 values; lj = 0, no column pass)
    int32_t set = 0;     // prime set
};
// Limbs of a run of the last pass for R rows in the first one: fewer where R rows
// of every prime fill the shared memory sooner.
constexpr int word_run(int R) { return R > 16 ? 64 : 128; }
// Up to this many tiles a word product's last pass adds the carries between them
// itself: its limb tiles are followed by two count words.
constexpr int64_t WORD_FUSED_TILES = 2048;
// The smallest supported length >= nconv; false when there is none.
// coarse: up to 2^17 values only odd = 1 and 3, so that a batch of many lengths
// needs half the kernels at up to a fifth more work.
bool word_shape(int64_t nconv, WordShape& s, bool coarse = false);

// One launch's CTAs: products of one shape are consecutive, `cpp` CTAs each.
struct WSeg {
    int32_t begin;  // first CTA
    int32_t first;  // into the launch's product list
    int32_t cpp;    // CTAs per product
    int32_t pad_;
};

// Variant of a word launch: bits 20 on the prime set, below them
// (odd << 8) | (lj - j2) for column passes (bit 16: of 4096 columns), j2 for
// middle passes, (odd << 8) | lm for one-CTA products, 0 for the rest.
cudaError_t word_init();  // constant memory of the current device
cudaError_t launch_word(int kind, int variant, const DProd* prods, const WSeg* segs, int nseg, const int32_t* plist,
                        int64_t nctas, cudaStream_t st);
// The same for one product passed by value (no device tables).
cudaError_t launch_word_one(int kind, int variant, const DProd& P, int64_t nctas, cudaStream_t st);
// CTAs one product needs in a word launch (ntl: its limb tiles; of the FP64 passes where s is empty).
int64_t word_ctas(int kind, const WordShape& s, int sqr, int64_t ntl);

// Tables of one `odd` for heap sizes up to 2^L: per prime and block, fwd then inverse.
size_t word_table_bytes(int set, int odd, int L);
cudaError_t word_build_tables(int set, int odd, int L, void* fwd, void* inv, cudaStream_t st);
// Per-product scale constants of the unpack (the inverse transform's 1/(odd * 2^(k-2)) and the 2^-96 of packing and pointwise products).
void word_scales(const WordShape& s, uint32_t* out);

}  // namespace nbg
