// Exact modular arithmetic on the FP64 pipe, for moduli below 2^50.
//
// A residue is an integer-valued double, a multiplier w a centred one (|w| <= q/2) with
// its quotient wq = w * (1 / q), rounded. The product y w mod q takes six FP64 instructions: t = the
// integer nearest y wq (one fused multiply-add into 1.5 * 2^52, whose last place is 1),
// y w as the exact pair h + l, and y w - t q = (h - t q) + l. Every step is exact while
// |y| <= 2^52: |y wq| stays below 2^51, h and l are the rounded product and its exact
// remainder, h - t q is an integer below 2^51, so the result is the exact integer
// y w - t q, and |result| <= q (1/2 + |y| 2^-53) (the second term is the error of wq, two
// roundings at most).
//
// Why: the 64-bit integer Shoup product needs about 14 - 18 issue slots of the FMA-heavy
// pipe, the FP64 pipe (64 lanes a clock and SM on B200) is idle meanwhile. A whole
// butterfly is 8 FP64 instructions; measured with operands in registers on B200
// (tb_measure_fp64_butterfly_rate): 2,200 G butterflies/s against 1,023 G for the
// estimated-quotient integer butterfly.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace tb {

// One modulus of the FP64 forms: twiddles as centred doubles in the order of the radix-8
// passes (fp_fwd_index, fp_inv_index), q and 1 / q, and the scaled last inverse stage's
// constants. p / ip hold {twiddle, quotient} for the passes whose warps share twiddles:
// the first N / 16 indices forward, the last N / 16 inverse (ip[i - (N - N / 16)]).
struct FpMod {
    const double *w, *iw;
    const double2 *p, *ip;
    double q, qinv;
    double inv_n, sroot;
};

constexpr double FP_ROUND = 6755399441055744.0;     // 1.5 * 2^52: adding it rounds to an integer
constexpr double FP_2P52 = 4503599627370496.0;
constexpr uint64_t FP_MAX_Q = 1ull << 50;            // moduli of the FP64 forms are below this
constexpr uint64_t FP_PLAIN_Q = 1ull << 48;          // below this no reductions between passes
constexpr uint64_t FP_MAX_IN = 1ull << 49;           // unreduced transform inputs are below this

// x in [0, 2^52) as a double (exponent bits OR-ed in, one subtraction).
__device__ __forceinline__ double fp_from_u64(uint64_t x) {
    return __dadd_rn(__longlong_as_double((long long)(x | 0x4330000000000000ull)), -FP_2P52);
}

__device__ __forceinline__ double fp_mulmod(double y, double w, double wq, double q) {
    const double t = __dadd_rn(__fma_rn(y, wq, FP_ROUND), -FP_ROUND);
    const double h = __dmul_rn(y, w);
    const double l = __fma_rn(y, w, -h);
    return __dadd_rn(__fma_rn(-t, q, h), l);
}

// x mod q in about [-q/2, q/2] for |x| < 2^53 and |x / q| < 2^51: |result| <= q/2 + |x| 2^-53.
__device__ __forceinline__ double fp_reduce(double x, double q, double qinv) {
    const double t = __dadd_rn(__fma_rn(x, qinv, FP_ROUND), -FP_ROUND);
    return __fma_rn(-t, q, x);
}

// [0, q) from an integer |x| < q: the two's complement value, and q added where it is
// negative (the unsigned minimum of x and x + q).
__device__ __forceinline__ uint64_t fp_to_residue(double x, uint64_t q) {
    const uint64_t u = (uint64_t)(__double_as_longlong(__dadd_rn(x, FP_ROUND)) - __double_as_longlong(FP_ROUND));
    return min(u, u + q);
}

__device__ __forceinline__ double fp_centred(uint64_t w, uint64_t q) {
    return w > (q >> 1) ? -fp_from_u64(q - w) : fp_from_u64(w);
}

// Where the pass-ordered tables (FP64, and the integer ones at roots + 2 N for N <= 2^14)
// keep the twiddles of the integer tables in natural order. The three stages of a
// radix-8 pass starting at stage s use 7 consecutive ranges of 2^s twiddles (forward:
// indices 2^s .. 8 2^s - 1); the ordered tables hold, inside the same range, twiddle k (0 ..
// 6, in stage order) of every group side by side, so a warp's loads of one k are
// consecutive. Radix-8 passes end at the last stage, so the stages before the first one
// (logn mod 3) keep their natural order. index 1 .. n - 1.
// Natural index i of stage s (2^s <= i < 2^(s+1)).
__host__ __device__ constexpr uint32_t fp_fwd_stage_index(uint32_t i, int s, int logn) {
    const int r = logn % 3;
    if (s < r) return i;
    const int s0 = r + (s - r) / 3 * 3, t = s - s0;
    return (((1u << t) - 1 + (i & ((1u << t) - 1))) << s0) + (i >> t);
}
__host__ __device__ inline uint32_t fp_fwd_index(uint32_t i, int logn) {
    int s = 0;
    while ((2u << s) <= i) s++;
    return fp_fwd_stage_index(i, s, logn);
}

// Inverse tables: stage sg uses indices n + 1 - (n >> sg) onwards, the radix-8 passes start
// at stages 0, 3, 6, ... and the remaining last stages keep their natural order. b: the
// twiddle's number in its stage.
__host__ __device__ constexpr uint32_t fp_inv_stage_index(uint32_t b, int sg, int logn) {
    const uint32_t n = 1u << logn;
    const int s = sg / 3 * 3, t = sg - s;
    if (s + 3 > logn) return n + 1 - (n >> sg) + b;
    const uint32_t j = b & ((4u >> t) - 1), blk = b >> (2 - t);
    const uint32_t k = t == 0 ? j : t == 1 ? 4 + j : 6;
    return n + 1 - (n >> s) + k * (n >> (s + 3)) + blk;
}
__host__ __device__ inline uint32_t fp_inv_index(uint32_t i, int logn) {
    const uint32_t n = 1u << logn;
    int sg = 0;
    while (sg + 1 < logn && n + 1 - (n >> (sg + 1)) <= i) sg++;
    return fp_inv_stage_index(i - (n + 1 - (n >> sg)), sg, logn);
}

}  // namespace tb
