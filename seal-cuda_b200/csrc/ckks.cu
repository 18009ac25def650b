// CKKS encoding and decoding (CKKSEncoder, src/ckks.cpp:32-579) on the device.
//
// Encode: slots -> conjugate-symmetric vector in bit-reversed index order ->
// inverse special FFT (Gentleman-Sande, scaled by scale/N in its last stage) ->
// round the real parts -> reduce into every prime -> NTT. Decode: inverse NTT ->
// CRT compose -> centre and scale to doubles -> forward special FFT -> slots.
// FP64 is used only here. The FFT butterflies follow the reference's DWTHandler
// order with complex products computed as (ac - bd, ad + bc) from individually
// rounded IEEE operations (no fused multiply-add), and the root tables are
// built on the host exactly like ComplexRoots (src/utils/croots.cpp:10-59).
#include <algorithm>
#include <cmath>
#include <complex>
#include <functional>
#include <mutex>
#include <vector>

#include "context.hpp"
#include "hostmath.hpp"
#include "trace.cuh"

namespace tb {

unsigned grid_for(uint64_t work, int threads);
void ensure_pool_retains(int device);
int slot_map(Context &c, const uint32_t **out);
int ntt_forward(const Context &c, const uint64_t *in, uint64_t *out, uint64_t polys, int first, int limbs, bool lazy,
                cudaStream_t s);
int ntt_inverse(const Context &c, const uint64_t *in, uint64_t *out, uint64_t polys, int first, int limbs, bool lazy,
                cudaStream_t s);

namespace {

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                        __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(__dmul_rn(a.x, s), __dmul_rn(a.y, s)); }

// One Gentleman-Sande stage (gap = 2^s) of transformFromRev over B vectors; the
// last stage (m == 1) multiplies by `scalar`.
__global__ void fft_inv_stage(double2 *__restrict__ a, const double2 *__restrict__ iroots, int logn, int s,
                              double scalar, uint64_t B) {
    const uint32_t n = 1u << logn, half = n >> 1;
    const uint64_t total = B * half;
    const uint32_t gap = 1u << s;
    const uint32_t m = n >> (s + 1);
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < total; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = w / half;
        const uint32_t k = (uint32_t)(w - b * half);
        const uint32_t i = k >> s, j = k & (gap - 1);
        double2 *x = a + b * n + 2 * i * gap + j, *y = x + gap;
        const uint32_t ri = n - 2 * m + 1 + i;
        const double2 r = iroots[ri];
        const double2 u = *x, v = *y;
        if (m > 1) {
            *x = cadd(u, v);
            *y = cmul(csub(u, v), r);
        } else {
            const double2 sr = cscale(r, scalar);
            *x = cscale(cadd(u, v), scalar);
            *y = cmul(csub(u, v), sr);
        }
    }
}

// One Cooley-Tukey stage (m = 2^s groups) of transformToRev.
__global__ void fft_fwd_stage(double2 *__restrict__ a, const double2 *__restrict__ roots, int logn, int s, uint64_t B) {
    const uint32_t n = 1u << logn, half = n >> 1;
    const uint64_t total = B * half;
    const uint32_t m = 1u << s, gap = n >> (s + 1);
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < total; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = w / half;
        const uint32_t k = (uint32_t)(w - b * half);
        const uint32_t i = k / gap, j = k - i * gap;
        double2 *x = a + b * n + 2 * i * gap + j, *y = x + gap;
        const double2 r = roots[m + i];
        const double2 u = *x, v = cmul(*y, r);
        *x = cadd(u, v);
        *y = csub(u, v);
    }
}

// The special FFT's stages inside blocks of 2^logb <= 4096 consecutive points run in shared
// memory (64 KB of complex doubles), two stages per pass; the stages that join blocks (up
// to 3) run in registers in the kernels around it. One kernel per stage over global memory
// spent its time on launches and latency (N = 16384: 14 launches, 65 us for 16 vectors).
// Every butterfly is computed as before, so the words are too.
constexpr int FFT_LOGB = 12;
constexpr int FFT_THREADS = 512;

// Slot of point e: 16-byte points, the low three bits XORed with the next three so that
// strides of 2 .. 64 points spread over the banks.
__device__ __forceinline__ uint32_t fft_slot(uint32_t e) { return e ^ ((e >> 3) & 7) ^ ((e >> 6) & 7); }

__device__ __forceinline__ void fft_inv_butterfly(double2 &x, double2 &y, double2 r, bool last, double scalar) {
    const double2 u = x, v = y;
    if (!last) {
        x = cadd(u, v);
        y = cmul(csub(u, v), r);
    } else {
        x = cscale(cadd(u, v), scalar);
        y = cmul(csub(u, v), cscale(r, scalar));
    }
}

__device__ __forceinline__ void fft_fwd_butterfly(double2 &x, double2 &y, double2 r) {
    const double2 u = x, v = cmul(y, r);
    x = cadd(u, v);
    y = csub(u, v);
}

// Inverse stages 0 .. logb - 1 of block blockIdx.x of vector blockIdx.y: point p of the
// conjugate-symmetric vector is the value of slot inv[p] (its conjugate for slots of the
// second half, zero from `count` on).
__global__ void __launch_bounds__(FFT_THREADS) fft_inv_block(const double2 *__restrict__ vals, uint64_t vstride,
                                                             uint32_t count, double2 *__restrict__ a,
                                                             const double2 *__restrict__ iroots,
                                                             const uint32_t *__restrict__ inv, int logn, int logb,
                                                             double scalar) {
    extern __shared__ double2 fsm[];
    const uint32_t n = 1u << logn, slots = n >> 1, nb = 1u << logb, p0 = blockIdx.x << logb;
    const double2 *v = vals + blockIdx.y * vstride;
    for (uint32_t e = threadIdx.x; e < nb; e += blockDim.x) {
        const uint32_t i = __ldg(inv + p0 + e), j = i & (slots - 1);
        double2 x = make_double2(0.0, 0.0);
        if (j < count) x = v[j];
        fsm[fft_slot(e)] = i < slots ? x : make_double2(x.x, -x.y);
    }
    __syncthreads();
    int s = 0;
    for (; s + 2 <= logb; s += 2) {   // stages s and s + 1
        const uint32_t m0 = n >> (s + 1), m1 = m0 >> 1, gap = 1u << s;
        for (uint32_t g = threadIdx.x; g < nb / 4; g += blockDim.x) {
            const uint32_t i = g >> s, e = (i << (s + 2)) + (g & (gap - 1)), gi = (p0 >> (s + 2)) + i;
            double2 x[4];
#pragma unroll
            for (int k = 0; k < 4; k++) x[k] = fsm[fft_slot(e + k * gap)];
            const double2 r0 = __ldg(iroots + (n - 2 * m0 + 1 + 2 * gi)), r1 = __ldg(iroots + (n - 2 * m0 + 2 + 2 * gi)),
                          r2 = __ldg(iroots + (n - 2 * m1 + 1 + gi));
            fft_inv_butterfly(x[0], x[1], r0, false, scalar);
            fft_inv_butterfly(x[2], x[3], r1, false, scalar);
            fft_inv_butterfly(x[0], x[2], r2, m1 == 1, scalar);
            fft_inv_butterfly(x[1], x[3], r2, m1 == 1, scalar);
#pragma unroll
            for (int k = 0; k < 4; k++) fsm[fft_slot(e + k * gap)] = x[k];
        }
        __syncthreads();
    }
    if (s < logb) {
        const uint32_t m0 = n >> (s + 1), gap = 1u << s;
        for (uint32_t g = threadIdx.x; g < nb / 2; g += blockDim.x) {
            const uint32_t i = g >> s, e = (i << (s + 1)) + (g & (gap - 1)), gi = (p0 >> (s + 1)) + i;
            double2 x = fsm[fft_slot(e)], y = fsm[fft_slot(e + gap)];
            fft_inv_butterfly(x, y, __ldg(iroots + (n - 2 * m0 + 1 + gi)), m0 == 1, scalar);
            fsm[fft_slot(e)] = x;
            fsm[fft_slot(e + gap)] = y;
        }
        __syncthreads();
    }
    double2 *out = a + ((size_t)blockIdx.y << logn) + p0;
    for (uint32_t e = threadIdx.x; e < nb; e += blockDim.x) out[e] = fsm[fft_slot(e)];
}

// Forward stages of block blockIdx.x of vector blockIdx.y: the first H_LOG stages join the
// 2^H_LOG blocks, and every CTA computes its own block's points of them from the real
// coefficients (coeff, `cplx` 0) or the complex points (`cplx` 1); the rest runs in shared
// memory, and point p goes to slot inv[p] (slots of the second half are conjugates and are
// not written).
template <int H_LOG>
__global__ void __launch_bounds__(FFT_THREADS) fft_fwd_block(const double2 *__restrict__ a,
                                                             const double *__restrict__ coeff, double2 *__restrict__ out,
                                                             uint64_t ostride, const double2 *__restrict__ roots,
                                                             const uint32_t *__restrict__ inv, int logn, int logb) {
    extern __shared__ double2 fsm[];
    constexpr int H = 1 << H_LOG;
    const uint32_t n = 1u << logn, slots = n >> 1, nb = 1u << logb, blk = blockIdx.x, p0 = blk << logb;
    const size_t vec = (size_t)blockIdx.y << logn;
    const int top = logn - logb;         // stages before the block's
    const uint32_t sup = blk >> H_LOG;   // which group of H blocks
    for (uint32_t e = threadIdx.x; e < nb; e += blockDim.x) {
        double2 x[H];
        const size_t base = vec + (((size_t)sup << H_LOG) << logb) + e;
#pragma unroll
        for (int k = 0; k < H; k++)
            x[k] = coeff ? make_double2(coeff[base + ((size_t)k << logb)], 0.0) : a[base + ((size_t)k << logb)];
        // keep only the side of each stage that leads to this block
#pragma unroll
        for (int t = 0; t < H_LOG; t++) {
            const int half = H >> (t + 1);
            const int s = top - H_LOG + t;   // global stage: 2^s groups
            const bool hi = (blk >> (H_LOG - 1 - t)) & 1;
            const double2 r = __ldg(roots + (1u << s) + (blk >> (top - s)));
#pragma unroll
            for (int k = 0; k < half; k++) {
                double2 p = x[k], q = x[k + half];
                fft_fwd_butterfly(p, q, r);
                x[k] = hi ? q : p;
            }
        }
        fsm[fft_slot(e)] = x[0];
    }
    __syncthreads();
    int s = 0;   // stage inside the block
    if (logb & 1) {
        const uint32_t gap = nb >> 1;
        const double2 r = __ldg(roots + (1u << top) + blk);
        for (uint32_t e = threadIdx.x; e < gap; e += blockDim.x) {
            double2 x = fsm[fft_slot(e)], y = fsm[fft_slot(e + gap)];
            fft_fwd_butterfly(x, y, r);
            fsm[fft_slot(e)] = x;
            fsm[fft_slot(e + gap)] = y;
        }
        s = 1;
        __syncthreads();
    }
    for (; s < logb; s += 2) {   // stages s and s + 1
        const int ls = logb - s - 2;
        const uint32_t gap = 1u << ls;
        for (uint32_t g = threadIdx.x; g < nb / 4; g += blockDim.x) {
            const uint32_t i = g >> ls, e = (i << (ls + 2)) + (g & (gap - 1));
            const uint32_t X = ((1u << top) + blk << s) + i;
            double2 x[4];
#pragma unroll
            for (int k = 0; k < 4; k++) x[k] = fsm[fft_slot(e + k * gap)];
            const double2 r0 = __ldg(roots + X), r1 = __ldg(roots + 2 * X), r2 = __ldg(roots + 2 * X + 1);
            fft_fwd_butterfly(x[0], x[2], r0);
            fft_fwd_butterfly(x[1], x[3], r0);
            fft_fwd_butterfly(x[0], x[1], r1);
            fft_fwd_butterfly(x[2], x[3], r2);
#pragma unroll
            for (int k = 0; k < 4; k++) fsm[fft_slot(e + k * gap)] = x[k];
        }
        __syncthreads();
    }
    double2 *o = out + blockIdx.y * ostride;
    for (uint32_t e = threadIdx.x; e < nb; e += blockDim.x) {
        const uint32_t i = __ldg(inv + p0 + e);
        if (i < slots) o[i] = fsm[fft_slot(e)];
    }
}

// Round the real parts and reduce into primes 0..L-1 (src/ckks.cpp:158-230); flags
// coefficients of 128 bits or more.
// The last H_LOG stages of the inverse FFT (the ones that join blocks) run first, in
// registers, on the 2^H_LOG points of a thread.
template <int H_LOG>
__global__ void ckks_round_reduce(const double2 *__restrict__ a, const double2 *__restrict__ iroots,
                                  uint64_t *__restrict__ out, const Mod *__restrict__ mods, int L, int logn, uint64_t B,
                                  int *__restrict__ err, int total_bits, double scalar) {
    constexpr int H = 1 << H_LOG;
    const uint32_t n = 1u << logn;
    const int logsub = logn - H_LOG;
    const uint64_t total = B << logsub;
    const double two64 = 18446744073709551616.0;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < total; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = w >> logsub;
        const uint32_t j = (uint32_t)(w & ((1u << logsub) - 1));
        double2 x[H];
#pragma unroll
        for (int k = 0; k < H; k++) x[k] = a[(b << logn) + ((size_t)k << logsub) + j];
#pragma unroll
        for (int t = 0; t < H_LOG; t++) {
            const int h = 1 << t;
            const uint32_t m = n >> (logsub + t + 1);
#pragma unroll
            for (int k = 0; k < H; k++) {
                if (k & h) continue;
                fft_inv_butterfly(x[k], x[k + h], __ldg(iroots + (n - 2 * m + 1 + (k >> (t + 1)))), t == H_LOG - 1, scalar);
            }
        }
#pragma unroll
        for (int k = 0; k < H; k++) {
            const double mag = fabs(x[k].x);
            // max_coeff_bit_count = ceil(log2(max(|x|, 1))) + 1 must stay below the modulus bits
            if ((mag > 1.0 ? (int)ceil(log2(mag)) : 0) + 1 >= total_bits) atomicOr(err, 1);
            double c = round(x[k].x);
            const bool neg = signbit(c);
            c = fabs(c);
            if (!(c < 170141183460469231731687303715884105728.0)) {  // 2^127
                atomicOr(err, 1);
                c = 0.0;
            }
            const uint64_t lo = (uint64_t)fmod(c, two64), hi = (uint64_t)(c / two64);
            uint64_t *o = out + ((b * L) << logn) + ((size_t)k << logsub) + j;
            for (int l = 0; l < L; l++) {
                const Mod &m = mods[l];
                uint64_t r = hi ? reduce128(hi, lo, m) : reduce64(lo, m);
                if (neg) r = neg_mod(r, m.value);
                o[(size_t)l << logn] = r;
            }
        }
    }
}

// CRT compose, centre and scale (src/ckks.cpp:520-563): per coefficient the
// multi-word x = sum_j [c_j (Q/q_j)^-1]_{q_j} (Q/q_j) mod Q, then the word-wise
// signed sum scaled by inv_scale * 2^(64 j).
// LT > 0: the limb count is fixed, and the words stay in registers; LT = 0: any count.
constexpr int MAXW = 34;
constexpr int MAX_COMPOSE_LT = 12;
template <int LT>
__global__ void __launch_bounds__(128) ckks_compose(const uint64_t *__restrict__ coeff, double *__restrict__ out,
                                                    uint64_t ostride, const Mod *__restrict__ mods,
                                                    const uint64_t *__restrict__ consts, int L_, int logn,
                                                    double inv_scale, uint64_t B) {
    constexpr int NW = LT > 0 ? LT + 1 : MAXW, UNROLL = LT > 0 ? NW : 1;
    const int L = LT > 0 ? LT : L_;
    const uint64_t *ip = consts, *punct = consts + 2 * L, *Qw = punct + L * L, *thr = Qw + L;
    const uint32_t n = 1u << logn;
    const uint64_t total = B << logn;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < total; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = w >> logn;
        const uint32_t i = (uint32_t)(w & (n - 1));
        uint64_t x[NW];
#pragma unroll UNROLL
        for (int k = 0; k < NW; k++) {
            if (k > L) break;
            x[k] = 0;
        }
        for (int j = 0; j < L; j++) {
            const uint64_t q = mods[j].value;
            const uint64_t t = mul_shoup(coeff[((b * L + j) << logn) + i], ip[2 * j], ip[2 * j + 1], q);
            // x += t * punct_j (L words)
            uint64_t carry = 0;
#pragma unroll UNROLL
            for (int k = 0; k < NW - 1; k++) {
                if (k >= L) break;
                const uint64_t pk = punct[j * L + k];
                const uint64_t lo = t * pk, hi = mulhi(t, pk);
                uint64_t s = x[k] + lo;
                uint64_t c1 = s < lo;
                s += carry;
                c1 += s < carry;
                x[k] = s;
                carry = hi + c1;
            }
            x[L] += carry;
        }
        // reduce mod Q: x < L Q, subtract Q while x >= Q
        for (int rep = 0; rep < L + 1; rep++) {
            bool ge = x[L] != 0, decided = ge;
#pragma unroll UNROLL
            for (int k = NW - 2; k >= 0; k--) {
                if (k >= L) continue;
                if (!decided && x[k] != Qw[k]) {
                    ge = x[k] > Qw[k];
                    decided = true;
                }
            }
            if (decided && !ge) break;
            uint64_t borrow = 0;
#pragma unroll UNROLL
            for (int k = 0; k < NW - 1; k++) {
                if (k >= L) break;
                const uint64_t d = x[k] - Qw[k] - borrow;
                borrow = (x[k] < Qw[k]) || (x[k] - Qw[k] < borrow);
                x[k] = d;
            }
            x[L] -= borrow;
        }
        // compare with the upper-half threshold (Q + 1) / 2
        bool upper = true, decided = false;
#pragma unroll UNROLL
        for (int k = NW - 2; k >= 0; k--) {
            if (k >= L) continue;
            if (!decided && x[k] != thr[k]) {
                upper = x[k] > thr[k];
                decided = true;
            }
        }
        double res = 0.0, sc = inv_scale;
        const double two64 = 18446744073709551616.0;
#pragma unroll UNROLL
        for (int k = 0; k < NW - 1; k++) {
            if (k >= L) break;
            if (upper) {
                if (x[k] > Qw[k]) {
                    const uint64_t d = x[k] - Qw[k];
                    res = __dadd_rn(res, d ? __dmul_rn((double)d, sc) : 0.0);
                } else {
                    const uint64_t d = Qw[k] - x[k];
                    res = __dsub_rn(res, d ? __dmul_rn((double)d, sc) : 0.0);
                }
            } else {
                res = __dadd_rn(res, x[k] ? __dmul_rn((double)x[k], sc) : 0.0);
            }
            sc = __dmul_rn(sc, two64);
        }
        out[b * ostride + i] = res;
    }
}

// a[b][i] = (v[b][i] * scale, 0) for i < count, 0 elsewhere (coefficient encode).
__global__ void ckks_load_real(const double *__restrict__ vals, uint64_t vstride, uint32_t count, double scale,
                               double2 *__restrict__ out, int logn, uint64_t B) {
    const uint32_t n = 1u << logn;
    const uint64_t total = B << logn;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < total; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = w >> logn;
        const uint32_t i = (uint32_t)(w & (n - 1));
        out[w] = make_double2(i < count ? __dmul_rn(vals[b * vstride + i], scale) : 0.0, 0.0);
    }
}

}  // namespace

// Complex root tables of the special FFT (CKKSEncoder constructor, src/ckks.cpp:62-77).
static std::mutex g_ckks_mu;

static int ckks_tables(Context &c, double2 **roots, double2 **iroots) {
    std::lock_guard<std::mutex> g(g_ckks_mu);
    if (!c.d_fft_roots) {
        const uint32_t n = c.n;
        const uint64_t m = 2ull * n;
        const double PI = 3.1415926535897932384626433832795028842;
        std::vector<std::complex<double>> base(m / 8 + 1);
        for (size_t i = 0; i <= m / 8; i++) base[i] = std::polar<double>(1.0, 2 * PI * (double)i / (double)m);
        std::function<std::complex<double>(uint64_t)> get = [&](uint64_t idx) -> std::complex<double> {
            idx &= m - 1;
            if (idx <= m / 8) return base[idx];
            if (idx <= m / 4) {
                auto a = base[m / 4 - idx];
                return {a.imag(), a.real()};
            }
            if (idx <= m / 2) return -std::conj(get(m / 2 - idx));
            if (idx <= 3 * m / 4) return -get(idx - m / 2);
            return std::conj(get(m - idx));
        };
        std::vector<double2> r(2ull * n, make_double2(0, 0));   // forward, inverse
        double2 *ir = r.data() + n;
        if (m >= 8) {
            for (uint32_t i = 1; i < n; i++) {
                auto a = get(host::bitrev(i, c.logn));
                auto b = std::conj(get(host::bitrev(i - 1, c.logn) + 1));
                r[i] = make_double2(a.real(), a.imag());
                ir[i] = make_double2(b.real(), b.imag());
            }
        } else if (m == 4) {
            r[1] = make_double2(0, 1);
            ir[1] = make_double2(0, -1);
        }
        double2 *d = nullptr;
        const cudaError_t e = to_device(r.data(), r.size(), &d);
        if (e != cudaSuccess) return status_from(e);
        c.d_fft_roots = d;
    }
    *roots = (double2 *)c.d_fft_roots;
    *iroots = (double2 *)c.d_fft_roots + c.n;
    return TB_OK;
}

static int total_bits(const Context &c, int L) {
    return host::bit_count(host::product(c.chain.data(), L));
}

// Rounds the real parts of buf [B][N], after the last h inverse FFT stages, into plaintexts
// [B][L][N] and transforms them; fails with "encoded values are too large" when a
// coefficient reaches the modulus. The check's result is read after the last launch.
static int round_reduce_ntt(Context &c, int L, double2 *buf, const double2 *iroots, int h, double scalar, uint64_t *out,
                            uint64_t B, cudaStream_t s) {
    int *err = nullptr;
    cudaError_t e = cudaMallocAsync(&err, sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), s);
    if (e != cudaSuccess) return status_from(e);
    const int bits = total_bits(c, L);
    const unsigned grid = grid_for((B * c.n) >> h, 256);
    if (h == 0) ckks_round_reduce<0><<<grid, 256, 0, s>>>(buf, iroots, out, c.d_mods, L, c.logn, B, err, bits, scalar);
    else if (h == 1) ckks_round_reduce<1><<<grid, 256, 0, s>>>(buf, iroots, out, c.d_mods, L, c.logn, B, err, bits, scalar);
    else if (h == 2) ckks_round_reduce<2><<<grid, 256, 0, s>>>(buf, iroots, out, c.d_mods, L, c.logn, B, err, bits, scalar);
    else ckks_round_reduce<3><<<grid, 256, 0, s>>>(buf, iroots, out, c.d_mods, L, c.logn, B, err, bits, scalar);
    int r = ntt_forward(c, out, out, B, 0, L, false, s);
    int herr = 0;
    e = cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaFreeAsync(err, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return status_from(e);
    if (herr) return set_error(TB_ERR_INVALID_ARGUMENT, "encoded values are too large");
    return r;
}

// values [B][vstride] complex (count used) -> plaintexts [B][L][N], NTT form.
int ckks_encode(Context &c, int L, const double *values, uint64_t vstride, uint32_t count, double scale, uint64_t *out,
                uint64_t B, cudaStream_t s) {
    if (c.scheme != SCHEME_CKKS) return set_error(TB_ERR_UNSUPPORTED, "unsupported scheme");
    const uint32_t n = c.n;
    if (L < 1 || L > (int)c.chain.size()) return set_error(TB_ERR_INVALID_ARGUMENT, "level outside the chain");
    if (count > n / 2) return set_error(TB_ERR_INVALID_ARGUMENT, "values_size is too large");
    if (!(scale > 0) || (int)std::log2(scale) + 1 >= total_bits(c, L))
        return set_error(TB_ERR_INVALID_ARGUMENT, "scale out of bounds");
    if (!out || (count && !values)) return set_error(TB_ERR_INVALID_ARGUMENT, "null buffer");
    if (!B) return TB_OK;
    if (!vstride) vstride = count;
    const uint32_t *map = nullptr;
    double2 *roots, *iroots;
    int r = slot_map(c, &map);
    if (r == TB_OK) r = ckks_tables(c, &roots, &iroots);
    if (r != TB_OK) return r;
    ensure_pool_retains(c.device);
    double2 *buf = nullptr;
    cudaError_t e = cudaMallocAsync(&buf, B * n * sizeof(double2), s);
    if (e != cudaSuccess) return status_from(e);
    {
        TraceScope ts("ckks_encode", s);
        const int logb = std::min(c.logn, FFT_LOGB);
        const size_t smem = sizeof(double2) << logb;
        if (smem > 48 * 1024) e = cudaFuncSetAttribute(fft_inv_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        for (uint64_t b0 = 0; e == cudaSuccess && b0 < B; b0 += 65535) {
            const unsigned nb = (unsigned)std::min<uint64_t>(B - b0, 65535);
            fft_inv_block<<<dim3(n >> logb, nb), FFT_THREADS, smem, s>>>((const double2 *)values + b0 * vstride, vstride,
                                                                         count, buf + b0 * n, iroots, map + n, c.logn,
                                                                         logb, scale / (double)n);
            e = cudaGetLastError();
        }
        // degrees above 2^15: the stages between the blocks' and the last three
        for (int st = logb; st < c.logn - 3; st++)
            fft_inv_stage<<<grid_for(B * n / 2, 256), 256, 0, s>>>(buf, iroots, c.logn, st, scale / (double)n, B);
    }
    r = e == cudaSuccess ? round_reduce_ntt(c, L, buf, iroots, std::min(3, std::max(0, c.logn - FFT_LOGB)),
                                            scale / (double)n, out, B, s)
                         : status_from(e);
    cudaFreeAsync(buf, s);
    return r;
}

// Real coefficients [B][vstride] (count <= N used) times scale, rounded, reduced and
// transformed: CKKSEncoderCuda::encodePolynomialInternal (src/ckks_cuda.cu:455-565).
int ckks_encode_polynomial(Context &c, int L, const double *values, uint64_t vstride, uint32_t count, double scale,
                           uint64_t *out, uint64_t B, cudaStream_t s) {
    if (c.scheme != SCHEME_CKKS) return set_error(TB_ERR_UNSUPPORTED, "unsupported scheme");
    if (L < 1 || L > (int)c.chain.size()) return set_error(TB_ERR_INVALID_ARGUMENT, "level outside the chain");
    if (count > c.n) return set_error(TB_ERR_INVALID_ARGUMENT, "values_size is too large");
    if (!out || (count && !values)) return set_error(TB_ERR_INVALID_ARGUMENT, "null buffer");
    if (!B) return TB_OK;
    if (!vstride) vstride = count;
    ensure_pool_retains(c.device);
    double2 *buf = nullptr;
    cudaError_t e = cudaMallocAsync(&buf, B * c.n * sizeof(double2), s);
    if (e != cudaSuccess) return status_from(e);
    {
        TraceScope ts("ckks_encode", s);
        ckks_load_real<<<grid_for(B * c.n, 256), 256, 0, s>>>(values, vstride, count, scale, buf, c.logn, B);
    }
    const int r = round_reduce_ntt(c, L, buf, nullptr, 0, 1.0, out, B, s);
    cudaFreeAsync(buf, s);
    return r;
}

int fill_limbs(Context &c, int L, const uint64_t *vals, uint64_t *out, uint64_t B, cudaStream_t s);

// |x| mod q for a non-negative integral double x, through its base-2^64 digits.
static uint64_t double_mod(double x, uint64_t q) {
    const double two64 = 18446744073709551616.0;
    std::vector<uint64_t> words;
    while (x >= 1) {
        words.push_back((uint64_t)std::fmod(x, two64));
        x /= two64;
    }
    unsigned __int128 r = 0;
    for (size_t k = words.size(); k-- > 0;) r = ((r << 64) | words[k]) % q;
    return (uint64_t)r;
}

// The constant round(value * scale) in every slot: every NTT coefficient of limb l
// equals the constant mod q_l (CKKSEncoder::encodeInternal(double), src/ckks.cpp:279-400).
int ckks_encode_double(Context &c, int L, double value, double scale, uint64_t *out, cudaStream_t s) {
    if (c.scheme != SCHEME_CKKS) return set_error(TB_ERR_UNSUPPORTED, "unsupported scheme");
    if (L < 1 || L > (int)c.chain.size()) return set_error(TB_ERR_INVALID_ARGUMENT, "level outside the chain");
    const int bits = total_bits(c, L);
    if (!(scale > 0) || (int)std::log2(scale) >= bits) return set_error(TB_ERR_INVALID_ARGUMENT, "scale out of bounds");
    value *= scale;
    if (value != 0.0 && (int)std::log2(std::fabs(value)) + 2 >= bits)
        return set_error(TB_ERR_INVALID_ARGUMENT, "encoded value is too large");
    double cd = std::round(value);
    const bool neg = std::signbit(cd);
    cd = std::fabs(cd);
    std::vector<uint64_t> vals(L);
    for (int l = 0; l < L; l++) {
        const uint64_t q = c.chain[l];
        const uint64_t r = double_mod(cd, q);
        vals[l] = (neg && r) ? q - r : r;
    }
    TraceScope ts("ckks_encode", s);
    return fill_limbs(c, L, vals.data(), out, 1, s);
}

// The integer `value` in every slot, scale 1 (CKKSEncoder::encodeInternal(int64_t),
// src/ckks.cpp:402-440): residue ((uint64)value + q) mod q for negative values.
int ckks_encode_int64(Context &c, int L, int64_t value, uint64_t *out, cudaStream_t s) {
    if (c.scheme != SCHEME_CKKS) return set_error(TB_ERR_UNSUPPORTED, "unsupported scheme");
    if (L < 1 || L > (int)c.chain.size()) return set_error(TB_ERR_INVALID_ARGUMENT, "level outside the chain");
    const uint64_t mag = value < 0 ? 0 - (uint64_t)value : (uint64_t)value;
    if (host::bit_count(mag) + 2 >= total_bits(c, L))
        return set_error(TB_ERR_INVALID_ARGUMENT, "encoded value is too large");
    std::vector<uint64_t> vals(L);
    for (int l = 0; l < L; l++) {
        const uint64_t q = c.chain[l];
        const uint64_t fill = value < 0 ? (uint64_t)value + q : (uint64_t)value;
        vals[l] = fill % q;
    }
    TraceScope ts("ckks_encode", s);
    return fill_limbs(c, L, vals.data(), out, 1, s);
}

// CRT constants of level L: pairs (Q/q_j)^-1 mod q_j, the words of Q/q_j, of Q and of the
// threshold (Q + 1) / 2, built and uploaded on first use.
static int compose_consts(Context &c, int L, const uint64_t **out) {
    using namespace host;
    std::lock_guard<std::mutex> g(g_ckks_mu);
    RnsLevel &lv = c.levels[L];
    if (!lv.d_compose) {
        const uint64_t *q = c.chain.data();
        auto Q = product(q, L);
        Q.resize(L, 0);
        std::vector<uint64_t> hc(2 * L + L * L + L + L);
        for (int j = 0; j < L; j++) {
            const uint64_t ipj = invmod(punctured_mod(q, L, j, q[j]), q[j]);
            hc[2 * j] = ipj;
            hc[2 * j + 1] = shoup(ipj, q[j]);
            uint64_t rem = 0;
            auto pj = div_words(Q, q[j], rem);
            pj.resize(L, 0);
            for (int k = 0; k < L; k++) hc[2 * L + j * L + k] = pj[k];
        }
        for (int k = 0; k < L; k++) hc[2 * L + L * L + k] = Q[k];
        std::vector<uint64_t> t(Q);
        int k = 0;
        while (k < L && ++t[k] == 0) k++;
        uint64_t carry = 0;
        for (int i = L - 1; i >= 0; i--) {
            const uint64_t v = t[i];
            t[i] = (v >> 1) | (carry << 63);
            carry = v & 1;
        }
        for (int i = 0; i < L; i++) hc[2 * L + L * L + L + i] = t[i];
        const cudaError_t e = to_device(hc.data(), hc.size(), &lv.d_compose);
        if (e != cudaSuccess) return status_from(e);
    }
    *out = lv.d_compose;
    return TB_OK;
}

template <int LT>
static void launch_compose(int L, const uint64_t *coeff, double *out, uint64_t ostride, const Context &c,
                           const uint64_t *consts, double inv_scale, uint64_t B, cudaStream_t s) {
    if constexpr (LT > 0) {
        if (L != LT) return launch_compose<LT - 1>(L, coeff, out, ostride, c, consts, inv_scale, B, s);   // ends at 0
    }
    ckks_compose<LT><<<grid_for(B * c.n, 128), 128, 0, s>>>(coeff, out, ostride, c.d_mods, consts, L, c.logn, inv_scale, B);
}

// Inverse NTT, CRT compose, centre and scale by 1/scale: out [B][ostride] real coefficients.
static int compose_level(Context &c, int L, const uint64_t *plain, double scale, double *out, uint64_t ostride,
                         uint64_t B, cudaStream_t s) {
    const uint64_t *consts = nullptr;
    int r = refuse_capture(s);
    if (r == TB_OK) r = compose_consts(c, L, &consts);
    if (r != TB_OK) return r;
    uint64_t *tmp = nullptr;
    cudaError_t e = cudaMallocAsync(&tmp, 8ull * B * L * c.n, s);
    if (e != cudaSuccess) return status_from(e);
    // the transform loads pairs of words; a plaintext that starts inside a pair is copied first
    if (reinterpret_cast<uintptr_t>(plain) & 15) {
        r = status_from(cudaMemcpyAsync(tmp, plain, 8ull * B * L * c.n, cudaMemcpyDeviceToDevice, s));
        plain = tmp;
    }
    if (r == TB_OK) r = ntt_inverse(c, plain, tmp, B, 0, L, false, s);
    if (r == TB_OK) {
        TraceScope ts("ckks_decode", s);
        launch_compose<MAX_COMPOSE_LT>(L, tmp, out, ostride, c, consts, 1.0 / scale, B, s);
        r = status_from(cudaGetLastError());
    }
    cudaFreeAsync(tmp, s);
    return r;
}

static int decode_checks(const Context &c, int L, const uint64_t *plain, double scale, const double *values) {
    if (c.scheme != SCHEME_CKKS) return set_error(TB_ERR_UNSUPPORTED, "unsupported scheme");
    if (L < 1 || L > (int)c.chain.size() || L + 1 > MAXW) return set_error(TB_ERR_INVALID_ARGUMENT, "bad level");
    if (!(scale > 0) || (int)std::log2(scale) >= total_bits(c, L))
        return set_error(TB_ERR_INVALID_ARGUMENT, "scale out of bounds");
    if (!plain || !values) return set_error(TB_ERR_INVALID_ARGUMENT, "null buffer");
    return TB_OK;
}

// plaintexts [B][L][N] (NTT form) -> slot values [B][ostride] complex (N/2 used).
int ckks_decode(Context &c, int L, const uint64_t *plain, double scale, double *values, uint64_t ostride, uint64_t B,
                cudaStream_t s) {
    int r = decode_checks(c, L, plain, scale, values);
    if (r != TB_OK || !B) return r;
    const uint32_t n = c.n;
    if (!ostride) ostride = n / 2;
    const uint32_t *map = nullptr;
    double2 *roots, *iroots;
    r = slot_map(c, &map);
    if (r == TB_OK) r = ckks_tables(c, &roots, &iroots);
    if (r != TB_OK) return r;
    ensure_pool_retains(c.device);
    const int logb = std::min(c.logn, FFT_LOGB), top = c.logn - logb, h = std::min(top, 3);
    // real coefficients, and complex points where stages come before the last three (N > 2^15)
    double *buf = nullptr;
    cudaError_t e = cudaMallocAsync(&buf, B * n * (top > 3 ? sizeof(double) + sizeof(double2) : sizeof(double)), s);
    if (e != cudaSuccess) return status_from(e);
    r = compose_level(c, L, plain, scale, buf, n, B, s);
    if (r == TB_OK) {
        TraceScope ts("ckks_decode", s);
        double2 *pts = nullptr;
        if (top > 3) {
            pts = (double2 *)(buf + B * n);
            ckks_load_real<<<grid_for(B * n, 256), 256, 0, s>>>(buf, n, n, 1.0, pts, c.logn, B);
            for (int st = 0; st < top - 3; st++)
                fft_fwd_stage<<<grid_for(B * n / 2, 256), 256, 0, s>>>(pts, roots, c.logn, st, B);
        }
        auto kernel = h == 0 ? fft_fwd_block<0> : h == 1 ? fft_fwd_block<1> : h == 2 ? fft_fwd_block<2> : fft_fwd_block<3>;
        const size_t smem = sizeof(double2) << logb;
        e = cudaGetLastError();
        if (e == cudaSuccess && smem > 48 * 1024)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        for (uint64_t b0 = 0; e == cudaSuccess && b0 < B; b0 += 65535) {
            const unsigned nb = (unsigned)std::min<uint64_t>(B - b0, 65535);
            kernel<<<dim3(n >> logb, nb), FFT_THREADS, smem, s>>>(pts ? pts + b0 * n : nullptr, pts ? nullptr : buf + b0 * n,
                                                                  (double2 *)values + b0 * ostride, ostride, roots, map + n,
                                                                  c.logn, logb);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) r = status_from(e);
    }
    cudaFreeAsync(buf, s);
    return r;
}

// plaintexts [B][L][N] (NTT form) -> N real coefficients each, divided by scale
// (CKKSEncoderCuda::decodePolynomialInternal, src/ckks_cuda.cu:983-1040).
int ckks_decode_polynomial(Context &c, int L, const uint64_t *plain, double scale, double *values, uint64_t ostride,
                           uint64_t B, cudaStream_t s) {
    int r = decode_checks(c, L, plain, scale, values);
    if (r != TB_OK || !B) return r;
    const uint32_t n = c.n;
    if (!ostride) ostride = n;
    ensure_pool_retains(c.device);
    return compose_level(c, L, plain, scale, values, ostride, B, s);
}

}  // namespace tb
