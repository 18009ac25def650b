// Device-side PRNG stream and samplers.
//
// The reference's Blake2xbPRNG (src/randomgen.cpp:188-198) emits the concatenation
// of 4096-byte BLAKE2Xb outputs keyed by the 64-byte seed with the 8-byte
// little-endian counter 0, 1, 2, ... as message. That makes the stream counter
// based: byte p lives in refill p / 4096, output block (p % 4096) / 64, and every
// 64-byte block is one BLAKE2b compression of the refill's root hash. prng_fill
// computes any byte range in parallel (four lanes per 64-byte block; BLAKE2b as in
// RFC 7693, BLAKE2X parameters per the BLAKE2X specification).
//
// A PRNG is a device-resident PrngState {seed, offset}: samplers read the offset,
// consume bytes and advance it, so data-dependent consumption (rejection sampling)
// needs no host round trip. The samplers reproduce the reference's consumption
// exactly (src/utils/rlwe.cpp:21-150): ternary draws 32-bit words through
// libstdc++'s uniform_int_distribution<uint64_t>(0, 2), which rejects only a zero
// word; CBD takes 6 bytes per coefficient; uniform takes L*N 64-bit words, then
// replaces each rejected word, in order, by the next acceptable word of the stream.
#include <cstring>
#include <random>

#include "context.hpp"
#include "prng.hpp"
#include "trace.cuh"

namespace tb {

unsigned grid_for(uint64_t work, int threads);

namespace {

__constant__ uint64_t c_iv[8] = {0x6a09e667f3bcc908ULL, 0xbb67ae8584caa73bULL, 0x3c6ef372fe94f82bULL,
                                 0xa54ff53a5f1d36f1ULL, 0x510e527fade682d1ULL, 0x9b05688c2b3e6c1fULL,
                                 0x1f83d9abfb41bd6bULL, 0x5be0cd19137e2179ULL};
__constant__ __align__(16) uint8_t c_sigma[12][16] = {
    {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3},
    {11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4}, {7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8},
    {9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13}, {2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9},
    {12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11}, {13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10},
    {6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5}, {10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0},
    {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3}};

__device__ __forceinline__ uint64_t rotr(uint64_t x, int c) { return (x >> c) | (x << (64 - c)); }

// BLAKE2b by four lanes: lane l of a quad holds column l of the state (words l, 4 + l, 8 + l,
// 12 + l), runs one G of the column step and, after rotating the rows by shuffles, one of
// the diagonal step. A compression is a chain of 24 G steps either way, but one thread
// issues all eight G of a round, and a warp that runs alone (the root hashes; a single
// encryption's stream) is bound by its own issue rate: a quad issues a quarter of that. The
// message is in shared memory, m[0 .. 15]; sg[r] holds the lane's four message indices of
// round r. Generating the 64 KB of one encryption at N = 4096: 60 us in three launches with
// one thread per block and the message in local memory, 23 us in one launch with one thread
// per block and the message in shared memory, 15 us with quads.
constexpr int FILL_THREADS = 256;
constexpr int FILL_QUADS = FILL_THREADS / 4;   // 64: the blocks of one refill
constexpr int FILL_REFILLS = 4;                // most refills of a CTA
constexpr int MSG = 17;                        // words between the quads' messages (no bank conflicts)

__device__ __forceinline__ void b2_sigma(uint32_t (&sg)[10]) {
    const int l = threadIdx.x & 3;
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint8_t *s = c_sigma[r];
        sg[r] = s[2 * l] | (uint32_t)s[2 * l + 1] << 8 | (uint32_t)s[8 + 2 * l] << 16 | (uint32_t)s[9 + 2 * l] << 24;
    }
}

__device__ __forceinline__ void b2_g(uint64_t &a, uint64_t &b, uint64_t &c, uint64_t &d, uint64_t x, uint64_t y) {
    a = a + b + x;
    d = rotr(d ^ a, 32);
    c = c + d;
    b = rotr(b ^ c, 24);
    a = a + b + y;
    d = rotr(d ^ a, 16);
    c = c + d;
    b = rotr(b ^ c, 63);
}

// lo, hi: words l and 4 + l of the chain value.
__device__ __noinline__ void b2_compress(uint64_t &lo, uint64_t &hi, const uint64_t *m, const uint32_t (&sg)[10], uint64_t t,
                                         bool last) {
    const int l = threadIdx.x & 3;
    uint64_t a = lo, b = hi, c = c_iv[l], d = c_iv[4 + l];
    if (l == 0) d ^= t;
    if (l == 2 && last) d = ~d;
#pragma unroll
    for (int r = 0; r < 12; r++) {
        const uint32_t s = sg[r % 10];
        const uint64_t x0 = m[s & 255], y0 = m[(s >> 8) & 255], x1 = m[(s >> 16) & 255], y1 = m[s >> 24];
        b2_g(a, b, c, d, x0, y0);
        b = __shfl_sync(0xffffffffu, b, l + 1, 4);
        c = __shfl_sync(0xffffffffu, c, l + 2, 4);
        d = __shfl_sync(0xffffffffu, d, l + 3, 4);
        b2_g(a, b, c, d, x1, y1);
        b = __shfl_sync(0xffffffffu, b, l + 3, 4);
        c = __shfl_sync(0xffffffffu, c, l + 2, 4);
        d = __shfl_sync(0xffffffffu, d, l + 1, 4);
    }
    lo ^= a ^ c;
    hi ^= b ^ d;
}

// buf[k] = stream[st->offset + k] for k < nbytes, for each of `count` states (blockIdx.y).
// One CTA per `per` <= FILL_REFILLS refills of 4096 bytes: their root hashes (two
// compressions each) by the first quads, side by side, then one output node per quad and
// refill.
__global__ void __launch_bounds__(FILL_THREADS) prng_fill_kernel(const PrngState *__restrict__ st, uint8_t *__restrict__ buf,
                                                                 uint64_t nbytes, uint64_t bstride, int per) {
    __shared__ uint64_t msg[MSG * FILL_QUADS], root[8 * FILL_REFILLS];
    const PrngState &s = st[blockIdx.y];
    const uint64_t off = s.offset, xof = 4096;
    const uint64_t end = (off + nbytes + 4095) >> 12;
    uint8_t *b = buf + blockIdx.y * bstride;
    const int l = threadIdx.x & 3, quad = threadIdx.x >> 2;
    uint64_t *m = msg + MSG * quad;
    uint32_t sg[10];
    b2_sigma(sg);
    for (uint64_t first = (off >> 12) + (uint64_t)per * blockIdx.x; first < end; first += (uint64_t)per * gridDim.x) {
        __syncthreads();   // the previous refills' roots and messages are read
        if (threadIdx.x < 32) {   // the roots of refills first .. first + 3 (a whole warp: shuffles)
            uint64_t lo = c_iv[l], hi = c_iv[4 + l];
            // root: digest 64, key 64, fanout 1, depth 1, leaf 0; node offset 0, xof length 4096
            if (l == 0) lo ^= 64ull | (64ull << 8) | (1ull << 16) | (1ull << 24);
            if (l == 1) lo ^= xof << 32;
#pragma unroll
            for (int i = 0; i < 4; i++) m[4 * i + l] = i < 2 ? s.seed[4 * i + l] : 0;
            __syncwarp();
            b2_compress(lo, hi, m, sg, 128, false);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++) m[4 * i + l] = i == 0 && l == 0 ? first + quad : 0;
            __syncwarp();
            b2_compress(lo, hi, m, sg, 136, true);
            if (quad < FILL_REFILLS) {
                root[8 * quad + l] = lo;
                root[8 * quad + 4 + l] = hi;
            }
        }
        __syncthreads();
        for (int f = 0; f < per && first + f < end; f++) {
            // output node: digest 64, leaf length 64, node offset, xof 4096, inner length 64
            uint64_t lo = c_iv[l], hi = c_iv[4 + l];
            if (l == 0) lo ^= 64ull | (64ull << 32);
            if (l == 1) lo ^= (uint64_t)quad | (xof << 32);
            if (l == 2) lo ^= 64ull << 8;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++) m[4 * i + l] = i < 2 ? root[8 * f + 4 * i + l] : 0;
            __syncwarp();
            b2_compress(lo, hi, m, sg, 64, true);
            const uint64_t at = ((first + f) << 12) + ((uint64_t)quad << 6) + 8 * l;   // and 32 bytes on
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint64_t p = at + 32 * h, w = h ? hi : lo;
                if (p >= off && p + 8 <= off + nbytes && ((p - off) & 7) == 0) {
                    *reinterpret_cast<uint64_t *>(b + (p - off)) = w;
                } else {
                    for (int k = 0; k < 8; k++)
                        if (p + k >= off && p + k < off + nbytes) b[p + k - off] = (uint8_t)(w >> (8 * k));
                }
            }
        }
    }
}

// The small polynomials of an encryption as signed values: one ternary polynomial and two
// of the centred binomial distribution from the start of each state's stream (offset 0).
// The stream's first 16 N bytes are all they read unless a ternary word is rejected
// (probability 2^-32 a word), which encrypt_fixup_kernel handles: the state is flagged
// here and its polynomials are redone there.
__device__ __forceinline__ int ternary_of(uint32_t w) { return (int)(((uint64_t)w * 3u) >> 32) - 1; }

__device__ __forceinline__ int cbd_of(const uint8_t *x) {
    return __popc(x[0]) + __popc(x[1]) + __popc(x[2] & 0x1f) - __popc(x[3]) - __popc(x[4]) - __popc(x[5] & 0x1f);
}

__global__ void __launch_bounds__(128) encrypt_small_kernel(const uint8_t *__restrict__ buf, uint64_t bstride, uint32_t n,
                                                            int32_t *__restrict__ small, PrngState *st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint8_t *b = buf + blockIdx.y * bstride;
    int32_t *o = small + 3ull * n * blockIdx.y;
    const uint32_t w = reinterpret_cast<const uint32_t *>(b)[i];
    if (w == 0) atomicOr(&st[blockIdx.y].flag, 1u);
    o[i] = ternary_of(w);
    o[n + i] = cbd_of(b + 4ull * n + 6ull * i);
    o[2 * n + i] = cbd_of(b + 10ull * n + 6ull * i);
}

// A flagged state's polynomials by one thread: every ternary coefficient takes the next
// non-zero word, and the binomial bytes follow the last word taken. The buffer holds 64
// words more than a state without rejections needs.
__global__ void encrypt_fixup_kernel(const uint8_t *__restrict__ buf, uint64_t bstride, uint64_t nbytes, uint32_t n,
                                     int32_t *__restrict__ small, PrngState *st) {
    PrngState &s = st[blockIdx.x];
    if (threadIdx.x != 0 || !(s.flag & 1)) return;
    const uint8_t *b = buf + blockIdx.x * bstride;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(b);
    int32_t *o = small + 3ull * n * blockIdx.x;
    uint64_t p = 0;
    for (uint32_t i = 0; i < n; i++) {
        uint32_t x;
        do {
            if (4 * (p + 1) + 12ull * n > nbytes) {
                s.flag = 2;   // stream window exhausted
                return;
            }
            x = w[p++];
        } while (x == 0);
        o[i] = ternary_of(x);
    }
    for (uint32_t i = 0; i < 2 * n; i++) o[n + i] = cbd_of(b + 4 * p + 6ull * i);
    s.flag = 0;
}

// Seeds by kernel parameter: states first .. first + count - 1 start at offset 0.
constexpr int SEEDS_PER_LAUNCH = 32;
struct SeedBlock {
    uint64_t w[SEEDS_PER_LAUNCH][8];
};

__global__ void prng_seed_kernel(PrngState *st, SeedBlock seeds, int same) {
    PrngState &s = st[blockIdx.x];
    if (threadIdx.x < 8) s.seed[threadIdx.x] = seeds.w[same ? 0 : blockIdx.x][threadIdx.x];
    if (threadIdx.x == 8) {
        s.offset = 0;
        s.flag = 0;
        s.pad = 0;
    }
}

// Ternary sampling; a zero word would be rejected by the distribution, which the
// fix-up pass then handles sequentially (probability 2^-32 per word).
__global__ void ternary_kernel(const uint8_t *__restrict__ buf, uint64_t bstride, uint32_t n,
                               const Mod *__restrict__ mods, int L, uint64_t *__restrict__ out, uint64_t ostride,
                               PrngState *st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint8_t *b = buf + blockIdx.y * bstride;
    uint64_t *o = out + blockIdx.y * ostride;
    const uint32_t w = reinterpret_cast<const uint32_t *>(b)[i];
    if (w == 0) atomicOr(&st[blockIdx.y].flag, 1u);
    const uint64_t r = ((uint64_t)w * 3u) >> 32;
    for (int j = 0; j < L; j++) o[(size_t)j * n + i] = r == 0 ? mods[j].value - 1 : r - 1;
}

__global__ void ternary_fixup_kernel(const uint8_t *__restrict__ buf, uint64_t bstride, uint64_t avail_words,
                                     uint32_t n, const Mod *__restrict__ mods, int L, uint64_t *__restrict__ out,
                                     uint64_t ostride, PrngState *st) {
    PrngState &s = st[blockIdx.x];
    if (threadIdx.x != 0) return;
    if (!(s.flag & 1)) {
        s.offset += 4ull * n;
        return;
    }
    const uint32_t *w = reinterpret_cast<const uint32_t *>(buf + blockIdx.x * bstride);
    uint64_t *o = out + blockIdx.x * ostride;
    uint64_t p = 0;
    for (uint32_t i = 0; i < n; i++) {
        uint32_t x;
        do {
            if (p >= avail_words) {
                s.flag = 2;  // more rejections (2^-32 a word) than the window has words to spare
                return;
            }
            x = w[p++];
        } while (x == 0);
        const uint64_t r = ((uint64_t)x * 3u) >> 32;
        for (int j = 0; j < L; j++) o[(size_t)j * n + i] = r == 0 ? mods[j].value - 1 : r - 1;
    }
    s.offset += 4 * p;
    s.flag = 0;
}

// Centered binomial, 6 bytes per coefficient (src/utils/rlwe.cpp:89-104).
__global__ void cbd_kernel(const uint8_t *__restrict__ buf, uint64_t bstride, uint32_t n,
                           const Mod *__restrict__ mods, int L, uint64_t *__restrict__ out, uint64_t ostride) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint8_t *x = buf + blockIdx.y * bstride + 6ull * i;
    uint64_t *o = out + blockIdx.y * ostride;
    const int v = __popc(x[0]) + __popc(x[1]) + __popc(x[2] & 0x1f) - __popc(x[3]) - __popc(x[4]) -
                  __popc(x[5] & 0x1f);
    for (int j = 0; j < L; j++) o[(size_t)j * n + i] = v < 0 ? mods[j].value - (uint64_t)(-v) : (uint64_t)v;
}

__global__ void advance_kernel(PrngState *st, uint64_t bytes) { st[blockIdx.x].offset += bytes; }

constexpr uint64_t REJECTED = ~0ull;

// Words below 2^64 - 1 - ((2^64 - 1) mod q) - 1 are accepted for modulus q.
__device__ __forceinline__ uint64_t uniform_limit(const Mod &m) { return ~0ull - reduce64(~0ull, m) - 1; }

// Uniform mod q_j: word (j, i) is accepted below uniform_limit (src/utils/rlwe.cpp:126-149).
__global__ void uniform_kernel(const uint8_t *__restrict__ buf, uint64_t bstride, uint32_t n,
                               const Mod *__restrict__ mods, int L, uint64_t *__restrict__ out, uint64_t ostride,
                               PrngState *st) {
    const uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (idx >= (uint64_t)L * n) return;
    const int j = (int)(idx / n);
    const uint64_t w = reinterpret_cast<const uint64_t *>(buf + blockIdx.y * bstride)[idx];
    uint64_t *o = out + blockIdx.y * ostride;
    if (w >= uniform_limit(mods[j])) {
        o[idx] = REJECTED;
        atomicOr(&st[blockIdx.y].flag, 1u);
    } else {
        o[idx] = reduce64(w, mods[j]);
    }
}

// One warp per state: rejected positions in (limb, coefficient) order take the next
// acceptable words after the first L*N.
__global__ void uniform_fixup_kernel(const uint8_t *__restrict__ buf, uint64_t bstride, uint64_t avail_words,
                                     uint32_t n, const Mod *__restrict__ mods, int L, uint64_t *__restrict__ out,
                                     uint64_t ostride, PrngState *st) {
    PrngState &s = st[blockIdx.x];
    const int lane = threadIdx.x;
    const uint64_t total = (uint64_t)L * n;
    if (!(s.flag & 1)) {
        if (lane == 0) s.offset += 8 * total;
        return;
    }
    const uint64_t *w = reinterpret_cast<const uint64_t *>(buf + blockIdx.x * bstride);
    uint64_t *o = out + blockIdx.x * ostride;
    uint64_t p = total;
    for (int j = 0; j < L; j++) {
        const Mod m = mods[j];
        const uint64_t mm = uniform_limit(m);
        for (uint32_t i0 = 0; i0 < n; i0 += 32) {
            const uint32_t i = i0 + lane;
            unsigned rej = __ballot_sync(0xffffffffu, i < n && o[(uint64_t)j * n + i] == REJECTED);
            while (rej) {
                const int k = __ffs(rej) - 1;
                rej &= rej - 1;
                uint64_t val = 0;
                bool found = false;
                while (!found) {
                    if (p + lane >= avail_words && p >= avail_words) {
                        if (lane == 0) s.flag = 2;
                        return;
                    }
                    const uint64_t x = p + lane < avail_words ? w[p + lane] : REJECTED;
                    const unsigned acc = __ballot_sync(0xffffffffu, p + lane < avail_words && x < mm);
                    if (acc) {
                        const int f = __ffs(acc) - 1;
                        val = __shfl_sync(0xffffffffu, x, f);
                        p += f + 1;
                        found = true;
                    } else {
                        p += 32;
                    }
                }
                if (lane == 0) o[(uint64_t)j * n + i0 + k] = reduce64(val, m);
            }
        }
    }
    __syncwarp();
    if (lane == 0) {
        s.offset += 8 * p;
        s.flag = 0;
    }
}

}  // namespace

// Stream bytes of `count` states: four refills to a CTA where that still gives every SM
// work (a CTA's root hashes then cost one quad group for four refills), else one.
static void launch_fill(const PrngState *st, int count, uint8_t *buf, uint64_t nbytes, uint64_t bstride, cudaStream_t s) {
    const uint64_t refills = (nbytes + 4095) / 4096 + 1;   // a range that starts inside a refill spans one more
    const int per = refills * count >= 592 ? FILL_REFILLS : 1;
    const dim3 grid((unsigned)std::min<uint64_t>((refills + per - 1) / per, 1024), count);
    prng_fill_kernel<<<grid, FILL_THREADS, 0, s>>>(st, buf, nbytes, bstride, per);
}

// Samples `count` polynomials over table moduli [first, first + L) from `count`
// device PRNG states into out (polynomial b at out + b*ostride, [L][N]).
int sample_poly(const Context &c, int kind, PrngState *st, int count, int first, int L, uint64_t *out,
                uint64_t ostride, cudaStream_t s) {
    if (count <= 0) return TB_OK;
    const uint32_t n = c.n;
    if (!ostride) ostride = (uint64_t)L * n;
    uint64_t nbytes;
    if (kind == SAMPLE_TERNARY) nbytes = 4ull * n + 256;
    else if (kind == SAMPLE_CBD) nbytes = 6ull * n;
    else nbytes = 8ull * ((uint64_t)L * n + (uint64_t)L * n / 4 + 1024);
    const uint64_t bstride = (nbytes + 255) & ~255ull;
    uint8_t *buf = nullptr;
    cudaError_t e = cudaMallocAsync(&buf, bstride * count, s);
    if (e != cudaSuccess) return status_from(e);
    const Mod *mods = c.d_mods + first;
    {
        TraceScope ts("prng_fill", s);
        launch_fill(st, count, buf, nbytes, bstride, s);
    }
    TraceScope ts("sample", s);
    if (kind == SAMPLE_TERNARY) {
        dim3 g((n + 255) / 256, count);
        ternary_kernel<<<g, 256, 0, s>>>(buf, bstride, n, mods, L, out, ostride, st);
        ternary_fixup_kernel<<<count, 32, 0, s>>>(buf, bstride, nbytes / 4, n, mods, L, out, ostride, st);
    } else if (kind == SAMPLE_CBD) {
        dim3 g((n + 255) / 256, count);
        cbd_kernel<<<g, 256, 0, s>>>(buf, bstride, n, mods, L, out, ostride);
        advance_kernel<<<count, 1, 0, s>>>(st, 6ull * n);
    } else {
        dim3 g((unsigned)(((uint64_t)L * n + 255) / 256), count);
        uniform_kernel<<<g, 256, 0, s>>>(buf, bstride, n, mods, L, out, ostride, st);
        uniform_fixup_kernel<<<count, 32, 0, s>>>(buf, bstride, nbytes / 8, n, mods, L, out, ostride, st);
    }
    e = cudaGetLastError();
    cudaFreeAsync(buf, s);
    return e == cudaSuccess ? TB_OK : status_from(e);
}

// `nbytes` raw stream bytes of each of `count` states (advances them), `ostride` bytes apart.
int prng_bytes(PrngState *st, int count, uint64_t nbytes, uint8_t *out, uint64_t ostride, cudaStream_t s) {
    launch_fill(st, count, out, nbytes, ostride, s);
    advance_kernel<<<count, 1, 0, s>>>(st, nbytes);
    return status_from(cudaGetLastError());
}

// The ternary and the two binomial polynomials of `count` encryptions from fresh states
// (offset 0) into small [count][3][N].
int sample_encryption(const Context &c, PrngState *st, int count, int32_t *small, cudaStream_t s) {
    const uint32_t n = c.n;
    const uint64_t nbytes = 16ull * n + 256, bstride = (nbytes + 255) & ~255ull;
    uint8_t *buf = nullptr;
    cudaError_t e = cudaMallocAsync(&buf, bstride * count, s);
    if (e != cudaSuccess) return status_from(e);
    {
        TraceScope ts("prng_fill", s);
        launch_fill(st, count, buf, nbytes, bstride, s);
    }
    TraceScope ts("sample", s);
    encrypt_small_kernel<<<dim3((n + 127) / 128, count), 128, 0, s>>>(buf, bstride, n, small, st);
    encrypt_fixup_kernel<<<count, 32, 0, s>>>(buf, bstride, nbytes, n, small, st);
    e = cudaGetLastError();
    cudaFreeAsync(buf, s);
    return status_from(e);
}

// Fresh states: a seeded factory gives every PRNG the same seed and offset 0
// (src/randomgen.h:412-427); without a seed each state gets random bytes. The seeds travel
// as kernel parameters, so nothing is copied and nothing waits.
int prng_init(PrngState *st, int count, const uint64_t *seed8, cudaStream_t s) {
    const int r = refuse_capture(s);   // a graph would replay the same seeds for every run
    if (r != TB_OK) return r;
    SeedBlock b{};
    if (seed8) {
        for (int i = 0; i < 8; i++) b.w[0][i] = seed8[i];
        prng_seed_kernel<<<count, 32, 0, s>>>(st, b, 1);
        return status_from(cudaGetLastError());
    }
    std::random_device rd;
    for (int first = 0; first < count; first += SEEDS_PER_LAUNCH) {
        const int k = std::min(SEEDS_PER_LAUNCH, count - first);
        for (int j = 0; j < k; j++)
            for (int i = 0; i < 8; i++) b.w[j][i] = (uint64_t)rd() << 32 | rd();
        prng_seed_kernel<<<k, 32, 0, s>>>(st + first, b, 0);
    }
    return status_from(cudaGetLastError());
}

}  // namespace tb
