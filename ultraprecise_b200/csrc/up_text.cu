// up_text.cu — decimal text in and out on the GPU.
//
// Parsing follows the reference's string constructor of a typed decimal
// (Decimal::Decimal(precision, scale, mode, str), decimal.cu:158-165): the
// text is read by StringToDecimal (decimal.cu:2980-3025) — an optional
// leading '-', digits and at most one '.'; the magnitude is every digit, the
// scale is the number of digits after the '.' — and then cast to the column's
// scale (Decimal::cast, decimal.cu:471-533): more fraction digits than the
// column keeps are cut off (truncation toward zero, no rounding), fewer are
// padded with zeros.  The compact value keeps the low B(p) bytes with the
// sign in bit 7 of the last byte (ToCompactDecimal, decimal.cu:337-341).
// Where the reference reads past the text or turns other characters into
// digits (a second '.', any non-digit), this parser flags UP_ROWERR_DOMAIN and
// stores 0; lost magnitude bits flag UP_ROWERR_OVERFLOW.
//
// Formatting writes one fixed-width slot per row: either the reference's
// output image (Decimal::GetDecimal, decimal.cu:362-398: '+' or '-', eight
// upper-case hex digits per 32-bit limb from the highest nonzero limb down,
// then the scale as "(fff)"), or the plain decimal string ("-123.4500": a '-'
// when the sign bit is set, the digits, a '.' before the last `scale`
// digits).  The decimal string parses back to the same compact bytes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "../../include/ultraprecise.h"
#include "up_dev.cuh"
#include "up_internal.h"

namespace upi {
namespace {

using u8 = uint8_t;
using u32 = uint32_t;
using u64 = uint64_t;

constexpr int kMaxPrecisionText = 1000;
constexpr int kMaxDigits = 1500;  // digits of one field
// 8960 bits: 1500 digits plus up to 1000 zeros of scale padding
constexpr int kMaxLimbs = 280;

__device__ __forceinline__ void mul_add_small(u32* m, int& nl, u32 k, u32 add) {
    u64 c = add;
    for (int i = 0; i < nl; i++) {
        const u64 t = (u64)m[i] * k + c;
        m[i] = (u32)t;
        c = t >> 32;
    }
    if (c && nl < kMaxLimbs) m[nl++] = (u32)c;
}

// m = floor(m / d), d < 2^32
__device__ __forceinline__ u32 div_small(u32* m, int& nl, u32 d) {
    u64 r = 0;
    for (int i = nl - 1; i >= 0; i--) {
        const u64 cur = (r << 32) | m[i];
        m[i] = (u32)(cur / d);
        r = cur % d;
    }
    while (nl > 1 && m[nl - 1] == 0u) nl--;
    return (u32)r;
}

__device__ __forceinline__ u32 pow10_u32(int k) {
    u32 p = 1;
    for (int i = 0; i < k; i++) p *= 10u;
    return p;
}

// One field of any length: magnitude in local memory.
__device__ __noinline__ u32 parse_row_general(const char* s, int64_t n, int scale, int B, u8* o) {
    u32 err = 0u;
    u32 m[kMaxLimbs];
    int nl = 1;
    m[0] = 0u;
    u32 sign = 0u;
    int64_t i = 0;
    if (n > 0 && s[0] == '-') {
        sign = 1u;
        i = 1;
    }
    bool dot = false, bad = false;
    int frac = 0, digits = 0, clen = 0;
    u32 chunk = 0;
    for (; i < n; i++) {
        const char c = s[i];
        if (c == '.' && !dot) {
            dot = true;
            continue;
        }
        if (c < '0' || c > '9' || digits >= kMaxDigits) {
            bad = true;
            break;
        }
        chunk = chunk * 10u + (u32)(c - '0');
        clen++;
        digits++;
        if (dot) frac++;
        if (clen == 9) {
            mul_add_small(m, nl, 1000000000u, chunk);
            chunk = 0u;
            clen = 0;
        }
    }
    if (!bad && clen) mul_add_small(m, nl, pow10_u32(clen), chunk);
    if (!bad) {
        // to the column's scale: pad with zeros or cut digits off
        for (int d = scale - frac; d > 0; d -= 9) mul_add_small(m, nl, pow10_u32(d < 9 ? d : 9), 0u);
        for (int d = frac - scale; d > 0; d -= 9) div_small(m, nl, pow10_u32(d < 9 ? d : 9));
    }
    if (bad) {
        err |= UP_ROWERR_DOMAIN;
        for (int b = 0; b < B; b++) o[b] = 0;
        return err;
    }
    // low B bytes; magnitude bits at or above 8B-1 are lost (sign bit)
    bool lost = false;
    for (int b = 0; b < 4 * nl; b++) {
        const u32 byte = (m[b >> 2] >> (8 * (b & 3))) & 0xffu;
        if (b < B) {
            u32 v = byte;
            if (b == B - 1) {
                lost |= (v & 0x80u) != 0u;
                v |= sign << 7;
            }
            o[b] = (u8)v;
        } else {
            lost |= byte != 0u;
        }
    }
    for (int b = 4 * nl; b < B; b++) o[b] = (u8)(b == B - 1 ? sign << 7 : 0u);
    if (lost) err |= UP_ROWERR_OVERFLOW;
    return err;
}

// Rows per CTA of the staged kernels (one row per thread).
constexpr int kTextRows = 128;
// Widest staged values: 32 limbs (308 digits); wider ones take the general kernels.
constexpr int kStagedLimbs = 32;

// Contiguous bytes global -> shared, 16-byte vectors between the unaligned
// ends; dst and src have the same address modulo 16.
__device__ __forceinline__ void copy_bytes_in(u8* dst, const u8* src, int n) {
    const int head = min(n, (int)((16u - (u32)(uintptr_t)src) & 15u));
    const int vecs = (n - head) >> 4, tail = head + (vecs << 4);
    for (int i = threadIdx.x; i < head; i += kTextRows) dst[i] = src[i];
    const uint4* v = (const uint4*)(src + head);
    uint4* d = (uint4*)(dst + head);
    for (int i = threadIdx.x; i < vecs; i += kTextRows) d[i] = v[i];
    for (int i = tail + threadIdx.x; i < n; i += kTextRows) dst[i] = src[i];
}

// Contiguous bytes shared -> global, the same way.
__device__ __forceinline__ void copy_bytes_out(u8* dst, const u8* src, int n) {
    const int head = min(n, (int)((16u - (u32)(uintptr_t)dst) & 15u));
    const int vecs = (n - head) >> 4, tail = head + (vecs << 4);
    for (int i = threadIdx.x; i < head; i += kTextRows) dst[i] = src[i];
    const uint4* v = (const uint4*)(src + head);
    uint4* d = (uint4*)(dst + head);
    for (int i = threadIdx.x; i < vecs; i += kTextRows) d[i] = v[i];
    for (int i = tail + threadIdx.x; i < n; i += kTextRows) dst[i] = src[i];
}

__constant__ const u32 kPow10[10] = {1u,      10u,      100u,      1000u,      10000u,
                                     100000u, 1000000u, 10000000u, 100000000u, 1000000000u};

// m = m * k + add over N limbs (the caller keeps the value below 2^(32N))
template <int N>
__device__ __forceinline__ void mul_add_limbs(u32 (&m)[N], u32 k, u32 add) {
    u64 c = add;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const u64 t = (u64)m[i] * k + c;
        m[i] = (u32)t;
        c = t >> 32;
    }
}

// Decimal digits that always fit N limbs: floor(32 N log10 2).
__host__ __device__ constexpr int digits_of_limbs(int n) { return (int)(32.0 * n * 0.30102999566398); }

// A row's characters in shared memory, four at a time: two aligned words
// around the next character (the text is padded past its end).
struct TextReader {
    const u32* w;
    u32 w0, w1, off;
    __device__ __forceinline__ explicit TextReader(const u8* s) {
        off = (u32)(uintptr_t)s & 3u;
        w = (const u32*)(s - off);
        w0 = w[0];
        w1 = w[1];
    }
    // the next four characters, each xor '0'
    __device__ __forceinline__ u32 peek() const { return __funnelshift_r(w0, w1, 8u * off) ^ 0x30303030u; }
    __device__ __forceinline__ void skip4() {
        w++;
        w0 = w1;
        w1 = w[1];
    }
    __device__ __forceinline__ void skip1() {
        if (++off == 4u) {
            off = 0u;
            skip4();
        }
    }
};
__device__ __forceinline__ bool four_are_digits(u32 x) { return (((x + 0x06060606u) | x) & 0xf0f0f0f0u) == 0u; }
__device__ __forceinline__ u32 four_digit_value(u32 x) {
    const u32 v = (x * 10u + (x >> 8)) & 0x00ff00ffu;
    return (v * 100u + (v >> 16)) & 0xffffu;
}

// Consecutive digits of [i, end): eight per step into the limbs, the last
// ones of a run left in (chunk, scale10 = 10^digits of it).  Stops at end or at
// the first other character.
template <int N>
__device__ __forceinline__ void parse_digits(TextReader& t, int& i, int end, u32 (&m)[N], u32& chunk, u32& scale10) {
    while (i + 8 <= end) {
        const u32 x = t.peek();
        if (!four_are_digits(x)) break;
        t.skip4();
        const u32 y = t.peek();
        const u32 a = four_digit_value(x);
        if (!four_are_digits(y)) {  // four digits only
            if (scale10 > 10000u) {
                mul_add_limbs(m, scale10, chunk);
                chunk = 0u;
                scale10 = 1u;
            }
            chunk = chunk * 10000u + a;
            scale10 *= 10000u;
            i += 4;
            break;
        }
        t.skip4();
        i += 8;
        if (scale10 != 1u) {
            mul_add_limbs(m, scale10, chunk);
            chunk = 0u;
            scale10 = 1u;
        }
        mul_add_limbs(m, 100000000u, a * 10000u + four_digit_value(y));
    }
    if (i + 4 <= end && scale10 <= 10000u) {
        const u32 x = t.peek();
        if (four_are_digits(x)) {
            t.skip4();
            i += 4;
            chunk = chunk * 10000u + four_digit_value(x);
            scale10 *= 10000u;
        }
    }
    while (i < end) {
        const u32 d = t.peek() & 0xffu;
        if (d > 9u) break;
        t.skip1();
        i++;
        if (scale10 == 1000000000u) {
            mul_add_limbs(m, scale10, chunk);
            chunk = 0u;
            scale10 = 1u;
        }
        chunk = chunk * 10u + d;
        scale10 *= 10u;
    }
}

// A field of a row staged in shared memory: N limbs in registers.  Fraction
// digits past the scale are only checked (cutting digits off is the
// truncation), missing ones are multiplied in.  False: more digits than N
// limbs are sure to hold.
template <int N>
__device__ __forceinline__ bool parse_row_limbs(const u8* s, int n, int scale, u32 (&m)[N], u32& sign, bool& bad) {
#pragma unroll
    for (int i = 0; i < N; i++) m[i] = 0u;
    sign = 0u;
    bad = false;
    int i = 0;
    if (n > 0 && s[0] == '-') {
        sign = 1u;
        i = 1;
    }
    TextReader t(s + i);
    u32 chunk = 0u, scale10 = 1u;
    const int int0 = i;
    parse_digits(t, i, n, m, chunk, scale10);
    const int ints = i - int0;
    int frac = 0;
    if (i < n && (t.peek() & 0xffu) == ('.' ^ '0')) {
        t.skip1();
        i++;
        const int frac0 = i;
        parse_digits(t, i, min(n, i + scale), m, chunk, scale10);
        frac = i - frac0;
        if (frac == scale)
            for (; i < n && (t.peek() & 0xffu) <= 9u; i++) t.skip1();
    }
    bad = i < n;
    if (bad) return true;
    if (scale10 != 1u) mul_add_limbs(m, scale10, chunk);
    for (int z = scale - frac; z > 0; z -= 9) mul_add_limbs(m, kPow10[z < 9 ? z : 9], 0u);
    return ints + scale <= digits_of_limbs(N);
}

// Whether a field [a, b) lies in the staged text [lo, hi) and is short enough
// for the limbs in registers.  Fields that end before they start (offsets that
// do not ascend) read nothing: the general routine stores their 0.
__host__ __device__ constexpr bool staged_field(int64_t a, int64_t b, int64_t lo, int64_t hi) {
    return a >= lo && a <= b && b <= hi && b - a <= 1024;
}

// Bound by the instructions per character; a byte of text from global memory
// per step and limbs in local memory waited on both.  The CTA's text (its
// fields are consecutive) is staged in shared memory when it fits `cap`
// bytes, the values leave through shared memory.  Measured on B200, 4M fields
// of DECIMAL(38,9): 0.39 -> 0.18 ms with the call's allocations, the kernel 0.15 ms.
template <int N>
__global__ void __launch_bounds__(kTextRows) k_parse_staged(const char* __restrict__ text, const int64_t* __restrict__ off,
                                                            int64_t rows, int scale, int B, int cap, u8* __restrict__ out,
                                                            u32* __restrict__ err_word) {
    extern __shared__ __align__(16) u8 sm[];
    u8* const area = sm + cap + 32;  // 16 bytes of alignment before the text, readable words after it
    u32 err = 0u;
    const int64_t tiles = (rows + kTextRows - 1) / kTextRows;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int64_t r0 = t * kTextRows;
        const int nr = rows - r0 < kTextRows ? (int)(rows - r0) : kTextRows;
        const int64_t lo = off[r0], hi = off[r0 + nr];
        const bool fits = hi >= lo && hi - lo <= cap;
        u8* buf = sm + ((uintptr_t)(text + lo) & 15u);
        u8* vals = area + ((uintptr_t)(out + r0 * B) & 15u);
        const bool words = (B & 3) == 0 && ((uintptr_t)vals & 3u) == 0u;
        if (fits) copy_bytes_in(buf, (const u8*)text + lo, (int)(hi - lo));
        __syncthreads();
        if ((int)threadIdx.x < nr) {
            const int64_t a = off[r0 + threadIdx.x], b = off[r0 + threadIdx.x + 1];
            u8* o = vals + threadIdx.x * B;
            bool done = false;
            if (fits && staged_field(a, b, lo, hi)) {
                u32 m[N], sign;
                bool bad;
                if (parse_row_limbs<N>(buf + (a - lo), (int)(b - a), scale, m, sign, bad)) {
                    done = true;
                    if (bad) {
                        err |= UP_ROWERR_DOMAIN;
                        for (int i = 0; i < B; i++) o[i] = 0;
                    } else {
                        // low B bytes, the sign in the last one's bit 7; lost: bits at or above 8B-1
                        const int top = 8 * B - 1;
                        u32 lost = 0u;
#pragma unroll
                        for (int l = 0; l < N; l++) {
                            if (32 * l + 32 > top) lost |= 32 * l >= top ? m[l] : m[l] >> (top - 32 * l);
                            const u32 x = m[l] | (l == (B - 1) >> 2 ? sign << (top & 31) : 0u);
                            if (words) {
                                if (4 * l < B) ((u32*)o)[l] = x;
                            } else {
#pragma unroll
                                for (int k = 0; k < 4; k++)
                                    if (4 * l + k < B) o[4 * l + k] = (u8)(x >> (8 * k));
                            }
                        }
                        if (lost) err |= UP_ROWERR_OVERFLOW;
                    }
                }
            }
            if (!done) err |= parse_row_general(text + a, b - a, scale, B, o);
        }
        __syncthreads();
        copy_bytes_out(out + r0 * B, vals, nr * B);
    }
    if (err && err_word) atomicOr(err_word, err);
}

__global__ void k_parse_decimal(const char* __restrict__ text, const int64_t* __restrict__ off, int64_t rows,
                                int scale, int B, u8* __restrict__ out, u32* __restrict__ err_word) {
    u32 err = 0u;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += stride)
        err |= parse_row_general(text + off[r], off[r + 1] - off[r], scale, B, out + r * B);
    if (err && err_word) atomicOr(err_word, err);
}

// Chunks of eight decimal digits that N limbs (32 N - 1 bits) and one more
// leading zero need.
__host__ __device__ constexpr int chunks_of_limbs(int n) { return ((int)((32.0 * n - 1.0) * 0.30102999566398) + 2 + 7) / 8; }

// x = floor(x / 10^8) over the low K of N limbs (the others are zero), the
// remainder returned: 2/1 steps by the divisor normalised to 32 bits (10^8 << 5).
template <int K, int N>
__device__ __forceinline__ u32 div_1e8(u32 (&x)[N]) {
    constexpr u32 D = 100000000u << 5;
    constexpr u32 V = (u32)(~0ull / D - (1ull << 32));
    u32 r = x[K - 1] >> 27;
#pragma unroll
    for (int i = K - 1; i >= 0; i--) {
        const u32 lo = __funnelshift_l(i > 0 ? x[i > 0 ? i - 1 : 0] : 0u, x[i], 5);
        x[i] = up::div2by1(r, lo, D, V, r);
    }
    return r >> 5;
}

// four decimal digits of v < 10^4 as bytes, the first in the lowest byte
__device__ __forceinline__ u32 four_digits(u32 v) {
    const u32 h = (v * 5243u) >> 19;             // v / 100
    const u32 y = h | ((v - 100u * h) << 16);    // two values below 100
    const u32 t = ((y * 103u) >> 10) & 0x000f000fu;  // their tens
    return t | ((y - 10u * t) << 8);
}

// The C chunks of eight digits of x, least significant first (chunk k divides
// what 26.5 bits per chunk before it have left of 32 N - 1 bits).
template <int K, int C, int N>
__device__ __forceinline__ void decimal_chunks(u32 (&x)[N], u32 (&dig)[2 * C]) {
    if constexpr (K < C) {
        constexpr int bits = 32 * N - 1 - (int)(26.57 * K);
        u32 v;
        if constexpr (bits > 32) {
            v = div_1e8<(bits + 31) / 32>(x);
        } else {
            v = x[0] % 100000000u;
            x[0] /= 100000000u;
        }
        const u32 h = v / 10000u;
        dig[2 * (C - 1 - K)] = four_digits(h);
        dig[2 * (C - 1 - K) + 1] = four_digits(v - 10000u * h);
        decimal_chunks<K + 1, C>(x, dig);
    }
}

// The decimal string of every row: N limbs to eight-digit chunks in
// registers, characters into a shared-memory image of the CTA's slots (loaded
// first, so that characters past a row's length stay what they were), which
// leaves in vectors.  Bound by the instructions and byte stores per
// character; digits in local memory and byte stores to global memory waited
// on both.  Measured on B200, 4M values of DECIMAL(38,9): 1.16 -> 0.19 ms.
// CTAs per SM asked for (registers of 64, 102 and 255 at most): p=6 0.066 ms (0.083
// with none asked for), p=38 0.187 (0.230), p=77 0.355 (0.357), p=200 0.477
// (0.481); p=120 is the exception, 0.379 (0.344).
template <int N>
__global__ void __launch_bounds__(kTextRows, N <= 4 ? 8 : N <= 8 ? 5 : 2)
    k_format_staged(const u8* __restrict__ in, int64_t rows, int B, int scale, char* __restrict__ out, int width,
                    int32_t* __restrict__ out_len) {
    constexpr int C = chunks_of_limbs(N), D = 8 * C;
    extern __shared__ __align__(16) u8 sm[];
    // a warp's byte stores go to rows whose slots start in different banks: four
    // rows apart (width words) where a slot is no whole number of words
    const int row = width & 3 ? (int)((threadIdx.x & 31u) * 4u + (threadIdx.x >> 5)) : (int)threadIdx.x;
    u8* const area = sm + (kTextRows * B + 32 + 15) / 16 * 16;
    const int64_t tiles = (rows + kTextRows - 1) / kTextRows;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int64_t r0 = t * kTextRows;
        const int nr = rows - r0 < kTextRows ? (int)(rows - r0) : kTextRows;
        u8* src = sm + ((uintptr_t)(in + r0 * B) & 15u);
        u8* img = area + ((uintptr_t)(out + r0 * width) & 15u);
        copy_bytes_in(src, in + r0 * B, nr * B);
        copy_bytes_in(img, (const u8*)out + r0 * width, nr * width);
        __syncthreads();
        const u32 active = __ballot_sync(0xffffffffu, row < nr);
        if (row < nr) {
            const u8* p = src + row * B;
            const u32 po = (u32)(uintptr_t)p & 3u;
            const u32* w = (const u32*)(p - po);
            u32 x[N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int left = B - 4 * i;  // bytes of the value from limb i on
                x[i] = left > 0 ? __funnelshift_r(w[i], w[i + 1], 8u * po) : 0u;
                if (left > 0 && left < 4) x[i] &= (1u << (8 * left)) - 1u;
            }
            const u32 sign = (u32)p[B - 1] >> 7;
#pragma unroll
            for (int i = 0; i < N; i++)
                if (i == (B - 1) >> 2) x[i] &= ~(0x80u << (8 * ((B - 1) & 3)));
            u32 dig[2 * C];  // four digits per word, most significant word first
            decimal_chunks<0, C>(x, dig);
            int first = D - 1 - scale;  // at least a 0 before the point
#pragma unroll
            for (int k = 2 * C - 1; k >= 0; k--)
                if (dig[k]) first = min(D - 1 - scale, 4 * k + ((__ffs((int)dig[k]) - 1) >> 3));
            const int point = D - scale;  // the point comes before this digit
            int at = (int)sign - first;   // digit i's place is at + i, one more after the point
            const int len = at + D + (scale > 0 ? 1 : 0);
            u8* o = img + row * width;
            if (sign) o[0] = '-';
            if (scale > 0 && at + point < width) o[at + point] = '.';
            // words of four digits on one side of the point that every row of
            // the warp writes whole take no tests per character
            const bool cut = __any_sync(active, len > width);
            const int some = __reduce_min_sync(active, first);
            const int whole = cut ? D : __reduce_max_sync(active, first);
#pragma unroll
            for (int k = 0; k < 2 * C; k++) {
                const u32 x = dig[k] + 0x30303030u;
                if (4 * k >= whole && (4 * k + 4 <= point || 4 * k >= point)) {
                    u8* c = o + at + (4 * k >= point ? 1 : 0) + 4 * k;
                    c[0] = (u8)x;
                    c[1] = (u8)(x >> 8);
                    c[2] = (u8)(x >> 16);
                    c[3] = (u8)(x >> 24);
                } else if (4 * k + 3 >= some) {
#pragma unroll
                    for (int i = 4 * k; i < 4 * k + 4; i++) {
                        const int c = at + i + (i >= point ? 1 : 0);
                        if (i >= first && c < width) o[c] = (u8)(x >> (8 * (i & 3)));
                    }
                }
            }
            out_len[r0 + row] = len <= width ? len : -1;
        }
        __syncthreads();
        copy_bytes_out((u8*)out + r0 * width, img, nr * width);
        __syncthreads();
    }
}

// The reference's hex image, and values wider than the staged kernels'.
__global__ void k_format_decimal(const u8* __restrict__ in, int64_t rows, int B, int scale, int hex,
                                 char* __restrict__ out, int width, int32_t* __restrict__ out_len) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += stride) {
        const u8* p = in + r * B;
        u32 m[kMaxLimbs];
        const int nl0 = (B + 3) / 4;
        for (int i = 0; i < nl0; i++) m[i] = 0u;
        for (int b = 0; b < B; b++) m[b >> 2] |= (u32)p[b] << (8 * (b & 3));
        const u32 sign = (u32)(p[B - 1] >> 7);
        m[(B - 1) >> 2] &= ~(0x80u << (8 * ((B - 1) & 3)));
        char* o = out + r * width;
        int len = 0;
        auto put = [&](char c) {
            if (len < width) o[len] = c;
            len++;
        };
        if (hex) {
            // Decimal::GetDecimal: sign, 8 hex digits per limb from the highest
            // nonzero one, then "(fff)"
            const char* dig = "0123456789ABCDEF";
            put(sign ? '-' : '+');
            int top = nl0 - 1;
            while (top >= 0 && m[top] == 0u) top--;
            for (int i = top; i >= 0; i--)
                for (int j = 7; j >= 0; j--) put(dig[(m[i] >> (4 * j)) & 0xfu]);
            put('(');
            put((char)('0' + scale / 100 % 10));
            put((char)('0' + scale / 10 % 10));
            put((char)('0' + scale % 10));
            put(')');
        } else {
            // decimal digits, least significant first, in base 10^9 chunks
            int nl = nl0;
            while (nl > 1 && m[nl - 1] == 0u) nl--;
            char rev[kMaxDigits + 16];
            int nd = 0;
            do {
                u32 rem = div_small(m, nl, 1000000000u);
                const bool last = nl == 1 && m[0] == 0u;
                for (int k = 0; k < 9 && (nd < kMaxDigits + 16); k++) {
                    rev[nd++] = (char)('0' + rem % 10u);
                    rem /= 10u;
                    if (last && rem == 0u) break;
                }
                if (last) break;
            } while (true);
            while (nd > 1 && rev[nd - 1] == '0') nd--;  // no leading zeros
            while (nd < scale + 1) rev[nd++] = '0';      // at least "0." before the fraction
            if (sign) put('-');
            for (int k = nd - 1; k >= 0; k--) {
                put(rev[k]);
                if (k == scale && scale > 0) put('.');
            }
        }
        out_len[r] = len <= width ? len : -1;
    }
}

// The staged kernels' instances, by limbs of the compact value.
template <template <int> class L, class... A>
cudaError_t by_limbs(int limbs, A... args) {
    if (limbs <= 1) return L<1>::launch(args...);
    if (limbs <= 2) return L<2>::launch(args...);
    if (limbs <= 3) return L<3>::launch(args...);
    if (limbs <= 4) return L<4>::launch(args...);
    if (limbs <= 6) return L<6>::launch(args...);
    if (limbs <= 8) return L<8>::launch(args...);
    if (limbs <= 12) return L<12>::launch(args...);
    if (limbs <= 16) return L<16>::launch(args...);
    if (limbs <= 24) return L<24>::launch(args...);
    return L<kStagedLimbs>::launch(args...);
}

int staged_grid(int64_t rows) {
    const int64_t tiles = (rows + kTextRows - 1) / kTextRows;
    return (int)std::min<int64_t>(tiles, (int64_t)std::max(1, sm_count_current()) * 16);
}

template <int N>
struct ParseStaged {
    static cudaError_t launch(const char* text, const int64_t* off, int64_t rows, int scale, int B, u8* out, u32* err,
                              cudaStream_t s) {
        // text per CTA: fields of the digits the limbs hold, a sign, a point
        // and two separators; with the values within 48 KB
        const int cap = std::min(kTextRows * (digits_of_limbs(N) + 4), 48 * 1024 - 64 - kTextRows * B) / 16 * 16;
        k_parse_staged<N><<<staged_grid(rows), kTextRows, cap + 32 + 16 + kTextRows * B, s>>>(text, off, rows, scale, B, cap, out,
                                                                                         err);
        return cudaGetLastError();
    }
};

// Bytes of the format kernel's shared memory: the staged values and the slots.
int64_t format_smem(int B, int width) { return (kTextRows * B + 32 + 15) / 16 * 16 + (int64_t)kTextRows * width + 16; }
constexpr int kFormatSmem = 48 * 1024;

template <int N>
struct FormatStaged {
    static cudaError_t launch(const u8* in, int64_t rows, int B, int scale, char* out, int width, int32_t* lens,
                              cudaStream_t s) {
        k_format_staged<N><<<staged_grid(rows), kTextRows, (size_t)format_smem(B, width), s>>>(in, rows, B, scale, out, width,
                                                                                               lens);
        return cudaGetLastError();
    }
};

int grid_for(int64_t rows) {
    const int64_t blocks = (rows + 127) / 128;
    const int sms = std::max(1, sm_count_current());
    return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, (int64_t)sms * 16));
}

}  // namespace
}  // namespace upi

using namespace upi;

extern "C" {

up_status up_parse_decimal(const char* text, const int64_t* offsets, int64_t rows, int32_t precision, int32_t scale,
                           void* out, uint32_t* err_word, void* stream) {
    if (rows < 0) return fail(UP_ERR_INVALID_ARG, "negative row count");
    if (precision < 1 || precision > kMaxPrecisionText || scale < 0 || scale > precision)
        return fail(UP_ERR_INVALID_ARG, "precision 1..1000 and 0 <= scale <= precision");
    if (rows == 0) return UP_OK;
    if (!text || !offsets || !out) return fail(UP_ERR_INVALID_ARG, "NULL buffers");
    const int B = compact_bytes(precision);
    const int limbs = (B + 3) / 4;
    cudaError_t e;
    if (limbs <= kStagedLimbs) {
        e = by_limbs<ParseStaged>(limbs, text, offsets, rows, scale, B, (u8*)out, err_word, (cudaStream_t)stream);
    } else {
        k_parse_decimal<<<grid_for(rows), 128, 0, (cudaStream_t)stream>>>(text, offsets, rows, scale, B, (u8*)out,
                                                                          err_word);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess)
        return fail(e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver ? UP_ERR_NO_DEVICE : UP_ERR_CUDA,
                    std::string("parse launch: ") + cudaGetErrorString(e));
    return UP_OK;
}

int32_t up_format_width(int32_t precision, int32_t hex) {
    if (precision < 1 || precision > kMaxPrecisionText) return -1;
    const int B = compact_bytes(precision);
    if (hex) return 1 + 8 * ((B + 3) / 4) + 5;
    // digits of the largest magnitude B bytes can hold (2^(8B-1) - 1), a sign,
    // a '.' and a leading 0
    const int digits = (int)std::floor((8.0 * B - 1.0) * std::log10(2.0)) + 1;
    return digits + 3;
}

up_status up_format_decimal(const void* compact, int64_t rows, int32_t precision, int32_t scale, int32_t hex,
                            char* out_text, int32_t width, int32_t* out_len, void* stream) {
    if (rows < 0 || width < 1) return fail(UP_ERR_INVALID_ARG, "negative row count or width");
    if (precision < 1 || precision > kMaxPrecisionText || scale < 0 || scale > precision)
        return fail(UP_ERR_INVALID_ARG, "precision 1..1000 and 0 <= scale <= precision");
    if (rows == 0) return UP_OK;
    if (!compact || !out_text || !out_len) return fail(UP_ERR_INVALID_ARG, "NULL buffers");
    const int B = compact_bytes(precision);
    const int limbs = (B + 3) / 4;
    cudaError_t e;
    if (!hex && limbs <= kStagedLimbs && format_smem(B, width) <= kFormatSmem) {
        e = by_limbs<FormatStaged>(limbs, (const u8*)compact, rows, B, scale, out_text, width, out_len,
                                   (cudaStream_t)stream);
    } else {
        k_format_decimal<<<grid_for(rows), 128, 0, (cudaStream_t)stream>>>((const u8*)compact, rows, B, scale, hex ? 1 : 0,
                                                                           out_text, width, out_len);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess)
        return fail(e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver ? UP_ERR_NO_DEVICE : UP_ERR_CUDA,
                    std::string("format launch: ") + cudaGetErrorString(e));
    return UP_OK;
}

}  // extern "C"
