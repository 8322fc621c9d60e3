// chaincheck.cpp — TEST INFRASTRUCTURE: the carry-chain arithmetic of
// up_dev.cuh (products, sums, differences, comparisons), compiled for the
// host, against schoolbook sums limb by limb.  Prints "<name> <cases> <bad>".
#include "host_shims.h"

#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "../../ultraprecise_b200/csrc/up_dev.cuh"

using namespace up;

static uint64_t state = 88172645463325252ull;
static u32 rnd() {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return (u32)(state >> 11);
}
// limbs from the values carries run through: 0, all ones, one, random
template <int N>
static void gen(u32 (&a)[N]) {
    const int mode = rnd() % 4;
    for (int i = 0; i < N; i++) {
        const u32 r = rnd();
        a[i] = mode == 0 ? 0xffffffffu : (mode == 1 ? r : (r % 3 == 0 ? 0u : (r % 3 == 1 ? 0xffffffffu : rnd())));
    }
    if (rnd() % 8 == 0)
        for (int i = 0; i < N; i++) a[i] = i ? 0u : rnd() % 2;
}

template <int N, int NA, int NB>
static long check_mul(long n) {
    long bad = 0;
    for (long c = 0; c < n; c++) {
        u32 a[NA], b[NB], r[N], want[N + NA + NB + 1] = {0};
        gen(a);
        gen(b);
        mul(r, a, b);
        for (int i = 0; i < NA; i++) {
            uint64_t carry = 0;
            for (int j = 0; j < NB; j++) {
                const uint64_t t = (uint64_t)a[i] * b[j] + want[i + j] + carry;
                want[i + j] = (u32)t;
                carry = t >> 32;
            }
            want[i + NB] = (u32)carry;
        }
        bool ok = true;
        for (int i = 0; i < N; i++) ok &= r[i] == want[i];
        u32 k[N + 1], wk[NA + 1];
        mul_u32(k, a, b[0]);
        uint64_t carry = 0;
        for (int i = 0; i <= NA; i++) {
            const uint64_t t = (i < NA ? (uint64_t)a[i < NA ? i : 0] * b[0] : 0ull) + carry;
            wk[i] = (u32)t;
            carry = t >> 32;
        }
        for (int i = 0; i < N + 1; i++) ok &= k[i] == (i <= NA ? wk[i <= NA ? i : 0] : 0u);
        bad += !ok;
    }
    std::printf("mul<%d,%d,%d> %ld %ld\n", N, NA, NB, n, bad);
    return bad;
}

template <int N, int NA, int NB>
static long check_sums(long n) {
    long bad = 0;
    for (long c = 0; c < n; c++) {
        u32 a[NA], b[NB], r[N], d[N], w[N], v[N], s[N];
        gen(a);
        gen(b);
        if (rnd() % 4 == 0)
            for (int i = 0; i < NB; i++) b[i] = i < NA ? a[i < NA ? i : 0] : 0u;
        const u32 co = add(r, a, b), bo = sub(d, a, b);
        uint64_t carry = 0, borrow = 0;
        for (int i = 0; i < N; i++) {
            const uint64_t x = i < NA ? a[i < NA ? i : 0] : 0u, y = i < NB ? b[i < NB ? i : 0] : 0u;
            uint64_t t = x + y + carry;
            w[i] = (u32)t;
            carry = t >> 32;
            t = x - y - borrow;
            v[i] = (u32)t;
            borrow = t >> 63;
        }
        bool ok = co == carry && bo == borrow;
        int cmpv = 0;
        for (int i = (NA > NB ? NA : NB) - 1; i >= 0 && cmpv == 0; i--) {
            const u32 x = i < NA ? a[i < NA ? i : 0] : 0u, y = i < NB ? b[i < NB ? i : 0] : 0u;
            cmpv = x < y ? -1 : x > y;
        }
        ok &= less(a, b) == (cmpv < 0);
        u32 g[N];
        for (int i = 0; i < N; i++) g[i] = d[i];
        negate(g);
        u32 back[N];
        add(back, g, d);
        for (int i = 0; i < N; i++) ok &= r[i] == w[i] && d[i] == v[i] && back[i] == 0u;
        const u32 sa = rnd() & 1u, sb = rnd() & 1u;
        u32 sr;
        add_signed(s, sr, a, sa, b, sb);
        if (sa == sb) {
            for (int i = 0; i < N; i++) ok &= s[i] == w[i];
            ok &= sr == sa;
        } else {
            for (int i = 0; i < N; i++) ok &= s[i] == (cmpv < 0 ? g[i] : d[i]);
            ok &= sr == (cmpv == 0 ? 0u : (cmpv < 0 ? sb : sa));
        }
        bad += !ok;
    }
    std::printf("sums<%d,%d,%d> %ld %ld\n", N, NA, NB, n, bad);
    return bad;
}

// x = q*b + r with r < b and quotients around every bound of
// div_small_quotient (2^47, 2^79: above it the function declines)
template <int NX, int NB>
static long check_quotient(long n) {
    long bad = 0, ran = 0;
    for (long c = 0; c < n; c++) {
        u32 b[NB], r[NB], q[NX] = {0}, x[NX], got[NX];
        gen(b);
        for (int i = 2 + (int)(rnd() % (NB - 1)); i < NB; i++) b[i] = 0u;
        if (NB > 1 && rnd() % 2) b[1] |= 1u;
        bool wide = false;
        for (int i = 1; i < NB; i++) wide |= b[i] != 0u;
        if (!wide) continue;
        const int bits = (int)(rnd() % 83);  // of the quotient
        for (int i = 0; i < NX; i++) {
            const int left = bits - 32 * i;
            const u32 v = rnd() % 3 == 0 ? 0xffffffffu : (rnd() % 2 ? rnd() : 0u);
            q[i] = left <= 0 ? 0u : (left >= 32 ? v : v & ((1u << left) - 1u));
        }
        if (rnd() % 4 == 0)
            for (int i = 0; i < NX; i++) q[i] = i == bits / 32 ? 1u << (bits % 32) : 0u;
        const int rm = rnd() % 4;  // 0, b - 1, b / 2 and neighbours
        for (int i = 0; i < NB; i++)
            r[i] = rm == 0 ? 0u : (rm == 1 ? b[i] : (b[i] >> 1) | (i + 1 < NB ? b[i + 1 < NB ? i + 1 : 0] << 31 : 0u));
        if (rm == 1) {
            u32 one[1] = {1u};
            sub(r, r, one);
        }
        if (rm == 3) {
            u32 one[1] = {1u};
            add(r, r, one);
            if (!less(r, b)) continue;
        }
        u32 full[NX + NB + 1];
        mul(full, q, b);
        add(full, full, r);
        bool fits = true;
        for (int i = NX; i < NX + NB + 1; i++) fits &= full[i] == 0u;
        if (!fits) continue;
        for (int i = 0; i < NX; i++) x[i] = full[i];
        bool up = false;
        ran++;
        if (!div_small_quotient(got, up, x, b)) {
            bad += bits < 78;
            continue;
        }
        u32 dbl[NB + 1];
        add(dbl, r, r);
        bool ok = up == !less(dbl, b);
        for (int i = 0; i < NX; i++) ok &= got[i] == q[i];
        if (!ok && bad < 3) std::printf("quotient<%d,%d> of %d bits, rm %d\n", NX, NB, bits, rm);
        bad += !ok;
    }
    std::printf("quotient<%d,%d> %ld %ld\n", NX, NB, ran, bad);
    return bad;
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 20000;
    long bad = 0;
    bad += check_mul<2, 1, 1>(n) + check_mul<4, 2, 2>(n) + check_mul<5, 3, 2>(n) + check_mul<6, 4, 2>(n);
    bad += check_mul<7, 4, 3>(n) + check_mul<8, 4, 4>(n) + check_mul<9, 5, 4>(n) + check_mul<8, 3, 5>(n);
    bad += check_mul<16, 8, 8>(n) + check_mul<13, 11, 2>(n) + check_mul<22, 11, 11>(n / 4) + check_mul<32, 16, 16>(n / 8);
    bad += check_mul<64, 32, 32>(n / 32) + check_mul<41, 32, 9>(n / 16);
    bad += check_mul<3, 4, 4>(n) + check_mul<7, 8, 8>(n) + check_mul<20, 16, 16>(n / 8);  // low limbs only
    // long operands by halves (with small limits when built for that), the
    // second half as long as the other operand, or a limb shorter
    bad += check_mul<12, 8, 4>(n) + check_mul<11, 7, 4>(n) + check_mul<13, 8, 5>(n) + check_mul<14, 9, 5>(n);
    bad += check_mul<16, 12, 4>(n) + check_mul<13, 5, 8>(n) + check_mul<10, 8, 5>(n) + check_mul<9, 9, 5>(n);
    bad += check_mul<141, 94, 47>(n / 200) + check_mul<187, 125, 63>(n / 200) + check_mul<150, 63, 125>(n / 200);
    bad += check_sums<1, 1, 1>(n) + check_sums<4, 4, 3>(n) + check_sums<5, 5, 5>(n) + check_sums<6, 4, 5>(n);
    bad += check_sums<9, 8, 3>(n) + check_sums<33, 32, 32>(n / 4);
    bad += check_quotient<3, 2>(n) + check_quotient<5, 2>(n) + check_quotient<6, 4>(n) + check_quotient<7, 4>(n);
    bad += check_quotient<8, 4>(n) + check_quotient<7, 5>(n) + check_quotient<6, 6>(n);
    return bad ? 1 : 0;
}
