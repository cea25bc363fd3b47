// Exact integer arithmetic shared by host and device code.
//
//  * Z_q with q = 2^112 - 75 on four 32-bit limbs (little endian, the 16-byte
//    serde form of src/algebra/field.rs:112-129).  Multiplication is a 4x4 limb
//    schoolbook product reduced with 2^112 = 75 (mod q), the same pseudo-Mersenne
//    identity as field.rs:229-258; host code multiplies reduced values with
//    64-bit halves instead (same results).
//  * Arithmetic modulo the nine NTT primes p < 2^28 (p = 1 mod 2^14) that carry
//    every ring product: Shoup products by constants give [0, 2p), so the
//    transforms run four stages on values below 16p < 2^32 without reducing
//    (lazy Harvey butterflies), and products of two reduced residues fit 56 bits.
//  * CRT recombination of the nine residues into Z_q with a centred lift
//    (the integer result of src/algebra/ntt.rs:372-427; P = 2^251.98 leaves room
//    for any commitment sum, |X| < 2^250, up to depth 13).
#pragma once

#include <cstring>

#include "dm_common.cuh"

namespace dm {

struct fq {
    uint32_t w[4];
};

DM_HD fq fq_zero() { return fq{{0u, 0u, 0u, 0u}}; }
DM_HD fq fq_from_u32(uint32_t v) { return fq{{v, 0u, 0u, 0u}}; }
DM_HD bool fq_is_zero(const fq& a) { return (a.w[0] | a.w[1] | a.w[2] | a.w[3]) == 0u; }
DM_HD bool fq_eq(const fq& a, const fq& b) {
    return a.w[0] == b.w[0] && a.w[1] == b.w[1] && a.w[2] == b.w[2] && a.w[3] == b.w[3];
}

// q = 2^112 - 75 in limbs.
constexpr uint32_t kQ0 = 0xFFFFFFB5u, kQ1 = 0xFFFFFFFFu, kQ2 = 0xFFFFFFFFu, kQ3 = 0x0000FFFFu;

// x < 2^113 -> x mod q, using x >= q  <=>  x + 75 >= 2^112.
DM_HD fq fq_canon(const fq& x) {
    uint64_t c = (uint64_t)x.w[0] + 75u;
    uint32_t t0 = (uint32_t)c;
    c = (c >> 32) + x.w[1];
    uint32_t t1 = (uint32_t)c;
    c = (c >> 32) + x.w[2];
    uint32_t t2 = (uint32_t)c;
    c = (c >> 32) + x.w[3];
    uint32_t t3 = (uint32_t)c;
    if (t3 >> 16) return fq{{t0, t1, t2, t3 & 0xFFFFu}};
    return x;
}

DM_HD fq fq_add(const fq& a, const fq& b) {
    fq s;
    uint64_t c = (uint64_t)a.w[0] + b.w[0];
    s.w[0] = (uint32_t)c;
    c = (c >> 32) + a.w[1] + b.w[1];
    s.w[1] = (uint32_t)c;
    c = (c >> 32) + a.w[2] + b.w[2];
    s.w[2] = (uint32_t)c;
    c = (c >> 32) + a.w[3] + b.w[3];
    s.w[3] = (uint32_t)c;
    return fq_canon(s);
}

DM_HD fq fq_sub(const fq& a, const fq& b) {
    // d = a - b (mod 2^128); if it borrowed, add q.
    uint64_t br;
    fq d;
    uint64_t t = (uint64_t)a.w[0] - b.w[0];
    d.w[0] = (uint32_t)t;
    br = (t >> 63) & 1u;
    t = (uint64_t)a.w[1] - b.w[1] - br;
    d.w[1] = (uint32_t)t;
    br = (t >> 63) & 1u;
    t = (uint64_t)a.w[2] - b.w[2] - br;
    d.w[2] = (uint32_t)t;
    br = (t >> 63) & 1u;
    t = (uint64_t)a.w[3] - b.w[3] - br;
    d.w[3] = (uint32_t)t;
    br = (t >> 63) & 1u;
    if (br) {
        uint64_t c = (uint64_t)d.w[0] + kQ0;
        d.w[0] = (uint32_t)c;
        c = (c >> 32) + d.w[1] + kQ1;
        d.w[1] = (uint32_t)c;
        c = (c >> 32) + d.w[2] + kQ2;
        d.w[2] = (uint32_t)c;
        c = (c >> 32) + d.w[3] + kQ3;
        d.w[3] = (uint32_t)c;
    }
    return d;
}

DM_HD fq fq_neg(const fq& a) { return fq_sub(fq_zero(), a); }

// r[0..7] < 2^256 -> r mod q.
DM_HD fq fq_reduce8(const uint32_t r[8]) {
    // hi = r >> 112 (144 bits), t = (r mod 2^112) + 75 * hi < 2^152.
    uint32_t h0 = (r[3] >> 16) | (r[4] << 16);
    uint32_t h1 = (r[4] >> 16) | (r[5] << 16);
    uint32_t h2 = (r[5] >> 16) | (r[6] << 16);
    uint32_t h3 = (r[6] >> 16) | (r[7] << 16);
    uint32_t h4 = r[7] >> 16;
    uint64_t c = (uint64_t)r[0] + (uint64_t)h0 * 75u;
    uint32_t t0 = (uint32_t)c;
    c = (c >> 32) + r[1] + (uint64_t)h1 * 75u;
    uint32_t t1 = (uint32_t)c;
    c = (c >> 32) + r[2] + (uint64_t)h2 * 75u;
    uint32_t t2 = (uint32_t)c;
    c = (c >> 32) + (r[3] & 0xFFFFu) + (uint64_t)h3 * 75u;
    uint32_t t3 = (uint32_t)c;
    c = (c >> 32) + (uint64_t)h4 * 75u;
    uint32_t t4 = (uint32_t)c;
    // second fold: hi2 = t >> 112 < 2^40.
    uint64_t m = ((uint64_t)(t3 >> 16) | ((uint64_t)t4 << 16)) * 75u;  // < 2^47
    fq o;
    c = (uint64_t)t0 + (uint32_t)m;
    o.w[0] = (uint32_t)c;
    c = (c >> 32) + t1 + (m >> 32);
    o.w[1] = (uint32_t)c;
    c = (c >> 32) + t2;
    o.w[2] = (uint32_t)c;
    c = (c >> 32) + (t3 & 0xFFFFu);
    o.w[3] = (uint32_t)c;  // o < 2^112 + 2^47 < 2q
    return fq_canon(o);
}

DM_HD fq fq_mul_limbs(const fq& a, const fq& b) {
    uint32_t r[8] = {0, 0, 0, 0, 0, 0, 0, 0};
DM_UNROLL
    for (int i = 0; i < 4; ++i) {
        uint64_t c = 0;
DM_UNROLL
        for (int j = 0; j < 4; ++j) {
            c += (uint64_t)a.w[i] * b.w[j] + r[i + j];
            r[i + j] = (uint32_t)c;
            c >>= 32;
        }
        r[i + 4] = (uint32_t)c;
    }
    return fq_reduce8(r);
}

#if !defined(__CUDA_ARCH__) && defined(__SIZEOF_INT128__)
// Host form for inputs below 2^112 (every reduced value): four 64 x 64-bit
// products instead of sixteen 32 x 32, the same reduction 2^112 = 75 (mod q) to
// the canonical value, so the result equals fq_mul_limbs bit for bit.  False
// for wider inputs (words of an unchecked proof), which take the limb form.
inline bool fq_mul_wide(const fq& a, const fq& b, fq* out) {
    if ((a.w[3] | b.w[3]) >> 16) return false;
    typedef unsigned __int128 u128;
    const uint64_t a0 = a.w[0] | (uint64_t)a.w[1] << 32, a1 = a.w[2] | (uint64_t)a.w[3] << 32;
    const uint64_t b0 = b.w[0] | (uint64_t)b.w[1] << 32, b1 = b.w[2] | (uint64_t)b.w[3] << 32;
    const u128 p00 = (u128)a0 * b0;
    const u128 mid = (u128)a0 * b1 + (u128)a1 * b0;  // a1, b1 < 2^48: < 2^113
    const u128 p11 = (u128)a1 * b1;                  // < 2^96
    const uint64_t r0 = (uint64_t)p00;
    u128 t = (p00 >> 64) + (uint64_t)mid;
    const uint64_t r1 = (uint64_t)t;
    t = (t >> 64) + (mid >> 64) + p11;  // the product's bits from 128 on (< 2^96)
    const u128 m112 = ((u128)1 << 112) - 1;
    const u128 lo = ((u128)(r1 & ((1ull << 48) - 1)) << 64) | r0;  // product mod 2^112
    const u128 hi = (t << 16) | (r1 >> 48);                         // product >> 112, < 2^112
    u128 r = lo + hi * 75u;                                         // < 2^119
    r = (r & m112) + (r >> 112) * 75u;                              // < 2^112 + 2^14 < 2q
    const u128 q = ((u128)1 << 112) - 75u;
    if (r >= q) r -= q;
    out->w[0] = (uint32_t)r;
    out->w[1] = (uint32_t)(r >> 32);
    out->w[2] = (uint32_t)(r >> 64);
    out->w[3] = (uint32_t)(r >> 96);
    return true;
}
#endif

DM_HD fq fq_mul(const fq& a, const fq& b) {
#if !defined(__CUDA_ARCH__) && defined(__SIZEOF_INT128__)
    fq w;
    if (fq_mul_wide(a, b, &w)) return w;
#endif
    return fq_mul_limbs(a, b);
}

// a + c * b (mod q): the fold map of src/protocol/prover.rs:332-457.
DM_HD fq fq_fma(const fq& a, const fq& c, const fq& b) { return fq_add(a, fq_mul(c, b)); }

// ---- conversions between 16-byte little-endian words and limbs (host side) ----
inline fq fq_from_bytes(const uint8_t* p) {
    fq r;
    for (int i = 0; i < 4; ++i)
        r.w[i] = (uint32_t)p[4 * i] | ((uint32_t)p[4 * i + 1] << 8) | ((uint32_t)p[4 * i + 2] << 16) |
                 ((uint32_t)p[4 * i + 3] << 24);
    return r;
}
inline void fq_to_bytes(const fq& a, uint8_t* p) {
    for (int i = 0; i < 4; ++i) {
        p[4 * i] = (uint8_t)a.w[i];
        p[4 * i + 1] = (uint8_t)(a.w[i] >> 8);
        p[4 * i + 2] = (uint8_t)(a.w[i] >> 16);
        p[4 * i + 3] = (uint8_t)(a.w[i] >> 24);
    }
}
// Arbitrary 128-bit value reduced mod q (deserialisation, field.rs:121-129).
inline fq fq_from_u128_words(const fq& x) {
    uint32_t r[8] = {x.w[0], x.w[1], x.w[2], x.w[3], 0, 0, 0, 0};
    return fq_reduce8(r);
}
// Exponentiation and inversion by Fermat (field.rs:89-109).
inline fq fq_pow(fq base, const fq& e) {
    fq r = fq_from_u32(1);
    for (int limb = 0; limb < 4; ++limb)
        for (int bit = 0; bit < 32; ++bit) {
            if ((e.w[limb] >> bit) & 1u) r = fq_mul(r, base);
            base = fq_mul(base, base);
        }
    return r;
}
inline fq fq_inv(const fq& a) {
    const fq qm2{{kQ0 - 2u, kQ1, kQ2, kQ3}};
    return fq_pow(a, qm2);
}

// Inverse by division steps (D. J. Bernstein, B.-Y. Yang, "Fast constant-time gcd
// computation and modular inversion", 2019): the chain of one thread, for challenges
// on the device.
//
// (f, g) starts as (q, a), f always odd.  A step replaces it by (g, (g - f) / 2) if
// delta > 0 and g is odd, else by (f, (g + (g mod 2) f) / 2); delta becomes 1 - delta
// or 1 + delta.  Thirty steps depend on the lowest thirty bits, so they run on 32-bit
// words and leave a matrix, which is then applied to the whole numbers (30-bit limbs)
// and to (d, e) with f = d a, g = e a (mod q); 8 matrices on average, 11 at most (327
// steps, the paper's bound).
//
// Five steps depend on delta and on g / f mod 32 only, and on delta only between -4
// and 4: below, no step swaps, above, just the first with odd g.  Their matrices come
// from a table of 9 x 32 words that a kernel fills in shared memory.  Step by step
// (37 cycles each, what the integer pipe takes for 18 instructions), or by runs of
// zeros (133 cycles for 4 steps), an inverse took about as long as by binary gcd steps
// on whole numbers, 11,200 cycles; now 7,440.  A proof of 52 KB went from 351 to 339 us, of 1 MiB
// from 902 to 889; twelve verifications of 50 KB to 1 MiB files from 4.34 to 4.21 ms.
constexpr uint32_t kInvTable = 9 * 32;
// Word i of the table: steps for delta = i / 32 - 4 and -g / f = i mod 32.  Seven bits
// each of u, v, q, r with 32 f' = u f + v g, 32 g' = q f + r g, then (c + 5) / 2 and the
// sign s of delta' = s delta + c.
DM_HD uint32_t inv_table_word(uint32_t i) {
    int32_t delta = (int32_t)(i / 32) - 4, f = 1, g = -(int32_t)(i % 32), u = 1, v = 0, q = 0, r = 1, c = 0;
    uint32_t minus = 0;
    for (int k = 0; k < 5; ++k) {
        const bool odd = (g & 1) != 0;
        if (odd && delta > 0) {
            const int32_t tf = f, tu = u, tv = v;
            f = g;
            u = q;
            v = r;
            g -= tf;
            q -= tu;
            r -= tv;
            delta = 1 - delta;
            c = 1 - c;
            minus ^= 1u;
        } else {
            if (odd) g += f, q += u, r += v;
            delta += 1;
            c += 1;
        }
        g >>= 1;
        u *= 2;
        v *= 2;
    }
    return ((uint32_t)u & 127u) | ((uint32_t)v & 127u) << 7 | ((uint32_t)q & 127u) << 14 | ((uint32_t)r & 127u) << 21 |
           (uint32_t)((c + 5) / 2) << 28 | minus << 31;
}
// a^-1 mod q, 0 for 0; table: the kInvTable words.
DM_HD fq fq_inv_steps(const fq& a, const uint32_t* table) {
    if (fq_is_zero(a)) return fq_zero();
    constexpr uint32_t kMask = (1u << 30) - 1u;
    constexpr uint32_t kInv75 = 0x162FC963u;  // 75^-1 mod 2^30
    static_assert(((75u * kInv75) & kMask) == 1u, "75^-1");
    int32_t f[4] = {(int32_t)(kMask - 74u), (int32_t)kMask, (int32_t)kMask, (1 << 22) - 1};
    int32_t g[4] = {(int32_t)(a.w[0] & kMask), (int32_t)((a.w[0] >> 30 | a.w[1] << 2) & kMask),
                    (int32_t)((a.w[1] >> 28 | a.w[2] << 4) & kMask), (int32_t)(a.w[2] >> 26 | a.w[3] << 6)};
    int32_t d[4] = {0, 0, 0, 0}, e[4] = {1, 0, 0, 0};
    int32_t delta = 1;
    for (int matrix = 0; matrix < 11 && (g[0] | g[1] | g[2] | g[3]) != 0; ++matrix) {
        uint32_t lf = (uint32_t)f[0] | (uint32_t)f[1] << 30, lg = (uint32_t)g[0] | (uint32_t)g[1] << 30;
        int32_t su = 1, sv = 0, sq = 0, sr = 1;
        DM_UNROLL
        for (int five = 0; five < 6; ++five) {
            const uint32_t w = lf * lg * (lf * lf - 2u);  // -g / f mod 64
            const int32_t near = delta < -4 ? -4 : delta > 4 ? 4 : delta;
            const uint32_t t = table[(uint32_t)((near + 4) * 32) + (w & 31u)];
            const int32_t tu = (int32_t)(t << 25) >> 25, tv = (int32_t)(t << 18) >> 25, tq = (int32_t)(t << 11) >> 25,
                          tr = (int32_t)(t << 4) >> 25;
            const uint32_t nf = (uint32_t)tu * lf + (uint32_t)tv * lg, ng = (uint32_t)tq * lf + (uint32_t)tr * lg;
            lf = nf >> 5;
            lg = ng >> 5;
            const int32_t nu = tu * su + tv * sq, nv = tu * sv + tv * sr;
            sq = tq * su + tr * sq;
            sr = tq * sv + tr * sr;
            su = nu;
            sv = nv;
            delta = ((int32_t)t < 0 ? -delta : delta) + (int32_t)(t >> 27 & 14u) - 5;
        }
        // (f, g) and (d, e) over 2^30, the second made divisible by multiples of q, which
        // is -75 mod 2^30; |d| and |e| grow by q a matrix at most
        int64_t cf = ((int64_t)su * f[0] + (int64_t)sv * g[0]) >> 30, cg = ((int64_t)sq * f[0] + (int64_t)sr * g[0]) >> 30;
        int64_t cd = (int64_t)su * d[0] + (int64_t)sv * e[0], ce = (int64_t)sq * d[0] + (int64_t)sr * e[0];
        const int32_t td = (int32_t)((uint32_t)cd * kInv75 & kMask), te = (int32_t)((uint32_t)ce * kInv75 & kMask);
        cd = (cd - (int64_t)td * 75) >> 30;
        ce = (ce - (int64_t)te * 75) >> 30;
        DM_UNROLL
        for (int i = 1; i < 4; ++i) {
            cf += (int64_t)su * f[i] + (int64_t)sv * g[i];
            cg += (int64_t)sq * f[i] + (int64_t)sr * g[i];
            cd += (int64_t)su * d[i] + (int64_t)sv * e[i];
            ce += (int64_t)sq * d[i] + (int64_t)sr * e[i];
            if (i == 3) {  // q's 2^112 is 2^22 in the last limb
                cd += (int64_t)td << 22;
                ce += (int64_t)te << 22;
            }
            f[i - 1] = (int32_t)((uint32_t)cf & kMask);
            g[i - 1] = (int32_t)((uint32_t)cg & kMask);
            d[i - 1] = (int32_t)((uint32_t)cd & kMask);
            e[i - 1] = (int32_t)((uint32_t)ce & kMask);
            cf >>= 30;
            cg >>= 30;
            cd >>= 30;
            ce >>= 30;
        }
        f[3] = (int32_t)cf;
        g[3] = (int32_t)cg;
        d[3] = (int32_t)cd;
        e[3] = (int32_t)ce;
    }
    // f = +-1 and d = +-a^-1 in (-12 q, 12 q): with 16 q = 2^116 - 1200 added, nonnegative
    const int32_t sign = f[3] < 0 ? -1 : 1;
    int32_t l[4];
    int32_t c = -1200;
    DM_UNROLL
    for (int i = 0; i < 4; ++i) {
        c += sign * d[i] + (i == 3 ? 1 << 26 : 0);
        l[i] = i < 3 ? (int32_t)((uint32_t)c & kMask) : c;
        c >>= 30;
    }
    fq o{{(uint32_t)l[0] | (uint32_t)l[1] << 30, (uint32_t)l[1] >> 2 | (uint32_t)l[2] << 28,
          (uint32_t)l[2] >> 4 | (uint32_t)l[3] << 26, (uint32_t)l[3] >> 6}};
    const uint32_t high = o.w[3] >> 16;  // below 32
    o.w[3] &= 0xFFFFu;
    return fq_add(o, fq_from_u32(75u * high));
}
#if !defined(__CUDA_ARCH__)
// On the host, with a table of its own.
inline fq fq_inv_gcd(const fq& a) {
    static const struct Table {
        uint32_t w[kInvTable];
        Table() {
            for (uint32_t i = 0; i < kInvTable; ++i) w[i] = inv_table_word(i);
        }
    } table;
    return fq_inv_steps(a, table.w);
}
#endif

// ====================== arithmetic modulo an NTT prime ======================

DM_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
DM_HD uint32_t umin32(uint32_t a, uint32_t b) { return a < b ? a : b; }

// x mod p in [0, m) for x in [0, 2m): min(x, x - m) (x - m wraps when x < m).
DM_HD uint32_t red_below(uint32_t x, uint32_t m) { return umin32(x, x - m); }

// Shoup product x * w mod p in [0, 2p) for any x < 2^32, with w < p < 2^31 and
// ws = floor(w * 2^32 / p): q = floor(x * ws / 2^32) is floor(x w / p) or one less.
DM_HD uint32_t shoup_mul(uint32_t x, uint32_t w, uint32_t ws, uint32_t p) {
    const uint32_t q = mulhi32(x, ws);
    return x * w - q * p;
}

// A twiddle (or any constant factor) with its Shoup constant, loaded as one 8-byte word.
struct alignas(8) Tw {
    uint32_t w, s;
};
DM_HD uint32_t shoup_mul(uint32_t x, Tw t, uint32_t p) { return shoup_mul(x, t.w, t.s, p); }

// Generic reductions (any p < 2^32) used by the reference-prime FFI path too.
DM_HD uint32_t add_mod(uint32_t a, uint32_t b, uint32_t p) {
    uint32_t s = a + b;
    return (s < a || s >= p) ? s - p : s;
}
DM_HD uint32_t sub_mod(uint32_t a, uint32_t b, uint32_t p) {
    uint32_t d = a - b;
    return a < b ? d + p : d;
}

// Constants of the nine NTT primes handed to kernels by value.
struct PrimeConsts {
    uint32_t p[kPrimes];
    uint32_t one_s[kPrimes];  // floor(2^32 / p): Shoup constant of 1
    uint32_t c1[kPrimes];     // 2^32 mod p
    uint32_t c1s[kPrimes];    // floor(c1 * 2^32 / p)
    uint32_t c2[kPrimes];     // 2^64 mod p
    uint32_t c2s[kPrimes];
    uint32_t c3[kPrimes];     // 2^96 mod p
};

// A 64-bit value mod p in [0, 4p): hi * (2^32 mod p) + lo * 1, two Shoup products.
DM_HD uint32_t red64_lazy(uint64_t t, const PrimeConsts& c, int i) {
    const uint32_t p = c.p[i];
    return shoup_mul((uint32_t)(t >> 32), c.c1[i], c.c1s[i], p) + shoup_mul((uint32_t)t, 1u, c.one_s[i], p);
}
DM_HD uint32_t red64(uint64_t t, const PrimeConsts& c, int i) {
    const uint32_t p = c.p[i];
    return red_below(red_below(red64_lazy(t, c, i), 2 * p), p);
}
// hi * 2^64 + lo (hi < 2^32) mod p in [0, p).
DM_HD uint32_t red96(uint32_t hi, uint64_t lo, const PrimeConsts& c, int i) {
    const uint32_t p = c.p[i];
    const uint32_t a = red_below(red64_lazy(lo, c, i), 2 * p);            // [0, 2p)
    const uint32_t b = shoup_mul(hi, c.c2[i], c.c2s[i], p);                 // [0, 2p)
    return red_below(red_below(a + b, 2 * p), p);
}

// Residue of a 128-bit word x = sum_j x_j 2^(32 j) modulo prime i, in [0, 4p):
// x_0 + x_1 c1 + x_2 c2 + x_3 c3 < 2^32 + 3 * 2^62 fits one 64-bit accumulation.
DM_HD uint32_t residue_lazy(const fq& x, const PrimeConsts& c, int i) {
    const uint64_t t = (uint64_t)x.w[0] + (uint64_t)x.w[1] * c.c1[i] + (uint64_t)x.w[2] * c.c2[i] +
                       (uint64_t)x.w[3] * c.c3[i];
    return red64_lazy(t, c, i);
}
// The same residue below 8p with one multiply fewer, as a forward transform
// input: the low word (< 2^32 < 16.01p) is brought below 4.01p by two
// conditional subtractions instead of a Shoup product by 1.
DM_HD uint32_t residue_fwd(const fq& x, const PrimeConsts& c, int i) {
    const uint32_t p = c.p[i];
    const uint64_t t = (uint64_t)x.w[0] + (uint64_t)x.w[1] * c.c1[i] + (uint64_t)x.w[2] * c.c2[i] +
                       (uint64_t)x.w[3] * c.c3[i];
    return shoup_mul((uint32_t)(t >> 32), c.c1[i], c.c1s[i], p) + red_below(red_below((uint32_t)t, 8 * p), 4 * p);
}
DM_HD uint32_t residue(const fq& x, const PrimeConsts& c, int i) {
    const uint32_t p = c.p[i];
    return red_below(red_below(residue_lazy(x, c, i), 2 * p), p);
}

// Constants for recombining residues into Z_q (the centred lift that
// src/algebra/ntt.rs:400-427 takes with BigUint): X = sum_i y_i P/p_i - alpha P with
// y_i = r_i (P/p_i)^-1 mod p_i and alpha = round(sum_i y_i / p_i).
struct CrtConsts {
    uint32_t yinv[kPrimes];   // (P / p_i)^-1 mod p_i
    uint32_t yinvs[kPrimes];  // its Shoup constant
    float scale[kPrimes];     // 2^8 / p_i
    float bias;               // -sum_i 2^23 scale_i
    fq cofactor[kPrimes];     // P / p_i mod q
    fq neg_p;                 // -P mod q
};

DM_HD float float_of_bits(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(x);
#else
    float f;
    memcpy(&f, &x, 4);
    return f;
#endif
}
DM_HD uint32_t bits_of_float(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t x;
    memcpy(&x, &f, 4);
    return x;
#endif
}
// 2^23 + (y >> 8) as a float, for y < 2^31 (the bytes of y above the lowest under
// the exponent of 2^23).
DM_HD float float_of_top(uint32_t y) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(__byte_perm(y, 0x4B000000u, 0x7321));
#else
    return float_of_bits(0x4B000000u | (y >> 8));
#endif
}

// y_i = r_i (P/p_i)^-1 mod p_i in [0, p_i) -> the integer X with |X| <= 2^250 < 0.254 P
// congruent to every r_i, reduced mod q.  sum_i y_i / p_i = alpha + X / P lies within
// 0.26 of the integer alpha (2^250 at the largest commitment, 2^26 coefficients) and each
// term drops at most 2^-20 (its lowest byte) plus rounding, so rounding the float
// sum gives alpha exactly.  The four limb columns hold nine products below 2^60 and
// alpha times a limb: below 2^64, with no carry until the end.  Against Garner's
// mixed radix (36 chained Shoup products) it takes nine independent products that
// the inverse transform's final scale already carries, and 40 multiply-adds:
// 4,096 products of degree 512 went from 215.6 to 187.3 us.
DM_HD fq crt_from_scaled(const uint32_t y[kPrimes], const CrtConsts& cc) {
    uint64_t acc[4] = {0, 0, 0, 0};
    float s = cc.bias;
    DM_UNROLL
    for (int i = 0; i < kPrimes; ++i) {
        s += float_of_top(y[i]) * cc.scale[i];
        DM_UNROLL
        for (int w = 0; w < 4; ++w) acc[w] += (uint64_t)y[i] * cc.cofactor[i].w[w];
    }
    // round to the nearest integer in the low bits of 1.5 * 2^23 + s, -0.26 < s < 9.26
    const uint32_t alpha = bits_of_float(s + 12582912.0f) & 15u;
    DM_UNROLL
    for (int w = 0; w < 4; ++w) acc[w] += (uint64_t)alpha * cc.neg_p.w[w];
    uint32_t x[4];
    uint64_t c = acc[0];
    x[0] = (uint32_t)c;
    c = (c >> 32) + acc[1];
    x[1] = (uint32_t)c;
    c = (c >> 32) + acc[2];
    x[2] = (uint32_t)c;
    c = (c >> 32) + acc[3];  // bits 96 and up of a sum below 2^144
    x[3] = (uint32_t)c & 0xFFFFu;
    const uint64_t m = (c >> 16) * 75u;  // 2^112 = 75 (mod q); below 2^39
    fq o;
    c = (uint64_t)x[0] + (uint32_t)m;
    o.w[0] = (uint32_t)c;
    c = (c >> 32) + x[1] + (m >> 32);
    o.w[1] = (uint32_t)c;
    c = (c >> 32) + x[2];
    o.w[2] = (uint32_t)c;
    o.w[3] = (uint32_t)(c >> 32) + x[3];  // o < 2^112 + 2^39
    return fq_canon(o);
}

// The same from the residues r_i < p_i themselves.
DM_HD fq crt_to_fq(const uint32_t r[kPrimes], const PrimeConsts& pc, const CrtConsts& cc) {
    uint32_t y[kPrimes];
    DM_UNROLL
    for (int i = 0; i < kPrimes; ++i) y[i] = red_below(shoup_mul(r[i], cc.yinv[i], cc.yinvs[i], pc.p[i]), pc.p[i]);
    return crt_from_scaled(y, cc);
}

}  // namespace dm
