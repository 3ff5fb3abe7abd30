// fp64_int.cuh -- lbc's FP64 moments and collision, bit for bit, mostly on the
// integer pipes.
//
// GB300 issues an FP64 instruction of a warp every 64 cycles per SM
// sub-partition (76 with all four busy), an integer instruction every 2
// (measured: DADD, DMUL, DFMA 76, LOP3 / SHF / IMAD 2.1, IMAD.WIDE 6.5). The
// exact step (moments_exact, collide_exact) is 125 FP64 instructions per node
// and bound by them: 1024 x 1024 periodic 253 us per step, 4.1 GLUPS. An
// addition of numbers of known range is about a dozen integer instructions on
// 64-bit fixed point, its round-to-nearest-even included, and a product of two
// 53-bit mantissas about twenty. In this form a force-free node takes 24 FP64
// instructions (the relaxation's product and the final additions, u.u and the
// diagonal velocities) beside 1020 ALU and 580 multiply-add instructions:
// 71.5 us per step, 14.7 GLUPS, with the FP64 pipe 57 % and the ALU 77 % busy,
// so that neither alone bounds it. (80 registers, three blocks of 256 threads
// or six of 128 per SM; in an earlier form of 72.8 us 64 registers took 74.5, 99
// registers 77.2, and additions moved to the multiply-add pipe by hand, as
// multiplications by 1, 81.6.)
//
// Nothing is approximated: every operation returns the FP64 result that
// moments_exact / collide_exact round to. The fixed-point forms hold for the
// ranges of an ordinary flow, checked per node; any other node takes
// moments_exact and collide_exact, or the latter alone. Ranges: populations in
// [2^-8, 1) (f_1 .. f_8 below 1/2), 9/16 <= rho < 2, |c.u| < 1/4 (the equilibria
// are then above 2^-8), |f - f_eq| < 2^-9 (2^-6 where no f or f_eq is below 2^-6).
// Zeros come out with lbc's value; their sign is not kept.
//
// The division by the density is an integer one: a 64-bit reciprocal by Newton
// steps from the FP32 one, shared by both velocities, and the exact remainder
// to decide the last bit.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define LBM_HD __host__ __device__ __forceinline__
#else
#define LBM_HD inline
#endif

namespace lbm {
namespace fi {

struct W2 { uint32_t lo, hi; };

LBM_HD W2 words(double x) {
#ifdef __CUDA_ARCH__
    return W2{(uint32_t)__double2loint(x), (uint32_t)__double2hiint(x)};
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return W2{(uint32_t)b, (uint32_t)(b >> 32)};
#endif
}
LBM_HD double make_double(uint32_t lo, uint32_t hi) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t b = ((uint64_t)hi << 32) | lo;
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
LBM_HD uint64_t u64(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
LBM_HD uint32_t lo32(uint64_t v) { return (uint32_t)v; }
LBM_HD uint32_t hi32(uint64_t v) { return (uint32_t)(v >> 32); }

// (hi:lo << (s mod 32)) >> 32
LBM_HD uint32_t shl_wide(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    s &= 31;
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
// low word of hi:lo >> (s mod 32)
LBM_HD uint32_t shr_wide(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    s &= 31;
    return s ? (lo >> s) | (hi << (32 - s)) : lo;
#endif
}
// Position of the highest set bit, -1 for 0; of the highest bit that differs
// from the sign for the signed form.
LBM_HD int top_bit(uint32_t x) {
#ifdef __CUDA_ARCH__
    int r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
#else
    return x ? 31 - __builtin_clz(x) : -1;
#endif
}
LBM_HD int top_bit_signed(int32_t x) {
#ifdef __CUDA_ARCH__
    int r;
    asm("bfind.s32 %0, %1;" : "=r"(r) : "r"(x));
    return r;
#else
    return top_bit(x < 0 ? ~(uint32_t)x : (uint32_t)x);
#endif
}
// 2^n - 1; all ones for n > 31 (unsigned).
LBM_HD uint32_t ones(int n) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(r) : "r"(n));
    return r;
#else
    return (uint32_t)n > 31u ? 0xFFFFFFFFu : (1u << n) - 1u;
#endif
}
// x >> (n mod 32)
LBM_HD uint32_t shr32(uint32_t x, int n) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(x, 0u, (uint32_t)n);
#else
    return x >> (n & 31);
#endif
}
// Shifts with the PTX meaning (64 or more gives 0).
LBM_HD uint64_t shr(uint64_t v, uint32_t n) {
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
#else
    return n >= 64 ? 0 : v >> n;
#endif
}
LBM_HD uint64_t shl(uint64_t v, uint32_t n) {
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
#else
    return n >= 64 ? 0 : v << n;
#endif
}
LBM_HD double add(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
LBM_HD double mul(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}

// Round v to 53 significant bits, ties to even, by clearing the low
// d = (bit length - 53) bits, d >= 1. Works on two's complement as it stands
// (rounding v + half - 1 + odd down is to nearest even for either sign).
LBM_HD uint64_t round_low(uint64_t v, int d) {
    v += (uint64_t)(ones(d - 1) + (shr32(lo32(v), d) & 1u));
    return u64(lo32(v) & ~ones(d), hi32(v));
}
// v of 54 to 64 bits, or 0.
LBM_HD uint64_t round53(uint64_t v) { return round_low(v, top_bit(hi32(v)) - 20); }
// Signed, |v| < 2^63, bit 0 clear when |v| < 2^53 (one bit is always dropped).
LBM_HD int64_t round53_signed(int64_t v) {
    const int d = top_bit_signed((int32_t)hi32((uint64_t)v)) - 20;
    return (int64_t)round_low((uint64_t)v, d > 1 ? d : 1);
}

// A population as fixed point of 2^-61: needs 2^-8 <= x < 1, else bad gets
// bits above 7 (negative, infinite and NaN values included).
LBM_HD uint64_t pop_fixed(double x, uint32_t &bad) {
    const W2 b = words(x);
    const uint32_t t = (b.hi >> 20) - (1023u - 8u);  // exponent + 8
    bad |= t;
    const uint32_t m = (b.hi & 0xFFFFFu) | 0x100000u, s = t + 1;
    return u64(shl_wide(0, b.lo, s), shl_wide(b.lo, m, s));
}

LBM_HD uint64_t negate_if(uint64_t v, uint32_t sgn) {
    const uint64_t s = u64(sgn, sgn);
    return (v ^ s) - s;
}
// v 2^-n, bits shifted out kept as a sticky bit 0. 64 or more give zero: below
// 2^-62 beside numbers near 1 of 53 bits, which no rounding here sees.
LBM_HD uint64_t shr_sticky(uint64_t v, uint32_t n) {
    const uint64_t lost = shl(v, 64u - n);
    return shr(v, n) | (uint64_t)((lo32(lost) | hi32(lost)) != 0u);
}
// a * b: the high 64 bits, with bit 0 set when the low 64 are not zero.
LBM_HD uint64_t mul_high_sticky(uint64_t a, uint64_t b) {
    const uint64_t ll = (uint64_t)lo32(a) * lo32(b);
    const uint64_t lh = (uint64_t)lo32(a) * hi32(b) + hi32(ll);
    const uint64_t m = (uint64_t)hi32(a) * lo32(b) + lo32(lh);
    const uint64_t h = (uint64_t)hi32(a) * hi32(b) + hi32(lh) + hi32(m);
    return h | (uint64_t)((lo32(ll) | lo32(m)) != 0u);
}
// The high 64 bits of a * b.
LBM_HD uint64_t mul_high(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// A number as sign (all ones when negative), mantissa and exponent:
// |x| = m 2^-e, m left-justified (bit 63 set) unless x = 0 (m = 0, e large).
struct Num {
    uint64_t m;
    uint32_t e, sgn;
};

LBM_HD Num num_of(double x) {  // normal x or zero
    const W2 b = words(x);
    const uint32_t ex = (b.hi >> 20) & 0x7FFu;
    Num r;
    r.sgn = (uint32_t)((int32_t)b.hi >> 31);
    r.e = 1023u + 63u - ex;
    r.m = ex ? u64(b.lo << 11, shl_wide(b.lo, b.hi, 11) | 0x80000000u) : 0;
    return r;
}
LBM_HD Num num_of_fixed(int64_t v, uint32_t lsb) {  // v 2^-lsb, |v| < 2^63
    Num r;
    r.sgn = (uint32_t)((int32_t)hi32((uint64_t)v) >> 31);
    const uint64_t a = negate_if((uint64_t)v, r.sgn);
    const int ph = top_bit(hi32(a)), pl = top_bit(lo32(a));
    const int z = 63 - (ph >= 0 ? ph + 32 : pl);  // 64 for v = 0
    r.m = shl(a, (uint32_t)z);
    r.e = lsb + (uint32_t)z;
    return r;
}
// The FP64 value of x (53 significant bits; normal or zero).
LBM_HD double value_of(const Num &x) {
    const uint32_t e = (1023u + 62u - x.e) << 20;
    const uint64_t m = x.m >> 11;
    return x.m ? make_double(lo32(m), (hi32(m) + e) | (x.sgn & 0x80000000u)) : 0.0;
}

// The FP64 value of a fixed-point integer of LSB 2^-lsb with at most 53
// significant bits, highest bit at 53 or above.
LBM_HD double from_fixed(uint64_t v, int lsb) {
    const int d = top_bit(hi32(v)) - 20;
    const uint64_t m = shr(v, (uint32_t)d);
    return make_double(lo32(m), hi32(m) + ((uint32_t)(1023 + 52 - 1 - lsb + d) << 20));
}
// 1/d for d = D 2^-63 in [1/2, 1), as an integer of LSB 2^-63, below the true
// value by less than 8 units: the FP32 reciprocal, then two Newton steps.
// The FP32 number that stands for d: above d's first 24 bits by 3 2^-24 at most,
// and so far above 1/2 that a reciprocal 2^-23 off (the bound of rcp.approx) is
// below 2.
LBM_HD uint32_t recip_arg(uint64_t D) {
    return 0x3F000000u | (hi32(D << 1) >> 8 & 0x7FFFFFu) | 3u;
}
// yb: the bits of its reciprocal, between 1 - 2^-24 and 2.
LBM_HD uint64_t recip_refine(uint64_t D, uint32_t yb) {
    const uint32_t dh = hi32(D) << 1 | lo32(D) >> 31, dl = lo32(D) << 1;  // LSB 2^-64
    // LSB 2^-31: the exponent's last bit is 2^31; 1 - 2^-24 (exponent one less,
    // mantissa of ones) gives 2^31 - 2^8 of its own accord
    const uint32_t y0 = yb << 8;
    // e = 1 - d y0, |e| < 2^-20, LSB 2^-63
    const uint64_t t = (uint64_t)dh * y0 + (((uint64_t)dl * y0) >> 32);
    const int32_t e0 = (int32_t)((int64_t)(0x8000000000000000ull - t) >> 11);  // LSB 2^-52
    const uint64_t y1 = ((uint64_t)y0 << 32) + (uint64_t)(((int64_t)e0 * (int64_t)(y0 >> 1)) >> 19);
    // |1 - d y1| < 2^-40
    const int32_t e1 = (int32_t)(uint32_t)(0x8000000000000000ull - mul_high(u64(dl, dh), y1));
    // 4 units off keep 1/d = 2 inside 64 bits
    return y1 + (uint64_t)(((int64_t)e1 * (int64_t)(hi32(y1) >> 1)) >> 30) - 4u;
}
LBM_HD uint64_t recip_fixed(uint64_t D) {
    const uint32_t db = recip_arg(D);
    uint32_t yb;
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(db)));
    yb = __float_as_uint(y);
#else
    float df, y;
    std::memcpy(&df, &db, 4);
    y = 1.0f / df;
    std::memcpy(&yb, &y, 4);
#endif
    return recip_refine(D, yb);
}

// a / d rounded to FP64 for a of at most 53 significant bits and d = D 2^-63
// in [1/2, 1) of 53, Y = recip_fixed(D). The quotient of the left-justified
// mantissas to within a few units of 2^-63 gives its nearest 54-bit number m.
// An even m is half the result; an odd one is a midpoint, and the side on
// which the quotient lies is the sign of the remainder (exact modulo 2^64;
// never zero: a 54-bit odd number times D is no 53-bit number).
LBM_HD Num divide(const Num &a, uint64_t D, uint64_t Y) {
    const uint64_t Q = mul_high(a.m, Y);      // LSB 2^-63, [2^62, 2^64)
    const uint32_t big = hi32(Q) >> 31;       // quotient of 1 or more: 11 bits go, else 10
    const uint64_t m = shr(Q + ((uint64_t)256u << big), 9u + big);
    const uint64_t md = m * D;
    const int32_t rem = (int32_t)((lo32(a.m) << (21u - big)) - hi32(md) - (lo32(md) != 0u));
    const uint32_t up = (uint32_t)(~rem) >> 31;  // 1 when the remainder is not negative
    const uint64_t r = (m >> 1) + (lo32(m) & up);
    // r of 53 bits (2^53 after a carry)
    const uint32_t carry = hi32(r) >> 21;
    Num q;
    q.m = shl(r, 11u - carry);
    q.e = a.e - big - carry;
    q.sgn = a.sgn;
    return q;
}

struct Moments {
    uint64_t s;        // rho, LSB 2^-61
    uint64_t D;        // rho = D 2^-(61 + sb), bit 62 of D set
    uint32_t sb;       // 1 or 2
    Num ux, uy;
};

// Moments (moments_exact) of the populations F of LSB 2^-61, all in
// [2^-8, 1) and F[1..8] < 1/2; bad as in pop_fixed.
LBM_HD Moments moments(const uint64_t F[9], bool force, double hFx, double hFy, uint32_t &bad) {
    Moments q;
    uint64_t s = F[0];
#pragma unroll
    for (int k = 1; k < 9; k++) s = round53(s + F[k]);
    int64_t a = round53_signed((int64_t)(F[1] - F[3]));
    a = round53_signed(a + (int64_t)F[5]);
    a = round53_signed(a - (int64_t)F[6]);
    a = round53_signed(a - (int64_t)F[7]);
    a = round53_signed(a + (int64_t)F[8]);
    int64_t b = round53_signed((int64_t)(F[2] - F[4]));
    b = round53_signed(b + (int64_t)F[5]);
    b = round53_signed(b + (int64_t)F[6]);
    b = round53_signed(b - (int64_t)F[7]);
    b = round53_signed(b - (int64_t)F[8]);
    // 9/16 <= rho < 2
    bad |= (hi32(s) - 0x12000000u >= 0x40000000u - 0x12000000u) ? 0x80000000u : 0u;
    q.s = s;
    q.sb = 1u + ((hi32(s) >> 29) ^ 1u);
    q.D = shl(s, q.sb);
    const uint64_t Y = recip_fixed(q.D);
    Num jx = num_of_fixed(a, 61), jy = num_of_fixed(b, 61);
    if (force) {
        const double fx = add(value_of(jx), hFx), fy = add(value_of(jy), hFy);
        jx = num_of(fx);
        jy = num_of(fy);
        // subnormal quotients are the FP64 pipe's
        bad |= ((jx.e > 563u && fx != 0.0) || (jy.e > 563u && fy != 0.0)) ? 0x80000000u : 0u;
    }
    q.ux = divide(jx, q.D, Y);
    q.uy = divide(jy, q.D, Y);
    q.ux.e += 2u - q.sb;
    q.uy.e += 2u - q.sb;
    return q;
}

// f - f_eq for f_eq = (w rho) * bracket, as sign (bit 63) and magnitude of LSB
// 2^-61, exact. Br: the bracket, LSB 2^-62, 53 significant bits; wr: w_1 rho, LSB
// 2^-(65 + sb); n = sb, 2 + sb, 4 + sb for w_0 = 4 w_1, w_1 and w_5 = w_1 / 4
// (exact in FP64: powers of two apart). big and low collect the magnitudes'
// words.
LBM_HD uint64_t excess(uint64_t F, uint64_t wr, uint32_t n, uint64_t Br, uint32_t &big, uint32_t &low) {
    // f_eq: product rounded to 53 bits, then to LSB 2^-61 (exact: f_eq >= 2^-8)
    const uint64_t d = F - shr(round53(mul_high_sticky(wr, Br)), n);
    const uint64_t a = (int32_t)hi32(d) < 0 ? 0ull - d : d;
    big |= hi32(a);
    low |= lo32(a);
    return u64(lo32(a), hi32(a) | (hi32(d) & 0x80000000u));
}

// -omega (f - f_eq), one rounding: 2^(s-9) + |f - f_eq| is the FP64 number whose
// mantissa is the magnitude (its low s bits, which are zero, dropped), and
// omega times that minus omega 2^(s-9) is exact but for the multiply-add's own
// rounding. om_m = -omega 2^(s-9).
LBM_HD double relax(uint64_t x, uint32_t s, double om, double om_m) {
    const uint32_t h = hi32(x) & 0x7FFFFFFFu;
    const double m = make_double(shr_wide(lo32(x), h, s), (h >> s) | ((1023u - 9u + s) << 20));
    const W2 w = words(fma(om, m, om_m));
    return make_double(w.lo, w.hi ^ (~hi32(x) & 0x80000000u));
}

// How far step_node_parts got: a range check failed before the moments, after
// them (rho, ux, uy are lbc's), or none did.
enum Done : int { DONE_NOTHING = 0, DONE_MOMENTS = 1, DONE_ALL = 2 };

// One node: moments, then (COLLIDE) the collided populations in f, which stays
// as it was when a range check fails. Needs lbc's weights w and an ordinary
// omega (the caller's checks). A node whose collision is out of range keeps its
// moments, so that the FP64 pipe only collides it, and one whose populations are
// is refused before anything else. Vortices at speeds up to 0.3, us per step: 64^2
// 8.3, 256^2 20.7, 512^2 51, 1024^2 165 (with the moments taken again 256^2 25.7,
// 1024^2 217; all on the FP64 pipe 12.5, 21.7, 67, 252). Density 2.5: 7.0, 20.9,
// 66.9, 251.
template <bool COLLIDE>
LBM_HD int step_node_parts(double f[9], const double w[9], bool force, double hFx, double hFy, double om, double Fx,
                      double Fy, double &rho, double &ux, double &uy) {
    uint32_t bad = 0, half = 0;
    uint64_t F[9];
    F[0] = pop_fixed(f[0], bad);
#pragma unroll
    for (int k = 1; k < 9; k++) {
        F[k] = pop_fixed(f[k], bad);
        half |= hi32(F[k]);
    }
    bad |= half & 0xF0000000u;
    if (bad > 7u) return DONE_NOTHING;
    const Moments q = moments(F, force, hFx, hFy, bad);
    if (bad > 7u) return DONE_NOTHING;
    rho = from_fixed(q.s, 61);
    ux = value_of(q.ux);
    uy = value_of(q.uy);
    if (!COLLIDE) return DONE_ALL;

    const uint64_t kNinth = 0xE38E38E38E38E000ull;  // the FP64 number 1/9, LSB 2^-67
    const uint64_t wr = round53(mul_high_sticky(kNinth, q.D << 1));
    const Num tn = num_of(mul(1.5, add(mul(ux, ux), mul(uy, uy))));
    uint32_t far = 0, big = 0, low = 0;
    const uint64_t T = shr_sticky(tn.m, tn.e - 62u);
    const uint64_t one = 1ull << 62;
    const Num c[4] = {q.ux, q.uy, num_of(add(ux, uy)), num_of(add(uy, -ux))};
    uint64_t x[9];
    // For |c.u| < 1/4 every bracket is above 1/4.
    const uint64_t b0 = round_low(one - T, 9);  // 3/4 < 1 - T <= 1
    x[0] = excess(F[0], wr, q.sb, b0, big, low);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int ka = i < 2 ? 1 + i : 3 + i, kb = ka + 2;  // (1,3) (2,4) (5,7) (6,8)
        far |= c[i].e - 66u;                                 // |c.u| < 1/4
        const uint64_t m = c[i].m >> 11;
        // 3 c.u and (4.5 c.u) c.u, each operation rounded to 53 bits
        const bool neg = c[i].sgn != 0;
        const uint64_t B = shr_sticky(round53(3u * m) << 8, c[i].e - 65u);
        const uint64_t A = shr_sticky(round53(mul_high_sticky(round53(9u * m) << 7, c[i].m)), 2u * c[i].e - 129u);
        // 1 + |B| + A in [1, 2) (bit 31 of far otherwise): 10 bits go
        const uint64_t p2 = round_low(round_low(one + B, 10) + A, 10);
        far |= hi32(p2);
        const uint64_t p3 = round53(p2 - T), m3 = round53(round53(round53(one - B) + A) - T);
        const uint64_t bp = neg ? m3 : p3, bm = neg ? p3 : m3;
        x[ka] = excess(F[ka], wr, (i < 2 ? 2u : 4u) + q.sb, bp, big, low);
        x[kb] = excess(F[kb], wr, (i < 2 ? 2u : 4u) + q.sb, bm, big, low);
    }
    // Below 2^-9 as they are; below 2^-6 without their low three bits, which are
    // zero when f and f_eq are 2^-6 or more.
    const uint32_t sh = big >> 20 ? 3u : 0u;
    if ((big >> 23) || (sh && (low & 7u)) || (far >> 31)) return DONE_MOMENTS;
    const double om_m = make_double(words(om).lo, words(om).hi + 0x80000000u - ((9u - sh) << 20));
    double r[9];
#pragma unroll
    for (int k = 0; k < 9; k++) r[k] = relax(x[k], sh, om, om_m);
    if (!force) {
#pragma unroll
        for (int k = 0; k < 9; k++) f[k] = add(f[k], r[k]);
        return DONE_ALL;
    }
    // Guo's term (collide_exact): w (3 c.F + 9 (c.u)(c.F) - 3 u.F), in the FP64
    // sequence. The pair's product (9 c.u)(c.F) is the same for both directions;
    // a direction across the force has 3 u.F alone, and its w_1 multiple serves
    // the rest population (w_0 = 4 w_1). Zero terms are left out: x + 0 = x.
    const bool fx = Fx != 0.0, fy = Fy != 0.0;
    const double uF = !fy ? mul(ux, Fx) : !fx ? mul(uy, Fy) : add(mul(ux, Fx), mul(uy, Fy));
    const double uF3 = mul(3.0, uF);
    const double g = add(1.0, -mul(0.5, om));
    const double across = mul(g, mul(w[1], -uF3));
    f[0] = add(f[0], add(r[0], mul(4.0, across)));
    const double cF[4] = {Fx, Fy, add(Fx, Fy), add(Fy, -Fx)};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int ka = i < 2 ? 1 + i : 3 + i, kb = ka + 2;
        double ta = across, tb = across;
        if (i == 0 ? fx : i == 1 ? fy : true) {
            const double cu = i == 0 ? ux : i == 1 ? uy : i == 2 ? add(ux, uy) : add(uy, -ux);
            const double L = mul(3.0, cF[i]), X = mul(mul(9.0, cu), cF[i]);
            ta = mul(g, mul(w[ka], add(add(L, X), -uF3)));
            tb = mul(g, mul(w[kb], add(add(-L, X), -uF3)));
        }
        f[ka] = add(f[ka], add(r[ka], ta));
        f[kb] = add(f[kb], add(r[kb], tb));
    }
    return DONE_ALL;
}

// The same, all or nothing.
template <bool COLLIDE>
LBM_HD bool step_node(double f[9], const double w[9], bool force, double hFx, double hFy, double om, double Fx,
                      double Fy, double &rho, double &ux, double &uy) {
    return step_node_parts<COLLIDE>(f, w, force, hFx, hFy, om, Fx, Fy, rho, ux, uy) == DONE_ALL;
}

}  // namespace fi
}  // namespace lbm
