// 64-bit modular arithmetic shared by host precompute and device kernels.
//
// Device code keeps residues lazily reduced inside an operation (the ranges are stated at the butterflies), between the two
// kernels of a transform also in memory, and leaves the canonical residue in [0,q) when the operation is done, as every stage of
// the reference library does (cahel-main/src/ntt/fntt_2d.cu:860-866, cahel-main/include/uintmodmath.cuh:112-259).
#pragma once
#include <cstdint>
#include <type_traits>

namespace lb {

typedef uint64_t u64;
typedef unsigned __int128 u128;

#if defined(__CUDACC__)
#define LB_HD __host__ __device__ __forceinline__
#define LB_D __device__ __forceinline__
#else
#define LB_HD inline
#define LB_D inline
#endif

// ---- host-only helpers (precompute) ---------------------------------------------------
#if defined(__x86_64__) && !defined(__CUDA_ARCH__)
// 128-by-64 division in one instruction; valid whenever the high half is below q
inline u64 h_div128(u64 hi, u64 lo, u64 q, u64 *rem)
{
    u64 quo, r;
    __asm__("divq %4" : "=a"(quo), "=d"(r) : "a"(lo), "d"(hi), "r"(q) : "cc");
    *rem = r;
    return quo;
}
inline u64 h_mulmod(u64 a, u64 b, u64 q)
{
    if (a >= q) a %= q;
    if (b >= q) b %= q;
    const u128 p = (u128)a * b;
    u64 r;
    h_div128((u64)(p >> 64), (u64)p, q, &r);
    return r;
}
#else
inline u64 h_mulmod(u64 a, u64 b, u64 q) { return (u64)((u128)a * b % q); }
#endif
inline u64 h_powmod(u64 b, u64 e, u64 q)
{
    u64 r = 1 % q;
    b %= q;
    for (; e; e >>= 1) {
        if (e & 1) r = h_mulmod(r, b, q);
        b = h_mulmod(b, b, q);
    }
    return r;
}
inline u64 h_invmod(u64 a, u64 q) { return h_powmod(a % q, q - 2, q); } // q prime
#if defined(__x86_64__) && !defined(__CUDA_ARCH__)
inline u64 h_shoup(u64 w, u64 q)
{
    if (w >= q) return (u64)(((u128)w << 64) / q);
    u64 r;
    return h_div128(w, 0, q, &r);
}
#else
inline u64 h_shoup(u64 w, u64 q) { return (u64)(((u128)w << 64) / q); }
#endif

// ---- the FP64 pipe in the transform kernels -----------------------------------------------------
// Primes below 2^50: the whole butterfly runs on the FP64 pipe.  Residues travel through the
// transform as integer-valued doubles (their bit patterns sit in the same 64-bit words), products
// are formed error-free with fused multiply-adds.  Below 2^47 values may grow over all forward stages
// without a reduction (13.5 q < 2^51); from 2^47 up they are centred every three or four stages.
// Their twiddle entries are (double(w), double(w / q)) with w the representative in (-q/2, q/2).
constexpr u64 kF64TightPrimeLimit = u64(1) << 50; // below it the butterflies run on the FP64 pipe: 2q stays below 2^51
constexpr u64 kF64PrimeLimit = u64(1) << 47;

inline u64 h_bits_of(double d)
{
    u64 bits;
    static_assert(sizeof(bits) == sizeof(d), "double is 64 bits");
    __builtin_memcpy(&bits, &d, sizeof(bits));
    return bits;
}
// the representative of w in (-q/2, q/2) as a double: half the magnitude leaves the butterflies twice the range
inline double h_centred(u64 w, u64 q) { return w > q / 2 ? (double)w - (double)q : (double)w; }
inline u64 h_fp_quot(u64 w, u64 q)
{
    return h_bits_of(h_centred(w, q) / (double)q); // both exact in double, so the quotient is correctly rounded
}
// the two words of a twiddle-table entry for the power w of a root modulo prime q
// (primes below 2^50 run their butterflies on the FP64 pipe: the power as a double, and its quotient by q)
inline u64 h_twiddle_value(u64 w, u64 q) { return q < kF64TightPrimeLimit ? h_bits_of(h_centred(w, q)) : w; }
inline u64 h_twiddle_quot(u64 w, u64 q) { return q < kF64TightPrimeLimit ? h_fp_quot(w, q) : h_shoup(w, q); }

// Per-modulus constants as laid out in device memory (one entry per prime of QP).
struct alignas(16) ModConst {
    u64 q;
    u64 r0, r1;      // floor(2^128 / q), low and high word
    u64 ninv, ninvs; // N^-1 mod q and its Shoup quotient
    u64 iw1n, iw1ns; // psi^-bitrev(1) * N^-1 (last inverse stage fused with the scaling)
    uint32_t kind;   // how 128-bit sums are reduced, one of the three below
    uint32_t near_d; // kWideNear: 2^60 - q
    double qd, qi;   // kWideF64: q, 1 / q, 2^32 / q, the residue of 2^64 nearest zero and its quotient by q
    double qi32, c64, c64q;
    u64 pad;
};
// near 2^60: integer primes with 2^60 - q < 2^28 (what CoeffModulus hands out for 60 bits)
constexpr u64 kNearTop = u64(1) << 60, kNearSpan = u64(1) << 28;
enum : uint32_t { kWideBarrett = 0, kWideNear = 1, kWideF64 = 2 };
inline void h_wide_constants(ModConst &c)
{
    c.kind = c.q < kF64TightPrimeLimit && (c.q >> 34) ? kWideF64 : c.q < kNearTop && kNearTop - c.q < kNearSpan ? kWideNear : kWideBarrett;
    c.near_d = c.kind == kWideNear ? (uint32_t)(kNearTop - c.q) : 0;
    c.qd = (double)c.q;
    c.qi = 1.0 / c.qd;
    c.qi32 = 4294967296.0 * c.qi;
    c.c64 = h_centred((u64)(((u128)1 << 64) % c.q), c.q);
    c.c64q = c.c64 / c.qd;
    c.pad = 0;
}

#if defined(__CUDACC__)
// ---- device arithmetic ----------------------------------------------------------------

// ---- residues as integer-valued doubles (primes below 2^50) --------------------------------------
LB_D double f64_of(u64 bits) { return __longlong_as_double((long long)bits); }
LB_D u64 bits_of(double d) { return (u64)__double_as_longlong(d); }
// an integer below 2^52 as a double: its bits under the exponent of 2^52, minus 2^52
LB_D double f64_from_u52(u64 x) { return __dadd_rn(__longlong_as_double((long long)(x | 0x4330000000000000ull)), -4503599627370496.0); }
// back: a double holding an integer of [0, 2^52)
LB_D u64 u52_from_f64(double d) { return (u64)__double_as_longlong(__dadd_rn(d, 4503599627370496.0)) & 0x000FFFFFFFFFFFFFull; }

// r = y w - Q q with Q an integer next to y w / q: r is congruent to y w and |r| <= 0.75 q.
// Needs integer-valued |y| <= 2^52, |w| <= q < 2^50, |y w / q| <= 2^51 and wq = w / q rounded once; rounded
// twice (w times the rounded 1 / q) the remainder is bounded by q.  y w is split error-free into h + l
// (l = fma(y, w, -h) is exact); Q comes from one fused multiply-add into 1.5 * 2^52, whose rounding is the
// rounding to an integer (the sum stays inside [2^52, 2^53)); the estimate is off by at most 0.5 and the
// error of wq, 2^51 * 2^-53.  h - Q q = r - l with |l| <= 2^48 (half a unit of |y w| <= 2^101) is an integer
// below 2^52 in magnitude, so the second fused multiply-add is exact, and so is the final sum.
LB_D double f64_mulmod(const double y, const double w, const double wq, const double q)
{
    const double h = __dmul_rn(y, w);
    const double l = __fma_rn(y, w, -h);
    const double Q = __dadd_rn(__fma_rn(y, wq, 6755399441055744.0), -6755399441055744.0);
    return __dadd_rn(__fma_rn(-Q, q, h), l);
}
// the residue of an integer-valued |v| < 2^52 nearest to zero: |result| <= q / 2 (+ rounding of 1 / q)
LB_D double f64_centre(const double v, const double q, const double qinv)
{
    const double Q = __dadd_rn(__fma_rn(v, qinv, 6755399441055744.0), -6755399441055744.0);
    return __fma_rn(-Q, q, v);
}
// the canonical residue in [0, q) as an integer
LB_D u64 f64_canon(const double v, const double q, const double qinv)
{
    const double r = f64_centre(v, q, qinv);
    return u52_from_f64(r < 0.0 ? __dadd_rn(r, q) : r);
}

// x * w mod q in [0, 2q) for any 64-bit x, given ws = floor(w 2^64 / q), w < q.
LB_D u64 shoup_lazy(u64 x, u64 w, u64 ws, u64 q)
{
    u64 hi = __umul64hi(x, ws);
    return x * w - hi * q;
}

// The same with the high product formed from three 32 x 32 multiplications instead of four: the quotient comes out at
// most two too small (the product of the low halves and the carries of the cross terms are dropped, each worth less
// than one), so the result is congruent to x w and lies in [0, 4q).  For the butterflies, which only need a bound.
// Spelled out in 32-bit steps: the quotient's cross terms join the high product on a carry chain and both low products go
// into one accumulator (with -q, so that both only add, and a multiply-add takes its addend for free): nine multiplier and
// four adder instructions.  Against the same steps on 64-bit words (shoup_lazy4_words below), which the compiler pads with
// moves: 37.9 instead of 42.9 cycles per butterfly and SM partition in the four stages of a prime near 2^60 on registers only,
// 768 limbs of N = 2^16 near 2^60 542 instead of 590 us forward and 598 instead of 636 inverse.  B200 issues a 32 x 32 + 32
// multiplication at 64 lanes per clock and SM and one whose high half is used at 32, so the quotient is two thirds of the cost.
LB_D u64 shoup_lazy4(u64 x, u64 w, u64 ws, u64 q)
{
    u64 r;
    asm("{\n\t"
        ".reg .u32 xl, xh, wl, wh, sl, sh, t, c, ql, qh, nl, nh, rl, rh;\n\t"
        ".reg .u64 h, p;\n\t"
        "mov.b64 {xl, xh}, %1;\n\t"
        "mov.b64 {wl, wh}, %2;\n\t"
        "mov.b64 {sl, sh}, %3;\n\t"
        "mov.b64 {nl, nh}, %4;\n\t"
        "mul.hi.u32 t, xh, sl;\n\t"
        "mul.hi.u32 c, xl, sh;\n\t"
        "mul.wide.u32 h, xh, sh;\n\t"
        "mov.b64 {ql, qh}, h;\n\t"
        "add.cc.u32 ql, ql, t;\n\t"
        "addc.u32 qh, qh, 0;\n\t"
        "add.cc.u32 ql, ql, c;\n\t"
        "addc.u32 qh, qh, 0;\n\t"
        "mul.wide.u32 p, xl, wl;\n\t"
        "mad.wide.u32 p, ql, nl, p;\n\t"
        "mov.b64 {rl, rh}, p;\n\t"
        "mad.lo.u32 rh, xl, wh, rh;\n\t"
        "mad.lo.u32 rh, xh, wl, rh;\n\t"
        "mad.lo.u32 rh, ql, nh, rh;\n\t"
        "mad.lo.u32 rh, qh, nl, rh;\n\t"
        "mov.b64 %0, {rl, rh};\n\t"
        "}"
        : "=l"(r)
        : "l"(x), "l"(w), "l"(ws), "l"(0 - q));
    return r;
}

// The same on 64-bit words, for the one-kernel transforms (ntt.cu): their passes of three stages lost with the steps above
// (inverse of one to six limbs of N = 2048 and 57 to 60 bits 8.2 to 9.3 us against 9.2 to 10.3), the two-kernel ones gain.
LB_D u64 shoup_lazy4_words(u64 x, u64 w, u64 ws, u64 q)
{
    const uint32_t xh = (uint32_t)(x >> 32), xl = (uint32_t)x, sh = (uint32_t)(ws >> 32), sl = (uint32_t)ws;
    const u64 hi = (u64)xh * sh + __umulhi(xh, sl) + __umulhi(xl, sh);
    return x * w - hi * q;
}

LB_D u64 shoup_mul(u64 x, u64 w, u64 ws, u64 q)
{
    u64 r = shoup_lazy(x, w, ws, q);
    return r >= q ? r - q : r;
}

LB_D u64 csub(u64 x, u64 q) { return x >= q ? x - q : x; }

LB_D u64 add_mod(u64 a, u64 b, u64 q) { return csub(a + b, q); }
LB_D u64 sub_mod(u64 a, u64 b, u64 q) { return a >= b ? a - b : a + q - b; }

// x mod q for any 64-bit x, bhi = floor(2^64 / q)
LB_D u64 barrett64(u64 x, u64 q, u64 bhi)
{
    u64 s = __umul64hi(x, bhi);
    u64 r = x - s * q;
    return r >= q ? r - q : r;
}

struct u128d {
    u64 lo, hi;
};

LB_D u128d mul_wide(u64 a, u64 b)
{
    u128d r;
    r.lo = a * b;
    r.hi = __umul64hi(a, b);
    return r;
}

// acc += a * b; the 128-bit integer type lets the compiler share partial products between the
// two halves and keep the additions on the carry chain
LB_D void mac_wide(u128d &acc, u64 a, u64 b)
{
    const u128 s = ((u128)acc.hi << 64 | acc.lo) + (u128)a * b;
    acc.lo = (u64)s;
    acc.hi = (u64)(s >> 64);
}

// (hi:lo) mod q with the two-word ratio floor(2^128 / q) = (r1:r0); exact for q < 2^62.
LB_D u64 barrett128(u128d z, u64 q, u64 r0, u64 r1)
{
    // quotient estimate: floor(z * ratio / 2^128), dropping the lowest partial product
    u64 carry = __umul64hi(z.lo, r0);
    u64 t_lo = z.lo * r1;
    u64 t_hi = __umul64hi(z.lo, r1);
    u64 s = t_lo + carry;
    u64 c1 = t_hi + (s < t_lo);
    u64 u_lo = z.hi * r0;
    u64 u_hi = __umul64hi(z.hi, r0);
    u64 s2 = s + u_lo;
    u64 c2 = u_hi + (s2 < u_lo);
    u64 qhat = z.hi * r1 + c1 + c2;
    u64 r = z.lo - qhat * q;
    // the estimate is short by at most 2
    r = csub(r, q << 1);
    return csub(r, q);
}

// ---- reductions of products and sums of products ---------------------------------------------------
// Two classes of primes have cheaper reductions than the two-word Barrett quotient (18 products of 32 x 32 bits):
//   near 2^60   2^64 = 16 d and 2^60 = d modulo q with d = 2^60 - q < 2^28, so the high half folds onto the low one with
//               four products;
//   FP64        2^34 <= q < 2^50: the high half times 2^64 mod q and the quotient of the low half are formed on the
//               FP64 pipe, which these kernels leave idle otherwise.
// The reductions, not the products they belong to, were what bounded the element-wise kernels and the inner product.

// any 64-bit word -> congruent word below 2^60 + 15 (2^60 - q)
LB_D u64 near_reduce(const u64 v, const uint32_t d)
{
    return (v & (kNearTop - 1)) + (u64)(uint32_t)(v >> 60) * d;
}
// any 128-bit word -> congruent word below 2^60 + 15 (2^60 - q).  The first fold leaves 96 bits: (2^64 - 1) 16 d + 2^64 < 2^96;
// the second 64 and a carry, whose 16 d fit because the wrapped sum is below 2^64 - 16 d.
LB_D u64 near_fold(const u128d z, const uint32_t d)
{
    const uint32_t d16 = d << 4;
    const u64 p0 = (u64)(uint32_t)z.hi * d16, p1 = (u64)(uint32_t)(z.hi >> 32) * d16;
    const u128 t = (u128)z.lo + p0 + ((u128)p1 << 32);
    const u64 lo = (u64)t, p2 = (u64)(uint32_t)(t >> 64) * d16;
    u64 r = lo + p2;
    r += r < lo ? d16 : 0u;
    return near_reduce(r, d);
}

// x mod q for any 64-bit x as an integer of magnitude at most q / 2 + 2^32, for 2^34 <= q < 2^50.  The quotient, below 2^30, is
// taken from the upper half of x and read out of the mantissa of 1.5 * 2^52 + quotient.
LB_D u64 f64_fold64(const u64 x, const ModConst &m)
{
    const double xh = __dadd_rn(__hiloint2double(0x43300000, (int)(x >> 32)), -4503599627370496.0);
    const uint32_t Q = (uint32_t)__double2loint(__fma_rn(xh, m.qi32, 6755399441055744.0));
    return x - (u64)Q * m.q;
}
// a signed integer of magnitude below 2^51 (two's complement) as a double
LB_D double f64_from_s52(const u64 x) { return __dadd_rn(f64_of(x + 0x4338000000000000ull), -6755399441055744.0); }
// (hi:lo) mod q as an integer-valued double of magnitude at most 1.5 q (0.75 q from the high half, q / 2 + 2^32 from the low one),
// for 2^34 <= q < 2^50 and hi < 2^52: |hi c64 / q| <= 2^51 is the range of the quotient in f64_mulmod
LB_D double f64_fold(const u128d z, const ModConst &m)
{
    const double h = f64_mulmod(f64_from_u52(z.hi), m.c64, m.c64q, m.qd);
    return __dadd_rn(__dadd_rn(h, f64_of(f64_fold64(z.lo, m) + 0x4338000000000000ull)), -6755399441055744.0);
}

// (hi:lo) mod q, canonical.  kWideF64 takes hi < 2^52: sums of 2^15 products of residues, or of 64 products of a residue
// with a 60-bit word.
template <uint32_t KIND>
LB_D u64 reduce_wide(const u128d z, const ModConst &m)
{
    if (KIND == kWideNear) return csub(near_fold(z, m.near_d), m.q);
    if (KIND == kWideF64) return f64_canon(f64_fold(z, m), m.qd, m.qi);
    return barrett128(z, m.q, m.r0, m.r1);
}
LB_D u64 reduce_wide(const u128d z, const ModConst &m)
{
    if (m.kind == kWideNear) return reduce_wide<kWideNear>(z, m);
    if (m.kind == kWideF64) return reduce_wide<kWideF64>(z, m);
    return reduce_wide<kWideBarrett>(z, m);
}

// canonical product of residues.  FP64: |a b / q| < 2^50, so the quotient is off by at most 0.5 + 2^-2 as in f64_mulmod
// although its factor b / q is rounded twice.
template <uint32_t KIND>
LB_D u64 mul_mod(const u64 a, const u64 b, const ModConst &m)
{
    if (KIND == kWideF64) {
        const double w = f64_from_u52(b);
        return f64_canon(f64_mulmod(f64_from_u52(a), w, __dmul_rn(w, m.qi), m.qd), m.qd, m.qi);
    }
    return reduce_wide<KIND>(mul_wide(a, b), m);
}
LB_D u64 mul_mod(const u64 a, const u64 b, const ModConst &m)
{
    if (m.kind == kWideNear) return mul_mod<kWideNear>(a, b, m);
    if (m.kind == kWideF64) return mul_mod<kWideF64>(a, b, m);
    return mul_mod<kWideBarrett>(a, b, m);
}

// calls body with the prime's class as a compile-time constant
template <class F>
LB_D void with_wide_kind(const uint32_t kind, const F &body)
{
    if (kind == kWideNear) body(std::integral_constant<uint32_t, kWideNear>());
    else if (kind == kWideF64) body(std::integral_constant<uint32_t, kWideF64>());
    else body(std::integral_constant<uint32_t, kWideBarrett>());
}
#endif

} // namespace lb
