// Register-level stages of the two-kernel transforms (ntt_twopass.cuh): up to four consecutive
// butterfly stages on 2^S values a thread holds, with the range of every value known at compile time.
//
// The stage loops are unrolled in full, so the bounds below (in hundredths of q) are constants to the
// compiler and a reduction is emitted only for the elements that need one:
//   FP64 pipe    residues as integer-valued doubles, twiddles in (-q/2, q/2), so |y w / q| <= |y| / 2 and a
//                product is at most 0.75 q.  With q < 2^50 a multiplicand may reach 4q and a value 4q
//                before 2^51 (the quotient's range) and 2^52 come into reach.
//   near 2^60    integer primes with 2^60 - q < 2^28 (what CoeffModulus hands out for 60 bits): any 64-bit
//                word v comes back to about q by (v mod 2^60) + (v >> 60) (2^60 - q), three instructions
//                against six of a conditional subtraction, and 64 bits hold 16 q, so the forward stages reduce
//                half of the values once per four stages instead of a value per butterfly.
//   integer      the remaining primes of 50 bits and more keep values in [0, 8q) with a conditional subtraction per butterfly.
//                A class of its own for primes below 2^58, without that subtraction but with the four-multiplication product,
//                was 1 to 4 % slower (768 limbs of 57 bits at N = 2^15 292 us against 282).
#pragma once
#include "ntt_butterfly.cuh"

namespace lb {

// butterfly kinds of the two-kernel transforms
enum { kTpStrict = 0, kTpNear = 1, kTpF64Tight = 2, kTpF64 = 3 };
LB_D constexpr bool tp_f64(const int m) { return m == kTpF64 || m == kTpF64Tight; }

// primes below 2^42 need no reduction inside a kernel of an inverse transform (sums of at most nine stages)
constexpr u64 kF64InvPrimeLimit = u64(1) << 42;

LB_HD int tp_fwd_mode(const u64 q)
{
    if (q < kF64PrimeLimit) return kTpF64;
    if (q < kF64TightPrimeLimit) return kTpF64Tight;
    return q < kNearTop && kNearTop - q < kNearSpan ? kTpNear : kTpStrict;
}
LB_D int tp_inv_mode(const u64 q)
{
    if (q < kF64InvPrimeLimit) return kTpF64;
    if (q < kF64TightPrimeLimit) return kTpF64Tight;
    return q < kNearTop && kNearTop - q < kNearSpan ? kTpNear : kTpStrict;
}

// the scalars of a mode: q and 2^60 - q, or double(q) and double(1 / q)
struct TpPrime {
    u64 q;
    double qd, qi;
    uint32_t d;
};
template <int M>
LB_D TpPrime tp_prime(const u64 q)
{
    TpPrime p;
    p.q = q;
    if (tp_f64(M)) {
        p.qd = (double)q;
        p.qi = 1.0 / p.qd;
    }
    p.d = (uint32_t)(kNearTop - q);
    return p;
}

template <int M>
LB_D u64 tp_load(const u64 canonical) // a canonical residue in the form the stages take
{
    return tp_f64(M) ? bits_of(f64_from_u52(canonical)) : canonical;
}

// a small signed value (a ternary or error coefficient) in that form
template <int M>
LB_D u64 tp_small(const int e, const TpPrime &p)
{
    if (tp_f64(M)) return bits_of(f64_from_s52((u64)(long long)e));
    if (M == kTpNear) return p.q + (u64)(long long)e; // the stages of this class start from any word of a few q
    return e < 0 ? p.q - (u64)(-e) : (u64)e;
}

template <int M>
LB_D u64 tp_centre(const u64 v, const TpPrime &p) { return bits_of(f64_centre(f64_of(v), p.qd, p.qi)); }

// values left by up to four stages -> values the next ones may start from (at most q, or nothing to do)
template <int M, int R>
LB_D void tp_settle(u64 (&v)[R], const TpPrime &p)
{
    if (M == kTpF64Tight) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = tp_centre<M>(v[i], p);
    }
    if (M == kTpNear) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = near_reduce(v[i], p.d);
    }
}

// value left by the stages -> canonical residue
template <int M>
LB_D u64 tp_canon(const u64 v, const TpPrime &p)
{
    if (tp_f64(M)) return f64_canon(f64_of(v), p.qd, p.qi);
    if (M == kTpNear) return csub(near_reduce(v, p.d), p.q);
    return csub(csub(csub(v, p.q << 2), p.q << 1), p.q);
}

// How the values of a row end in a fused epilogue, without a canonical form in between.  A forward transform leaves at
// most 13.5 q (FP64, q < 2^47), 4.5 q (FP64, tight: centred here first) or 5 q + 2^32 (near 2^60).
struct TpScale { // a fixed factor in a mode's form
    u64 w, ws;
};
template <int M>
LB_D TpScale tp_scale(const u64 w, const u64 ws, const TpPrime &p)
{
    if (!tp_f64(M)) return TpScale{w, ws};
    const double wd = w > p.q / 2 ? (double)w - p.qd : (double)w;
    return TpScale{bits_of(wd), bits_of(__dmul_rn(wd, p.qi))};
}
// (x - v) w + y, canonical; x, y canonical residues
template <int M>
LB_D u64 tp_end_scaled(const u64 v, const u64 x, const u64 y, const TpScale &w, const TpPrime &p)
{
    if (tp_f64(M)) {
        const double d = __dadd_rn(f64_from_u52(x), -f64_of(M == kTpF64Tight ? tp_centre<M>(v, p) : v));
        return f64_canon(__dadd_rn(f64_mulmod(d, f64_of(w.w), f64_of(w.ws), p.qd), f64_from_u52(y)), p.qd, p.qi);
    }
    if (M == kTpNear) return csub(near_reduce(shoup_lazy4(x + 6 * p.q - v, w.w, w.ws, p.q) + y, p.d), p.q);
    return add_mod(shoup_mul(sub_mod(x, tp_canon<M>(v, p), p.q), w.w, w.ws, p.q), y, p.q);
}
// v x, canonical; x a canonical residue
template <int M>
LB_D u64 tp_end_product(const u64 v, const u64 x, const TpPrime &p, const u64 r0, const u64 r1)
{
    if (tp_f64(M)) {
        const double w = f64_from_u52(x);
        return f64_canon(f64_mulmod(f64_of(M == kTpF64Tight ? tp_centre<M>(v, p) : v), w, __dmul_rn(w, p.qi), p.qd), p.qd, p.qi);
    }
    if (M == kTpNear) return csub(near_fold(mul_wide(v, x), p.d), p.q);
    return barrett128(mul_wide(tp_canon<M>(v, p), x), p.q, r0, r1);
}

// S forward stages on canonical or settled values; tw(u, b): twiddle of block b at stage u
template <int S, int M, class TW>
LB_D void tp_fwd(u64 (&v)[1 << S], const TpPrime &p, const TW &tw)
{
#pragma unroll
    for (int u = 0; u < S; ++u) {
        const int half = 1 << (S - 1 - u);
#pragma unroll
        for (int b = 0; b < (1 << u); ++b) {
            const ulonglong2 w = tw(u, b);
#pragma unroll
            for (int i = 0; i < half; ++i) {
                u64 &x = v[b * 2 * half + i], &y = v[b * 2 * half + i + half];
                if (tp_f64(M)) {
                    const double xd = f64_of(x), r = f64_mulmod(f64_of(y), f64_of(w.x), f64_of(w.y), p.qd);
                    y = bits_of(__dadd_rn(xd, -r));
                    x = bits_of(__dadd_rn(xd, r));
                } else if (M == kTpNear) {
                    // 1, 5, 9, 13 q; the multiplicand may be any word, so only x is brought back before the fourth stage
                    if (u == 3) x = near_reduce(x, p.d);
                    const u64 t = shoup_lazy4(y, w.x, w.y, p.q);
                    y = x + (p.q << 2) - t;
                    x = x + t;
                } else {
                    const u64 q4 = p.q << 2, t = shoup_lazy4(y, w.x, w.y, p.q);
                    x = csub(x, q4);
                    y = x + q4 - t;
                    x = x + t;
                }
            }
        }
    }
}

// closing constants of an inverse transform in a mode's form
struct TpClose {
    u64 cn, cns, cw, cws;
};
template <int M>
LB_D TpClose tp_close(const u64 q, const u64 cn, const u64 cns, const u64 cw, const u64 cws)
{
    if (!tp_f64(M)) return TpClose{cn, cns, cw, cws};
    const double qd = (double)q, n = cn > q / 2 ? (double)cn - qd : (double)cn, w = cw > q / 2 ? (double)cw - qd : (double)cw;
    return TpClose{bits_of(n), bits_of(n / qd), bits_of(w), bits_of(w / qd)};
}

// The reductions of S <= 4 inverse stages on canonical or settled values, worked out from the bounds of the values
// (hundredths of q) while compiling: bit 16 u + i of `reduce`: the pair whose lower element is i is reduced before
// stage u; nibble i of offset[u]: the multiple of q that covers the pair's upper element.
struct TpInvPlan {
    u64 reduce, offset[4];
};
constexpr TpInvPlan tp_inv_plan(const int S, const bool f64)
{
    TpInvPlan pl = {};
    int bound[16] = {};
    for (int i = 0; i < 16; ++i) bound[i] = 100;
    for (int u = 0; u < S; ++u)
        for (int ix = 0; ix < (1 << S); ++ix) {
            const int iy = ix + (1 << u);
            if (ix & (1 << u)) continue;
            if (bound[ix] + bound[iy] > (f64 ? 400 : 1400)) {
                pl.reduce |= u64(1) << (16 * u + ix);
                bound[ix] = bound[iy] = f64 ? 51 : 100;
            }
            if (!f64) pl.offset[u] |= u64(bound[iy] / 100 + 1) << (4 * ix);
            bound[ix] += bound[iy];
            bound[iy] = f64 ? 75 : 400;
        }
    return pl;
}

// stage U of S: pairs at distance 2^U.  REDUCE, OFFSET: the stage's part of the plan
template <int S, int M, int U, bool CLOSING, u64 REDUCE, u64 OFFSET, class TW>
LB_D void tp_inv_stage(u64 (&v)[1 << S], const TpPrime &p, const TW &tw, const TpClose &c)
{
    constexpr int DIST = 1 << U;
    ulonglong2 w = make_ulonglong2(c.cw, c.cws);
#pragma unroll
    for (int j = 0; j < (1 << (S - 1)); ++j) {
        const int b = j >> U, ix = b * 2 * DIST + (j & (DIST - 1)), iy = ix + DIST;
        if (!CLOSING && (j & (DIST - 1)) == 0) w = tw(U, b);
        u64 x = v[ix], y = v[iy];
        if (tp_f64(M)) {
            if (M == kTpF64Tight && (REDUCE >> ix & 1)) {
                x = tp_centre<M>(x, p);
                y = tp_centre<M>(y, p);
            }
            const double xd = f64_of(x), yd = f64_of(y);
            const double s = __dadd_rn(xd, yd), d = f64_mulmod(__dadd_rn(xd, -yd), f64_of(w.x), f64_of(w.y), p.qd);
            v[ix] = CLOSING ? f64_canon(f64_mulmod(s, f64_of(c.cn), f64_of(c.cns), p.qd), p.qd, p.qi) : bits_of(s);
            v[iy] = CLOSING ? f64_canon(d, p.qd, p.qi) : bits_of(d);
        } else if (M == kTpNear) {
            // the difference is offset by the multiple of q that covers y
            if (REDUCE >> ix & 1) {
                x = near_reduce(x, p.d);
                y = near_reduce(y, p.d);
            }
            const u64 s = x + y, d = x + (OFFSET >> (4 * ix) & 15) * p.q - y;
            v[ix] = CLOSING ? shoup_mul(s, c.cn, c.cns, p.q) : s;
            v[iy] = CLOSING ? shoup_mul(d, c.cw, c.cws, p.q) : shoup_lazy4(d, w.x, w.y, p.q);
        } else {
            const u64 q4 = p.q << 2, s = x + y, d = x + q4 - y; // inputs below 4q
            v[ix] = CLOSING ? shoup_mul(s, c.cn, c.cns, p.q) : csub(s, q4);
            v[iy] = CLOSING ? shoup_mul(d, c.cw, c.cws, p.q) : shoup_lazy4(d, w.x, w.y, p.q);
        }
    }
}

// S inverse stages (distances 1, 2, .., 2^(S-1)); tw(u, b): twiddle of block b at stage u.
// CLOSE: the last stage is the transform's last one, carries the N^-1 scaling and leaves canonical residues.
template <int S, int M, bool CLOSE, class TW>
LB_D void tp_inv(u64 (&v)[1 << S], const TpPrime &p, const TW &tw, const TpClose &c)
{
    constexpr TpInvPlan plan = tp_inv_plan(S, tp_f64(M));
    tp_inv_stage<S, M, 0, CLOSE && S == 1, (plan.reduce & 0xFFFF), plan.offset[0]>(v, p, tw, c);
    if constexpr (S > 1) tp_inv_stage<S, M, 1, CLOSE && S == 2, (plan.reduce >> 16 & 0xFFFF), plan.offset[1]>(v, p, tw, c);
    if constexpr (S > 2) tp_inv_stage<S, M, 2, CLOSE && S == 3, (plan.reduce >> 32 & 0xFFFF), plan.offset[2]>(v, p, tw, c);
    if constexpr (S > 3) tp_inv_stage<S, M, 3, CLOSE && S == 4, (plan.reduce >> 48), plan.offset[3]>(v, p, tw, c);
}

} // namespace lb
