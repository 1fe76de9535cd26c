// Two-kernel negacyclic transforms for rings of 4096 to 65536 points (included by ntt.cu).
//
// A limb of N = 2^A * 256 coefficients is a matrix of 2^A rows of 256.  The column kernel runs the A stages
// with spans N/2 .. 256 on tiles of adjacent columns, the row kernel the eight stages with spans 128 .. 1 on single rows;
// the inverse runs them the other way round.  A thread holds 16 values (8 on the shorter columns) and takes four stages at
// a time in registers, so a kernel of eight stages exchanges its values once through shared memory:
//   column kernel  one block barrier; loads and stores are 128-byte segments of a matrix row
//   row kernel     a row belongs to half a warp, so exchanges need a warp barrier only
// What bounds them: the integer multiplier / FP64 pipe and the issue slots.  The schedule before this one (one kernel, a
// cluster of N / 8192 blocks per limb, five radix-8 passes through shared memory) kept issue slots half busy: every
// pass was a barrier for 256 threads that each walked 32 values, the first one for the whole cluster, and a single
// limb, a chain of 5 x 4 such steps on N / 8192 SMs, took 20 to 27 us whatever the batch.  Here a limb of 65536 is
// spread over 4096 threads and a pass over the matrix is a chain of two register steps.  The price is a second trip of the
// data through L2 / HBM (16 more bytes per coefficient).
//
// Code size: the two register groups of a kernel are one loop body, because the bodies of the prime classes (integer and
// FP64) run side by side on an SM and unrolled in full they missed the instruction cache (2 stalls per issue).  Twiddles are
// stored in the order the groups read them (twiddle_slot in params.h).
#pragma once
#include "ntt_stages.cuh"

namespace lb {

constexpr int kRowLog = 8, kRowThreads = 128, kRowsPerCta = kRowThreads / 16; // half warps per block of the row kernels
constexpr int kRowPad = 272; // a row in shared memory: one spare word per 16

// shape of the column kernel for 2^A rows: first S1 stages, then S2; 2^S1 values and 2^S2 threads per column
template <int A>
struct ColShape {
    static constexpr int S1 = column_first_stages(A), S2 = A - S1;
    static constexpr int V = 1 << S1, TPC = 1 << S2;
    static constexpr int THREADS = A >= 7 ? 256 : 128;
    static constexpr int COLS = THREADS / TPC; // 128, 32, 16, 32, 16 columns for A = 4 .. 8
    static constexpr int TILES = 256 / COLS;   // blocks per limb
    static constexpr int G = 1 << (S1 - S2);   // register groups of the second part per thread (S2 > 0)
};

// A kernel launched with programmatic stream serialisation may start before its predecessor's writes are visible: nothing is
// read or written before this.  No kernel signals its successor before it ends.  With the signal at the top, blocks of two or
// three later kernels sat on the SMs waiting and the next ones were placed around them, up to six on one SM while others had
// none: 20 inverse transforms of N = 2^15 one call after the other took 24.2 us a call against 16.3, 100 of N = 2^12 19.6
// against 10.3, a small 4-client round 1345 us against 1295.  Signals after the wait or before the last stores lie in between.
LB_D void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Sums of products of 60-bit words without carries: operands in halves of 30 bits, three products per term
// (x0 y0, x1 y1, and (x0 - x1)(y0 - y1) for the mixed ones), and eight terms fit the 64-bit sums.
struct Mac30 {
    u64 ll, hh, df;
};
LB_D void mac30(Mac30 &s, const u64 x, const uint32_t yl, const uint32_t yh, const int yd)
{
    const uint32_t xl = (uint32_t)x & 0x3FFFFFFFu, xh = (uint32_t)(x >> 30);
    s.ll += (u64)xl * yl;
    s.hh += (u64)xh * yh;
    s.df += (u64)((long long)((int)xl - (int)xh) * yd);
}
LB_D u128 mac30_sum(const Mac30 &s) // the mixed products sum to at most 16 (2^30 - 1)^2 < 2^64
{
    return (u128)s.ll + ((u128)(s.ll + s.hh - s.df) << 30) + ((u128)s.hh << 60);
}

// The transform's input at column-kernel positions j + (k << LOGST), k < V (see FwdIn), in the form the stages take.  FP64
// values start at up to 1.5 q (a folded conversion and the plaintext's product), words near 2^60 at up to 2 q: each
// stage adds 0.75 q (4 q), which keeps four stages within 4.5 q (within 16 q, see tp_fwd), and all sixteen of a prime
// below 2^47 within 13.5 q.
template <int V, int LOGST, int THREADS, bool PLAIN, int M>
LB_D void col_load(u64 (&v)[V], const FwdIn &in, const TpPrime &p, const int j, u64 *own)
{
    const u64 q = in.q;
    if (PLAIN || (in.n == 0 && in.sub == nullptr && in.small == nullptr)) {
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = in.src[j + (k << LOGST)];
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = tp_load<M>(v[k]);
        return;
    }
    const ModConst &m = *in.mc;
    const bool folds = tp_f64(M) && m.kind == kWideF64;
    if (in.small) {
        // the small polynomial of an encryption as signed bytes, the same for every prime
        int ev[V];
#pragma unroll
        for (int k = 0; k < V; ++k) ev[k] = in.small[j + (k << LOGST)];
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = tp_small<M>(ev[k], p);
    } else if (in.n == 1 && in.mat == nullptr) {
        // One source row reduced into this prime (every conversion of a chain with one special prime), eight words at a
        // time.  The branches on the optional parts stay outside the loops so that all loads of a part are in flight together.
        const TpScale w = tp_scale<M>(in.sub_w, in.sub_ws, p);
#pragma unroll
        for (int h = 0; h < V; h += 8) {
            u64 x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = in.src[j + ((h + k) << LOGST)];
            if (in.es) {
                int ev[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) ev[k] = in.es[j + ((h + k) << LOGST)];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    x[k] = add_mod(x[k], ev[k] < 0 ? in.es_p - (u64)(-ev[k]) : (u64)ev[k], in.es_p);
                    if (folds) x[k] = bits_of(f64_from_s52(f64_fold64(x[k], m) - (u64)(long long)ev[k]));
                    else if (M == kTpNear) x[k] += q - (u64)(long long)ev[k];
                    else x[k] = tp_load<M>(sub_mod(barrett64(x[k], q, in.r1), ev[k] < 0 ? q - (u64)(-ev[k]) : (u64)ev[k], q));
                }
            } else if (folds) {
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = bits_of(f64_from_s52(f64_fold64(x[k], m)));
            } else if (M != kTpNear) { // there a word of another prime, below 2^60, is hardly more than q
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = tp_load<M>(barrett64(x[k], q, in.r1));
            }
            if (in.sub) {
                u64 t[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) t[k] = in.sub[j + ((h + k) << LOGST)];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (tp_f64(M)) x[k] = bits_of(__dadd_rn(f64_of(x[k]), -f64_mulmod(f64_from_u52(t[k]), f64_of(w.w), f64_of(w.ws), p.qd)));
                    else if (M == kTpNear) x[k] = near_reduce(x[k] + (q << 2) - shoup_lazy4(t[k], w.w, w.ws, q), p.d);
                    else x[k] = sub_mod(x[k], shoup_mul(t[k], w.w, w.ws, q), q);
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) v[h + k] = x[k];
        }
    } else if (in.mat != nullptr && in.sub == nullptr) {
        // Base conversion of several source rows: four outputs share one walk over the rows, and the words of the next row
        // are requested before those of this one are multiplied.  Finished outputs wait in the thread's own words of shared
        // memory (the ones its first exchange writes): the sums and two rows of operands need the registers.
        constexpr int STEP = V < 4 ? V : 4;
#pragma unroll 1
        for (int h = 0; h < V; h += STEP) {
            const u64 *src = in.src + j + (h << LOGST);
            u64 x[STEP];
#pragma unroll
            for (int k = 0; k < STEP; ++k) x[k] = src[k << LOGST];
            u128d acc[STEP];
#pragma unroll
            for (int k = 0; k < STEP; ++k) acc[k] = u128d{0, 0};
            for (int i0 = 0; i0 < in.n; i0 += 8) {
                Mac30 s[STEP];
#pragma unroll
                for (int k = 0; k < STEP; ++k) s[k] = Mac30{0, 0, 0};
                const int i1 = min(i0 + 8, in.n);
#pragma unroll 2
                for (int i = i0; i < i1; ++i) {
                    u64 nx[STEP];
                    if (i + 1 < in.n) src += (size_t)1 << in.logN;
#pragma unroll
                    for (int k = 0; k < STEP; ++k) nx[k] = src[k << LOGST];
                    const u64 y = __ldg(in.mat + i);
                    const uint32_t yl = (uint32_t)y & 0x3FFFFFFFu, yh = (uint32_t)(y >> 30);
#pragma unroll
                    for (int k = 0; k < STEP; ++k) mac30(s[k], x[k], yl, yh, (int)yl - (int)yh);
#pragma unroll
                    for (int k = 0; k < STEP; ++k) x[k] = nx[k];
                }
#pragma unroll
                for (int k = 0; k < STEP; ++k) {
                    const u128 t = ((u128)acc[k].hi << 64 | acc[k].lo) + mac30_sum(s[k]);
                    acc[k] = u128d{(u64)t, (u64)(t >> 64)};
                }
            }
#pragma unroll
            for (int k = 0; k < STEP; ++k) {
                u64 r;
                if (folds) r = bits_of(f64_fold(acc[k], m));
                else if (M == kTpNear) r = near_fold(acc[k], p.d);
                else r = tp_load<M>(barrett128(acc[k], q, in.r0, in.r1));
                own[(h + k) * THREADS] = r;
            }
        }
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = own[k * THREADS];
    } else {
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = tp_load<M>(load_in(in, j + (k << LOGST)));
    }
}

template <int A, int M, bool PLAIN>
LB_D void col_fwd_body(u64 *sm, const FwdRow &fr, u64 *mid, const int tile)
{
    using C = ColShape<A>;
    const int cl = threadIdx.x & (C::COLS - 1), t = threadIdx.x / C::COLS;
    const int col = tile * C::COLS + cl;
    const TpPrime p = tp_prime<M>(fr.q);
    const ulonglong2 *tw = fr.tw;
    u64 v[C::V];
    col_load<C::V, kRowLog + C::S2, C::THREADS, PLAIN, M>(v, fr.in, p, (t << kRowLog) + col, sm + threadIdx.x);
    if constexpr (C::S1 == C::S2) {
        const ulonglong2 *tg = tw + 1;
#pragma unroll 1
        for (int half = 0;; ++half) {
            tp_fwd<C::S1, M>(v, p, [&](const int u, const int b) { return __ldg(tg + (1 << u) - 1 + b); });
            tp_settle<M>(v, p);
            if (half) break;
#pragma unroll
            for (int k = 0; k < C::V; ++k) sm[((k << C::S2) + t) * C::COLS + cl] = v[k];
            __syncthreads();
#pragma unroll
            for (int k = 0; k < C::V; ++k) v[k] = sm[((t << C::S2) + k) * C::COLS + cl];
            tg = tw + (1 << C::S1) + t * ((1 << C::S2) - 1);
        }
#pragma unroll
        for (int k = 0; k < C::V; ++k) mid[(((t << C::S2) + k) << kRowLog) + col] = v[k];
    } else {
        tp_fwd<C::S1, M>(v, p, [&](const int u, const int b) { return __ldg(tw + (1 << u) + b); });
        tp_settle<M>(v, p);
        if constexpr (C::S2 == 0) {
#pragma unroll
            for (int k = 0; k < C::V; ++k) mid[(k << kRowLog) + col] = v[k];
        } else {
#pragma unroll
            for (int k = 0; k < C::V; ++k) sm[((k << C::S2) + t) * C::COLS + cl] = v[k];
            __syncthreads();
#pragma unroll
            for (int i = 0; i < C::G; ++i) {
                const int g = t + i * C::TPC;
                const ulonglong2 *tg = tw + (1 << C::S1) + g * ((1 << C::S2) - 1);
                u64 w[1 << C::S2];
#pragma unroll
                for (int k = 0; k < (1 << C::S2); ++k) w[k] = sm[((g << C::S2) + k) * C::COLS + cl];
                tp_fwd<C::S2, M>(w, p, [&](const int u, const int b) { return __ldg(tg + (1 << u) - 1 + b); });
                tp_settle<M>(w, p);
#pragma unroll
                for (int k = 0; k < (1 << C::S2); ++k) mid[(((g << C::S2) + k) << kRowLog) + col] = w[k];
            }
        }
    }
}

template <int A, bool PLAIN>
__global__ void __launch_bounds__(ColShape<A>::THREADS, ColShape<A>::THREADS == 256 ? 3 : 6) ntt_fwd_col_kernel(const __grid_constant__ NttK a)
{
    using C = ColShape<A>;
    __shared__ __align__(16) u64 sm[C::S2 || !PLAIN ? C::V * C::THREADS : 1];
    grid_wait();
    const int row = blockIdx.x / C::TILES, tile = blockIdx.x % C::TILES;
    FwdRow fr;
    if (!fwd_row_setup(a, row, fr)) return;
    u64 *mid = a.mid ? a.mid + ((size_t)row << a.logN) : fr.dst;
    // the order of the classes is the order of their code, here and in the row kernel: with the FP64 classes first, 768 limbs of
    // 50 bits took 379.8 us instead of 362.9 and the 10-client round at N = 2^15 14.20 ms instead of 14.02
    switch (tp_fwd_mode(fr.q)) {
    case kTpNear: col_fwd_body<A, kTpNear, PLAIN>(sm, fr, mid, tile); break;
    case kTpF64Tight: col_fwd_body<A, kTpF64Tight, PLAIN>(sm, fr, mid, tile); break;
    case kTpF64: col_fwd_body<A, kTpF64, PLAIN>(sm, fr, mid, tile); break;
    default: col_fwd_body<A, kTpStrict, PLAIN>(sm, fr, mid, tile); break;
    }
}

// Which limb row and which matrix row a half warp of a row kernel works on.  The eight half warps of a block take
// 2^log_polys polynomials of the same prime times 8 / 2^log_polys matrix rows: polynomials that share a matrix row share its
// 510 twiddles (4 KB of table against 2 KB of data per row), which then come from L1 instead of L2.
struct RowPlace {
    int rr, grp, r; // limb within its group (the same for the whole block), group (n_groups or more: nothing to do), matrix row
};
LB_D RowPlace row_place(const NttK &a)
{
    const int h = threadIdx.x >> 4, log_tiles = a.logN - kRowLog - 3 + a.log_polys;
    const int tile = blockIdx.x & ((1 << log_tiles) - 1);
    int rest = blockIdx.x >> log_tiles;
    RowPlace w;
    w.rr = rest % a.per_group;
    rest /= a.per_group;
    const int sub = rest % a.poly_step;
    w.grp = (((rest / a.poly_step) << a.log_polys) + (h & ((1 << a.log_polys) - 1))) * a.poly_step + sub;
    w.r = (tile << (3 - a.log_polys)) + (h >> a.log_polys);
    return w;
}

// the 16 x 16 values of a matrix row change hands: thread t has (t, k) and gets (k, t)
LB_D void row_transpose(u64 (&v)[16], u64 *srow, const int t)
{
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 16; ++k) srow[t + 17 * k] = v[k];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = srow[17 * t + k];
}

// a thread's twiddles of a row's first (spans 128 .. 16) and second (spans 8 .. 1) register group, 16 entries apart
LB_D const ulonglong2 *row_twiddles(const ulonglong2 *tw, const int logN, const int r, const int t, const bool second)
{
    return second ? tw + (1 << (logN - 4)) + r * 240 + t : tw + (1 << (logN - kRowLog)) + (r >> 4) * 240 + (r & 15);
}

template <int M, bool PLAIN>
LB_D void row_fwd_body(u64 *srow, const NttK &a, const RowPlace &w, const ModConst *mc, const ulonglong2 *tw)
{
    const int t = threadIdx.x & 15, logN = a.logN;
    const u64 q = mc->q;
    const TpPrime p = tp_prime<M>(q);
    const long go = w.grp / a.split, gi = w.grp - go * a.split;
    const size_t base = ((size_t)w.r << kRowLog) + t;
    u64 *const dst = a.dst + ((size_t)(go * a.dst_outer + gi * a.dst_group_stride + w.rr) << logN) + base;
    const u64 *const mid = a.mid ? a.mid + ((size_t)((long)w.grp * a.per_group + w.rr) << logN) + base : dst;
    u64 v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = mid[16 * k];
    const ulonglong2 *tg = row_twiddles(tw, logN, w.r, t, false);
#pragma unroll 1
    for (int half = 0;; ++half) {
        tp_fwd<4, M>(v, p, [&](const int u, const int b) { return __ldg(tg + 16 * ((1 << u) - 1 + b)); });
        if (half) break;
        tp_settle<M>(v, p);
        row_transpose(v, srow, t);
        tg = row_twiddles(tw, logN, w.r, t, true);
    }
    if (PLAIN || (!a.aux && !a.mul2)) {
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = tp_canon<M>(v[k], p);
    }
    row_transpose(v, srow, t); // back to neighbouring threads on neighbouring coefficients
    if (!PLAIN && a.aux) {
        const u64 *aux = a.aux + ((size_t)(go * a.aux_outer + gi * a.aux_group_stride + w.rr) << logN) + base;
        const u64 *add = a.add1 && gi == 1 ? a.add1 + ((size_t)(go * a.add1_outer + w.rr) << logN) + base
                         : a.add && gi < a.add_inner ? a.add + ((size_t)(go * a.add_outer + gi * a.add_group_stride + w.rr) << logN) + base
                                                     : nullptr;
        const TpScale scal = tp_scale<M>(a.scal[w.rr], a.scal_s[w.rr], p);
#pragma unroll
        for (int h = 0; h < 16; h += 4) {
            u64 x[4], y[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = aux[16 * (h + k)];
#pragma unroll
            for (int k = 0; k < 4; ++k) y[k] = 0;
            if (add) {
#pragma unroll
                for (int k = 0; k < 4; ++k) y[k] = add[16 * (h + k)];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) v[h + k] = tp_end_scaled<M>(v[h + k], x[k], y[k], scal, p);
        }
    } else if (!PLAIN && a.mul2) {
        const u64 *mul0 = a.mul2 + ((size_t)w.rr << logN) + base, *mul1 = mul0 + ((size_t)a.per_group << logN);
        u64 *const dst1 = dst + ((size_t)a.per_group << logN);
        const u64 r0 = mc->r0, r1 = mc->r1;
#pragma unroll
        for (int h = 0; h < 16; h += 4) {
            u64 x[4], y[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                x[k] = mul0[16 * (h + k)];
                y[k] = mul1[16 * (h + k)];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                dst1[16 * (h + k)] = tp_end_product<M>(v[h + k], y[k], p, r0, r1);
                v[h + k] = tp_end_product<M>(v[h + k], x[k], p, r0, r1);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) dst[16 * k] = v[k];
}

LB_D int row_table(const NttK &a, const int rr) { return rr < a.size_l ? rr + a.tbl_off : a.size_Q + (rr - a.size_l); }

template <bool PLAIN>
__global__ void __launch_bounds__(kRowThreads, 6) ntt_fwd_row_kernel(const __grid_constant__ NttK a)
{
    __shared__ __align__(16) u64 sm[kRowsPerCta * kRowPad];
    grid_wait();
    const RowPlace w = row_place(a);
    if (w.grp >= a.n_polys * a.poly_step || (w.rr >= a.skip_lo && w.rr < a.skip_hi)) return;
    if (a.digit_alpha > 0) { // the digit's own limbs stay in NTT form
        const int s = (w.grp % a.split) * a.digit_alpha;
        if (w.rr >= s && w.rr < min(s + a.digit_alpha, a.size_l)) return;
    }
    const int tbl = row_table(a, w.rr);
    const ModConst *mc = a.mc + tbl;
    const ulonglong2 *tw = a.tw + ((size_t)tbl << a.logN);
    u64 *srow = sm + (threadIdx.x >> 4) * kRowPad;
    switch (tp_fwd_mode(mc->q)) {
    case kTpNear: row_fwd_body<kTpNear, PLAIN>(srow, a, w, mc, tw); break;
    case kTpF64Tight: row_fwd_body<kTpF64Tight, PLAIN>(srow, a, w, mc, tw); break;
    case kTpF64: row_fwd_body<kTpF64, PLAIN>(srow, a, w, mc, tw); break;
    default: row_fwd_body<kTpStrict, PLAIN>(srow, a, w, mc, tw); break;
    }
}

// ---- inverse ---------------------------------------------------------------------------

// Where an inverse transform's row comes from and goes to
struct InvRow {
    const u64 *src;
    u64 *dst;
    const ulonglong2 *itw;
    u64 q, cn, cns, cw, cws;
};

LB_D bool inv_row_setup(const NttK &a, const int row, InvRow &r)
{
    const int grp = row / a.per_group, rr = row - grp * a.per_group;
    if (rr >= a.skip_lo && rr < a.skip_hi) return false;
    const int tbl = rr < a.size_l ? rr + a.tbl_off : a.size_Q + (rr - a.size_l);
    const ModConst mc = a.mc[tbl];
    const int go = grp / a.split, gi = grp - go * a.split;
    r.q = mc.q;
    r.itw = a.tw + ((size_t)tbl << a.logN);
    r.src = a.src + (((size_t)go * a.src_outer + (size_t)gi * a.src_group_stride + rr + a.src_row_off) << a.logN);
    r.dst = a.dst + (((size_t)go * a.dst_outer + (size_t)gi * a.dst_group_stride + rr) << a.logN);
    r.cn = mc.ninv; r.cns = mc.ninvs; r.cw = mc.iw1n; r.cws = mc.iw1ns;
    if (a.fold) {
        const u64 *f = a.fold + 4 * rr;
        r.cn = f[0]; r.cns = f[1]; r.cw = f[2]; r.cws = f[3];
    }
    return true;
}

template <int M>
LB_D void row_inv_body(u64 *srow, const NttK &a, const RowPlace &w, const u64 q, const ulonglong2 *tw)
{
    const int t = threadIdx.x & 15, logN = a.logN;
    const TpPrime p = tp_prime<M>(q);
    const long go = w.grp / a.split, gi = w.grp - go * a.split;
    const size_t base = ((size_t)w.r << kRowLog) + t;
    const u64 *const src = a.src + ((size_t)(go * a.src_outer + gi * a.src_group_stride + w.rr + a.src_row_off) << logN) + base;
    u64 *const dst = a.dst + ((size_t)(go * a.dst_outer + gi * a.dst_group_stride + w.rr) << logN) + base;
    const TpClose none = {0, 0, 0, 0};
    u64 v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = src[16 * k];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = tp_load<M>(v[k]);
#pragma unroll 1
    for (int half = 1; half >= 0; --half) {
        row_transpose(v, srow, t);
        const ulonglong2 *tg = row_twiddles(tw, logN, w.r, t, half);
        tp_inv<4, M, false>(v, p, [&](const int u, const int b) { return __ldg(tg + 16 * ((1 << (3 - u)) - 1 + b)); }, none);
        tp_settle<M>(v, p);
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) dst[16 * k] = v[k];
}

__global__ void __launch_bounds__(kRowThreads, 6) ntt_inv_row_kernel(const __grid_constant__ NttK a)
{
    __shared__ __align__(16) u64 sm[kRowsPerCta * kRowPad];
    grid_wait();
    const RowPlace w = row_place(a);
    if (w.grp >= a.n_polys * a.poly_step || (w.rr >= a.skip_lo && w.rr < a.skip_hi)) return;
    const int tbl = row_table(a, w.rr);
    const u64 q = a.mc[tbl].q;
    const ulonglong2 *tw = a.tw + ((size_t)tbl << a.logN);
    u64 *srow = sm + (threadIdx.x >> 4) * kRowPad;
    switch (tp_inv_mode(q)) {
    case kTpF64: row_inv_body<kTpF64>(srow, a, w, q, tw); break;
    case kTpF64Tight: row_inv_body<kTpF64Tight>(srow, a, w, q, tw); break;
    case kTpNear: row_inv_body<kTpNear>(srow, a, w, q, tw); break;
    default: row_inv_body<kTpStrict>(srow, a, w, q, tw); break;
    }
}

template <int A, int M>
LB_D void col_inv_body(u64 *sm, const InvRow &ir, const int tile)
{
    using C = ColShape<A>;
    const int cl = threadIdx.x & (C::COLS - 1), t = threadIdx.x / C::COLS;
    const int col = tile * C::COLS + cl;
    const TpPrime p = tp_prime<M>(ir.q);
    const TpClose close = tp_close<M>(ir.q, ir.cn, ir.cns, ir.cw, ir.cws);
    const ulonglong2 *tw = ir.itw;
    u64 *dst = ir.dst;
    u64 v[C::V];
    if constexpr (C::S2 == 0) {
#pragma unroll
        for (int k = 0; k < C::V; ++k) v[k] = dst[(k << kRowLog) + col];
        if (M == kTpF64) { // small primes are brought back once per transform
#pragma unroll
            for (int k = 0; k < C::V; ++k) v[k] = tp_centre<M>(v[k], p);
        }
    } else {
#pragma unroll
        for (int i = 0; i < C::G; ++i) {
            const int g = t + i * C::TPC;
            const ulonglong2 *tg = tw + (1 << C::S1) + g * ((1 << C::S2) - 1);
            u64 w[1 << C::S2];
#pragma unroll
            for (int k = 0; k < (1 << C::S2); ++k) w[k] = dst[(((g << C::S2) + k) << kRowLog) + col];
            if (M == kTpF64) {
#pragma unroll
                for (int k = 0; k < (1 << C::S2); ++k) w[k] = tp_centre<M>(w[k], p);
            }
            tp_inv<C::S2, M, false>(w, p, [&](const int u, const int b) { return __ldg(tg + (1 << (C::S2 - 1 - u)) - 1 + b); }, close);
            tp_settle<M>(w, p);
#pragma unroll
            for (int k = 0; k < (1 << C::S2); ++k) sm[((g << C::S2) + k) * C::COLS + cl] = w[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < C::V; ++k) v[k] = sm[((k << C::S2) + t) * C::COLS + cl];
    }
    tp_inv<C::S1, M, true>(v, p, [&](const int u, const int b) { return __ldg(tw + (1 << (C::S1 - 1 - u)) + b); }, close);
#pragma unroll
    for (int k = 0; k < C::V; ++k) dst[((((k << C::S2) + t)) << kRowLog) + col] = v[k];
}

template <int A>
__global__ void __launch_bounds__(ColShape<A>::THREADS, ColShape<A>::THREADS == 256 ? 3 : 6) ntt_inv_col_kernel(const __grid_constant__ NttK a)
{
    using C = ColShape<A>;
    __shared__ __align__(16) u64 sm[C::S2 ? C::V * C::THREADS : 1];
    grid_wait();
    const int row = blockIdx.x / C::TILES, tile = blockIdx.x % C::TILES;
    InvRow ir;
    if (!inv_row_setup(a, row, ir)) return;
    switch (tp_inv_mode(ir.q)) {
    case kTpF64: col_inv_body<A, kTpF64>(sm, ir, tile); break;
    case kTpF64Tight: col_inv_body<A, kTpF64Tight>(sm, ir, tile); break;
    case kTpNear: col_inv_body<A, kTpNear>(sm, ir, tile); break;
    default: col_inv_body<A, kTpStrict>(sm, ir, tile); break;
    }
}

} // namespace lb
