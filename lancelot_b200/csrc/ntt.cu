// Batched negacyclic NTT / inverse NTT over RNS limbs for sm_100a.
//
// Mathematical definition (must equal the reference's, cahel-main/src/ntt/ntt_1d.cu:38-74,
// :129-171 and butterfly.cuh:10-43; its production path is the two-kernel radix-8 pair in
// cahel-main/src/ntt/fntt_2d.cu:8,126,872 and intt_2d.cu:8,103,693):
//   forward: stages m = 1,2,..,N/2, butterfly (x,y) -> (x + w y, x - w y), w = psi^bitrev(m+k);
//            natural order in, bit-reversed order out, canonical residues out.
//   inverse: the exact inverse map (the reference halves in every butterfly; here N^-1 is
//            folded into the last stage).
//
// Schedules: rings of 4096 to 65536 points take the two-kernel transforms of ntt_twopass.cuh.  The kernels in this
// file serve the rest: rings below 4096 points (one block holds a limb in shared memory) and 131072 points, where a
// thread-block cluster of 16 blocks owns a limb: the first log2(C) stages run in registers on coalesced strided global
// loads, their outputs are scattered to the owning block through distributed shared memory, and each block finishes
// an independent 8192-point transform in its own shared memory with register-blocked radix-8 passes.  The inverse
// mirrors this.
#include <cooperative_groups.h>

#include "context.h"
#include "ntt_stages.cuh"

namespace cg = cooperative_groups;

namespace lb {

// Launch shape of the single-kernel transforms: threads per CTA, CTAs per SM the register allocation aims at, and log2 of the points one
// CTA keeps in shared memory (8192 points: 64 KiB + padding, three CTAs per SM).  Register passes take at most
// three stages (radix 8).
constexpr int kNttThreads = 256;
constexpr int kNttMinBlocks = 3;
constexpr int kMaxLocalLog = 13;
constexpr int kMaxRadixLog = 3;

struct NttK {
    const u64 *src;
    u64 *dst;
    const ulonglong2 *tw;
    const ModConst *mc;
    int logN, per_group, split, size_l, size_Q, tbl_off;
    long src_group_stride, dst_group_stride, aux_group_stride, add_group_stride;
    long src_outer, dst_outer, aux_outer, add_outer;
    int src_row_off, skip_lo, skip_hi;
    int bconv_n, digit_alpha, add_inner;
    const u64 *bconv_mat;
    long mat_group_stride, mat_row_stride;
    const u64 *aux, *scal, *scal_s, *add, *fold;
    const u64 *add1; // addend rows of the groups with inner == 1, if they sit elsewhere (see NttJob::add1)
    long add1_outer;
    const u64 *mul2; // forward epilogue: two products per row (see NttJob::mul2)
    int n_polys, poly_step, log_polys; // row kernels: how polynomials of one prime share a block (see row_place)
    u64 *mid;        // two-kernel forward transform: rows between the kernels, or nullptr: the dst rows
    const u64 *presub, *presub_scal, *presub_scal_s;
    const signed char *esmall;
    const signed char *small;
    u64 esmall_p;
    long presub_outer;
    int presub_inner;
    int npass;
    int nwide; // passes whose butterflies cross warp chunks (forward: the first nwide, inverse: the last nwide)
    int wlog;  // log2 of the contiguous chunk one warp owns in the other passes
    unsigned char S[8];
};

// one spare word per 16 keeps the stride-8 and stride-1 passes off the same banks
LB_D int sidx(int i) { return i + (i >> 4); }

// S consecutive forward stages on 2^S register values; stage u uses twiddle (t0 << u) + block
template <int S, int MODE>
LB_D void fwd_core(u64 (&v)[1 << S], const ulonglong2 *__restrict__ tw, const unsigned t0, const u64 q, const u64 q2)
{
#pragma unroll
    for (int u = 0; u < S; ++u) {
        const int half = 1 << (S - 1 - u);
        if (MODE == kF64Tight && u == 3) { // three stages since the values were centred: centre them again
#pragma unroll
            for (int i = 0; i < (1 << S); ++i) v[i] = bits_of(f64_centre(f64_of(v[i]), f64_of(q), f64_of(q2)));
        }
#pragma unroll
        for (int b = 0; b < (1 << u); ++b) {
            const ulonglong2 w = __ldg(tw + ((t0 << u) + b));
#pragma unroll
            for (int i = 0; i < half; ++i) fwd_bf<MODE>(v[b * 2 * half + i], v[b * 2 * half + i + half], w, q, q2);
        }
    }
}

// S consecutive inverse stages; stage u pairs distance 2^u and uses twiddle (tb >> u) + block.
// CLOSE: the last of them is the transform's last stage and carries the N^-1 scaling; it leaves
// canonical residues (as integers in every mode).  In kInvF64 mode q, q2 carry double(q), double(1 / q)
// and (cn, cns), (cw, cws) the closing constants and their quotients by q, all as doubles.
template <int S, bool CLOSE, int IM>
LB_D void inv_core(u64 (&v)[1 << S], const ulonglong2 *__restrict__ itw, const unsigned tb, const u64 q, const u64 q2,
                   const u64 cn, const u64 cns, const u64 cw, const u64 cws)
{
#pragma unroll
    for (int u = 0; u < S; ++u) {
        const int dist = 1 << u;
        if (IM == kInvF64Tight && u > 0 && (u & 1) == 0) { // two stages since the values were centred
#pragma unroll
            for (int i = 0; i < (1 << S); ++i) v[i] = bits_of(f64_centre(f64_of(v[i]), f64_of(q), f64_of(q2)));
        }
#pragma unroll
        for (int b = 0; b < (1 << (S - 1 - u)); ++b) {
            if (CLOSE && u == S - 1) {
#pragma unroll
                for (int i = 0; i < dist; ++i) {
                    u64 &x = v[b * 2 * dist + i], &y = v[b * 2 * dist + i + dist];
                    if (is_inv_f64(IM)) {
                        const double xd = f64_of(x), yd = f64_of(y), qd = f64_of(q), qi = f64_of(q2);
                        x = f64_canon(f64_mulmod(__dadd_rn(xd, yd), f64_of(cn), f64_of(cns), qd), qd, qi);
                        y = f64_canon(f64_mulmod(__dadd_rn(xd, -yd), f64_of(cw), f64_of(cws), qd), qd, qi);
                    } else {
                        const u64 s = x + y, d = x + (q2 << 1) - y; // inputs below 4q
                        x = shoup_mul(s, cn, cns, q);
                        y = shoup_mul(d, cw, cws, q);
                    }
                }
            } else {
                const ulonglong2 w = __ldg(itw + ((tb >> u) + b));
#pragma unroll
                for (int i = 0; i < dist; ++i) inv_bf<IM>(v[b * 2 * dist + i], v[b * 2 * dist + i + dist], w, q, q2);
            }
        }
    }
}

template <int R>
LB_D void load_contig(u64 (&v)[R], const u64 *p)
{
    if (R == 1) {
        v[0] = p[0];
    } else {
#pragma unroll
        for (int i = 0; i < R; i += 2) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(p + i);
            v[i] = t.x;
            v[i + 1] = t.y;
        }
    }
}

template <int R>
LB_D void store_contig(const u64 (&v)[R], u64 *p)
{
#pragma unroll
    for (int i = 0; i < R; i += 2) *reinterpret_cast<ulonglong2 *>(p + i) = make_ulonglong2(v[i], v[i + 1]);
}

// ---- forward --------------------------------------------------------------------------

// Where a transform input comes from: a plain row, one row reduced into this row's prime,
// or an approximate fast base conversion of up to alpha rows (cahel-main/src/rns_bconv.cu:
// 562-623 for mod-up, :847-866 and :166-199 for mod-down), evaluated while loading.
struct FwdIn {
    const u64 *src;
    const u64 *mat;
    const u64 *sub; // optional: the loaded value becomes value - sub[k] * sub_w (plaintext folded into a mod-down)
    const signed char *es; // optional small error polynomial e of an encryption (see the encrypt path)
    const signed char *small; // the input itself as signed bytes (then src is not read)
    int n, logN;
    u64 q, r0, r1, sub_w, sub_ws, es_p;
    const ModConst *mc;
};

LB_D u64 load_in(const FwdIn &in, const int idx)
{
    u64 v;
    if (in.small) {
        const int ev = in.small[idx];
        v = ev < 0 ? in.q - (u64)(-ev) : (u64)ev;
    } else if (in.n == 0) {
        v = in.src[idx];
    } else if (in.mat == nullptr) {
        u64 x = in.src[idx];
        if (in.es) {
            // x is INTT(pk u) on the special prime p: add e mod p first (INTT is linear, so this is the
            // special limb of pk u + e), convert, then take e off again on this prime, because the
            // caller's aux rows hold pk u without e:  (pk u + e) - NTT(delta) = pk u - NTT(delta - e)
            const int ev = in.es[idx];
            x = add_mod(x, ev < 0 ? in.es_p - (u64)(-ev) : (u64)ev, in.es_p);
            v = barrett64(x, in.q, in.r1);
            v = sub_mod(v, ev < 0 ? in.q - (u64)(-ev) : (u64)ev, in.q);
        } else {
            v = barrett64(x, in.q, in.r1);
        }
    } else {
        u128d acc;
        acc.lo = 0;
        acc.hi = 0;
        for (int i = 0; i < in.n; ++i) mac_wide(acc, in.src[((size_t)i << in.logN) + idx], __ldg(in.mat + i));
        v = barrett128(acc, in.q, in.r0, in.r1);
    }
    if (in.sub) v = sub_mod(v, shoup_mul(in.sub[idx], in.sub_w, in.sub_ws, in.q), in.q);
    return v;
}

struct FwdEpi {
    const u64 *aux; // nullptr: plain store
    const u64 *add; // optional addend
    u64 scal, scal_s;
    // optional: instead of the transform itself, store its products with two fixed rows (the two polynomials of a
    // public key): dst <- NTT(x) * mul0, dst + dst1_off <- NTT(x) * mul1
    const u64 *mul0, *mul1;
    long dst1_off;
    u64 r0, r1; // floor(2^128 / q) for those products
};

// Work split of one register pass.  A pass whose largest butterfly span exceeds a warp's chunk
// is shared out over the whole CTA; in every other pass a warp keeps to the groups of its own
// contiguous 2^wlog-point chunk, so that consecutive such passes only need a warp-level barrier.
struct PassSplit {
    int first, end, step;
};

template <int S>
LB_D PassSplit pass_split(const int logn_loc, const int wlog)
{
    PassSplit ps;
    if (wlog < 0) {
        ps.first = threadIdx.x;
        ps.end = 1 << (logn_loc - S);
        ps.step = kNttThreads;
    } else {
        const int gpw = 1 << (wlog - S), warp = threadIdx.x >> 5;
        ps.first = warp * gpw + (threadIdx.x & 31);
        ps.end = (warp + 1) * gpw;
        ps.step = 32;
    }
    return ps;
}

template <int S, int MODE>
LB_D void fwd_pass(u64 *sm, const bool from_global, u64 *gdst, const FwdIn &in, const int logn_loc, const int logt,
                   const unsigned cc, const ulonglong2 *tw, const u64 q, const u64 q2, const FwdEpi &epi, const int wlog)
{
    constexpr int R = 1 << S;
    const int logst = logt - (S - 1);
    const int logm0 = logn_loc - 1 - logt;
    const PassSplit ps = pass_split<S>(logn_loc, wlog);
    for (int g = ps.first; g < ps.end; g += ps.step) {
        const int lo = g & ((1 << logst) - 1), hi = g >> logst;
        const int base = (hi << (logt + 1)) + lo;
        u64 v[R];
        if (from_global) {
#pragma unroll
            for (int i = 0; i < R; ++i) v[i] = load_in(in, base + (i << logst));
            if (is_f64_mode(MODE)) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = bits_of(f64_from_u52(v[i]));
            }
        } else {
#pragma unroll
            for (int i = 0; i < R; ++i) v[i] = sm[sidx(base + (i << logst))];
        }
        if (MODE == kF64Tight) {
#pragma unroll
            for (int i = 0; i < R; ++i) v[i] = bits_of(f64_centre(f64_of(v[i]), f64_of(q), f64_of(q2)));
        }
        fwd_core<S, MODE>(v, tw, (cc << logm0) + hi, q, q2);
        if (gdst) { // closing pass: logst == 0, the 2^S results are contiguous
            const u64 qi = in.q; // the prime as an integer (q, q2 are the butterflies' scalars)
            if (is_f64_mode(MODE)) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = f64_canon(f64_of(v[i]), f64_of(q), f64_of(q2));
            } else if (MODE == kIntLazy) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = barrett64(v[i], qi, in.r1);
            } else {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = csub(csub(csub(v[i], q2 << 1), q2), q);
            }
            if (epi.aux) {
                u64 t[R];
                load_contig<R>(t, epi.aux + base);
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = shoup_mul(sub_mod(t[i], v[i], qi), epi.scal, epi.scal_s, qi);
                if (epi.add) {
                    load_contig<R>(t, epi.add + base);
#pragma unroll
                    for (int i = 0; i < R; ++i) v[i] = add_mod(v[i], t[i], qi);
                }
            }
            if (epi.mul0) {
                u64 t[R], w[R];
                load_contig<R>(t, epi.mul1 + base);
#pragma unroll
                for (int i = 0; i < R; ++i) w[i] = barrett128(mul_wide(v[i], t[i]), qi, epi.r0, epi.r1);
                store_contig<R>(w, gdst + epi.dst1_off + base);
                load_contig<R>(t, epi.mul0 + base);
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = barrett128(mul_wide(v[i], t[i]), qi, epi.r0, epi.r1);
            }
            store_contig<R>(v, gdst + base);
        } else {
#pragma unroll
            for (int i = 0; i < R; ++i) sm[sidx(base + (i << logst))] = v[i];
        }
    }
}

template <int MODE>
LB_D void fwd_pass_any(const int S, u64 *sm, const bool from_global, u64 *gdst, const FwdIn &in, const int logn_loc, const int logt,
                       const unsigned cc, const ulonglong2 *tw, const u64 q, const u64 q2, const FwdEpi &epi, const int wlog)
{
    if (S == 3) fwd_pass<3, MODE>(sm, from_global, gdst, in, logn_loc, logt, cc, tw, q, q2, epi, wlog);
    else if (S == 2) fwd_pass<2, MODE>(sm, from_global, gdst, in, logn_loc, logt, cc, tw, q, q2, epi, wlog);
    else fwd_pass<1, MODE>(sm, from_global, gdst, in, logn_loc, logt, cc, tw, q, q2, epi, wlog);
}

// Everything a forward CTA derives from its row index: where the limb comes from, which prime
// and tables it uses, and what the closing pass does with the result.
struct FwdRow {
    FwdIn in;
    FwdEpi epi;
    u64 *dst;
    const ulonglong2 *tw;
    u64 q;
    int mode;
};

// false: this row has nothing to transform (uniform over the cluster that owns the row)
LB_D bool fwd_row_setup(const NttK &a, const int row, FwdRow &r)
{
    const int grp = row / a.per_group, rr = row - grp * a.per_group;
    if (rr >= a.skip_lo && rr < a.skip_hi) return false;
    const int go = grp / a.split, gi = grp - go * a.split;
    int n_in = a.bconv_n;
    size_t src_row = (size_t)go * a.src_outer + a.src_row_off;
    const u64 *mat = a.bconv_mat;
    if (a.digit_alpha > 0) {
        const int s = gi * a.digit_alpha;
        const int e = min(s + a.digit_alpha, a.size_l);
        if (rr >= s && rr < e) return false; // the digit's own limbs stay in NTT form
        src_row += s;
        n_in = e - s;
        if (mat) mat += (size_t)gi * a.mat_group_stride;
    } else {
        src_row += (size_t)gi * a.src_group_stride;
    }
    if (n_in == 0) src_row += rr;
    if (mat) mat += (size_t)rr * a.mat_row_stride;
    const int tbl = rr < a.size_l ? rr + a.tbl_off : a.size_Q + (rr - a.size_l);
    const ModConst mc = a.mc[tbl];
    const int logN = a.logN;
    r.q = mc.q;
    r.tw = a.tw + ((size_t)tbl << logN);
    FwdIn &in = r.in;
    in.n = n_in;
    in.logN = logN;
    in.q = mc.q;
    in.mc = a.mc + tbl;
    in.r0 = mc.r0;
    in.r1 = mc.r1;
    in.src = a.src + (src_row << logN);
    in.mat = mat;
    in.sub = (a.presub && gi < a.presub_inner) ? a.presub + (((size_t)go * a.presub_outer + rr) << logN) : nullptr;
    in.sub_w = in.sub ? a.presub_scal[rr] : 0;
    in.sub_ws = in.sub ? a.presub_scal_s[rr] : 0;
    in.es = a.esmall ? a.esmall + ((size_t)go << logN) : nullptr;
    in.small = a.small ? a.small + ((size_t)grp << logN) : nullptr;
    in.es_p = a.esmall_p;
    r.mode = butterfly_mode(mc.q);
    r.dst = a.dst + (((size_t)go * a.dst_outer + (size_t)gi * a.dst_group_stride + rr) << logN);
    FwdEpi &epi = r.epi;
    epi.aux = a.aux ? a.aux + (((size_t)go * a.aux_outer + (size_t)gi * a.aux_group_stride + rr) << logN) : nullptr;
    epi.add = (a.add && gi < a.add_inner) ? a.add + (((size_t)go * a.add_outer + (size_t)gi * a.add_group_stride + rr) << logN) : nullptr;
    if (a.add1 && gi == 1) epi.add = a.add1 + (((size_t)go * a.add1_outer + rr) << logN);
    epi.scal = a.aux ? a.scal[rr] : 0;
    epi.scal_s = a.aux ? a.scal_s[rr] : 0;
    epi.mul0 = a.mul2 ? a.mul2 + ((size_t)rr << logN) : nullptr;
    epi.mul1 = a.mul2 ? a.mul2 + ((size_t)(a.per_group + rr) << logN) : nullptr;
    epi.dst1_off = (long)a.per_group << logN;
    epi.r0 = mc.r0;
    epi.r1 = mc.r1;
    return true;
}

template <int LOGC>
__global__ void __launch_bounds__(kNttThreads, kNttMinBlocks) ntt_fwd_kernel(const NttK a)
{
    extern __shared__ __align__(16) u64 sm[];
    constexpr int C = 1 << LOGC;
    FwdRow fr;
    if (!fwd_row_setup(a, blockIdx.x >> LOGC, fr)) return;
    const FwdIn &in = fr.in;
    FwdEpi &epi = fr.epi;
    u64 *dst = fr.dst;
    const ulonglong2 *tw = fr.tw;
    const int mode = fr.mode;
    // the butterflies' two scalars: (q, 2q), or (double(q), double(1 / q)) when they run on the FP64 pipe
    const u64 q = is_f64_mode(mode) ? bf_scalar_q<kF64>(fr.q) : fr.q, q2 = is_f64_mode(mode) ? bf_scalar_q2<kF64>(fr.q) : fr.q << 1;
    const int logn_loc = a.logN - LOGC, n_loc = 1 << logn_loc;

    unsigned c = 0;
    if constexpr (LOGC > 0) {
        cg::cluster_group cluster = cg::this_cluster();
        c = cluster.block_rank();
        // Every CTA of the cluster must be running before its shared memory is written; the
        // first loads and butterflies do not touch it, so only the first scatter waits.
        cluster.barrier_arrive();
        u64 *remote[C];
#pragma unroll
        for (int k = 0; k < C; ++k) remote[k] = cluster.map_shared_rank(sm, k);
        const int share = n_loc >> LOGC;
        auto column = [&](const int jj, const bool first) {
            const int j = c * share + jj;
            u64 v[C];
#pragma unroll
            for (int k = 0; k < C; ++k) v[k] = load_in(in, j + k * n_loc);
            if (is_f64_mode(mode)) {
#pragma unroll
                for (int k = 0; k < C; ++k) v[k] = bits_of(f64_from_u52(v[k]));
            }
            if (mode == kF64Tight) {
#pragma unroll
                for (int k = 0; k < C; ++k) v[k] = bits_of(f64_centre(f64_of(v[k]), f64_of(q), f64_of(q2)));
            }
            switch (mode) {
            case kF64: fwd_core<LOGC, kF64>(v, tw, 1u, q, q2); break;
            case kF64Tight: fwd_core<LOGC, kF64Tight>(v, tw, 1u, q, q2); break;
            case kIntLazy: fwd_core<LOGC, kIntLazy>(v, tw, 1u, q, q2); break;
            default: fwd_core<LOGC, kIntStrict>(v, tw, 1u, q, q2); break;
            }
            if (first) cluster.barrier_wait();
#pragma unroll
            for (int k = 0; k < C; ++k) remote[k][sidx(j)] = v[k];
        };
        if ((int)threadIdx.x < share) column(threadIdx.x, true);
        else cluster.barrier_wait();
        for (int jj = threadIdx.x + kNttThreads; jj < share; jj += kNttThreads) column(jj, false);
        cluster.sync(); // all scatters into this CTA have landed; from here on it only touches its own memory
        const size_t off = (size_t)c * n_loc;
        if (epi.aux) epi.aux += off;
        if (epi.add) epi.add += off;
        if (epi.mul0) { epi.mul0 += off; epi.mul1 += off; }
    }

    int logt = logn_loc - 1;
    const unsigned cc = C + c;
    for (int p = 0; p < a.npass; ++p) {
        const int S = a.S[p];
        const bool from_global = (LOGC == 0 && p == 0);
        u64 *gdst = (p == a.npass - 1) ? dst + (size_t)c * n_loc : nullptr;
        const int wlog = p < a.nwide ? -1 : a.wlog;
        switch (mode) {
        case kF64: fwd_pass_any<kF64>(S, sm, from_global, gdst, in, logn_loc, logt, cc, tw, q, q2, epi, wlog); break;
        case kF64Tight: fwd_pass_any<kF64Tight>(S, sm, from_global, gdst, in, logn_loc, logt, cc, tw, q, q2, epi, wlog); break;
        case kIntLazy: fwd_pass_any<kIntLazy>(S, sm, from_global, gdst, in, logn_loc, logt, cc, tw, q, q2, epi, wlog); break;
        default: fwd_pass_any<kIntStrict>(S, sm, from_global, gdst, in, logn_loc, logt, cc, tw, q, q2, epi, wlog); break;
        }
        logt -= S;
        if (p + 1 < a.npass) {
            if (wlog < 0) __syncthreads();
            else __syncwarp();
        }
    }
}

// ---- inverse --------------------------------------------------------------------------

// Stages a run of FP64 inverse butterflies may take before the sums, which double per stage, must be brought
// back to the residue nearest zero: operands of a butterfly stay below 2^50 (their difference below 2^51).
// `fresh`: the run starts from canonical residues below 2^bits; otherwise from |v| <= 2^(bits - 1).
struct F64Run {
    int bits, since, allowed;
    LB_D explicit F64Run(const u64 q) : bits(0), since(0), allowed(0)
    {
        while (bits < 64 && (q >> bits) != 0) ++bits; // q < 2^bits
        allowed = 51 - bits;
    }
    // true: reduce before the next `stages` stages
    LB_D bool before(const int stages)
    {
        const bool reduce = since + stages > allowed;
        if (reduce) {
            since = 0;
            allowed = 52 - bits;
        }
        since += stages;
        return reduce;
    }
};

// IM == kInvF64: `reduce` asks for the centred reduction of the loaded values (see F64Run)
template <int S, bool CLOSE, int IM>
LB_D void inv_pass(u64 *sm, const u64 *gsrc, u64 *gdst, const int logn_loc, const int logt, const unsigned cc,
                   const ulonglong2 *itw, const u64 q, const u64 q2, const u64 cn, const u64 cns, const u64 cw,
                   const u64 cws, const int wlog, const bool reduce)
{
    constexpr int R = 1 << S;
    const int logst = logt;
    const int logm0 = logn_loc - 1 - logt;
    const PassSplit ps = pass_split<S>(logn_loc, wlog);
    for (int g = ps.first; g < ps.end; g += ps.step) {
        const int lo = g & ((1 << logst) - 1), hi = g >> logst;
        const int base = (hi << (logst + S)) + lo;
        u64 v[R];
        if (gsrc) { // opening pass: logst == 0, contiguous
            load_contig<R>(v, gsrc + base);
            if (is_inv_f64(IM)) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = bits_of(f64_from_u52(v[i]));
            }
        } else {
#pragma unroll
            for (int i = 0; i < R; ++i) v[i] = sm[sidx(base + (i << logst))];
        }
        if ((IM == kInvF64 && reduce && !gsrc) || IM == kInvF64Tight) {
#pragma unroll
            for (int i = 0; i < R; ++i) v[i] = bits_of(f64_centre(f64_of(v[i]), f64_of(q), f64_of(q2)));
        }
        inv_core<S, CLOSE, IM>(v, itw, (cc << logm0) + (hi << (S - 1)), q, q2, cn, cns, cw, cws);
        if (gdst) {
#pragma unroll
            for (int i = 0; i < R; ++i) gdst[base + (i << logst)] = v[i];
        } else {
#pragma unroll
            for (int i = 0; i < R; ++i) sm[sidx(base + (i << logst))] = v[i];
        }
    }
}

template <bool CLOSE, int IM>
LB_D void inv_pass_any(const int S, u64 *sm, const u64 *gsrc, u64 *gdst, const int logn_loc, const int logt, const unsigned cc,
                       const ulonglong2 *itw, const u64 q, const u64 q2, const u64 cn, const u64 cns, const u64 cw, const u64 cws,
                       const int wlog, const bool reduce)
{
    if (S == 3) inv_pass<3, CLOSE, IM>(sm, gsrc, gdst, logn_loc, logt, cc, itw, q, q2, cn, cns, cw, cws, wlog, reduce);
    else if (S == 2) inv_pass<2, CLOSE, IM>(sm, gsrc, gdst, logn_loc, logt, cc, itw, q, q2, cn, cns, cw, cws, wlog, reduce);
    else inv_pass<1, CLOSE, IM>(sm, gsrc, gdst, logn_loc, logt, cc, itw, q, q2, cn, cns, cw, cws, wlog, reduce);
}

// The closing constants of an inverse transform for the butterflies' mode: integers with their Shoup quotients,
// or (kInvF64) the constants and their quotients by q as doubles.
struct InvConst {
    u64 q, q2, cn, cns, cw, cws;
};
LB_D InvConst inv_constants(const int im, const u64 q, const u64 cn, const u64 cns, const u64 cw, const u64 cws)
{
    InvConst k;
    if (is_inv_f64(im)) {
        const double qd = (double)q;
        k.q = bits_of(qd);
        k.q2 = bits_of(1.0 / qd);
        k.cn = bits_of((double)cn);
        k.cns = bits_of((double)cn / qd);
        k.cw = bits_of((double)cw);
        k.cws = bits_of((double)cw / qd);
    } else {
        k.q = q; k.q2 = q << 1; k.cn = cn; k.cns = cns; k.cw = cw; k.cws = cws;
    }
    return k;
}

template <int LOGC>
__global__ void __launch_bounds__(kNttThreads, kNttMinBlocks) ntt_inv_kernel(const NttK a)
{
    extern __shared__ __align__(16) u64 sm[];
    constexpr int C = 1 << LOGC;
    const int row = blockIdx.x >> LOGC;
    const int grp = row / a.per_group, rr = row - grp * a.per_group;
    if (rr >= a.skip_lo && rr < a.skip_hi) return;
    const int tbl = rr < a.size_l ? rr + a.tbl_off : a.size_Q + (rr - a.size_l);
    const ModConst mc = a.mc[tbl];
    const u64 q = mc.q, q2 = q << 1;
    const int logN = a.logN, logn_loc = logN - LOGC, n_loc = 1 << logn_loc;
    const ulonglong2 *itw = a.tw + ((size_t)tbl << logN);
    const int go = grp / a.split, gi = grp - go * a.split;
    const u64 *src = a.src + (((size_t)go * a.src_outer + (size_t)gi * a.src_group_stride + rr + a.src_row_off) << logN);
    u64 *dst = a.dst + (((size_t)go * a.dst_outer + (size_t)gi * a.dst_group_stride + rr) << logN);
    u64 cn = mc.ninv, cns = mc.ninvs, cw = mc.iw1n, cws = mc.iw1ns;
    if (a.fold) {
        const u64 *f = a.fold + 4 * rr;
        cn = f[0]; cns = f[1]; cw = f[2]; cws = f[3];
    }
    unsigned c = 0;
    if constexpr (LOGC > 0) c = cg::this_cluster().block_rank();
    const unsigned cc = C + c;
    const int im = inverse_mode(q);
    const InvConst ic = inv_constants(im, q, cn, cns, cw, cws);
    F64Run run(q);
    int logt = 0;
    for (int p = 0; p < a.npass; ++p) {
        const int S = a.S[p];
        const u64 *gsrc = (p == 0) ? src + (size_t)c * n_loc : nullptr;
        const bool closing = (LOGC == 0 && p == a.npass - 1);
        u64 *gdst = closing ? dst : nullptr;
        const int wlog = p >= a.npass - a.nwide ? -1 : a.wlog;
        if (p > 0) {
            if (wlog < 0) __syncthreads();
            else __syncwarp();
        }
        const bool red = run.before(S);
        if (im == kInvF64) {
            if (closing) inv_pass_any<true, kInvF64>(S, sm, gsrc, gdst, logn_loc, logt, cc, itw, ic.q, ic.q2, ic.cn, ic.cns, ic.cw, ic.cws, wlog, red);
            else inv_pass_any<false, kInvF64>(S, sm, gsrc, gdst, logn_loc, logt, cc, itw, ic.q, ic.q2, ic.cn, ic.cns, ic.cw, ic.cws, wlog, red);
        } else if (im == kInvF64Tight) {
            if (closing) inv_pass_any<true, kInvF64Tight>(S, sm, gsrc, gdst, logn_loc, logt, cc, itw, ic.q, ic.q2, ic.cn, ic.cns, ic.cw, ic.cws, wlog, true);
            else inv_pass_any<false, kInvF64Tight>(S, sm, gsrc, gdst, logn_loc, logt, cc, itw, ic.q, ic.q2, ic.cn, ic.cns, ic.cw, ic.cws, wlog, true);
        } else {
            if (closing) inv_pass_any<true, kInvInt>(S, sm, gsrc, gdst, logn_loc, logt, cc, itw, q, q2, cn, cns, cw, cws, wlog, false);
            else inv_pass_any<false, kInvInt>(S, sm, gsrc, gdst, logn_loc, logt, cc, itw, q, q2, cn, cns, cw, cws, wlog, false);
        }
        logt += S;
    }
    if constexpr (LOGC > 0) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync(); // all local transforms of the cluster are in shared memory (and every peer is running)
        const u64 *remote[C];
#pragma unroll
        for (int k = 0; k < C; ++k) remote[k] = cluster.map_shared_rank(sm, k);
        const int share = n_loc >> LOGC;
        const bool red = run.before(LOGC);
        for (int jj = threadIdx.x; jj < share; jj += kNttThreads) {
            const int j = c * share + jj;
            u64 v[C];
#pragma unroll
            for (int kk = 0; kk < C; ++kk) v[kk] = remote[kk][sidx(j)];
            if (im == kInvF64) {
                if (red) {
#pragma unroll
                    for (int kk = 0; kk < C; ++kk) v[kk] = bits_of(f64_centre(f64_of(v[kk]), f64_of(ic.q), f64_of(ic.q2)));
                }
                inv_core<LOGC, true, kInvF64>(v, itw, C / 2, ic.q, ic.q2, ic.cn, ic.cns, ic.cw, ic.cws);
            } else if (im == kInvF64Tight) {
#pragma unroll
                for (int kk = 0; kk < C; ++kk) v[kk] = bits_of(f64_centre(f64_of(v[kk]), f64_of(ic.q), f64_of(ic.q2)));
                inv_core<LOGC, true, kInvF64Tight>(v, itw, C / 2, ic.q, ic.q2, ic.cn, ic.cns, ic.cw, ic.cws);
            } else {
                inv_core<LOGC, true, kInvInt>(v, itw, C / 2, q, q2, cn, cns, cw, cws);
            }
#pragma unroll
            for (int kk = 0; kk < C; ++kk) dst[j + kk * n_loc] = v[kk];
        }
        cluster.sync(); // shared memory stays alive until every peer has read it
    }
}

} // namespace lb

#include "ntt_twopass.cuh"

namespace lb {

// ---- launchers ------------------------------------------------------------------------

// Splits `stages` into as few register passes of at most R stages as possible, evenly.
static int split_even(int stages, int R, unsigned char *out)
{
    const int count = (stages + R - 1) / R;
    int n = 0;
    for (int i = 0; i < count; ++i) {
        const int s = (stages + (count - i) - 1) / (count - i);
        out[n++] = (unsigned char)s;
        stages -= s;
    }
    return n;
}

struct PassPlan {
    int npass, nwide, wlog;
    unsigned char S[8];
};

static PassPlan plan_passes(int logn_loc, bool forward)
{
    // The log2(warps) stages whose butterflies span more than one warp's chunk run as
    // CTA-wide passes; the rest stay inside a warp's contiguous chunk.  Of those, the pass
    // that touches global memory with contiguous per-thread data (forward: last, inverse:
    // first) takes the largest radix.  Short transforms keep every pass CTA-wide.
    const int R = kMaxRadixLog;
    int lw = 0;
    while ((32 << lw) < kNttThreads) ++lw;
    PassPlan pl;
    unsigned char wide[8], mid[8];
    int nw = 0, local = logn_loc;
    pl.wlog = -1;
    if (logn_loc - lw >= 8) {
        local = logn_loc - lw;
        pl.wlog = local;
        nw = split_even(lw, R, wide);
    }
    const int edge = local >= R ? R : local;
    const int nm = split_even(local - edge, R, mid);
    int n = 0;
    if (forward) {
        for (int i = 0; i < nw; ++i) pl.S[n++] = wide[i];
        for (int i = 0; i < nm; ++i) pl.S[n++] = mid[i];
        pl.S[n++] = (unsigned char)edge;
    } else {
        pl.S[n++] = (unsigned char)edge;
        for (int i = nm - 1; i >= 0; --i) pl.S[n++] = mid[i];
        for (int i = nw - 1; i >= 0; --i) pl.S[n++] = wide[i];
    }
    pl.npass = n;
    pl.nwide = nw;
    if (pl.wlog < 0) pl.nwide = n; // every pass CTA-wide
    return pl;
}

static bool plain_input(const NttK &k)
{
    return k.bconv_n == 0 && k.digit_alpha == 0 && !k.presub && !k.esmall && !k.small && !k.aux && !k.mul2;
}

static const char *kernel_label(bool forward, const NttK &k)
{
    return !forward ? "ntt_inv_kernel" : plain_input(k) ? "ntt_fwd_kernel(plain input)" : "ntt_fwd_kernel(fused input)";
}

// algorithmic bytes of a transform for the diagnostics: what its source, its limb rows (once) and its fused ends hold
struct NttBytes {
    double in, rows, ends;
};

// rings below 4096 points (LOGC == 0) and of 131072 points (LOGC == 4)
template <int LOGC>
static int launch(bool forward, const NttK &k, int rows, size_t smem, cudaStream_t stream, const NttBytes &b)
{
    auto kern = forward ? ntt_fwd_kernel<LOGC> : ntt_inv_kernel<LOGC>;
    // function attributes belong to the device the kernel image is loaded on
    static bool configured[64][2] = {};
    int dev = 0;
    LB_CUDA(cudaGetDevice(&dev));
    bool &done = configured[dev & 63][forward];
    if (!done) {
        // largest request any ring degree makes: 8192 points plus one pad word per 16
        LB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 72 * 1024));
        if (LOGC > 3) LB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        done = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows << LOGC);
    cfg.blockDim = dim3(kNttThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1 << LOGC;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    count_launch(kernel_label(forward, k), stream, b.in + b.rows + b.ends);
    LB_CUDA(cudaLaunchKernelEx(&cfg, kern, k));
    return LB_OK;
}

// `grid` blocks of `threads`; the kernel is set up while its predecessor in the stream ends (see grid_wait)
static int launch_serial(void (*kern)(const NttK), const NttK &k, long grid, int threads, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    LB_CUDA(cudaLaunchKernelEx(&cfg, kern, k));
    return LB_OK;
}

// Polynomials of one prime that share a block of the row kernels: as many as divide the batch without leaving more than
// an eighth of the half warps idle.  In mod-up the digits of one ciphertext skip different rows, so there a block takes
// the same digit of several ciphertexts.
static void share_rows(NttK &k, int n_groups)
{
    k.poly_step = k.digit_alpha > 0 ? k.split : 1;
    k.n_polys = n_groups / k.poly_step;
    k.log_polys = 3;
    while (k.log_polys > 0 && ((k.n_polys + (1 << k.log_polys) - 1) >> k.log_polys << k.log_polys) * 8L > k.n_polys * 9L) --k.log_polys;
}

template <int A>
static int launch_twopass(bool forward, NttK &k, int rows, cudaStream_t stream, const NttBytes &b)
{
    using C = ColShape<A>;
    share_rows(k, rows / k.per_group);
    const long col_grid = (long)rows * C::TILES;
    const long row_grid = (long)((k.n_polys + (1 << k.log_polys) - 1) >> k.log_polys) * k.poly_step * k.per_group << (A - 3 + k.log_polys);
    const bool plain = plain_input(k);
    int rc;
    if (forward) {
        // a conversion of several rows reads them again for every target: its own label, so that no other launch's traffic stands for it
        count_launch(plain ? "ntt_fwd_col_kernel(plain)" : k.bconv_mat ? "ntt_fwd_col_kernel(conversion)" : "ntt_fwd_col_kernel(fused)", stream,
                     b.in + b.rows);
        if ((rc = launch_serial(plain ? ntt_fwd_col_kernel<A, true> : ntt_fwd_col_kernel<A, false>, k, col_grid, C::THREADS, stream))) return rc;
        count_launch(plain ? "ntt_fwd_row_kernel(plain)" : "ntt_fwd_row_kernel(fused)", stream, 2 * b.rows + b.ends);
        return launch_serial(plain ? ntt_fwd_row_kernel<true> : ntt_fwd_row_kernel<false>, k, row_grid, kRowThreads, stream);
    }
    count_launch("ntt_inv_row_kernel", stream, b.in + b.rows);
    if ((rc = launch_serial(ntt_inv_row_kernel, k, row_grid, kRowThreads, stream))) return rc;
    count_launch("ntt_inv_col_kernel", stream, 2 * b.rows);
    return launch_serial(ntt_inv_col_kernel<A>, k, col_grid, C::THREADS, stream);
}

static int run(Context *ctx, const NttJob &job, bool forward, cudaStream_t stream)
{
    const HostParams &hp = ctx->hp;
    const int rows = job.n_groups * job.per_group;
    if (rows <= 0) return LB_OK;
    NttK k;
    k.src = job.src;
    k.dst = job.dst;
    k.tw = forward ? ctx->d_tw : ctx->d_itw;
    k.mc = ctx->d_mc;
    k.logN = hp.logN;
    k.per_group = job.per_group;
    k.size_l = job.size_l;
    k.size_Q = hp.size_Q;
    k.tbl_off = job.tbl_off;
    k.split = job.split > 0 ? job.split : 1;
    k.src_group_stride = job.src_group_stride >= 0 ? job.src_group_stride : job.per_group;
    k.dst_group_stride = job.dst_group_stride >= 0 ? job.dst_group_stride : job.per_group;
    k.aux_group_stride = job.aux_group_stride >= 0 ? job.aux_group_stride : job.per_group;
    k.add_group_stride = job.add_group_stride >= 0 ? job.add_group_stride : job.per_group;
    k.src_outer = job.src_outer >= 0 ? job.src_outer : k.split * k.src_group_stride;
    k.dst_outer = job.dst_outer >= 0 ? job.dst_outer : k.split * k.dst_group_stride;
    k.aux_outer = job.aux_outer >= 0 ? job.aux_outer : k.split * k.aux_group_stride;
    k.add_outer = job.add_outer >= 0 ? job.add_outer : k.split * k.add_group_stride;
    k.src_row_off = job.src_row_off;
    k.skip_lo = job.skip_lo;
    k.skip_hi = job.skip_hi;
    k.bconv_n = job.bconv_n;
    k.digit_alpha = job.digit_alpha;
    k.add_inner = job.add_inner;
    k.add1 = job.add1;
    k.add1_outer = job.add1_outer;
    k.bconv_mat = job.bconv_mat;
    k.mat_group_stride = job.mat_group_stride;
    k.mat_row_stride = job.mat_row_stride;
    k.aux = job.aux;
    k.scal = job.scal;
    k.scal_s = job.scal_s;
    k.add = job.add;
    k.fold = job.fold;
    k.mul2 = job.mul2;
    k.mid = job.mid;
    k.presub = job.presub;
    k.esmall = job.esmall;
    k.small = job.small;
    k.esmall_p = job.esmall_p;
    k.presub_scal = job.presub_scal;
    k.presub_scal_s = job.presub_scal_s;
    k.presub_outer = job.presub_outer >= 0 ? job.presub_outer : job.per_group;
    k.presub_inner = job.presub ? job.presub_inner : 0;
    const int logc = hp.logN > kMaxLocalLog ? hp.logN - kMaxLocalLog : 0;
    const int logn_loc = hp.logN - logc;
    const PassPlan pl = plan_passes(logn_loc, forward);
    k.npass = pl.npass;
    k.nwide = pl.nwide;
    k.wlog = pl.wlog;
    for (int i = 0; i < pl.npass; ++i) k.S[i] = pl.S[i];
    const size_t n_loc = size_t(1) << logn_loc;
    const size_t smem = (n_loc + (n_loc >> 4) + 2) * sizeof(u64);
    // diagnostics: rows written once; plain rows read once; fused loaders read the group's source rows once per group, plus the
    // rows the prologue and the epilogue fold in
    const double limb = 8.0 * (double)hp.N;
    const int live = job.per_group - (job.skip_hi > job.skip_lo ? job.skip_hi - job.skip_lo : 0);
    const double out_rows = (double)job.n_groups * live;
    NttBytes b = {0, out_rows * limb, 0};
    if (job.digit_alpha > 0) b.in = (double)job.n_groups * job.digit_alpha * limb;
    else if (job.bconv_n > 0) b.in = (double)job.n_groups * job.bconv_n * limb;
    else if (job.small) b.in = (double)job.n_groups * (double)hp.N; // one byte per coefficient and group
    else b.in = out_rows * limb;
    const double outer = (double)job.n_groups / k.split;
    if (job.aux) b.ends += out_rows * limb;
    if (job.add) b.ends += outer * (job.add_inner < k.split ? job.add_inner : k.split) * live * limb;
    if (job.add1) b.ends += outer * live * limb;
    if (job.presub) b.in += outer * (k.presub_inner < k.split ? k.presub_inner : k.split) * live * limb;
    if (job.esmall) b.in += outer * (double)hp.N;
    if (job.mul2) b.ends += out_rows * limb + 2.0 * job.per_group * limb; // a second output row per row, the two fixed rows once
    switch (hp.logN) {
    case 12: return launch_twopass<4>(forward, k, rows, stream, b);
    case 13: return launch_twopass<5>(forward, k, rows, stream, b);
    case 14: return launch_twopass<6>(forward, k, rows, stream, b);
    case 15: return launch_twopass<7>(forward, k, rows, stream, b);
    case 16: return launch_twopass<8>(forward, k, rows, stream, b);
    case 17: return launch<4>(forward, k, rows, smem, stream, b);
    default: return launch<0>(forward, k, rows, smem, stream, b);
    }
}

int ntt_forward(Context *ctx, const NttJob &job, cudaStream_t stream) { return run(ctx, job, true, stream); }
int ntt_inverse(Context *ctx, const NttJob &job, cudaStream_t stream) { return run(ctx, job, false, stream); }

} // namespace lb
