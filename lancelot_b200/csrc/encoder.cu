// CKKS encoder: canonical-embedding special FFT in double precision plus RNS decompose /
// compose (cahel-main/src/ckks.cu:104-209,292-465, fft.cu:54-344, rns_base.cu:121-156,325-459).
//
// Encoding is bit-sensitive: a coefficient is round()ed after the inverse FFT, so the
// butterfly expression shapes of the reference are kept exactly (x0 + x1, (x0 - x1) * w with
// the complex product's difference/sum contracted into one fused multiply-add each, scale/n
// multiplied in after the last stage).  Only the schedule differs: one kernel per batch of
// messages, a thread-block cluster per message, local stages in shared memory, the last
// log2(C) stages through distributed shared memory, and the rounding + residue step fused
// into the final store, instead of one global pass per stage plus a host round trip.
#include <cooperative_groups.h>

#include <utility>

#include "context.h"

namespace cg = cooperative_groups;

namespace lb {

constexpr int kFftThreads = 256;
constexpr int kFftLocalLog = 12; // 4096 complex points (64 KiB + padding) per CTA

struct cplx {
    double x, y;
};

LB_D cplx c_add(cplx a, cplx b) { return {__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)}; }
LB_D cplx c_sub(cplx a, cplx b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)}; }
// cuCmul as the device compiler contracts it in the reference's kernels: one rounded product feeding one fused
// multiply-add per part.  Which product of the imaginary part is the rounded one differs between the reference's two
// inverse-FFT kernels: the multi-stage kernel that runs the first eleven stages (cahel-main/src/fft.cu:194-268,
// SWITCH_POINT = 2048) rounds a.x * b.y, the per-stage kernel of the later stages (fft.cu:279-344) rounds a.y * b.x.
// Plaintexts at scale 2^50, whose largest coefficients keep two or three bits below the rounding point, pin this
// (reference-made fixtures n4096_s50, n8192_s50, n65536_a8).
constexpr int kRefIfftFirstKernelStages = 11;
LB_D cplx c_mul(cplx a, cplx b, const bool first_kernel_stage = false)
{
    cplx r;
    r.x = __fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y));
    r.y = first_kernel_stage ? __fma_rn(a.y, b.x, __dmul_rn(a.x, b.y)) : __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x));
    return r;
}

LB_D int fidx(int i) { return i + (i >> 4); }

struct EncK {
    const void *values; // [batch][value_stride] of dtype
    int dtype;          // 0 double real, 1 float real, 2 complex double
    long value_stride;  // elements between messages
    int n_values;
    u64 *pt;            // [batch][size_l][N]
    const double2 *roots;
    const uint32_t *group;
    const double2 *tw; // stage-ordered copy of the twiddles (see Context::d_ifft_tw), or nullptr
    const ModConst *mc;
    int logN, logn, size_l;
    double fix;
    double too_large;
    int *status;
    int npass;
    unsigned char S[8];
};

LB_D cplx load_value(const EncK &a, const long msg, const unsigned idx)
{
    cplx v = {0.0, 0.0};
    if (idx < (unsigned)a.n_values) {
        if (a.dtype == 0) v.x = reinterpret_cast<const double *>(a.values)[msg * a.value_stride + idx];
        else if (a.dtype == 1) v.x = (double)reinterpret_cast<const float *>(a.values)[msg * a.value_stride + idx];
        else {
            const double2 t = reinterpret_cast<const double2 *>(a.values)[msg * a.value_stride + idx];
            v.x = t.x;
            v.y = t.y;
        }
    }
    return v;
}

// twiddle of butterfly group k at stage u (pairs = 2^u): fft.cu:216-222
LB_D cplx ifft_twiddle(const EncK &a, const unsigned k, const int u)
{
    if (a.tw) { // one load instead of two dependent ones
        const unsigned n = 1u << a.logn;
        const double2 w = __ldg(a.tw + (n - (n >> u)) + k);
        return {w.x, w.y};
    }
    const int logRatio = a.logN + 1 - a.logn - 2;
    const unsigned M = 2u << a.logN;
    const unsigned rev = a.logn > 1 ? (__brev(k << u) >> (33 - a.logn)) : 0u;
    unsigned p = a.group[rev];
    p <<= (u + logRatio);
    p &= M - 1;
    const double2 w = a.roots[M - p];
    return {w.x, w.y};
}

// round, reduce into every prime, and store coefficient `pos` of the plaintext (rns_base.cu:121-156)
// QUOT_F64: coefficients below 2^51 take their quotients on the FP64 pipe.  Not in the cluster kernels: their unrolled copies
// of the longer code cost a product chain at N = 2^13 30 us.
template <bool QUOT_F64>
LB_D void emit_coeff(const EncK &a, u64 *pt_msg, const unsigned pos, const double value)
{
    const double r = round(value);
    const bool neg = signbit(r);
    const double av = fabs(r);
    // ceil(log2(av)) + 1 >= total bit count  <=>  av > 2^(total - 2)   (ckks.cu:185-191)
    if (av > a.too_large) atomicOr(a.status, 1);
    const long N = 1L << a.logN;
    if (QUOT_F64 && av < 2251799813685248.0) { // 2^51: what a message at Lancelot's scale of 2^40 encodes to
        const u64 m = u52_from_f64(av);
        for (int l = 0; l < a.size_l; ++l) {
            const ModConst &mc = a.mc[l];
            u64 t;
            if (mc.kind == kWideF64) t = f64_canon(r, mc.qd, mc.qi);
            else {
                t = mc.q >> 51 ? m : barrett64(m, mc.q, mc.r1);
                if (neg && t) t = mc.q - t;
            }
            pt_msg[l * N + pos] = t;
        }
    } else if (av < 18446744073709551616.0) {
        const u64 m = (u64)av;
        for (int l = 0; l < a.size_l; ++l) {
            const ModConst mc = a.mc[l];
            u64 t = barrett64(m, mc.q, mc.r1);
            if (neg && t) t = mc.q - t;
            pt_msg[l * N + pos] = t;
        }
    } else {
        u128d z;
        z.lo = (u64)fmod(av, 18446744073709551616.0);
        z.hi = (u64)(av / 18446744073709551616.0);
        for (int l = 0; l < a.size_l; ++l) {
            const ModConst mc = a.mc[l];
            u64 t = barrett128(z, mc.q, mc.r0, mc.r1);
            if (neg && t) t = mc.q - t;
            pt_msg[l * N + pos] = t;
        }
    }
}

template <int S>
LB_D void ifft_pass(cplx *sm, const EncK &a, const long msg, const bool first, const bool last_global, u64 *pt_msg,
                    const int logn_loc, const int logt, const unsigned c, const int ratio_log)
{
    constexpr int R = 1 << S;
    const int groups = 1 << (logn_loc - S);
    for (int g = threadIdx.x; g < groups; g += kFftThreads) {
        const int lo = g & ((1 << logt) - 1), hi = g >> logt;
        const int base = (hi << (logt + S)) + lo;
        cplx v[R];
        if (first) { // logt == 0: the bit-reversal placement is folded into the load
            const unsigned gbase = (c << logn_loc) + base;
            // the type switch sits outside the element loop so that the R loads are in flight together
            unsigned idx[R];
#pragma unroll
            for (int i = 0; i < R; ++i) idx[i] = __brev(gbase + i) >> (32 - a.logn);
            if (a.dtype == 1) {
                const float *f = reinterpret_cast<const float *>(a.values) + msg * a.value_stride;
                float t[R];
#pragma unroll
                for (int i = 0; i < R; ++i) t[i] = idx[i] < (unsigned)a.n_values ? f[idx[i]] : 0.0f;
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = {(double)t[i], 0.0};
            } else if (a.dtype == 0) {
                const double *f = reinterpret_cast<const double *>(a.values) + msg * a.value_stride;
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = {idx[i] < (unsigned)a.n_values ? f[idx[i]] : 0.0, 0.0};
            } else {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = load_value(a, msg, idx[i]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < R; ++i) v[i] = sm[fidx(base + (i << logt))];
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int u = logt + s;
            const int dist = 1 << s;
#pragma unroll
            for (int b = 0; b < (1 << (S - 1 - s)); ++b) {
                // global butterfly group index of this pair
                const unsigned k = ((c << logn_loc) >> (u + 1)) + (hi << (S - 1 - s)) + b;
                const cplx w = ifft_twiddle(a, k, u);
                const bool early = u < kRefIfftFirstKernelStages; // uniform over the CTA
#pragma unroll
                for (int i = 0; i < dist; ++i) {
                    cplx &x0 = v[b * 2 * dist + i], &x1 = v[b * 2 * dist + i + dist];
                    const cplx s0 = c_add(x0, x1), s1 = c_sub(x0, x1);
                    x0 = s0;
                    x1 = c_mul(s1, w, early);
                }
            }
        }
        if (last_global) { // single-CTA transform: this pass holds the final stage
            const unsigned n = 1u << a.logn;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const unsigned e = base + (i << logt);
                cplx z = v[i];
                if (a.fix != 0.0) {
                    z.x = __dmul_rn(z.x, a.fix);
                    z.y = __dmul_rn(z.y, a.fix);
                }
                emit_coeff<false>(a, pt_msg, e << ratio_log, z.x);
                emit_coeff<false>(a, pt_msg, (e + n) << ratio_log, z.y);
            }
        } else {
#pragma unroll
            for (int i = 0; i < R; ++i) sm[fidx(base + (i << logt))] = v[i];
        }
    }
}

// fills the stage-ordered twiddle table from the root table: the same values, found once
__global__ void ifft_twiddle_table_kernel(EncK a, double2 *out)
{
    const unsigned n = 1u << a.logn;
    a.tw = nullptr;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i + 1 < n; i += gridDim.x * blockDim.x) {
        // stage u holds the entries [n - (n >> u), n - (n >> (u + 1)))
        int u = 0;
        while (i >= n - (n >> (u + 1))) ++u;
        const unsigned k = i - (n - (n >> u));
        const cplx w = ifft_twiddle(a, k, u);
        out[i] = make_double2(w.x, w.y);
    }
}

template <int LOGC>
__global__ void __launch_bounds__(kFftThreads) encode_ifft_kernel(const EncK a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx *sm = reinterpret_cast<cplx *>(smraw);
    constexpr int C = 1 << LOGC;
    const long msg = blockIdx.x >> LOGC;
    const int logn_loc = a.logn - LOGC, n_loc = 1 << logn_loc;
    const int ratio_log = (a.logN - 1) - a.logn;
    u64 *pt_msg = a.pt + ((msg * a.size_l) << a.logN);
    unsigned c = 0;
    if constexpr (LOGC > 0) {
        c = cg::this_cluster().block_rank();
        cg::this_cluster().sync();
    }
    int logt = 0;
    for (int p = 0; p < a.npass; ++p) {
        const int S = a.S[p];
        const bool last_global = (LOGC == 0 && p == a.npass - 1);
        if (p > 0) __syncthreads();
        if (S == 3) ifft_pass<3>(sm, a, msg, p == 0, last_global, pt_msg, logn_loc, logt, c, ratio_log);
        else if (S == 2) ifft_pass<2>(sm, a, msg, p == 0, last_global, pt_msg, logn_loc, logt, c, ratio_log);
        else ifft_pass<1>(sm, a, msg, p == 0, last_global, pt_msg, logn_loc, logt, c, ratio_log);
        logt += S;
    }
    if constexpr (LOGC > 0) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        const cplx *remote[C];
#pragma unroll
        for (int k = 0; k < C; ++k) remote[k] = cluster.map_shared_rank(sm, k);
        const int share = n_loc >> LOGC;
        const unsigned n = 1u << a.logn;
        for (int jj = threadIdx.x; jj < share; jj += kFftThreads) {
            const int j = c * share + jj;
            cplx v[C];
#pragma unroll
            for (int k = 0; k < C; ++k) v[k] = remote[k][fidx(j)];
#pragma unroll
            for (int s = 0; s < LOGC; ++s) {
                const int u = logn_loc + s;
                const int dist = 1 << s;
#pragma unroll
                for (int b = 0; b < (1 << (LOGC - 1 - s)); ++b) {
                    // element j + kk * n_loc with kk = b * 2 * dist + i: group index (j + kk n_loc) >> (u + 1) = b
                    const cplx w = ifft_twiddle(a, (unsigned)b, u);
#pragma unroll
                    for (int i = 0; i < dist; ++i) {
                        cplx &x0 = v[b * 2 * dist + i], &x1 = v[b * 2 * dist + i + dist];
                        const cplx s0 = c_add(x0, x1), s1 = c_sub(x0, x1);
                        x0 = s0;
                        x1 = c_mul(s1, w);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const unsigned e = j + k * n_loc;
                cplx z = v[k];
                if (a.fix != 0.0) {
                    z.x = __dmul_rn(z.x, a.fix);
                    z.y = __dmul_rn(z.y, a.fix);
                }
                emit_coeff<false>(a, pt_msg, e << ratio_log, z.x);
                emit_coeff<false>(a, pt_msg, (e + n) << ratio_log, z.y);
            }
        }
        cluster.sync();
    }
}

// ---- inverse FFT in two kernels, for 4096 slots and more where scratch for the values in between is at hand ----
// A message is a matrix of n / 256 rows of 256 values.  The row kernel gathers the input in bit-reversed order and runs the
// stages with spans 1 .. 128, the column kernel the rest and the rounding; a thread holds 16 values and takes four
// stages at a time in registers, with one exchange per kernel.  The cluster kernel above walks six passes with a block or
// cluster barrier each, eight values per thread and three blocks of eight warps per SM, and waits at those barriers:
// 51 messages of 32768 slots 110 -> 65 us.  The price is a second trip of 16 bytes per value through L2 / HBM.
constexpr int kRowVals = 256, kEncThreads = 128, kRowsPerBlock = 8;
constexpr int kRowStride = kRowVals + 17; // one spare value per 16 of a row, and the rows on different banks

// S stages on values AT .. AT + 2^S - 1, whose lowest position bits are the register index: stage U + s, group (g << (S - 1 - s)) + b
template <int S, int U, int AT = 0>
LB_D void ifft_stages(double (&re)[16], double (&im)[16], const double2 *__restrict__ tw, const unsigned n, const unsigned g)
{
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const double2 *t = tw + (n - (n >> (U + s))) + ((size_t)g << (S - 1 - s));
#pragma unroll
        for (int j = 0; j < (1 << (S - 1)); ++j) {
            const int b = j >> s, x0 = AT + (b << (s + 1)) + (j & ((1 << s) - 1)), x1 = x0 + (1 << s);
            const double2 w = __ldg(t + b);
            const cplx p = {re[x0], im[x0]}, q = {re[x1], im[x1]};
            const cplx s0 = c_add(p, q), s1 = c_mul(c_sub(p, q), cplx{w.x, w.y}, U + s < kRefIfftFirstKernelStages);
            re[x0] = s0.x;
            im[x0] = s0.y;
            re[x1] = s1.x;
            im[x1] = s1.y;
        }
    }
}
// the last S stages of a column's groups of 2^S rows, whose twiddles are those of group 0
template <int S, int... I>
LB_D void ifft_groups(double (&re)[16], double (&im)[16], const double2 *__restrict__ tw, const unsigned n, std::integer_sequence<int, I...>)
{
    (ifft_stages<S, 12, I * (1 << S)>(re, im, tw, n, 0), ...);
}

// A block takes the eight rows whose input positions are neighbours (32 bytes of floats per sector read).
__global__ void __launch_bounds__(kEncThreads, 4) encode_row_kernel(const __grid_constant__ EncK a, cplx *__restrict__ mid)
{
    __shared__ __align__(16) cplx sm[kRowsPerBlock * kRowStride];
    const unsigned n = 1u << a.logn, rows_log = a.logn - 8;
    const long msg = blockIdx.y;
    const unsigned first = blockIdx.x * kRowsPerBlock; // the rows' bit-reversed numbers start here
    double re[16], im[16];
    {
        const unsigned h = threadIdx.x & (kRowsPerBlock - 1), t = threadIdx.x / kRowsPerBlock;
        const unsigned low = first + h + ((__brev(t) >> 28) << rows_log); // input position of value k: bitrev4(k) n / 16 + low
        if (a.dtype == 1) {
            const float *f = reinterpret_cast<const float *>(a.values) + msg * a.value_stride;
            float x[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const unsigned idx = ((__brev((unsigned)k) >> 28) << (a.logn - 4)) + low;
                x[k] = idx < (unsigned)a.n_values ? f[idx] : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                re[k] = (double)x[k];
                im[k] = 0.0;
            }
        } else if (a.dtype == 0) {
            const double *f = reinterpret_cast<const double *>(a.values) + msg * a.value_stride;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const unsigned idx = ((__brev((unsigned)k) >> 28) << (a.logn - 4)) + low;
                re[k] = idx < (unsigned)a.n_values ? f[idx] : 0.0;
                im[k] = 0.0;
            }
        } else {
            const double2 *f = reinterpret_cast<const double2 *>(a.values) + msg * a.value_stride;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const unsigned idx = ((__brev((unsigned)k) >> 28) << (a.logn - 4)) + low;
                const double2 x = idx < (unsigned)a.n_values ? f[idx] : make_double2(0.0, 0.0);
                re[k] = x.x;
                im[k] = x.y;
            }
        }
        const unsigned r = __brev(first + h) >> (32 - rows_log);
        ifft_stages<4, 0>(re, im, a.tw, n, r * 16 + t);
        cplx *row = sm + h * kRowStride + t * 17;
#pragma unroll
        for (int k = 0; k < 16; ++k) row[k] = cplx{re[k], im[k]};
    }
    __syncthreads();
    const unsigned h = threadIdx.x >> 4, t = threadIdx.x & 15, r = __brev(first + h) >> (32 - rows_log);
    const cplx *row = sm + h * kRowStride + t;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const cplx z = row[17 * k];
        re[k] = z.x;
        im[k] = z.y;
    }
    ifft_stages<4, 4>(re, im, a.tw, n, r);
    cplx *dst = mid + ((size_t)msg << a.logn) + r * kRowVals + t;
#pragma unroll
    for (int k = 0; k < 16; ++k) dst[16 * k] = cplx{re[k], im[k]};
}

// A: log2 of the rows (4 .. 7).  2^(A - 4) threads per column; the twiddles depend on the row only.
template <int A>
__global__ void __launch_bounds__(kEncThreads, 4) encode_col_kernel(const __grid_constant__ EncK a, const cplx *__restrict__ mid)
{
    constexpr int S2 = A - 4, TPC = 1 << S2, COLS = kEncThreads / TPC, G = 16 >> S2;
    __shared__ __align__(16) cplx sm[16 * kEncThreads];
    const unsigned n = 1u << (A + 8);
    const long msg = blockIdx.y;
    const int cl = threadIdx.x % COLS, t = threadIdx.x / COLS, col = blockIdx.x * COLS + cl;
    const cplx *src = mid + ((size_t)msg << (A + 8)) + col;
    double re[16], im[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const cplx z = src[(16 * t + k) * kRowVals];
        re[k] = z.x;
        im[k] = z.y;
    }
    ifft_stages<4, 8>(re, im, a.tw, n, t);
    if constexpr (S2 > 0) {
#pragma unroll
        for (int k = 0; k < 16; ++k) sm[(16 * t + k) * COLS + cl] = cplx{re[k], im[k]};
        __syncthreads();
        // group i of the thread: rows t + TPC i + 16 k
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const cplx z = sm[(t + TPC * (i / TPC) + 16 * (i % TPC)) * COLS + cl];
            re[i] = z.x;
            im[i] = z.y;
        }
        ifft_groups<S2>(re, im, a.tw, n, std::make_integer_sequence<int, G>());
        __syncthreads();
    }
    u64 *pt_msg = a.pt + ((msg * a.size_l) << a.logN);
    const int ratio_log = a.logN - 1 - a.logn;
    // the rounding is long: one copy of it, fed from the thread's own words of shared memory
#pragma unroll
    for (int i = 0; i < 16; ++i) sm[i * kEncThreads + threadIdx.x] = cplx{re[i], im[i]};
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
        const int row = S2 > 0 ? t + TPC * (i / TPC) + 16 * (i % TPC) : i;
        const unsigned e = (unsigned)(row * kRowVals + col);
        cplx z = sm[i * kEncThreads + threadIdx.x];
        if (a.fix != 0.0) {
            z.x = __dmul_rn(z.x, a.fix);
            z.y = __dmul_rn(z.y, a.fix);
        }
        emit_coeff<true>(a, pt_msg, e << ratio_log, z.x);
        emit_coeff<true>(a, pt_msg, (e + n) << ratio_log, z.y);
    }
}

template <int A>
static void launch_encode_two(const EncK &k, int batch, cplx *mid, cudaStream_t stream)
{
    constexpr int COLS = kEncThreads >> (A - 4);
    count_launch("encode_row_kernel", stream);
    encode_row_kernel<<<dim3((1u << A) / kRowsPerBlock, (unsigned)batch), kEncThreads, 0, stream>>>(k, mid);
    count_launch("encode_col_kernel", stream);
    encode_col_kernel<A><<<dim3(kRowVals / COLS, (unsigned)batch), kEncThreads, 0, stream>>>(k, mid);
}

static int plan(int logn_loc, unsigned char *S)
{
    // first pass (contiguous, gathers the input) at radix 8 when possible, then radix 8 / 4
    int n = 0, rem = logn_loc;
    while (rem > 0) {
        int s = rem >= 3 ? 3 : rem;
        if (rem == 4) s = 2;
        S[n++] = (unsigned char)s;
        rem -= s;
    }
    return n;
}

template <int LOGC>
static int launch_encode(const EncK &k, int batch, size_t smem, cudaStream_t stream)
{
    auto kern = encode_ifft_kernel<LOGC>;
    static bool configured = false;
    if (!configured) {
        LB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 72 * 1024));
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)batch << LOGC);
    cfg.blockDim = dim3(kFftThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1 << LOGC;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    count_launch("encode_ifft_kernel", stream);
    LB_CUDA(cudaLaunchKernelEx(&cfg, kern, k));
    return LB_OK;
}

// values -> plaintexts [batch][size_l][N] in NTT form
// mid: scratch for batch * sparse_slots complex values, or nullptr
int encode(Context *ctx, int size_l, const void *values, int dtype, long value_stride, int n_values, int sparse_slots, int batch,
           double scale, u64 *pt, int *d_status, int skip_ntt, cudaStream_t stream, double *mid)
{
    const HostParams &hp = ctx->hp;
    int logn = 0;
    while ((1 << logn) < sparse_slots) ++logn;
    if ((1 << logn) != sparse_slots || sparse_slots < 2 || (u64)sparse_slots > hp.N / 2) {
        set_error("single value encoding is not available / slot count must be a power of two up to N/2");
        return LB_ERR_INVALID_ARG;
    }
    if (n_values > sparse_slots) { set_error("values_size is too large"); return LB_ERR_INVALID_ARG; }
    int total_bits = 0;
    for (int l = 0; l < size_l; ++l) total_bits += 64 - __builtin_clzll(hp.q[l]);
    // the reference bounds by the bit count of the product; the sum of prime bit counts is within size_l of it
    {
        long double prod = 1.0L;
        for (int l = 0; l < size_l; ++l) prod *= (long double)hp.q[l];
        int e = 0;
        frexpl(prod, &e);
        total_bits = e;
    }
    if (scale <= 0 || ((int)log2(scale) + 1 >= total_bits)) { set_error("scale out of bounds"); return LB_ERR_INVALID_ARG; }
    if (batch <= 0) return LB_OK;
    if ((u64)sparse_slots < hp.N / 2)
        LB_CUDA(cudaMemsetAsync(pt, 0, ((size_t)batch * size_l << hp.logN) * 8, stream));
    EncK k;
    k.values = values;
    k.dtype = dtype;
    k.value_stride = value_stride;
    k.n_values = n_values;
    k.pt = pt;
    k.roots = ctx->d_croots;
    k.group = ctx->d_rot_group;
    k.tw = nullptr;
    k.mc = ctx->d_mc;
    k.logN = hp.logN;
    k.logn = logn;
    if (!ctx->d_ifft_tw[logn]) {
        // one table per slot count, built once and kept with the context; the build is synchronous so that a
        // later encode on another stream never reads a table still being filled
        double2 *tbl = nullptr;
        LB_CUDA(cudaMalloc((void **)&tbl, sizeof(double2) << logn));
        ctx->owned.push_back(tbl);
        count_launch("ifft_twiddle_table_kernel", stream);
        ifft_twiddle_table_kernel<<<(unsigned)(((1u << logn) + 255) / 256), 256, 0, stream>>>(k, tbl);
        LB_CUDA(cudaGetLastError());
        LB_CUDA(cudaStreamSynchronize(stream));
        ctx->d_ifft_tw[logn] = tbl;
    }
    k.tw = ctx->d_ifft_tw[logn];
    k.size_l = size_l;
    k.fix = scale / (double)sparse_slots;
    k.too_large = ldexp(1.0, total_bits - 2);
    k.status = d_status;
    const int logc = logn > kFftLocalLog ? logn - kFftLocalLog : 0;
    const int logn_loc = logn - logc;
    k.npass = plan(logn_loc, k.S);
    const size_t n_loc = size_t(1) << logn_loc;
    const size_t smem = (n_loc + (n_loc >> 4) + 2) * sizeof(cplx);
    int rc = LB_OK;
    if (mid && logn >= 12 && logn <= 15 && batch <= 65535) {
        cplx *m = reinterpret_cast<cplx *>(mid);
        switch (logn) {
        case 12: launch_encode_two<4>(k, batch, m, stream); break;
        case 13: launch_encode_two<5>(k, batch, m, stream); break;
        case 14: launch_encode_two<6>(k, batch, m, stream); break;
        default: launch_encode_two<7>(k, batch, m, stream); break;
        }
        LB_CUDA(cudaGetLastError());
    } else {
        switch (logc) {
        case 0: rc = launch_encode<0>(k, batch, smem, stream); break;
        case 1: rc = launch_encode<1>(k, batch, smem, stream); break;
        case 2: rc = launch_encode<2>(k, batch, smem, stream); break;
        case 3: rc = launch_encode<3>(k, batch, smem, stream); break;
        default: set_error("slot count above 32768 is not supported"); return LB_ERR_INVALID_ARG;
        }
    }
    if (rc) return rc;
    if (skip_ntt) return LB_OK; // coefficient form, for an encryption that folds the plaintext in
    NttJob j;
    j.src = pt;
    j.dst = pt;
    j.n_groups = batch;
    j.per_group = size_l;
    j.size_l = size_l;
    return ntt_forward(ctx, j, stream);
}

// ---- decode -----------------------------------------------------------------------------

constexpr int kMaxComposeLimbs = 32; // the constants travel as a kernel argument (17 KiB at 32 limbs, below the 32 KiB limit)

struct ComposeConst {
    u64 radix[kMaxComposeLimbs][kMaxComposeLimbs + 1]; // q_0 ... q_{r-1} as a multi-word integer
    u64 Q[kMaxComposeLimbs + 1], Qhalf[kMaxComposeLimbs + 1];
    u64 ginv[kMaxComposeLimbs], ginv_s[kMaxComposeLimbs];
    u64 radix_mod[kMaxComposeLimbs][kMaxComposeLimbs]; // (q_0...q_{s-1}) mod q_r
};

// Exact centred CRT composition by Garner's mixed radix, then one conversion to double.
// (The reference accumulates word by word in double, rns_base.cu:325-459; both are within
// an ulp of the true quotient, and decoding is compared by tolerance.)
__global__ void __launch_bounds__(256) compose_kernel(cplx *__restrict__ out, const u64 *__restrict__ coef,
                                                      const ModConst *__restrict__ mc, const ComposeConst cc, const int logN,
                                                      const int logn, const int size_l, const double inv_scale)
{
    const unsigned n = 1u << logn;
    const int ratio_log = (logN - 1) - logn;
    const int W = size_l + 1;
    coef += ((size_t)blockIdx.y * size_l) << logN;
    out += (size_t)blockIdx.y * n;
    for (unsigned id = blockIdx.x * blockDim.x + threadIdx.x; id < 2 * n; id += gridDim.x * blockDim.x) {
        u64 v[kMaxComposeLimbs];
        for (int r = 0; r < size_l; ++r) {
            const ModConst m = mc[r];
            const u64 t = coef[((size_t)r << logN) + ((size_t)id << ratio_log)];
            u64 acc = 0;
            for (int s = 0; s < r; ++s) acc = add_mod(acc, mul_mod(barrett64(v[s], m.q, m.r1), cc.radix_mod[r][s], m), m.q);
            v[r] = shoup_mul(sub_mod(t, acc, m.q), cc.ginv[r], cc.ginv_s[r], m.q);
        }
        u64 x[kMaxComposeLimbs + 1];
        for (int i = 0; i < W; ++i) x[i] = 0;
        for (int r = 0; r < size_l; ++r) {
            u64 carry = 0;
            for (int i = 0; i < W; ++i) {
                u128d t = mul_wide(cc.radix[r][i], v[r]);
                t.lo += x[i];
                t.hi += t.lo < x[i];
                t.lo += carry;
                t.hi += t.lo < carry;
                x[i] = t.lo;
                carry = t.hi;
            }
        }
        bool gt = false, decided = false;
        for (int i = W - 1; i >= 0 && !decided; --i)
            if (x[i] != cc.Qhalf[i]) { gt = x[i] > cc.Qhalf[i]; decided = true; }
        if (gt) { // x > floor(Q/2): represent x - Q
            u64 borrow = 0;
            for (int i = 0; i < W; ++i) {
                const u64 a = cc.Q[i], b = x[i];
                const u64 d = a - b - borrow;
                borrow = (a < b) || (a == b && borrow);
                x[i] = d;
            }
        }
        // only the non-zero words count: with many limbs 2^(64 i) leaves the range of a double long before the
        // words of a centred coefficient stop being zero, and 0 * inf would poison the sum
        double val = 0.0;
        for (int i = 0; i < W; ++i)
            if (x[i]) val += ldexp((double)x[i], 64 * i);
        if (gt) val = -val;
        val *= inv_scale;
        if (id < n) out[id].x = val;
        else out[id - n].y = val;
    }
}

// The same for the few limbs a decoded ciphertext has in practice (Lancelot's chain: three, and two after the rescale), with
// every word in registers: the general kernel's arrays are indexed at run time and live in local memory.
// 342 messages of three limbs at N = 2^16: 1003 -> 338 us.
constexpr int kSmallLimbs = 4;
template <int L>
struct SmallCompose {
    u64 radix[L][L + 1], Q[L + 1], Qhalf[L + 1];
    u64 ginv[L], ginv_s[L], radix_mod[L][L], radix_mod_s[L][L];
};
template <int L>
__global__ void __launch_bounds__(256) compose_small_kernel(cplx *__restrict__ out, const u64 *__restrict__ coef,
                                                            const ModConst *__restrict__ mc, const __grid_constant__ SmallCompose<L> cc,
                                                            const int logN, const int logn, const double inv_scale)
{
    constexpr int W = L + 1;
    const unsigned n = 1u << logn, id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= 2 * n) return;
    coef += (((size_t)blockIdx.y * L) << logN) + ((size_t)id << (logN - 1 - logn));
    u64 t[L], v[L], x[W];
#pragma unroll
    for (int r = 0; r < L; ++r) t[r] = coef[(size_t)r << logN];
#pragma unroll
    for (int r = 0; r < L; ++r) {
        const u64 q = mc[r].q;
        u64 acc = 0;
#pragma unroll
        for (int s = 0; s < r; ++s) acc = add_mod(acc, shoup_mul(v[s], cc.radix_mod[r][s], cc.radix_mod_s[r][s], q), q);
        v[r] = shoup_mul(sub_mod(t[r], acc, q), cc.ginv[r], cc.ginv_s[r], q);
    }
#pragma unroll
    for (int i = 0; i < W; ++i) x[i] = 0;
#pragma unroll
    for (int r = 0; r < L; ++r) {
        u64 carry = 0;
#pragma unroll
        for (int i = 0; i < W; ++i) {
            if (i > r) { // the radix has r words and a product with it r + 1
                x[i] += carry;
                carry = x[i] < carry;
            } else {
                const u128 p = (u128)cc.radix[r][i] * v[r] + x[i] + carry;
                x[i] = (u64)p;
                carry = (u64)(p >> 64);
            }
        }
    }
    bool gt = false, decided = false;
#pragma unroll
    for (int i = W - 1; i >= 0; --i)
        if (!decided && x[i] != cc.Qhalf[i]) { gt = x[i] > cc.Qhalf[i]; decided = true; }
    if (gt) { // x > floor(Q/2): represent x - Q
        u64 borrow = 0;
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const u64 a = cc.Q[i], b = x[i];
            const u64 d = a - b - borrow;
            borrow = (a < b) || (a == b && borrow);
            x[i] = d;
        }
    }
    double val = 0.0, word = 1.0; // L <= 4 words: 2^256 is far inside the range of a double
#pragma unroll
    for (int i = 0; i < W; ++i) {
        val = __dadd_rn(val, __dmul_rn((double)x[i], word));
        word *= 18446744073709551616.0;
    }
    if (gt) val = -val;
    val *= inv_scale;
    cplx *o = out + (size_t)blockIdx.y * n;
    if (id < n) o[id].x = val;
    else o[id - n].y = val;
}

// twiddle of butterfly group k at stage u of the forward transform: the conjugate of the inverse one (fft.cu:54-182)
LB_D cplx fft_twiddle(const double2 *__restrict__ tw, const double2 *__restrict__ roots, const uint32_t *__restrict__ group, const int logN,
                      const int logn, const unsigned k, const int u)
{
    if (tw) {
        const unsigned n = 1u << logn;
        const double2 w = __ldg(tw + (n - (n >> u)) + k);
        return {w.x, -w.y};
    }
    const unsigned rev = logn > 1 ? (__brev(k << u) >> (33 - logn)) : 0u;
    const double2 w = roots[(group[rev] << (u + logN - 1 - logn)) & ((2u << logN) - 1)];
    return {w.x, w.y};
}

// S consecutive forward stages (spans 2^u .. 2^(u-S+1)) on 2^S values per thread: (x0, x1) <- (x0 + w x1, x0 - w x1).
// Bound by its trips over memory, so a transform of 32768 points takes four of them instead of one per stage and one for
// the order: 342 messages 1024 -> 353 us.  The last pass writes natural order.  There thread t takes group bitrev(t),
// so that neighbouring threads write neighbouring values and read whole 2^S-value rows.
constexpr int kFftPassThreads = 128;
template <int S>
__global__ void __launch_bounds__(kFftPassThreads) fft_pass_kernel(const cplx *in, cplx *out, const double2 *__restrict__ tw,
                                                                   const double2 *__restrict__ roots, const uint32_t *__restrict__ group,
                                                                   const int logN, const int logn, const int u)
{
    constexpr int R = 1 << S;
    const int ul = u - S + 1; // log2 of the smallest span
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >> (logn - S)) return;
    in += (size_t)blockIdx.y << logn;
    out += (size_t)blockIdx.y << logn;
    const unsigned lo = t & ((1u << ul) - 1);
    const unsigned hi = ul > 0 ? t >> ul : logn > S ? __brev(t) >> (32 - (logn - S)) : 0u;
    const unsigned base = (hi << (u + 1)) + lo;
    cplx v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = in[base + ((unsigned)i << ul)];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int half = 1 << (S - 1 - s);
#pragma unroll
        for (int b = 0; b < (1 << s); ++b) {
            const cplx w = fft_twiddle(tw, roots, group, logN, logn, (hi << s) + b, u - s);
#pragma unroll
            for (int i = 0; i < half; ++i) {
                cplx &a0 = v[b * 2 * half + i], &a1 = v[b * 2 * half + i + half];
                const cplx x1 = c_mul(a1, w), x0 = a0;
                a0 = c_add(x0, x1);
                a1 = c_sub(x0, x1);
            }
        }
    }
    if (ul > 0) {
#pragma unroll
        for (int i = 0; i < R; ++i) out[base + ((unsigned)i << ul)] = v[i];
    } else {
#pragma unroll
        for (int i = 0; i < R; ++i) out[((__brev((unsigned)i) >> (32 - S)) << (logn - S)) + t] = v[i];
    }
}

template <int S>
static void launch_fft_pass(const Context *ctx, const cplx *in, cplx *out, int logn, int u, int batch, cudaStream_t stream)
{
    const unsigned threads = 1u << (logn - S);
    count_launch("fft_pass_kernel", stream);
    fft_pass_kernel<S><<<dim3((threads + kFftPassThreads - 1) / kFftPassThreads, batch), kFftPassThreads, 0, stream>>>(
        in, out, ctx->d_ifft_tw[logn], ctx->d_croots, ctx->d_rot_group, ctx->hp.logN, logn, u);
}

template <int L>
static void launch_compose_small(const ComposeConst &cc, const Context *ctx, cplx *buf, const u64 *coef, int logn, int batch, double inv_scale,
                                 cudaStream_t stream)
{
    SmallCompose<L> sc;
    for (int r = 0; r < L; ++r) {
        for (int i = 0; i <= L; ++i) sc.radix[r][i] = cc.radix[r][i];
        for (int s = 0; s < L; ++s) {
            sc.radix_mod[r][s] = cc.radix_mod[r][s];
            sc.radix_mod_s[r][s] = h_shoup(cc.radix_mod[r][s], ctx->hp.q[r]);
        }
        sc.ginv[r] = cc.ginv[r];
        sc.ginv_s[r] = cc.ginv_s[r];
    }
    for (int i = 0; i <= L; ++i) {
        sc.Q[i] = cc.Q[i];
        sc.Qhalf[i] = cc.Qhalf[i];
    }
    compose_small_kernel<L><<<dim3(((2u << logn) + 255) / 256, batch), 256, 0, stream>>>(buf, coef, ctx->d_mc, sc, ctx->hp.logN, logn, inv_scale);
}

size_t decode_workspace_bytes(const Context *ctx, int size_l, int batch)
{
    return (((size_t)size_l << ctx->hp.logN) + ctx->hp.N) * 8 * batch + 256;
}

// plaintext [size_l][N] (NTT form) -> sparse_slots complex doubles on the device
int decode(Context *ctx, int size_l, int batch, const u64 *pt, double scale, int sparse_slots, double *out_complex, cudaStream_t stream)
{
    const HostParams &hp = ctx->hp;
    if (size_l > kMaxComposeLimbs) { set_error("decode supports at most 32 limbs"); return LB_ERR_INVALID_ARG; }
    int logn = 0;
    while ((1 << logn) < sparse_slots) ++logn;
    if ((1 << logn) != sparse_slots || sparse_slots < 2 || (u64)sparse_slots > hp.N / 2) {
        set_error("slot count must be a power of two between 2 and N/2");
        return LB_ERR_INVALID_ARG;
    }
    if (scale <= 0) { set_error("scale out of bounds"); return LB_ERR_INVALID_ARG; }
    int rc = ctx->ensure_workspace(decode_workspace_bytes(ctx, size_l, batch));
    if (rc) return rc;
    u64 *coef = reinterpret_cast<u64 *>(ctx->ws);
    cplx *buf = reinterpret_cast<cplx *>(coef + (((size_t)size_l * batch) << hp.logN));
    NttJob inv;
    inv.src = pt;
    inv.dst = coef;
    inv.n_groups = batch;
    inv.per_group = size_l;
    inv.size_l = size_l;
    if ((rc = ntt_inverse(ctx, inv, stream))) return rc;
    ComposeConst cc;
    memset(&cc, 0, sizeof(cc));
    const int W = size_l + 1;
    u64 Q[kMaxComposeLimbs + 1] = {1};
    for (int r = 0; r < size_l; ++r) {
        for (int i = 0; i < W; ++i) cc.radix[r][i] = Q[i];
        u64 carry = 0;
        for (int i = 0; i < W; ++i) {
            const u128 t = (u128)Q[i] * hp.q[r] + carry;
            Q[i] = (u64)t;
            carry = (u64)(t >> 64);
        }
        u64 radix = 1;
        for (int s = 0; s < r; ++s) {
            cc.radix_mod[r][s] = radix;
            radix = h_mulmod(radix, hp.q[s] % hp.q[r], hp.q[r]);
        }
        cc.ginv[r] = h_invmod(radix, hp.q[r]);
        cc.ginv_s[r] = h_shoup(cc.ginv[r], hp.q[r]);
    }
    for (int i = 0; i < W; ++i) {
        cc.Q[i] = Q[i];
        cc.Qhalf[i] = (Q[i] >> 1) | (i + 1 < W ? Q[i + 1] << 63 : 0);
    }
    const unsigned n = (unsigned)sparse_slots;
    count_launch("compose_kernel", stream);
    switch (size_l) {
    case 1: launch_compose_small<1>(cc, ctx, buf, coef, logn, batch, 1.0 / scale, stream); break;
    case 2: launch_compose_small<2>(cc, ctx, buf, coef, logn, batch, 1.0 / scale, stream); break;
    case 3: launch_compose_small<3>(cc, ctx, buf, coef, logn, batch, 1.0 / scale, stream); break;
    case kSmallLimbs: launch_compose_small<kSmallLimbs>(cc, ctx, buf, coef, logn, batch, 1.0 / scale, stream); break;
    default: compose_kernel<<<dim3((2 * n + 255) / 256, batch), 256, 0, stream>>>(buf, coef, ctx->d_mc, cc, hp.logN, logn, size_l, 1.0 / scale);
    }
    LB_CUDA(cudaGetLastError());
    // as few passes of at most four stages as possible, evenly
    for (int u = logn - 1, left = (logn + 3) / 4; left > 0; --left) {
        const int S = (u + left) / left;
        cplx *dst = left == 1 ? reinterpret_cast<cplx *>(out_complex) : buf;
        switch (S) {
        case 4: launch_fft_pass<4>(ctx, buf, dst, logn, u, batch, stream); break;
        case 3: launch_fft_pass<3>(ctx, buf, dst, logn, u, batch, stream); break;
        case 2: launch_fft_pass<2>(ctx, buf, dst, logn, u, batch, stream); break;
        default: launch_fft_pass<1>(ctx, buf, dst, logn, u, batch, stream); break;
        }
        u -= S;
    }
    LB_CUDA(cudaGetLastError());
    return LB_OK;
}

} // namespace lb
