// Diagnostics for benchmarks (include/lancelot_b200_diag.h): launch counter, per-kernel device
// times of whatever the library launches while the timer is on, and the register-only butterfly
// rate probe.  Nothing here is on the compute path; with the timer off a launch costs one
// counter increment.
#include <cstdio>
#include <cstring>
#include <mutex>

#include "../../include/lancelot_b200_diag.h"
#include "context.h"
#include "ntt_stages.cuh"

namespace lb {

// the column kernels' launch shape (ntt_twopass.cuh): the probe runs at their occupancy
constexpr int kProbeThreads = 256;
constexpr int kProbeBlocks = 3;

static unsigned long long g_launches = 0;
unsigned long long launch_count() { return g_launches; }

// ---- kernel timer ---------------------------------------------------------------------------
// While enabled, an event is recorded on the launching stream in front of every kernel of this
// library.  A kernel's time is the span to the next event on the same stream (the next launch, or
// the closing event the report records), so copies and idle gaps between two launches count towards
// the first.  One stream at a time is timed correctly: a launch on another stream closes the
// current span with an event on the previous stream.
constexpr int kMaxMarks = 1 << 15;
struct Mark {
    const char *name;
    cudaEvent_t ev;
    cudaStream_t stream;
    double bytes;
};
static std::mutex g_diag_mu;
static bool g_timing = false;
static std::vector<cudaEvent_t> g_pool;
static std::vector<Mark> g_marks;
static bool g_overflow = false;

void count_launch(const char *name, cudaStream_t stream, double bytes)
{
    ++g_launches;
    if (!g_timing) return;
    std::lock_guard<std::mutex> lock(g_diag_mu);
    if ((int)g_marks.size() >= kMaxMarks) {
        g_overflow = true;
        return;
    }
    cudaEvent_t ev;
    if (g_marks.size() < g_pool.size()) {
        ev = g_pool[g_marks.size()];
    } else {
        if (cudaEventCreate(&ev) != cudaSuccess) return;
        g_pool.push_back(ev);
    }
    cudaEventRecord(ev, stream);
    g_marks.push_back(Mark{name ? name : "other", ev, stream, bytes});
}

// ---- arithmetic ceiling probe -------------------------------------------------------------------
// The four forward stages a thread of the two-kernel transforms takes at a time, with the reduction behind them, on registers only
// but for twiddles from a table that stays in L1, at the column kernels' occupancy.  Its rate is the ceiling the modular arithmetic
// of a prime class sets for these transforms on this GPU; one limb of N points needs (N/2) log2 N butterflies.
constexpr int kProbeTwiddles = 16 * 16;
template <int M>
__global__ void __launch_bounds__(kProbeThreads, kProbeBlocks) butterfly_probe_kernel(u64 *out, const u64 q, const ulonglong2 *tw,
                                                                                      const int iters)
{
    const TpPrime p = tp_prime<M>(q);
    u64 v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = tp_load<M>((u64)threadIdx.x * 16 + i + blockIdx.x);
    for (int it = 0; it < iters; ++it) {
        const ulonglong2 *t = tw + (it & 15) * 16; // others each time, so that nothing is hoisted out of the loop
        tp_fwd<4, M>(v, p, [&](const int u, const int b) { return __ldg(t + (1 << u) - 1 + b); });
        tp_settle<M>(v, p); // nothing for primes below 2^47: the 3000 q their values grow to here stay finite
    }
    u64 acc = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) acc ^= v[i];
    out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = acc;
}

// variant: 0 near 2^60, 1 the other integers, 2 all on the FP64 pipe at a 50-bit prime, 3 the same at a 40-bit prime,
// -1 the one the context's first prime takes.
int probe_butterfly_rate(Context *ctx, int variant, double *butterflies_per_second)
{
    static const int mode_of[4] = {kTpNear, kTpStrict, kTpF64Tight, kTpF64};
    if (variant > 3) {
        set_error("butterfly variant must be 0..3 or -1");
        return LB_ERR_INVALID_ARG;
    }
    for (int v = 0; variant < 0 && v < 4; ++v)
        if (mode_of[v] == tp_fwd_mode(ctx->hp.q[0])) variant = v;
    const int blocks = ctx->sm_count * kProbeBlocks, iters = 1000;
    int rc = ctx->ensure_workspace(kProbeTwiddles * sizeof(ulonglong2) + (size_t)blocks * kProbeThreads * sizeof(u64));
    if (rc) return rc;
    ulonglong2 *tw = reinterpret_cast<ulonglong2 *>(ctx->ws);
    u64 *out = reinterpret_cast<u64 *>(tw + kProbeTwiddles);
    // any odd modulus of the variant's size gives the variant's instruction stream
    static const u64 modulus_of[4] = {(u64(1) << 60) - 93, (u64(1) << 57) - 13, (u64(1) << 50) - 27, (u64(1) << 40) - 87};
    const u64 q = modulus_of[variant];
    ulonglong2 table[kProbeTwiddles];
    for (int i = 0; i < kProbeTwiddles; ++i) {
        const u64 w = (u64(0x9E3779B97F4A7C15) * (i + 1)) % q;
        table[i] = make_ulonglong2(h_twiddle_value(w, q), h_twiddle_quot(w, q));
    }
    LB_CUDA(cudaMemcpy(tw, table, sizeof(table), cudaMemcpyHostToDevice));
    cudaEvent_t e0, e1;
    LB_CUDA(cudaEventCreate(&e0));
    LB_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    for (int rep = 0; rep < 4; ++rep) {
        LB_CUDA(cudaEventRecord(e0, 0));
        count_launch("butterfly_probe_kernel", nullptr);
        switch (mode_of[variant]) {
        case kTpNear: butterfly_probe_kernel<kTpNear><<<blocks, kProbeThreads>>>(out, q, tw, iters); break;
        case kTpStrict: butterfly_probe_kernel<kTpStrict><<<blocks, kProbeThreads>>>(out, q, tw, iters); break;
        case kTpF64Tight: butterfly_probe_kernel<kTpF64Tight><<<blocks, kProbeThreads>>>(out, q, tw, iters); break;
        default: butterfly_probe_kernel<kTpF64><<<blocks, kProbeThreads>>>(out, q, tw, iters); break;
        }
        LB_CUDA(cudaGetLastError());
        LB_CUDA(cudaEventRecord(e1, 0));
        LB_CUDA(cudaEventSynchronize(e1));
        float ms = 0;
        LB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (rep > 0 && ms < best) best = ms;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *butterflies_per_second = (double)blocks * kProbeThreads * iters * 32.0 / (best * 1e-3);
    return LB_OK;
}

} // namespace lb

using namespace lb;

extern "C" {

unsigned long long lb_launch_count(void) { return launch_count(); }

int lb_diag_kernel_timing(int enable)
{
    std::lock_guard<std::mutex> lock(g_diag_mu);
    g_marks.clear();
    g_overflow = false;
    g_timing = enable != 0;
    return LB_OK;
}

int lb_diag_kernel_report(char *buf, size_t capacity)
{
    std::lock_guard<std::mutex> lock(g_diag_mu);
    if (!buf || capacity < 64) {
        set_error("report buffer is too small");
        return LB_ERR_INVALID_ARG;
    }
    struct Row {
        const char *name;
        long launches;
        double ms, bytes;
    };
    std::vector<Row> rows;
    if (!g_marks.empty()) {
        cudaEvent_t last;
        LB_CUDA(cudaEventCreateWithFlags(&last, cudaEventDefault));
        LB_CUDA(cudaEventRecord(last, g_marks.back().stream));
        LB_CUDA(cudaEventSynchronize(last));
        for (size_t i = 0; i < g_marks.size(); ++i) {
            cudaEvent_t end = i + 1 < g_marks.size() ? g_marks[i + 1].ev : last;
            float ms = 0.f;
            if (cudaEventElapsedTime(&ms, g_marks[i].ev, end) != cudaSuccess) {
                (void)cudaGetLastError();
                ms = 0.f;
            }
            size_t r = 0;
            while (r < rows.size() && std::strcmp(rows[r].name, g_marks[i].name)) ++r;
            if (r == rows.size()) rows.push_back(Row{g_marks[i].name, 0, 0.0, 0.0});
            rows[r].launches += 1;
            rows[r].ms += ms;
            rows[r].bytes += g_marks[i].bytes;
        }
        cudaEventDestroy(last);
    }
    size_t off = 0;
    auto put = [&](const char *fmt, auto... a) {
        if (off < capacity) {
            int n = std::snprintf(buf + off, capacity - off, fmt, a...);
            if (n > 0) off += (size_t)n;
        }
    };
    put("{");
    for (size_t r = 0; r < rows.size(); ++r)
        put("%s\"%s\": {\"launches\": %ld, \"ms\": %.4f, \"bytes\": %.0f}", r ? ", " : "", rows[r].name, rows[r].launches, rows[r].ms,
            rows[r].bytes);
    put("%s\"_overflow\": %s}", rows.empty() ? "" : ", ", g_overflow ? "true" : "false");
    g_marks.clear();
    if (off >= capacity) {
        set_error("report buffer is too small");
        return LB_ERR_INVALID_ARG;
    }
    return LB_OK;
}

int lb_probe_butterfly_rate(lb_context *h, int variant, double *butterflies_per_second)
{
    Context *c = lb_context_impl(h);
    if (!c || !butterflies_per_second) {
        set_error("context or destination is null");
        return LB_ERR_INVALID_ARG;
    }
    LB_CUDA(cudaSetDevice(c->device));
    return probe_butterfly_rate(c, variant, butterflies_per_second);
}

} // extern "C"
