// finalize.cu -- pair histograms as doubles: the last kernel of every pair count (in
// a file of its own, so that it does not load a pair kernel's module).
#include "pcf_internal.cuh"

namespace {

// A bin of k_pairs_lean's weighted sums: 128-bit whole numbers, low and high.
__device__ __forceinline__ double exact_sum(unsigned long long lo, double hi) {
    return (double)(unsigned long long)__double_as_longlong(hi) * 0x1p64 + (double)lo;
}

// How a histogram arrives: u64 counts, FP64 sums, or exact sums (whose scale the
// caller's multiplier includes).
enum { SUM_COUNTS = 0, SUM_FP64 = 1, SUM_EXACT = 2 };

// Several histograms: out[s*nb + k] = mult[s] * hist[s*nb + k].
__global__ void k_finalize_slots(const unsigned long long *__restrict__ cnt,
                                 const double *__restrict__ ws, int weighted,
                                 const double *__restrict__ mult, int nb, int nslots,
                                 double *__restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nb * nslots) return;
    const int s = (int)(t / nb);
    out[t] = mult[s] * (weighted == SUM_EXACT ? exact_sum(cnt[t], ws[t]) : weighted ? ws[t] : (double)cnt[t]);
}

// out[k] = mult * hist[k] (u64 counts or FP64 sums); with host_stats, the four
// statistics words too.
__global__ void k_finalize(const unsigned long long *__restrict__ cnt, const double *__restrict__ ws,
                           int weighted, double mult, int nb, double *__restrict__ out,
                           const unsigned long long *__restrict__ stats, unsigned long long *host_stats) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (host_stats && k < 4) host_stats[k] = stats[k];
    if (k >= nb) return;
    double v = weighted == SUM_EXACT ? exact_sum(cnt[k], ws[k]) : weighted ? ws[k] : (double)cnt[k];
    out[k] = mult * v;
}

}  // namespace

static int sum_kind(bool weighted, bool exact) { return !weighted ? SUM_COUNTS : exact ? SUM_EXACT : SUM_FP64; }

cudaError_t launch_finalize_slots(const unsigned long long *d_count, const double *d_wsum,
                                  bool weighted, bool exact, const double *d_mult, int nb, int nslots,
                                  double *d_out, cudaStream_t st) {
    const long long n = (long long)nb * nslots;
    k_finalize_slots<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_count, d_wsum, sum_kind(weighted, exact),
                                                                   d_mult, nb, nslots, d_out);
    return cudaGetLastError();
}

cudaError_t launch_finalize(const unsigned long long *d_count, const double *d_wsum, bool weighted,
                            double mult, int nb, double *d_out, cudaStream_t st) {
    k_finalize<<<(nb + 255) / 256, 256, 0, st>>>(d_count, d_wsum, weighted ? 1 : 0, mult, nb, d_out, nullptr, nullptr);
    return cudaGetLastError();
}

pcf_status finalize_hist(pcf_ctx *ctx, const unsigned long long *d_count, const double *d_wsum,
                         bool weighted, bool exact, double mult, int nb, double *out,
                         const unsigned long long *d_stats, unsigned long long *host_stats) {
    k_finalize<<<(nb + 255) / 256, 256, 0, ctx->stream>>>(d_count, d_wsum, sum_kind(weighted, exact), mult,
                                                          nb, out, d_stats, host_stats);
    PCF_CU(ctx, cudaGetLastError());
    ++ctx->launches;
    return PCF_OK;
}
