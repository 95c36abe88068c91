// pairs_common.cuh -- what the pair kernels share: launch arguments, candidate
// ranges, the FP64 rule of one pair, ticket shapes.  Included by pairs.cu (the
// general kernel) and pairs_lean.cuh (the branch-free one, which has source files of
// its own for unit and for weighted counts).
#pragma once
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <type_traits>

#include "pcf_internal.cuh"

constexpr int kChunkMax = 8;            // work items per ticket, at most
constexpr int kLeanWideBins = 120;      // bins up to which k_pairs_lean reads out 16 fraction bits

// Fast-path cut constants for one range type (0: unshifted, 1: image-shifted).
struct FastCuts {
    float dsf;        // (float)ds
    float ds2;        // dsf * dsf
    float lo[2];      // d2 below lo (and >= tiny) is safely inside dmax
    float hi[2];      // d2 at or above hi is safely outside dmax
    unsigned w[2];    // edge window in 2^-15 units of r
    // k_pairs_lean: the edge window in units of its readout, dmax included; 0
    // where it does not apply (see make_cuts)
    unsigned wl[2];
    float tiny;
};

struct PairArgs {
    const PairJob *jobs;  // histograms of this launch, items laid out job after job
    int n_jobs;
    long long n_items;
    unsigned long long *counter;  // work tickets handed out so far
    long long n_chunked;          // items [0, n_chunked) go out `kchunk` per ticket,
    long long t_chunked;          // in t_chunked tickets; later tickets: one item each
    int kchunk;
    float box;
    int bpc;
    float zreach;  // dmax * (1 + 1e-5): the z reach of a home tile's rows
    PairRule rule;
    FastCuts fc;
    unsigned long long *g_count;
    double *g_wsum;
    unsigned long long *g_stats;
    int chunk;   // candidates per budget check (even)
    int budget;  // adds one shared counter absorbs between flushes
    int fast;    // 0: every pair in range takes the FP64 rule (bins > 255: r + 256
                 // no longer has a fixed exponent)
    const unsigned *ctrl;  // abort request polled at every ticket (null: none)
    unsigned *status;      // where a warp that gives up records why (null: none)
    long long max_tickets; // iteration cap: tickets one warp may take
};

namespace {

constexpr unsigned kFull = 0xffffffffu;

// Kinds of one launch: the isotropic histogram, the anisotropic one, or both
// from one pass over the candidates (the anisotropic stencil covers the
// isotropic one).
enum { K_ISO = 0, K_ANI = 1, K_BOTH = 2 };

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Shared reductions on 32-bit shared-window addresses.  They are not
// predicated: a lane without a pair adds 0 to a private dummy slot, which
// keeps the candidate loop free of branches around memory operations.
__device__ __forceinline__ void red_s_u32(unsigned a, unsigned v) {
    asm volatile("red.shared.add.u32 [%0], %1;" :: "r"(a), "r"(v));
}

// Point j of a pair-packed view.
__device__ __forceinline__ void load_point(const float4 *pk, int j, float &x, float &y, float &z, float &w) {
    const float4 a = __ldg(pk + (j & ~1)), b = __ldg(pk + (j & ~1) + 1);
    const bool o = j & 1;
    x = o ? a.y : a.x;
    y = o ? a.w : a.z;
    z = o ? b.y : b.x;
    w = o ? b.w : b.z;
}

// Canonical FP64 decision for one pair (rare path): histogram slot or -1.
template <bool ANI>
__device__ __noinline__ int slow_slot(float hx, float hy, float hz, float cx, float cy, float cz,
                                      float sx, float sy, float sz, PairRule rule) {
    double dx, dy, dz;
    exact_sep(hx, hy, hz, cx, cy, cz, sx, sy, sz, dx, dy, dz);
    return exact_slot<ANI>(dx, dy, dz, rule);
}

// Candidate ranges of one stencil row for the current home tile: [a0, b0)
// unshifted in z, [a1, b1) image-shifted by sz1 (periodic wrap in z); the
// column's image shift is (sx, sy).  kind 1: forward half of the home column.
struct RowRange {
    int a0, b0, a1, b1;
    float sx, sy, sz1;
    int kind;
};

// The candidate ranges of stencil row rw for home tile t of job J, whose
// points lie in [zmn, zmx].
__device__ __forceinline__ RowRange row_range(const PairArgs &A, const PairJob &J, const RowDesc rw, const TileDesc &t,
                                              float zmn, float zmx) {
    RowRange rr{0, 0, 0, 0, 0.f, 0.f, 0.f, 0};
    int nx = t.ix + rw.dx, ny = t.iy + rw.dy;
    const int P = J.P;
    bool ok = true;
    if (A.bpc) {
        if (nx < 0) { nx += P; rr.sx = -A.box; } else if (nx >= P) { nx -= P; rr.sx = A.box; }
        if (ny < 0) { ny += P; rr.sy = -A.box; } else if (ny >= P) { ny -= P; rr.sy = A.box; }
    } else if (nx < 0 || nx >= P || ny < 0 || ny >= P) {
        ok = false;
    }
    if (ok) {
        const int col = (nx * P + ny) * P;
        // the row's cells, clipped to those the home points reach in z:
        // a candidate within dmax of a home point has z in (zmn - dmax,
        // zmx + dmax), so its cell lies in [zcut_lo, zcut_hi] (with
        // 1e-3 of a cell to spare for the rounding of z / cell here
        // and in the grid build; the tile's own cells always stay);
        // periodic images follow the same cell arithmetic past 0 and P
        const float rcell = (float)P / A.box;
        const int zcut_lo = min((int)floorf((zmn - A.zreach) * rcell - 1e-3f), (int)t.z0);
        const int zcut_hi = max((int)floorf((zmx + A.zreach) * rcell + 1e-3f), (int)t.z1);
        const int zhi = min(t.z1 + rw.kz, zcut_hi);
        rr.kind = rw.kind;
        const int *cs = J.cand.cstart;
        if (rw.kind == 1) {  // forward half of the home column (XX): j > home index
            rr.a0 = t.start;
            rr.b0 = cs[col + min(zhi, P - 1) + 1];
            if (A.bpc && zhi >= P) { rr.a1 = cs[col]; rr.b1 = cs[col + zhi - P + 1]; rr.sz1 = A.box; }
        } else {
            const int zlo = max(t.z0 - rw.kz, zcut_lo);
            rr.a0 = cs[col + max(zlo, 0)];
            rr.b0 = cs[col + min(zhi, P - 1) + 1];
            if (A.bpc) {
                if (zlo < 0) { rr.a1 = cs[col + zlo + P]; rr.b1 = cs[col + P]; rr.sz1 = -A.box; }
                else if (zhi >= P) { rr.a1 = cs[col]; rr.b1 = cs[col + zhi - P + 1]; rr.sz1 = A.box; }
            }
        }
    }
    return rr;
}

}  // namespace

// The ticket shape of a launch of `warps` warps: runs of k items per ticket
// while a queue holds >= 32 runs per warp (k at most 8, or the tuned cap that
// A.kchunk carries in).
static PairArgs with_tickets(const PairArgs &A, long long n_items, long long warps) {
    PairArgs B = A;
    const long long cap = A.kchunk > 0 ? std::min<long long>(A.kchunk, kChunkMax) : kChunkMax;
    B.kchunk = (int)std::max(1LL, std::min<long long>(cap, n_items / (warps * 32)));
    B.n_chunked = B.kchunk > 1 ? std::max(0LL, n_items - 2 * warps) : 0;
    B.t_chunked = (B.n_chunked + B.kchunk - 1) / B.kchunk;
    // a warp can take at most every ticket of the queue plus the one that
    // finds it empty
    B.max_tickets = B.t_chunked + (n_items - B.n_chunked) + 2;
    return B;
}

// CTAs of `kfn` per SM (occupancy queries cost microseconds: cached per device
// and shared-memory size, under a lock, as several host threads launch).
struct OccCache {
    std::mutex mu;
    std::map<std::pair<int, size_t>, int> per_sm;
    cudaError_t get(const void *kfn, int threads, int device, size_t smem, int *out) {
        std::lock_guard<std::mutex> lk(mu);
        auto it = per_sm.find({device, smem});
        if (it == per_sm.end()) {
            int per = 0;
            const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kfn, threads, smem);
            if (e != cudaSuccess) return e;
            it = per_sm.insert({{device, smem}, std::max(1, per)}).first;
        }
        *out = it->second;
        return cudaSuccess;
    }
};
