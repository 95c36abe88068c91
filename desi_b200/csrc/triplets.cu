// triplets.cu -- isotropic triplet histograms DDD / RRR / DDR / DRR on the
// CUDA cores.
//
// Reference kernels replaced: XXX3iso / XXY3iso (cuda/kernels/3iso_k.cuh:8,94)
// and the periodic count123 / count123_mixed / XXX3iso_BPC / XXY3iso_BPC
// (cuda/kernels/3isoBPC_k.cuh:8,98,191,940), which run one thread per cell
// *triple* with a global FP64 atomic per triangle and spell out 64 image
// combinations.  Here:
//
//  * A group of warps of a persistent CTA takes one anchor point i at a time.  It
//    lists the point ranges of the anchor's neighbour rows (the pair stencil,
//    periodic images by index wrap), walks the candidates of all of them at
//    full width, and compacts into shared memory the X neighbours j > i (list J)
//    and, for XXY, all Y neighbours (list K), each with its FP32 image
//    displacement from i (in bins) and its exact side bin (FP32 fast path +
//    FP64 recheck, as in the pair kernel).
//  * It then runs the pairs of that list: XXX pairs (j < k) of J, XXY all of
//    J x K.  The third side is |v_k - v_j| -- the consistent embedding of
//    count123 (3isoBPC_k.cuh:56-75) -- tested and binned in FP32 with the
//    same edge-window recheck.  Each unordered XXX triangle is seen once (i
//    its lowest index), each unordered XX pair of an XXY triangle once.
//  * Counts go to a shared u32 histogram (one orientation per triangle), exact
//    weight products to one of three limbs per counter; the finalize pass symmetrises it into the reference's ordered-triple
//    histogram: XXX sums the 6 axis permutations, XXY the two orders of the
//    XX pair (b_jk <-> b_ki).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

#include "pcf_internal.cuh"
#include "node_gates.cuh"

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kTThreads = 768;  // 24 warps, one CTA per SM (16 warps left 30% of issue slots empty, 24 leave 20%)
constexpr int kTWarps = kTThreads / 32;
constexpr float kMagic = 256.0f;
constexpr int kFracBits = 15;
constexpr unsigned kFracMask = (1u << kFracBits) - 1u;
struct TripCuts {
    float dsf, ds2;
    float lo, hi;    // d2 window around dd (image-aware bound for periodic boxes)
    float lo3, hi3;  // the same in bins^2 (third sides: list entries are in bins)
    unsigned w;      // edge window, 2^-15 units of r
    // tiles (tri_tiles): the window in 2^-16 units with the distance from dmax
    // to the last bin edge, where that is small (far = 0); else the window
    // around dmax as values of r + 128 + w
    unsigned wt;
    int far;
    float qlo, qhi;
};

struct Cat {
    const float *x, *y, *z, *w;
    const int *cstart;
};

struct TripArgs {
    Cat X, Y;
    int nX;
    const RowDesc *rows;
    int n_rows;
    int P;
    float cell;
    float box;
    int bpc;
    PairRule rXX, rXY;  // side rules (X-X side, X-Y sides)
    TripCuts fc;
    int capJ, capK;          // shared-memory list capacities (entries)
    float4 *gJ, *gK;         // per-CTA overflow lists in global memory
    float *gwJ, *gwK;        // weights of the overflow lists
    int gcap;                // entries per CTA in the overflow lists
    unsigned long long *counter;
    unsigned long long *g_count;  // bins^3 (unit weights)
    double *g_wsum;               // bins^3 (weighted)
    int hist_in_smem;
    // weighted: the catalogs' weights are exact integers q (Cat::w holds their
    // bits), w_i w_j w_k = q_i q_j q_k * wunscale
    int wfix;
    double wunscale;
    int list_bytes;          // shared memory of a group's lists
    unsigned long long *g_stats;
    // adds the shared u32 histogram absorbs between flushes into g_count
    // (a counter then never wraps: one slot gets at most that many adds)
    unsigned long long flush_budget;
    const unsigned *ctrl;  // abort request, polled with every anchor (null: none)
    unsigned *status;      // where a CTA that gives up records why (null: none)
    int mixed;  // XXY
    GateGeom gate;  // the reference's node grid (PCF_REF_NODE_GATES)
};

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ bool fix_safe(unsigned q, unsigned w) {
    return ((q + w) & kFracMask) >= 2u * w;
}

// Exact FP64 side between two catalog points (minimum image when periodic),
// returned as components.
__device__ __forceinline__ void sep_exact(float ax, float ay, float az, float bx, float by,
                                          float bz, int bpc, double L, double &dx, double &dy,
                                          double &dz) {
    dx = __dsub_rn((double)bx, (double)ax);
    dy = __dsub_rn((double)by, (double)ay);
    dz = __dsub_rn((double)bz, (double)az);
    if (bpc) {
        const double h = 0.5 * L;
        if (dx > h) dx = __dsub_rn(dx, L); else if (dx < -h) dx = __dadd_rn(dx, L);
        if (dy > h) dy = __dsub_rn(dy, L); else if (dy < -h) dy = __dadd_rn(dy, L);
        if (dz > h) dz = __dsub_rn(dz, L); else if (dz < -h) dz = __dadd_rn(dz, L);
    }
}

// Side bin of the anchor -> candidate pair in the canonical FP64 rule.
__device__ __noinline__ int exact_side(float ax, float ay, float az, float bx, float by, float bz,
                                       int bpc, float box, PairRule rule) {
    double dx, dy, dz;
    sep_exact(ax, ay, az, bx, by, bz, bpc, (double)box, dx, dy, dz);
    return exact_slot<false>(dx, dy, dz, rule);
}

// Bin of side j-k in the consistent embedding anchored at i: v_jk = v_ik - v_ij.
__device__ __noinline__ int exact_third(float ix, float iy, float iz, float jx, float jy, float jz,
                                        float kx, float ky, float kz, int bpc, float box,
                                        PairRule rule) {
    double ax, ay, az, bx, by, bz;
    sep_exact(ix, iy, iz, jx, jy, jz, bpc, (double)box, ax, ay, az);
    sep_exact(ix, iy, iz, kx, ky, kz, bpc, (double)box, bx, by, bz);
    return exact_slot<false>(__dsub_rn(bx, ax), __dsub_rn(by, ay), __dsub_rn(bz, az), rule);
}

// FP32 fast-path bin of a squared distance, or -1 (recheck needed), -2 (out).
__device__ __forceinline__ int fast_bin(float d2, const TripCuts &c, int bins) {
    if (!(d2 < c.hi)) return -2;
    const float r = sqrt_approx(d2 * c.ds2);
    const unsigned q = __float_as_uint(r + kMagic) & 0x7FFFFFu;
    if (d2 < c.lo && fix_safe(q, c.w)) return min((int)(q >> kFracBits), bins - 1);
    return -1;
}

// The same for a third side, from the squared difference of two list entries
// (in bins^2).
__device__ __forceinline__ int fast_bin3(float r2, const TripCuts &c, int bins) {
    if (!(r2 < c.hi3)) return -2;
    const unsigned q = __float_as_uint(sqrt_approx(r2) + kMagic) & 0x7FFFFFu;
    if (r2 < c.lo3 && fix_safe(q, c.w)) return min((int)(q >> kFracBits), bins - 1);
    return -1;
}

// Angle bin of the anisotropic 3-point histograms for the side anchor->point:
// t = (int)((1 + dz/d) * (float)(bins/2)) (3ani_k.cuh:79-91), dz signed, or
// with periodic boxes dz = |z2-z1| - L*f (3aniBPC_k.cuh:57,73); -1 when >= bins.
__device__ __noinline__ int exact_angle(float ax, float ay, float az, float bx, float by, float bz,
                                        int bpc, float box, int bins, float ds_th) {
    double dx, dy, dz;
    sep_exact(ax, ay, az, bx, by, bz, bpc, (double)box, dx, dy, dz);
    const double d = __dsqrt_rn(exact_d2(dx, dy, dz));
    double dzr = dz;
    if (bpc) {
        const double raw = fabs(__dsub_rn((double)bz, (double)az));
        dzr = raw > 0.5 * (double)box ? __dsub_rn(raw, (double)box) : raw;
    }
    const double c = __dadd_rn(1.0, __ddiv_rn(dzr, d));
    const int t = (int)__dmul_rn(c, (double)ds_th);
    return (t >= 0 && t < bins) ? t : -1;
}

// The candidate ranges of an anchor's stencil rows, two per row (a periodic
// row may wrap in z): first point with the image shifts (2 bits per axis
// above bit 24: 0 -L, 1 none, 2 +L) and the number of candidates before it.
//
// The list builds and the counting of an anchor run in a group of NW warps, of
// which a CTA holds one or more, each with anchors of its own: lane, warp and
// thread numbers below are the group's, gsync its barrier.
constexpr int kGroupWarps = 8;  // of a group, where a CTA or an SM holds several
template <int NW>
struct SegTable {
    int first[NW * 32], before[NW * 32];
    int wsum[NW];
};
template <int NW>
__device__ __forceinline__ int group_tid() { return (int)(threadIdx.x % (NW * 32)); }
template <int NW>
__device__ __forceinline__ void gsync() {
    if (NW == kTWarps) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + threadIdx.x / (NW * 32)), "n"(NW * 32) : "memory");
}

// Ranges of rows [rb, rb + NW * 16), one per thread, in catalog C around the
// anchor's cell; only_after >= 0 keeps the points after that index.  Returns
// the number of candidates.  Called by the whole group; ends synchronised, and
// needs no barrier before it (the table is written after its first barrier).
template <int NW>
__device__ __forceinline__ int seg_table(const TripArgs &A, const Cat &C, int cix, int ciy, int ciz,
                                         int only_after, int rb, SegTable<NW> &T) {
    const int tid = group_tid<NW>(), lane = tid & 31, warp = tid >> 5;
    const int r = rb + (tid >> 1), P = A.P;
    int a = 0, len = 0;
    if (r < A.n_rows) {
        const RowDesc rw = A.rows[r];
        int nx = cix + rw.dx, ny = ciy + rw.dy, ix = 1, iy = 1, iz = 1;
        bool ok = true;
        if (A.bpc) {
            if (nx < 0) { nx += P; ix = 0; } else if (nx >= P) { nx -= P; ix = 2; }
            if (ny < 0) { ny += P; iy = 0; } else if (ny >= P) { ny -= P; iy = 2; }
        } else {
            ok = nx >= 0 && nx < P && ny >= 0 && ny < P;
        }
        if (ok) {
            const int col = (nx * P + ny) * P;
            int zlo = ciz - rw.kz, zhi = ciz + rw.kz;
            if (tid & 1) {  // the part past the box's z face, through its image
                ok = A.bpc && (zlo < 0 || zhi >= P);
                iz = zlo < 0 ? 0 : 2;
                if (zlo < 0) { zlo += P; zhi = P - 1; } else { zlo = 0; zhi -= P; }
            } else {
                zlo = max(zlo, 0);
                zhi = min(zhi, P - 1);
            }
            if (ok) {
                a = C.cstart[col + zlo];
                const int b = C.cstart[col + zhi + 1];
                if (only_after >= 0) a = max(a, only_after + 1);
                len = max(b - a, 0);
                a |= (ix | (iy << 2) | (iz << 4)) << 24;
            }
        }
    }
    int x = len;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) T.wsum[warp] = x;
    gsync<NW>();
    const int ws = lane < NW ? T.wsum[lane] : 0;
    int w = ws;
    #pragma unroll
    for (int o = 1; o < NW; o <<= 1) {
        const int y = __shfl_up_sync(kFull, w, o);
        if (lane >= o) w += y;
    }
    const int total = __shfl_sync(kFull, w, NW - 1);
    T.first[tid] = a;
    T.before[tid] = x - len + __shfl_sync(kFull, w - ws, warp);
    gsync<NW>();
    return total;
}

// Scratch of a group's list builds.
template <int NW>
struct ListScratch {
    SegTable<NW> seg;
    int kept[2][NW];  // entries of each warp's chunk, alternating rounds
};

// Lists the neighbours of anchor (hx,hy,hz) found in catalog C, in the order of
// the stencil's cells, and returns their number; entries past cap are not
// written.  Entries: {dx, dy, dz in bins, bits(idx << 8 | bin)}.  ang: their
// angle bins (ANG).  ginfo (PCF_REF_NODE_GATES): per entry, its node on the
// reference's grid and the axes of its image relative to the anchor
// (gate_pack).  WRAPPED: only the neighbours through an image.  Called by the
// whole CTA; ends synchronised.
//
// All rows' candidates form one index space that the group takes NW * 32 at a time
// (the range of an index by binary search): a row holds 10 to 100 candidates,
// so a loop over rows kept 1 to 3 warps busy and cost a dependent
// cell-table load per row.  The order is kept (a barrier per round) so that
// runs of entries stay close in space, for the culling of tri_tiles.
template <int NW, bool ANG, bool WRAPPED = false>
__device__ int build_list(const TripArgs &A, const Cat &C, float hx, float hy, float hz, int cix, int ciy,
                          int ciz, int only_after, const PairRule &rule, float4 *list, float *wlist, int cap,
                          unsigned &n_rechk, ListScratch<NW> &S, unsigned char *ang = nullptr,
                          unsigned *ginfo = nullptr) {
    const int tid = group_tid<NW>(), lane = tid & 31, warp = tid >> 5;
    int n = 0, par = 0;
    for (int rb = 0; rb < A.n_rows; rb += NW * 16) {
        const int total = seg_table<NW>(A, C, cix, ciy, ciz, only_after, rb, S.seg);
        const int nseg = 2 * min(NW * 16, A.n_rows - rb);
        const int top = 1 << (31 - __clz(nseg));
        // candidate of index q: its point, or -1 past the end; image axes in sh
        auto locate = [&](int q, int &sh) -> int {
            if (q >= total) return -1;
            int s = 0;
            for (int o = top; o > 0; o >>= 1)
                if (s + o < nseg && S.seg.before[s + o] <= q) s += o;
            const int f = S.seg.first[s];
            sh = f >> 24;
            return (f & 0xFFFFFF) + q - S.seg.before[s];
        };
        int sh = 0, c = locate(tid, sh);
        float px = 0.f, py = 0.f, pz = 0.f;
        if (c >= 0) { px = C.x[c]; py = C.y[c]; pz = C.z[c]; }
        for (int base = 0; base < total; base += NW * 32) {
            // the next round's points are on their way while this one is tested
            int shn = 0;
            const int cn = locate(base + NW * 32 + tid, shn);
            float nx = 0.f, ny = 0.f, nz = 0.f;
            if (cn >= 0) { nx = C.x[cn]; ny = C.y[cn]; nz = C.z[cn]; }
            int bin = -2, tang = 0;
            float vx = 0.f, vy = 0.f, vz = 0.f;
            if (c >= 0 && !(WRAPPED && sh == (1 | (1 << 2) | (1 << 4)))) {
                vx = px - (hx - (float)((sh & 3) - 1) * A.box);
                vy = py - (hy - (float)(((sh >> 2) & 3) - 1) * A.box);
                vz = pz - (hz - (float)((sh >> 4) - 1) * A.box);
                const float d2 = fmaf(vz, vz, fmaf(vy, vy, vx * vx));
                bin = fast_bin(d2, A.fc, rule.bins);
                if (bin == -1) {
                    ++n_rechk;
                    bin = exact_side(hx, hy, hz, px, py, pz, A.bpc, A.box, rule);
                }
                if (ANG && bin >= 0) {
                    tang = exact_angle(hx, hy, hz, px, py, pz, A.bpc, A.box, rule.bins,
                                       (float)rule.bins / 2.0f);
                    if (tang < 0) bin = -2;  // the side can close no triangle
                }
            }
            const bool keep = bin >= 0;
            const unsigned m = __ballot_sync(kFull, keep);
            if (lane == 0) S.kept[par][warp] = __popc(m);
            gsync<NW>();
            const int wk = lane < NW ? S.kept[par][lane] : 0;
            int x = wk;
            #pragma unroll
            for (int o = 1; o < NW; o <<= 1) {
                const int y = __shfl_up_sync(kFull, x, o);
                if (lane >= o) x += y;
            }
            const int pos = n + __shfl_sync(kFull, x - wk, warp) + __popc(m & ((1u << lane) - 1u));
            n += __shfl_sync(kFull, x, NW - 1);
            par ^= 1;
            if (keep && pos < cap) {
                list[pos] = make_float4(vx * A.fc.dsf, vy * A.fc.dsf, vz * A.fc.dsf,
                                        __int_as_float((c << 8) | bin));
                if (wlist) wlist[pos] = C.w[c];
                if (ANG) ang[pos] = (unsigned char)tang;
                if (ginfo)
                    ginfo[pos] = gate_pack(A.gate, px, py, pz,
                                           ((sh & 3) != 1 ? 1u : 0u) | (((sh >> 2) & 3) != 1 ? 2u : 0u) |
                                               ((sh >> 4) != 1 ? 4u : 0u));
            }
            c = cn;
            sh = shn;
            px = nx;
            py = ny;
            pz = nz;
        }
    }
    gsync<NW>();
    return n;
}

// The shared histogram U of the unit-weight counts: bins^2 rows [b_ij][b_ki]
// of bins + 1 counters over b_jk, the last of which takes the tests out of
// range and is never read.
__host__ __device__ __forceinline__ int u_words(int bins) { return bins * bins * (bins + 1); }

// The shared histogram of the weighted counts: sums of exact integer weight
// products, three 32-bit limbs each, over [b_ij] and the unordered pair of b_ki and
// b_jk, which the final sums take together.  FP64 adds in global memory queued in
// L2; FP64 adds to shared memory, loops of compare-and-swaps, lay between (us, XXX
// clustered, XXX, XXY of 4100 points, 25 bins, dmax 70: 633 424 1316, 557 342 786, and
// 377 310 682 by limbs; 8000 points 3790 2987 8535, 3222 1861 4779, 2111 1618 3980;
// with XXX rows by ticket since, 309 260 683 and 1587 1237 3978).
__host__ __device__ __forceinline__ int w_slots(int bins) { return bins * (bins * (bins + 1) / 2); }
__device__ __forceinline__ int w_slot(int bins, int bij, int bki, int bjk) {
    const int lo = min(bki, bjk), hi = max(bki, bjk);
    return bij * (bins * (bins + 1) / 2) + hi * (hi + 1) / 2 + lo;
}
// Bytes of a shared histogram, rounded up to 16.
__host__ __device__ __forceinline__ size_t hist_bytes(int bins, bool weighted) {
    const size_t b = weighted ? (size_t)w_slots(bins) * 12 : (size_t)u_words(bins) * 4;
    return (b + 15) & ~(size_t)15;
}
// Adds it into g (bins^3, at [b_ij][lo][hi]) and clears it (whole group; others may
// be adding meanwhile: the limbs are taken one by one, and what a carry brings to
// one afterwards stays for the next flush).
template <int NW>
__device__ __forceinline__ void flush_limbs(unsigned *U, int bins, double unscale, double *g) {
    gsync<NW>();
    const int half = bins * (bins + 1) / 2, n = w_slots(bins);
    for (int k = group_tid<NW>(); k < n; k += NW * 32) {
        if (!(U[k] | U[k + n] | U[k + 2 * n])) continue;
        const double l0 = (double)atomicExch(U + k, 0u), l1 = (double)atomicExch(U + k + n, 0u),
                     l2 = (double)atomicExch(U + k + 2 * n, 0u);
        const int a = k / half, p = k - a * half;
        int hi = (int)((sqrtf(8.f * (float)p + 1.f) - 1.f) * 0.5f);  // hi (hi + 1) / 2 <= p, up to rounding
        if (hi * (hi + 1) / 2 > p) --hi;
        if ((hi + 1) * (hi + 2) / 2 <= p) ++hi;
        atomicAdd(g + ((long long)a * bins + (p - hi * (hi + 1) / 2)) * bins + hi,
                  (l2 * 0x1p64 + (l1 * 0x1p32 + l0)) * unscale);
    }
    gsync<NW>();
}

// Adds U into the u64 histogram g (bins^3, [b_ij][b_ki][b_jk]) and clears it
// (whole group); returns the triangles this thread added.  SHARED: other groups
// may be counting into U meanwhile, so a counter is taken by an exchange, and one
// that settle lowers after its count was taken reads as -1.
template <int NW, bool SHARED>
__device__ __forceinline__ unsigned long long flush_hist(unsigned *U, int bins, unsigned long long *g) {
    gsync<NW>();
    unsigned long long n = 0;
    const int nu = u_words(bins);
    for (int k = group_tid<NW>(); k < nu; k += NW * 32) {
        unsigned v = U[k];
        if (v) {
            const int row = k / (bins + 1), c = k - row * (bins + 1);
            if (SHARED) v = atomicExch(&U[k], 0u);
            else U[k] = 0u;
            if (c < bins) {
                const unsigned long long d = SHARED ? (unsigned long long)(long long)(int)v : v;
                atomicAdd(g + row * bins + c, d);
                n += d;
            }
        }
    }
    gsync<NW>();
    return n;
}

// The extent of one chunk of the K list (in bins).
struct ChunkBox {
    float lo[3], hi[3];
};

// State of a group's anchor loop.
template <int NW>
struct TripCta {
    unsigned *U;                      // shared histogram (hist_in_smem)
    unsigned char *lists;             // shared neighbour lists
    ListScratch<NW> *scr;
    ChunkBox *boxes;                  // max_boxes<NW>() chunks of the K list
    uint2 *queue;                     // 64 tests per warp on their way to the FP64 rule
    int *s_unit;                      // shared counter
    int slot;                         // of the overflow lists
    unsigned n_rechk;
    unsigned long long n_tri;
    unsigned long long since;         // pair tests since U's last flush
};

// A list position past the end: farther than dmax from every entry, and a
// tile's j from a padded k too (they carry opposite signs).
constexpr float kFarAway = 1e15f;
constexpr int kTile = 8;        // j per tile
constexpr int kChunkK = 32;     // K lists are padded to whole chunks of one k per lane
constexpr int kMaxBoxes = 256;  // chunks of K lists that take part in the culling, over the groups
template <int NW>
__host__ __device__ constexpr int max_boxes() { return kMaxBoxes * NW / kTWarps; }
// Fixed-point readout of a third side: bits(128 + r) >> 16 = kSideBias + bin
constexpr float kSideMagic = 128.0f;
constexpr int kSideBits = 16;
constexpr unsigned kSideBias = 0x43000000u >> kSideBits;

// Pads the K list to whole chunks and finds the chunks' extents.  Whole group;
// ends synchronised.
template <int NW>
__device__ __forceinline__ void finish_k(TripCta<NW> &C, float4 *L, int nK) {
    const int lane = threadIdx.x & 31, warp = group_tid<NW>() >> 5;
    const int nchunk = (nK + kChunkK - 1) / kChunkK;
    for (int c = warp; c < nchunk; c += NW) {
        const int k = c * kChunkK + lane;
        float4 e = make_float4(kFarAway, kFarAway, kFarAway, 0.f);
        if (k < nK) e = L[k];
        else L[k] = e;
        if (c < max_boxes<NW>()) {
            const float v[3] = {e.x, e.y, e.z};
            #pragma unroll
            for (int a = 0; a < 3; ++a) {
                float lo = v[a], hi = k < nK ? v[a] : -kFarAway;
                #pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    lo = fminf(lo, __shfl_xor_sync(kFull, lo, o));
                    hi = fmaxf(hi, __shfl_xor_sync(kFull, hi, o));
                }
                if (lane == 0) {
                    C.boxes[c].lo[a] = lo;
                    C.boxes[c].hi[a] = hi;
                }
            }
        }
    }
    gsync<NW>();
}

// The canonical rule for up to 32 tests that fell into a window, one per lane
// (queue entries: j | fast bin << 24, k); corrects their counts in U.
template <bool MIXED>
__device__ __noinline__ void settle(const TripArgs &A, unsigned *U, const float4 *LJ, const float4 *LK,
                                    const uint2 *queue, int n, float hx, float hy, float hz) {
    const int lane = threadIdx.x & 31;
    if (lane >= n) return;
    const uint2 t = queue[lane];
    const int bins = A.rXX.bins, fast = (int)(t.x >> 24);
    const float4 ej = LJ[t.x & 0xFFFFFFu], ek = LK[t.y];
    const int jidx = (int)((unsigned)__float_as_int(ej.w) >> 8);
    const int kidx = (int)((unsigned)__float_as_int(ek.w) >> 8);
    const Cat &CK = MIXED ? A.Y : A.X;
    const int b = exact_third(hx, hy, hz, A.X.x[jidx], A.X.y[jidx], A.X.z[jidx], CK.x[kidx], CK.y[kidx],
                              CK.z[kidx], A.bpc, A.box, MIXED ? A.rXY : A.rXX);
    if (b == fast) return;
    unsigned *row = U + ((__float_as_int(ej.w) & 255) * bins + (__float_as_int(ek.w) & 255)) * (bins + 1);
    atomicSub(row + fast, 1u);
    if (b >= 0) atomicAdd(row + b, 1u);
}

// Pass 2 of the unit-weight counts into U: tiles of kTile consecutive j
// against the K list, one k per lane.  A step loads one k and tests it
// against the tile's j.
//
// What bounds it is instruction issue.  Tiles divide the list loads by kTile,
// and the step is kept branch-free and short: every test adds 1 to a counter,
// tests out of range (their r clamped to bins + 1/2) to the row's last one, and
// tests within the window of a bin edge as the fast path has them; those are
// queued (a rare vote finds them) and, 32 at a time, corrected by the FP64
// rule.  The constant increment lets the hardware add lanes that hit one
// counter together (32 cycles for a register operand where all lanes collide,
// 1 for the constant).  The separations are scalar FP32: packed pairs issue
// half as many FP instructions, but the moves that assemble the pairs come to
// as many again, all on the FMA pipe's heavy half.
// Half of all tests between two neighbours of one anchor are out of range: a
// chunk whose extent is out of the tile's reach is skipped whole (the rounded
// differences are monotone, so no test inside could have been in range).
// FAR: dmax lies more than the window below the last bin's edge (bins / dmax
// rounded down to 1e-6, large dmax), so it needs a window of its own.
template <int NW, bool MIXED, bool FAR>
__device__ __forceinline__ void tri_tiles(const TripArgs &A, TripCta<NW> &C, const float4 *__restrict__ LJ,
                                          const float4 *__restrict__ LK, int nJ, int nK, float hx, float hy,
                                          float hz) {
    const int lane = threadIdx.x & 31, warp = group_tid<NW>() >> 5;
    const int bins = A.rXX.bins;
    const float mgw = kSideMagic + (float)A.fc.wt * 0x1p-16f, qout = kSideMagic + (float)bins + 0.5f;
    const float qlo = A.fc.qlo, qhi = A.fc.qhi, qedge = kSideMagic + (float)bins;
    const unsigned w2 = 2u * A.fc.wt;
    const unsigned Us = (unsigned)__cvta_generic_to_shared(C.U) - 4u * kSideBias;
    const unsigned kstride = 4u * (unsigned)(bins + 1), jstride = kstride * (unsigned)bins;
    const int ntile = (nJ + kTile - 1) / kTile, nchunk = (nK + kChunkK - 1) / kChunkK;
    uint2 *queue = C.queue + warp * 64;
    int queued = 0;
    // units: tiles (XXX: the longest rows first), split along K while there
    // are few tiles per warp
    int segs = 1;
    if (MIXED)
        while (segs < nchunk && ntile * segs < 8 * NW) segs <<= 1;
    const int units = ntile * segs;
    for (;;) {
        int u0 = 0;
        if (lane == 0) u0 = atomicAdd(C.s_unit, 1);
        u0 = __shfl_sync(kFull, u0, 0);
        if (u0 >= units) break;
        const int tile = u0 / segs, sg = u0 - tile * segs, j0 = tile * kTile;
        float JX[kTile], JY[kTile], JZ[kTile];
        unsigned jb[kTile];
        float blo[3] = {kFarAway, kFarAway, kFarAway}, bhi[3] = {-kFarAway, -kFarAway, -kFarAway};
        #pragma unroll
        for (int q = 0; q < kTile; ++q) {
            float4 e = make_float4(-kFarAway, -kFarAway, -kFarAway, 0.f);
            if (j0 + q < nJ) {
                e = LJ[j0 + q];
                blo[0] = fminf(blo[0], e.x);
                bhi[0] = fmaxf(bhi[0], e.x);
                blo[1] = fminf(blo[1], e.y);
                bhi[1] = fmaxf(bhi[1], e.y);
                blo[2] = fminf(blo[2], e.z);
                bhi[2] = fmaxf(bhi[2], e.z);
            }
            JX[q] = e.x;
            JY[q] = e.y;
            JZ[q] = e.z;
            jb[q] = Us + (unsigned)(__float_as_int(e.w) & 255) * jstride;
        }
        // head (XXX): the chunk that holds the tile itself, where k <= j is no test
        auto step = [&](int k, bool head) {
            const float4 e = LK[k];
            const unsigned kb = (unsigned)(__float_as_int(e.w) & 255) * kstride;
            unsigned u[kTile], nearest = 0xffffffffu;  // the smallest fractions, two 16-bit lanes
            #pragma unroll
            for (int q = 0; q < kTile; ++q) {
                const float dx = __fsub_rn(e.x, JX[q]), dy = __fsub_rn(e.y, JY[q]), dz = __fsub_rn(e.z, JZ[q]);
                const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
                float s = __fadd_rn(sqrt_approx(r2), mgw);
                if (head && k <= j0 + q) s = qout;
                // FAR: inside dmax's window the unread counter, marked for the FP64 rule
                if (FAR) s = s < qlo ? s : s < qhi ? qedge : qout;
                else s = fminf(s, qout);
                u[q] = __float_as_uint(s);
                asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(jb[q] + kb + 4u * (u[q] >> kSideBits)));
                if ((q & 3) == 3)
                    nearest = __vimin3_u16x2(nearest, __byte_perm(u[q - 3], u[q - 2], 0x5410),
                                             __byte_perm(u[q - 1], u[q], 0x5410));
            }
            if (__any_sync(kFull, min(nearest & 0xFFFFu, nearest >> 16) < w2)) {
                #pragma unroll
                for (int q = 0; q < kTile; ++q) {
                    const bool hit = (u[q] & 0xFFFFu) < w2;
                    const unsigned m = __ballot_sync(kFull, hit);
                    if (!m) continue;
                    if (hit)
                        queue[queued + __popc(m & ((1u << lane) - 1u))] =
                            make_uint2((unsigned)(j0 + q) | (((u[q] >> kSideBits) - kSideBias) << 24), (unsigned)k);
                    C.n_rechk += hit;
                    queued += __popc(m);
                    __syncwarp();
                    if (queued >= 32) {
                        queued -= 32;
                        settle<MIXED>(A, C.U, LJ, LK, queue + queued, 32, hx, hy, hz);
                        __syncwarp();
                    }
                }
            }
        };
        int c = MIXED ? (int)((long long)nchunk * sg / segs) : j0 / kChunkK;
        const int c1 = MIXED ? (int)((long long)nchunk * (sg + 1) / segs) : nchunk;
        if (!MIXED) step(c++ * kChunkK + lane, true);
        for (; c < c1; c += 32) {
            bool in = c + lane < c1;
            if (in && c + lane < max_boxes<NW>()) {
                const ChunkBox &b = C.boxes[c + lane];
                float g[3];
                #pragma unroll
                for (int a = 0; a < 3; ++a)
                    g[a] = fmaxf(0.f, fmaxf(__fsub_rn(b.lo[a], bhi[a]), __fsub_rn(blo[a], b.hi[a])));
                in = !(fmaf(g[2], g[2], fmaf(g[1], g[1], __fmul_rn(g[0], g[0]))) >= A.fc.hi3);
            }
            unsigned todo = __ballot_sync(kFull, in);
            for (int k = c * kChunkK + lane; todo; k += kChunkK, todo >>= 1)
                if (todo & 1u) step(k, false);
        }
    }
    if (queued) settle<MIXED>(A, C.U, LJ, LK, queue, queued, hx, hy, hz);
}

// All triangles of anchor i of job A: pass 1 builds the anchor's
// neighbour lists in shared memory (or, past their capacity, in the group's
// global scratch), pass 2 counts the neighbour pairs.
template <int NW, bool MIXED, bool WEIGHTED>
__device__ __forceinline__ void tri_anchor(const TripArgs &A, int i, TripCta<NW> &C) {
    const int bins = A.rXX.bins;
    const int tid = group_tid<NW>(), lane = tid & 31, warp = tid >> 5;
    unsigned &n_rechk = C.n_rechk;
    float4 *sJ = reinterpret_cast<float4 *>(C.lists);
    float4 *sK = sJ + A.capJ;
    float *swJ = reinterpret_cast<float *>(sK + (MIXED ? A.capK : 0));
    float *swK = swJ + (WEIGHTED ? A.capJ : 0);
    float4 *gJ = A.gJ + (size_t)C.slot * A.gcap;
    float4 *gK = A.gK ? A.gK + (size_t)C.slot * A.gcap : nullptr;
    float *gwJ = A.gwJ ? A.gwJ + (size_t)C.slot * A.gcap : nullptr;
    float *gwK = A.gwK ? A.gwK + (size_t)C.slot * A.gcap : nullptr;
    const float hx = A.X.x[i], hy = A.X.y[i], hz = A.X.z[i];
    const float hw = WEIGHTED ? A.X.w[i] : 1.f;
    const int P = A.P;
    const int cix = min(max((int)__fdiv_rn(hx, A.cell), 0), P - 1);
    const int ciy = min(max((int)__fdiv_rn(hy, A.cell), 0), P - 1);
    const int ciz = min(max((int)__fdiv_rn(hz, A.cell), 0), P - 1);
    // pass 1: lists into shared memory (sizes counted even past capacity).
    // Pooled (unit weights, shared histogram): one buffer of capJ entries, J
    // and behind it K, each list that is walked in chunks padded to them.
    const bool pool = !WEIGHTED && A.hist_in_smem;
    auto padded = [](int n) { return (n + kChunkK - 1) / kChunkK * kChunkK; };
    int nJ = build_list<NW, false>(A, A.X, hx, hy, hz, cix, ciy, ciz, i, A.rXX, sJ, WEIGHTED ? swJ : nullptr, A.capJ,
                               n_rechk, *C.scr);
    int capK = A.capK, nK = nJ;
    if (MIXED) {
        if (pool) {
            sK = sJ + min(nJ, A.capJ);
            capK = max(0, A.capJ - nJ);
        }
        nK = build_list<NW, false>(A, A.Y, hx, hy, hz, cix, ciy, ciz, -1, A.rXY, sK, WEIGHTED ? swK : nullptr, capK,
                               n_rechk, *C.scr);
    }
    const float4 *LJ = sJ;
    const float4 *LK = MIXED ? sK : sJ;
    const float *WJ = swJ, *WK = MIXED ? swK : swJ;
    const bool spill = nJ > A.capJ || (MIXED && nK > capK) || (pool && padded(nK) > (MIXED ? capK : A.capJ));
    if (spill) {
        // overflow: the lists in the group's global scratch (L2), which holds any anchor's
        nJ = min(A.gcap, build_list<NW, false>(A, A.X, hx, hy, hz, cix, ciy, ciz, i, A.rXX, gJ,
                                           WEIGHTED ? gwJ : nullptr, A.gcap, n_rechk, *C.scr));
        nK = nJ;
        if (MIXED)
            nK = min(A.gcap, build_list<NW, false>(A, A.Y, hx, hy, hz, cix, ciy, ciz, -1, A.rXY, gK,
                                               WEIGHTED ? gwK : nullptr, A.gcap, n_rechk, *C.scr));
        LJ = gJ;
        LK = MIXED ? gK : gJ;
        WJ = gwJ;
        WK = MIXED ? gwK : gwJ;
    }
    // Flush budget of the shared histogram: this anchor adds at most
    // `tests` times.  Flush first if the total could pass the budget; an
    // anchor whose tests alone exceed it counts into global memory.
    bool smem_hist = A.hist_in_smem;
    if (smem_hist) {
        const unsigned long long tests =
            MIXED ? (unsigned long long)nJ * (unsigned long long)nK
                  : (unsigned long long)nJ * (unsigned long long)(nJ > 0 ? nJ - 1 : 0) / 2;
        if (tests > A.flush_budget) {
            smem_hist = false;
        } else {
            if (C.since + tests > A.flush_budget) {
                if (WEIGHTED) flush_limbs<NW>(C.U, bins, A.wunscale, A.g_wsum);
                else C.n_tri += flush_hist<NW, NW != kTWarps>(C.U, bins, A.g_count);
                C.since = 0;
            }
            C.since += tests;
        }
    }
    // pass 2: pairs of neighbours
    if (smem_hist && !WEIGHTED) {
        // the lists' address space is fixed per instantiation, so the
        // shared-memory case (all but overflowing anchors) uses shared loads
        if (spill) {
            finish_k(C, MIXED ? gK : gJ, nK);
            if (A.fc.far) tri_tiles<NW, MIXED, true>(A, C, gJ, MIXED ? gK : gJ, nJ, nK, hx, hy, hz);
            else tri_tiles<NW, MIXED, false>(A, C, gJ, MIXED ? gK : gJ, nJ, nK, hx, hy, hz);
        } else {
            finish_k(C, MIXED ? sK : sJ, nK);
            if (A.fc.far) tri_tiles<NW, MIXED, true>(A, C, sJ, MIXED ? sK : sJ, nJ, nK, hx, hy, hz);
            else tri_tiles<NW, MIXED, false>(A, C, sJ, MIXED ? sK : sJ, nJ, nK, hx, hy, hz);
        }
        return;
    }
    auto weight = [&](float w) { return A.wfix ? (double)__float_as_uint(w) : (double)w; };
    const int nw = WEIGHTED ? w_slots(bins) : 0;
    // XXX, whose rows shrink with j: rows by ticket, the longest first.  Dealt out
    // beforehand (0, n-1, 1, n-2, ...) the warps waited for one another a third of
    // their time (4100 points, dmax 70, 25 bins, weighted: 377 and 310 -> 320 and
    // 260 us).  XXY rows are of one length.
    for (int jj = warp;; jj += NW) {
        if (!MIXED) {
            if (lane == 0) jj = atomicAdd(C.s_unit, 1);
            jj = __shfl_sync(kFull, jj, 0);
        }
        if (jj >= nJ) break;
        const float4 ej = LJ[jj];
        const int bj = __float_as_int(ej.w) & 255;
        const int jidx = (int)((unsigned)__float_as_int(ej.w) >> 8);
        const double wij = WEIGHTED ? weight(hw) * weight(WJ[jj]) * (A.wfix ? A.wunscale : 1.0) : 1.0;
        const unsigned long long qij =
            WEIGHTED ? (unsigned long long)__float_as_uint(hw) * __float_as_uint(WJ[jj]) : 0ull;
        const int ubase = bj * bins * bins;
        const int k0 = MIXED ? 0 : jj + 1;
        for (int kk = k0 + lane; kk < nK; kk += 32) {
            const float4 ek = LK[kk];
            const float dx = ek.x - ej.x, dy = ek.y - ej.y, dz = ek.z - ej.z;
            const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            const PairRule &r3 = MIXED ? A.rXY : A.rXX;
            int bjk = fast_bin3(r2, A.fc, bins);
            if (bjk == -1) {
                ++n_rechk;
                const int kidx = (int)((unsigned)__float_as_int(ek.w) >> 8);
                const Cat &CK = MIXED ? A.Y : A.X;
                bjk = exact_third(hx, hy, hz, A.X.x[jidx], A.X.y[jidx], A.X.z[jidx], CK.x[kidx], CK.y[kidx],
                                  CK.z[kidx], A.bpc, A.box, r3);
            }
            if (bjk >= 0) {
                const int bk = __float_as_int(ek.w) & 255;
                // (b_jk before b_ki, which the final sums do not tell apart: lanes of one
                // list stretch then add to neighbouring words.  16000 points, dmax 60 of
                // 250, signed weights, XXX, 18, 25 and 30 bins: 39.3 15.6 10.9 ms -> 32.2 11.7 8.1)
                const int slot = ubase + bjk * bins + bk;
                ++C.n_tri;
                if (!WEIGHTED) {
                    atomicAdd(A.g_count + slot, 1ull);
                } else if (smem_hist) {
                    // q_i q_j q_k in three limbs, the carries by the values that the
                    // adds return (an FP64 add to shared memory is a loop of
                    // compare-and-swaps, one to global memory queues in L2)
                    const unsigned qk = __float_as_uint(WK[kk]);
                    const unsigned long long p0 = (qij & 0xffffffffull) * qk, p1 = (qij >> 32) * qk + (p0 >> 32);
                    unsigned *u = C.U + w_slot(bins, bj, bk, bjk);
                    const unsigned l0 = (unsigned)p0, l1 = (unsigned)p1;
                    const unsigned c0 = atomicAdd(u, l0) > ~l0 ? 1u : 0u;
                    const unsigned long long m = (unsigned long long)l1 + c0;
                    const unsigned m0 = (unsigned)m;
                    const unsigned c1 = atomicAdd(u + nw, m0) > ~m0 ? 1u : 0u;
                    const unsigned h = (unsigned)(p1 >> 32) + (unsigned)(m >> 32) + c1;
                    if (h) atomicAdd(u + 2 * nw, h);
                } else {
                    atomicAdd(A.g_wsum + slot, wij * weight(WK[kk]));
                }
            }
        }
    }
}

template <bool MIXED, bool WEIGHTED, int NW>
__global__ void __launch_bounds__(kTThreads, 1) k_triplets(const __grid_constant__ TripArgs A) {
    constexpr int G = kTWarps / NW;
    extern __shared__ __align__(16) unsigned char smem[];
    const int bins = A.rXX.bins;
    const size_t u_bytes = A.hist_in_smem ? hist_bytes(bins, WEIGHTED) : 0;
    __shared__ ListScratch<NW> s_scr[G];
    __shared__ ChunkBox s_boxes[kMaxBoxes];
    __shared__ uint2 s_queue[64 * kTWarps];
    __shared__ int s_anchor[G], s_unit[G];
    __shared__ unsigned s_stop[G];
    const int tid = group_tid<NW>(), lane = tid & 31, g = (int)threadIdx.x / (NW * 32);
    TripCta<NW> C{reinterpret_cast<unsigned *>(smem), smem + u_bytes + (size_t)g * A.list_bytes, &s_scr[g],
                  s_boxes + g * max_boxes<NW>(), s_queue + g * NW * 64, &s_unit[g], (int)blockIdx.x * G + g, 0u,
                  0ull, 0ull};
    if (A.hist_in_smem)
        for (int k = threadIdx.x; k < (int)(u_bytes / 4); k += kTThreads) C.U[k] = 0u;
    if (G > 1) __syncthreads();
    long long taken = 0;  // anchors this group took (iteration cap: nX + 1)
    int ticket = 0;       // thread 0: the next anchor, taken while the last one is counted
    if (tid == 0) ticket = (int)atomicAdd(A.counter, 1ull);
    for (;;) {
        if (tid == 0) {
            s_anchor[g] = ticket;
            s_unit[g] = 0;
            unsigned stop = (A.ctrl && ctrl_load(A.ctrl)) ? PCF_GAVE_UP_ABORT : 0u;
            if (++taken > (long long)A.nX + 1) stop |= PCF_GAVE_UP_CAP;
            if (stop && A.status) ctrl_store(A.status, stop);
            s_stop[g] = stop;
        }
        gsync<NW>();
        const int i = s_anchor[g];
        if (i >= A.nX || s_stop[g]) break;
        if (tid == 0) ticket = (int)atomicAdd(A.counter, 1ull);
        tri_anchor<NW, MIXED, WEIGHTED>(A, i, C);
        gsync<NW>();
    }
    if (A.hist_in_smem) {
        if (G > 1) __syncthreads();  // every group's counts are in
        if (WEIGHTED) flush_limbs<kTWarps>(C.U, bins, A.wunscale, A.g_wsum);
        else C.n_tri += flush_hist<kTWarps, (G > 1)>(C.U, bins, A.g_count);
    }
    unsigned long long rr = C.n_rechk, nt = C.n_tri;
    for (int off = 16; off > 0; off >>= 1) {
        rr += __shfl_down_sync(kFull, rr, off);
        nt += __shfl_down_sync(kFull, nt, off);
    }
    if (lane == 0) {
        if (rr) atomicAdd(A.g_stats + 0, rr);
        if (nt) atomicAdd(A.g_stats + 2, nt);
    }
}

// Anisotropic triplets (3ani_k.cuh:8,109; 3aniBPC_k.cuh:210,959): ordered
// triples anchored at point 1 = the anchor i; the lists hold every X (and
// for XXY every Y) neighbour with its exact side bin and angle bin, and all
// ordered (j, k), j != k, are counted into the bins^5 histogram
// [b(d12)][b(d31)][b(d23)][t12][t31] in global memory.  XXX without gates, where
// (k, j) counts what (j, k) does with points 2 and 3 exchanged: j < k alone, and
// k_to_double adds the exchanged bin (3000 points, 12 bins, dmax 60: 844 us for
// DDD and RRR -> 507, with rows by ticket 483).
// GATES (periodic, PCF_REF_NODE_GATES): each ordered triangle counts as many
// times as the reference's node-gate blocks count it (node_gates.cuh), on the
// reference's node grid A.gate.  ISO3 (with GATES): the isotropic bins^3
// histogram [b(d12)][b(d23)][b(d31)] of the same ordered triangles
// (3isoBPC_k.cuh:191,940), from lists without angle bins.
template <int NW, bool MIXED, bool WEIGHTED, bool GATES = false, bool ISO3 = false>
__global__ void __launch_bounds__(NW * 32, kTWarps / NW) k_triplets_ani(const TripArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int bins = A.rXX.bins;
    float4 *sJ = reinterpret_cast<float4 *>(smem);
    float4 *sK = sJ + A.capJ;
    float *swJ = reinterpret_cast<float *>(sK + (MIXED ? A.capK : 0));
    float *swK = swJ + (WEIGHTED ? A.capJ : 0);
    // node / image words of the gated counts, then the angle bins
    unsigned *gJ = reinterpret_cast<unsigned *>(swK + (WEIGHTED && MIXED ? A.capK : 0));
    unsigned *gK = gJ + (GATES ? A.capJ : 0);
    unsigned char *aJ = reinterpret_cast<unsigned char *>(gK + (GATES && MIXED ? A.capK : 0));
    unsigned char *aK = aJ + A.capJ;
    __shared__ ListScratch<NW> s_scr;
    __shared__ int s_anchor, s_unit;
    __shared__ unsigned s_stop;
    __shared__ GateBlock s_gates[GATES ? 64 : 1];
    __shared__ signed char s_gate_by[GATES ? 64 : 1][2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (GATES) {
        for (int k = tid; k < 64; k += NW * 32) {
            s_gates[k] = kGateBlocks[k];
            s_gate_by[k][0] = kGateByImage[k][0];
            s_gate_by[k][1] = kGateByImage[k][1];
        }
    }
    unsigned n_rechk = 0;
    unsigned long long n_tri = 0;
    long long taken = 0;
    const long long B = bins, B2 = B * B, B3 = B2 * B, B4 = B3 * B;
    constexpr bool HALF = !MIXED && !GATES;
    for (;;) {
        if (tid == 0) {
            s_anchor = (int)atomicAdd(A.counter, 1ull);
            s_unit = 0;
            unsigned stop = (A.ctrl && ctrl_load(A.ctrl)) ? PCF_GAVE_UP_ABORT : 0u;
            if (++taken > (long long)A.nX + 1) stop |= PCF_GAVE_UP_CAP;
            if (stop && A.status) ctrl_store(A.status, stop);
            s_stop = stop;
        }
        __syncthreads();
        const int i = s_anchor;
        if (i >= A.nX || s_stop) break;
        const float hx = A.X.x[i], hy = A.X.y[i], hz = A.X.z[i];
        const float hw = WEIGHTED ? A.X.w[i] : 1.f;
        const int P = A.P;
        const int cix = min(max((int)__fdiv_rn(hx, A.cell), 0), P - 1);
        const int ciy = min(max((int)__fdiv_rn(hy, A.cell), 0), P - 1);
        const int ciz = min(max((int)__fdiv_rn(hz, A.cell), 0), P - 1);
        const int nJ = build_list<NW, !ISO3>(A, A.X, hx, hy, hz, cix, ciy, ciz, -1, A.rXX, sJ,
                                         WEIGHTED ? swJ : nullptr, A.capJ, n_rechk, s_scr, aJ,
                                         GATES ? gJ : nullptr);
        const int nK = MIXED ? build_list<NW, !ISO3>(A, A.Y, hx, hy, hz, cix, ciy, ciz, -1, A.rXY, sK,
                                                 WEIGHTED ? swK : nullptr, A.capK, n_rechk, s_scr, aK,
                                                 GATES ? gK : nullptr)
                             : nJ;
        GateNode n1{};
        if (GATES) n1 = gate_unpack(A.gate, gate_pack(A.gate, hx, hy, hz, 0u));
        if (nJ > A.capJ || (MIXED && nK > A.capK)) {
            // lists beyond shared memory: flagged for the host, anchor skipped
            if (tid == 0) atomicAdd(A.g_stats + 3, 1ull);
            __syncthreads();
            continue;
        }
        const float4 *LK = MIXED ? sK : sJ;
        const unsigned char *AK = MIXED ? aK : aJ;
        const float *WK = MIXED ? swK : swJ;
        for (int jj = warp;; jj += NW) {
            if (HALF) {  // rows shrink with j: by ticket, the longest first
                if (lane == 0) jj = atomicAdd(&s_unit, 1);
                jj = __shfl_sync(0xffffffffu, jj, 0);
            }
            if (jj >= nJ) break;
            const float4 ej = sJ[jj];
            const int jidx = (int)((unsigned)__float_as_int(ej.w) >> 8);
            const int bj = __float_as_int(ej.w) & 255;
            const long long base = ISO3 ? (long long)bj * B2 : (long long)bj * B4 + (long long)aJ[jj] * B;
            const double wij = WEIGHTED ? (double)hw * (double)swJ[jj] : 1.0;
            GateNode n2{};
            if (GATES) n2 = gate_unpack(A.gate, gJ[jj]);
            const unsigned *GK = MIXED ? gK : gJ;
            for (int kk = (HALF ? jj + 1 : 0) + lane; kk < nK; kk += 32) {
                if (!MIXED && kk == jj) continue;
                const float4 ek = LK[kk];
                const float dx = ek.x - ej.x, dy = ek.y - ej.y, dz = ek.z - ej.z;
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                const PairRule &r3 = MIXED ? A.rXY : A.rXX;
                int c = fast_bin3(r2, A.fc, bins);
                if (c == -1) {
                    ++n_rechk;
                    const int kidx = (int)((unsigned)__float_as_int(ek.w) >> 8);
                    const Cat &CK = MIXED ? A.Y : A.X;
                    c = exact_third(hx, hy, hz, A.X.x[jidx], A.X.y[jidx], A.X.z[jidx], CK.x[kidx],
                                    CK.y[kidx], CK.z[kidx], A.bpc, A.box, r3);
                }
                if (c >= 0) {
                    int mult = 1;
                    if (GATES) {
                        mult = gate_mult(A.gate, n1, n2, gate_unpack(A.gate, GK[kk]), s_gates, s_gate_by);
                        if (mult == 0) continue;
                    }
                    long long slot;
                    if (ISO3) {
                        slot = base + (long long)c * B + (__float_as_int(ek.w) & 255);
                    } else {
                        slot = base + (long long)(__float_as_int(ek.w) & 255) * B3 + (long long)c * B2 + AK[kk];
                    }
                    n_tri += (unsigned long long)mult;
                    if (WEIGHTED) atomicAdd(A.g_wsum + slot, wij * (double)WK[kk] * (double)mult);
                    else atomicAdd(A.g_count + slot, (unsigned long long)mult);
                }
            }
        }
        __syncthreads();
    }
    unsigned long long rr = n_rechk;
    for (int off = 16; off > 0; off >>= 1) {
        rr += __shfl_down_sync(kFull, rr, off);
        n_tri += __shfl_down_sync(kFull, n_tri, off);
    }
    if (lane == 0) {
        if (rr) atomicAdd(A.g_stats + 0, rr);
        if (n_tri) atomicAdd(A.g_stats + 2, n_tri);
    }
}

// Node-gated isotropic counts (unit weights) as corrections of the plain ones.
// Where gates_hold, a regular block (node_gates.cuh) counts each of its triangles
// once, so the gated histogram is the plain one, which k_triplets makes from
// unordered triangles, plus (multiplicity - 1) of the ordered triangles whose
// images (F2, F3) have no regular block: eight of the 64 combinations, both points
// through an image and two axes involved.  This kernel evaluates those alone, from
// the anchors near two or more faces and their neighbours through an image.
// Evaluating every ordered triangle's gates, with a global atomic each, took 50.7 ms
// for 4096 and 4100 points (DDD, RRR, DDR, DRR; bins 30, dmax 80 of 250).
// Histogram: A.g_count, bins^3 signed, [b(d12)][b(d23)][b(d31)]; g_stats[1]: their sum.
template <int NW, bool MIXED>
__global__ void __launch_bounds__(NW * 32, kTWarps / NW) k_gate_fix(const __grid_constant__ TripArgs A, float reach) {
    extern __shared__ __align__(16) unsigned char smem[];
    float4 *sJ = reinterpret_cast<float4 *>(smem), *sK = sJ + A.capJ;
    unsigned *gJ = reinterpret_cast<unsigned *>(sK + A.capK), *gK = gJ + A.capJ;
    // the third points by image: indices in `by`, those of images f at s_class[f] ..
    unsigned short *by = reinterpret_cast<unsigned short *>(gK + A.capK);
    __shared__ int s_class[9], s_fill[8];
    __shared__ ListScratch<NW> s_scr;
    __shared__ int s_anchor;
    __shared__ unsigned s_stop;
    __shared__ GateBlock s_gates[64];
    __shared__ signed char s_gate_by[64][2];
    __shared__ unsigned s_irr[8];  // per F2: the F3 without a regular block
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bins = A.rXX.bins;
    if (tid < 8) s_irr[tid] = 0u;
    if (tid < 64) {
        s_gates[tid] = kGateBlocks[tid];
        s_gate_by[tid][0] = kGateByImage[tid][0];
        s_gate_by[tid][1] = kGateByImage[tid][1];
    }
    __syncthreads();
    if (tid < 64 && !gate_regular(tid & 7, tid >> 3, s_gates, s_gate_by)) atomicOr(&s_irr[tid & 7], 1u << (tid >> 3));
    unsigned n_rechk = 0;
    long long n_fix = 0, taken = 0;
    for (;;) {
        if (tid == 0) {
            s_anchor = (int)atomicAdd(A.counter, 1ull);
            unsigned stop = (A.ctrl && ctrl_load(A.ctrl)) ? PCF_GAVE_UP_ABORT : 0u;
            if (++taken > (long long)A.nX + 1) stop |= PCF_GAVE_UP_CAP;
            if (stop && A.status) ctrl_store(A.status, stop);
            s_stop = stop;
        }
        __syncthreads();
        const int i = s_anchor;
        if (i >= A.nX || s_stop) break;
        const float hx = A.X.x[i], hy = A.X.y[i], hz = A.X.z[i];
        const int near = (hx <= reach || hx >= A.box - reach) + (hy <= reach || hy >= A.box - reach) +
                         (hz <= reach || hz >= A.box - reach);
        if (near >= 2) {
            const int P = A.P;
            const int cix = min(max((int)__fdiv_rn(hx, A.cell), 0), P - 1);
            const int ciy = min(max((int)__fdiv_rn(hy, A.cell), 0), P - 1);
            const int ciz = min(max((int)__fdiv_rn(hz, A.cell), 0), P - 1);
            const int nJ = build_list<NW, false, true>(A, A.X, hx, hy, hz, cix, ciy, ciz, -1, A.rXX, sJ, nullptr, A.capJ,
                                                   n_rechk, s_scr, nullptr, gJ);
            const int nK = MIXED ? build_list<NW, false, true>(A, A.Y, hx, hy, hz, cix, ciy, ciz, -1, A.rXY, sK, nullptr,
                                                           A.capK, n_rechk, s_scr, nullptr, gK)
                                 : nJ;
            const bool fits = nJ <= A.capJ && (!MIXED || nK <= A.capK);
            if (!fits && tid == 0) atomicAdd(A.g_stats + 3, 1ull);  // not reached: the host bounds the lists
            const GateNode n1 = gate_unpack(A.gate, gate_pack(A.gate, hx, hy, hz, 0u));
            const float4 *LK = MIXED ? sK : sJ;
            const unsigned *GK = MIXED ? gK : gJ;
            if (tid < 8) s_fill[tid] = 0;
            __syncthreads();
            for (int kk = tid; fits && kk < nK; kk += NW * 32) atomicAdd(&s_fill[GK[kk] >> 27 & 7u], 1);
            __syncthreads();
            if (tid == 0) {
                int n = 0;
                for (int f = 0; f < 8; ++f) {
                    s_class[f] = n;
                    n += s_fill[f];
                    s_fill[f] = s_class[f];
                }
                s_class[8] = n;
            }
            __syncthreads();
            for (int kk = tid; fits && kk < nK; kk += NW * 32)
                by[atomicAdd(&s_fill[GK[kk] >> 27 & 7u], 1)] = (unsigned short)kk;
            __syncthreads();
            for (int jj = warp; fits && jj < nJ; jj += NW) {
                unsigned irr = s_irr[(gJ[jj] >> 27) & 7u];
                if (!irr) continue;
                const float4 ej = sJ[jj];
                const GateNode n2 = gate_unpack(A.gate, gJ[jj]);
                const int jidx = (int)((unsigned)__float_as_int(ej.w) >> 8), bj = __float_as_int(ej.w) & 255;
                for (; irr; irr &= irr - 1u)
                for (int q = s_class[__ffs(irr) - 1] + lane; q < s_class[__ffs(irr)]; q += 32) {
                    const int kk = by[q];
                    if (!MIXED && kk == jj) continue;
                    const float4 ek = LK[kk];
                    const float dx = ek.x - ej.x, dy = ek.y - ej.y, dz = ek.z - ej.z;
                    int c = fast_bin3(fmaf(dz, dz, fmaf(dy, dy, dx * dx)), A.fc, bins);
                    if (c == -1) {
                        ++n_rechk;
                        const int kidx = (int)((unsigned)__float_as_int(ek.w) >> 8);
                        const Cat &CK = MIXED ? A.Y : A.X;
                        c = exact_third(hx, hy, hz, A.X.x[jidx], A.X.y[jidx], A.X.z[jidx], CK.x[kidx], CK.y[kidx],
                                        CK.z[kidx], A.bpc, A.box, MIXED ? A.rXY : A.rXX);
                    }
                    if (c < 0) continue;
                    const int fix = gate_mult(A.gate, n1, n2, gate_unpack(A.gate, GK[kk]), s_gates, s_gate_by) - 1;
                    if (fix == 0) continue;
                    n_fix += fix;
                    atomicAdd(A.g_count + ((long long)bj * bins + c) * bins + (__float_as_int(ek.w) & 255),
                              (unsigned long long)(long long)fix);
                }
            }
        }
        __syncthreads();
    }
    unsigned long long rr = n_rechk;
    for (int off = 16; off > 0; off >>= 1) {
        rr += __shfl_down_sync(kFull, rr, off);
        n_fix += __shfl_down_sync(kFull, n_fix, off);
    }
    if (lane == 0) {
        if (rr) atomicAdd(A.g_stats + 0, rr);
        if (n_fix) atomicAdd(A.g_stats + 1, (unsigned long long)n_fix);
    }
}

// bins5 > 0: the histogram [b12][b31][b23][t12][t31] holds half the ordered
// triangles; the others are in the bin with points 2 and 3 exchanged.
__global__ void k_to_double(const unsigned long long *__restrict__ c, const double *__restrict__ w,
                            int weighted, long long n, double *__restrict__ out,
                            const unsigned long long *__restrict__ stats, unsigned long long *host_stats, int bins5) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 4) host_stats[t] = stats[t];
    if (t >= n) return;
    long long u = t;
    if (bins5) {
        const long long B = bins5, B2 = B * B;
        const long long t31 = t % B, t12 = t / B % B, b23 = t / B2 % B, b31 = t / (B2 * B) % B, b12 = t / (B2 * B2);
        u = ((((b31 * B) + b12) * B + b23) * B + t31) * B + t12;
        out[t] = weighted ? w[t] + w[u] : (double)(c[t] + c[u]);
        return;
    }
    out[t] = weighted ? w[t] : (double)c[t];
}

// fix: the node gates' corrections of an unweighted count.
// Ordered-triple histogram from the oriented counts U[b_ij][b_ki][b_jk] (both
// sums below are the same for U[b_ij][b_jk][b_ki]).
__global__ void k_trip_finalize(const unsigned long long *__restrict__ cnt,
                                const double *__restrict__ ws, int weighted, int mixed, int bins,
                                double *__restrict__ out, const unsigned long long *__restrict__ stats,
                                unsigned long long *host_stats, const unsigned long long *__restrict__ fix) {
    const int n3 = bins * bins * bins;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (host_stats && t < 4) host_stats[t] = stats[t];
    if (t >= n3) return;
    const int a = t / (bins * bins), b = (t / bins) % bins, c = t % bins;
    auto U = [&](int x, int y, int z) -> double {
        const int s = (x * bins + y) * bins + z;
        return weighted ? ws[s] : (double)cnt[s];
    };
    if (fix) {  // k_gate_fix, in whole numbers
        auto N = [&](int x, int y, int z) { return cnt[(x * bins + y) * bins + z]; };
        const unsigned long long n =
            mixed ? N(a, b, c) + N(a, c, b)
                  : N(a, b, c) + N(b, c, a) + N(c, a, b) + N(a, c, b) + N(c, b, a) + N(b, a, c);
        out[t] = (double)(n + fix[t]);
        return;
    }
    double v;
    if (mixed) v = U(a, b, c) + U(a, c, b);
    else v = U(a, b, c) + U(b, c, a) + U(c, a, b) + U(a, c, b) + U(c, b, a) + U(b, a, c);
    out[t] = v;
}

}  // namespace

constexpr int64_t kCheapBound = 8192;
// Bound of an anchor's list in a catalog of n points gridded as g: n itself
// up to `cheap` (while overflow lists of that size are small), else the largest stencil
// population of any cell (memoised per cell structure, dmax and periodicity: the
// rows are fixed by them and the structure's P).
static pcf_status list_bound(pcf_ctx *ctx, const CellGrid &g, int64_t n, float dmax, const RowDesc *d_rows, int n_rows,
                             bool bpc, int64_t *out, int64_t cheap = kCheapBound) {
    *out = n;
    if (n <= cheap) return PCF_OK;
    for (const auto &m : g.stencil_memo)
        if (m.first.first == dmax && m.first.second == bpc) {
            *out = m.second;
            return PCF_OK;
        }
    const pcf_status s = stencil_max(ctx, g, d_rows, n_rows, bpc, out);
    if (s == PCF_OK) g.stencil_memo.push_back({{dmax, bpc}, *out});
    return s;
}

// FP32 windows of the triplet kernels (u = 2^-24, R = dmax, L = box).  A list
// entry, candidate - (anchor - shift), is off by u of itself (at most uR), where
// an axis is image-shifted by 2uL more, and by u of itself again when scaled to
// bins; the third side's difference of two entries adds u of itself.  Its vector
// is thus off by at most sqrt(3) (4uR + 4uL) = 6.9uR + 6.9uL (no L term without a
// periodic box), and d2 and r carry the pair kernel's 5u and 6.5u (make_cuts) and
// the scale's u beside that.  The windows keep more than twice these bounds; the
// anchor's sides, with one entry's error, lie well inside.
static TripCuts trip_cuts(const PairRule &rule, float box, float dmax, bool bpc) {
    TripCuts c;
    const double dd = rule.dd, R = (double)dmax, L = bpc ? (double)box : 0.0;
    const double rmax = R * rule.ds + 1.0;
    const double e_d2 = dd * std::ldexp(1.0, -18) + R * L * std::ldexp(1.0, -19);
    const double wr = rmax * std::ldexp(1.0, -20) + rule.ds * (R + L) * std::ldexp(1.0, -20);
    c.dsf = (float)rule.ds;
    c.ds2 = c.dsf * c.dsf;
    c.lo = (float)(dd - e_d2);
    c.hi = (float)(dd + e_d2);
    c.lo3 = (float)((dd - e_d2) * rule.ds * rule.ds);
    c.hi3 = (float)((dd + e_d2) * rule.ds * rule.ds);
    // + the rounding of the fixed-point readout (2^-16)
    c.w = std::min(8000u, (unsigned)std::ceil((wr + std::ldexp(1.0, -16)) * 32768.0));
    // The tiles' window, in units of 2^-16: 1.25 times the bound and the rounding
    // of the readout (a test in it costs about 40 instructions of its warp).  dmax lies `gap` units below the last bin's edge: ds is rounded down to
    // 1e-6, so gap is at most dmax * 0.066.  Up to 16 units (dmax of about 250)
    // the window takes it in; beyond, dmax gets a window of its own.
    const double edge = std::sqrt(dd) * rule.ds;
    const double gap = std::ceil(std::max(0.0, (double)rule.bins - edge) * 65536.0);
    c.far = gap > 16.0 ? 1 : 0;
    const double bound = (rmax * 7.5 + rule.ds * (R + L) * 6.93) / 256.0;
    c.wt = std::min(16000u, (unsigned)std::ceil(bound * 1.25 + 0.5 + (c.far ? 0.0 : gap)));
    // r in [edge - w, edge + w] as values of r + 128 + w, one unit wider
    c.qlo = (float)(128.0 + edge) - 0x1p-16f;
    c.qhi = (float)(128.0 + edge) + (float)(2u * c.wt + 1u) * 0x1p-16f;
    return c;
}

// Shared memory of the isotropic kernels' lists and histogram.
constexpr size_t kTripSmem = 227 * 1024 - 256 - sizeof(ListScratch<kTWarps>) - sizeof(ChunkBox) * kMaxBoxes -
                             sizeof(uint2) * 64 * kTWarps;
static size_t trip_hist_bytes(int bins, bool weighted) {
    const size_t b = hist_bytes(bins, weighted);
    return b <= (weighted ? 166 : 150) * 1024 ? b : 0;
}
// Adds that a three-limb counter of the weighted counts takes (0: the weights are
// no exact integers, or their products too large).
static unsigned long long limb_budget(const pcf_grid *X, const pcf_grid *Y) {
    if (!X->wfix_ok || (Y && !Y->wfix_ok)) return 0;
    const double q = (double)X->wqmax * (double)X->wqmax * (double)(Y ? Y : X)->wqmax;
    const double adds = std::floor(std::ldexp(1.0, 96) / std::max(q, 1.0) * (1.0 - 1e-9));
    return adds < 262144.0 ? 0 : (unsigned long long)std::min(adds, 2147483648.0);
}

// Groups of warps per CTA, each with anchors of its own.  Three overlap the
// latencies of one anchor's list builds (about 6 us, most of the time of a short
// list) with the counting of others; their lists share the room, and lists that
// spill into global memory cost more than that.  us, 1 -> 3 groups (XXX
// clustered, XXX, XXY): 1000 points, dmax 45 of 250, 20 bins 42 39 55 -> 29 23 35;
// 4100: 153 136 254 -> 86 71 176; 16000: 969 817 2848 -> 698 524 1755; 30 bins, dmax 80: 4100: 279
// 257 852 -> 221 193 567; 8000: 986 883 2939 -> 952 805 2468; 16000, where they
// spill: 5057 4401 15533 -> 5652 4770 18544.  Weighted counts take three up to half
// that: 1000 points, 20 bins 45 37 58 -> 32 24 37, 4100 points, dmax 70, 25 bins 412
// 354 731 -> 377 310 682, 8000: 2133 1732 3980 -> 2111 1618 4036, 30 bins, dmax 80 3568 3104
// 7501 -> 3901 3058 11834; without exact integer weights, bound by atomics in
// global memory, one.  (Four groups of 6 warps and two of 12 lie between.)
// The lists meant are those of uniform catalogs.  bx, by: the longest there can be
// (list_bound), which a dense clump in a large box makes much longer.  Then one group where
//  * the anchors are few, so that a group more is a tail more (clumps of 800 and
//    100000 points, dmax 20: 4432 us by one group, 7939 by three; 2000 and 30000, dmax 15:
//    1722 and 2934; 3000 and 3000: 703 and 582),
//  * the room for all groups' spilled lists grows past 2 GB (of 148 or 444 lists each), or
//  * an anchor's tests may pass a third of the shared counters' budget, which sends
//    its triangles to global memory.
static int trip_groups(pcf_ctx *ctx, const pcf_grid *X, const pcf_grid *Y, int bins, float dmax, bool weighted,
                       int64_t bx, int64_t by) {
    const size_t hist = trip_hist_bytes(bins, weighted);
    if (!hist || (weighted && !limb_budget(X, Y))) return 1;
    const double L = X->box, in = std::min(1.0, 4.18879 * (double)dmax * dmax * dmax / (L * L * L));
    const double list = Y ? (0.5 * (double)X->n + (double)Y->n) * in : (double)X->n * in;
    constexpr int G = kTWarps / kGroupWarps;
    const double room = (double)((kTripSmem - hist) / G / (weighted ? 40 : 16));
    if (list > room) return 1;
    const int64_t longest = std::max(X->n > kCheapBound ? bx : 0, Y && Y->n > kCheapBound ? by : 0);
    if (X->n < (int64_t)6 * G * ctx->sm_count && (double)longest > 2.0 * room) return 1;
    if ((double)longest * 16.0 * (Y ? 2 : 1) * G * ctx->sm_count > 2147483648.0) return 1;
    const double tests = Y ? (double)bx * (double)by : 0.5 * (double)bx * (double)bx;
    return tests <= (double)(1 << 30) / G ? G : 1;
}

// Arguments of one isotropic triplet histogram over the cell structures of
// x (and y for XXY) at P partitions: catalogs, side rules, FP32 windows and
// the shared-memory layout (smem: dynamic bytes).  The buffers (rows,
// counter, histograms, overflow lists) are the caller's.
static void trip_setup(pcf_ctx *ctx, const pcf_grid *X, const pcf_grid *Y, int P, int n_rows, int bins,
                       float dmax, uint32_t flags, bool weighted, TripArgs &A, size_t &smem, int groups = 1) {
    const bool bpc = (flags & PCF_BPC) != 0, mixed = Y != nullptr;
    const CellGrid &gx = *X->cells;
    const CellGrid &gy = mixed ? *Y->cells : gx;
    // side rules: X-X sides need d > 0; X-Y sides only with periodic boxes
    // (3iso_k.cuh:158,160 vs 3isoBPC_k.cuh:165,170)
    PairRule rXX = make_pair_rule(bins, dmax, flags & ~PCF_DS_EXACT, false, bpc, false);
    PairRule rXY = rXX;
    rXY.flags = bpc ? PCF_RULE_EXCL : 0u;
    if (flags & PCF_RULE_CUSTOM) rXY.flags = rXX.flags;
    memset(&A, 0, sizeof(A));
    A.X = {gx.x(), gx.y(), gx.z(), gx.w(), gx.cell_start.as<int>()};
    A.Y = {gy.x(), gy.y(), gy.z(), gy.w(), gy.cell_start.as<int>()};
    A.nX = (int)X->n;
    A.n_rows = n_rows;
    A.P = P;
    A.cell = gx.cell;
    A.box = X->box;
    A.bpc = bpc ? 1 : 0;
    A.rXX = rXX;
    A.rXY = rXY;
    A.flush_budget = ctx->trip_flush_budget;
    A.ctrl = ctx->d_abort;
    A.status = ctx->d_status;
    A.mixed = mixed ? 1 : 0;
    A.fc = trip_cuts(rXX, X->box, dmax, bpc);
    const size_t hist_b = weighted && !limb_budget(X, Y) ? 0 : trip_hist_bytes(bins, weighted);
    A.hist_in_smem = hist_b > 0 ? 1 : 0;
    if (hist_b && weighted) {
        A.wfix = 1;
        A.wunscale = std::ldexp(1.0, -(2 * X->wshift + (mixed ? Y : X)->wshift));
        A.X.w = reinterpret_cast<const float *>(gx.qw.as<unsigned>());
        A.Y.w = reinterpret_cast<const float *>(gy.qw.as<unsigned>());
        A.flush_budget = std::min(A.flush_budget, limb_budget(X, Y));
    }
    const size_t ent = 16 + (weighted ? 4 : 0);
    const size_t room = (kTripSmem - hist_b) / groups;
    if (mixed && !(A.hist_in_smem && !weighted)) {
        A.capJ = (int)(room / ent / 3);
        A.capK = (int)(room / ent) - A.capJ;
    } else {  // XXX, or XXY with one pooled buffer (see tri_anchor)
        A.capJ = (int)(room / ent);
        A.capK = 0;
    }
    A.list_bytes = (int)(((size_t)(A.capJ + A.capK) * ent + 15) & ~(size_t)15);
    if (groups > 1) A.flush_budget = std::min<unsigned long long>(A.flush_budget, 1ull << 30) / (unsigned)groups;
    smem = hist_b + (size_t)A.list_bytes * groups;
}

static void (*trip_kernel(bool mixed, bool weighted, bool several))(const TripArgs) {
    if (several)
        return mixed ? (weighted ? k_triplets<true, true, kGroupWarps> : k_triplets<true, false, kGroupWarps>)
                     : (weighted ? k_triplets<false, true, kGroupWarps> : k_triplets<false, false, kGroupWarps>);
    return mixed ? (weighted ? k_triplets<true, true, kTWarps> : k_triplets<true, false, kTWarps>)
                 : (weighted ? k_triplets<false, true, kTWarps> : k_triplets<false, false, kTWarps>);
}

// Per-group overflow lists for lists of up to gcap entries (J, K and weights).
static pcf_status trip_overflow(pcf_ctx *ctx, int64_t gmax, bool mixed, bool weighted, int grid,
                                TripArgs &A) {
    A.gcap = (int)std::min<int64_t>(gmax, 1 << 24);
    PCF_CU(ctx, ctx->scratch_c.ensure(sizeof(float4) * (size_t)A.gcap * grid * (mixed ? 2 : 1) +
                                      (weighted ? sizeof(float) * (size_t)A.gcap * grid * 2 : 0) + 256));
    char *sc = ctx->scratch_c.as<char>();
    A.gJ = reinterpret_cast<float4 *>(sc);
    A.gK = mixed ? A.gJ + (size_t)A.gcap * grid : nullptr;
    float *wbase = reinterpret_cast<float *>(sc + sizeof(float4) * (size_t)A.gcap * grid * (mixed ? 2 : 1));
    A.gwJ = weighted ? wbase : nullptr;
    A.gwK = weighted && mixed ? wbase + (size_t)A.gcap * grid : nullptr;
    return PCF_OK;
}

static pcf_status count_triplets_ordered(pcf_ctx *ctx, const pcf_grid *x_, const pcf_grid *y_, int bins,
                                         float dmax, uint32_t flags, double *hist, pcf_stats *stats,
                                         bool iso3);

// Entries that the ordered counts' lists hold in shared memory with `ctas` CTAs
// per SM; returns the bytes of one (the row table of the list build takes one of
// them).  Several small CTAs overlap one's list builds with another's counting;
// they are taken where no list can be longer than theirs hold, which leaves the
// calls that the large one refuses as they are.
static size_t ordered_caps(bool mixed, bool weighted, bool gates, int ctas, TripArgs &A) {
    const size_t ent = 16 + 2 + (weighted ? 4 : 0) + (gates ? 4 : 0);
    const size_t fixed = 256 + (gates ? 64 * sizeof(GateBlock) + 128 + 64 : 0);
    const size_t room = ctas == 1 ? 227 * 1024 - fixed
                                  : 228 * 1024 / ctas - 1024 - 256 - sizeof(ListScratch<kGroupWarps>) - fixed;
    if (mixed) {
        A.capJ = (int)(room / ent / 3);
        A.capK = (int)(room / ent) - A.capJ - 8;
    } else {
        A.capJ = (int)(room / ent) - 8;
        A.capK = 0;
    }
    return ent;
}

extern "C" pcf_status pcf_count_triplets(pcf_ctx *ctx, int kind, const pcf_grid *x_,
                                         const pcf_grid *y_, int bins, float dmax, uint32_t flags,
                                         double *hist, pcf_stats *stats) {
    if (!ctx || !x_ || !hist || bins < 1 || !(dmax > 0.f)) return PCF_ERR_INVALID_ARG;
    if (kind == PCF_ANI) return pcf_count_triplets_ani(ctx, x_, y_, bins, dmax, flags, hist, stats);
    if (kind != PCF_ISO) return PCF_ERR_INVALID_ARG;
    // Node gates of unit-weight counts: corrections of the plain count where the
    // gates hold on the grid's nodes; else (weights, whose corrections would
    // cancel; long lists; a touching diagonal; invalid calls) every ordered triangle.
    const bool gates = (flags & PCF_REF_NODE_GATES) != 0;
    auto ordered = [&] { return count_triplets_ordered(ctx, x_, y_, bins, dmax, flags, hist, stats, true); };
    GateGeom geom{};
    if (gates) {
        if (!(flags & PCF_BPC) || x_->user_P < 1 || x_->user_P > 512 || bins > 255 ||
            (int64_t)bins * bins * bins > (1 << 26) ||
            (y_ && (y_->user_P != x_->user_P || y_->box != x_->box)))
            return ordered();
        geom = gate_geometry(x_->box, dmax, x_->user_P);
        if (!gates_hold(geom, make_pair_rule(bins, dmax, flags & ~PCF_DS_EXACT, false, true, false).dd))
            return ordered();
    }
    if (bins > 255 || (int64_t)bins * bins * bins > (1 << 26)) return PCF_ERR_UNSUPPORTED;
    cudaSetDevice(ctx->device);
    {
        pcf_status s0 = grid_finish(ctx, x_);
        if (s0 == PCF_OK && y_) s0 = grid_finish(ctx, y_);
        if (s0 != PCF_OK) return s0;
    }
    pcf_grid *X = const_cast<pcf_grid *>(x_);
    pcf_grid *Y = const_cast<pcf_grid *>(y_);
    const bool bpc = (flags & PCF_BPC) != 0, mixed = Y != nullptr;
    if (X->n >= (1 << 24) || (Y && Y->n >= (1 << 24))) return PCF_ERR_UNSUPPORTED;
    if (ctx_abort_requested(ctx) != PCF_OK) return PCF_ERR_TIMEOUT;
    int P = 0;
    pcf_status s = prepare_grids(ctx, X, Y, dmax, kTripletCells, bpc, &P);
    if (s != PCF_OK) return s;
    const CellGrid &gx = *X->cells;
    const CellGrid &gy = mixed ? *Y->cells : gx;
    PairPlan plan;
    plan_pairs(gx, X->box, dmax, false, false, plan, ctx->sm_count * 24);
    const bool weighted = !(X->unit_weights && (!mixed || Y->unit_weights));
    if (gates && weighted) return ordered();
    TripArgs A;
    size_t smem = 0;
    const int n3 = bins * bins * bins, n_rows = (int)plan.rows.size();
    // rows + counter through the plan slot
    PlanSlot *sl = nullptr;
    s = stage_plan(ctx, plan, &sl);
    if (s != PCF_OK) return s;
    // overflow lists
    int64_t bx = 0, by = 0;
    s = list_bound(ctx, gx, X->n, dmax, sl->rows(), n_rows, bpc, &bx);
    if (s == PCF_OK && mixed) s = list_bound(ctx, gy, Y->n, dmax, sl->rows(), n_rows, bpc, &by);
    const int groups = trip_groups(ctx, X, Y, bins, dmax, weighted, bx, by);
    trip_setup(ctx, X, Y, P, n_rows, bins, dmax, flags, weighted, A, smem, groups);
    A.rows = sl->rows();
    A.counter = sl->counter();
    TripArgs F;  // the gates' corrections
    size_t fix_smem = 0;
    int fix_ctas = kTWarps / kGroupWarps;
    if (s == PCF_OK && gates) {
        int capJ = 0, capK = 0;
        for (;; fix_ctas = 1) {
            ordered_caps(mixed, false, true, fix_ctas, F);
            // an entry also has its place in the order by image (two bytes; the row
            // table's share of the room comes off here)
            capJ = F.capJ - 300;
            capK = mixed ? F.capK : 0;
            int64_t fx = bx, fy = by;
            if (fx > capJ) s = list_bound(ctx, gx, X->n, dmax, A.rows, A.n_rows, bpc, &fx, capJ);
            if (s == PCF_OK && mixed && fy > capK)
                s = list_bound(ctx, gy, Y->n, dmax, A.rows, A.n_rows, bpc, &fy, capK);
            if (s != PCF_OK) return s;
            if (fx <= capJ && (!mixed || fy <= capK)) break;
            if (fix_ctas == 1) return ordered();
        }
        F = A;
        F.capJ = capJ;
        F.capK = capK;
        F.gate = geom;
        fix_smem = (size_t)(capJ + capK) * 20 + 2 * (size_t)(mixed ? capK : capJ);
    }
    const int grid = ctx->sm_count;
    if (s == PCF_OK) s = trip_overflow(ctx, std::max(bx, by) + 32, mixed, weighted, grid * groups, A);
    if (s != PCF_OK) return s;
    // histogram scratch: [u64 n3][f64 n3][stats 8][f64 out n3]
    PCF_CU(ctx, ctx->d_hist.ensure((size_t)n3 * 24 + 64));
    char *hp = ctx->d_hist.as<char>();
    A.g_count = reinterpret_cast<unsigned long long *>(hp);
    A.g_wsum = reinterpret_cast<double *>(hp + (size_t)n3 * 8);
    A.g_stats = reinterpret_cast<unsigned long long *>(hp + (size_t)n3 * 16);
    double *d_out = reinterpret_cast<double *>(hp + (size_t)n3 * 16 + 64);
    PCF_CU(ctx, cudaMemsetAsync(hp, 0, (size_t)n3 * 16 + 64, ctx->stream));
    // unweighted: the sums' place holds the gates' corrections
    unsigned long long *fix = gates ? reinterpret_cast<unsigned long long *>(A.g_wsum) : nullptr;

    const auto kfn = trip_kernel(mixed, weighted, groups > 1);
    PCF_CU(ctx, ensure_smem_limit(reinterpret_cast<const void *>(kfn), ctx->device, smem));
    cudaEvent_t pe0 = nullptr, pe1 = nullptr;
    if (ctx->profile) {
        s = profile_events(ctx, &pe0, &pe1);
        if (s != PCF_OK) return s;
        PCF_CU(ctx, cudaEventRecord(pe0, ctx->stream));
    }
    PCF_CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
    kfn<<<grid, kTThreads, smem, ctx->stream>>>(A);
    PCF_CU(ctx, cudaGetLastError());
    if (gates) {
        F.g_count = fix;
        F.g_stats = A.g_stats;
        F.counter = A.counter + 1;
        const bool few = fix_ctas == 1;
        auto ffn = mixed ? (few ? k_gate_fix<kTWarps, true> : k_gate_fix<kGroupWarps, true>)
                         : (few ? k_gate_fix<kTWarps, false> : k_gate_fix<kGroupWarps, false>);
        PCF_CU(ctx, ensure_smem_limit(reinterpret_cast<const void *>(ffn), ctx->device, fix_smem));
        const float reach = (float)(std::sqrt(A.rXX.dd) * (1.0 + 1e-6) + (double)A.box * 1e-6);
        ffn<<<grid * fix_ctas, kTThreads / fix_ctas, fix_smem, ctx->stream>>>(F, reach);
        PCF_CU(ctx, cudaGetLastError());
        ++ctx->launches;
    }
    PCF_CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    if (pe1) PCF_CU(ctx, cudaEventRecord(pe1, ctx->stream));
    PCF_CU(ctx, cudaEventRecord(sl->done, ctx->stream));
    ++ctx->launches;
    const bool dev_out = (flags & PCF_DEVICE_OUT) != 0;
    OutPath o;
    s = out_open(ctx, n3, dev_out, hist, d_out, &o);
    if (s != PCF_OK) return s;
    k_trip_finalize<<<(n3 + 255) / 256, 256, 0, ctx->stream>>>(A.g_count, A.g_wsum, weighted ? 1 : 0,
                                                                mixed ? 1 : 0, bins, o.to, A.g_stats,
                                                                stats || !dev_out || gates ? o.stats : nullptr, fix);
    PCF_CU(ctx, cudaGetLastError());
    ++ctx->launches;
    if (stats || !dev_out || gates) {
        unsigned long long hs[4];
        s = out_close(ctx, o, n3, dev_out, hist, hs);
        if (s != PCF_OK) return s;
        if (gates && hs[3]) return PCF_ERR_UNSUPPORTED;
        if (stats) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
            stats->pairs = (double)hs[2];  // unordered triangles (XXY: per unordered XX pair)
            if (gates) stats->pairs = (double)(hs[2] * (mixed ? 2 : 6) + hs[1]);  // counts of ordered ones
            stats->candidates = 0;
            stats->rechecks = (double)hs[0];
            stats->kernel_ms = ms;
            stats->partitions = P;
            stats->work_items = (int)X->n;
        }
    }
    return PCF_OK;
}

// One data catalog against n_rand random catalogs: DDD once, RRR_i, DDR_i
// and DRR_i per random catalog: their kernels queued one behind the other, one
// wait for all.  All grids take one partition count (the one a call on the largest
// catalog would use; results do not depend on it).  (All jobs' anchors as one queue
// of a persistent launch saved the tails between kernels, but a CTA's groups of
// warps had to stay in one job: 32768 points against 8 randoms of 4k to 32k, dmax 40 of
// 250, 20 bins 84.6 ms; 53.7 so.)
extern "C" pcf_status pcf_batch_triplets(pcf_ctx *ctx, const pcf_grid *d_, const pcf_grid *const *r_,
                                         int n_rand, int bins, float dmax, uint32_t flags, double *ddd,
                                         double *rrr, double *ddr, double *drr, pcf_stats *stats) {
    if (!ctx || !d_ || bins < 1 || !(dmax > 0.f) || n_rand < 0 || (n_rand > 0 && !r_) ||
        (!ddd && !rrr && !ddr && !drr))
        return PCF_ERR_INVALID_ARG;
    if (bins > 255 || (int64_t)bins * bins * bins > (1 << 26)) return PCF_ERR_UNSUPPORTED;
    if (flags & PCF_REF_NODE_GATES) {
        ctx->last_error = "PCF_REF_NODE_GATES counts run per call (pcf_count_triplets)";
        return PCF_ERR_UNSUPPORTED;
    }
    if (ctx_abort_requested(ctx) != PCF_OK) return PCF_ERR_TIMEOUT;
    cudaSetDevice(ctx->device);
    {
        pcf_status s0 = grid_finish(ctx, d_);
        for (int i = 0; s0 == PCF_OK && i < n_rand; ++i)
            if (r_[i]) s0 = grid_finish(ctx, r_[i]);
        if (s0 != PCF_OK) return s0;
    }
    const bool bpc = (flags & PCF_BPC) != 0;
    pcf_grid *D = const_cast<pcf_grid *>(d_);
    std::vector<pcf_grid *> R((size_t)n_rand);
    pcf_grid *big = D;
    bool weighted = !D->unit_weights;
    for (int i = 0; i < n_rand; ++i) {
        R[i] = const_cast<pcf_grid *>(r_[i]);
        if (!R[i]) return PCF_ERR_INVALID_ARG;
        if (R[i]->box != D->box) return PCF_ERR_MISMATCH;
        if (R[i]->n >= (1 << 24)) return PCF_ERR_UNSUPPORTED;
        if (R[i]->n > big->n) big = R[i];
        weighted = weighted || !R[i]->unit_weights;
    }
    if (D->n >= (1 << 24)) return PCF_ERR_UNSUPPORTED;
    int P = 0;
    pcf_status s = prepare_grids(ctx, big, nullptr, dmax, kTripletCells, bpc, &P);
    if (s != PCF_OK) return s;
    // every structure queued before the first is completed
    if ((s = grid_ensure_cells(ctx, D, P, true)) != PCF_OK) return s;
    for (pcf_grid *g : R)
        if ((s = grid_ensure_cells(ctx, g, P, true)) != PCF_OK) return s;
    if ((s = grid_finish(ctx, D)) != PCF_OK) return s;
    for (pcf_grid *g : R)
        if ((s = grid_finish(ctx, g)) != PCF_OK) return s;
    PairPlan plan;
    plan_pairs(*D->cells, D->box, dmax, false, false, plan, ctx->sm_count * 24);
    const int n3 = bins * bins * bins;

    // jobs: (X, Y) in output order
    struct Job { pcf_grid *x, *y; double *out; };
    std::vector<Job> jobs;
    if (ddd) jobs.push_back({D, nullptr, ddd});
    for (int i = 0; i < n_rand; ++i) {
        if (rrr) jobs.push_back({R[i], nullptr, rrr + (size_t)i * n3});
        if (ddr) jobs.push_back({D, R[i], ddr + (size_t)i * n3});
        if (drr) jobs.push_back({R[i], D, drr + (size_t)i * n3});
    }
    const int nj = (int)jobs.size();
    std::vector<TripArgs> args((size_t)nj);
    long long anchors = 0;
    bool any_mixed = false;
    int most = 1;
    std::vector<size_t> smem((size_t)nj);
    std::vector<int> groups((size_t)nj);
    // rows + counters through the plan slot
    PlanSlot *sl = nullptr;
    s = stage_plan(ctx, plan, &sl);
    if (s != PCF_OK) return s;
    auto bound = [&](const pcf_grid *g, int64_t *b) {
        return list_bound(ctx, *g->cells, g->n, dmax, sl->rows(), (int)plan.rows.size(), bpc, b);
    };
    int64_t gmax = 0, bD = 0;
    s = bound(D, &bD);
    if (s != PCF_OK) return s;
    gmax = bD;
    std::map<const pcf_grid *, int64_t> bounds{{D, bD}};
    for (pcf_grid *g : R) {
        int64_t b = 0;
        s = bound(g, &b);
        if (s != PCF_OK) return s;
        gmax = std::max(gmax, b);
        bounds[g] = b;
    }
    for (int k = 0; k < nj; ++k) {
        groups[k] = trip_groups(ctx, jobs[k].x, jobs[k].y, bins, dmax, weighted, bounds[jobs[k].x],
                                jobs[k].y ? bounds[jobs[k].y] : 0);
        trip_setup(ctx, jobs[k].x, jobs[k].y, P, (int)plan.rows.size(), bins, dmax, flags, weighted,
                   args[k], smem[k], groups[k]);
        most = std::max(most, groups[k]);
        anchors += jobs[k].x->n;
        any_mixed = any_mixed || jobs[k].y;
    }
    const int grid = ctx->sm_count;
    TripArgs ov;
    s = trip_overflow(ctx, gmax + 32, any_mixed, weighted, grid * most, ov);
    if (s != PCF_OK) return s;

    // histograms per job, a counter per job, statistics, results
    const size_t nh = (size_t)nj * n3, cb = ((size_t)nj * 8 + 63) & ~(size_t)63;
    PCF_CU(ctx, ctx->d_hist.ensure(nh * 24 + cb + 64));
    char *hp = ctx->d_hist.as<char>();
    unsigned long long *cnt = reinterpret_cast<unsigned long long *>(hp);
    double *wsum = reinterpret_cast<double *>(hp + nh * 8);
    unsigned long long *ctr = reinterpret_cast<unsigned long long *>(hp + nh * 16);
    unsigned long long *gstats = reinterpret_cast<unsigned long long *>(hp + nh * 16 + cb);
    double *d_out = reinterpret_cast<double *>(hp + nh * 16 + cb + 64);
    PCF_CU(ctx, cudaMemsetAsync(hp, 0, nh * 16 + cb + 64, ctx->stream));
    for (int k = 0; k < nj; ++k) {
        TripArgs &A = args[k];
        A.gcap = ov.gcap;
        A.gJ = ov.gJ;
        A.gK = ov.gK;
        A.gwJ = ov.gwJ;
        A.gwK = ov.gwK;
        A.rows = sl->rows();
        A.counter = ctr + k;
        A.g_count = cnt + (size_t)k * n3;
        A.g_wsum = wsum + (size_t)k * n3;
        A.g_stats = gstats;
    }
    cudaEvent_t pe0 = nullptr, pe1 = nullptr;
    if (ctx->profile) {
        s = profile_events(ctx, &pe0, &pe1);
        if (s != PCF_OK) return s;
        PCF_CU(ctx, cudaEventRecord(pe0, ctx->stream));
    }
    PCF_CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
    for (int k = 0; k < nj; ++k) {
        const auto kfn = trip_kernel(jobs[k].y != nullptr, weighted, groups[k] > 1);
        PCF_CU(ctx, ensure_smem_limit(reinterpret_cast<const void *>(kfn), ctx->device, smem[k]));
        kfn<<<grid, kTThreads, smem[k], ctx->stream>>>(args[k]);
        PCF_CU(ctx, cudaGetLastError());
        ++ctx->launches;
    }
    PCF_CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    if (pe1) PCF_CU(ctx, cudaEventRecord(pe1, ctx->stream));
    PCF_CU(ctx, cudaEventRecord(sl->done, ctx->stream));
    for (int k = 0; k < nj; ++k) {
        k_trip_finalize<<<(n3 + 255) / 256, 256, 0, ctx->stream>>>(
            cnt + (size_t)k * n3, wsum + (size_t)k * n3, weighted ? 1 : 0, jobs[k].y ? 1 : 0, bins,
            d_out + (size_t)k * n3, nullptr, nullptr, nullptr);
        PCF_CU(ctx, cudaGetLastError());
        ++ctx->launches;
    }
    std::vector<char> spill;
    const char *hb = nullptr;
    s = fetch_block(ctx, gstats, 64 + sizeof(double) * nh, spill, &hb);  // [stats | out]
    if (s == PCF_OK) s = ctx_queue_status(ctx);
    if (s != PCF_OK) return s;
    unsigned long long hs[4];
    memcpy(hs, hb, sizeof(hs));
    for (int k = 0; k < nj; ++k) memcpy(jobs[k].out, hb + 64 + (size_t)k * n3 * sizeof(double), sizeof(double) * n3);
    if (stats) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        stats->pairs = (double)hs[2];
        stats->candidates = 0;
        stats->rechecks = (double)hs[0];
        stats->kernel_ms = ms;
        stats->partitions = P;
        stats->work_items = (int)std::min<long long>(anchors, INT32_MAX);
    }
    return PCF_OK;
}

template <int NW>
static void (*ordered_kernel(bool mixed, bool weighted, bool gates, bool iso3))(const TripArgs) {
    if (iso3)
        return mixed ? (weighted ? k_triplets_ani<NW, true, true, true, true> : k_triplets_ani<NW, true, false, true, true>)
                     : (weighted ? k_triplets_ani<NW, false, true, true, true>
                                 : k_triplets_ani<NW, false, false, true, true>);
    if (gates)
        return mixed ? (weighted ? k_triplets_ani<NW, true, true, true> : k_triplets_ani<NW, true, false, true>)
                     : (weighted ? k_triplets_ani<NW, false, true, true> : k_triplets_ani<NW, false, false, true>);
    return mixed ? (weighted ? k_triplets_ani<NW, true, true> : k_triplets_ani<NW, true, false>)
                 : (weighted ? k_triplets_ani<NW, false, true> : k_triplets_ani<NW, false, false>);
}

// Anisotropic triplets (bins^5).  The histogram lives in global memory (u64
// counts or FP64 sums); lists stay in shared memory (an anchor whose lists
// do not fit makes the call fail with PCF_ERR_UNSUPPORTED).
// Ordered-triangle counts through k_triplets_ani: the bins^5 anisotropic
// histogram, or (iso3, with PCF_REF_NODE_GATES) the bins^3 isotropic one.
static pcf_status count_triplets_ordered(pcf_ctx *ctx, const pcf_grid *x_, const pcf_grid *y_, int bins,
                                         float dmax, uint32_t flags, double *hist, pcf_stats *stats,
                                         bool iso3) {
    const int64_t nh = iso3 ? (int64_t)bins * bins * bins : (int64_t)bins * bins * bins * bins * bins;
    if (bins > 255 || nh > ((int64_t)1 << 31)) return PCF_ERR_UNSUPPORTED;
    const bool gates = (flags & PCF_REF_NODE_GATES) != 0;
    if (gates) {
        if (!(flags & PCF_BPC)) {
            ctx->last_error = "PCF_REF_NODE_GATES applies to periodic counts (PCF_BPC)";
            return PCF_ERR_INVALID_ARG;
        }
        if (x_->user_P < 1 || x_->user_P > 512 ||
            (y_ && (y_->user_P != x_->user_P || y_->box != x_->box))) {
            ctx->last_error = "PCF_REF_NODE_GATES: the reference's node grid is the partitions given to "
                              "pcf_grid_build (1 to 512), the same for both grids";
            return PCF_ERR_INVALID_ARG;
        }
    }
    cudaSetDevice(ctx->device);
    {
        pcf_status s0 = grid_finish(ctx, x_);
        if (s0 == PCF_OK && y_) s0 = grid_finish(ctx, y_);
        if (s0 != PCF_OK) return s0;
    }
    pcf_grid *X = const_cast<pcf_grid *>(x_);
    pcf_grid *Y = const_cast<pcf_grid *>(y_);
    const bool bpc = (flags & PCF_BPC) != 0, mixed = Y != nullptr;
    if (X->n >= (1 << 24) || (Y && Y->n >= (1 << 24))) return PCF_ERR_UNSUPPORTED;
    if (ctx_abort_requested(ctx) != PCF_OK) return PCF_ERR_TIMEOUT;
    int P = 0;
    pcf_status s = prepare_grids(ctx, X, Y, dmax, kTripletCells, bpc, &P);
    if (s != PCF_OK) return s;
    const CellGrid &gx = *X->cells;
    const CellGrid &gy = mixed ? *Y->cells : gx;
    PairPlan plan;
    plan_pairs(gx, X->box, dmax, false, false, plan, ctx->sm_count * 24);
    PairRule rXX = make_pair_rule(bins, dmax, flags & ~PCF_DS_EXACT, false, bpc, false);
    PairRule rXY = rXX;
    rXY.flags = bpc ? PCF_RULE_EXCL : 0u;
    if (flags & PCF_RULE_CUSTOM) rXY.flags = rXX.flags;
    TripArgs A;
    memset(&A, 0, sizeof(A));
    A.X = {gx.x(), gx.y(), gx.z(), gx.w(), gx.cell_start.as<int>()};
    A.Y = {gy.x(), gy.y(), gy.z(), gy.w(), gy.cell_start.as<int>()};
    A.nX = (int)X->n;
    A.n_rows = (int)plan.rows.size();
    A.P = P;
    A.cell = gx.cell;
    A.box = X->box;
    A.bpc = bpc ? 1 : 0;
    A.rXX = rXX;
    A.rXY = rXY;
    A.ctrl = ctx->d_abort;
    A.status = ctx->d_status;
    if (gates) A.gate = gate_geometry(X->box, dmax, X->user_P);
    A.fc = trip_cuts(rXX, X->box, dmax, bpc);
    const bool weighted = !(X->unit_weights && (!mixed || Y->unit_weights));
    const int64_t n5 = nh;
    PlanSlot *sl = nullptr;
    s = stage_plan(ctx, plan, &sl);
    if (s != PCF_OK) return s;
    A.rows = sl->rows();
    A.counter = sl->counter();
    int ctas = kTWarps / kGroupWarps;
    size_t ent = ordered_caps(mixed, weighted, gates, ctas, A);
    int64_t bx = 0, by = 0;
    s = list_bound(ctx, gx, X->n, dmax, A.rows, A.n_rows, bpc, &bx, A.capJ);
    if (s == PCF_OK && mixed) s = list_bound(ctx, gy, Y->n, dmax, A.rows, A.n_rows, bpc, &by, A.capK);
    if (s != PCF_OK) return s;
    if (bx > A.capJ || (mixed && by > A.capK)) {
        ctas = 1;
        ent = ordered_caps(mixed, weighted, gates, ctas, A);
    }
    // (an entry's angle bin takes one of the two bytes `ent` counts)
    const size_t smem = (size_t)(A.capJ + A.capK) * (ent - 1) + 64;
    PCF_CU(ctx, ctx->d_hist.ensure((size_t)n5 * 16 + 128));
    char *hp = ctx->d_hist.as<char>();
    A.g_count = reinterpret_cast<unsigned long long *>(hp);
    A.g_wsum = reinterpret_cast<double *>(hp);  // one of the two is used
    A.g_stats = reinterpret_cast<unsigned long long *>(hp + (size_t)n5 * 8);
    double *d_out = reinterpret_cast<double *>(hp + (size_t)n5 * 8 + 128);
    PCF_CU(ctx, cudaMemsetAsync(hp, 0, (size_t)n5 * 8 + 128, ctx->stream));
    const auto kfn = ctas == 1 ? ordered_kernel<kTWarps>(mixed, weighted, gates, iso3)
                               : ordered_kernel<kGroupWarps>(mixed, weighted, gates, iso3);
    PCF_CU(ctx, ensure_smem_limit(reinterpret_cast<const void *>(kfn), ctx->device, smem));
    PCF_CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
    kfn<<<ctx->sm_count * ctas, kTThreads / ctas, smem, ctx->stream>>>(A);
    PCF_CU(ctx, cudaGetLastError());
    PCF_CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    PCF_CU(ctx, cudaEventRecord(sl->done, ctx->stream));
    const bool dev_out = (flags & PCF_DEVICE_OUT) != 0, half = !mixed && !gates;
    OutPath o;
    s = out_open(ctx, n5, dev_out, hist, d_out, &o);
    if (s != PCF_OK) return s;
    k_to_double<<<(unsigned)((n5 + 255) / 256), 256, 0, ctx->stream>>>(A.g_count, A.g_wsum, weighted ? 1 : 0, n5, o.to,
                                                                       A.g_stats, o.stats, half ? bins : 0);
    PCF_CU(ctx, cudaGetLastError());
    ctx->launches += 2;
    unsigned long long hs[4];
    s = out_close(ctx, o, n5, dev_out, hist, hs);
    if (s != PCF_OK) return s;
    if (hs[3]) {
        ctx->last_error = "neighbour lists of the anisotropic triplet kernel exceed shared memory";
        return PCF_ERR_UNSUPPORTED;
    }
    if (stats) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        stats->pairs = (double)hs[2] * (half ? 2 : 1);  // ordered triangles
        stats->rechecks = (double)hs[0];
        stats->candidates = 0;
        stats->kernel_ms = ms;
        stats->partitions = P;
        stats->work_items = (int)X->n;
    }
    return PCF_OK;
}

pcf_status pcf_count_triplets_ani(pcf_ctx *ctx, const pcf_grid *x_, const pcf_grid *y_, int bins,
                                  float dmax, uint32_t flags, double *hist, pcf_stats *stats) {
    return count_triplets_ordered(ctx, x_, y_, bins, dmax, flags, hist, stats, false);
}
