// pairs_lean.cuh -- the pair kernel of unit weights and of weights with exact
// integer images, at the bin counts where its copies leave room for enough warps
// (lean_columns in pairs.cu, which holds the windows and the general kernel for
// everything else).
//
// Same work items as the general kernel: one warp takes (home tile, stencil
// rows), one home point per lane, candidates two at a time as packed f32x2.
// The candidate loop is what is different:
//  * Nothing is selected or predicated per pair.  The fixed-point readout
//    r + magic is clamped to bins + 1/2, so a pair out of range adds to a
//    counter past the last bin that is never read; a pair inside an edge window
//    is added where the fast path has it, queued, and moved by the FP64 rule,
//    32 queued pairs at a time (one lane alone cost its warp 500 instructions).
//  * The counter's address is one FMA per readout: the readout with its
//    fraction cleared is the float magic + bin, and an FMA with the stride and
//    the base as denormals (multiples of 2^-149) leaves the address in the bits.
//  * Unit weights add the constant 1: the hardware then adds lanes that hit one
//    counter together (1 cycle where a register operand takes one per lane), so
//    neither kind needs private columns.
//  * Weighted sums: the exact 64-bit product q_a * q_b goes into 32-bit limbs
//    with carries -- an add that returns the old value tells the carry -- two
//    reductions instead of three 16/16/32-bit ones.  Isotropic: two limbs in
//    columns private to the lane (or to two or four), flushed before the upper one could wrap.
//    Anisotropic: a third limb takes the rare carry out of the second, so it is
//    never flushed before the job ends.
//  * Candidates are staged into shared memory by cp.async, 32 at a time, the next
//    window (across rows) on its way while one is counted: an L2 access takes
//    longer than the registers of a prefetch can cover.
//  * Both kinds come from one pass: its candidate tests and products are shared.
//  * The anisotropic copy is shared by the CTA's warps (a reduction costs the
//    same whichever warps share a copy), so 16 to 20 warps are resident at any
//    usual bin count; the warps of a CTA that has one meet where their items leave a job.
// What bounds it: instruction issue (67 to 74% of slots at 16 to 20 warps; the
// general kernel 37 to 61% with half as many instructions again) and, for
// weighted anisotropic counts, the shared-memory pipe beside it (76 to 86%: two
// returning adds to scattered counters per pair).
// Kernel time of one DR histogram, general -> this (us, one B200): periodic,
// 32768 + 32768 points, 30 bins, dmax 80, weighted: isotropic 679 -> 569,
// anisotropic 931 -> 734, both 1379 (one pass) -> 1083; 100003 + 200000 points,
// box 1000, 40 bins, dmax 120, weighted, anisotropic: 1488 -> 822; 200001 +
// 300000 points, periodic, 50 bins, dmax 100, unit weights: isotropic 1013 -> 703,
// anisotropic 1400 -> 883.
//
// Unit and weighted counts are compiled in files of their own (pairs_lean_unit.cu,
// pairs_lean_weighted.cu): a process loads a file's kernels with the first of them
// it launches, and with the general kernel and the last kernel of every count they
// had grown to a 14 MB module, which took the first count of a process 15 ms to
// load (unit weights, without them: 0.8 ms).
#pragma once

#include "pairs_common.cuh"

cudaError_t launch_lean_unit(const PairArgs &A, const PairLaunch &pl, cudaStream_t st, int sm_count, int device);
// nc: lean_columns
cudaError_t launch_lean_weighted(const PairArgs &A, const PairLaunch &pl, int nc, cudaStream_t st, int sm_count,
                                 int device);

namespace {

// CTA shapes, steps per vote and resident CTAs.  Weighted: 8 warps, two CTAs at
// 128 registers (the anisotropic copy is large, so few CTAs share an SM); unit: 4
// warps, five CTAs at 96.  Four steps (8 candidates per lane) per vote: one took
// 35% longer, two 10%, eight spilled.
template <bool W>
struct LeanShape {
    static constexpr int warps = W ? 8 : 4, threads = 32 * warps, ctas = W ? 2 : 5;
};
constexpr int kN = 4;
constexpr int kLQueue = 64;   // pairs waiting for the FP64 rule, per warp

// A pair inside a window.  home, cand: points, with the candidate's x / y image
// (0 -L, 1 none, 2 +L) above bit 29; code: the fast path's bins, perpendicular
// and z (8 bits each) and isotropic (9), the lane whose column it went to (5), z image (2).
struct LeanQueued {
    unsigned home, cand, code;
};

// One contiguous candidate range of an item: [a, b) with its image shift; fwd:
// the forward half of the home column (candidates after the home point only).
struct LeanRange {
    int a, b;
    float sx, sy, sz;
    int fwd;
};

constexpr int kWindow = 32;  // candidates staged at a time

struct LeanWarp {
    float4 pts[2][kWindow];      // two windows of pair-packed candidates
    unsigned q[2][kWindow];      // and their integer weights
    float4 home[32];
    LeanRange ranges[64];        // the item's rows, two ranges each at most, without the empty ones
    LeanQueued queue[kLQueue];
};

// Shared-memory layout of one CTA (after the static part): isotropic copies per
// warp, then the CTA's anisotropic copy; in bytes.
// NC columns of two limbs per isotropic bin (weighted): 32, or fewer where that
// is what lets two CTAs share an SM (lanes l and l + NC then share one).
template <int KIND, bool W, int NC>
struct LeanCopies {
    static constexpr int iso_slot = W ? 8 * NC : 4;   // [bin][limb][column] or [bin]
    static constexpr int ani_slot = W ? 12 : 4;    // [z][perp][limb] or [z][perp]
    // Rows and columns past the last bin: pairs out of range go to row or column
    // bins + lane % pad.  Weighted adds of many lanes to one counter serialise
    // (unit ones merge), so these spread.
    static constexpr int pad = W ? 8 : 1;  // (kMag + bins + pad stays in the magic's binade)
    __host__ __device__ static int row(int bins) { return bins + pad; }
    __host__ __device__ static int iso_warp(int bins) { return KIND == K_ANI ? 0 : (bins + 1) * iso_slot; }
    __host__ __device__ static int ani(int bins) { return KIND == K_ISO ? 0 : row(bins) * row(bins) * ani_slot; }
    __host__ __device__ static int bytes(int bins) { return (LeanShape<W>::warps * iso_warp(bins) + ani(bins) + 15) & ~15; }
};

// An integer of magnitude below 2^23 as a multiple of 2^-149.
__device__ __forceinline__ float tiny_of(int n) { return __int_as_float(n < 0 ? (int)(0x80000000u | (unsigned)-n) : n); }

__device__ __forceinline__ unsigned atom_s_u32(unsigned a, unsigned v) {
    unsigned old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(v));
    return old;
}
__device__ __forceinline__ void red_s_one(unsigned a) { asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(a)); }

// The second half of a two-limb add: old is what the lower limb held.
__device__ __forceinline__ unsigned carry_of(unsigned old, unsigned lo) { return old + lo < lo ? 1u : 0u; }

// v added to (or, neg, taken from) the limbs at byte addresses a, a + D,
// a + 2 D (the third if LIMBS == 3).
template <int LIMBS, int D>
__device__ __forceinline__ void add_limbs(unsigned a, unsigned long long v, bool neg) {
    const unsigned long long x = neg ? 0ull - v : v;
    const unsigned lo = (unsigned)x, hi = (unsigned)(x >> 32);
    const unsigned c = carry_of(atom_s_u32(a, lo), lo);
    if (LIMBS == 2) {
        red_s_u32(a + D, hi + c);
    } else {
        const unsigned h = hi + c, old = atom_s_u32(a + D, h);
        // the limbs above the product's: its sign, and the carry out of the second
        const unsigned up = (neg && v ? 0xffffffffu : 0u) + (h < c ? 1u : 0u) + carry_of(old, h);
        if (up) red_s_u32(a + 2 * D, up);
    }
}

// The FP64 rule for n queued pairs, one per lane: a pair that belongs elsewhere
// than the fast path put it is moved.  Returns the change of this lane's count
// of pairs in range.
template <int KIND, bool W, int NC>
__device__ __noinline__ int lean_settle(const PairArgs &A, const PairJob &J, const LeanQueued *q, int n,
                                        unsigned iso_copy, unsigned ani_copy) {
    constexpr bool DO_I = KIND != K_ANI, DO_A = KIND != K_ISO;
    typedef LeanCopies<KIND, W, NC> Copies;
    const int lane = threadIdx.x & 31, bins = A.rule.bins, row1 = Copies::row(bins);
    if (lane >= n) return 0;
    int change = 0;
    const LeanQueued t = q[lane];
    const int hi = (int)(t.home & 0x3FFFFFFFu), cj = (int)(t.cand & 0x3FFFFFFFu);
    const float sx = (float)((int)(t.home >> 30) - 1) * A.box, sy = (float)((int)(t.cand >> 30) - 1) * A.box;
    const float sz = (float)((int)(t.code >> 30) - 1) * A.box;
    float hx, hy, hz, hw, cx, cy, cz, cw;
    load_point(J.home.pk, hi, hx, hy, hz, hw);
    load_point(J.cand.pk, cj, cx, cy, cz, cw);
    const unsigned long long v = W ? (unsigned long long)__ldg(J.home.qw + hi) * __ldg(J.cand.qw + cj) : 1ull;
    PairRule rule = A.rule;
    if (DO_I) {
        rule.flags = J.rule_flags;
        const int s = slow_slot<false>(hx, hy, hz, cx, cy, cz, sx, sy, sz, rule);
        const int fast = (int)((t.code >> 16) & 511u), to = s >= 0 ? s : bins;
        if (to != fast) {
            const unsigned col = iso_copy + (W ? ((t.code >> 25) & (NC - 1)) * 4u : 0u);
            if (W) {
                add_limbs<2, 4 * NC>(col + fast * Copies::iso_slot, v, true);
                add_limbs<2, 4 * NC>(col + to * Copies::iso_slot, v, false);
            } else {
                red_s_u32(col + fast * 4u, 0xffffffffu);
                red_s_u32(col + to * 4u, 1u);
            }
            change += (to < bins) - (fast < bins);
        }
    }
    if (DO_A) {
        rule.flags = KIND == K_BOTH ? J.rule_flags2 : J.rule_flags;
        const int s = slow_slot<true>(hx, hy, hz, cx, cy, cz, sx, sy, sz, rule);
        const int fz = (int)((t.code >> 8) & 255u), fp = (int)(t.code & 255u);  // bins past the last: bins
        const bool was = fz < bins && fp < bins;
        const int fast = was ? fz * row1 + fp : bins * row1 + bins;
        const int to = s >= 0 ? s / bins * row1 + s % bins : bins * row1 + bins;
        if (to != fast) {
            if (W) {
                add_limbs<3, 4>(ani_copy + fast * 12u, v, true);
                add_limbs<3, 4>(ani_copy + to * 12u, v, false);
            } else {
                red_s_u32(ani_copy + fast * 4u, 0xffffffffu);
                red_s_u32(ani_copy + to * 4u, 1u);
            }
            change += (s >= 0) - was;
        }
    }
    return change;
}

template <int KIND, bool W, bool COUNT, int FB, int NC>
__global__ void __launch_bounds__(LeanShape<W>::threads, LeanShape<W>::ctas) k_pairs_lean(const __grid_constant__ PairArgs A) {
    constexpr bool DO_I = KIND != K_ANI, DO_A = KIND != K_ISO;
    typedef LeanCopies<KIND, W, NC> Copies;
    constexpr int kLWarps = LeanShape<W>::warps, kLThreads = LeanShape<W>::threads;
    constexpr int kMag = FB == 16 ? 128 : 256;
    constexpr unsigned kMask = (1u << FB) - 1u, kBias = (FB == 16 ? 0x43000000u : 0x43800000u) >> FB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ LeanWarp s_w[kLWarps];
    // The job being counted: the CTA's where its warps share a copy (MEET), else each
    // warp's own.  A CTA that counts one job at a time leaves most of its warps waiting
    // where jobs are small: a batch of 100 catalogs of 250 to 940 points, exact weights,
    // isotropic, took 752 us so, 211 with a job per warp (and the cheaper flush below).
    constexpr bool MEET = DO_A;
    __shared__ PairJob s_job[MEET ? 1 : kLWarps];
    __shared__ int s_want[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    LeanWarp &ws = s_w[warp];
    PairJob &J = s_job[MEET ? 0 : warp];
    const int bins = A.rule.bins, row1 = Copies::row(bins);
    const int nbi = bins, nbt = (DO_I ? bins : 0) + (DO_A ? bins * bins : 0);
    unsigned char *iso_copy = smem_raw + warp * Copies::iso_warp(bins);
    unsigned char *ani_copy = smem_raw + kLWarps * Copies::iso_warp(bins);
    for (int k = tid; k < Copies::bytes(bins) / 4; k += kLThreads) reinterpret_cast<unsigned *>(smem_raw)[k] = 0u;
    if (tid < 2) s_want[tid] = INT_MAX;
    const int iso_base = (int)__cvta_generic_to_shared(iso_copy) + (W ? (lane & (NC - 1)) * 4 : 0);
    const int ani_base = (int)__cvta_generic_to_shared(ani_copy);
    const float ci = tiny_of(Copies::iso_slot), bi = tiny_of(iso_base - kMag * Copies::iso_slot);
    const float cz = tiny_of(row1 * Copies::ani_slot), cp = tiny_of(Copies::ani_slot);
    const float ba = tiny_of(ani_base - kMag * Copies::ani_slot * (row1 + 1));
    const float qout = (float)kMag + (float)bins + 0.5f, aout = qout + (float)(lane % Copies::pad);
    unsigned long long n_cand = 0;
    int n_pairs = 0;
    unsigned n_rechk = 0;
    long long n_pairs_all = 0;
    int queued = 0;

    // ---- rare parts -------------------------------------------------------
    auto settle = [&](int from, int n) {
        __syncwarp();
        const int d = lean_settle<KIND, W, NC>(A, J, ws.queue + from, n, (unsigned)__cvta_generic_to_shared(iso_copy),
                                               (unsigned)ani_base);
        if (COUNT) n_pairs += d;
        __syncwarp();
    };
    auto drain = [&]() {
        if (queued) settle(0, queued);
        queued = 0;
    };
    // Adds an exact weighted sum to a bin: 128 bits in g_count (low) and g_wsum's
    // place (high), which the finalize kernels convert (exact_sum).
    auto add_exact = [&](size_t bin, unsigned long long lo, unsigned long long hi) {
        const unsigned long long old = atomicAdd(A.g_count + bin, lo);
        hi += old > ~lo ? 1u : 0u;
        if (hi) atomicAdd(reinterpret_cast<unsigned long long *>(A.g_wsum) + bin, hi);
    };
    // Adds this warp's isotropic copy into job slot J.slot and clears it.
    auto flush_iso = [&]() {
        if (!DO_I) return;
        __syncwarp();
        const size_t off = (size_t)J.slot * nbt;
        if (!W) {
            unsigned *c = reinterpret_cast<unsigned *>(iso_copy);
            for (int k = lane; k < bins; k += 32) {
                const unsigned v = c[k];
                c[k] = 0u;
                if (v) atomicAdd(A.g_count + off + k, (unsigned long long)v);
            }
        } else {
            // a bin per lane, its columns from a different one on in each lane (a bin
            // per column group and shuffles took four times the instructions)
            unsigned *c = reinterpret_cast<unsigned *>(iso_copy);
            for (int k = lane; k < bins; k += 32) {
                unsigned long long lo = 0, hi = 0;
                #pragma unroll 4
                for (int o = 0; o < NC; ++o) {
                    unsigned *p = c + 2 * NC * k + ((o + lane) & (NC - 1));
                    lo += p[0];
                    hi += p[NC];
                    p[0] = p[NC] = 0u;
                }
                hi += lo >> 32;
                if (hi | lo) add_exact(off + k, hi << 32 | (lo & 0xffffffffull), hi >> 32);
            }
        }
        __syncwarp();
    };
    // Adds the CTA's anisotropic copy into job slot J.slot and clears it, shared
    // out to `nthr` threads; each counter is exchanged, so other warps may add
    // meanwhile (unit counts are signed: a queued pair may be taken back after).
    auto flush_ani = [&](int t, int nthr) {
        if (!DO_A) return;
        const size_t off = (size_t)J.slot * nbt + (DO_I ? nbi : 0);
        unsigned *c = reinterpret_cast<unsigned *>(ani_copy);
        for (int k = t; k < bins * bins; k += nthr) {
            const int z = k / bins, s = z * row1 + (k - z * bins);
            if (!W) {
                const int v = (int)atomicExch(c + s, 0u);
                if (v) atomicAdd(A.g_count + off + k, (unsigned long long)(long long)v);
            } else {
                const unsigned l0 = c[3 * s], l1 = c[3 * s + 1], l2 = c[3 * s + 2];
                c[3 * s] = c[3 * s + 1] = c[3 * s + 2] = 0u;
                if (l0 | l1 | l2) add_exact(off + k, (unsigned long long)l1 << 32 | l0, l2);
            }
        }
    };

    // ---- work queue: tickets as in the general kernel ------------------------
    auto ticket_items = [&](long long t, long long &ib, long long &ie) {
        if (t < A.t_chunked) {
            ib = t * A.kchunk;
            ie = min(ib + A.kchunk, A.n_chunked);
        } else {
            ib = A.n_chunked + (t - A.t_chunked);
            ie = ib + 1;
        }
        ie = min(ie, A.n_items);
    };
    long long tk = 0, it = 0, ie = 0;  // this warp's next item and its ticket's end
    if (lane == 0) tk = (long long)atomicAdd(A.counter, 1ull);
    tk = __shfl_sync(kFull, tk, 0);
    ticket_items(tk, it, ie);
    long long taken = 1;  // tickets this warp has taken (iteration cap)
    unsigned stop = 0;    // set at a ticket's end: abort request or iteration cap
    unsigned asked = 0;   // lane 0: the abort request, read with each ticket
    bool fetched = false; // the next ticket is on its way (lane 0's tk)
    int cur = -1, phase = 0;
    long long job_end = 0;
    int since_i = 0, since_a = 0;  // adds since this warp's last flush (bounds)
    __syncthreads();
    for (;;) {
        // the job of this warp's next item
        int want = INT_MAX;
        if (it < A.n_items && !stop) {
            want = max(cur, 0);
            while (want + 1 < A.n_jobs && it >= A.jobs[want + 1].item_begin) ++want;
        }
        if (MEET && lane == 0 && want != INT_MAX) atomicMin(&s_want[phase], want);
        if (cur >= 0) {
            drain();
            flush_iso();
            since_i = since_a = 0;
        }
        if (MEET) __syncthreads();
        const int next = MEET ? s_want[phase] : want;
        if (cur >= 0) flush_ani(tid, kLThreads);
        if (next == INT_MAX) break;
        if (MEET) __syncthreads();  // J is read by the flush until here
        else __syncwarp();
        static_assert(sizeof(PairJob) % 4 == 0, "PairJob words");
        for (int q = MEET ? tid : lane; q < (int)(sizeof(PairJob) / 4); q += MEET ? kLThreads : 32)
            reinterpret_cast<int *>(&J)[q] = reinterpret_cast<const int *>(A.jobs + next)[q];
        if (tid == 0) s_want[phase ^ 1] = INT_MAX;
        phase ^= 1;
        cur = next;
        job_end = cur + 1 < A.n_jobs ? A.jobs[cur + 1].item_begin : A.n_items;
        if (MEET) __syncthreads();
        else __syncwarp();
        while (!stop && it < job_end && it < A.n_items && want == cur) {
            if (!fetched) {  // the ticket after this one (and the abort word with it)
                if (lane == 0) {
                    tk = (long long)atomicAdd(A.counter, 1ull);
                    if (A.ctrl) asked = ctrl_load(A.ctrl);
                }
                fetched = true;
            }
            // ---- one item ----------------------------------------------------
            const long long loc = it - J.item_begin;
            const int tile = (int)(loc / J.n_chunks);
            const int chunk = (int)(loc - (long long)tile * J.n_chunks);
            const int row_begin = chunk * J.rows_per_item;
            const int nrows = min(row_begin + J.rows_per_item, J.n_rows) - row_begin;  // <= 32
            const TileDesc t = J.tiles[tile];
            const int H = t.count;                            // 1..32 home points
            const int S = min(32 / H, kWindow / 2);           // candidate streams per warp
            const int sidx = lane / H < S ? lane / H : 0;     // this lane's stream
            const bool idle = lane >= S * H;
            const int hidx = t.start + (idle ? 0 : lane - sidx * H);
            unsigned hq = 0;
            int nranges;
            {
                float4 h;
                load_point(J.home.pk, hidx, h.x, h.y, h.z, h.w);
                if (W) hq = __ldg(J.home.qw + hidx);
                if (idle) h.x = h.y = h.z = __int_as_float(0x7fc00000);  // NaN: clamped out of range
                ws.home[lane] = h;
                // the home points' z extent (NaN lanes drop out of fminf / fmaxf)
                float zmn = h.z, zmx = h.z;
                #pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    zmn = fminf(zmn, __shfl_xor_sync(kFull, zmn, o));
                    zmx = fmaxf(zmx, __shfl_xor_sync(kFull, zmx, o));
                }
                RowRange rr{0, 0, 0, 0, 0.f, 0.f, 0.f, 0};
                if (lane < nrows) rr = row_range(A, J, J.rows[row_begin + lane], t, zmn, zmx);
                const unsigned m0 = __ballot_sync(kFull, rr.a0 < rr.b0), m1 = __ballot_sync(kFull, rr.a1 < rr.b1);
                const unsigned below = (1u << lane) - 1u;
                int at = __popc(m0 & below) + __popc(m1 & below);
                if (rr.a0 < rr.b0) ws.ranges[at++] = LeanRange{rr.a0, rr.b0, rr.sx, rr.sy, 0.f, rr.kind == 1 ? 1 : 0};
                if (rr.a1 < rr.b1) ws.ranges[at] = LeanRange{rr.a1, rr.b1, rr.sx, rr.sy, rr.sz1, 0};
                nranges = __popc(m0) + __popc(m1);
            }
            __syncwarp();
            const float4 *__restrict__ cpk = J.cand.pk;
            const unsigned *__restrict__ cqw = J.cand.qw;
            const int stride = 2 * S, wsize = kWindow / stride * stride;
            // copies window [lo, min(lo + wsize, b)) of a range into buffer `buf`
            auto stage = [&](int buf, int lo, int b) {
                const int n = min(wsize, ((b + 1) & ~1) - lo);
                if (lane < n)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                                     (unsigned)__cvta_generic_to_shared(&ws.pts[buf][lane])), "l"(cpk + lo + lane));
                if (W && 2 * lane < n)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                     (unsigned)__cvta_generic_to_shared(&ws.q[buf][2 * lane])), "l"(cqw + lo + 2 * lane));
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            int buf = 0, next_r = 0, next_lo = 0, next_b = 0;  // the next window to stage
            if (nranges) {
                next_lo = ws.ranges[0].a & ~1;
                next_b = ws.ranges[0].b;
                stage(0, next_lo, next_b);
            }
            auto stage_next = [&](int to) {  // the window after the one staged last, if any
                next_lo += wsize;
                if (next_lo >= next_b && ++next_r < nranges) {
                    next_lo = ws.ranges[next_r].a & ~1;
                    next_b = ws.ranges[next_r].b;
                }
                if (next_r < nranges) stage(to, next_lo, next_b);
                else asm volatile("cp.async.commit_group;" ::: "memory");
            };
            for (int r = 0; r < nranges; ++r) {
                const LeanRange &rg = ws.ranges[r];
                const int a = rg.a, b = rg.b;
                const float sx = rg.sx, sy = rg.sy, sz = rg.sz;
                {
                    const int sh = (sx != 0.f || sy != 0.f || sz != 0.f) ? 1 : 0;
                    const unsigned wl = A.fc.wl[sh], w2 = 2u * wl;
                    const float mgw = (float)kMag + (float)wl * (FB == 16 ? 0x1p-16f : 0x1p-15f);
                    const float2 MG = make_float2(mgw, mgw);
                    const float4 h = ws.home[lane];
                    const float2 NHX = make_float2(sx - h.x, sx - h.x), NHY = make_float2(sy - h.y, sy - h.y),
                                 NHZ = make_float2(sz - h.z, sz - h.z);
                    const int jmin = rg.fwd ? hidx : a - 1;
                    const int chk = rg.fwd ? t.start + H : a;  // from here on every pair is one to count
                    if (lane == 0) n_cand += (unsigned long long)(b - a) * (unsigned long long)H;

                    struct Cand {
                        float4 a, b;
                        uint2 q;
                    };
                    auto load = [&](int lo, int p) -> Cand {
                        Cand c;
                        c.a = ws.pts[buf][p - lo];
                        c.b = ws.pts[buf][p - lo + 1];
                        c.q = W ? *reinterpret_cast<const uint2 *>(&ws.q[buf][p - lo]) : make_uint2(0u, 0u);
                        return c;
                    };
                    // Readouts of two candidates: clamped bits, and addresses.
                    struct Read {
                        unsigned i[2], z[2], p[2];   // iso, z and perp readouts
                        unsigned ai[2], aa[2];       // counters
                    };
                    auto clip = [&](float q, float out, bool v) -> unsigned {
                        return __float_as_uint(v ? fminf(q, out) : out);
                    };
                    auto whole = [&](unsigned u0, unsigned u1) -> float2 {
                        return make_float2(__uint_as_float(u0 & ~kMask), __uint_as_float(u1 & ~kMask));
                    };
                    auto eval = [&](const Cand &c, bool v0, bool v1) -> Read {
                        Read e;
                        const float2 DX = __fadd2_rn(make_float2(c.a.x, c.a.y), NHX);
                        const float2 DY = __fadd2_rn(make_float2(c.a.z, c.a.w), NHY);
                        const float2 DZ = __fadd2_rn(make_float2(c.b.x, c.b.y), NHZ);
                        const float2 PP = __ffma2_rn(DY, DY, __fmul2_rn(DX, DX));
                        const float2 DS2 = make_float2(A.fc.ds2, A.fc.ds2);
                        if (DO_I) {
                            const float2 U = __fmul2_rn(__ffma2_rn(DZ, DZ, PP), DS2);
                            const float2 Q = __fadd2_rn(make_float2(sqrt_approx(U.x), sqrt_approx(U.y)), MG);
                            e.i[0] = clip(Q.x, qout, v0);
                            e.i[1] = clip(Q.y, qout, v1);
                            const float2 AD = __ffma2_rn(whole(e.i[0], e.i[1]), make_float2(ci, ci), make_float2(bi, bi));
                            e.ai[0] = __float_as_uint(AD.x);
                            e.ai[1] = __float_as_uint(AD.y);
                        }
                        if (DO_A) {
                            const float2 U = __fmul2_rn(PP, DS2);
                            const float2 Q = __fadd2_rn(make_float2(sqrt_approx(U.x), sqrt_approx(U.y)), MG);
                            const float2 RZ = __fmul2_rn(DZ, make_float2(A.fc.dsf, A.fc.dsf));
                            e.z[0] = clip(fabsf(RZ.x) + mgw, aout, v0);
                            e.z[1] = clip(fabsf(RZ.y) + mgw, aout, v1);
                            e.p[0] = clip(Q.x, aout, v0);  // (an invalid pair is in no window)
                            e.p[1] = clip(Q.y, aout, v1);
                            const float2 AD = __ffma2_rn(whole(e.z[0], e.z[1]), make_float2(cz, cz),
                                                         __ffma2_rn(whole(e.p[0], e.p[1]), make_float2(cp, cp),
                                                                    make_float2(ba, ba)));
                            e.aa[0] = __float_as_uint(AD.x);
                            e.aa[1] = __float_as_uint(AD.y);
                        }
                        return e;
                    };
                    // the fractions of two readouts, 16 bits each
                    auto fractions = [&](const unsigned *u) -> unsigned {
                        const unsigned f = __byte_perm(u[0], u[1], 0x5410);
                        return FB == 16 ? f : f & 0x7fff7fffu;
                    };
                    // N steps (of `stride` candidates for the warp): all evaluated,
                    // then all lower limbs, then the rest, so the returned values are
                    // waited for once; then the vote.
                    auto steps = [&](auto nst, const Cand *c, int p, bool v0, bool v1) {
                        constexpr int N = decltype(nst)::value;
                        Read e[N];
                        unsigned near = 0xffffffffu;
                        #pragma unroll
                        for (int k = 0; k < N; ++k) {
                            e[k] = eval(c[k], v0, v1);
                            if (DO_I) near = __vminu2(near, fractions(e[k].i));
                            if (DO_A) {
                                near = __vminu2(near, fractions(e[k].z));
                                near = __vminu2(near, fractions(e[k].p));
                            }
                            if (COUNT) {
                                #pragma unroll
                                for (int x = 0; x < 2; ++x) {
                                    if (DO_I) n_pairs += (e[k].i[x] >> FB) - kBias < (unsigned)bins;
                                    if (DO_A) n_pairs += (e[k].z[x] >> FB) - kBias < (unsigned)bins &&
                                                         (e[k].p[x] >> FB) - kBias < (unsigned)bins;
                                }
                            }
                        }
                        if (!W) {
                            #pragma unroll
                            for (int k = 0; k < N; ++k) {
                                #pragma unroll
                                for (int x = 0; x < 2; ++x) {
                                    if (DO_I) red_s_one(e[k].ai[x]);
                                    if (DO_A) red_s_one(e[k].aa[x]);
                                }
                            }
                        } else {
                            unsigned lo[N][2], hi[N][2], oi[N][2], oa[N][2];
                            #pragma unroll
                            for (int k = 0; k < N; ++k) {
                                #pragma unroll
                                for (int x = 0; x < 2; ++x) {
                                    const unsigned long long v = (unsigned long long)hq * (x ? c[k].q.y : c[k].q.x);
                                    lo[k][x] = (unsigned)v;
                                    hi[k][x] = (unsigned)(v >> 32);
                                    if (DO_I) oi[k][x] = atom_s_u32(e[k].ai[x], lo[k][x]);
                                    if (DO_A) oa[k][x] = atom_s_u32(e[k].aa[x], lo[k][x]);
                                }
                            }
                            #pragma unroll
                            for (int k = 0; k < N; ++k) {
                                #pragma unroll
                                for (int x = 0; x < 2; ++x) {
                                    if (DO_I) red_s_u32(e[k].ai[x] + 4u * NC, hi[k][x] + carry_of(oi[k][x], lo[k][x]));
                                    if (DO_A) {  // hi + carry < 2^32: hi is at most 2^32 - 2
                                        hi[k][x] += carry_of(oa[k][x], lo[k][x]);
                                        oa[k][x] = atom_s_u32(e[k].aa[x] + 4u, hi[k][x]);
                                    }
                                }
                            }
                            if (DO_A) {
                                #pragma unroll
                                for (int k = 0; k < N; ++k) {
                                    #pragma unroll
                                    for (int x = 0; x < 2; ++x)
                                        if (carry_of(oa[k][x], hi[k][x])) red_s_one(e[k].aa[x] + 8u);
                                }
                            }
                        }
                        near = __vminu2(near, near >> 16) & 0xffffu;
                        if (__any_sync(kFull, near < w2)) {
                            #pragma unroll
                            for (int k = 0; k < N; ++k) {
                                #pragma unroll
                                for (int x = 0; x < 2; ++x) {
                                    unsigned f = 0xffffffffu;
                                    if (DO_I) f = min(f, e[k].i[x] & kMask);
                                    if (DO_A) f = min(f, min(e[k].z[x] & kMask, e[k].p[x] & kMask));
                                    const bool hit = f < w2;
                                    const unsigned m = __ballot_sync(kFull, hit);
                                    if (!m) continue;
                                    if (hit) {
                                        ++n_rechk;
                                        const unsigned si = DO_I ? (e[k].i[x] >> FB) - kBias : 0u;
                                        const unsigned sa = DO_A ? min((e[k].z[x] >> FB) - kBias, (unsigned)bins) << 8 |
                                                                       min((e[k].p[x] >> FB) - kBias, (unsigned)bins)
                                                                 : 0u;
                                        LeanQueued q;
                                        q.home = (unsigned)hidx | ((sx < 0.f ? 0u : sx > 0.f ? 2u : 1u) << 30);
                                        q.cand = (unsigned)(p + k * stride + x) | ((sy < 0.f ? 0u : sy > 0.f ? 2u : 1u) << 30);
                                        q.code = sa | (si << 16) | ((unsigned)lane << 25) |
                                                 ((sz < 0.f ? 0u : sz > 0.f ? 2u : 1u) << 30);
                                        ws.queue[queued + __popc(m & ((1u << lane) - 1u))] = q;
                                    }
                                    queued += __popc(m);
                                    if (queued >= 32) {
                                        queued -= 32;
                                        settle(queued, 32);
                                    }
                                }
                            }
                        }
                    };
                    for (int lo = a & ~1; lo < b; lo += wsize) {
                        // flush before a counter could wrap: the limb of a lane's
                        // column takes at most one add per candidate of its stream,
                        // a unit counter one per pair
                        if (DO_I) {
                            const int adds = W ? (wsize / S) * (32 / NC) : wsize * H;
                            if (since_i + adds > A.budget) {
                                drain();
                                flush_iso();
                                since_i = 0;
                            }
                            since_i += adds;
                        }
                        if (DO_A && !W) {
                            if (since_a > (1 << 27)) {
                                flush_ani(lane, 32);
                                since_a = 0;
                            }
                            since_a += wsize * H;
                        }
                        stage_next(buf ^ 1);
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
                        __syncwarp();
                        const int hi = min(lo + wsize, b);
                        // one step whose candidates may lie outside (jmin, hi)
                        auto edge = [&](int blk) {
                            const int p = blk + 2 * sidx;
                            const Cand c = load(lo, min(p, (hi - 1) & ~1));
                            steps(std::integral_constant<int, 1>(), &c, p, p > jmin && p < hi, p + 1 > jmin && p + 1 < hi);
                        };
                        int blk = lo;
                        for (; blk < hi && blk < chk; blk += stride) edge(blk);
                        for (; blk + kN * stride <= hi; blk += kN * stride) {
                            Cand c[kN];
                            const int p = blk + 2 * sidx;
                            #pragma unroll
                            for (int k = 0; k < kN; ++k) c[k] = load(lo, p + k * stride);
                            steps(std::integral_constant<int, kN>(), c, p, true, true);
                        }
                        for (; blk < hi; blk += stride) edge(blk);
                        __syncwarp();  // every lane is done with this window
                        buf ^= 1;
                    }
                    if (COUNT) {
                        n_pairs_all += n_pairs;
                        n_pairs = 0;
                    }
                }
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");  // (the empty group after the last window)
            __syncwarp();  // the next item overwrites this item's ranges, homes and windows
            // ---- the next item -------------------------------------------------
            if (++it >= ie) {
                tk = __shfl_sync(kFull, tk, 0);
                ticket_items(tk, it, ie);
                fetched = false;
                // give up the queue on an abort request or past the iteration cap
                // (the copies are still flushed; the host discards them)
                stop = __shfl_sync(kFull, asked, 0) ? PCF_GAVE_UP_ABORT : 0u;
                if (++taken > A.max_tickets) stop |= PCF_GAVE_UP_CAP;
                if (stop && lane == 0 && A.status) ctrl_store(A.status, stop);
            }
        }
    }
    n_pairs_all += n_pairs;
    unsigned long long rp = (unsigned long long)n_pairs_all, rr = n_rechk;
    for (int off = 16; off > 0; off >>= 1) {
        rr += __shfl_down_sync(kFull, rr, off);
        rp += __shfl_down_sync(kFull, rp, off);
    }
    if (lane == 0) {
        if (rr) atomicAdd(A.g_stats + 0, rr);
        if (n_cand) atomicAdd(A.g_stats + 1, n_cand);
        if (COUNT && rp) atomicAdd(A.g_stats + 2, rp);
    }
}

}  // namespace

template <int KIND, bool W, bool C, int FB, int NC>
static cudaError_t launch_lean(const PairArgs &A, cudaStream_t st, int sm_count, int device) {
    auto kfn = k_pairs_lean<KIND, W, C, FB, NC>;
    const size_t smem = (size_t)LeanCopies<KIND, W, NC>::bytes(A.rule.bins);
    static OccCache occ;
    cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(kfn), device, smem);
    int per_sm = 0;
    if (e == cudaSuccess) e = occ.get(reinterpret_cast<const void *>(kfn), LeanShape<W>::threads, device, smem, &per_sm);
    if (e != cudaSuccess) return e;
    constexpr int kLWarps = LeanShape<W>::warps;
    const long long want = (A.n_items + kLWarps - 1) / kLWarps;
    const int grid = (int)std::max(1LL, std::min<long long>(want, (long long)sm_count * per_sm));
    kfn<<<grid, LeanShape<W>::threads, smem, st>>>(with_tickets(A, A.n_items, (long long)grid * kLWarps));
    return cudaGetLastError();
}
