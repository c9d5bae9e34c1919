// Alignment of every candidate of every anchor in both orientations, the
// orientation choice and the mismatch-ratio filter.
//
// reference: src/cpu_alignment.cpp:32-497 (shifted-Hamming alignment),
// include/alignmentorientation.hpp:10-92 (orientation),
// include/corrector.hpp:982-1211 (flag and mismatch-ratio filters).
//
// The reference takes, per orientation, the first shift of smallest score in
// its scan order among the shifts whose mismatches stay under int(overlap *
// maxErrorRate); its early exits only skip shifts that cannot win.  Nearly
// every shift of nearly every candidate fails that limit by a wide margin, so
// the work is a test of all shifts, and that test is a contraction: with the
// reads' hi planes as +-1 and zero outside the read, the sum over i of
// a[i + s] * c[i] is overlap - 2 * (hi plane mismatches), and the hi plane
// mismatches are a lower bound of the mismatches.  The tensor cores take it for
// 128 shifts x 64 candidates per product (the anchor's Toeplitz matrix times the
// candidates); the few shifts that pass are then counted exactly on both planes.
//
// Float work keeps the reference's operand order and uses explicitly rounded
// intrinsics, so every compare sees the reference's values.

#include <algorithm>
#include <type_traits>

#include "care_device.cuh"
#include "care_internal.h"
#include "care_tc.cuh"

namespace cg {

namespace {

constexpr unsigned kFull = 0xffffffffu;

struct AlnRes {
    int score, overlap, shift, nOps;
    bool valid;
};

// nOps / overlap as the reference's float division gives it (overlap > 0).  An
// exact overlap, the most frequent case, is kept out of the division: a zero
// dividend takes its slow path.
__device__ __forceinline__ float mismatch_ratio(int nOps, int overlap) {
    const float q = __fdiv_rn((float)(nOps == 0 ? 1 : nOps), (float)overlap);
    return nOps == 0 ? 0.0f : q;
}

// reference: include/alignmentorientation.hpp:12-66; 1 fwd, 2 rc, 3 none
__device__ __forceinline__ int choose_orientation(const AlnRes& f, const AlnRes& r, int La, float ratioParam,
                                                  int minOverlap, float maxErr, float* chosen) {
    const int minimumOverlap = max((int)__fmul_rn((float)La, ratioParam), minOverlap);
    const bool fok = f.valid && f.overlap >= minimumOverlap, rok = r.valid && r.overlap >= minimumOverlap;
    float ratio = 0.0f, rratio = 0.0f;
    if (fok) ratio = mismatch_ratio(f.nOps, f.overlap);
    if (rok) rratio = mismatch_ratio(r.nOps, r.overlap);
    const bool both = fok && rok;
    const bool forward = both ? ratio < rratio || (ratio == rratio && f.overlap > r.overlap) : fok;
    *chosen = forward ? ratio : rratio;
    if (!fok && !rok) return 3;
    return !(*chosen < maxErr) ? 3 : forward ? 1 : 2;
}

// reference: include/hostdevicefunctions.cuh:93-95 (calculateOverlapWeight)
__device__ __forceinline__ float overlap_weight(int nOps, int overlap, float maxErrorRate) {
    const float x = __fdiv_rn((float)(nOps == 0 ? 1 : nOps), __fmul_rn((float)overlap, maxErrorRate));
    return nOps == 0 ? 1.0f : __fsub_rn(1.0f, __fsqrt_rn(x));  // as mismatch_ratio
}

__device__ __forceinline__ uint2 pack_aln(const AlnRes& r, int ori) {
    return make_uint2((uint32_t)(uint16_t)(int16_t)r.shift | ((uint32_t)r.overlap << 16),
                      (uint32_t)(uint16_t)r.nOps | ((uint32_t)ori << 16));
}

// Mismatch-ratio filter of one anchor (include/corrector.hpp:1053-1149 single
// end, 1151-1211 paired end) over its nc aligned candidates in b.aln, writing
// the kept candidates in order; one warp (an anchor of several units).
__device__ void filter_anchor(const StoreArg& st, const Params& p, const BatchArg& b, int a, uint32_t base,
                              uint32_t nc) {
    auto aln = [&](uint32_t j) { return __ldcg(&b.aln[base + j]); };  // other blocks' results
    const int lane = (int)lane_id();
    float thr;
    if (!p.paired) {
        uint32_t c0 = 0, c1 = 0, c2 = 0;
        for (uint32_t j = lane; j < nc; j += 32) {
            const uint2 v = aln(j);
            if ((v.y >> 16) != 3u) {
                const float ratio = mismatch_ratio((int)(int16_t)(v.y & 0xffffu), (int)(v.x >> 16));
                c0 += ratio < p.mm2;
                c1 += ratio < p.mm3;
                c2 += ratio < p.mm4;
            }
        }
        c0 = __reduce_add_sync(kFull, c0);
        c1 = __reduce_add_sync(kFull, c1);
        c2 = __reduce_add_sync(kFull, c2);
        thr = -3.402823466e+38f;  // std::numeric_limits<float>::lowest()
        if (c0 > 0 || c1 > 0 || c2 > 0) {
            if ((float)c0 >= p.goodAlignmentsCountThreshold) thr = p.mm2;
            else if ((float)c1 >= p.goodAlignmentsCountThreshold) thr = p.mm3;
            else if ((float)c2 >= p.goodAlignmentsCountThreshold) thr = p.mm4;
        }
    } else {
        thr = p.pairedThreshold;
    }
    uint32_t kept = 0, aligned = 0;
    for (uint32_t j0 = 0; j0 < nc; j0 += 32) {
        const uint32_t j = j0 + lane;
        bool keep = false, isAligned = false;
        uint2 v = make_uint2(0, 0);
        if (j < nc) {
            v = aln(j);
            const int ori = (int)(v.y >> 16);
            if (ori != 3) {
                isAligned = true;
                const int ov = (int)(v.x >> 16);
                const int nOps = (int)(int16_t)(v.y & 0xffffu);
                const float ratio = mismatch_ratio(nOps, ov);
                keep = ratio < thr;
                if (p.paired && b.paired[base + j]) keep = true;
            }
        }
        const uint32_t m = __ballot_sync(kFull, keep);
        aligned += __popc(__ballot_sync(kFull, isAligned));
        if (keep) {
            const uint32_t pos = kept + __popc(m & ((1u << lane) - 1u));
            const int ov = (int)(v.x >> 16);
            const int nOps = (int)(int16_t)(v.y & 0xffffu);
            const uint32_t id = b.cand[base + j];
            b.fid[base + pos] = id;
            b.fshift[base + pos] = (int16_t)(v.x & 0xffffu);
            b.forient[base + pos] = (uint8_t)(v.y >> 16);
            b.flen[base + pos] = st.len[id];
            b.fweight[base + pos] = overlap_weight(nOps, ov, p.maxErrorRate);
        }
        kept += __popc(m);
    }
    if (lane == 0) {
        b.nfinal[a] = kept;
        atomicAdd(&b.counters[kCounterAligned], (unsigned long long)aligned);
        atomicAdd(&b.counters[kCounterMsaCands], (unsigned long long)kept);
    }
}

// ---------------------------------------------------------------- the shift test

constexpr int kAlignThreads = 128;         // a thread per TMEM lane
constexpr uint32_t kAlignTmemCols = kAlignUnit;  // a column per candidate of a unit
constexpr int kAlignQueue = 256;
constexpr uint32_t kOnes = 0x38383838u;    // four e4m3 +1 (the sign bit makes -1)

// `keep` most significant bits (any keep: all from 32 up, none from 0 down)
__device__ __forceinline__ uint32_t top_bits(int keep) {
    return __funnelshift_lc(0u, 0xffffffffu, (uint32_t)min(max(32 - keep, 0), 32));
}

// The 16 positions in the upper half of `bits` as 16 e4m3 values: -1 where the
// bit is set, +1 where it is not.  The order of the positions within the 16
// bytes is fixed but not ascending: both operands use it, so the products do not
// see it.
__device__ __forceinline__ uint32_t spread16(uint32_t v) {
    // byte 3: positions 0-7, byte 2: 8-15, byte 1: 4-11, byte 0: 12-15; word i takes bit 7 - i of each
    return __byte_perm(v, v << 4, 0x3276);
}
__device__ __forceinline__ uint4 expand16(uint32_t bits) {
    const uint32_t x = spread16(bits);
    return make_uint4((x & 0x80808080u) | kOnes, ((x << 1) & 0x80808080u) | kOnes, ((x << 2) & 0x80808080u) | kOnes,
                      ((x << 3) & 0x80808080u) | kOnes);
}
// the same with 0 before position `from` and from position `to` on
__device__ __forceinline__ uint4 expand16_part(uint32_t bits, int from, int to) {
    const uint32_t x = spread16(bits);
    const uint32_t v = spread16((0xffffffffu >> min(max(from, 0), 31)) & top_bits(to));
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t m = (v << i) & 0x80808080u;
        w[i] = ((x << i) & m) | ((m >> 4) * 7u);  // 0x80 -> 0x38
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// The sign bits of 16 or 32 consecutive FP32 accumulator columns of this
// thread's TMEM lane shifted into p, the first column's highest.
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_signs16(uint32_t taddr, uint32_t& p) {
    uint32_t r[16];
    tc_ld16(taddr, r);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; i++) p = __funnelshift_l(r[i], p, 1);
}
__device__ __forceinline__ void tc_signs32(uint32_t taddr, uint32_t& p) {
    uint32_t r[16], q[16];
    tc_ld16(taddr, r);
    tc_ld16(taddr + 16u, q);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; i++) p = __funnelshift_l(r[i], p, 1);
#pragma unroll
    for (int i = 0; i < 16; i++) p = __funnelshift_l(q[i], p, 1);
}

// a barrier of the two warps of one half of the block
__device__ __forceinline__ void half_sync(int half) { asm volatile("bar.sync %0, 64;" ::"r"(half + 1) : "memory"); }

// the same value into 8 consecutive columns of this thread's TMEM lane
__device__ __forceinline__ void tc_fill8(uint32_t taddr, float v) {
    const uint32_t r = __float_as_uint(v);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr), "r"(r)
                 : "memory");
}
// and into its first ncol columns (16, 32, 48 or 64).  zero: 0, unknown to the
// compiler, which would otherwise fill a register vector for every store (64 moves
// instead of 16).
__device__ __forceinline__ void tc_fill(uint32_t taddr, float v, int ncol, uint32_t zero) {
    uint32_t r[16];
#pragma unroll
    for (int i = 0; i < 16; i++) r[i] = __float_as_uint(v) + (uint32_t)i * zero;
#pragma unroll
    for (int c = 0; c < 64; c += 16) {
        if (c >= ncol) break;
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
                taddr + (uint32_t)c),
            "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
            "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
            : "memory");
    }
}

struct AlignUnit {
    int a, n;            // anchor of the batch, candidates (0: no unit left)
    uint32_t base, nc;   // the anchor's first slot and number of candidates
    uint32_t j0;         // the unit's first candidate
    int len;             // the anchor's length
};

// One block's shared memory, for reads of up to 32 W bases.
template <int W>
struct AlignBlock {
    static constexpr int kPlane = align_plane_words(W);  // words per plane
    static constexpr int kCopy = 2 * W + 15;             // 16-byte windows per copy (odd: no bank conflicts)
    alignas(128) uint4 toeplitz[16 * kCopy];              // of two tiles
    alignas(128) uint4 cands[kAlignUnit * 2 * W];
    alignas(16) uint32_t planes[kAlignUnit][2 * kPlane];  // the candidates' hi and lo planes
    uint32_t anch[2][2][kPlane];                          // the anchor's, forward and reverse complement
    uint32_t hi[2][W + 2];                                // its hi planes between two zero words
    alignas(16) uint4 queue[kAlignQueue];                 // passing shifts
    alignas(16) uint4 res[kAlignUnit];                    // packed result, its mismatch ratio, length; list order
    uint32_t best[kAlignUnit][2];                         // per orientation: score << 16 | scan position
    alignas(16) uint32_t keys[kAlignUnit];                // length << 6 | position, while they are ordered
    uint4 votes[2];
    // the unit in work and the next one
    AlignUnit unit[2];
    uint32_t ids[2][kAlignUnit];
    uint16_t lens[2][kAlignUnit];                         // in column order
    uint8_t ord[2][kAlignUnit];                           // a column's position in the list
    uint32_t queued, next;
    uint32_t tmem;
    alignas(8) unsigned long long mbar;
};

// Blocks per SM: at most 8 (512 tensor-memory columns), as many as the shared
// memory holds.  An instance for 640 bp gives those reads three blocks where the one
// for 1024 has two: alignment of 30,000 anchors of 640 bp 2.50 ms, 6.05 with one block
// of the largest instance; 20,000 of 1000 bp 4.03 ms with two, 7.37 with one; 60,000 of
// 300 bp 1.42 ms with five, 1.63 with four.
constexpr int align_blocks_per_sm(int w) { return w <= 5 ? 8 : w <= 8 ? 6 : w <= 10 ? 5 : w <= 20 ? 3 : 2; }

// One block per unit (up to 64 candidates of one anchor; a counter hands the
// batch's units out).
//
// The shift test.  Orientation o of a candidate against the anchor at shift
// s equals the forward candidate against the anchor (o = 0) or its reverse
// complement at shift La - Lc - s (o = 1), over the same range of shifts, so
// one set of candidate values serves both.  A product has 128 consecutive shifts
// as rows (M), the candidates as columns (N, a multiple of 16) and the candidates'
// positions as K, 32 per tcgen05.mma (kind::f8f6f4, e4m3, FP32 accumulators:
// sums of +-1 are exact).  The Toeplitz operand is not stored as a matrix: row 8
// r + i is shift 16 i + r, so that the rows of a core matrix (8 rows of 16 bytes)
// and its neighbours along K are 16 bytes apart in one copy of the anchor's
// values moved by r positions, and the 16 copies are the 8-row groups.  A tile is
// 16 (2 W + 15) windows of 16 values for two tiles, each expanded once from the
// bit plane.  The accumulators start at minus the smallest sum that a shift under its
// mismatch limit can have -- (1 - 2 maxErrorRate) * overlap -- so a shift passes
// where the sign bit is clear, and each lane shifts its row's signs into a word per
// 32 columns, one instruction per element.  With a limit above half the overlap that
// sum is negative and the test could rule out next to nothing: every shift passes to
// the exact count.  (60,000 anchors of 150 bp, whole call: 1.2 ms with limits to 0.3,
// 2.1 at 0.4, 3.7 at 0.45, 7.1 at 0.5, 8.9 at 0.7; the scan of every shift 1.9, 3.6, 3.7,
// 3.8 and 3.6.)
//
// With several read lengths the columns are in order of length, and the start
// value of a group of 8 columns is that of its shortest candidate (higher than the
// others' own: more shifts pass, none that should is lost).
//
// The shifts that pass are queued and counted exactly: mismatches of both planes
// over the overlap, the reference's limit and score, and the first smallest
// score per candidate and orientation by an atomic minimum over (score, scan
// position); a shift that can no longer win is not counted.  Then warps 0 and 1 choose the orientations and filter (an anchor of
// several units: warp 0 of the last of them to finish) while warps 2 and 3 load
// the next unit, whose chain of dependent loads would otherwise be the longest
// part of a unit.
//
// Measured, alignment and filter of 2M anchors of 150 bp (105M candidates, 10 Mbp
// genome with repeats): 22.1 ms; the scan of every shift by XOR and popcount that
// this replaces, 33.2 ms with its filter kernel (integer pipe 85% busy, popcounts at
// a quarter of its rate).  60k anchors of 300 bp: 1.4 ms against 16.1.  Issue is 65%
// busy, the tensor pipe 18%: what is left is bound by the instructions around the
// products (about 7,800 warp instructions a unit, a quarter of them signs and start
// values) and by waiting for the products in between.  The same test with mma.sync
// took 61 ms: e4m3 operands are unpacked to FP16 there, at a quarter of this rate.
//
// Limited: the waits end after p.alignPolls polls instead of kWaitPolls (an instance of
// its own, since a limit that may be zero costs 0.5% of the time).
template <int W, bool Limited>
__global__ void __launch_bounds__(kAlignThreads, align_blocks_per_sm(W))
align_kernel(StoreArg st, Params p, BatchArg b, const uint32_t* __restrict__ rawOff, int varies) {
    using Sm = AlignBlock<W>;
    extern __shared__ __align__(1024) unsigned char smraw[];
    // The block's shared memory by an address kept in a register: left to itself the
    // compiler builds it anew at every access.
    uint32_t smAt = smem_u32(smraw);
    asm volatile("" : "+r"(smAt));
    Sm& sm = *static_cast<Sm*>(__cvta_shared_to_generic(smAt));
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = (int)warp_uniform((uint32_t)tid >> 5);
    const float rate = p.maxErrorRate, slope = fmaxf(1.0f - 2.0f * rate, 0.0f);
    unsigned int next = 0;  // thread 64: the unit after the one in work
    if (tid == 64) next = atomicAdd(b.unitCursor, 1u);
    if (tid == 0) {
        sm.queued = 0;
        sm.unit[0].n = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)),
                     "r"(kAlignTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < 2 * (W + 2); i += kAlignThreads) (&sm.hi[0][0])[i] = 0u;
    if (tid < kAlignUnit) sm.best[tid][0] = sm.best[tid][1] = 0xffffffffu;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem, acc = tmem + ((uint32_t)(warp * 32) << 16);  // acc: this thread's TMEM lane
    const uint32_t mb = smem_u32(&sm.mbar);
    const uint32_t zero = (uint32_t)st.lmax >> 20;
    const uint64_t adesc = smem_desc(smem_u32(sm.toeplitz), 16, 16 * Sm::kCopy);
    const uint64_t bdesc = smem_desc(smem_u32(sm.cands), 128, 256 * W);
    const int rowShift = 16 * (tid & 7) + (tid >> 3);  // this thread's row of a tile
    const uint64_t first = batch_first(b);
    // Warps 2 and 3 load the next unit, a thread per candidate.  Its chain of
    // dependent loads (unit, slots, read ids, planes) is taken one step per tile
    // of the unit in work, so that each load arrives meanwhile; load() takes the
    // steps that are left and fills buffer u.
    const unsigned int total = *b.unitCount;
    int steps = 0;
    uint2 part = make_uint2(0u, 0u);
    uint32_t base2 = 0, nc2 = 0, id = 0;
    int len2 = 0, n2 = 0;
    auto step = [&]() {
        const int t = tid - 64, k = steps++;
        if (k == 0) {
            if (t == 0) sm.next = next;
        } else if (k == 1) {
            half_sync(1);
            const unsigned int at = sm.next;
            part.x = 0xffffffffu;
            if (at < total) part = b.units[at];
        } else if (part.x == 0xffffffffu) {
            n2 = 0;
        } else if (k == 2) {
            base2 = rawOff[part.x];
            nc2 = b.ncand[part.x];
            len2 = st.len[first + (uint64_t)part.x];
        } else {
            const uint32_t j0 = part.y * (uint32_t)kAlignUnit;
            n2 = (int)min((uint32_t)kAlignUnit, nc2 - j0);
            id = t < n2 ? b.cand[base2 + j0 + t] : 0u;
        }
    };
    auto load = [&](int u) {
        const int t = tid - 64;
        while (steps < 4) step();
        steps = 0;
        AlignUnit& un = sm.unit[u];
        if (n2 == 0) {
            if (t == 0) un.n = 0;
            return;
        }
        const int n = n2, La = len2;
        const uint64_t aid = first + (uint64_t)part.x;
        const uint32_t len = t < n ? st.len[id] : 0u;
        // the anchor's planes, forward and reversed and complemented, and both hi planes for the windows
        const uint32_t* ga = st.hilo + aid * (2 * Sm::kPlane);
        for (int i = t; i < 2 * Sm::kPlane; i += 64) {
            const int pl = i >= Sm::kPlane, w = i - pl * Sm::kPlane;
            const uint32_t* gp = ga + pl * Sm::kPlane;
            const int d = 32 * W - La, x = w + (d >> 5);
            const uint32_t r0 = x < W ? __brev(gp[W - 1 - x]) : 0u, r1 = x + 1 < W ? __brev(gp[W - 2 - x]) : 0u;
            const uint32_t f = gp[w], v = ~__funnelshift_l(r1, r0, d & 31) & top_bits(La - 32 * w);
            sm.anch[0][pl][w] = f;
            sm.anch[1][pl][w] = v;
            if (pl == 0 && w < W) {
                sm.hi[0][w + 1] = f;
                sm.hi[1][w + 1] = v;
            }
        }
        int col = t;  // a column per candidate, by length where lengths differ
        if (varies) {
            const uint32_t key = ((t < n ? len : 0xffffu) << 6) | (uint32_t)t;
            sm.keys[t] = key;
            half_sync(1);
            const uint4* k4 = reinterpret_cast<const uint4*>(sm.keys);
            col = 0;
#pragma unroll 4
            for (int i = 0; i < kAlignUnit / 4; i++) {
                const uint4 k = k4[i];
                col += (int)(k.x < key) + (int)(k.y < key) + (int)(k.z < key) + (int)(k.w < key);
            }
        }
        sm.ids[u][t] = id;
        sm.lens[u][col] = (uint16_t)len;
        sm.ord[u][col] = (uint8_t)t;
        if (t < n) {
            const uint32_t* gc = st.hilo + (uint64_t)id * (2 * Sm::kPlane);
#pragma unroll
            for (int q = 0; q < Sm::kPlane / 2; q++) cp_async16(&sm.planes[col][4 * q], gc + 4 * q);
        }
        if (t == 0) {
            un.a = (int)part.x;
            un.n = n;
            un.base = base2;
            un.nc = nc2;
            un.j0 = part.y * (uint32_t)kAlignUnit;
            un.len = La;
        }
        cp_async_wait_all();
    };
    uint32_t phase = 0;
    bool failed = false;
    for (int u = 0;; u ^= 1) {
        // n == 0: the first unit is still to be loaded
        const int n = (int)warp_uniform((uint32_t)sm.unit[u].n), La = (int)warp_uniform((uint32_t)sm.unit[u].len);
        if (tid == 64 && n) next = atomicAdd(b.unitCursor, 1u);  // arrives while this unit is in work
        const int minov = max(p.minOverlap, (int)__fmul_rn((float)La, p.minOverlapRatio));
        const uint16_t* lens = sm.lens[u];
        const int lcMin = (int)warp_uniform(lens[0]), lcMax = (int)warp_uniform(lens[max(n - 1, 0)]);
        const int right = max(La - minov + 1, 0);  // the reference's shifts 0 .. right - 1, then the left ones
        // the forward candidates' shifts (a read shorter than minov overlaps by its whole length,
        // and then the other orientation's shifts reach further)
        const int spMin = -max(lcMax - min(minov, La), 0), spMax = La - min(minov, lcMin);
        const int jobs = n && spMax >= spMin ? 2 * ((spMax - spMin) / 128 + 1) : 0;  // orientations x tiles
        const int ksteps = (lcMax + 31) >> 5, ncol = (n + 15) & ~15;
        const uint32_t idesc = (1u << 4) | ((uint32_t)(ncol >> 3) << 17) | (8u << 24);  // FP32 += e4m3 e4m3, M 128
        // the windows of up to two tiles from shift x0 on: window x (positions x .. x + 15) of
        // copy x0 + x mod 16; this thread's windows are 128 positions apart
        auto build = [&](int o, int x0, int pair) {
            uint4* dst = sm.toeplitz + (tid & 15) * Sm::kCopy + (tid >> 4);
            const uint4* const end = dst + (2 * ksteps + 8 * pair - 1 - (tid >> 4));
            int x = x0 + tid;
            const uint32_t inside = (uint32_t)max(La - 15, 0);  // windows [0, inside) hold 16 bases
            const uint32_t* h = sm.hi[o] + 1 + (x >> 5);
            for (; dst < end; dst += 8, x += 128, h += 4) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if ((uint32_t)x < inside) v = expand16(__funnelshift_l(h[1], h[0], x & 31));
                else if (x > -16 && x < La) v = expand16_part(__funnelshift_l(h[1], h[0], x & 31), -x, La - x);
                *dst = v;
            }
        };
        // the accumulators' start values for this thread's row, shift sp
        auto start = [&](int sp) {
            const int low = min(minov, La);
            auto value = [&](int lc) {
                const int ov = sp >= 0 ? min(La - sp, lc) : min(La, lc + sp);
                return p.alignLift - slope * (float)max(ov, min(low, lc));
            };
            if (!varies) {
                tc_fill(acc, value(lcMin), ncol, zero);
            } else {
#pragma unroll 1
                for (int c = 0; c < ncol; c += 8) tc_fill8(acc + (uint32_t)c, c < n ? value(lens[c]) : -1e6f);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        };
        // the exact count of the queued shifts
        // unrolled where registers are to spare: 75 bp 3%, 640 and 1000 bp 1% of the
        // alignment (150 to 300 bp lose up to 1% with it)
        constexpr int kCountUnroll = W <= 4 || W > 10 ? 4 : 1;
        auto count = [&](int entries) {
            for (int e0 = tid; e0 < entries; e0 += kAlignThreads) {
                uint4 e = sm.queue[e0];  // columns 0-31, columns 32-63 (first column highest), shift, orientation
                const int sp = (int)e.z, o = (int)e.w;
                const uint32_t* ap = sm.anch[o][0];
                while (e.x | e.y) {
                    const bool second = e.x == 0u;
                    const int bit = __clz(second ? e.y : e.x), c = second ? 32 + bit : bit;
                    if (second) e.y ^= 0x80000000u >> bit;
                    else e.x ^= 0x80000000u >> bit;
                    if (c >= n) continue;
                    const int lc = lens[c];
                    const int s = o ? La - lc - sp : sp;  // the reference's shift
                    if (s >= 0 ? s > La - minov : -s > lc - minov) continue;
                    const int ov = s >= 0 ? min(La - s, lc) : min(La, lc + s);
                    if (ov <= 0) continue;
                    // out from this many mismatches on: the shift's limit, or a score above
                    // the best so far (of equal scores the first in scan order counts)
                    const int beaten = (int)(*(volatile uint32_t*)&sm.best[c][o] >> 16) - La - lc + 2 * ov + 1;
                    const int out = min((int)__fmul_rn((float)ov, rate), beaten);
                    if (out <= 0) continue;
                    const int sl = abs(sp), ws = sl >> 5, bs = sl & 31, parts = (ov + 31) >> 5;
                    const uint32_t* sh = (sp >= 0 ? ap : sm.planes[c]) + ws;
                    const uint32_t* ot = sp >= 0 ? sm.planes[c] : ap;
                    uint32_t ch = sh[0], cl = sh[Sm::kPlane];
                    int m = 0;
#pragma unroll kCountUnroll
                    for (int i = 0; i < parts; i++) {
                        const uint32_t nh = sh[i + 1], nl = sh[Sm::kPlane + i + 1];
                        const uint32_t x = (__funnelshift_l(nh, ch, bs) ^ ot[i]) |
                                           (__funnelshift_l(nl, cl, bs) ^ ot[Sm::kPlane + i]);
                        m += __popc(x & top_bits(ov - 32 * i));
                        ch = nh;
                        cl = nl;
                    }
                    if (m < out)
                        atomicMin(&sm.best[c][o], ((uint32_t)(m + La + lc - 2 * ov) << 16) |
                                                      (uint32_t)(s >= 0 ? s : right - s - 1));
                }
            }
        };
        if ((tid & 63) < ncol) {  // the candidates' values, 32 positions of a column per step
            const int c = tid & 63, lc = lens[c];
            uint4* dst = sm.cands + (c >> 3) * (16 * W) + (c & 7);
            for (int q = tid >> 6; q < ksteps; q += 2) {
                const uint32_t h = sm.planes[c][q];
                const int rest = lc - 32 * q;
                if (rest >= 32) {
                    dst[16 * q] = expand16(h);
                    dst[16 * q + 8] = expand16(h << 16);
                } else {
                    dst[16 * q] = expand16_part(h, 0, rest);
                    dst[16 * q + 8] = expand16_part(h << 16, 0, rest - 16);
                }
            }
        }
        for (int job = 0;; job++) {
            const int o = 2 * job >= jobs, t = job - (o ? jobs >> 1 : 0);
            const int sp = spMin + 128 * t + rowShift;
            if (job < jobs) {
                if ((t & 1) == 0) build(o, spMin + 128 * t, min((jobs >> 1) - t, 2));
                start(sp);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // operands, for the tensor core
                tc_fence_before();
            }
            __syncthreads();
            const int entries = (int)warp_uniform(sm.queued);
            if (job == jobs || entries > kAlignQueue - kAlignThreads) {  // done, or no room for a tile's worst case
                count(entries);
                __syncthreads();
                if (job == jobs) break;
                if (tid == 0) sm.queued = 0;
            }
            tc_fence_after();
            if (tid == 0) {
                for (int k = 0; k < ksteps; k++)
                    tc_mma_e4m3(tmem, adesc + (uint64_t)(2 * k + 8 * (t & 1)), bdesc + (uint64_t)(16 * k), idesc);
                tc_commit(mb);
            }
            if (warp >= 2 && steps < 4) step();
            bool ok = true;
            if (warp == 0) ok = mbar_wait(mb, phase, Limited ? p.alignPolls : kWaitPolls);  // the other warps wait at the barrier
            phase ^= 1u;
            if (__syncthreads_or(!ok)) {
                failed = true;
                break;
            }
            tc_fence_after();
            uint32_t fails[2] = {0xffffffffu, 0xffffffffu};
#pragma unroll
            for (int c = 0; c < 2; c++) {
                if (32 * c >= ncol) break;
                if (32 * c + 16 < ncol) {
                    tc_signs32(acc + 32u * c, fails[c]);
                } else {
                    tc_signs16(acc + 32u * c, fails[c]);
                    fails[c] = (fails[c] << 16) | 0xffffu;
                }
            }
            const bool any = (fails[0] & fails[1]) != 0xffffffffu;
            const unsigned m = __ballot_sync(kFull, any);
            if (m) {
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&sm.queued, (uint32_t)__popc(m));
                at = __shfl_sync(kFull, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
                if (any)
                    sm.queue[at] = make_uint4(~fails[0], ~fails[1], (uint32_t)sp, (uint32_t)o);
            }
        }
        if (failed) break;
        if (warp >= 2) {
            load(u ^ 1);
        } else if (n) {
            // orientation choice; the results in list order
            const AlignUnit un = sm.unit[u];
            const bool whole = un.nc <= (uint32_t)kAlignUnit;  // the anchor's only unit
            if (tid < n) {
                const int pos = sm.ord[u][tid], lc = lens[tid], tb = La + lc;
                AlnRes res[2];
#pragma unroll
                for (int o = 0; o < 2; o++) {
                    const uint32_t key = sm.best[tid][o];
                    const int t = (int)(key & 0xffffu);
                    AlnRes& r = res[o];
                    r.valid = key != 0xffffffffu;
                    r.shift = !r.valid ? -lc : t < right ? t : right - t - 1;
                    r.score = r.valid ? (int)(key >> 16) : tb;
                    r.overlap = min(lc, La - r.shift) - max(-r.shift, 0);
                    r.nOps = r.score - tb + 2 * r.overlap;
                }
                float ratio;
                const int ori = choose_orientation(res[0], res[1], La, p.minOverlapRatio, p.minOverlap,
                                                   p.orientMaxErrorRate, &ratio);
                const uint2 v = pack_aln(ori == 2 ? res[1] : res[0], ori);
                if (whole) {
                    sm.res[pos] = make_uint4(v.x, v.y, __float_as_uint(ratio), (uint32_t)lc);
                } else {
                    b.aln[un.base + un.j0 + pos] = v;
                    __threadfence();
                }
            }
            sm.best[tid][0] = sm.best[tid][1] = 0xffffffffu;
            if (tid == 0) sm.queued = 0;
            half_sync(0);
            if (whole) {
                // the filter of filter_anchor with a thread per candidate
                uint4 r = make_uint4(0u, 3u << 16, 0u, 0u);
                if (tid < n) r = sm.res[tid];
                const bool aligned = (r.y >> 16) != 3u;
                const float ratio = __uint_as_float(r.z);
                unsigned k0, k1 = 0u, k2 = 0u;
                if (!p.paired) {
                    k0 = __ballot_sync(kFull, aligned && ratio < p.mm2);
                    k1 = __ballot_sync(kFull, aligned && ratio < p.mm3);
                    k2 = __ballot_sync(kFull, aligned && ratio < p.mm4);
                } else {
                    k0 = __ballot_sync(kFull, aligned && (ratio < p.pairedThreshold || b.paired[un.base + tid]));
                }
                const unsigned al = __ballot_sync(kFull, aligned);
                const uint4 mine = make_uint4(__popc(k0), __popc(k1), __popc(k2), __popc(al));
                if (lane == 0) sm.votes[warp] = mine;
                half_sync(0);
                const uint4 other = sm.votes[1 - warp];
                const uint32_t c0 = mine.x + other.x, c1 = mine.y + other.y, c2 = mine.z + other.z;
                unsigned kept = 0u;
                uint32_t beside = 0u, total = 0u;  // kept by the other warp, and by both
                auto take = [&](unsigned k, uint32_t o, uint32_t c) {
                    kept = k;
                    beside = o;
                    total = c;
                };
                const float good = p.goodAlignmentsCountThreshold;
                if (p.paired) take(k0, other.x, c0);
                else if ((c0 | c1 | c2) == 0u) take(0u, 0u, 0u);
                else if ((float)c0 >= good) take(k0, other.x, c0);
                else if ((float)c1 >= good) take(k1, other.y, c1);
                else if ((float)c2 >= good) take(k2, other.z, c2);
                if ((kept >> lane) & 1u) {
                    const uint32_t at = un.base + __popc(kept & ((1u << lane) - 1u)) + (warp ? beside : 0u);
                    b.fid[at] = sm.ids[u][tid];
                    b.fshift[at] = (int16_t)(r.x & 0xffffu);
                    b.forient[at] = (uint8_t)(r.y >> 16);
                    b.flen[at] = (uint16_t)r.w;
                    b.fweight[at] = overlap_weight((int)(int16_t)(r.y & 0xffffu), (int)(r.x >> 16), rate);
                }
                if (tid == 0) {
                    b.nfinal[un.a] = total;
                    atomicAdd(&b.counters[kCounterAligned], (unsigned long long)(mine.w + other.w));
                    atomicAdd(&b.counters[kCounterMsaCands], (unsigned long long)total);
                }
            } else if (warp == 0) {  // the last of the anchor's units to finish filters it
                uint32_t done = 0;
                if (lane == 0) done = atomicAdd(&b.unitsDone[un.a], 1u);
                done = __shfl_sync(kFull, done, 0);
                if (done == (un.nc - 1) / (uint32_t)kAlignUnit) {
                    __threadfence();
                    filter_anchor(st, p, b, un.a, un.base, un.nc);
                }
            }
        }
        __syncthreads();
        if (sm.unit[u ^ 1].n == 0) break;
    }
    if (failed) {
        if (tid == 0) atomicAdd(&b.counters[kCounterAlignTimeouts], 1ull);
        mbar_wait(mb, phase ^ 1u, kWaitPolls);  // the products in flight, bounded again
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAlignTmemCols)
                     : "memory");
}

template <int W>
struct AlignInstance {
    static cudaError_t launch(StoreArg st, const Params& p, const BatchArg& b, bool varies, unsigned blocks,
                              cudaStream_t s) {
        const auto kernel = p.alignPolls == kWaitPolls ? align_kernel<W, false> : align_kernel<W, true>;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)sizeof(AlignBlock<W>));
        if (e != cudaSuccess) return e;
        kernel<<<blocks, kAlignThreads, sizeof(AlignBlock<W>), s>>>(st, p, b, b.rawCount, varies);
        return cudaGetLastError();
    }
    static int occupancy() {
        static_assert(align_blocks_per_sm(W) * (sizeof(AlignBlock<W>) + 1024) <= 228 * 1024, "shared memory of an SM");
        return align_blocks_per_sm(W);
    }
};

// calls f with the instance for this store
template <class F>
auto with_instance(StoreArg st, F f) {
    switch (align_words(st.lmax)) {
        case 3: return f(AlignInstance<3>{});
        case 4: return f(AlignInstance<4>{});
        case 5: return f(AlignInstance<5>{});
        case 8: return f(AlignInstance<8>{});
        case 10: return f(AlignInstance<10>{});
        case 16: return f(AlignInstance<16>{});
        case 20: return f(AlignInstance<20>{});
        default: return f(AlignInstance<32>{});
    }
}

}  // namespace

int align_occupancy(StoreArg st) {
    return with_instance(st, [](auto k) { return k.occupancy(); });
}

cudaError_t launch_align(StoreArg st, Params p, BatchArg b, bool varies, unsigned blocks, cudaStream_t s) {
    if (b.count <= 0 || blocks == 0) return cudaSuccess;
    // a shift without overlap has no mismatch limit to stay under: a negative minimum is none
    p.minOverlap = std::max(p.minOverlap, 0);
    p.alignLift = p.maxErrorRate > 0.5f ? 0.25f + (float)st.lmax : 0.25f;  // no sum is below -lmax
    return with_instance(st, [&](auto k) { return k.launch(st, p, b, varies, blocks, s); });
}

}  // namespace cg
