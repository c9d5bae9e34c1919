// Per-anchor correction: MSA build, region refinement and the anchor
// correction decision.
//
// reference: include/corrector.hpp:1260-1421 (weights, MSA build, refinement),
// src/msa.cpp:9-173,304-453,532-734 (MSA, properties, corrected anchor,
// different-region search).
//
// Float work keeps the reference's operand order and uses explicitly rounded
// intrinsics (the library is also built with --fmad=false): every compare the
// decision makes sees the same float values as the reference's host code.

#include <algorithm>
#include <type_traits>

#include "care_device.cuh"
#include "care_internal.h"

namespace cg {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// reference: include/classification.hpp:748-797 (extract_anchor_v3) and
// include/forest.hpp:70-81,217-226 (tree walk; decide: running mean of the
// trees' probabilities, true as soon as it reaches the threshold)
__device__ bool forest_decide(const Params& p, const float* f) {
    float sum = 0.0f;
    for (int t = 0; t < p.numTrees; t++) {
        const ForestNode* tree = p.forestNodes + p.treeOffsets[t];
        uint32_t i = 0;
        float prob = 0.0f;
        for (int guard = 0; guard < (1 << 20); guard++) {
            const ForestNode n = tree[i];
            if ((double)f[n.att] <= n.split) {
                if (n.flag & 2u) { prob = __uint_as_float(n.lhs); break; }
                i = n.lhs;
            } else {
                if (n.flag & 1u) { prob = __uint_as_float(n.rhs); break; }
                i = n.rhs;
            }
        }
        sum = __fadd_rn(sum, prob);
        if (__fdiv_rn(sum, (float)p.numTrees) >= p.forestThreshold) return true;
    }
    return false;
}

__device__ __forceinline__ int base_index(char c) { return c == 'A' ? 0 : c == 'C' ? 1 : c == 'G' ? 2 : 3; }

// ---------------------------------------------------------------- candidate correction
//
// reference: src/msa.cpp:457-522 (getCorrectedCandidates), include/corrector.hpp
// :293-299 and 1504-1512 (HQ anchors correct their candidates), :1674-1748 (the
// record: the consensus slice, reverse complemented back for a reverse-
// complement candidate).  A row of the final MSA with shift s and length len
// qualifies when -nc <= s <= nc and s + len <= La + nc (nc =
// new_columns_to_correct; the support and coverage test computed there is
// overwritten by `candidateShouldBeCorrected = true`).  Its record votes for
// read `id` (see Params::candVotes).

__device__ __forceinline__ void vote_word(const Params& p, uint64_t read, int w, unsigned long long v) {
    const uint64_t i = read * (uint64_t)p.candPitch + (uint64_t)w;
    atomicAnd(&p.candAnd[i], v);
    atomicOr(&p.candOr[i], v);
}

// Quality score of position `pos` (aligned orientation) of a candidate row
// (reference: include/corrector.hpp:1214-1239).  Rows hold Lmax scores; past
// the read's end the store holds what the reference's decoded row holds there
// (zero, or the first bin's score with lossy qualities; include/
// chunkedreadstorage.hpp:532-610), and a reverse-complement candidate's whole
// row is reversed, so a read shorter than Lmax starts with that padding: its
// position pos reads score Lmax - 1 - pos.
__device__ __forceinline__ uint8_t row_quality(const uint8_t* q, int lmax, bool rc, int pos) {
    return q[rc ? lmax - 1 - pos : pos];
}

// ---------------------------------------------------------------- MSA, warp per anchor

// A column's weights and counts and the statistics derived from them
// (src/msa.cpp:135-157).
struct ColInfo {
    float w[4];
    uint32_t n[4];
    char cons;
    float consW, colW;
    __device__ float wOf(uint32_t i) const { return i == 0 ? w[0] : i == 1 ? w[1] : i == 2 ? w[2] : w[3]; }
    __device__ uint32_t nOf(uint32_t i) const { return i == 0 ? n[0] : i == 1 ? n[1] : i == 2 ? n[2] : n[3]; }
    __device__ int cov() const { return (int)(n[0] + n[1] + n[2] + n[3]); }
};

// wc[q * cp + c]: weight bits (x) and count (y) of base q in column c, read
// as one 8-byte entry per base
__device__ __forceinline__ ColInfo col_info(const uint2* wc, int cp, int c) {
    ColInfo r;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint2 v = wc[q * cp + c];
        r.w[q] = __uint_as_float(v.x);
        r.n[q] = v.y;
    }
    const float wA = r.w[0], wC = r.w[1], wG = r.w[2], wT = r.w[3];
    r.cons = 'A';
    r.consW = wA;
    if (wC > r.consW) { r.cons = 'C'; r.consW = wC; }
    if (wG > r.consW) { r.cons = 'G'; r.consW = wG; }
    if (wT > r.consW) { r.cons = 'T'; r.consW = wT; }
    r.colW = __fadd_rn(__fadd_rn(__fadd_rn(wA, wC), wG), wT);
    return r;
}

// One warp per anchor.
//
// Everything the path reads from an MSA -- the different-region search, the
// properties and both decisions -- lies in the anchor's columns, so only the
// part of each row that overlaps the anchor is accumulated, in anchor
// coordinates (column = anchor position).  Lane l owns the columns c with c % 32
// == l in every pass.
//
// Nearly every base of a row equals its column's base, so the build separates the
// two.  For 32 rows at a time, lane r brings row r's bit planes into the anchor's
// columns and compares them with the columns' bases: one word of matches and one
// of mismatches per 32 columns.  The match words are transposed across the warp,
// so that a lane holds its columns' rows as bits, and each lane adds the rows'
// weights to its columns' sums in registers, in list order: a test and an addition
// per row and 32 columns, the counts by population count.  The mismatches (one or
// two per row) go to a list in row order and are added to their (base, column)
// entries in shared memory 32 at a time, entries that meet in one place by their
// order in the list.  A column's base is the anchor's, unless the first 32 rows say
// that the anchor errs there.  A column's sum of a base thus receives the
// reference's additions in the reference's order (anchor, then the kept candidates
// in list order); sums of different bases are independent.
// With quality scores, and for reads longer than 320 bp (msa_planes), the rows are
// added one at a time in shared memory instead, each lane to its columns.
// Measured, MSA stage: 2M anchors of 150 bp with repeats 12.9 ms (row by row in
// shared memory 17.2 ms: 116 instructions per row); 60,000 anchors of 300 bp
// 0.70 ms, 30,000 of 640 bp 1.01 ms, 20,000 of 1000 bp 1.51 ms (a block per anchor,
// which reads longer than 256 bp used to take, 2.9, 3.1 and 4.3 ms).  It issues in
// 6 of 10 cycles: a warp's steps depend on one another, and registers and the sums
// in shared memory leave room for 27 one-warp blocks per SM (150 bp; the occupancy
// query's figure, as those below).
//
// `sm` is the warp's own slice of shared memory (MsaSlice), `qw` the block's
// quality weights.

// Whether a store of reads of up to lp bases (a multiple of 32) adds its rows by
// planes or one at a time.  With quality scores every base has its own weight: see
// rowPass.  Without them, a row of many words holds more in registers, and the few
// warps that its sums leave room for do not hide the steps from word to word.  MSA
// stage, by planes and one row at a time: 60,000 anchors of 300 bp 0.70 and 0.75 ms,
// 40,000 of 321 bp 1.00 and 0.62, of 500 bp 1.26 and 0.93, 30,000 of 640 bp 1.64 and
// 1.01, 20,000 of 1000 bp 4.58 and 1.50.
__host__ __device__ constexpr bool msa_planes(bool quality, int lp) { return !quality && lp <= 320; }

// Offsets in bytes of one warp's shared memory.  Its first 16 lp bytes hold the
// weights and counts [4][lp].
struct MsaSlice {
    size_t sup, stage, weight, ref, meta, cons, bytes;
    // rows: the rows are added one at a time
    __host__ __device__ MsaSlice(int lp, int pitch, int wp, const Params& p, bool rows) {
        const int words = pitch > 2 * wp ? pitch : 2 * wp;
        sup = (size_t)lp * 4 * sizeof(uint2);
        stage = sup + (size_t)lp * sizeof(float);           // 32 rows' planes or 2-bit words; the mismatch list
        weight = stage + (size_t)32 * words * sizeof(uint32_t);  // [32]
        ref = weight + 32 * sizeof(float);                   // planes of the columns' bases [2][wp]
        meta = ref + (size_t)(2 * wp + 3) / 4 * 16;          // [32]: shift, len | orient << 16, weight, id
        cons = meta + (rows || p.candidates ? 32 * sizeof(int4) : 0);
        // candidate correction: the consensus codes of Lmax + 2 new_columns_to_correct columns
        const size_t cols = (size_t)lp + 2 * (size_t)p.newColumns;
        bytes = cons + (p.candidates ? (cols + 15) / 16 * 16 + 2 * ((cols + 31) / 32 + 1) * sizeof(uint64_t) : 0);
    }
};

// x's bits from the n-th most significant on (none from 32 up), and its n most
// significant bits
__device__ __forceinline__ uint32_t bits_from(int n) { return __funnelshift_rc(0xffffffffu, 0u, (uint32_t)max(n, 0)); }
__device__ __forceinline__ uint32_t bits_to(int n) { return ~bits_from(n); }

// x[k] and its assignment for a k known at run time only, x in registers
template <int K, typename T>
__device__ __forceinline__ T pick(const T (&x)[K], int k) {
    T v = x[0];
#pragma unroll
    for (int q = 1; q < K; q++) v = q == k ? x[q] : v;
    return v;
}
template <int K, typename T>
__device__ __forceinline__ void put(T (&x)[K], int k, T v) {
#pragma unroll
    for (int q = 0; q < K; q++) x[q] = q == k ? v : x[q];
}

// Transposes K 32 x 32 bit matrices, lane r holding row r, most significant bit
// first: afterwards lane c holds column c.
template <int K>
__device__ __forceinline__ void transpose_bits(uint32_t (&x)[K], int lane) {
    uint32_t half = 0xffff0000u;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const bool low = (lane & s) != 0;
        const uint32_t keep = low ? ~half : half, turn = low ? s : 32 - s;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const uint32_t y = __shfl_xor_sync(kFull, x[k], s);
            x[k] = (x[k] & keep) | (__funnelshift_l(y, y, turn) & ~keep);
        }
        half = s == 16 ? 0xff00ff00u : s == 8 ? 0xf0f0f0f0u : s == 4 ? 0xccccccccu : 0xaaaaaaaau;
    }
}

template <bool QUAL, int K>
__device__ __forceinline__ void msa_warp_anchor(const StoreArg& st, const Params& p, const BatchArg& b,
                                             const uint32_t* __restrict__ rawOff, int lp, int a, uint64_t first,
                                             unsigned char* sm, const MsaSlice& sl, const float* qw) {
    const int lane = (int)lane_id();
    uint2* wc = reinterpret_cast<uint2*>(sm);                    // [4][lp]: weight bits, count
    float* sup = reinterpret_cast<float*>(sm + sl.sup);          // [lp]
    uint32_t* stage = reinterpret_cast<uint32_t*>(sm + sl.stage);
    uint32_t* list = stage;
    float* weight = reinterpret_cast<float*>(sm + sl.weight);
    uint32_t* ref = reinterpret_cast<uint32_t*>(sm + sl.ref);
    int4* meta = reinterpret_cast<int4*>(sm + sl.meta);  // [32]: shift, len | orient << 16, weight, id
    const uint64_t aid = first + (uint64_t)a;
    const uint64_t oi = (first - out_first(b)) + (uint64_t)a;   // output row
    const uint32_t nf = warp_uniform(b.nfinal[a]);
    char* out = b.out + oi * b.outPitch;
    if (nf == 0) {
        if (lane == 0) b.flags[oi] = 0;
        return;
    }
    const uint32_t base = warp_uniform(rawOff[a]);
    const int La = (int)warp_uniform((uint32_t)st.len[aid]);
    const int pitch = st.pitch;
    const uint32_t* aenc = st.enc + aid * (uint64_t)pitch;
    const uint8_t* aq = QUAL ? st.qual + aid * (uint64_t)st.lmax : nullptr;
    constexpr uint8_t kRm = 0x80;

    constexpr uint8_t kNew = 0x40;
    constexpr bool kPlanes = msa_planes(QUAL, 32 * K);
    const int wp = st.wp;
    const uint32_t mine = 0x80000000u >> lane;  // the lane's column in a 32-column word
    const int listMax = 64 * wp;  // entries the staging area holds
    using Bits = std::conditional_t<(K <= 16), uint32_t, uint64_t>;  // two bits per 32 columns
    Bits anchorBits = 0;  // bits 2 k: the anchor's base in column 32 k + lane
#pragma unroll
    for (int k = 0; k < K; k++) {
        const uint32_t* planes = st.hilo + aid * (2 * (uint64_t)wp) + k;
        anchorBits |= (Bits)((planes[0] & mine ? 2u : 0u) + (planes[wp] & mine ? 1u : 0u)) << (2 * k);
    }
    Bits refBits = 0;  // bits 2 k: the base of column 32 k + lane
    auto ref_entry = [&](int k) -> uint2* { return wc + (uint32_t)((refBits >> (2 * k)) & 3u) * (uint32_t)lp + (uint32_t)(32 * k + lane); };
    // The rows still in the MSA (add), or the rows just removed (marked kNew, the
    // mark is cleared) with their weights' signs turned, are added to wc.  Returns
    // their number.
    auto planePass = [&](const bool add) -> int {
        int selected = 0;
#pragma unroll 1
        for (uint32_t j0 = 0; j0 < nf; j0 += 32) {
            const uint32_t jr = j0 + lane;
            uint32_t mo = kRm, mid = 0;
            int shift = 0, len = 0;
            float mw = 0.0f;
            if (jr < nf) {
                mo = b.forient[base + jr];
                shift = b.fshift[base + jr];
                len = b.flen[base + jr];
                mid = b.fid[base + jr];
                mw = b.fweight[base + jr];
            }
            const bool sel = jr < nf && (add ? !(mo & kRm) : (mo & kNew) != 0);
            const unsigned selRows = __ballot_sync(kFull, sel);
            if (!selRows) continue;
            if (sel) {  // the row's planes
                const uint32_t* src = st.hilo + (uint64_t)mid * (2 * wp);
                for (int q = 0; q < 2 * wp; q += 4) cp_async16(stage + lane * 2 * wp + q, src + q);
            }
            if (!add && sel) b.forient[base + jr] = (uint8_t)(mo & ~kNew);
            if (!add) mw = -mw;
            weight[lane] = sel ? mw : 0.0f;
            const bool rc = (mo & 3u) == 2;
            cp_async_wait_all();
            __syncwarp();
            // Columns 32 k .. 32 k + 31 of the row.  Forward they are the stored bases
            // from -shift + 32 k on; for a reverse complement the last of them is base
            // len - 32 + shift - 32 k, their order turned.  Words in front of or behind
            // the row's are whatever lies there in the warp's slice (at most K words before
            // and K after the staged rows, wp being at least K); the valid columns
            // leave them out.
            uint32_t hi[K], lo[K], miss[K];
            uint32_t rowsOf[K];  // bit 31 - r: row r matches in the lane's column
            const int to = sel ? min(La, shift + len) : 0;  // its columns: shift .. to - 1
            int cnt = 0;
            {
                const int p0 = rc ? len - 32 + shift : -shift, step = rc ? -1 : 1;
                const uint32_t* h = stage + lane * 2 * wp + (p0 >> 5) + (rc ? 1 : 0);
                const uint32_t turn = rc ? 32u - (uint32_t)(p0 & 31) : (uint32_t)(p0 & 31), flip = rc ? ~0u : 0u;
                uint32_t h0 = h[0], l0 = h[wp];
                if (rc) {
                    h0 = __brev(h0);
                    l0 = __brev(l0);
                }
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (K > 5 && 32 * k >= La) {  // (a store of reads of many lengths)
                        hi[k] = lo[k] = miss[k] = rowsOf[k] = 0;
                        continue;
                    }
                    h += step;
                    uint32_t h1 = h[0], l1 = h[wp];
                    if (rc) {
                        h1 = __brev(h1);
                        l1 = __brev(l1);
                    }
                    hi[k] = __funnelshift_lc(h1, h0, turn) ^ flip;
                    lo[k] = __funnelshift_lc(l1, l0, turn) ^ flip;
                    h0 = h1;
                    l0 = l1;
                    const uint32_t valid = bits_from(shift - 32 * k) & bits_to(to - 32 * k);
                    const uint32_t x = (hi[k] ^ ref[k]) | (lo[k] ^ ref[wp + k]);
                    rowsOf[k] = valid & ~x;
                    miss[k] = valid & x;
                }
            }
            transpose_bits(rowsOf, lane);
            if (add && !selected) {
                // a column in which far fewer rows match than in the next one: most
                // likely the anchor's error; its base is then the first mismatching
                // row's
                unsigned odd[K], some = 0;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const int have = __popc(rowsOf[k]);
                    odd[k] = __ballot_sync(kFull, 4 * have < __shfl_xor_sync(kFull, have, 1));
                    some |= (odd[k] ? 1u : 0u) << k;
                }
#pragma unroll 1
                while (some) {  // (one copy of the code for the K words)
                    const int k = __ffs(some) - 1;
                    unsigned cols = pick<K>(odd, k);
                    const int c = __ffs(cols) - 1;
                    cols &= cols - 1;
                    put<K>(odd, k, cols);
                    if (!cols) some &= some - 1;
                    const uint32_t bit = 0x80000000u >> c, h = pick<K>(hi, k) & bit, l = pick<K>(lo, k) & bit;
                    uint32_t m = pick<K>(miss, k);
                    const unsigned differ = __ballot_sync(kFull, (m & bit) != 0);
                    if (!differ) continue;
                    const uint32_t nh = __shfl_sync(kFull, h, __ffs(differ) - 1);
                    const uint32_t nl = __shfl_sync(kFull, l, __ffs(differ) - 1);
                    const bool in = 32 * k + c >= shift && 32 * k + c < to;
                    const bool same = in && h == nh && l == nl;
                    m = (m & ~bit) | (in && !same ? bit : 0u);
                    put<K>(miss, k, m);
                    const unsigned now = __ballot_sync(kFull, same);
                    if (lane == c) {
                        put<K>(rowsOf, k, __brev(now));
                        refBits ^= (((refBits >> (2 * k)) & 3u) ^ (Bits)((nh ? 2u : 0u) | (nl ? 1u : 0u))) << (2 * k);
                        ref[k] = (ref[k] & ~bit) | nh;
                        ref[wp + k] = (ref[wp + k] & ~bit) | nl;
                    }
                    __syncwarp();
                }
            }
            selected += __popc(selRows);
            // the mismatches, listed as row << 20 | base << 16 | column
#pragma unroll
            for (int k = 0; k < K; k++) cnt += __popc(miss[k]);
            int incl = cnt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(kFull, incl, d);
                if (lane >= d) incl += y;
            }
            const int total = __shfl_sync(kFull, incl, 31);  // all rows' planes have been read
            for (int from = 0; from < total; from += listMax) {
                int at = incl - cnt - from;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    for (uint32_t x = miss[k]; x != 0u;) {
                        const int bit = __clz(x);
                        x ^= 0x80000000u >> bit;
                        const uint32_t q = 2u * ((hi[k] << bit) >> 31) + ((lo[k] << bit) >> 31);
                        if ((unsigned)at < (unsigned)listMax)
                            list[at] = ((uint32_t)lane << 20) | (q << 16) | (uint32_t)(32 * k + bit);
                        at++;
                    }
                }
                __syncwarp();
                const int n0 = min(listMax, total - from);
                for (int e0 = 0; e0 < n0; e0 += 32) {
                    const bool has = e0 + lane < n0;
                    const uint32_t e = has ? list[e0 + lane] : 0xffffffffu;
                    const uint32_t c = e & 0xffffu, slot = ((e >> 16) & 3u) * (uint32_t)lp + c, r = (e >> 20) & 31u;
                    const float wt = weight[r];
                    const uint32_t before = __popc(__match_any_sync(kFull, e & 0xfffffu) & ((1u << lane) - 1u));
                    const uint32_t rounds = __reduce_max_sync(kFull, has ? before : 0u);
                    for (uint32_t t = 0; t <= rounds; t++) {
                        if (has && before == t) {
                            uint2 v = wc[slot];
                            v.x = __float_as_uint(__fadd_rn(__uint_as_float(v.x), wt));
                            v.y += add ? 1u : ~0u;
                            wc[slot] = v;
                        }
                        __syncwarp();
                    }
                }
            }
            // the matches
            const int rows = 32 - __clz(selRows);
            float w[K];
#pragma unroll
            for (int k = 0; k < K; k++) w[k] = rowsOf[k] ? __uint_as_float(ref_entry(k)->x) : 0.0f;
            uint32_t left[K];
#pragma unroll
            for (int k = 0; k < K; k++) left[k] = rowsOf[k];
#pragma unroll 1
            for (int r0 = 0; r0 < rows; r0 += 8) {
                float wr[8];
                *reinterpret_cast<float4*>(wr) = *reinterpret_cast<const float4*>(weight + r0);
                *reinterpret_cast<float4*>(wr + 4) = *reinterpret_cast<const float4*>(weight + r0 + 4);
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (K > 5 && 32 * k >= La) break;
#pragma unroll
                    for (int r = 0; r < 8; r++)
                        if (left[k] & (0x80000000u >> r)) w[k] = __fadd_rn(w[k], wr[r]);
                    left[k] <<= 8;
                }
            }
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (!rowsOf[k]) continue;
                uint2* const entry = ref_entry(k);
                const int n = __popc(rowsOf[k]);
                *entry = make_uint2(__float_as_uint(w[k]), entry->y + (add ? n : -n));
            }
            __syncwarp();  // the next chunk overwrites the staged rows and weights
        }
        __syncwarp();
        return selected;
    };

    // The same a row at a time, with the lanes over the row's columns: for quality
    // scores, where every base has its own weight, and for the longest reads
    // (msa_planes).  (With qualities the other pass needs a load per row and 32 columns for the matches' qualities as well, and
    // then measured 6.5 ms where this one takes 5.5: 300,000 reads of 50 to 250 bp.)
    auto rowPass = [&](const bool add) -> int {
        int selected = 0;
        const uint32_t one = add ? 1u : ~0u;
#pragma unroll 1
        for (uint32_t j0 = 0; j0 < nf; j0 += 32) {
            const uint32_t jr = j0 + lane;
            const int rows = (int)min(32u, nf - j0);
            uint32_t mo = kRm, mid = 0;
            int shift = 0, len = 0;
            float mw = 0.0f;
            if (jr < nf) {
                mo = b.forient[base + jr];
                shift = b.fshift[base + jr];
                len = b.flen[base + jr];
                mid = b.fid[base + jr];
                mw = b.fweight[base + jr];
            }
            const bool sel = jr < nf && (add ? !(mo & kRm) : (mo & kNew) != 0);
            const unsigned selRows = __ballot_sync(kFull, sel);
            if (!selRows) continue;
            selected += __popc(selRows);
            if (!add && sel) b.forient[base + jr] = (uint8_t)(mo & ~kNew);
            if (sel) {
                const uint32_t* src = st.hilo + (uint64_t)mid * (2 * wp);
                for (int q = 0; q < 2 * wp; q += 4) cp_async16(stage + lane * 2 * wp + q, src + q);
            }
            meta[lane] = make_int4(shift, len | (int)((mo & 3u) << 16), __float_as_int(add ? mw : -mw), (int)mid);
            cp_async_wait_all();
            __syncwarp();
#pragma unroll 1
            for (int r = 0; r < rows; r++) {
                if (!((selRows >> r) & 1u)) continue;
                const int4 md = meta[r];
                const bool rc = ((uint32_t)md.y >> 16) == 2;
                const int rshift = md.x, rlen = md.y & 0xffff;
                const float wr = __int_as_float(md.z);
                const uint32_t* h = stage + r * 2 * wp;
                const int c0 = max(rshift, 0), c1 = min(La, rshift + rlen);  // overlap with the anchor
                int c = c0 + ((lane - c0) & 31);                             // this lane's first column
                // the row position moves by 32 per column step of the lane, so its
                // word moves by one and its bit stays
                int sp = rc ? rlen - 1 - (c - rshift) : c - rshift;
                const int dsp = rc ? -32 : 32, dwi = rc ? -1 : 1;
                const int up = sp & 31;
                const uint32_t flip = rc ? 3u : 0u;
                // quality of position sp (row_quality; padding past the read's end is
                // read as stored)
                const uint8_t* q = QUAL ? st.qual + (uint64_t)(uint32_t)md.w * st.lmax + (rc ? st.lmax - rlen : 0)
                                        : nullptr;
                auto weightAt = [&](int p) { return QUAL ? __fmul_rn(wr, qw[q[p]]) : wr; };
                auto baseAt = [&](int w) -> uint32_t {
                    return (((h[w] << up) >> 31) * 2u + ((h[wp + w] << up) >> 31)) ^ flip;
                };
                auto upd = [&](uint2& v, float wt) {
                    v.x = __float_as_uint(__fadd_rn(__uint_as_float(v.x), wt));
                    v.y += one;
                };
                int wi = sp >> 5;
                // two of the lane's columns (c and c + 32) per iteration: both words and
                // both entries are read before either is written (distinct columns,
                // distinct entries)
                for (; c + 32 < c1; c += 64, wi += 2 * dwi, sp += 2 * dsp) {
                    const uint32_t b0 = baseAt(wi), b1 = baseAt(wi + dwi);
                    const float w0 = weightAt(sp), w1 = weightAt(sp + dsp);
                    uint2* p0 = wc + b0 * lp + c;
                    uint2* p1 = wc + b1 * lp + (c + 32);
                    uint2 v0 = *p0, v1 = *p1;
                    upd(v0, w0);
                    upd(v1, w1);
                    *p0 = v0;
                    *p1 = v1;
                }
                if (c < c1) {
                    uint2* p0 = wc + baseAt(wi) * lp + c;
                    uint2 v0 = *p0;
                    upd(v0, weightAt(sp));
                    *p0 = v0;
                }
            }
            __syncwarp();  // the next chunk overwrites the staged rows
        }
        __syncwarp();
        return selected;
    };
    // add: builds the MSA of the rows still in it as the reference does, from the
    // anchor row (weight 1 times the quality weight) and the rows in order.
    // Otherwise takes the rows just removed out of wc.  Returns the number of rows.
    auto rowsPass = [&](const bool add) -> int {
        if (add) {
            refBits = anchorBits;
            if (kPlanes)
                for (int i = lane; i < 2 * wp; i += 32) ref[i] = st.hilo[aid * (2 * (uint64_t)wp) + i];
#pragma unroll
            for (int k = 0; k < K; k++) {
                const int c = 32 * k + lane;
                if (c >= La) break;
#pragma unroll
                for (int q = 0; q < 4; q++) wc[q * lp + c] = make_uint2(0u, 0u);
                *ref_entry(k) = make_uint2(__float_as_uint(QUAL ? __fmul_rn(1.0f, qw[aq[c]]) : 1.0f), 1u);
            }
        }
        if constexpr (kPlanes)
            return planePass(add);
        else
            return rowPass(add);
    };

    // Rounds of refinement.  A round begins with a build, or with the removal of
    // the rows that the one before it took out; `last` ends them after the next
    // build.  Everything that is read from a column's sums is read once a round,
    // and stays in registers: the consensus (consBits, as anchorBits), whether at
    // most two rows have the anchor's base (fewBits), the support, the coverage.
    int builds = 1, iter = 0, nActive = -1;
    bool build = true, haveS = false, last = false;
    Bits consBits;
    uint32_t fewBits;
    float support[K];
    int minc, maxc;
    const float tol = __fmul_rn(2.5f * 5.9604645e-8f, (float)(3 * nf + 4));  // 2 E_c / S_c with slack
    while (true) {
        const int rows = rowsPass(build);
        if (nActive < 0) nActive = rows;
        const bool exact = build;
        bool close = false, mism = false;
        int firstSig = 0x7fffffff;
        consBits = 0;
        fewBits = 0;
        minc = 0x7fffffff;
        maxc = -1;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int c = 32 * k + lane;
            support[k] = 0.0f;
            if (c >= La) continue;
            float v[4];
            int n[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint2 e = wc[q * lp + c];
                v[q] = __uint_as_float(e.x);
                n[q] = (int)e.y;
            }
            const float colW = __fadd_rn(__fadd_rn(__fadd_rn(v[0], v[1]), v[2]), v[3]);
            float consW = v[0];
            uint32_t cons = 0;
#pragma unroll
            for (int q = 1; q < 4; q++)
                if (v[q] > consW) {
                    consW = v[q];
                    cons = q;
                }
            if (!exact) {  // are the two largest weights too close to tell them apart?
                float t1 = 0.0f, t2 = 0.0f;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    t2 = fmaxf(t2, fminf(t1, v[q]));
                    t1 = fmaxf(t1, v[q]);
                }
                close |= !(__fsub_rn(t1, t2) > __fmul_rn(tol, sup[c]));
            }
            const uint32_t ab = (uint32_t)(anchorBits >> (2 * k)) & 3u;
            mism |= cons != ab;
            bool sig = false;
#pragma unroll
            for (int q = 0; q < 4; q++) sig |= (uint32_t)q != cons && p.significantCount <= n[q];
            if (sig) firstSig = min(firstSig, c);
            consBits |= (Bits)cons << (2 * k);
            if ((ab & 2u ? (ab & 1u ? n[3] : n[2]) : (ab & 1u ? n[1] : n[0])) <= 2) fewBits |= 1u << k;
            support[k] = __fdiv_rn(consW, colW);
            const int cov = n[0] + n[1] + n[2] + n[3];
            minc = min(minc, cov);
            maxc = max(maxc, cov);
        }
        if (last) break;
        last = build = true;  // unless rows are removed below
        if (iter == 5 || nActive == 0) {
            if (exact) break;
            continue;
        }
        if (__any_sync(kFull, close)) {
            last = false;  // the round again, from an exact MSA
            continue;
        }
        // findCandidatesOfDifferentRegion (src/msa.cpp:532-734), in anchor coordinates
        const int col = __reduce_min_sync(kFull, firstSig);
        if (!__any_sync(kFull, mism) || col == 0x7fffffff) {
            if (exact) break;
            continue;
        }
        int found;
        {
            const ColInfo ci = col_info(wc, lp, col);
            const int cidx = base_index(ci.cons);
            found = -1;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (i != cidx && p.significantCount <= (int)ci.n[i]) found = i;
        }
        const uint32_t orig = get2bit(aenc, col);
        const bool keepMatching = orig == (uint32_t)found;
        auto differs = [&](uint32_t j) -> bool {
            const uint32_t g = base + j;
            const int sh = b.fshift[g];
            const int len = b.flen[g];
            if (col < sh || col >= sh + len) return false;
            const uint32_t* e = st.enc + (uint64_t)b.fid[g] * pitch;
            const int pos = col - sh;
            const bool rc = (b.forient[g] & 3) == 2;
            uint32_t bb = get2bit(e, rc ? len - 1 - pos : pos);
            if (rc) bb = 3u - bb;
            return keepMatching ? (bb != (uint32_t)found) : (bb == (uint32_t)found);
        };
        bool veto = false, any = false;
#pragma unroll 1
        for (uint32_t j = lane; j < nf; j += 32) {
            if ((b.forient[base + j] & kRm) || !differs(j)) continue;
            any = true;
            veto |= b.fweight[base + j] >= 0.90f;
        }
        // a veto (or nothing to remove) leaves the MSA as it is; the
        // reference then rebuilds the same MSA and reaches the same decision
        if (__any_sync(kFull, veto) || !__any_sync(kFull, any)) {
            if (exact) break;
            continue;
        }
        int act = 0;
#pragma unroll 1
        for (uint32_t j = lane; j < nf; j += 32) {
            const uint8_t o = b.forient[base + j];
            if (!(o & kRm) && differs(j)) b.forient[base + j] = o | kRm | kNew;
            else act += !(o & kRm);
        }
        nActive = __reduce_add_sync(kFull, act);
        if (!haveS) {  // S_c (the first build, which wc still holds), kept in `sup` until the properties
#pragma unroll 1
            for (int c = lane; c < La; c += 32) sup[c] = col_info(wc, lp, c).colW;
            haveS = true;
        }
        __syncwarp();
        last = build = false;
        iter++;
        builds++;
    }
    // getMSAProperties (src/msa.cpp:304-376) and the decision
    float mins = 3.402823466e+38f;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int c = 32 * k + lane;
        if (c >= La) continue;
        sup[c] = support[k];
        mins = fminf(mins, support[k]);
    }
    for (int d = 16; d > 0; d >>= 1) mins = fminf(mins, __shfl_xor_sync(kFull, mins, d));
    minc = __reduce_min_sync(kFull, minc);
    maxc = __reduce_max_sync(kFull, maxc);
    __syncwarp();
    float avg = 0.0f;
    if (lane == 0) {  // in column order, four columns per shared-memory load
        float sum = 0.0f;
        const float4* s4 = reinterpret_cast<const float4*>(sup);
        int i = 0;
#pragma unroll 4
        for (; i + 4 <= La; i += 4) {
            const float4 v = s4[i >> 2];
            sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
        }
#pragma unroll 1
        for (; i < La; i++) sum = __fadd_rn(sum, sup[i]);
        avg = __fdiv_rn(sum, (float)La);
    }
    avg = __shfl_sync(kFull, avg, 0);
    const bool good = fgeq(avg, p.avgSupportThreshold) && fgeq(mins, p.minSupportThreshold) &&
                      fgeq((float)minc, p.minCoverageThreshold);
    bool hq = false;
    if (good) {
        int smallest = 100;
#pragma unroll 1
        for (int percent = p.errPercent; percent >= 0; percent--) {
            if (fgeq(avg, p.hqAvg[percent]) && fgeq(mins, p.hqMin[percent])) smallest = percent;
        }
        hq = fgeq((float)minc, p.minCoverageThreshold) && fleq((float)smallest, p.hqPercentLimit);
    }
    const bool forest = p.correctionType == CG_CORR_FOREST;
    const bool corrected = forest || nActive > 0;
    if (lane == 0) {
        if (corrected) {
            atomicAdd(&b.counters[kCounterCorrected], 1ull);
            if (hq) atomicAdd(&b.counters[kCounterHQ], 1ull);
        }
        atomicAdd(&b.counters[kCounterMsaBuilds], (unsigned long long)builds);
        b.flags[oi] = corrected ? (uint8_t)(CG_RESULT_CORRECTED | (hq ? CG_RESULT_HQ : 0)) : (uint8_t)0;
    }
    if (!corrected) return;
    if (!forest) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int c = 32 * k + lane;
            const bool take = good || (support[k] > 0.90f && ((fewBits >> k) & 1u));
            const uint32_t code = (uint32_t)((take ? consBits : anchorBits) >> (2 * k)) & 3u;
            if (c < La) out[c] = (char)__byte_perm(0x54474341u, 0u, code);  // "ACGT"[code]
        }
    }
#pragma unroll 1
    for (int c = lane; forest && c < La; c += 32) {
        const uint32_t ab = get2bit(aenc, c);
        const char orig = "ACGT"[ab];
        const ColInfo ci = col_info(wc, lp, c);
        const int origCov = (int)ci.nOf(ab);
        // correctAnchorClf (include/corrector.hpp:1448-1472), features of
        // include/classification.hpp:748-797
        char r = ci.cons;
        if (!hq && r != orig) {
            const int ci_ = base_index(ci.cons);
            const float wCons = ci.wOf((uint32_t)ci_);
            const float nCons = (float)ci.nOf((uint32_t)ci_);
            const float wOrig = ci.wOf(ab);
            const float cv = (float)ci.cov();
            const float oc = (float)origCov;
            const float ec = p.estimatedCoverage;
            const float f[13] = {__fdiv_rn(oc, cv),      __fdiv_rn(wOrig, ci.colW), __fdiv_rn(wOrig, oc),
                                 __fdiv_rn(nCons, cv),   sup[c],                    __fdiv_rn(wCons, nCons),
                                 __fdiv_rn(ci.colW, cv), __fdiv_rn(cv, ec),         __fdiv_rn(ci.colW, ec),
                                 avg,                    mins,                      __fdiv_rn((float)maxc, ec),
                                 __fdiv_rn((float)minc, ec)};
            if (!forest_decide(p, f)) r = orig;
        }
        out[c] = r;
    }
    if (p.candidates && hq) {
        // Candidate correction.  The MSA above holds the anchor's columns
        // only; the consensus of the nc columns on either side is summed here,
        // rows in list order, lane e0 + lane owning extension column e (column
        // e - nc left of the anchor, or La + e - nc right of it).  cons8[x] =
        // consensus base code of column x - nc, for x in [0, La + 2 nc).
        const int nc = p.newColumns;
        uint8_t* cons8 = reinterpret_cast<uint8_t*>(sm + sl.cons);
#pragma unroll 1
        for (int c = lane; c < La; c += 32) cons8[nc + c] = (uint8_t)base_index(col_info(wc, lp, c).cons);
#pragma unroll 1
        for (int e0 = 0; e0 < 2 * nc; e0 += 32) {  // warp-uniform trip count
            const int e = e0 + lane;
            const int col = e < nc ? e - nc : La + (e - nc);
            float w4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
            for (uint32_t j0 = 0; j0 < nf; j0 += 32) {
                const uint32_t jr = j0 + lane;
                const int rows = (int)min(32u, nf - j0);
                uint32_t mo = kRm, mid = 0;
                int mshift = 0, mlen = 0;
                float mw = 0.0f;
                if (jr < nf) {
                    mo = b.forient[base + jr];
                    mshift = b.fshift[base + jr];
                    mlen = b.flen[base + jr];
                    mid = b.fid[base + jr];
                    mw = b.fweight[base + jr];
                }
                // rows still in the MSA that reach past either end of the anchor
                const bool sel = jr < nf && !(mo & kRm) && (mshift < 0 || mshift + mlen > La);
                const unsigned selRows = __ballot_sync(kFull, sel);
                if (!selRows) continue;
#pragma unroll 1
                for (int i0 = 0; i0 < rows * pitch; i0 += 32) {
                    const int idx = i0 + lane;
                    const int r = min(idx / pitch, rows - 1);
                    const uint32_t rid = __shfl_sync(kFull, mid, r);
                    if (idx < rows * pitch && ((selRows >> r) & 1u))
                        stage[idx] = st.enc[(uint64_t)rid * pitch + (idx - r * pitch)];
                }
                meta[lane] = make_int4(mshift, mlen | (int)((mo & 3u) << 16), __float_as_int(mw), (int)mid);
                __syncwarp();
#pragma unroll 1
                for (int r = 0; r < rows; r++) {
                    if (!((selRows >> r) & 1u)) continue;
                    const int4 md = meta[r];
                    const bool rc = ((uint32_t)md.y >> 16) == 2;
                    const int len = md.y & 0xffff;
                    const int pos = col - md.x;
                    if (e >= 2 * nc || pos < 0 || pos >= len) continue;
                    const int sp = rc ? len - 1 - pos : pos;
                    const uint32_t bb = ((stage[r * pitch + (sp >> 4)] >> (30u - 2u * (uint32_t)(sp & 15))) & 3u) ^
                                        (rc ? 3u : 0u);
                    float wt = __int_as_float(md.z);
                    if (QUAL)
                        wt = __fmul_rn(wt, qw[row_quality(st.qual + (uint64_t)(uint32_t)md.w * st.lmax, st.lmax, rc,
                                                          pos)]);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if ((uint32_t)q == bb) w4[q] = __fadd_rn(w4[q], wt);
                }
                __syncwarp();  // the next chunk overwrites the staged rows
            }
            if (e < 2 * nc) {  // src/msa.cpp:135-157: the first largest weight, A C G T
                int cb = 0;
                float cw = w4[0];
#pragma unroll
                for (int q = 1; q < 4; q++)
                    if (w4[q] > cw) {
                        cb = q;
                        cw = w4[q];
                    }
                cons8[e < nc ? e : La + e] = (uint8_t)cb;
            }
        }
        __syncwarp();
        // The consensus packed 32 columns per word, forward (fw: column x at
        // position x) and reverse complemented (rv: position y holds the
        // complement of column X - 1 - y), one zero word past each; a row's
        // slice is then a run of whole words at a bit offset in one of them.
        const int X = La + 2 * nc, nw = (X + 31) / 32;
        unsigned long long* fw =
            reinterpret_cast<unsigned long long*>(cons8 + ((size_t)lp + 2 * (size_t)nc + 15) / 16 * 16);
        unsigned long long* rv = fw + nw + 1;
        __syncwarp();
#pragma unroll 1
        for (int u = lane; u <= nw; u += 32) {
            unsigned long long f = 0, r = 0;
#pragma unroll 1
            for (int t = 0; t < 32; t++) {
                const int x = 32 * u + t;
                if (x < X) {
                    f |= (unsigned long long)cons8[x] << (62 - 2 * t);
                    r |= (unsigned long long)(3u - cons8[X - 1 - x]) << (62 - 2 * t);
                }
            }
            fw[u] = f;
            rv[u] = r;
        }
        __syncwarp();
        // one row per lane
        int votes = 0;
#pragma unroll 1
        for (uint32_t j = lane; j < nf; j += 32) {
            const uint32_t g = base + j;
            const uint8_t o = b.forient[g];
            if (o & kRm) continue;
            const int s = b.fshift[g], len = b.flen[g];
            if (s < -nc || s > nc || s + len > La + nc) continue;
            const bool rc = (o & 3) == 2;
            const unsigned long long* src = rc ? rv : fw;
            const int y0 = rc ? X - (nc + s) - len : nc + s;  // the slice's first position in src
            const uint32_t id = b.fid[g];
#pragma unroll 1
            for (int w = 0; w * 32 < len; w++) {
                const int y = y0 + 32 * w, u = y >> 5, off = 2 * (y & 31);
                unsigned long long v = src[u] << off;
                if (off) v |= src[u + 1] >> (64 - off);
                const int rest = len - 32 * w;
                if (rest < 32) v &= ~0ull << (64 - 2 * rest);
                vote_word(p, id, w, v);
            }
            atomicAdd((uint64_t)id > aid ? &p.candVotes[id].x : &p.candVotes[id].y, 1u);
            votes++;
        }
        votes = __reduce_add_sync(kFull, votes);
        if (lane == 0 && votes) atomicAdd(&b.counters[kCounterCandidateVotes], (unsigned long long)votes);
        return;
    }
    if (p.correctionType != CG_CORR_LEARNED || hq) return;
    // Learned decision: record every column whose consensus differs from the
    // anchor's base, with its features; the classifier then replaces the
    // decision written above (the fallback) where it is confident.
    // The columns are listed first, in order, so that a lane takes one each.
    uint32_t differ = 0;  // bit k: column 32 k + lane
#pragma unroll
    for (int k = 0; k < K; k++)
        if (32 * k + lane < La && ((consBits ^ anchorBits) >> (2 * k) & 3u) != 0) differ |= 1u << k;
    int nd = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const unsigned m = __ballot_sync(kFull, (differ >> k) & 1u);
        if ((differ >> k) & 1u) list[nd + __popc(m & ((1u << lane) - 1u))] = (uint32_t)(32 * k + lane);
        nd += __popc(m);
    }
    if (nd == 0) return;
    unsigned slot0 = 0;
    if (lane == 0) slot0 = atomicAdd(b.colCount, (unsigned)nd);
    slot0 = __shfl_sync(kFull, slot0, 0);
    __syncwarp();
    const float ec = p.estimatedCoverage;
    const float invLa = __fdiv_rn(1.0f, (float)La);
#pragma unroll 1
    for (int i = lane; i < nd; i += 32) {
        const unsigned slot = slot0 + (unsigned)i;
        if (slot >= b.colCap) break;
        const int c = (int)list[i];
        const uint32_t ab = get2bit(aenc, c);
        const ColInfo ci = col_info(wc, lp, c);
        const int cb = base_index(ci.cons);
        float n4[4], w4[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            n4[q] = (float)ci.n[q];
            w4[q] = ci.w[q];
        }
        auto pick = [](const float (&v)[4], uint32_t i) {
            return i == 0 ? v[0] : i == 1 ? v[1] : i == 2 ? v[2] : v[3];
        };
        const float cov = __fadd_rn(__fadd_rn(__fadd_rn(n4[0], n4[1]), n4[2]), n4[3]);
        const float icov = __fdiv_rn(1.0f, cov);
        const float icw = ci.colW > 0.0f ? __fdiv_rn(1.0f, ci.colW) : 0.0f;
        // Ratios that sit near 1 enter as 1 - ratio: BF16 keeps about three
        // significant digits, so 0.983 and 0.987 would be the same value but
        // 0.017 and 0.013 are not.
        const float na = pick(n4, ab), nc = pick(n4, (uint32_t)cb);
        float second = 0.0f;  // the second largest base weight
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (q != cb) second = fmaxf(second, w4[q]);
        float f[kLearnedFeatures];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            f[q] = __fmul_rn(n4[q], icov);                 // base counts / coverage
            f[4 + q] = __fmul_rn(w4[q], icw);              // weights / column weight
            f[18 + q] = q == cb ? 1.0f : 0.0f;             // consensus base
        }
        f[8] = __fdiv_rn(cov, ec);
        f[9] = __fdiv_rn(ci.colW, ec);
        f[10] = __fsub_rn(1.0f, sup[c]);
        f[11] = __fmul_rn(pick(w4, ab), icw);
        f[12] = __fmul_rn(na, icov);
        f[13] = __fsub_rn(1.0f, __fmul_rn(nc, icov));
        f[14] = __fsub_rn(1.0f, __fdiv_rn(pick(w4, ab), na));                   // mean weight of the anchor base's rows
        f[15] = nc > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(ci.consW, nc)) : 1.0f;   // ... of the consensus base's rows
        f[16] = __fsub_rn(1.0f, __fmul_rn(ci.colW, icov));                      // ... of all rows
        f[17] = __fmul_rn(second, icw);                                          // runner-up weight / column weight
        f[22] = __fmul_rn((float)c, invLa);
        f[23] = __fmul_rn((float)min(c, La - 1 - c), invLa);
        f[24] = __fsub_rn(1.0f, avg);
        f[25] = __fsub_rn(1.0f, mins);
        f[26] = __fdiv_rn((float)minc, ec);
        f[27] = __fdiv_rn((float)maxc, ec);
        f[28] = __fmul_rn((float)La, 1.0f / 256.0f);
        f[29] = __fmul_rn((float)nd, invLa);
        f[30] = __fdiv_rn((float)nActive, ec);
        f[31] = QUAL ? qw[aq[c]] : 1.0f;
        uint32_t wd[kLearnedFeatures / 2];
#pragma unroll
        for (int k = 0; k < kLearnedFeatures / 2; k++) {
            const __nv_bfloat162 v = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
            wd[k] = *reinterpret_cast<const uint32_t*>(&v);
        }
        uint4* dst = reinterpret_cast<uint4*>(b.colFeat + (uint64_t)slot * kLearnedFeatures);
#pragma unroll
        for (int k = 0; k < kLearnedFeatures / 8; k++)
            dst[k] = make_uint4(wd[4 * k], wd[4 * k + 1], wd[4 * k + 2], wd[4 * k + 3]);
        b.colMeta[slot] = make_uint2((uint32_t)oi, (uint32_t)c | ((uint32_t)(uint8_t)ci.cons << 16));
    }
}

// `warps` warps per block, each on its own anchors.  Plain form: anchor
// blockIdx.x * warps + warp.  Persistent form (b.work set): warps take the
// next anchor from the counter b.work[0] until the batch is done.
// Registers: as many as the K-word arrays need without lowering the number of
// resident one-warp blocks much, which shared memory bounds: 27 per SM at K = 5 (23
// with quality scores), 16 at K = 8, 14 at K = 10, 9, 7 and 4 at 16, 20 and 32.  MSA
// stage: 2M anchors of 150 bp 12.9 ms with 72 (13.7 with 64, which spill, 13.8 with
// 88), 300,000 with qualities 3.98 with 72 (4.02 with 64, 4.17 with 88); 200,000 of
// 250 bp 2.57 with 112 (2.99 with 80, 2.49 with 96), 100,000 with qualities 2.22 (2.20
// with 80, 2.25 with 96, 2.39 with 128); 60,000 of 300 bp 0.70 with 128 (0.71 with
// 112; 0.75 with 144 and 168, which leave room for 12 blocks), with qualities 1.39 with
// any of them.  At K = 16 and above the
// rows are added one at a time and need fewer: with qualities, 40,000 of 500 bp 2.08,
// 30,000 of 640 bp 2.18 and 20,000 of 1000 bp 3.56 with 168 (2.14, 2.23 and 3.67 with
// 128; 2.12, 2.35 and 3.64 with 224, 255 and 255).  256 threads, the most a block has,
// fit the register file in each case.
template <bool QUAL, int K>
__global__ void __maxnreg__(K > 10 ? 168 : K > 8 ? 128 : K > 5 ? 112 : 72)
    msa_warp_kernel(StoreArg st, Params p, BatchArg b, const uint32_t* __restrict__ rawOff, int lp) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int warp = (int)(threadIdx.x >> 5), warps = (int)(blockDim.x >> 5);
    const MsaSlice sl(lp, st.pitch, st.wp, p, !msa_planes(QUAL, 32 * K));
    // The slice's address is kept in a register: left to itself the compiler builds
    // a shared address from the block's number in its cluster for every access.
    uint32_t at = (uint32_t)__cvta_generic_to_shared(sm + (QUAL ? 256 * sizeof(float) : 0) + (size_t)warp * sl.bytes);
    asm volatile("" : "+r"(at));
    unsigned char* slice = static_cast<unsigned char*>(__cvta_shared_to_generic(at));
    uint32_t qwAt = (uint32_t)__cvta_generic_to_shared(sm);
    asm volatile("" : "+r"(qwAt));
    float* qw = static_cast<float*>(__cvta_shared_to_generic(qwAt));  // [256] (quality scores only)
    if (QUAL) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) qw[i] = p.qweight[i];
        __syncthreads();
    }
    const uint64_t first = batch_first(b);
    const int lane = (int)lane_id();
    const bool persistent = b.work != nullptr;
    int i = blockIdx.x * warps + warp;
    do {
        if (persistent) {
            i = lane == 0 ? (int)atomicAdd(&b.work[0], 1u) : 0;
        }
        i = (int)warp_uniform((uint32_t)i);
        if (i >= b.count) return;
        const int a = (int)warp_uniform(b.order ? b.order[i] : (uint32_t)i);
        msa_warp_anchor<QUAL, K>(st, p, b, rawOff, lp, a, first, slice, sl, qw);
        __syncwarp();
    } while (persistent);
}

constexpr int kOrderBuckets = 16;

// bucket 0 holds the anchors with the most kept rows (nf >= 2^14), bucket 15
// those with none
__device__ __forceinline__ int order_bucket(uint32_t nf) { return 15 - min(15, 32 - __clz(nf)); }

__global__ void msa_order_hist_kernel(const uint32_t* __restrict__ nfinal, int count, unsigned int* hist) {
    __shared__ unsigned int h[kOrderBuckets];
    if (threadIdx.x < kOrderBuckets) h[threadIdx.x] = 0;
    __syncthreads();
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < count; a += gridDim.x * blockDim.x)
        atomicAdd(&h[order_bucket(nfinal[a])], 1u);
    __syncthreads();
    if (threadIdx.x < kOrderBuckets && h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], h[threadIdx.x]);
}

// Each block reserves its slots of every bucket with one global atomic per
// bucket per round (the per-anchor tickets come from shared memory).
__global__ void msa_order_scatter_kernel(const uint32_t* __restrict__ nfinal, int count,
                                         const unsigned int* __restrict__ hist, unsigned int* cursor,
                                         uint32_t* __restrict__ order) {
    __shared__ unsigned int start[kOrderBuckets], local[kOrderBuckets], base[kOrderBuckets];
    if (threadIdx.x == 0) {
        unsigned int acc = 0;
        for (int i = 0; i < kOrderBuckets; i++) {
            start[i] = acc;
            acc += hist[i];
        }
    }
    for (int a0 = blockIdx.x * blockDim.x; a0 < count; a0 += gridDim.x * blockDim.x) {
        if (threadIdx.x < kOrderBuckets) local[threadIdx.x] = 0;
        __syncthreads();
        const int a = a0 + threadIdx.x;
        int k = 0;
        unsigned int ticket = 0;
        if (a < count) {
            k = order_bucket(nfinal[a]);
            ticket = atomicAdd(&local[k], 1u);
        }
        __syncthreads();
        if (threadIdx.x < kOrderBuckets && local[threadIdx.x])
            base[threadIdx.x] = start[threadIdx.x] + atomicAdd(&cursor[threadIdx.x], local[threadIdx.x]);
        __syncthreads();
        if (a < count) order[base[k] + ticket] = (uint32_t)a;
        __syncthreads();
    }
}

}  // namespace

namespace {

// The instance for a store -- as many 32-column words as its longest read takes,
// every word costs a share of each pass -- and its shared memory per warp.
struct MsaInstance {
    void (*kernel)(StoreArg, Params, BatchArg, const uint32_t*, int);
    size_t slice;
};
template <int K>
MsaInstance msa_instance_of(StoreArg st, const Params& p) {
    return {p.useQuality ? msa_warp_kernel<true, K> : msa_warp_kernel<false, K>,
            MsaSlice((st.lmax + 31) / 32 * 32, st.pitch, st.wp, p, !msa_planes(p.useQuality, 32 * K)).bytes};
}
MsaInstance msa_instance(StoreArg st, const Params& p) {
    const int words = (st.lmax + 31) / 32;
    return words <= 4    ? msa_instance_of<4>(st, p)
           : words <= 5  ? msa_instance_of<5>(st, p)
           : words <= 8  ? msa_instance_of<8>(st, p)
           : words <= 10 ? msa_instance_of<10>(st, p)
           : words <= 16 ? msa_instance_of<16>(st, p)
           : words <= 20 ? msa_instance_of<20>(st, p)
                         : msa_instance_of<32>(st, p);
}

size_t msa_warp_smem(const MsaInstance& m, const Params& p, int warps) {
    return (p.useQuality ? 256 * sizeof(float) : 0) + (size_t)warps * m.slice;
}

// warps per block: as asked for, but no more than the shared memory of a block holds
int msa_fit_warps(const MsaInstance& m, const Params& p, int warps) {
    while (warps > 1 && msa_warp_smem(m, p, warps) > 227 * 1024) warps--;
    return warps < 1 ? 1 : warps;
}

cudaError_t msa_warp_prepare(const MsaInstance& m, size_t smem) {
    if (smem <= 40 * 1024) return cudaSuccess;  // leaves room for the kernel's static shared memory
    return cudaFuncSetAttribute(m.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

}  // namespace

int msa_warp_occupancy(StoreArg st, Params p, int warps) {
    const MsaInstance m = msa_instance(st, p);
    warps = msa_fit_warps(m, p, warps);
    const size_t smem = msa_warp_smem(m, p, warps);
    if (msa_warp_prepare(m, smem) != cudaSuccess) return 0;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, m.kernel, warps * 32, smem) != cudaSuccess) return 0;
    return blocks;
}

cudaError_t launch_msa_correct(StoreArg st, Params p, BatchArg b, cudaStream_t s, const Shape* shape) {
    const bool persistent = shape && b.work;
    const MsaInstance m = msa_instance(st, p);
    const int warps = persistent ? msa_fit_warps(m, p, shape->msaWarps) : 1;
    const size_t smem = msa_warp_smem(m, p, warps);
    const cudaError_t e = msa_warp_prepare(m, smem);
    if (e != cudaSuccess) return e;
    const unsigned blocks = persistent ? (unsigned)shape->msaBlocks : (unsigned)b.count;
    if (blocks == 0) return cudaSuccess;
    m.kernel<<<blocks, warps * 32, smem, s>>>(st, p, b, b.rawCount, (st.lmax + 31) / 32 * 32);
    return cudaGetLastError();
}

cudaError_t launch_msa_order(BatchArg b, unsigned int* scratch, uint32_t* order, cudaStream_t s) {
    if (b.count <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(scratch, 0, 2 * kOrderBuckets * sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    const unsigned blocks = (unsigned)min((b.count + 255) / 256, 304);
    msa_order_hist_kernel<<<blocks, 256, 0, s>>>(b.nfinal, b.count, scratch);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    msa_order_scatter_kernel<<<blocks, 256, 0, s>>>(b.nfinal, b.count, scratch, scratch + kOrderBuckets, order);
    return cudaGetLastError();
}

namespace {

// one warp per anchor of the batch; lane w packs word w of a low-quality
// anchor correction (the output row's bases) and votes with it
__global__ void __launch_bounds__(256) anchor_vote_kernel(StoreArg st, Params p, BatchArg b) {
    const int a = (int)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (a >= b.count) return;
    const uint64_t first = batch_first(b);
    const uint64_t aid = first + (uint64_t)a;
    const uint64_t oi = (first - out_first(b)) + (uint64_t)a;
    const uint8_t f = b.flags[oi];
    if (!(f & CG_RESULT_CORRECTED) || (f & CG_RESULT_HQ)) return;
    const int len = st.len[aid];
    const int w = (int)lane_id();
    if (w * 32 >= len) return;
    const char* o = b.out + oi * (uint64_t)b.outPitch;
    unsigned long long v = 0;
    const int pe = min(len, w * 32 + 32);
    for (int q = w * 32; q < pe; q++) v |= (unsigned long long)base_index(o[q]) << (62 - 2 * (q & 31));
    vote_word(p, aid, w, v);
}

// reference: src/correctionresultoutput.cpp:1256-1551 (combine), with the
// record filter of include/corrector.hpp:1678-1681 in a single-threaded run's
// order: read c's candidate records from anchors above c are not saved when c
// is a corrected HQ anchor.  One thread per read.
__global__ void combine_kernel(StoreArg st, Params p, uint64_t first, uint64_t n, uint8_t* __restrict__ flags,
                               unsigned long long* __restrict__ records) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long k = 0;
    if (i < n) {
        const uint64_t r = first + i;
        uint8_t f = flags[i];
        const uint2 v = p.candVotes[r];
        const bool hqAnchor = (f & CG_RESULT_CORRECTED) && (f & CG_RESULT_HQ);
        k = (unsigned long long)v.x + (hqAnchor ? 0ull : (unsigned long long)v.y);
        if (k) f |= CG_RESULT_CANDIDATE_RECORD;
        if ((f & CG_RESULT_CORRECTED) && !(f & CG_RESULT_HQ) && k >= 2) {
            const int words = (st.len[r] + 31) / 32;
            bool same = true;
            for (int w = 0; w < words; w++) {
                const uint64_t j = r * (uint64_t)p.candPitch + (uint64_t)w;
                same &= p.candAnd[j] == p.candOr[j];
            }
            f |= same ? CG_RESULT_CANDIDATES : CG_RESULT_REJECTED;
        }
        flags[i] = f;
    }
    for (int d = 16; d > 0; d >>= 1) k += __shfl_xor_sync(kFull, k, d);
    if ((threadIdx.x & 31) == 0 && k) atomicAdd(records, k);
}

__global__ void batch_advance_kernel(unsigned long long* cursor, unsigned int* work, unsigned long long stride) {
    cursor[0] += stride;
    work[0] = work[1] = work[2] = 0;
}
}  // namespace

cudaError_t launch_anchor_vote(StoreArg st, Params p, BatchArg b, cudaStream_t s) {
    if (b.count <= 0) return cudaSuccess;
    anchor_vote_kernel<<<(unsigned)((b.count + 7) / 8), 256, 0, s>>>(st, p, b);
    return cudaGetLastError();
}

cudaError_t launch_combine(StoreArg st, Params p, uint64_t first, uint64_t n, uint8_t* flags,
                           unsigned long long* records, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    combine_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(st, p, first, n, flags, records);
    return cudaGetLastError();
}

cudaError_t launch_batch_advance(unsigned long long* cursor, unsigned int* work, unsigned long long stride,
                                 cudaStream_t s) {
    batch_advance_kernel<<<1, 1, 0, s>>>(cursor, work, stride);
    return cudaGetLastError();
}

}  // namespace cg
