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

// ---------------------------------------------------------------- MSA

constexpr int kMsaThreadsMin = 128;
constexpr int kMsaCols = 4;  // columns owned per thread
constexpr int kMsaChunkRows = 512;

struct RowMeta {
    const uint32_t* enc;  // candidate's 2-bit row
    const uint8_t* qual;  // candidate's qualities (or null)
    float weight;
    int16_t shift;
    uint16_t len;
    uint8_t rc;
    uint8_t pad[7];
};
static_assert(sizeof(RowMeta) == 32, "row meta layout");

template <class T>
__device__ __forceinline__ T block_reduce(T v, T* red, int op /*0 min 1 max 2 sum*/) {
    for (int d = 16; d > 0; d >>= 1) {
        const T o = __shfl_xor_sync(kFull, v, d);
        v = op == 0 ? (o < v ? o : v) : op == 1 ? (o > v ? o : v) : v + o;
    }
    const int warp = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[warp] = v;
    __syncthreads();
    T r = red[0];
    for (int w = 1; w < nw; w++) r = op == 0 ? (red[w] < r ? red[w] : r) : op == 1 ? (red[w] > r ? red[w] : r) : r + red[w];
    return r;
}

// One block per anchor; column c belongs to thread c % blockDim (at most
// kMsaCols columns per thread, kept in registers while the rows stream by).
// Every column adds its rows in list order -- anchor first, then the kept
// candidates as the filters left them -- so each float sum is the
// reference's sequence of additions.  Row metadata is staged in shared memory
// in chunks of kMsaChunkRows rows; removed rows are a shared bitset.
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

// One thread votes for one row: cons(col) gives the consensus base code of
// column col (relative to the anchor's first column).  Returns 1 if it voted.
template <class Cons>
__device__ __forceinline__ int vote_candidate(const Params& p, int s, int len, bool rc, uint32_t id, uint64_t aid,
                                              int La, Cons cons) {
    const int nc = p.newColumns;
    if (s < -nc || s > nc || s + len > La + nc) return 0;
    for (int w = 0; w * 32 < len; w++) {
        unsigned long long v = 0;
        const int pe = min(len, w * 32 + 32);
        for (int q = w * 32; q < pe; q++) {
            uint32_t bb = cons(s + (rc ? len - 1 - q : q));
            if (rc) bb = 3u - bb;
            v |= (unsigned long long)bb << (62 - 2 * (q & 31));
        }
        vote_word(p, id, w, v);
    }
    atomicAdd((uint64_t)id > aid ? &p.candVotes[id].x : &p.candVotes[id].y, 1u);
    return 1;
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

__global__ void __launch_bounds__(1024) msa_correct_kernel(StoreArg st, Params p, BatchArg b,
                                                          const uint32_t* __restrict__ rawOff, int maxCols,
                                                          int bitsetWords, int storeWeights) {
    extern __shared__ __align__(16) unsigned char sm[];
    RowMeta* rows = reinterpret_cast<RowMeta*>(sm);
    uint32_t* removed = reinterpret_cast<uint32_t*>(rows + kMsaChunkRows);
    float* qw = reinterpret_cast<float*>(removed + bitsetWords);
    int* cntA = reinterpret_cast<int*>(qw + 256);
    int* cntC = cntA + maxCols;
    int* cntG = cntC + maxCols;
    int* cntT = cntG + maxCols;
    int* cov = cntT + maxCols;
    int* origCov = cov + maxCols;
    float* sup = reinterpret_cast<float*>(origCov + maxCols);
    // column weights, kept only for the forest's features
    float* colWA = storeWeights ? sup + maxCols : nullptr;
    float* colWC = storeWeights ? colWA + maxCols : nullptr;
    float* colWG = storeWeights ? colWC + maxCols : nullptr;
    float* colWT = storeWeights ? colWG + maxCols : nullptr;
    char* cons = reinterpret_cast<char*>(sup + maxCols + (storeWeights ? 4 * maxCols : 0));
    __shared__ float redf[32];
    __shared__ int redi[32];
    __shared__ int sCol, sFound, sByConsensus;

    const int a = blockIdx.x;
    const int tid = threadIdx.x;
    const int bd = blockDim.x;
    const uint64_t first = batch_first(b);
    const uint64_t aid = first + (uint64_t)a;
    const uint64_t oi = (first - out_first(b)) + (uint64_t)a;  // output row
    const uint32_t nf = b.nfinal[a];
    char* out = b.out + oi * b.outPitch;
    if (nf == 0) {
        if (tid == 0) b.flags[oi] = 0;
        return;
    }
    const uint32_t base = rawOff[a];
    const int La = st.len[aid];
    const uint32_t* aenc = st.enc + aid * (uint64_t)st.pitch;
    const uint8_t* aq = p.useQuality ? st.qual + aid * (uint64_t)st.lmax : nullptr;
    for (int i = tid; i < bitsetWords; i += bd) removed[i] = 0u;
    if (p.useQuality)
        for (int i = tid; i < 256; i += bd) qw[i] = p.qweight[i];
    const bool oneChunk = nf <= (uint32_t)kMsaChunkRows;
    auto loadRows = [&](uint32_t j0, uint32_t cnt) {
        for (uint32_t r = tid; r < cnt; r += bd) {
            const uint32_t j = base + j0 + r;
            const uint32_t id = b.fid[j];
            RowMeta m;
            m.enc = st.enc + (uint64_t)id * st.pitch;
            m.qual = p.useQuality ? st.qual + (uint64_t)id * st.lmax : nullptr;
            m.weight = b.fweight[j];
            m.shift = b.fshift[j];
            m.len = b.flen[j];
            m.rc = b.forient[j] == 2;
            rows[r] = m;
        }
    };
    if (oneChunk) loadRows(0, nf);
    __syncthreads();
    auto isRemoved = [&](uint32_t j) { return (removed[j >> 5] >> (j & 31)) & 1u; };

    int aBegin = 0, nActive = (int)nf, builds = 0;
    for (int iter = 0;; iter++) {
        // columns of the current MSA (src/msa.cpp:19-33)
        int lo = 0, hi = La, act = 0;
        for (uint32_t j = tid; j < nf; j += bd) {
            if (!isRemoved(j)) {
                const int s = b.fshift[base + j];
                lo = min(lo, s);
                hi = max(hi, s + (int)b.flen[base + j]);
                act++;
            }
        }
        lo = block_reduce<int>(lo, redi, 0);
        hi = block_reduce<int>(hi, redi, 1);
        nActive = block_reduce<int>(act, redi, 2);
        const int nCols = hi - lo;
        aBegin = -lo;
        const int aEnd = aBegin + La;
        // build: counts, weights (src/msa.cpp:93-112)
        int nA[kMsaCols], nC[kMsaCols], nG[kMsaCols], nT[kMsaCols];
        float wA[kMsaCols], wC[kMsaCols], wG[kMsaCols], wT[kMsaCols];
#pragma unroll
        for (int k = 0; k < kMsaCols; k++) {
            nA[k] = nC[k] = nG[k] = nT[k] = 0;
            wA[k] = wC[k] = wG[k] = wT[k] = 0.0f;
        }
        auto add = [&](int k, uint32_t bb, float w) {
            if (bb == 0) { nA[k]++; wA[k] = __fadd_rn(wA[k], w); }
            else if (bb == 1) { nC[k]++; wC[k] = __fadd_rn(wC[k], w); }
            else if (bb == 2) { nG[k]++; wG[k] = __fadd_rn(wG[k], w); }
            else { nT[k]++; wT[k] = __fadd_rn(wT[k], w); }
        };
#pragma unroll
        for (int k = 0; k < kMsaCols; k++) {
            const int c = tid + k * bd;
            if (c >= aBegin && c < aEnd) {
                const int pos = c - aBegin;
                const float w = p.useQuality ? __fmul_rn(1.0f, qw[aq[pos]]) : 1.0f;
                add(k, get2bit(aenc, pos), w);
            }
        }
        for (uint32_t j0 = 0; j0 < nf; j0 += kMsaChunkRows) {
            const uint32_t cnt = min((uint32_t)kMsaChunkRows, nf - j0);
            if (!oneChunk) {
                __syncthreads();
                loadRows(j0, cnt);
                __syncthreads();
            }
            for (uint32_t r = 0; r < cnt; r++) {
                if (isRemoved(j0 + r)) continue;
                const RowMeta m = rows[r];
                const int rb = aBegin + m.shift;
                const int re = rb + (int)m.len;
#pragma unroll
                for (int k = 0; k < kMsaCols; k++) {
                    const int c = tid + k * bd;
                    if (c >= rb && c < re) {
                        const int pos = c - rb;
                        const int sp = m.rc ? (int)m.len - 1 - pos : pos;
                        uint32_t bb = get2bit(m.enc, sp);
                        if (m.rc) bb = 3u - bb;
                        float w = m.weight;
                        if (p.useQuality) w = __fmul_rn(w, qw[row_quality(m.qual, st.lmax, m.rc, pos)]);
                        add(k, bb, w);
                    }
                }
            }
        }
        // findConsensus (src/msa.cpp:135-157), findOrigWeightAndCoverage (:159-173)
#pragma unroll
        for (int k = 0; k < kMsaCols; k++) {
            const int c = tid + k * bd;
            if (c < nCols) {
                char cs = 'A';
                float cw = wA[k];
                if (wC[k] > cw) { cs = 'C'; cw = wC[k]; }
                if (wG[k] > cw) { cs = 'G'; cw = wG[k]; }
                if (wT[k] > cw) { cs = 'T'; cw = wT[k]; }
                const float colW = __fadd_rn(__fadd_rn(__fadd_rn(wA[k], wC[k]), wG[k]), wT[k]);
                cntA[c] = nA[k]; cntC[c] = nC[k]; cntG[c] = nG[k]; cntT[c] = nT[k];
                cov[c] = nA[k] + nC[k] + nG[k] + nT[k];
                sup[c] = __fdiv_rn(cw, colW);
                cons[c] = cs;
                if (storeWeights) {
                    colWA[c] = wA[k]; colWC[c] = wC[k]; colWG[c] = wG[k]; colWT[c] = wT[k];
                }
                if (c >= aBegin && c < aEnd) {
                    const uint32_t ab = get2bit(aenc, c - aBegin);
                    origCov[c] = ab == 0 ? nA[k] : ab == 1 ? nC[k] : ab == 2 ? nG[k] : nT[k];
                }
            }
        }
        builds++;
        __syncthreads();
        if (iter == 5 || nActive == 0) break;
        // findCandidatesOfDifferentRegion (src/msa.cpp:532-734)
        bool mism = false;
        for (int c = aBegin + tid; c < aEnd; c += bd) mism |= cons[c] != "ACGT"[get2bit(aenc, c - aBegin)];
        if (!__syncthreads_or(mism)) break;
        if (tid == 0) sCol = 0x7fffffff;
        __syncthreads();
        for (int c = aBegin + tid; c < aEnd; c += bd) {
            const int counts[4] = {cntA[c], cntC[c], cntG[c], cntT[c]};
            const int ci = cons[c] == 'A' ? 0 : cons[c] == 'C' ? 1 : cons[c] == 'G' ? 2 : 3;
            bool sig = false;
            for (int i = 0; i < 4; i++) sig |= (i != ci && p.significantCount <= counts[i]);
            if (sig) atomicMin(&sCol, c);
        }
        __syncthreads();
        const int col = sCol;
        if (col == 0x7fffffff) break;
        if (tid == 0) {
            const int counts[4] = {cntA[col], cntC[col], cntG[col], cntT[col]};
            const int ci = cons[col] == 'A' ? 0 : cons[col] == 'C' ? 1 : cons[col] == 'G' ? 2 : 3;
            int si = -1;
            for (int i = 0; i < 4; i++)
                if (i != ci && p.significantCount <= counts[i]) si = i;
            sFound = si;
        }
        __syncthreads();
        const uint32_t found = (uint32_t)sFound;
        const uint32_t orig = get2bit(aenc, col - aBegin);
        const bool keepMatching = orig == found;
        auto differs = [&](uint32_t j) -> bool {  // row j lies on `col` and is to be removed
            const uint32_t g = base + j;
            const int rb = aBegin + b.fshift[g];
            const int len = b.flen[g];
            if (col < rb || col >= rb + len) return false;
            const uint32_t* e = st.enc + (uint64_t)b.fid[g] * st.pitch;
            const int pos = col - rb;
            const bool rc = b.forient[g] == 2;
            uint32_t bb = get2bit(e, rc ? len - 1 - pos : pos);
            if (rc) bb = 3u - bb;
            return keepMatching ? (bb != found) : (bb == found);
        };
        bool veto = false, any = false;
        for (uint32_t j = tid; j < nf; j += bd) {
            if (isRemoved(j) || !differs(j)) continue;
            any = true;
            veto |= b.fweight[base + j] >= 0.90f;
        }
        const bool anyVeto = __syncthreads_or(veto);
        const bool anyRemove = __syncthreads_or(any);
        // a veto (or nothing to remove) leaves the MSA as it is; the
        // reference then rebuilds the same MSA and reaches the same decision
        if (anyVeto || !anyRemove) break;
        for (uint32_t j = tid; j < nf; j += bd) {
            if (!isRemoved(j) && differs(j)) atomicOr(&removed[j >> 5], 1u << (j & 31));
        }
        __syncthreads();
    }
    // getMSAProperties (src/msa.cpp:304-376) and getCorrectedAnchor (:379-453)
    const int aEnd = aBegin + La;
    float mins = 3.402823466e+38f;
    int minc = 0x7fffffff, maxc = -1;
    for (int c = aBegin + tid; c < aEnd; c += bd) {
        mins = fminf(mins, sup[c]);
        minc = min(minc, cov[c]);
        maxc = max(maxc, cov[c]);
    }
    mins = block_reduce<float>(mins, redf, 0);
    minc = block_reduce<int>(minc, redi, 0);
    maxc = block_reduce<int>(maxc, redi, 1);
    __shared__ float sAvg;
    __shared__ int sHQ;
    if (tid == 0) {
        float sum = 0.0f;
        for (int c = aBegin; c < aEnd; c++) sum = __fadd_rn(sum, sup[c]);
        const float avg = __fdiv_rn(sum, (float)La);
        const bool good = fgeq(avg, p.avgSupportThreshold) && fgeq(mins, p.minSupportThreshold) &&
                          fgeq((float)minc, p.minCoverageThreshold);
        bool hq = false;
        if (good) {
            int smallest = 100;
            for (int percent = p.errPercent; percent >= 0; percent--) {
                if (fgeq(avg, p.hqAvg[percent]) && fgeq(mins, p.hqMin[percent])) smallest = percent;
            }
            hq = fgeq((float)minc, p.minCoverageThreshold) && fleq((float)smallest, p.hqPercentLimit);
        }
        sByConsensus = good;
        sAvg = avg;
        sHQ = hq;
        // the forest decision corrects every anchor that reached the MSA
        // (include/corrector.hpp:1448-1472); the classic one needs candidates
        const bool corrected = p.correctionType == CG_CORR_FOREST || nActive > 0;
        if (corrected) {
            atomicAdd(&b.counters[kCounterCorrected], 1ull);
            if (hq) atomicAdd(&b.counters[kCounterHQ], 1ull);
        }
        atomicAdd(&b.counters[kCounterMsaBuilds], (unsigned long long)builds);
        b.flags[oi] = corrected ? (uint8_t)(CG_RESULT_CORRECTED | (hq ? CG_RESULT_HQ : 0)) : (uint8_t)0;
    }
    __syncthreads();
    if (p.candidates && sHQ) {
        // candidate correction: one thread per row of the final MSA, whose
        // consensus covers every column of the rows
        int votes = 0;
        for (uint32_t j = tid; j < nf; j += bd) {
            if (isRemoved(j)) continue;
            const uint32_t g = base + j;
            votes += vote_candidate(p, b.fshift[g], b.flen[g], b.forient[g] == 2, b.fid[g], aid, La,
                                    [&](int col) { return (uint32_t)base_index(cons[aBegin + col]); });
        }
        votes = block_reduce<int>(votes, redi, 2);
        if (tid == 0 && votes) atomicAdd(&b.counters[kCounterCandidateVotes], (unsigned long long)votes);
    }
    if (p.correctionType == CG_CORR_FOREST) {
        const bool hq = sHQ;
        const float avg = sAvg;
        for (int i = tid; i < La; i += bd) {
            const int c = aBegin + i;
            const uint32_t ab = get2bit(aenc, i);
            const char orig = "ACGT"[ab];
            char r = cons[c];
            if (!hq && r != orig) {
                const float wsum = __fadd_rn(__fadd_rn(__fadd_rn(colWA[c], colWC[c]), colWG[c]), colWT[c]);
                float wCons, nCons;
                switch (r) {
                    case 'A': wCons = colWA[c]; nCons = (float)cntA[c]; break;
                    case 'C': wCons = colWC[c]; nCons = (float)cntC[c]; break;
                    case 'G': wCons = colWG[c]; nCons = (float)cntG[c]; break;
                    default: wCons = colWT[c]; nCons = (float)cntT[c]; break;
                }
                const float wOrig = ab == 0 ? colWA[c] : ab == 1 ? colWC[c] : ab == 2 ? colWG[c] : colWT[c];
                const float cv = (float)cov[c];
                const float oc = (float)origCov[c];
                const float ec = p.estimatedCoverage;
                const float f[13] = {__fdiv_rn(oc, cv),           __fdiv_rn(wOrig, wsum), __fdiv_rn(wOrig, oc),
                                     __fdiv_rn(nCons, cv),        sup[c],                 __fdiv_rn(wCons, nCons),
                                     __fdiv_rn(wsum, cv),         __fdiv_rn(cv, ec),      __fdiv_rn(wsum, ec),
                                     avg,                         mins,                   __fdiv_rn((float)maxc, ec),
                                     __fdiv_rn((float)minc, ec)};
                if (!forest_decide(p, f)) r = orig;
            }
            out[i] = r;
        }
        return;
    }
    if (nActive == 0) return;
    const bool byCons = sByConsensus;
    for (int i = tid; i < La; i += bd) {
        const int c = aBegin + i;
        char r;
        if (byCons) {
            r = cons[c];
        } else {
            r = (sup[c] > 0.90f && origCov[c] <= 2) ? cons[c] : "ACGT"[get2bit(aenc, i)];
        }
        out[i] = r;
    }
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

// One warp per anchor (one warp per block) for reads up to 256 bp.
//
// Everything the path reads from an MSA -- the different-region search, the
// properties and both decisions -- lies in the anchor's columns, so only the
// part of each row that overlaps the anchor is accumulated, in anchor
// coordinates (column = anchor position).  Shared memory holds per anchor
// position and base the weight and the count side by side (one 8-byte
// access per addition); rows are added one at a time
// (anchor, then the kept candidates in list order) with the lanes over the
// row's positions, so every column receives its additions in the reference's
// order.  Lane l owns the columns c with c % 32 == l in every pass (rows,
// consensus, properties, decision), so consecutive rows need no warp sync.
// The 2-bit words and the metadata of 32 rows are staged in shared memory per
// chunk.
//
// `sm` is the warp's own slice of shared memory (msa_warp_slice_bytes), `qw`
// the block's quality weights.
// Walk of the chunk staging loop: word i0 + lane of a chunk's rows is word
// off of row r (r = (i0 + lane) / pitch); (r0, off0) at i0 = 0 and the step
// (dr, doff) per 32 words, so that the loop divides nothing.
struct StageWalk {
    int r0, off0, dr, doff;
};

template <bool QUAL>
__device__ __forceinline__ void msa_warp_anchor(const StoreArg& st, const Params& p, const BatchArg& b,
                                             const uint32_t* __restrict__ rawOff, int lp, int a, uint64_t first,
                                             unsigned char* sm, const float* qw, const StageWalk sw) {
    const int lane = (int)lane_id();
    uint2* wc = reinterpret_cast<uint2*>(sm);                    // [4][lp]: weight bits, count
    float* sup = reinterpret_cast<float*>(wc + 4 * lp);          // [lp]
    uint32_t* stage = reinterpret_cast<uint32_t*>(sup + lp);     // [32][pitch]
    int4* meta = reinterpret_cast<int4*>(stage + 32 * st.pitch);  // [32]: shift, len | orient << 16, weight, id
    const uint64_t aid = first + (uint64_t)a;
    const uint64_t oi = (first - out_first(b)) + (uint64_t)a;   // output row
    const uint32_t nf = b.nfinal[a];
    char* out = b.out + oi * b.outPitch;
    if (nf == 0) {
        if (lane == 0) b.flags[oi] = 0;
        return;
    }
    const uint32_t base = rawOff[a];
    const int La = st.len[aid];
    const int pitch = st.pitch;
    const uint32_t* aenc = st.enc + aid * (uint64_t)pitch;
    const uint8_t* aq = QUAL ? st.qual + aid * (uint64_t)st.lmax : nullptr;
    constexpr uint8_t kRm = 0x80;

    // Rows are added (sign +1: every row still in the MSA, after the anchor
    // row) or taken out again (sign -1: the rows just removed, marked kNew).
    // Returns the number of rows added or taken out.
    constexpr uint8_t kNew = 0x40;
    auto rowsPass = [&](auto addTag) -> int {
        constexpr bool add = decltype(addTag)::value;
        int selected = 0;
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
            const bool sel = jr < nf && (add ? !(mo & kRm) : (mo & kNew) != 0);
            const unsigned selRows = __ballot_sync(kFull, sel);
            if (!selRows) continue;
            selected += __popc(selRows);
            if (!add && sel) b.forient[base + jr] = (uint8_t)(mo & ~kNew);
            // the selected rows' 2-bit words, copied without a register round
            // trip and waited for once
            {
                const int total = rows * pitch;
                int r = sw.r0, off = sw.off0;
                for (int i0 = 0; i0 < total; i0 += 32) {  // warp-uniform trip count
                    const int rr = min(r, rows - 1);
                    const uint32_t rid = __shfl_sync(kFull, mid, rr);
                    if (i0 + lane < total && ((selRows >> rr) & 1u))
                        cp_async4(stage + i0 + lane, st.enc + (uint64_t)rid * pitch + off);
                    r += sw.dr;
                    off += sw.doff;
                    if (off >= pitch) {
                        off -= pitch;
                        r++;
                    }
                }
            }
            meta[lane] = make_int4(mshift, mlen | (int)((mo & 3u) << 16), __float_as_int(mw), (int)mid);
            cp_async_wait_all();
            __syncwarp();
            for (int r = 0; r < rows; r++) {
                if (!((selRows >> r) & 1u)) continue;
                const int4 md = meta[r];
                const bool rc = ((uint32_t)md.y >> 16) == 2;
                const int shift = md.x, len = md.y & 0xffff;
                const float weight = __int_as_float(md.z);
                const uint32_t* e = stage + r * pitch;
                const uint8_t* q = QUAL ? st.qual + (uint64_t)(uint32_t)md.w * st.lmax : nullptr;
                const int c0 = max(shift, 0), c1 = min(La, shift + len);  // overlap with the anchor
                int c = c0 + ((lane - c0) & 31);                           // this lane's first column
                // the row position moves by 32 per column step of the lane, so
                // its word moves by 2 and its bit offset stays
                int sp = rc ? len - 1 - (c - shift) : c - shift;
                const int dsp = rc ? -32 : 32, dwi = rc ? -2 : 2;
                const uint32_t sh = 30u - 2u * (uint32_t)(sp & 15), flip = rc ? 3u : 0u;
                // quality index: sp, or for a reverse complement row Lmax - 1 - (c - shift)
                const int qd = rc ? st.lmax - len : 0;
                // padding past the read's end is read as stored
                auto wtAt = [&](int s) -> float { return QUAL ? __fmul_rn(weight, qw[q[s + qd]]) : weight; };
                auto upd = [&](uint2& v, float wt) {
                    if (add) {
                        v.x = __float_as_uint(__fadd_rn(__uint_as_float(v.x), wt));
                        v.y++;
                    } else {
                        v.x = __float_as_uint(__fsub_rn(__uint_as_float(v.x), wt));
                        v.y--;
                    }
                };
                int wi = sp >> 4;
                // two of the lane's columns (c and c + 32) per iteration: both
                // words and both entries are read before either is written
                // (distinct columns, distinct entries)
                for (; c + 32 < c1; c += 64, wi += 2 * dwi, sp += 2 * dsp) {
                    const uint32_t b0 = ((e[wi] >> sh) & 3u) ^ flip;
                    const uint32_t b1 = ((e[wi + dwi] >> sh) & 3u) ^ flip;
                    const float w0 = wtAt(sp), w1 = wtAt(sp + dsp);
                    uint2* p0 = wc + b0 * lp + c;
                    uint2* p1 = wc + b1 * lp + (c + 32);
                    uint2 v0 = *p0, v1 = *p1;
                    upd(v0, w0);
                    upd(v1, w1);
                    *p0 = v0;
                    *p1 = v1;
                }
                if (c < c1) {
                    const uint32_t b0 = ((e[wi] >> sh) & 3u) ^ flip;
                    uint2* p0 = wc + b0 * lp + c;
                    uint2 v0 = *p0;
                    upd(v0, wtAt(sp));
                    *p0 = v0;
                }
            }
            __syncwarp();  // the next chunk overwrites the staged rows
        }
        return selected;
    };
    // The MSA of the rows still in it, built as the reference builds it: the
    // anchor row (weight 1 times the quality weight), then the rows in order.
    // Returns the number of rows it holds besides the anchor.
    auto build = [&]() -> int {
        for (int pos = lane; pos < La; pos += 32) {
            const uint32_t bb = get2bit(aenc, pos);
            const float wt = QUAL ? __fmul_rn(1.0f, qw[aq[pos]]) : 1.0f;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                wc[q * lp + pos] = (uint32_t)q == bb ? make_uint2(__float_as_uint(__fadd_rn(0.0f, wt)), 1u)
                                                     : make_uint2(__float_as_uint(0.0f), 0u);
            }
        }
        __syncwarp();
        return rowsPass(std::true_type{});
    };

    int builds = 0;
    bool exact = true, haveS = false;
    int nActive = build();
    const float tol = __fmul_rn(2.5f * 5.9604645e-8f, (float)(3 * nf + 4));  // 2 E_c / S_c with slack
    for (int iter = 0;; iter++) {
        builds++;
        if (iter == 5 || nActive == 0) break;
        if (!exact) {
            bool close = false;
            for (int c = lane; c < La; c += 32) {
                float t1 = 0.0f, t2 = 0.0f;  // the two largest weights
                const ColInfo ci = col_info(wc, lp, c);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float v = ci.w[q];
                    t2 = fmaxf(t2, fminf(t1, v));
                    t1 = fmaxf(t1, v);
                }
                close |= !(__fsub_rn(t1, t2) > __fmul_rn(tol, sup[c]));
            }
            if (__any_sync(kFull, close)) {
                build();
                exact = true;
            }
        }
        // findCandidatesOfDifferentRegion (src/msa.cpp:532-734), in anchor coordinates
        bool mism = false;
        int firstSig = 0x7fffffff;
        for (int c = lane; c < La; c += 32) {
            const ColInfo ci = col_info(wc, lp, c);
            mism |= ci.cons != "ACGT"[get2bit(aenc, c)];
            const int cidx = base_index(ci.cons);
            bool sig = false;
#pragma unroll
            for (int i = 0; i < 4; i++) sig |= (i != cidx && p.significantCount <= (int)ci.n[i]);
            if (sig && c < firstSig) firstSig = c;
        }
        if (!__any_sync(kFull, mism)) break;
        const int col = __reduce_min_sync(kFull, firstSig);
        if (col == 0x7fffffff) break;
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
        for (uint32_t j = lane; j < nf; j += 32) {
            if ((b.forient[base + j] & kRm) || !differs(j)) continue;
            any = true;
            veto |= b.fweight[base + j] >= 0.90f;
        }
        // a veto (or nothing to remove) leaves the MSA as it is; the
        // reference then rebuilds the same MSA and reaches the same decision
        if (__any_sync(kFull, veto) || !__any_sync(kFull, any)) break;
        int act = 0;
        for (uint32_t j = lane; j < nf; j += 32) {
            const uint8_t o = b.forient[base + j];
            if (!(o & kRm) && differs(j)) b.forient[base + j] = o | kRm | kNew;
            else act += !(o & kRm);
        }
        nActive = __reduce_add_sync(kFull, act);
        if (!haveS) {  // S_c (the first build, which wc still holds), kept in `sup` until the properties
            for (int c = lane; c < La; c += 32) sup[c] = col_info(wc, lp, c).colW;
            haveS = true;
        }
        __syncwarp();
        rowsPass(std::false_type{});
        exact = false;
    }
    if (!exact) build();
    // getMSAProperties (src/msa.cpp:304-376) and the decision
    float mins = 3.402823466e+38f;
    int minc = 0x7fffffff, maxc = -1;
    for (int c = lane; c < La; c += 32) {
        const ColInfo ci = col_info(wc, lp, c);
        const float s = __fdiv_rn(ci.consW, ci.colW);
        sup[c] = s;
        mins = fminf(mins, s);
        const int cv = ci.cov();
        minc = min(minc, cv);
        maxc = max(maxc, cv);
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
        for (; i + 4 <= La; i += 4) {
            const float4 v = s4[i >> 2];
            sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
        }
        for (; i < La; i++) sum = __fadd_rn(sum, sup[i]);
        avg = __fdiv_rn(sum, (float)La);
    }
    avg = __shfl_sync(kFull, avg, 0);
    const bool good = fgeq(avg, p.avgSupportThreshold) && fgeq(mins, p.minSupportThreshold) &&
                      fgeq((float)minc, p.minCoverageThreshold);
    bool hq = false;
    if (good) {
        int smallest = 100;
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
    for (int c = lane; c < La; c += 32) {
        const uint32_t ab = get2bit(aenc, c);
        const char orig = "ACGT"[ab];
        const ColInfo ci = col_info(wc, lp, c);
        const int origCov = (int)ci.nOf(ab);
        char r;
        if (forest) {
            // correctAnchorClf (include/corrector.hpp:1448-1472), features of
            // include/classification.hpp:748-797
            r = ci.cons;
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
        } else if (good) {
            r = ci.cons;
        } else {
            r = (sup[c] > 0.90f && origCov <= 2) ? ci.cons : orig;
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
        uint8_t* cons8 = reinterpret_cast<uint8_t*>(meta + 32);
        for (int c = lane; c < La; c += 32) cons8[nc + c] = (uint8_t)base_index(col_info(wc, lp, c).cons);
        for (int e0 = 0; e0 < 2 * nc; e0 += 32) {  // warp-uniform trip count
            const int e = e0 + lane;
            const int col = e < nc ? e - nc : La + (e - nc);
            float w4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
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
                for (int i0 = 0; i0 < rows * pitch; i0 += 32) {
                    const int idx = i0 + lane;
                    const int r = min(idx / pitch, rows - 1);
                    const uint32_t rid = __shfl_sync(kFull, mid, r);
                    if (idx < rows * pitch && ((selRows >> r) & 1u))
                        stage[idx] = st.enc[(uint64_t)rid * pitch + (idx - r * pitch)];
                }
                meta[lane] = make_int4(mshift, mlen | (int)((mo & 3u) << 16), __float_as_int(mw), (int)mid);
                __syncwarp();
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
        for (int u = lane; u <= nw; u += 32) {
            unsigned long long f = 0, r = 0;
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
    int nd = 0;
    for (int c = lane; c < La; c += 32) nd += col_info(wc, lp, c).cons != "ACGT"[get2bit(aenc, c)];
    nd = __reduce_add_sync(kFull, nd);
    const float ec = p.estimatedCoverage;
    const float invLa = __fdiv_rn(1.0f, (float)La);
    for (int c0 = 0; c0 < La; c0 += 32) {  // warp-uniform trip count
        const int c = c0 + lane;
        bool rec = false;
        ColInfo ci{};
        uint32_t ab = 0;
        if (c < La) {
            ab = get2bit(aenc, c);
            ci = col_info(wc, lp, c);
            rec = ci.cons != "ACGT"[ab];
        }
        const unsigned m = __ballot_sync(kFull, rec);
        if (!m) continue;
        unsigned slot = 0;
        if (lane == 0) slot = atomicAdd(b.colCount, (unsigned)__popc(m));
        slot = __shfl_sync(kFull, slot, 0) + (unsigned)__popc(m & ((1u << lane) - 1u));
        if (!rec || slot >= b.colCap) continue;
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

// Bytes of shared memory one warp of msa_warp_kernel works in (with candidate
// correction, the consensus codes of Lmax + 2 new_columns_to_correct columns
// follow the row metadata).
__host__ __device__ inline size_t msa_warp_slice_bytes(int lp, int pitch, const Params& p) {
    const size_t cols = (size_t)lp + 2 * (size_t)p.newColumns;
    const size_t cand = p.candidates ? (cols + 15) / 16 * 16 + 2 * ((cols + 31) / 32 + 1) * sizeof(uint64_t) : 0;
    return (size_t)lp * (9 * sizeof(float)) + (size_t)32 * pitch * sizeof(uint32_t) + 32 * sizeof(int4) + cand;
}

// `warps` warps per block, each on its own anchors.  Plain form: anchor
// blockIdx.x * warps + warp.  Persistent form (b.work set): warps take the
// next anchor from the counter b.work[0] until the batch is done.
__global__ void __launch_bounds__(256, 4) msa_warp_kernel(StoreArg st, Params p, BatchArg b,
                                                       const uint32_t* __restrict__ rawOff, int lp) {
    extern __shared__ __align__(16) unsigned char sm[];
    float* qw = reinterpret_cast<float*>(sm);  // [256] (quality scores only)
    const int warp = (int)(threadIdx.x >> 5), warps = (int)(blockDim.x >> 5);
    const size_t qbytes = p.useQuality ? 256 * sizeof(float) : 0;
    unsigned char* slice = sm + qbytes + (size_t)warp * msa_warp_slice_bytes(lp, st.pitch, p);
    if (p.useQuality) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) qw[i] = p.qweight[i];
        __syncthreads();
    }
    const uint64_t first = batch_first(b);
    const int lane = (int)lane_id(), pitch = st.pitch;
    const StageWalk sw{lane / pitch, lane % pitch, 32 / pitch, 32 % pitch};
    auto anchor = [&](int i) {
        const int a = b.order ? (int)b.order[i] : i;
        if (p.useQuality) msa_warp_anchor<true>(st, p, b, rawOff, lp, a, first, slice, qw, sw);
        else msa_warp_anchor<false>(st, p, b, rawOff, lp, a, first, slice, qw, sw);
    };
    if (!b.work) {
        const int i = blockIdx.x * warps + warp;
        if (i < b.count) anchor(i);
        return;
    }
    while (true) {
        int i = 0;
        if (lane == 0) i = (int)atomicAdd(&b.work[0], 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= b.count) return;
        anchor(i);
        __syncwarp();
    }
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

int msa_threads(int maxCols) {
    int t = kMsaThreadsMin;
    while (t * kMsaCols < maxCols) t += 32;
    return t;
}

size_t msa_smem_bytes(int maxCols, int bitsetWords, int storeWeights) {
    return sizeof(RowMeta) * kMsaChunkRows + sizeof(uint32_t) * bitsetWords + 256 * sizeof(float) +
           (size_t)maxCols * (7 * sizeof(int) + 1 + (storeWeights ? 4 * sizeof(float) : 0));
}

namespace {

size_t msa_warp_smem(StoreArg st, Params p, int warps) {
    const int lp = (st.lmax + 31) / 32 * 32;
    return (p.useQuality ? 256 * sizeof(float) : 0) + (size_t)warps * msa_warp_slice_bytes(lp, st.pitch, p);
}

cudaError_t msa_warp_prepare(size_t smem) {
    if (smem <= 40 * 1024) return cudaSuccess;  // leaves room for the kernel's static shared memory
    return cudaFuncSetAttribute(msa_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

}  // namespace

int msa_warp_occupancy(StoreArg st, Params p, int warps) {
    if (st.lmax > 256 || warps < 1 || warps > 8) return 0;
    const size_t smem = msa_warp_smem(st, p, warps);
    if (msa_warp_prepare(smem) != cudaSuccess) return 0;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, msa_warp_kernel, warps * 32, smem) != cudaSuccess)
        return 0;
    return blocks;
}

cudaError_t launch_msa_correct(StoreArg st, Params p, BatchArg b, int maxRows, cudaStream_t s, const Shape* shape) {
    const int maxCols = 3 * st.lmax + 4;
    if (st.lmax <= 256) {
        const int lp = (st.lmax + 31) / 32 * 32;
        const bool persistent = shape && b.work;
        const int warps = persistent ? shape->msaWarps : 1;
        const size_t smem = msa_warp_smem(st, p, warps);
        cudaError_t e = msa_warp_prepare(smem);
        if (e != cudaSuccess) return e;
        const unsigned blocks = persistent ? (unsigned)shape->msaBlocks : (unsigned)b.count;
        if (blocks == 0) return cudaSuccess;
        msa_warp_kernel<<<blocks, warps * 32, smem, s>>>(st, p, b, b.rawCount, lp);
        return cudaGetLastError();
    }
    const int bitsetWords = (maxRows + 31) / 32 + 1;
    const int storeWeights = p.correctionType == CG_CORR_FOREST;
    const size_t smem = msa_smem_bytes(maxCols, bitsetWords, storeWeights);
    if (smem > 40 * 1024) {  // leaves room for the kernel's static shared memory
        cudaError_t e = cudaFuncSetAttribute(msa_correct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
    }
    if (b.count == 0) return cudaSuccess;
    msa_correct_kernel<<<b.count, msa_threads(maxCols), smem, s>>>(st, p, b, b.rawCount, maxCols, bitsetWords,
                                                                    storeWeights);
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
