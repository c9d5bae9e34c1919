// Internal declarations shared by the CUDA kernel files and the C ABI layer.
//
// Device layout (one context, one GPU):
//   read store      enc   u32 [N][pitch]      2-bit bases, 16 per word, first base in the MSBs
//                   len   u16 [N]
//                   hilo  u32 [N][2][wp]      hi and lo bit planes (32 bases per word), zero past the
//                                             read; wp = align_plane_words
//                   qual  u8  [N][Lmax]       Phred+33 (only with quality scores)
//                   ambig u8  [N]             read had a non-ACGT base
//   signatures      sig   u64 [maps][N]       minhash key of every read for every map
//   hash tables     per map: open-addressing slots {key, offset, count} and the
//                   read ids of every kept key, ascending
//   per batch       candidate lists, alignment results, filtered lists and the
//                   corrected anchors, all addressed by per-anchor offsets
#ifndef CARE_INTERNAL_H
#define CARE_INTERNAL_H

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "care_gpu.h"

namespace cg {

constexpr uint64_t kEmptyKey = ~0ull;
constexpr int kSegmentReads = 65536;  // N-replacement counter restarts per parser batch
constexpr int kMaxMaps = CG_MAX_HASHMAPS;
constexpr int kMaxBucket = 65535;     // BucketSize is uint16 in the reference
constexpr int kLearnedFeatures = 32;  // features of one MSA column for the learned decision

// The alignment kernel's instances take reads of up to 32 W bases: W of a
// store whose longest read has lmax bases (the read lengths in use: 75, 100 to
// 125, 150, 250 and 300 bp sequencing, and longer merged reads), the words of a
// bit plane it loads (W and at least one zero word, an even number so that a
// read's planes are 16-byte pieces), and the candidates per unit of its work
// (the columns of its products).
constexpr int align_words(int lmax) {
    const int need = (lmax + 31) / 32;
    return need <= 3 ? 3 : need <= 4 ? 4 : need <= 5 ? 5 : need <= 8 ? 8 : need <= 10 ? 10 : need <= 16 ? 16
           : need <= 20 ? 20 : 32;
}
constexpr int align_plane_words(int w) { return (w + 2) / 2 * 2; }
constexpr int kAlignUnit = 64;
constexpr uint32_t kWaitPolls = 1u << 20;  // polls of a wait for tensor-core products before it is declared failed

struct Slot {
    unsigned long long key;
    uint32_t offset;
    uint32_t count;
};
static_assert(sizeof(Slot) == 16, "slot layout");

// All maps' lookup tables, passed by value to the query kernels.
struct TablesArg {
    const Slot* slots[kMaxMaps];
    const uint32_t* values[kMaxMaps];
    uint32_t mask[kMaxMaps];
    int nmaps;
    int maxValuesPerKey;
};

// Read store view.
struct StoreArg {
    const uint32_t* enc;
    const uint16_t* len;
    const uint32_t* hilo;
    const uint8_t* qual;
    const uint8_t* ambig;
    int pitch;      // u32 words per read in enc
    int wp;         // u32 words per plane in hilo
    int lmax;
    uint64_t n;
};

// Float constants of the correction decision, computed once on the host in
// the reference's operand order (ISO C++, no contraction).
struct Params {
    int k;
    int nmaps;
    int minOverlap;
    float maxErrorRate;        // maxErrorRate (alignment)
    float minOverlapRatio;
    float orientMaxErrorRate;  // estimatedErrorrate * 4.0f
    float mmBase;              // estimatedErrorrate * 1.0f
    float mm2, mm3, mm4;       // 2/3/4 * mmBase
    float goodAlignmentsCountThreshold;  // estimatedCoverage * m_coverage
    float pairedThreshold;
    float avgSupportThreshold;  // 1 - 1*err
    float minSupportThreshold;  // 1 - 3*err
    float minCoverageThreshold; // m_coverage / 6 * cov
    int errPercent;             // ceil(err * 100)
    float hqPercentLimit;       // errPercent * 0.5f
    float hqAvg[101];           // 1 - 1*percent/100 for percent 0..100
    float hqMin[101];           // 1 - 3*percent/100
    int significantCount;       // int(int(cov) * 0.3f)
    uint32_t alignPolls;        // polls of an alignment block's wait for its products
    float alignLift;            // added to the start values of its accumulators (set by launch_align)
    int useQuality;
    int excludeAmbiguous;
    int paired;
    int correctionType;         // CG_CORR_*
    float estimatedCoverage;
    // forest decision (correctionType == CG_CORR_FOREST)
    const struct ForestNode* forestNodes;
    const uint32_t* treeOffsets;  // first node of each tree
    int numTrees;
    float forestThreshold;
    float qweight[256];
    // Candidate correction (correct_candidates).  Per read: votes = {number of
    // candidate corrections made by anchors with a smaller id, by anchors with a
    // larger id}; candAnd / candOr = bitwise AND / OR of every sequence voted
    // for the read (its candidate corrections and its own low-quality anchor
    // correction), 2 bits per base, 32 bases per word, first base in the most
    // significant bits, zero past the read's end.  All of them are equal
    // exactly when AND == OR over the read's words.
    int candidates;
    int newColumns;               // new_columns_to_correct
    int candPitch;                // words per read = ceil(Lmax / 32)
    uint2* candVotes;             // [N]
    unsigned long long* candAnd;  // [N][candPitch]
    unsigned long long* candOr;   // [N][candPitch]
};

// One forest node (reference: include/forest.hpp:21-30): go left when
// feature[att] <= split; flag bit 1 = lhs is a leaf, bit 0 = rhs is a leaf;
// a leaf side holds the float probability's bits, an inner side the index of
// the child within the tree.
struct ForestNode {
    double split;
    uint32_t lhs, rhs;
    uint8_t att, flag;
    uint8_t pad[6];
};
static_assert(sizeof(ForestNode) == 24, "forest node layout");

// ---------------------------------------------------------------- launches
// Every launcher enqueues on `s` and returns the launch status.

// exclusive scans, in place; `tmp` needs scan_tmp_bytes(n) bytes
size_t scan_tmp_bytes(size_t n);
cudaError_t scan_exclusive_u32(uint32_t* data, size_t n, void* tmp, cudaStream_t s);
cudaError_t scan_exclusive_u64(unsigned long long* data, size_t n, void* tmp, cudaStream_t s);
// kernels one scan of n elements launches
uint64_t scan_launches(uint64_t n);

// read store
// offs[i] -= base for i < count
cudaError_t launch_rebase_offsets(uint64_t* offs, uint64_t count, uint64_t base, cudaStream_t s);
cudaError_t launch_count_invalid(const char* chars, const uint64_t* offs, uint64_t n, uint32_t* invalid,
                                 cudaStream_t s);
cudaError_t launch_encode(const char* chars, const uint64_t* offs, const char* quals, uint64_t n,
                          uint64_t firstId, const uint32_t* invalidScan, const uint64_t* segStart,
                          uint32_t* enc, uint16_t* len, uint8_t* qual, uint8_t* ambig, int pitch, int lmax,
                          cudaStream_t s);
cudaError_t launch_hilo(StoreArg st, uint32_t* hilo, cudaStream_t s);
cudaError_t launch_signatures(StoreArg st, int k, int nmaps, unsigned long long* sig, cudaStream_t s);
// out[0] = shortest, out[1] = longest read of the store (out preset to {~0, 0})
cudaError_t launch_len_range(const uint16_t* len, uint64_t n, unsigned int* out, cudaStream_t s);
// qualityScoreBits 1 or 2: bins the stored scores of reads [0, n) in place
// (rows of lmax bytes) and fills each row past its read's end with the first bin
cudaError_t launch_quality_bins(uint8_t* qual, const uint16_t* len, uint64_t n, int lmax, int bits, cudaStream_t s);

// hash tables
// The maps of a build wave, one after the other: each map's n (key, read id)
// pairs sorted by key (read ids ascending within a key) into keys/vals
// [maps][n], from the first `bits` bits of keysIn's keys (values 0 .. n - 1 in
// every map); keysAlt/valsAlt hold as many pairs of scratch, temp
// radix_sort_temp_bytes(n, maps) bytes; n * maps < 2^32
size_t radix_sort_temp_bytes(uint64_t n, int maps);
cudaError_t radix_sort_pairs(const unsigned long long* keysIn, uint64_t n, int maps, int bits, unsigned long long* keys,
                             uint32_t* vals, unsigned long long* keysAlt, uint32_t* valsAlt, void* temp,
                             cudaStream_t s);
// Runs of equal keys in sorted pairs (total = n * maps): runOf[0..total]
// (scanned in place by the caller into run indices, runOf[total] = number of
// runs R), start[0..R], packed[0..R] (scanned by the caller into value offsets
// of the wave), then per map {kept keys << 32 | values, offset of its first
// value} into totals, the kept runs' ids into the wave's values and their keys
// into the maps' tables (and, with rawAll, each kept id's bucket size added to
// rawAll[id]).
struct WaveTables {
    Slot* slots[kMaxMaps];
    uint32_t mask[kMaxMaps];
    uint32_t firstValue[kMaxMaps];  // a map's first value in the wave's values
};
cudaError_t launch_run_heads(const unsigned long long* keys, uint64_t n, int maps, uint32_t* runOf, cudaStream_t s);
cudaError_t launch_run_starts(const unsigned long long* keys, uint64_t n, int maps, const uint32_t* runOf,
                              uint32_t* start, cudaStream_t s);
cudaError_t launch_run_pack(const unsigned long long* keys, const uint32_t* start, uint32_t runs, int maxValues,
                            unsigned long long* packed, cudaStream_t s);
cudaError_t launch_run_totals(const uint32_t* runOf, uint64_t n, int maps, const unsigned long long* packedScan,
                              ulonglong2* totals, cudaStream_t s);
cudaError_t launch_run_fill(const unsigned long long* keys, const uint32_t* ids, uint64_t n, int maps,
                            const uint32_t* runOf, const uint32_t* start, uint32_t runs,
                            const unsigned long long* packedScan, int maxValues, uint32_t* values, WaveTables tables,
                            cudaStream_t s, uint32_t* rawAll = nullptr);

// correction batch
struct BatchArg {
    uint64_t first;         // first anchor id
    int count;              // anchors in batch
    const unsigned long long* sig;  // [nmaps][N]
    uint2* qrange;          // [count][nmaps] (offset, count) per map
    uint32_t* rawCount;     // [count+2]: raw counts, exclusive-scanned in place into offsets
                            // ([count] = total after the scan); [count+1] = batch maximum
    uint32_t* cand;         // [totalRaw] unique candidate ids
    uint32_t* ncand;        // [count]
    uint8_t* paired;        // [totalRaw] pair flags (PE)
    uint2* aln;             // [totalRaw] packed alignment results (anchors of several units)
    uint32_t* fid;          // [totalRaw] filtered candidates: id
    int16_t* fshift;        // [totalRaw]
    uint8_t* forient;       // [totalRaw] 1 fwd, 2 rc
    float* fweight;         // [totalRaw]
    uint16_t* flen;         // [totalRaw] candidate length
    uint32_t* nfinal;       // [count] kept candidates; 0 until the anchor's filter has run
    // The alignment's work: units {anchor, part} of up to kAlignUnit candidates
    // (part k holds the anchor's candidates k kAlignUnit ..), appended by the
    // candidate kernel at *unitCount and taken at *unitCursor (both zero at the
    // start of a batch); null where only the candidates are wanted.
    uint2* units;
    unsigned int* unitCount;
    unsigned int* unitCursor;
    uint32_t* unitsDone;    // [count] finished units of an anchor of several (zero at the start of a batch)
    uint8_t* flags;         // [count] CG_RESULT_*
    char* out;              // [count][outPitch]
    int outPitch;
    unsigned long long* counters;  // device counters, see kCounter*
    // Output rows: anchor first + a goes to row (first - outFirst) + a of out
    // and flags.  The plain form sets outFirst = first.
    unsigned long long outFirst;
    // Batched form (graph replays), null in the plain form:
    //   cursor[0] = the batch's first anchor id, cursor[1] = outFirst, both
    //     read on the device so that one captured graph serves every batch
    //   rangeOff = exclusive scan of the raw id counts of the anchors
    //     outFirst, outFirst+1, ...; the candidate kernel takes the batch's raw
    //     offsets from it instead of a count pass and a scan per batch
    //   work[0] = the persistent MSA kernel's work-stealing counter (zero at the
    //     start of a batch)
    const unsigned long long* cursor;
    const unsigned long long* rangeOff;
    unsigned int* work;
    // Learned decision (correctionType CG_CORR_LEARNED): the MSA kernel records
    // every column of a non-HQ anchor whose consensus differs from the anchor's
    // base: 32 BF16 features (colFeat) and {output row, position | consensus
    // base << 16} (colMeta), at index atomicAdd(colCount); indexes past colCap
    // are not stored (those columns keep the fallback decision).
    __nv_bfloat16* colFeat;
    uint2* colMeta;
    unsigned int* colCount;
    unsigned int colCap;
    // MSA order: anchors by decreasing number of kept rows (null: batch order);
    // the heavy MSAs start first, so that none of them is left for the end
    const uint32_t* order;
};
enum {
    kCounterRaw = 0,
    kCounterUnique,
    kCounterAligned,
    kCounterMsaCands,
    kCounterMsaBuilds,
    kCounterCorrected,
    kCounterHQ,
    kCounterTimeouts,
    kCounterColumns,         // learned decision: columns recorded for the classifier
    kCounterColumnOverflow,  // columns beyond the buffer (decided by the fallback rule)
    kCounterLearnedTaken,    // columns the classifier corrected
    kCounterCandidateVotes,  // candidate corrections made by HQ anchors
    kCounterAlignTimeouts,   // alignment blocks that gave up waiting for their tensor-core products
    kNumCounters
};

cudaError_t launch_query_count(StoreArg st, TablesArg tb, Params p, BatchArg b, cudaStream_t s);
// with b.rangeOff set the kernel looks the buckets up itself and writes the
// batch's raw offsets into b.rawCount (no query_count pass, no scan)
// bigScratch (optional, count + 1 words): anchors with more than 1024 raw ids
// run in a second, large-table pass instead of sizing every block for them
cudaError_t launch_gather_unique(StoreArg st, TablesArg tb, Params p, BatchArg b, int maxRawPerAnchor,
                                 cudaStream_t s, uint32_t* bigScratch = nullptr);
cudaError_t launch_pair_flags(BatchArg b, cudaStream_t s);
// raw id count of every read as an anchor, raw[N]: raw holds every read's
// kept bucket sizes summed by launch_run_fill over all maps; reads that
// cannot be anchors get zero
cudaError_t launch_raw_count(StoreArg st, Params p, uint32_t* raw, cudaStream_t s);
// off[num+1] = exclusive scan of raw[0..num); maxima[0] = the largest raw
// total of a batch of `batch` anchors, maxima[1] = the largest raw count of
// one anchor; tmp needs scan_tmp_bytes(num + 1) bytes
cudaError_t launch_range_offsets(const uint32_t* raw, uint64_t num, uint64_t batch, unsigned long long* off,
                                 void* tmp, unsigned long long* maxima, cudaStream_t s);

// Launch shapes of the batched form's persistent kernels (b.work set).
struct Shape {
    int alignBlocks;  // persistent alignment blocks of 128 threads
    int msaWarps;     // warps (anchors in flight) per MSA block
    int msaBlocks;    // persistent MSA blocks
};

// Aligns every unit's candidates (b.units, *b.unitCount of them) and filters
// the anchors (b.nfinal and b.unitsDone zero before it; b.nfinal stays zero
// where a block gave up waiting for its products); varies: reads of several lengths.
// Persistent blocks: any number of them does.
cudaError_t launch_align(StoreArg st, Params p, BatchArg b, bool varies, unsigned blocks, cudaStream_t s);
// resident 128-thread blocks of it per SM
int align_occupancy(StoreArg st);
// MSA, refinement and decision of the batch's anchors, one warp each.  With
// b.work: persistent blocks of shape->msaWarps warps, or as many as a block's
// shared memory holds (long reads); otherwise a block of one warp per anchor.
cudaError_t launch_msa_correct(StoreArg st, Params p, BatchArg b, cudaStream_t s, const Shape* shape = nullptr);
// resident MSA blocks of `warps` warps per SM
int msa_warp_occupancy(StoreArg st, Params p, int warps);
// order[count] = the batch's anchors by decreasing b.nfinal (log2 buckets);
// scratch = 32 words, cleared by the launcher
cudaError_t launch_msa_order(BatchArg b, unsigned int* scratch, uint32_t* order, cudaStream_t s);
// candidate correction: the batch's low-quality anchor corrections join their
// reads' votes (after the MSA and any classifier pass)
cudaError_t launch_anchor_vote(StoreArg st, Params p, BatchArg b, cudaStream_t s);
// the combine step for reads [first, first + n): flags[i] of read first + i is
// rewritten (CG_RESULT_CANDIDATES / _REJECTED / _CANDIDATE_RECORD), *records
// (zeroed by the caller) gains the number of saved candidate records
cudaError_t launch_combine(StoreArg st, Params p, uint64_t first, uint64_t n, uint8_t* flags,
                           unsigned long long* records, cudaStream_t s);
// cursor[0] += stride, work[0..2] = 0 (the last node of a batch)
cudaError_t launch_batch_advance(unsigned long long* cursor, unsigned int* work, unsigned long long stride,
                                 cudaStream_t s);

}  // namespace cg

#endif
