// Learned correction classifier: a 32 -> 64 -> 64 -> 1 MLP over per-column
// MSA features, BF16 weights and activations, FP32 accumulation, sigmoid
// output.  It stands where the reference's forest/logistic-regression
// classifier stands in its correction path (include/classification.hpp:51-157,
// include/forest.hpp:217-226, used by correctAnchorClf in
// include/corrector.hpp:1448-1472); the network, its features and its training
// are this project's own.
//
// Every matrix product runs on the tcgen05 tensor cores (kind::f16: BF16
// operands in shared memory, FP32 accumulators in tensor memory).  Inference
// scores 128 columns per tile; training takes a 128-row tile of a minibatch
// per block through the forward pass, the hidden gradient and both weight
// gradients (one product over transposed tiles).  Training is deterministic:
// every block writes its partial gradients to its own slot and one kernel sums
// the slots in a fixed order before the Adam update.

#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "care_device.cuh"
#include "care_internal.h"
#include "care_learned.h"
#include "care_tc.cuh"

namespace cg {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// ---------------------------------------------------------------- inference (tcgen05)
//
// 128 columns (rows of the product, the MMA's M) per tile.  Operands sit in
// shared memory in the canonical K-major layout without swizzle (8-row x
// 16-byte core matrices; the K/8 core matrices of an 8-row group contiguous);
// one thread issues tcgen05.mma (kind::f16, BF16 A and B, FP32 accumulators
// in tensor memory), tcgen05.commit arrives on an mbarrier, and every thread
// reads its row of the accumulators back with tcgen05.ld (thread = TMEM lane).
// Layer 1 accumulates in TMEM columns 0-63, layer 2 in 64-127; the epilogue of
// layer 1 (bias, ReLU, BF16) writes layer 2's A operand back to shared memory.

constexpr int kTcRows = 128;
constexpr uint32_t kTmemCols = 128;

// Polls of the per-tile MMA waits (the waits whose failure ends a block);
// set from the host by set_classifier_wait_limit.  The wait that drains a
// failed block's MMAs before its tensor memory is released always uses
// kWaitPolls.
__device__ uint32_t g_tileWaitSpins = kWaitPolls;

// 32 consecutive FP32 accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                 : "=r"(r[0]),"=r"(r[1]),"=r"(r[2]),"=r"(r[3]),"=r"(r[4]),"=r"(r[5]),"=r"(r[6]),"=r"(r[7]),"=r"(r[8]),"=r"(r[9]),"=r"(r[10]),"=r"(r[11]),"=r"(r[12]),"=r"(r[13]),"=r"(r[14]),"=r"(r[15]),"=r"(r[16]),"=r"(r[17]),"=r"(r[18]),"=r"(r[19]),"=r"(r[20]),"=r"(r[21]),"=r"(r[22]),"=r"(r[23]),"=r"(r[24]),"=r"(r[25]),"=r"(r[26]),"=r"(r[27]),"=r"(r[28]),"=r"(r[29]),"=r"(r[30]),"=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// Inference over a column buffer, persistent over 128-column tiles.  Rows are
// BF16 (the column records) or FP32, rounded to BF16 as they are read.  With
// `logits` set the outputs are written there; otherwise every column whose
// logit reaches `minLogit` (the logit of the confidence threshold) gets the
// consensus base in its output row, and the others keep the fallback decision
// the MSA kernel already wrote.  A wait that does not end counts in
// counters[kCounterTimeouts] and ends the block (after a second bounded wait
// for its MMAs and the release of its tensor memory).  Measured: 1M FP32 rows 82 us
// (128 MB, 19 us at the memory's rate), bound by the chain of products and epilogues
// of a tile; with a conversion pass to BF16 in front a call took 1.02 ms, without
// it 0.95, nearly all of that the rows' copy from the host.
template <class Feature>
__global__ void __launch_bounds__(kTcRows) mlp_infer_kernel(const unsigned char* __restrict__ model,
                                                            const Feature* __restrict__ feat,
                                                            const uint2* __restrict__ meta,
                                                            const unsigned int* __restrict__ countPtr,
                                                            unsigned int count, unsigned int cap, float minLogit,
                                                            char* out, int outPitch, float* logits,
                                                            unsigned long long* counters) {
    __shared__ __align__(1024) unsigned char a1[kTcRows * kMlpFeatures * 2];
    __shared__ __align__(1024) unsigned char a2[kTcRows * kMlpHidden * 2];
    __shared__ __align__(1024) unsigned char b1[kMlpHidden * kMlpFeatures * 2];
    __shared__ __align__(1024) unsigned char b2[kMlpHidden * kMlpHidden * 2];
    __shared__ float bias1[kMlpHidden], bias2[kMlpHidden], wout[kMlpHidden];
    __shared__ float bias3;
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ uint32_t tmemBase;
    const int tid = (int)threadIdx.x, warp = tid >> 5;
    // weights into the canonical layout (B operands: N x K, K-major = the stored rows)
    const __nv_bfloat16* w1 = reinterpret_cast<const __nv_bfloat16*>(model + kMlpOffW1);
    const __nv_bfloat16* w2 = reinterpret_cast<const __nv_bfloat16*>(model + kMlpOffW2);
    const __nv_bfloat16* w3 = reinterpret_cast<const __nv_bfloat16*>(model + kMlpOffW3);
    for (int i = tid; i < kMlpHidden * kMlpFeatures; i += kTcRows)
        *reinterpret_cast<__nv_bfloat16*>(b1 + core_offset(i / kMlpFeatures, i % kMlpFeatures, kMlpFeatures)) = w1[i];
    for (int i = tid; i < kMlpHidden * kMlpHidden; i += kTcRows)
        *reinterpret_cast<__nv_bfloat16*>(b2 + core_offset(i / kMlpHidden, i % kMlpHidden, kMlpHidden)) = w2[i];
    const float* bsrc = reinterpret_cast<const float*>(model + kMlpOffB1);
    if (tid < kMlpHidden) {
        bias1[tid] = bsrc[tid];
        bias2[tid] = bsrc[kMlpHidden + tid];
        wout[tid] = __bfloat162float(w3[tid]);
    }
    if (tid == 0) {
        bias3 = bsrc[2 * kMlpHidden];
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemBase)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmemBase;
    const uint32_t lane0 = tbase + ((uint32_t)(warp * 32) << 16);  // this warp's 32 TMEM lanes
    const uint32_t mb = smem_u32(&mbar);
    constexpr uint32_t idesc = instr_desc(kTcRows, kMlpHidden);
    unsigned int n = countPtr ? *countPtr : count;
    if (countPtr && blockIdx.x == 0 && tid == 0 && counters) {
        atomicAdd(&counters[kCounterColumns], (unsigned long long)n);
        if (n > cap) atomicAdd(&counters[kCounterColumnOverflow], (unsigned long long)(n - cap));
    }
    if (n > cap) n = cap;
    uint32_t phase = 0;
    unsigned int taken = 0;
    bool failed = false;
    const uint32_t tilePolls = g_tileWaitSpins;
    for (unsigned int t0 = blockIdx.x * kTcRows; t0 < n; t0 += gridDim.x * kTcRows) {
        const unsigned int row = t0 + (unsigned int)tid;
        uint4 f[4];
#pragma unroll
        for (int j = 0; j < 4; j++) f[j] = make_uint4(0, 0, 0, 0);
        if (row < n) {
            if constexpr (sizeof(Feature) == 2) {
                const uint4* src = reinterpret_cast<const uint4*>(feat + (uint64_t)row * kMlpFeatures);
#pragma unroll
                for (int j = 0; j < 4; j++) f[j] = src[j];
            } else {
                const float4* src = reinterpret_cast<const float4*>(feat + (uint64_t)row * kMlpFeatures);
                float4 x[8];
#pragma unroll
                for (int j = 0; j < 8; j++) x[j] = src[j];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    f[j] = make_uint4(pack_bf16(x[2 * j].x, x[2 * j].y), pack_bf16(x[2 * j].z, x[2 * j].w),
                                      pack_bf16(x[2 * j + 1].x, x[2 * j + 1].y),
                                      pack_bf16(x[2 * j + 1].z, x[2 * j + 1].w));
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) *reinterpret_cast<uint4*>(a1 + core_offset(tid, 8 * j, kMlpFeatures)) = f[j];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // visible to the tensor core
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (tid == 0) {
#pragma unroll
            for (int k = 0; k < kMlpFeatures / 16; k++)
                tc_mma(tbase, smem_desc(smem_u32(a1) + 256u * k, 128, 512), smem_desc(smem_u32(b1) + 256u * k, 128, 512),
                       idesc, k > 0);
            tc_commit(mb);
        }
        bool ok = mbar_wait(mb, phase, tilePolls);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        tc_fence_after();
        // layer 1 epilogue: this thread's row -> bias, ReLU, BF16 -> layer 2's A operand
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[32];
            tc_ld32(lane0 + 32u * half, v);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t w[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int c = 32 * half + 8 * j + 2 * q;
                    w[q] = pack_bf16(fmaxf(__fadd_rn(v[8 * j + 2 * q], bias1[c]), 0.0f),
                                     fmaxf(__fadd_rn(v[8 * j + 2 * q + 1], bias1[c + 1]), 0.0f));
                }
                *reinterpret_cast<uint4*>(a2 + core_offset(tid, 32 * half + 8 * j, kMlpHidden)) =
                    make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (tid == 0) {
#pragma unroll
            for (int k = 0; k < kMlpHidden / 16; k++)
                tc_mma(tbase + kMlpHidden, smem_desc(smem_u32(a2) + 256u * k, 128, 1024),
                       smem_desc(smem_u32(b2) + 256u * k, 128, 1024), idesc, k > 0);
            tc_commit(mb);
        }
        ok = mbar_wait(mb, phase, tilePolls);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        tc_fence_after();
        float z = 0.0f;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[32];
            tc_ld32(lane0 + (uint32_t)kMlpHidden + 32u * half, v);
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const int c = 32 * half + i;
                const float h = __bfloat162float(__float2bfloat16_rn(fmaxf(__fadd_rn(v[i], bias2[c]), 0.0f)));
                z = __fadd_rn(z, __fmul_rn(h, wout[c]));
            }
        }
        z = __fadd_rn(z, bias3);
        if (row < n) {
            if (logits) {
                logits[row] = z;
            } else if (z >= minLogit) {
                const uint2 m = meta[row];
                out[(uint64_t)m.x * outPitch + (m.y & 0xffffu)] = (char)((m.y >> 16) & 0xffu);
                taken++;
            }
        }
        tc_fence_before();  // the next tile's MMAs overwrite the accumulators read here
    }
    if (failed) {
        if (tid == 0 && counters) atomicAdd(&counters[kCounterTimeouts], 1ull);
        mbar_wait(mb, phase ^ 1u, kWaitPolls);  // the MMAs in flight, bounded again at the full limit
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(kTmemCols) : "memory");
    if (counters && !logits) {
        taken = __reduce_add_sync(kFull, taken);
        if ((tid & 31) == 0 && taken) atomicAdd(&counters[kCounterLearnedTaken], (unsigned long long)taken);
    }
}

// ---------------------------------------------------------------- training (tcgen05)
//
// One block of 128 threads per 128-row tile of the minibatch (thread = row =
// TMEM lane): the forward pass and every gradient of the mean loss over the
// tile, as partial sums in part[tile][...] (parameter order of the model: w1,
// w2, w3, b1, b2, b3, loss) that mlp_reduce_kernel adds in tile order.  The
// matrix products run on tcgen05.mma (kind::f16, BF16 operands in shared
// memory in the canonical K-major layout, FP32 accumulators in tensor memory):
//   forward   D1 = X W1^T, D2 = H1 W2^T                (M = 128 rows)
//   backward  dH1 = dH2 W2                              (M = 128 rows)
//             [dW2; dW1] = [dH2^T; dH1^T] [H1^T | X^T]  (one M = 128, N = 96,
//             K = 128 product: rows 0-63 x columns 0-63 are dW2, rows 64-127
//             x columns 64-95 are dW1; the cross terms are not read)
// BF16 rounding at the same points as the oracle (oracle/mlp.py): the
// features, h1 and h2 after ReLU, dH2 before the products, dH1 before dW1;
// FP32 elsewhere.  Bound by latency: a minibatch is 32 tiles, one block each, and a
// tile is a chain of products and epilogues.  A training step (this kernel and the
// next) of 4,096 rows takes 17 us; 36 us with five shuffles per column sum, scalar
// weight loads and a kernel of its own for the step count.
// dW3 and the bias gradients are column sums over the tile's
// rows (warp shuffles, then the four warps in order).

constexpr int kTrainRows = 128;
constexpr uint32_t kTrainTmemCols = 256;  // D1/D2 (0-127, later [dW2 dW1] at 0-95), dH1 (128-191)
constexpr int kTrainOutCols = kMlpHidden + kMlpFeatures;  // N of the weight-gradient product
// The transposed operands, written two bytes at a time with a row of the
// minibatch per thread: 144 bytes between the core matrices along K keep a warp's
// stores (8 rows per core matrix) out of each other's banks.
constexpr uint32_t kTrainLbo = 144, kTrainSbo = kTrainLbo * (kTrainRows / 8);
__device__ __forceinline__ uint32_t train_offset(int row, int k) {
    return (uint32_t)(row >> 3) * kTrainSbo + (uint32_t)(k >> 3) * kTrainLbo + ((row & 7) << 4) + ((k & 7) << 1);
}

// Sums over the warp of 32 values per lane, column j's in lane j: every step
// halves the columns a lane carries, so 31 shuffles do for 32 sums.  Each sum is
// the butterfly's (lanes 16 apart first), in its order of additions.
__device__ __forceinline__ float warp_sums(float (&v)[32], int lane) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int j = 0; j < m; j++) {
            const float keep = up ? v[j + m] : v[j], send = up ? v[j] : v[j + m];
            v[j] = __fadd_rn(keep, __shfl_xor_sync(kFull, send, m));
        }
    }
    return v[0];
}

// shared memory of one block (every operand tile 1024-byte aligned)
struct TrainTc {
    unsigned char xa[kTrainRows * kMlpFeatures * 2];        // A of D1: X [128][32]
    unsigned char w1[kMlpHidden * kMlpFeatures * 2];        // B of D1: W1 [64][32]
    unsigned char h1a[kTrainRows * kMlpHidden * 2];         // A of D2: H1 [128][64]
    unsigned char w2[kMlpHidden * kMlpHidden * 2];          // B of D2: W2 [64 out][64 in]
    unsigned char d2a[kTrainRows * kMlpHidden * 2];         // A of dH1: dH2 [128][64]
    unsigned char w2t[kMlpHidden * kMlpHidden * 2];         // B of dH1: W2^T [64 in][64 out]
    unsigned char gA[kTrainRows / 8 * kTrainSbo];           // A of [dW2; dW1]: [dH2^T; dH1^T] [128][128 rows]
    unsigned char gB[kTrainOutCols / 8 * kTrainSbo];        // B of [dW2; dW1]: [H1^T | X^T] [96][128 rows]
    float b1[kMlpHidden], b2[kMlpHidden], w3[kMlpHidden];
    float red[4][3 * kMlpHidden + 2];                       // per-warp column sums: dW3, db2, db1, db3, loss
    float b3;
    unsigned long long mbar;
    uint32_t tmemBase;
};

__global__ void __launch_bounds__(kTrainRows, 1) mlp_grad_kernel(const unsigned char* __restrict__ model,
                                                                 const __nv_bfloat16* __restrict__ feat,
                                                                 const float* __restrict__ label,
                                                                 const uint32_t* __restrict__ perm,
                                                                 const unsigned long long* stepPtr,
                                                                 unsigned int stepsPerEpoch, unsigned int rows,
                                                                 float invTotal, float* __restrict__ part,
                                                                 unsigned long long* failed) {
    extern __shared__ __align__(1024) unsigned char smraw[];
    TrainTc& s = *reinterpret_cast<TrainTc*>(smraw);
    const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const __nv_bfloat16* w1g = reinterpret_cast<const __nv_bfloat16*>(model + kMlpOffW1);
    const __nv_bfloat16* w2g = reinterpret_cast<const __nv_bfloat16*>(model + kMlpOffW2);
    const __nv_bfloat16* w3g = reinterpret_cast<const __nv_bfloat16*>(model + kMlpOffW3);
    // 8 weights (a row of a core matrix) per load
    for (int i = tid; i < kMlpHidden * kMlpFeatures / 8; i += kTrainRows)
        *reinterpret_cast<uint4*>(s.w1 + core_offset(i / (kMlpFeatures / 8), 8 * (i % (kMlpFeatures / 8)), kMlpFeatures)) =
            reinterpret_cast<const uint4*>(w1g)[i];
    for (int i = tid; i < kMlpHidden * kMlpHidden / 8; i += kTrainRows) {
        const int o = i % kMlpHidden, in = 8 * (i / kMlpHidden);
        const uint4 v = reinterpret_cast<const uint4*>(w2g)[o * (kMlpHidden / 8) + in / 8];
        *reinterpret_cast<uint4*>(s.w2 + core_offset(o, in, kMlpHidden)) = v;
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            *reinterpret_cast<uint16_t*>(s.w2t + core_offset(in + 2 * q, o, kMlpHidden)) = (uint16_t)(w[q] & 0xffffu);
            *reinterpret_cast<uint16_t*>(s.w2t + core_offset(in + 2 * q + 1, o, kMlpHidden)) = (uint16_t)(w[q] >> 16);
        }
    }
    const float* bsrc = reinterpret_cast<const float*>(model + kMlpOffB1);
    if (tid < kMlpHidden) {
        s.b1[tid] = bsrc[tid];
        s.b2[tid] = bsrc[kMlpHidden + tid];
        s.w3[tid] = __bfloat162float(w3g[tid]);
    }
    if (tid == 0) {
        s.b3 = bsrc[2 * kMlpHidden];
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s.mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmemBase)),
                     "r"(kTrainTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // this thread's row of the minibatch (zero features past the end)
    const uint64_t base = stepPtr ? (*stepPtr % stepsPerEpoch) * (uint64_t)rows : 0;
    const unsigned row = blockIdx.x * kTrainRows + (unsigned)tid;
    const bool valid = row < rows;
    const uint64_t src = valid ? (perm ? perm[base + row] : base + row) : 0;
    {
        uint4 f[4];
#pragma unroll
        for (int j = 0; j < 4; j++) f[j] = make_uint4(0, 0, 0, 0);
        if (valid) {
            const uint4* x = reinterpret_cast<const uint4*>(feat + src * kMlpFeatures);
#pragma unroll
            for (int j = 0; j < 4; j++) f[j] = x[j];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) *reinterpret_cast<uint4*>(s.xa + core_offset(tid, 8 * j, kMlpFeatures)) = f[j];
        // X^T into rows 64-95 of the weight-gradient B operand (column = this row)
        const __nv_bfloat16* fv = reinterpret_cast<const __nv_bfloat16*>(f);
#pragma unroll
        for (int k = 0; k < kMlpFeatures; k++)
            *reinterpret_cast<__nv_bfloat16*>(s.gB + train_offset(kMlpHidden + k, tid)) = fv[k];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = s.tmemBase;
    const uint32_t laneAddr = tbase + ((uint32_t)(warp * 32) << 16);
    const uint32_t mb = smem_u32(&s.mbar);
    uint32_t phase = 0;
    bool ok = true;
    auto wait_mma = [&]() {
        if (!mbar_wait(mb, phase, kWaitPolls)) ok = false;
        phase ^= 1u;
        ok = !__syncthreads_or(!ok);
        tc_fence_after();
    };
    // ---- D1 = X W1^T (TMEM columns 0-63)
    if (tid == 0) {
#pragma unroll
        for (int k = 0; k < kMlpFeatures / 16; k++)
            tc_mma(tbase, smem_desc(smem_u32(s.xa) + 256u * k, 128, 512), smem_desc(smem_u32(s.w1) + 256u * k, 128, 512),
                   instr_desc(kTrainRows, kMlpHidden), k > 0);
        tc_commit(mb);
    }
    wait_mma();
    uint64_t h1pos = 0, h2pos = 0;  // ReLU masks of this row
    if (ok) {
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[32];
            tc_ld32(laneAddr + 32u * half, v);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t w[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int c = 32 * half + 8 * j + 2 * q;
                    const float a = fmaxf(__fadd_rn(v[8 * j + 2 * q], s.b1[c]), 0.0f);
                    const float b = fmaxf(__fadd_rn(v[8 * j + 2 * q + 1], s.b1[c + 1]), 0.0f);
                    h1pos |= (uint64_t)(a > 0.0f) << c;
                    h1pos |= (uint64_t)(b > 0.0f) << (c + 1);
                    w[q] = pack_bf16(a, b);
                }
                *reinterpret_cast<uint4*>(s.h1a + core_offset(tid, 32 * half + 8 * j, kMlpHidden)) =
                    make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
                for (int q = 0; q < 4; q++) {  // H1^T into rows 0-63 of the weight-gradient B operand
                    const int c = 32 * half + 8 * j + 2 * q;
                    *reinterpret_cast<uint16_t*>(s.gB + train_offset(c, tid)) = (uint16_t)(w[q] & 0xffffu);
                    *reinterpret_cast<uint16_t*>(s.gB + train_offset(c + 1, tid)) = (uint16_t)(w[q] >> 16);
                }
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // ---- D2 = H1 W2^T (TMEM columns 64-127)
    if (ok && tid == 0) {
#pragma unroll
        for (int k = 0; k < kMlpHidden / 16; k++)
            tc_mma(tbase + kMlpHidden, smem_desc(smem_u32(s.h1a) + 256u * k, 128, 1024),
                   smem_desc(smem_u32(s.w2) + 256u * k, 128, 1024), instr_desc(kTrainRows, kMlpHidden), k > 0);
        tc_commit(mb);
    }
    if (ok) wait_mma();
    // output layer, loss, dH2
    float h2[kMlpHidden];
    float dz = 0.0f, loss = 0.0f;
    if (ok) {
        float z = 0.0f;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[32];
            tc_ld32(laneAddr + (uint32_t)kMlpHidden + 32u * half, v);
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const int c = 32 * half + i;
                const float r = fmaxf(__fadd_rn(v[i], s.b2[c]), 0.0f);
                h2pos |= (uint64_t)(r > 0.0f) << c;
                h2[c] = __bfloat162float(__float2bfloat16_rn(r));
                z = __fadd_rn(z, __fmul_rn(h2[c], s.w3[c]));
            }
        }
        z = __fadd_rn(z, s.b3);
        if (valid) {
            const float y = label[src];
            const float pr = 1.0f / (1.0f + expf(-z));
            dz = (pr - y) * invTotal;
            const float sp = fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z)));
            loss = (sp - y * z) * invTotal;
        }
    }
    // column sums over the block's rows: four warps' sums, then in warp order
    auto colsum = [&](float v, int slot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(kFull, v, o));
        if (lane == 0) s.red[warp][slot] = v;
    };
    if (ok) {
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[32];
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = __fmul_rn(dz, h2[32 * half + i]);
            s.red[warp][32 * half + lane] = warp_sums(v, lane);  // dW3
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const int c = 32 * half + i;
                v[i] = (h2pos >> c) & 1ull ? __fmul_rn(dz, s.w3[c]) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t w[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int c = 32 * half + 8 * j + 2 * q;
                    w[q] = pack_bf16(v[8 * j + 2 * q], v[8 * j + 2 * q + 1]);
                    // dH2^T, rows 0-63
                    *reinterpret_cast<uint16_t*>(s.gA + train_offset(c, tid)) = (uint16_t)(w[q] & 0xffffu);
                    *reinterpret_cast<uint16_t*>(s.gA + train_offset(c + 1, tid)) = (uint16_t)(w[q] >> 16);
                }
                *reinterpret_cast<uint4*>(s.d2a + core_offset(tid, 32 * half + 8 * j, kMlpHidden)) =
                    make_uint4(w[0], w[1], w[2], w[3]);
            }
            s.red[warp][kMlpHidden + 32 * half + lane] = warp_sums(v, lane);  // db2
        }
        colsum(dz, 3 * kMlpHidden);      // db3
        colsum(loss, 3 * kMlpHidden + 1);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // ---- dH1 = dH2 W2 (TMEM columns 128-191)
    if (ok && tid == 0) {
#pragma unroll
        for (int k = 0; k < kMlpHidden / 16; k++)
            tc_mma(tbase + 2 * kMlpHidden, smem_desc(smem_u32(s.d2a) + 256u * k, 128, 1024),
                   smem_desc(smem_u32(s.w2t) + 256u * k, 128, 1024), instr_desc(kTrainRows, kMlpHidden), k > 0);
        tc_commit(mb);
    }
    if (ok) wait_mma();
    if (ok) {
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[32];
            tc_ld32(laneAddr + 2u * kMlpHidden + 32u * half, v);
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const int c = 32 * half + i;
                v[i] = (h1pos >> c) & 1ull ? v[i] : 0.0f;
                *reinterpret_cast<__nv_bfloat16*>(s.gA + train_offset(kMlpHidden + c, tid)) =
                    __float2bfloat16_rn(v[i]);  // dH1^T, rows 64-127
            }
            s.red[warp][2 * kMlpHidden + 32 * half + lane] = warp_sums(v, lane);  // db1
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // ---- [dW2; dW1] = [dH2^T; dH1^T] [H1^T | X^T] (TMEM columns 0-95; D1 and D2 were read)
    if (ok && tid == 0) {
#pragma unroll
        for (int k = 0; k < kTrainRows / 16; k++)
            tc_mma(tbase, smem_desc(smem_u32(s.gA) + 2 * kTrainLbo * k, kTrainLbo, kTrainSbo),
                   smem_desc(smem_u32(s.gB) + 2 * kTrainLbo * k, kTrainLbo, kTrainSbo),
                   instr_desc(kTrainRows, kTrainOutCols), k > 0);
        tc_commit(mb);
    }
    if (ok) wait_mma();
    float* out = part + (uint64_t)blockIdx.x * kMlpPartStride;
    if (ok) {
        if (tid < kMlpHidden) {  // row o of dW2: columns 0-63
#pragma unroll
            for (int half = 0; half < 2; half++) {
                float v[32];
                tc_ld32(laneAddr + 32u * half, v);
#pragma unroll
                for (int i = 0; i < 32; i += 4)
                    *reinterpret_cast<float4*>(out + kMlpOffW2 / 2 + tid * kMlpHidden + 32 * half + i) =
                        make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            }
        } else {  // row i of dW1: columns 64-95
            float v[32];
            tc_ld32(laneAddr + (uint32_t)kMlpHidden, v);
#pragma unroll
            for (int f = 0; f < kMlpFeatures; f += 4)
                *reinterpret_cast<float4*>(out + kMlpOffW1 / 2 + (tid - kMlpHidden) * kMlpFeatures + f) =
                    make_float4(v[f], v[f + 1], v[f + 2], v[f + 3]);
        }
    }
    __syncthreads();
    if (ok) {
        for (int i = tid; i < 3 * kMlpHidden + 2; i += kTrainRows) {
            const float v = __fadd_rn(__fadd_rn(__fadd_rn(s.red[0][i], s.red[1][i]), s.red[2][i]), s.red[3][i]);
            int dst;
            if (i < kMlpHidden) dst = kMlpOffW3 / 2 + i;
            else if (i < 2 * kMlpHidden) dst = kMlpParamB2 + (i - kMlpHidden);
            else if (i < 3 * kMlpHidden) dst = kMlpParamB1 + (i - 2 * kMlpHidden);
            else if (i == 3 * kMlpHidden) dst = kMlpParamB3;
            else dst = kMlpParamLoss;
            out[dst] = v;
        }
    } else {
        for (int i = tid; i < kMlpParams; i += kTrainRows) out[i] = 0.0f;
        if (tid == 0 && failed) atomicAdd(failed, 1ull);
        mbar_wait(mb, phase ^ 1u, kWaitPolls);  // the MMAs in flight, bounded again
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(kTrainTmemCols)
                     : "memory");
}

// One thread per parameter: the sum of the tiles' partials in tile order (eight
// loads in flight), then (with `state`) an Adam step on the FP32 master copy and
// the BF16/FP32 model the kernels read.  Thread kMlpParamLoss sums the loss into
// `lossOut`.  With stepPtr the last block to finish advances the step, after
// every thread has read the old powers.
__global__ void __launch_bounds__(128) mlp_reduce_kernel(const float* __restrict__ part, unsigned int parts,
                                                         float* __restrict__ grad, float* lossOut, MlpAdam* state,
                                                         unsigned char* model, unsigned long long* stepPtr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kMlpParams) {
        float sum = 0.0f;
        unsigned w = 0;
        for (; w + 8 <= parts; w += 8) {
            float x[8];
#pragma unroll
            for (int q = 0; q < 8; q++) x[q] = part[(uint64_t)(w + q) * kMlpPartStride + i];
#pragma unroll
            for (int q = 0; q < 8; q++) sum = __fadd_rn(sum, x[q]);
        }
        for (; w < parts; w++) sum = __fadd_rn(sum, part[(uint64_t)w * kMlpPartStride + i]);
        if (grad) grad[i] = sum;
        if (i == kMlpParamLoss) {
            if (lossOut) lossOut[stepPtr ? *stepPtr : 0] = sum;
        } else if (state) {
            MlpAdam& a = *state;
            const float m = a.beta1 * a.m[i] + (1.0f - a.beta1) * sum;
            const float v = a.beta2 * a.v[i] + (1.0f - a.beta2) * sum * sum;
            a.m[i] = m;
            a.v[i] = v;
            const float b1p = a.beta1Pow * a.beta1, b2p = a.beta2Pow * a.beta2;  // powers of this step
            const float mh = m / (1.0f - b1p), vh = v / (1.0f - b2p);
            const float w1 = a.master[i] - a.lr * mh / (sqrtf(vh) + a.eps);
            a.master[i] = w1;
            if (i < kMlpWeightCount) {
                reinterpret_cast<__nv_bfloat16*>(model)[i] = __float2bfloat16_rn(w1);
            } else {
                reinterpret_cast<float*>(model + kMlpOffB1)[i - kMlpWeightCount] = w1;
            }
        }
    }
    if (!state || !stepPtr) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&state->done, 1u) == gridDim.x - 1) {
            state->done = 0;
            state->beta1Pow *= state->beta1;
            state->beta2Pow *= state->beta2;
            *stepPtr += 1;
        }
    }
}

__global__ void to_bf16_kernel(const float* __restrict__ in, uint64_t n, __nv_bfloat16* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __float2bfloat16_rn(in[i]);
}

}  // namespace

size_t mlp_grad_smem_bytes() { return sizeof(TrainTc) + 1024; }

cudaError_t launch_mlp_infer(const unsigned char* model, const __nv_bfloat16* feat, const uint2* meta,
                             const unsigned int* countPtr, unsigned int count, unsigned int cap, float minLogit,
                             char* out, int outPitch, float* logits, unsigned long long* counters, int blocks,
                             cudaStream_t s) {
    if (blocks <= 0) blocks = 1;
    mlp_infer_kernel<<<blocks, kTcRows, 0, s>>>(model, feat, meta, countPtr, count, cap, minLogit, out, outPitch,
                                                 logits, counters);
    return cudaGetLastError();
}

cudaError_t launch_mlp_logits(const unsigned char* model, const float* feat, unsigned int count, float* logits,
                              unsigned long long* counters, int blocks, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    mlp_infer_kernel<<<std::max(blocks, 1), kTcRows, 0, s>>>(model, feat, static_cast<const uint2*>(nullptr),
                                                             static_cast<const unsigned int*>(nullptr), count, count,
                                                             0.0f, static_cast<char*>(nullptr), 0, logits, counters);
    return cudaGetLastError();
}

cudaError_t set_classifier_wait_limit(uint32_t polls) {
    return cudaMemcpyToSymbol(g_tileWaitSpins, &polls, sizeof(polls));
}

cudaError_t launch_mlp_grad(const unsigned char* model, const __nv_bfloat16* feat, const float* label,
                            const uint32_t* perm, const unsigned long long* stepPtr, unsigned int stepsPerEpoch,
                            unsigned int rows, float invTotal, float* part, unsigned long long* failed,
                            cudaStream_t s) {
    const size_t smem = mlp_grad_smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    mlp_grad_kernel<<<mlp_grad_parts(rows), kTrainRows, smem, s>>>(model, feat, label, perm, stepPtr,
                                                                   stepsPerEpoch ? stepsPerEpoch : 1u, rows, invTotal,
                                                                   part, failed);
    return cudaGetLastError();
}

unsigned int mlp_grad_parts(unsigned int rows) { return (rows + kTrainRows - 1) / kTrainRows; }

cudaError_t launch_mlp_reduce(const float* part, unsigned int parts, float* grad, float* lossOut, MlpAdam* state,
                              unsigned char* model, unsigned long long* stepPtr, cudaStream_t s) {
    mlp_reduce_kernel<<<(kMlpParams + 127) / 128, 128, 0, s>>>(part, parts, grad, lossOut, state, model, stepPtr);
    return cudaGetLastError();
}

cudaError_t launch_to_bf16(const float* in, uint64_t n, __nv_bfloat16* out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    to_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, n, out);
    return cudaGetLastError();
}

}  // namespace cg
