// Read store construction and minhash signatures.
//
// reference: include/chunkedreadstorageconstruction.hpp:29-485 (parse, N
// replacement, 2-bit encode), include/sequencehelpers.hpp:151-193 (encoding),
// :645-697 (hi/lo planes), include/cpusequencehasher.hpp:86-125 and
// include/sequencehelpers.hpp:842-930 (signatures over canonical k-mers).

#include "care_device.cuh"
#include "care_internal.h"

namespace cg {

// ---------------------------------------------------------------- scan
// Exclusive prefix sum, three phases: per-block scan + block totals, scan of
// the totals (recursively), add back.  4096 elements per block.

namespace {
constexpr int kScanBlock = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanBlock * kScanItems;

template <class T>
__global__ void scan_tile_kernel(T* __restrict__ data, size_t n, T* __restrict__ tileSums) {
    __shared__ T warpTot[kScanBlock / 32];
    const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    T run = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        const T x = (base + i < n) ? data[base + i] : T(0);
        v[i] = run;
        run += x;
    }
    // inclusive warp scan of thread totals
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T incl = run;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) warpTot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        T w = lane < kScanBlock / 32 ? warpTot[lane] : T(0);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        if (lane < kScanBlock / 32) warpTot[lane] = w;  // inclusive
    }
    __syncthreads();
    const T warpPrefix = warp == 0 ? T(0) : warpTot[warp - 1];
    const T threadPrefix = warpPrefix + incl - run;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) data[base + i] = threadPrefix + v[i];
    }
    if (tileSums && threadIdx.x == kScanBlock - 1) tileSums[blockIdx.x] = warpTot[kScanBlock / 32 - 1];
}

template <class T>
__global__ void scan_add_kernel(T* __restrict__ data, size_t n, const T* __restrict__ tileSums) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) data[i] += tileSums[i / kScanTile];
}

size_t tiles_of(size_t n) { return (n + kScanTile - 1) / kScanTile; }

template <class T>
cudaError_t scan_impl(T* data, size_t n, T* tmp, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const size_t tiles = tiles_of(n);
    if (tiles == 1) {
        scan_tile_kernel<T><<<1, kScanBlock, 0, s>>>(data, n, nullptr);
        return cudaGetLastError();
    }
    scan_tile_kernel<T><<<(unsigned)tiles, kScanBlock, 0, s>>>(data, n, tmp);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = scan_impl<T>(tmp, tiles, tmp + tiles, s);
    if (e != cudaSuccess) return e;
    scan_add_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(data, n, tmp);
    return cudaGetLastError();
}
}  // namespace

size_t scan_tmp_bytes(size_t n) {
    size_t total = 0;
    while (n > 1) {
        n = tiles_of(n);
        total += n;
    }
    return (total + 16) * sizeof(unsigned long long);
}

uint64_t scan_launches(uint64_t n) {
    uint64_t k = 0;
    while (true) {
        const uint64_t tiles = tiles_of(n);
        if (tiles <= 1) return k + 1;
        k += 2;
        n = tiles;
    }
}

cudaError_t scan_exclusive_u32(uint32_t* data, size_t n, void* tmp, cudaStream_t s) {
    return scan_impl<uint32_t>(data, n, static_cast<uint32_t*>(tmp), s);
}
cudaError_t scan_exclusive_u64(unsigned long long* data, size_t n, void* tmp, cudaStream_t s) {
    return scan_impl<unsigned long long>(data, n, static_cast<unsigned long long*>(tmp), s);
}

// ---------------------------------------------------------------- encode

namespace {

// Up to 16 characters of a read as a 2-bit word (first character highest, A C G T
// = 0 1 2 3 in either case) and, per character, whether it is another one
// (bad, same order, one bit each).  `have` >= 1 characters from p on.  The text is
// read by aligned words that hold at least one of them: up to three bytes past the
// text, within its block (blocks are multiples of 16 bytes).
struct Chars16 {
    uint32_t word, bad;
};
__device__ __forceinline__ Chars16 chars16(const char* p, int have) {
    const uint32_t skip = (uint32_t)((uintptr_t)p & 3u);
    const uint32_t* a = reinterpret_cast<const uint32_t*>(p - skip);
    const int words = ((int)skip + have + 3) / 4;
    uint32_t x[5];
#pragma unroll
    for (int i = 0; i < 5; i++) x[i] = i < words ? __ldg(a + i) : 0u;
    Chars16 r = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t y = __funnelshift_r(x[i], x[i + 1], 8 * skip), t = (y >> 1) & 0x03030303u;
        const uint32_t code = t ^ ((t >> 1) & 0x01010101u);  // per byte, right for ACGTacgt
        uint32_t sel = code | (code >> 4);                   // the codes as selectors of "ACGT"
        sel = (sel & 0xffu) | ((sel >> 8) & 0xff00u);
        const uint32_t d = __byte_perm(0x54474341u, 0u, sel) ^ (y & 0xdfdfdfdfu);
        const uint32_t other = (((d & 0x7f7f7f7fu) + 0x7f7f7f7fu) | d) & 0x80808080u;
        r.word |= ((code * 0x40100401u) >> 24) << (24 - 8 * i);
        r.bad |= ((((other >> 7) * 0x08040201u) >> 24) & 15u) << (12 - 4 * i);
    }
    r.bad &= 0xffff0000u >> have & 0xffffu;
    r.word &= have < 16 ? ~(0xffffffffu >> (2 * have)) : 0xffffffffu;
    return r;
}

__global__ void rebase_kernel(uint64_t* __restrict__ offs, uint64_t count, uint64_t base) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) offs[i] -= base;
}

// 16 lanes per read, 16 characters per lane: number of characters outside ACGTacgt
__global__ void count_invalid_kernel(const char* __restrict__ chars, const uint64_t* __restrict__ offs, uint64_t n,
                                     uint32_t* __restrict__ invalid) {
    const uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const int lane = (int)(threadIdx.x & 15);
    uint32_t cnt = 0;
    if (r < n) {
        const uint64_t b = offs[r];
        const int L = (int)(offs[r + 1] - b);
        for (int p = 16 * lane; p < L; p += 256) cnt += __popc(chars16(chars + b + p, min(16, L - p)).bad);
    }
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, d);
    if (r < n && lane == 0) invalid[r] = cnt;
}

// 16 lanes per read, a 2-bit word per lane.  Non-ACGT characters become A,C,G,T in turn; the turn
// counter starts at 0 at every multiple of 65536 reads of this call, as the
// reference's encoder threads restart it per parsed batch
// (include/chunkedreadstorageconstruction.hpp:243-282).  `invalidScan` is the
// exclusive scan of per-read invalid counts of this call (mod 2^32, which keeps
// the count mod 4).  Measured for 1M reads of 150 bp (200 MB moved, 0.03 ms at the
// memory's rate): 127 us, and 109 us for the count above; with a character per lane
// and a ballot per 32 of them 520 and 180 us.  Bound by instructions and, for the
// count, by the dependent loads of a read's offsets and text.
__global__ void encode_kernel(const char* __restrict__ chars, const uint64_t* __restrict__ offs,
                              const char* __restrict__ quals, uint64_t n, uint64_t firstId,
                              const uint32_t* __restrict__ invalidScan, uint32_t* __restrict__ enc,
                              uint16_t* __restrict__ len, uint8_t* __restrict__ qual, uint8_t* __restrict__ ambig,
                              int pitch, int lmax) {
    const uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    if (r >= n) return;
    const int lane = (int)(threadIdx.x & 15);
    const unsigned group = 0xffffu << (threadIdx.x & 16);  // the read's lanes
    const uint64_t b = offs[r];
    const int L = (int)(offs[r + 1] - b);
    const uint64_t seg = (r / kSegmentReads) * kSegmentReads;
    uint32_t ctr = invalidScan[r] - invalidScan[seg];
    const uint32_t ctr0 = ctr;
    const uint64_t id = firstId + r;
    uint32_t* row = enc + id * (uint64_t)pitch;
    for (int c = 0; c < L; c += 256) {
        const int p = c + 16 * lane;
        Chars16 v = {0u, 0u};
        if (p < L) v = chars16(chars + b + p, min(16, L - p));
        if (__any_sync(group, v.bad != 0u)) {
            const uint32_t own = __popc(v.bad);
            uint32_t incl = own;
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) {
                const uint32_t y = __shfl_up_sync(group, incl, d, 16);
                if (lane >= d) incl += y;
            }
            uint32_t turn = ctr + incl - own;
            for (uint32_t m = v.bad << 16; m != 0u; turn++) {
                const int i = __clz(m);
                m ^= 0x80000000u >> i;
                v.word = (v.word & ~(0xc0000000u >> (2 * i))) | ((turn & 3u) << (30 - 2 * i));
            }
            ctr += __shfl_sync(group, incl, 15, 16);
        }
        if (p < L) row[p >> 4] = v.word;
    }
    if (quals)
        for (int p = lane; p < L; p += 16) qual[id * (uint64_t)lmax + p] = (uint8_t)quals[b + p];
    if (lane == 0) {
        len[id] = (uint16_t)L;
        ambig[id] = ctr != ctr0;
    }
}

// the 16 odd (hi) or even (lo) bits of a 2-bit word, in order
__device__ __forceinline__ uint32_t odd_bits(uint32_t x) {
    x = (x >> 1) & 0x55555555u;
    x = (x | (x >> 1)) & 0x33333333u;
    x = (x | (x >> 2)) & 0x0f0f0f0fu;
    x = (x | (x >> 4)) & 0x00ff00ffu;
    return (x | (x >> 8)) & 0xffffu;
}

// hi/lo bit planes, 32 bases per word: one thread per word of a plane pair
// (the 2-bit rows are zero past the read, so the planes are too)
__global__ void hilo_kernel(StoreArg st, uint32_t* __restrict__ hilo) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t r = t / (uint32_t)st.wp;
    if (r >= st.n) return;
    const int w = (int)(t - r * (uint32_t)st.wp);
    const uint32_t* e = st.enc + r * (uint64_t)st.pitch;
    const uint32_t e0 = 2 * w < st.pitch ? e[2 * w] : 0u, e1 = 2 * w + 1 < st.pitch ? e[2 * w + 1] : 0u;
    uint32_t* row = hilo + r * 2 * (uint64_t)st.wp;
    row[w] = (odd_bits(e0) << 16) | odd_bits(e1);
    row[st.wp + w] = (odd_bits(e0 << 1) << 16) | odd_bits(e1 << 1);
}

// Signatures: one thread per (read, group of 16 maps); threads of a warp take
// consecutive reads of the same group so the map-major stores coalesce.
constexpr int kSigReads = 128;
constexpr int kSigGroup = 16;

__global__ void __launch_bounds__(kSigReads * 3) signature_kernel(StoreArg st, int k, int nmaps,
                                                                  unsigned long long* __restrict__ sig) {
    const uint64_t r = (uint64_t)blockIdx.x * kSigReads + (threadIdx.x % kSigReads);
    const int g = threadIdx.x / kSigReads;
    const int m0 = g * kSigGroup;
    if (r >= st.n || m0 >= nmaps) return;
    const uint64_t kmask = k == 32 ? ~0ull : ((1ull << (2 * k)) - 1ull);
    uint64_t mins[kSigGroup];
#pragma unroll
    for (int j = 0; j < kSigGroup; j++) mins[j] = ~0ull;
    const int L = st.len[r];
    if (L >= k) {
        const uint32_t* e = st.enc + r * (uint64_t)st.pitch;
        uint64_t fwd = 0, rc = 0;
        const int rcShift = 2 * (k - 1);
        for (int w = 0; w * 16 < L; w++) {
            const uint32_t word = e[w];
            const int lim = min(16, L - w * 16);
            for (int j = 0; j < lim; j++) {
                const uint64_t bb = (word >> (30 - 2 * j)) & 3u;
                fwd = ((fwd << 2) | bb) & kmask;
                rc = (rc >> 2) | ((3ull - bb) << rcShift);
                if (w * 16 + j >= k - 1) {
                    const uint64_t canon = fwd < rc ? fwd : rc;
#pragma unroll
                    for (int q = 0; q < kSigGroup; q++) {
                        const uint64_t hv = murmur64(canon + (uint64_t)(m0 + q));
                        mins[q] = hv < mins[q] ? hv : mins[q];
                    }
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kSigGroup; q++) {
        if (m0 + q < nmaps) sig[(uint64_t)(m0 + q) * st.n + r] = mins[q] & kmask;
    }
}

}  // namespace

cudaError_t launch_rebase_offsets(uint64_t* offs, uint64_t count, uint64_t base, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    rebase_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(offs, count, base);
    return cudaGetLastError();
}

cudaError_t launch_count_invalid(const char* chars, const uint64_t* offs, uint64_t n, uint32_t* invalid,
                                 cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint64_t threads = n * 16;
    count_invalid_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(chars, offs, n, invalid);
    return cudaGetLastError();
}

cudaError_t launch_encode(const char* chars, const uint64_t* offs, const char* quals, uint64_t n, uint64_t firstId,
                          const uint32_t* invalidScan, const uint64_t* /*segStart*/, uint32_t* enc, uint16_t* len,
                          uint8_t* qual, uint8_t* ambig, int pitch, int lmax, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint64_t threads = n * 16;
    encode_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(chars, offs, quals, n, firstId, invalidScan, enc,
                                                                    len, qual, ambig, pitch, lmax);
    return cudaGetLastError();
}

cudaError_t launch_hilo(StoreArg st, uint32_t* hilo, cudaStream_t s) {
    const uint64_t threads = st.n * (uint64_t)st.wp;
    hilo_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(st, hilo);
    return cudaGetLastError();
}

namespace {
__global__ void len_range_kernel(const uint16_t* __restrict__ len, uint64_t n, unsigned int* out) {
    unsigned int lo = 0xffffffffu, hi = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        lo = min(lo, (unsigned int)len[i]);
        hi = max(hi, (unsigned int)len[i]);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&out[0], lo);
        atomicMax(&out[1], hi);
    }
}
}  // namespace

namespace {
// Lossy quality store (qualityScoreBits 1 or 2): the binned score of every
// base, and the first bin's score past the read's end, where the reference's
// zero-filled encoded row decodes to bin 0 (include/qualityscorecompression.hpp:
// 25-140; scores are read as signed chars, as the reference's `int(quality[p])`
// on x86-64).  Four bytes per thread, rows of lmax bytes.
__global__ void quality_bin_kernel(uint8_t* __restrict__ qual, const uint16_t* __restrict__ len, uint64_t n,
                                   int lmax, int bits) {
    const uint64_t total = n * (uint64_t)lmax;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = i / (uint64_t)lmax;
        const int p = (int)(i - r * (uint64_t)lmax);
        const int q = (int)(int8_t)qual[i] - 33;
        uint8_t b;
        if (bits == 1) {
            b = (p >= len[r] || q <= 13) ? '(' : '5';
        } else {
            b = (p >= len[r] || q <= 4) ? '$' : q <= 13 ? '(' : q <= 20 ? '1' : '9';
        }
        qual[i] = b;
    }
}
}  // namespace

cudaError_t launch_quality_bins(uint8_t* qual, const uint16_t* len, uint64_t n, int lmax, int bits, cudaStream_t s) {
    if (n == 0 || (bits != 1 && bits != 2)) return cudaSuccess;
    const uint64_t total = n * (uint64_t)lmax;
    const unsigned blocks = (unsigned)std::min<uint64_t>((total + 255) / 256, 152 * 16);
    quality_bin_kernel<<<blocks, 256, 0, s>>>(qual, len, n, lmax, bits);
    return cudaGetLastError();
}

cudaError_t launch_len_range(const uint16_t* len, uint64_t n, unsigned int* out, cudaStream_t s) {
    len_range_kernel<<<(unsigned)std::min<uint64_t>((n + 255) / 256, 1216), 256, 0, s>>>(len, n, out);
    return cudaGetLastError();
}

cudaError_t launch_signatures(StoreArg st, int k, int nmaps, unsigned long long* sig, cudaStream_t s) {
    const unsigned blocks = (unsigned)((st.n + kSigReads - 1) / kSigReads);
    signature_kernel<<<blocks, kSigReads * 3, 0, s>>>(st, k, nmaps, sig);
    return cudaGetLastError();
}

}  // namespace cg
