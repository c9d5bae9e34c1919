// Library-internal hooks of the C ABI layer (care_capi.cu) for the device
// file path (care_files.cu): reads that are already in device memory, and
// results that stay there.
#ifndef CARE_CAPI_INTERNAL_H
#define CARE_CAPI_INTERNAL_H

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "care_gpu.h"

namespace cg {

// Device memory from the process's block cache (cg_release_cached_memory): at
// least n bytes, *got of them.  cached_release waits for stream s and keeps the
// block of the current device for a later request, or frees it where enough are
// kept.  It does not wait for the whole
// device: that fails, and breaks the capture, while another thread (of this
// library or of the program) captures one of its streams.
cudaError_t cached_alloc(void** p, size_t n, size_t* got);
void cached_release(void* p, size_t bytes, cudaStream_t s);

// Held while a stream is captured: no thread of this library waits for the device
// meanwhile.
struct CaptureScope {
    CaptureScope();
    ~CaptureScope();
    CaptureScope(const CaptureScope&) = delete;
    CaptureScope& operator=(const CaptureScope&) = delete;
};

// A block of it, given back on scope exit.  Allocated and given back with the
// same device current.  Work of other streams than `stream` that uses it has ended
// by then.
struct CachedMem {
    void* p = nullptr;
    size_t bytes = 0;
    cudaStream_t stream = nullptr;
    CachedMem() = default;
    CachedMem(const CachedMem&) = delete;
    CachedMem& operator=(const CachedMem&) = delete;
    ~CachedMem() { free(); }
    cudaError_t alloc(size_t n, cudaStream_t s) {
        free();
        stream = s;
        const cudaError_t e = cached_alloc(&p, n < 16 ? 16 : n, &bytes);
        if (e != cudaSuccess) p = nullptr;
        return e;
    }
    void free() {
        if (p) cached_release(p, bytes, stream);
        p = nullptr;
    }
    void* take() {  // the block is the caller's, to cudaFree
        void* q = p;
        p = nullptr;
        return q;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p);
    }
};

// cg_append_reads for one group of reads already on the device: bases back to
// back (dChars), offsets dOffs[n+1] from 0, qualities like the bases (or
// empty).  On success the context owns the blocks.
int append_device_chunk(cg_ctx* c, CachedMem& chars, CachedMem& offs, CachedMem& qual, uint64_t n, int lmax);

// cg_correct with flags[num] and sequences[num][pitch] in device memory.
int correct_into_device(cg_ctx* c, uint64_t first, uint64_t num, uint8_t* dFlags, char* dSeq, size_t pitch);

// cg_combine_results with flags[num] in device memory (candidate correction
// on); *records (may be null) gets the saved candidate records of the reads.
int combine_into_device(cg_ctx* c, uint64_t first, uint64_t num, uint8_t* dFlags, uint64_t* records);

}  // namespace cg

#endif
