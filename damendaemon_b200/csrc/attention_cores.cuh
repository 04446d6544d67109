// What the paged attention kernels on the CUDA cores share: where a key's row lies, which keys a query sees, clusters
// whose blocks share a token's (or a tile's) keys.
#pragma once
#include "common.cuh"
#include <math_constants.h>

namespace {

struct Pages {
    const int* block_table;      // [entries, max_blocks]
    int max_blocks, page_size, n_pages, kv_heads, d;
    int page_shift;              // log2 of the page size where that is a power of two, else -1
    // a key's page, as the table has it (negative or past the last page: there is none), and its place in the page
    struct Place { int page, row; };
    __device__ __forceinline__ Place place(int entry, int key) const {
        const int blk = page_shift >= 0 ? key >> page_shift : key / page_size;
        return {blk < max_blocks ? block_table[(size_t)entry * max_blocks + blk] : -1, key - blk * page_size};
    }
    // element offset of the row of head kh there, -1 without a page; the value row lies value_plane() further on
    __device__ __forceinline__ long long row_at(const Place& at, int kh) const {
        if (at.page < 0 || at.page >= n_pages) return -1;
        return at.page * (2 * value_plane()) + (long long)(kh * page_size + at.row) * d;
    }
    __device__ __forceinline__ long long key_row(int entry, int key, int kh) const { return row_at(place(entry, key), kh); }
    __device__ __forceinline__ long long value_plane() const { return (long long)kv_heads * page_size * d; }
};

struct Mask {
    int window, chunk;
    // the first key that a query at pos sees
    __device__ __forceinline__ int first_seen(int pos) const {
        int lo = window > 0 ? max(0, pos - window + 1) : 0;
        if (chunk > 0) lo = max(lo, pos - pos % chunk);
        return lo;
    }
};

__device__ __forceinline__ float logistic(float v) { return 1.0f / (1.0f + expf(-v)); }

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
[[maybe_unused]] int shift_of(int page_size) { return page_size > 0 && !(page_size & (page_size - 1)) ? __builtin_ctz(page_size) : -1; }

int check_sizes(const char* what, int n_heads, int kv_heads, int d, int page_size, const void* q, int q_stride, int element, const void* cache,
                int window, int chunk) {
    if (d <= 0 || d * element % 16 || d > 128) return dd_fail("%s: rows of a head of %d elements are not whole 16-byte pieces, or over 128", what, d);
    if (n_heads <= 0 || kv_heads <= 0 || n_heads % kv_heads || page_size <= 0)
        return dd_fail("%s: %d heads, %d key/value heads, pages of %d tokens", what, n_heads, kv_heads, page_size);
    if (q_stride * element % 16 || (((uintptr_t)q | (uintptr_t)cache) & 15)) return dd_fail("%s: rows must be 16-byte aligned", what);
    if (window < 0 || chunk < 0) return dd_fail("%s: window %d and chunk %d must not be negative", what, window, chunk);
    return 0;
}

template <typename... KArgs, typename... Args>
int launch_clusters(const char* what, void (*kernel)(KArgs...), long long blocks, int splits, int threads, int smem, cudaStream_t s, Args... args) {
    if (blocks * splits > 0x7fffffffLL) return dd_fail("%s: %lld x %d blocks are more than one launch takes", what, blocks, splits);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)(blocks * splits));
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = s;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = splits;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = dd_pdl_enabled ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&config, kernel, static_cast<KArgs>(args)...);
    if (e != cudaSuccess) return dd_fail("%s (clusters of %d): %s", what, splits, cudaGetErrorString(e));
    return dd_check_launch(what);
}

}  // namespace
