// sbf_kernels.cu -- the tile kernels compiled for the common configurations
// (the kernel is in sbf_tile.cuh; other DNA configurations are compiled at
// run time by sbf_jit.cpp) and the auxiliary kernels.
#include <cuda_runtime.h>

#include <cstdint>

#include "sbf_configs.h"
#include "sbf_device.cuh"
#include "sbf_internal.h"
#include "sbf_tile.cuh"

namespace sbf {

// First record whose end exceeds byte x (records sorted and non-overlapping).
__device__ __forceinline__ uint32_t first_record_past(const DevRange* ranges, uint64_t n,
                                                      int64_t x) {
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (static_cast<int64_t>(ranges[mid].offset + ranges[mid].bytes) > x)
            hi = mid;
        else
            lo = mid + 1;
    }
    return static_cast<uint32_t>(lo);
}

// tile_rec[t] = first record whose end exceeds the first byte tile t stages.
__global__ void tile_records_kernel(const DevRange* ranges, uint64_t n, int64_t sym_base,
                                    uint64_t tile_kmers, uint64_t n_tiles, uint32_t* tile_rec) {
    const uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n_tiles)
        tile_rec[t] = first_record_past(ranges, n, static_cast<int64_t>(t * tile_kmers) + sym_base);
}

// All that a ragged pass needs before its tile kernel, in one launch: the
// tiles' first records and, when given, the per-record tallies at zero.  (As a
// kernel and three memsets a small ragged query with counts took 17.7 us, this
// way 13.1.)
__global__ void ragged_prepare_kernel(const DevRange* ranges, uint64_t n, int64_t sym_base,
                                      uint64_t tile_kmers, uint64_t n_tiles, uint32_t* tile_rec,
                                      unsigned long long* zero_a, unsigned long long* zero_b) {
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t t = first; t < n_tiles; t += stride)
        tile_rec[t] = first_record_past(ranges, n, static_cast<int64_t>(t * tile_kmers) + sym_base);
    if (zero_a)
        for (uint64_t i = first; i < n; i += stride) zero_a[i] = zero_b[i] = 0;
}

// tile_records_kernel with the record and tile counts read on the device.
__global__ void tile_records_sized_kernel(const DevRange* ranges, const DevSizes* sizes,
                                          int64_t sym_base, uint32_t* tile_rec) {
    const uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < sizes->n_tiles)
        tile_rec[t] = first_record_past(ranges, sizes->n_ranges,
                                        static_cast<int64_t>(t * kTileKmers) + sym_base);
}

// ---------------------------------------------------------------------------
// Auxiliary kernels
// ---------------------------------------------------------------------------

// Dense packing: 32 symbols per word, symbol t at bits [2t, 2t+2), invalid
// bytes stored as their low two code bits (include/cusbf/dense_packed.hpp:26-50).
__global__ void pack_dense_kernel(const uint8_t* seq, uint64_t num_symbols, uint64_t* words) {
    const uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t n_words = (num_symbols + 31) / 32;
    if (w >= n_words) return;
    const uint64_t first = w * 32;
    uint64_t out = 0;
    for (int t = 0; t < 32; ++t) {
        const uint64_t s = first + t;
        if (s >= num_symbols) break;
        const uint8_t b = seq[s];
        const uint8_t upper = b & 0xDFu;
        const bool valid = upper == 'A' || upper == 'C' || upper == 'G' || upper == 'T';
        const uint64_t code = valid ? ((b >> 1) & 3u) : 3u;
        out |= code << (2 * t);
    }
    words[w] = out;
}

__global__ void popcount_kernel(const uint64_t* words, uint64_t n, unsigned long long* out) {
    unsigned long long local = 0;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        local += __popcll(words[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xFFFFFFFFu, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(out, local);
}

cudaError_t launch_pack_dense(const uint8_t* seq, uint64_t num_symbols, uint64_t* words,
                              cudaStream_t stream) {
    const uint64_t n_words = (num_symbols + 31) / 32;
    if (n_words == 0) return cudaSuccess;
    pack_dense_kernel<<<static_cast<unsigned>((n_words + 255) / 256), 256, 0, stream>>>(
        seq, num_symbols, words);
    return cudaGetLastError();
}

const void* tile_records_kernel_ptr() { return reinterpret_cast<const void*>(&tile_records_kernel); }

cudaError_t launch_ragged_prepare(const DevRange* ranges, uint64_t n_ranges, int64_t sym_base,
                                  uint64_t tile_kmers, uint64_t n_tiles, uint32_t* tile_rec,
                                  unsigned long long* zero_a, unsigned long long* zero_b,
                                  cudaStream_t stream) {
    const uint64_t work = zero_a && n_ranges > n_tiles ? n_ranges : n_tiles;
    const uint64_t blocks = (work + 255) / 256;
    ragged_prepare_kernel<<<static_cast<unsigned>(blocks < 4096 ? blocks : 4096), 256, 0, stream>>>(
        ranges, n_ranges, sym_base, tile_kmers, n_tiles, tile_rec, zero_a, zero_b);
    return cudaGetLastError();
}

cudaError_t launch_tile_records_sized(const DevRange* ranges, const DevSizes* sizes,
                                      int64_t sym_base, uint64_t max_tiles, uint32_t* tile_rec,
                                      cudaStream_t stream) {
    if (max_tiles == 0) return cudaSuccess;
    tile_records_sized_kernel<<<static_cast<unsigned>((max_tiles + 255) / 256), 256, 0, stream>>>(
        ranges, sizes, sym_base, tile_rec);
    return cudaGetLastError();
}

cudaError_t launch_popcount(const uint64_t* words, uint64_t n_words, unsigned long long* out,
                            cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return e;
    if (n_words == 0) return cudaSuccess;
    uint64_t blocks = (n_words + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    popcount_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(words, n_words, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Compiled configurations
// ---------------------------------------------------------------------------

template <class Fn>
const void* fn_ptr(Fn* f) {
    return reinterpret_cast<const void*>(f);
}

template <int K, int S, int M, int H>
KernelSet make_set() {
    using C = Cfg<K, S, M, H>;
    return KernelSet{K,
                     S,
                     M,
                     H,
                     fn_ptr(&tile_kernel<C, false, false, false>),
                     fn_ptr(&tile_kernel<C, true, false, false>),
                     fn_ptr(&tile_kernel<C, false, true, false>),
                     fn_ptr(&tile_kernel<C, true, true, false>),
                     fn_ptr(&tile_kernel<C, false, false, true>),
                     fn_ptr(&tile_kernel<C, true, false, true>)};
}

static const KernelSet kSets[] = {
#define SBF_SET(K, S, M, H) make_set<K, S, M, H>(),
    SBF_COMPILED_CONFIGS(SBF_SET)
#undef SBF_SET
};
constexpr int kNumSets = static_cast<int>(sizeof kSets / sizeof kSets[0]);

const KernelSet* find_kernels(int k, int s, int m, int h) {
    for (const KernelSet& ks : kSets)
        if (ks.k == k && ks.s == s && ks.m == m && ks.h == h) return &ks;
    return nullptr;
}

// Windows per thread of a launch.  A strip's windows are worked off one after
// the other, so a launch that gives every SM few warps takes as long as one
// strip; shorter strips cost more work per window (W - 1 m-mers and F - 1
// s-mers beyond its windows) but spread over more of the chip.  <31,28,16,4>
// insert / query with strips of 8, 16 and 32 windows, in us:
//    30 k windows   5.2 / 4.7    6.2 / 6.2    8.3 / 6.7
//   400 k           6.3 / 6.2    8.3 / 6.2    8.3 / 8.3
//   800 k          10.3 / 8.3    8.3 / 8.3   10.3 / 8.3
//   1.5 M          14.4 / 12.4  12.4 / 10.3  12.4 / 10.3 (<21,19,11,4> 12.4 / 12.4)
//     3 M          22.6 / 19.5  18.5 / 15.4  18.5 / 14.4
// so strips of 8 take up to 16 warps an SM, strips of 16 up to 24.
static int narrow_strip(uint64_t n_kmers, int sms) {
    const uint64_t per_sm = n_kmers / static_cast<uint64_t>(sms > 0 ? sms : 1);
    return per_sm < 16 * 32 * 8 ? 8 : per_sm < 24 * 32 * 16 ? 16 : kStrip;
}

const void* narrow16_kernel(int config, int which);
const void* narrow8_kernel(int config, int which);

// Index of a compiled set, kNumSets of any other.
static int config_of(const KernelSet* ks) {
    int config = 0;
    while (config < kNumSets && ks != &kSets[config]) ++config;
    return config;
}

StripKernel strip_kernel(const KernelSet* ks, int which, uint64_t n_kmers, int sms) {
    const int strip = narrow_strip(n_kmers, sms);
    const int config = config_of(ks);
    if (strip == kStrip || config == kNumSets) return {ks->fn(which), kStrip};
    return {strip == 16 ? narrow16_kernel(config, which) : narrow8_kernel(config, which), strip};
}

cudaError_t prepare_strip_kernels(const KernelSet* ks) {
    const int config = config_of(ks);
    for (int which = 0; which < 6 && config < kNumSets; ++which) {
        for (const void* fn : {narrow16_kernel(config, which), narrow8_kernel(config, which)}) {
            const cudaError_t e = cudaFuncSetAttribute(
                fn, cudaFuncAttributeMaxDynamicSharedMemorySize, ks->smem(which));
            if (e != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

cudaError_t launch_set_kernel(const KernelSet* ks, const void* fn, unsigned grid, int which,
                              const TileParams& p, cudaStream_t stream) {
    TileParams copy = p;
    void* args[] = {&copy};
    return cudaLaunchKernel(fn, dim3(grid), dim3(ks->threads(which)), args, ks->smem(which), stream);
}

}  // namespace sbf
