// sbf_internal.h -- types shared by the kernels and the C-ABI layer.
#pragma once

#ifndef __CUDACC_RTC__
#include <cuda_runtime.h>

#include <cstdint>
#endif

namespace sbf {

// Launch geometry of the tile kernels.
constexpr int kThreads = 128;                          // threads per CTA
constexpr int kStrip = 32;                             // consecutive k-mers per thread
constexpr int kTileKmers = kThreads * kStrip;          // k-mers per tile (4096)
constexpr int kStripWords = 4;                         // code words one strip reads
constexpr int kCodeWords = (kThreads - 1) * (kStrip / 16) + kStripWords;  // per tile
constexpr int kStageBytes = kCodeWords * 16 + 64;      // staged input bytes per buffer
constexpr int kFlushSlots = 8;                         // insert bulk-reduce staging slots
constexpr int kInsertSlotBytes = kFlushSlots * kThreads * 32;  // dynamic smem of flush rings

// Run-time compilation takes device functions only.
#ifdef __CUDACC_RTC__
#define SBF_SIZE_FN __device__ constexpr
#else
#define SBF_SIZE_FN constexpr
#endif

// Warps per SM that a tile kernel's registers are limited for: 24 (80 a
// thread), 16 (128) or 8 (255).  `w` m-mers and `f` s-mers a window, `h` hashes.
// The ring of a window's s-mers is held in registers, f entries of 8 in an
// insert and of 2 (h = 4, f <= 8: 4) in a query, and spills when they do not
// fit.  100 Mbp into 256 MiB, W = 16, in us with 24 / 16 / 8 warps:
//   insert h = 4   f = 5 483 / 515    7 571 / 569   10 1136 / 643 / 711
//                  f = 14 3227 / 771 / -    17 4633 / 1850 / 928
//          h = 8   f = 5 659 / 660   10 1174 / 841 / 882
//   query  h = 4   f = 7 517 / 538    8 605 / 576   10 714 / 653 / 773
//                  f = 17 1491 / 928 / 1039    20 2304 / 1308 / 1196
//          h = 8   f = 5 668 / 694    6 867 / 763   10 1712 / 1068 / 1232
//                  f = 13 2720 / 1757 / 1497
// Shorter windows change runs more often and need larger pools, longer ones
// and more than eight hashes more registers.
SBF_SIZE_FN int query_warps(int w, int h, int f) {
    return f > (h <= 4 ? 18 : 11)                              ? 8
           : w >= 10 && w <= 16 && h <= 8 && f <= (h <= 4 ? 7 : 5) ? 24
                                                               : 16;
}
SBF_SIZE_FN int insert_warps(int w, int h, int f) {
    return f > 15 ? 8 : w >= 12 && w <= 16 && h <= 8 && f <= 5 ? 24 : 16;
}

// A warp's dynamic shared memory in the query kernels: a pool of shard slots
// (first the run lists of its lanes, 32 entries each) and the shard id of
// every slot.  A warp of random sequence needs 121 slots at W = 16 m-mers a
// window and 171 at W = 11 (the runs of 32 strips less the borrowed ones),
// with a deviation of 6 to 8; a warp that needs more takes several rounds.
// 24 warps fit an SM with 208 slots each; W = 8 needs 252.
SBF_SIZE_FN int query_pool_slots(int w, int h, int f) {
    return query_warps(w, h, f) == 24 ? 208 : 336;
}
SBF_SIZE_FN int query_warp_bytes(int w, int h, int f) {
    return query_pool_slots(w, h, f) * (32 + 4);
}
SBF_SIZE_FN int query_cta_bytes(int w, int h, int f) {
    return kThreads / 32 * query_warp_bytes(w, h, f);
}

// The insert kernels' part of a warp: the same pool, filled with the runs' word
// masks, and a spare slot per lane for a run that a neighbour flushes.  184
// slots leave room for 24 warps and 4 deviations at W = 12 (158 slots).
SBF_SIZE_FN int insert_pool_slots(int w, int h, int f) {
    return insert_warps(w, h, f) == 24 ? 184 : 304;
}
SBF_SIZE_FN int insert_warp_bytes(int w, int h, int f) {
    return insert_pool_slots(w, h, f) * (32 + 4) + 32 * 32;
}
SBF_SIZE_FN int insert_cta_bytes(int w, int h, int f) {
    return kThreads / 32 * insert_warp_bytes(w, h, f);
}

// Threads per CTA of the ragged inserts with flush rings (sbf_generic.cuh), for
// windows of `w` m-mers and symbols of `width` bytes.  In us with 256 / 128: 64 M
// residues of <12,10,10,4> 898 / 1023, of <8,6,8,4> 1161 / 1278; 48 M triplets of
// <10,8,5,4> 853 / 920, of <6,5,6,4> (one m-mer a window) 1339 / 1211.
SBF_SIZE_FN int ragged_ring_threads(int w, int width) {
    return width > 1 && w == 1 ? kThreads : 256;
}

// A record of a ragged launch: bytes [offset, offset + bytes) of the input.
// Same layout as sbf_record_range of the C ABI.
struct DevRange {
    uint64_t offset;
    uint64_t bytes;
};

// Configuration of the runtime-parameterised kernels (sbf_generic.cu), used
// for every configuration and alphabet that has no specialised kernel.
struct GenericCfg {
    uint32_t k, s, m, h;
    uint32_t bits;      // bits per packed symbol
    uint32_t width;     // input bytes per symbol
    uint32_t alphabet;  // SBF_ALPHABET_*
};

// Sizes of a ragged launch that are known only on the device: a FASTX block
// parsed on the GPU and replayed as one CUDA graph finds its record count and
// sequence length on the device, so the graph's launches read them here.
struct DevSizes {
    uint64_t input_bytes;
    uint64_t n_kmers;
    uint64_t n_tiles;   // 0 skips the pass
    uint64_t n_ranges;
};

// One launch of a tile kernel.  With T windows a tile (StripKernel::tile_kmers:
// kTileKmers, fewer with narrower strips), tile n has the grid positions
// g = n * T + (0 .. T-1); position g holds window (k-mer) i = g + sym_base,
// and symbol i is the first base of that window.
struct TileParams {
    const uint8_t* input;    // device bytes (ASCII) or dense words viewed as bytes
    uint64_t input_bytes;    // readable bytes at `input`
    uint64_t n_kmers;        // windows to process
    int64_t sym_base;        // symbol index of grid position 0 (= -phase)
    uint64_t* words;         // filter: num_shards * 4 words
    uint32_t shard_mask;     // (uint32_t)(num_shards - 1)
    uint8_t* out;            // query: one byte per window (null in bit-packed mode)
    uint32_t* out_bits;      // query, bit-packed mode: bit i % 32 of word i / 32
    uint64_t n_tiles;
    int* err;                // device error word (non-zero = failure code)
    // Ragged launches only.  Records sorted by offset and non-overlapping; a
    // window is processed only when its K bytes lie inside one record.
    const DevRange* ranges;
    uint64_t n_ranges;
    const uint32_t* tile_rec;      // per tile: first record whose end > tile start
    unsigned long long* counts;    // [0] valid windows, [1] positive windows
    // Optional per-record tallies (zeroed before the launch): valid and
    // positive windows of record r are added to rec_valid[r << rec_shift]
    // and rec_pos[r << rec_shift] (rec_shift 1 interleaves the two arrays).
    unsigned long long* rec_valid;
    unsigned long long* rec_pos;
    uint32_t rec_shift;
    GenericCfg gen;  // read by the generic kernels only
    // Ragged tile kernels: when set, input_bytes, n_kmers, n_tiles and
    // n_ranges are read from here at kernel start (n_tiles above is then the
    // host's upper bound, used only for the launch shape).
    const DevSizes* sizes;
};

// Device error codes written to TileParams::err.
enum : int {
    kDevErrNone = 0,
    kDevErrStageTimeout = 1,  // a bulk-copy wait ran out of its time bound
    kDevErrRecordRange = 2,   // sharded insert: a run record outside the rank's shards
};

#ifndef __CUDACC_RTC__
// Which of a set's kernels: insert or query of bytes, dense words, records.
enum { kInsertBytes, kQueryBytes, kInsertDense, kQueryDense, kInsertRagged, kQueryRagged };

// Function table for one compiled configuration <K,S,M,H> (k = s = m = h = 0
// for the generic table, whose kernels read TileParams::gen).  Kernels are
// launched with cudaLaunchKernel(fn, ...): a compiled kernel's host stub, or a
// cudaKernel_t of a kernel compiled at run time (jit).
struct KernelSet {
    int k, s, m, h;
    const void* insert_bytes;
    const void* query_bytes;
    const void* insert_dense;
    const void* query_dense;
    const void* insert_ragged;
    const void* query_ragged;
    // Dynamic shared memory of the insert and query kernels: the tile kernels'
    // pools, the flush ring of the generic inserts compiled at run time, none
    // for the other generic kernels.
    int smem_insert = insert_cta_bytes(k - m + 1, h, k - s + 1);
    int smem_query = query_cta_bytes(k - m + 1, h, k - s + 1);
    bool jit = false;    // loaded from a run-time compiled library
    int jit_occupancy = 4;  // resident CTAs per SM assumed for run-time compiled sets
    const void* fn(int which) const {
        const void* const fns[6] = {insert_bytes, query_bytes,   insert_dense,
                                    query_dense,  insert_ragged, query_ragged};
        return fns[which];
    }
    // Sets of generic kernels; protein tile sets have generic dense kernels.
    bool generic = false, generic_dense = false;
    bool is_tile(int which) const {
        return !generic && !(generic_dense && (which == kInsertDense || which == kQueryDense));
    }
    int ragged_insert_threads = kThreads;  // of a generic set
    int threads(int which) const {
        return which == kInsertRagged ? ragged_insert_threads : kThreads;
    }
    int smem(int which) const {
        const bool query = (which & 1) != 0;
        if (!generic && !is_tile(which)) return query ? 0 : kInsertSlotBytes;
        return query ? smem_query : smem_insert / kThreads * threads(which);
    }
};

// Resident CTAs per SM of a pass that a tuning limits to `limit` units of 256
// threads (sbf_ragged_tuning::ctas_per_sm; tuning tables hold it), 0 for no
// limit, when `occupancy` CTAs of `threads` fit.
inline uint64_t limited_ctas(uint32_t limit, uint32_t occupancy, uint32_t threads) {
    const uint64_t ctas = limit ? uint64_t{limit} * 256 / threads : occupancy;
    return ctas < 1 ? 1 : ctas < occupancy ? ctas : occupancy;
}

// A kernel and the windows per thread it was compiled for.
struct StripKernel {
    const void* fn;
    int strip;
    uint64_t tile_kmers() const { return static_cast<uint64_t>(kThreads) * strip; }
};
// The kernel of a launch of `n_kmers` windows: a set's own, or one with
// narrower strips when the launch is small.
StripKernel strip_kernel(const KernelSet* ks, int which, uint64_t n_kmers, int sms);
// Loads a set's kernels with narrower strips on the current device and lets
// them use their dynamic shared memory.  At filter creation: a small call that
// loaded its kernel took 4 ms, which none takes now, in a stream capture or
// out of one.
cudaError_t prepare_strip_kernels(const KernelSet* ks);

// Returns the kernel table for a configuration, or nullptr when it is not
// compiled into this library.
const KernelSet* find_kernels(int k, int s, int m, int h);
// The runtime-parameterised kernels (sbf_generic.cu).
const KernelSet* generic_kernels();

// Auxiliary kernels (sbf_kernels.cu).
cudaError_t launch_pack_dense(const uint8_t* seq, uint64_t num_symbols, uint64_t* words,
                              cudaStream_t stream);
// Before a ragged pass (n_tiles > 0): tile_rec[t] = first record whose end
// exceeds the first input byte of tile t (n_ranges when none), and zero_a and
// zero_b (n_ranges entries each; both or neither) at zero.
cudaError_t launch_ragged_prepare(const DevRange* ranges, uint64_t n_ranges, int64_t sym_base,
                                  uint64_t tile_kmers, uint64_t n_tiles, uint32_t* tile_rec,
                                  unsigned long long* zero_a, unsigned long long* zero_b,
                                  cudaStream_t stream);
// The tile records with the record and tile counts read from `sizes` on the device;
// `max_tiles` bounds the launch.
cudaError_t launch_tile_records_sized(const DevRange* ranges, const DevSizes* sizes,
                                      int64_t sym_base, uint64_t max_tiles, uint32_t* tile_rec,
                                      cudaStream_t stream);
cudaError_t launch_popcount(const uint64_t* words, uint64_t n_words, unsigned long long* out,
                            cudaStream_t stream);
// Kernels compiled at run time for a configuration that is not compiled into
// the library (sbf_jit.cpp): the tile kernels for DNA and proteins, the generic
// kernels with the configuration as constants for the rest; nullptr when that
// is not possible.
const KernelSet* jit_kernels(int k, int s, int m, int h, int alphabet, int device);
// Launches one of a KernelSet's kernels.
cudaError_t launch_set_kernel(const KernelSet* ks, const void* fn, unsigned grid, int which,
                              const TileParams& p, cudaStream_t stream);
#endif

}  // namespace sbf
