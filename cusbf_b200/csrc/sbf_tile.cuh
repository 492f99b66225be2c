// sbf_tile.cuh -- sm_100a insert / query tile kernels of the Super Bloom engine
// (device code only: compiled into the library for the common configurations
// by sbf_kernels.cu and sbf_narrow*.cu, and for any other DNA configuration
// and for proteins at run time by sbf_jit.cpp).
//
// Reference path replaced: include/cusbf/detail/kernels.cuh:179-312 of
// tdortman/cuSBF (insert_sequence_kmers_kernel, contains_sequence_kmers_kernel
// and their dense-packed twins).  Results are bit-identical to it; the work
// decomposition is new:
//
//   * A CTA of 128 threads takes a tile of 4096 consecutive windows (1024 or
//     2048 in small launches).  The tile's input bytes are staged into shared
//     memory by a 1D bulk async copy (TMA) on an mbarrier.  Only the 16-byte
//     aligned interior goes through the bulk copy; ragged edges are read with
//     plain loads, so nothing outside the caller's buffer is touched.  Every
//     wait is bounded and reports kDevErrStageTimeout instead of hanging.
//   * Staged bytes are encoded with SWAR into 2-bit code words (16 bases per
//     32-bit word, earliest base in the top bits) plus invalid masks.
//   * Each thread owns a strip of 32 consecutive windows (8 or 16 in small
//     launches).  Every m-mer and s-mer of the strip is a funnel shift of the
//     code words, every position is hashed once, and the per-window minimizer
//     is a Gil-Werman sliding minimum over blocks of W positions (about 3
//     comparisons per window, one more for W > 16, where the reference hashes
//     and compares all W m-mers of every window).
//   * Both list a strip's super-k-mer runs (consecutive windows that select
//     one shard) and give the runs that hold a valid window consecutive slots
//     of a per-warp shared-memory pool; a run that crosses into the next
//     strip is one run.  (Windows of one or two m-mers go through the pool in
//     parts of 8 windows.)
//   * Query has the warp copy the runs' 32-byte shards to their slots with
//     cp.async, a lane pair per shard (one request each), and tests the
//     findere rule (all k-s+1 s-mers present) per window with byte permutes
//     of the current run's shard.
//   * Insert ORs the one-hot masks of a run's s-mers in registers, stores them
//     to the run's slot, and has the warp OR the slots into their shards, four
//     lanes and one request each.
//   * Ragged launches drop windows that cross a record boundary or touch a byte
//     outside every record (marked per tile in shared memory).
#pragma once

#include "sbf_device.cuh"
#include "sbf_internal.h"

namespace sbf {

// A filter configuration, the windows per thread (strip) and the bits of a
// symbol: 2 for DNA, 5 for proteins.
template <int K_, int S_, int M_, int H_, int Strip_ = kStrip, int Bits_ = 2>
struct Cfg {
    static constexpr int K = K_;
    static constexpr int S = S_;
    static constexpr int M = M_;
    static constexpr int H = H_;
    static constexpr int W = K - M + 1;  // m-mers per window
    static constexpr int F = K - S + 1;  // s-mers per window (findere span)
    static constexpr int kBits = Bits_;
    static constexpr int kStrip = Strip_;
    static constexpr int kTileKmers = kThreads * kStrip;
    // Code words of a strip and of a tile.  DNA words hold 16 bases; protein
    // symbols run on from word to word, five words a strip.
    static constexpr int kStripWords =
        kBits == 2 ? sbf::kStripWords : ((kStrip + K - 1) * kBits + 31) / 32;
    static constexpr int kCodeWords = kBits == 2 ? (kThreads - 1) * kStrip / 16 + kStripWords
                                                 : (kThreads + 1) * kStrip * kBits / 32;
    static constexpr int kSpan = kCodeWords * 32 / kBits;  // symbols staged and encoded
    static constexpr int kStageBytes = kSpan + 64;
    // The passes over a strip's windows take them in turns of at most 16.
    static constexpr int kTurn = kStrip < 16 ? kStrip : 16;
    static constexpr int kTurns = kStrip / kTurn;
    static constexpr uint32_t kAll = 0xFFFFFFFFu >> (32 - kStrip);  // a strip's windows
    // The windows of a strip that go through the warp's pool at a time: with one
    // or two m-mers a window, a run every 1 or 1.5 windows, strips overflow it.
    static constexpr int kPart = W <= 2 && kBits == 2 ? 8 : kStrip;
    static constexpr int kParts = kStrip / kPart;
    static_assert(kStrip == 8 || kStrip == 16 || kStrip == 32, "strips of 8, 16 or 32 windows");
    static_assert(kTileKmers / 4 % 16 == 0, "tiles start at one phase of 16 bytes");
    static_assert(kBits == 2 || (kBits == 5 && kStrip == 32), "DNA, or proteins in full strips");
    static_assert(K >= 1 && K * kBits <= 64, "k must fit a 64-bit packed window");
    static_assert(M >= 1 && M <= K, "m must satisfy 1 <= m <= k");
    static_assert(S >= 1 && S <= K, "s must satisfy 1 <= s <= k");
    static_assert(H % 4 == 0 && H >= 4 && H <= 16, "hash count must be 4, 8, 12 or 16");
};

// ---------------------------------------------------------------------------
// Tile geometry and staging
// ---------------------------------------------------------------------------

struct TileGeom {
    uint64_t a;      // 16-byte aligned address of stage byte 0
    uint32_t off;    // stage offset of the tile's first input byte
    uint64_t lo, hi; // bulk-copied address range [lo, hi), empty when lo >= hi
    uint64_t r0, r1; // readable range of the input [r0, r1)
    uint32_t span;   // staged bytes
    int64_t b_lo;    // input byte index of stage offset `off`
    int64_t s0;      // symbol index of the tile's first grid position
};

template <class C>
__device__ __forceinline__ int64_t tile_first_symbol(const TileParams& p, uint64_t tile) {
    return static_cast<int64_t>(tile) * C::kTileKmers + p.sym_base;
}

template <class C, bool kDense>
__device__ __forceinline__ TileGeom tile_geom(const TileParams& p, uint64_t tile) {
    TileGeom g;
    g.s0 = tile_first_symbol<C>(p, tile);
    uint32_t need;
    if constexpr (kDense) {
        // 2-bit symbols: symbol s sits at bit 2s of the byte stream.
        g.b_lo = g.s0 >= 0 ? g.s0 / 4 : -((-g.s0 + 3) / 4);
        need = (C::kCodeWords * 16 + 3) / 4 + 8;
    } else {
        g.b_lo = g.s0;
        need = C::kSpan + 4;
    }
    const uint64_t base = reinterpret_cast<uint64_t>(p.input);
    const uint64_t first = base + static_cast<uint64_t>(g.b_lo);  // wraps for b_lo < 0
    g.a = first & ~uint64_t{15};
    g.off = static_cast<uint32_t>(first & 15u);
    g.span = (g.off + need + 15u) & ~15u;
    g.r0 = base;
    g.r1 = base + p.input_bytes;
    const uint64_t in_lo = (base + 15u) & ~uint64_t{15};
    const uint64_t in_hi = g.r1 & ~uint64_t{15};
    // Signed comparisons: the stage window may start before the input.
    const int64_t a_s = static_cast<int64_t>(g.a - base);
    const int64_t lo_s = a_s > static_cast<int64_t>(in_lo - base) ? a_s
                                                                  : static_cast<int64_t>(in_lo - base);
    const int64_t hi_end = a_s + static_cast<int64_t>(g.span);
    const int64_t hi_s = hi_end < static_cast<int64_t>(in_hi - base)
                             ? hi_end
                             : static_cast<int64_t>(in_hi - base);
    g.lo = base + static_cast<uint64_t>(lo_s);
    g.hi = base + static_cast<uint64_t>(hi_s);
    if (hi_s <= lo_s) g.hi = g.lo;
    return g;
}

// Starts the tile's staging copy; returns whether it covers the whole stage
// window (every tile but those at the input's ends).
template <class C, bool kDense>
__device__ __forceinline__ bool issue_stage(const TileParams& p, uint64_t tile, uint8_t* buf,
                                            uint64_t* bar) {
    const TileGeom g = tile_geom<C, kDense>(p, tile);
    fence_proxy_async_smem();
    if (g.hi > g.lo) {
        const uint32_t bytes = static_cast<uint32_t>(g.hi - g.lo);
        mbar_arrive_expect_tx(bar, bytes);
        bulk_g2s(buf + (g.lo - g.a), reinterpret_cast<const void*>(g.lo), bytes, bar);
    } else {
        mbar_arrive(bar);
    }
    return g.lo == g.a && g.hi == g.a + g.span;
}

// Plain loads of the readable bytes of the stage window that the bulk copy
// did not cover (at most 15 at each end of the input).
template <bool kDense>
__device__ __forceinline__ void fill_ragged(const TileParams& p, const TileGeom& g, uint8_t* buf) {
    const int64_t base = static_cast<int64_t>(g.r0);
    const int64_t w0 = static_cast<int64_t>(g.a - g.r0);  // window start rel. to input
    const int64_t w1 = w0 + g.span;
    const int64_t in0 = 0, in1 = static_cast<int64_t>(p.input_bytes);
    const int64_t v0 = w0 > in0 ? w0 : in0;  // readable part of the window
    const int64_t v1 = w1 < in1 ? w1 : in1;
    if (v1 <= v0) return;
    const int64_t c0 = static_cast<int64_t>(g.lo) - base;
    const int64_t c1 = static_cast<int64_t>(g.hi) - base;
    // Head [v0, c0) and tail [c1, v1) when a bulk copy ran; otherwise all.
    int64_t h0 = v0, h1 = v1, t0 = 0, t1 = 0;
    if (c1 > c0) {
        h1 = c0 < v1 ? c0 : v1;
        t0 = c1 > v0 ? c1 : v0;
        t1 = v1;
    }
    const int tid = threadIdx.x;
    const int64_t nh = h1 > h0 ? h1 - h0 : 0;
    const int64_t nt = t1 > t0 ? t1 - t0 : 0;
    for (int64_t x = tid; x < nh + nt; x += kThreads) {
        const int64_t src = x < nh ? h0 + x : t0 + (x - nh);
        buf[src - w0] = p.input[src];
    }
}

// Where grid position 0 lies in the stage: its byte, or its bit for dense
// input.  The same for every tile, since a tile is a multiple of 16 bytes.
template <class C, bool kDense>
__device__ __forceinline__ uint32_t stage_origin(const TileParams& p) {
    const TileGeom g = tile_geom<C, kDense>(p, 0);
    return kDense ? 8u * g.off + 2u * static_cast<uint32_t>(g.s0 - 4 * g.b_lo) : g.off;
}
// Encodes code word q (16 symbols from grid position 16q) of the staged tile.
template <bool kDense>
__device__ __forceinline__ void encode_word(uint32_t origin, const uint8_t* buf, int q,
                                            uint32_t& code, uint32_t& inval) {
    const uint32_t* w32 = reinterpret_cast<const uint32_t*>(buf);
    if constexpr (kDense) {
        const uint32_t bitpos = origin + 32u * q;
        const uint32_t wi = bitpos >> 5;
        const uint32_t v = __funnelshift_r(w32[wi], w32[wi + 1], bitpos & 31u);
        code = dense16_to_code(v);
        inval = 0u;
    } else {
        const uint32_t bytepos = origin + 16u * q;
        const uint32_t wi = bytepos >> 2;
        const uint32_t sh = (bytepos & 3u) * 8u;
        const uint32_t x0 = w32[wi], x1 = w32[wi + 1], x2 = w32[wi + 2], x3 = w32[wi + 3],
                       x4 = w32[wi + 4];
        encode16(__funnelshift_r(x0, x1, sh), __funnelshift_r(x1, x2, sh),
                 __funnelshift_r(x2, x3, sh), __funnelshift_r(x3, x4, sh), code, inval);
    }
}

// Encodes the 32 protein symbols from grid position 32 t into five code words
// (5 bits a symbol, earliest symbol in the top bits) and a word of invalid
// bits.  Letters only, either case; code = letter - 'A'.  With the rest of the
// tile kernel as for DNA, 64 M residues of <12,10,6,4> take 260 us to query and
// 302 to insert, where a byte load and a whole window's hashes per window took
// 647 and 736 (sbf_generic.cuh).
__device__ __forceinline__ void encode_protein_strip(uint32_t origin, const uint8_t* buf, int t,
                                                     uint32_t* code, uint32_t* inval) {
    const uint32_t bytepos = origin + 32u * t;
    const uint32_t* x = reinterpret_cast<const uint32_t*>(buf) + (bytepos >> 2);
    const uint32_t sh = (bytepos & 3u) * 8u;
    uint32_t g[8], bad[8], any = 0;  // 20 bits of four symbols, their invalid bytes
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t v = __funnelshift_r(x[i], x[i + 1], sh);
        const uint32_t c = ((v & 0x1F1F1F1Fu) + 0x1F1F1F1Fu) & 0x1F1F1F1Fu;
        // Above 'Z' (code 26 and up, '@' wraps to 31), or not 01xxxxxx.
        bad[i] = ((c + 0x66666666u) & 0x80808080u) | ((v ^ 0x40404040u) & 0xC0C0C0C0u);
        any |= bad[i];
        const uint32_t pair = (c & 0x001F001Fu) * 32u + ((c >> 8) & 0x001F001Fu);
        g[i] = (pair & 0xFFFFu) * 1024u + (pair >> 16);
    }
    code[5 * t] = (g[0] << 12) | (g[1] >> 8);
    code[5 * t + 1] = (g[1] << 24) | (g[2] << 4) | (g[3] >> 16);
    code[5 * t + 2] = (g[3] << 16) | (g[4] >> 4);
    code[5 * t + 3] = (g[4] << 28) | (g[5] << 8) | (g[6] >> 12);
    code[5 * t + 4] = (g[6] << 20) | g[7];
    uint32_t bits = 0;
    if (any) {
#pragma unroll
        for (int i = 0; i < 8; ++i) bits |= nonzero_bytes_to_bits(bad[i]) << (4 * i);
    }
    inval[t] = bits;
}

// Expands the four low bits of `nib` into four 0/1 bytes (bit r -> byte r).
__device__ __forceinline__ uint32_t spread4(uint32_t nib) {
    return (nib * 0x00204081u) & 0x01010101u;
}

// ---------------------------------------------------------------------------
// Strip computation: kStrip consecutive windows per thread
// ---------------------------------------------------------------------------

// The 32 bits from bit `at` of the strip's code words (earliest bits on top).
// `at` is a compile-time constant after unrolling, so every access is a
// register; bits past the last word read 0.
template <class C>
__device__ __forceinline__ uint32_t bits32(const uint32_t* c, int at) {
    const int q = at >> 5, s = at & 31;
    if (s == 0) return c[q];
    return __funnelshift_l(q + 1 < C::kStripWords ? c[q + 1] : 0u, c[q], s);
}

// The `bits` bits from bit `at` on, right-aligned.
template <class C, int bits>
__device__ __forceinline__ uint64_t bits64(const uint32_t* c, int at) {
    if constexpr (bits > 32) {
        const uint64_t hi = bits32<C>(c, at) >> (64 - bits);
        return (hi << 32) | bits32<C>(c, at + bits - 32);
    } else {
        return bits32<C>(c, at) >> (32 - bits);
    }
}

// The hash of the m-mer, and the s-mer, at strip position r.
template <class C>
__device__ __forceinline__ uint64_t mh_at(const uint32_t* c, int r) {
    const uint64_t v = bits64<C, C::M * C::kBits>(c, r * C::kBits);
    if constexpr (C::M * C::kBits > 32)
        return mmer_hash(v);
    else
        return mmer_hash(static_cast<uint32_t>(v));
}

template <class C>
__device__ __forceinline__ uint64_t smer_at(const uint32_t* c, int r) {
    return bits64<C, C::S * C::kBits>(c, r * C::kBits);
}

// Calls fn(j, v) for j = 0..N-1 in order, v being the minimum hash of the W
// m-mers from position j on (2 <= W <= 16): a Gil-Werman sliding minimum over
// blocks of W positions.  Window b0 + r of the block starting at b0 is
// min(suffix_b0[r], prefix_{b0+W}[r-1]), about three 64-bit comparisons per
// window whatever W is (instead of W - 1).
template <class C, int W, int N, class Fn>
__device__ __forceinline__ void sliding_min(const uint32_t* c, Fn&& fn) {
#pragma unroll
    for (int b0 = 0; b0 < N; b0 += W) {
        uint64_t suf[W];
        suf[W - 1] = mh_at<C>(c, b0 + W - 1);
#pragma unroll
        for (int r = W - 2; r >= 0; --r) suf[r] = min64(mh_at<C>(c, b0 + r), suf[r + 1]);
        fn(b0, suf[0]);
        uint64_t pre = ~uint64_t{0};
#pragma unroll
        for (int r = 1; r < W; ++r) {
            if (b0 + r < N) {
                pre = min64(pre, mh_at<C>(c, b0 + W - 1 + r));
                fn(b0 + r, min64(suf[r], pre));
            }
        }
    }
}

// Calls fn(j, lo) for the strip's windows in order, lo being
// the low word of the window's minimum m-mer hash (its shard id, unmasked).
// Windows of more than 16 m-mers take the minimum of their first and their
// last 16.
template <class C, class Fn>
__device__ __forceinline__ void for_each_min(const uint32_t* c, Fn&& fn) {
    constexpr int W = C::W;
    if constexpr (W == 1) {
#pragma unroll
        for (int j = 0; j < C::kStrip; ++j) fn(j, static_cast<uint32_t>(mh_at<C>(c, j)));
    } else if constexpr (W <= 16) {
        sliding_min<C, W, C::kStrip>(
            c, [&](int j, uint64_t v) { fn(j, static_cast<uint32_t>(v)); });
    } else {
        constexpr int D = W - 16;
        uint64_t first[D];
        sliding_min<C, 16, C::kStrip + D>(c, [&](int j, uint64_t v) {
            if (j >= D) fn(j - D, static_cast<uint32_t>(min64(first[j % D], v)));
            first[j % D] = v;
        });
    }
}

// for_each_min with the shard id masked to the filter's shards.
template <class C, class Fn>
__device__ __forceinline__ void for_each_shard(const uint32_t* c, uint32_t shard_mask, Fn&& fn) {
    for_each_min<C>(c, [&](int j, uint32_t lo) { fn(j, lo & shard_mask); });
}

// Bit j of the result: some bit of x[j .. j + N - 1] is set (doubling spans,
// five steps for N = 31, where a test per window cost 200 instructions a
// strip as soon as one lane of the warp met an invalid base).
template <int N>
__device__ __forceinline__ uint64_t any_in_span(uint64_t x) {
#pragma unroll
    for (int n = 1; n < N; n += n) x |= x >> (n < N - n ? n : N - n);
    return x;
}

// Valid-window mask: window j holds K valid bases and lies in [0, n_kmers).
// Bit r of `bits` is set when the strip's base r is invalid.
template <class C>
__device__ __forceinline__ uint32_t strip_valid(uint64_t bits, int64_t first_kmer,
                                                uint64_t n_kmers) {
    constexpr int kStrip = C::kStrip;
    uint32_t vmask = C::kAll;
    if (bits) vmask = ~static_cast<uint32_t>(any_in_span<C::K>(bits)) & C::kAll;
    const int64_t left = static_cast<int64_t>(n_kmers) - first_kmer;  // windows from the first on
    if (first_kmer < 0) vmask = first_kmer > -kStrip ? vmask & (~0u << -first_kmer) : 0u;
    if (left < kStrip) vmask = left > 0 ? vmask & ((1u << left) - 1u) : 0u;
    return vmask;
}

// One-hot word masks of the s-mer at strip position r.  With four hashes each
// word gets one bit: the first word's mask is read from `onehot` (1 << b for
// b = 0..63 in the CTA's shared memory) and the others are 64-bit shifts.
// The table spares the logic pipe two instructions a word, but 32 random
// entries take about six passes of the shared-memory pipe: 100 Mbp plain and
// 200 Mbp of contigs take 429 and 936 us with two loads, 433 and 924 with one,
// 100 Mbp 444 with none.
template <class C>
__device__ __forceinline__ void smer_masks(const uint32_t* c, int r, uint64_t m[4],
                                           const uint64_t* onehot) {
    const uint64_t h = smer_hash(smer_at<C>(c, r));
    if constexpr (C::H == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            m[j] = j == 0 ? onehot[bit_address<4>(h, j)] : uint64_t{1} << bit_address<4>(h, j);
    } else {
        m[0] = m[1] = m[2] = m[3] = 0;
#pragma unroll
        for (int j = 0; j < C::H; ++j) m[j & 3] |= uint64_t{1} << bit_address<C::H>(h, j);
    }
}

// Fills the one-hot table of smer_masks (threads 0..63; the caller's next
// barrier publishes it).
__device__ __forceinline__ void onehot_init(uint64_t* onehot) {
    if (threadIdx.x < 64) onehot[threadIdx.x] = uint64_t{1} << threadIdx.x;
}

__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// One byte per window; the grid phase aligns whole strips to their size.
template <class C>
__device__ __forceinline__ void store_strip_bytes(uint32_t result, uint8_t* out, int64_t first_kmer,
                                                  uint64_t n_kmers) {
    constexpr int kStrip = C::kStrip;
    if (first_kmer >= 0 && first_kmer + kStrip <= static_cast<int64_t>(n_kmers)) {
        uint32_t v[kStrip / 4];
#pragma unroll
        for (int q = 0; q < kStrip / 4; ++q) v[q] = spread4((result >> (4 * q)) & 0xFu);
        if constexpr (kStrip == 8) {
            *reinterpret_cast<uint2*>(out + first_kmer) = make_uint2(v[0], v[1]);
        } else {
            uint4* dst = reinterpret_cast<uint4*>(out + first_kmer);
#pragma unroll
            for (int q = 0; q < kStrip / 16; ++q)
                dst[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < kStrip; ++j) {
            const int64_t i = first_kmer + j;
            if (i >= 0 && i < static_cast<int64_t>(n_kmers))
                out[i] = static_cast<uint8_t>((result >> j) & 1u);
        }
    }
}

// One bit per window (grid phase 0).  Strips up to the end of the last word
// are written, so that its unused bits are 0.
template <class C>
__device__ __forceinline__ void store_strip_bits(uint32_t result, uint32_t* out,
                                                 int64_t first_kmer, uint64_t n_kmers) {
    if ((first_kmer & ~int64_t{31}) >= static_cast<int64_t>(n_kmers)) return;
    if constexpr (C::kStrip == 32)
        out[first_kmer >> 5] = result;
    else if constexpr (C::kStrip == 16)
        reinterpret_cast<uint16_t*>(out)[first_kmer >> 4] = static_cast<uint16_t>(result);
    else
        reinterpret_cast<uint8_t*>(out)[first_kmer >> 3] = static_cast<uint8_t>(result);
}

// Windows of a turn of a strip of 32.  The ring of a window's F s-mers keeps
// position r at index r % F of the turn; its turn() renames it for the next.
constexpr int kTurn = 16;

// Moves the strip's code words on by the 16 windows of a turn.
template <class C>
__device__ __forceinline__ void next_turn_words(uint32_t (&c)[C::kStripWords]) {
    constexpr int kWords = kTurn * C::kBits / 32, kShift = kTurn * C::kBits % 32;
#pragma unroll
    for (int q = 0; q < C::kStripWords; ++q) {
        const uint32_t a = q + kWords < C::kStripWords ? c[q + kWords] : 0u;
        const uint32_t b = q + kWords + 1 < C::kStripWords ? c[q + kWords + 1] : 0u;
        c[q] = kShift ? __funnelshift_l(b, a, kShift) : a;
    }
}

// Loads a slot's shard words x[0..7] from shared address `addr` when `pred` is
// non-zero, leaves them unchanged otherwise, and advances `addr` to the next
// slot after a load: predicated, so that a run head costs no branch.
__device__ __forceinline__ void next_slot_if(uint32_t pred, uint32_t& addr, uint32_t (&x)[8]) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %9, 0;\n\t"
        "@p ld.shared.v4.u32 {%0, %1, %2, %3}, [%8];\n\t"
        "@p ld.shared.v4.u32 {%4, %5, %6, %7}, [%8+16];\n\t"
        "@p add.u32 %8, %8, 32;\n\t}"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]),
          "+r"(x[7]), "+r"(addr)
        : "r"(pred));
}

// Strip `strip` of the tile's code words at shared address `code`: the strip's
// first base comes to the top of c[0].
template <class C>
__device__ __forceinline__ void load_code_words(uint32_t code, uint32_t strip,
                                                uint32_t (&c)[C::kStripWords]) {
    if constexpr (C::kBits != 2) {
#pragma unroll
        for (int q = 0; q < C::kStripWords; ++q)
            asm volatile("ld.shared.u32 %0, [%1];"
                         : "=r"(c[q])
                         : "r"(code + (C::kStrip * C::kBits / 8) * strip + 4 * q)
                         : "memory");
    } else if constexpr (C::kStrip == 32) {
        asm volatile(
            "ld.shared.v2.u32 {%0, %1}, [%4];\n\tld.shared.v2.u32 {%2, %3}, [%4+8];"
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
            : "r"(code + 8 * strip)
            : "memory");
    } else {
        // 46 bases (16 windows of 31) are in three words.
        const uint32_t at = code + (strip * C::kStrip / 16) * 4;
        asm volatile(
            "ld.shared.u32 %0, [%3];\n\tld.shared.u32 %1, [%3+4];\n\tld.shared.u32 %2, [%3+8];"
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2])
            : "r"(at)
            : "memory");
        c[3] = 0;
        if constexpr (C::kStrip == 8) {
            const uint32_t sh = 16 * (strip & 1u);
            c[0] = __funnelshift_l(c[1], c[0], sh);
            c[1] = __funnelshift_l(c[2], c[1], sh);
            c[2] <<= sh;
        }
    }
}

// ---------------------------------------------------------------------------
// Query of one strip
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// (a & ~m) | (b & m) as one instruction (written in C it took two with a
// constant m, 15% of the test pass).
__device__ __forceinline__ uint32_t bit_select(uint32_t a, uint32_t b, uint32_t m) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xD8;" : "=r"(d) : "r"(a), "r"(b), "r"(m));
    return d;
}

// Appends `lo` to the strip's run list at shared address `at` (entries are a
// warp's 128 bytes apart) when it differs
// from `prev`, and sets `bit` in `chg`: predicated, since some lane of a warp
// starts a run on almost every window.
__device__ __forceinline__ void run_list_put(uint32_t lo, uint32_t prev, uint32_t bit,
                                             uint32_t& at, uint32_t& chg) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, %3;\n\t"
        "@p st.shared.u32 [%0], %2;\n\t"
        "@p add.u32 %0, %0, 128;\n\t"
        "@p or.b32 %1, %1, %4;\n\t}"
        : "+r"(at), "+r"(chg)
        : "r"(lo), "r"(prev), "r"(bit)
        : "memory");
}

// Copies a word of shared memory when `pred` is non-zero.
__device__ __forceinline__ void copy_u32_if(uint32_t pred, uint32_t dst, uint32_t src) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b32 v;\n\tsetp.ne.u32 p, %0, 0;\n\t"
        "@p ld.shared.u32 v, [%2];\n\t@p st.shared.u32 [%1], v;\n\t}" ::"r"(pred),
        "r"(dst), "r"(src)
        : "memory");
}

// The shard ids of a lane's slots, from its run list: head b's entry is the
// number of runs that start up to it.  Four heads a turn (the busiest lane of
// a warp has about 7): a 4 Mbp query took 19.8 us, with one head a turn 20.4.
__device__ __forceinline__ void list_shard_ids(uint32_t heads, uint32_t chg, uint32_t list,
                                               uint32_t ids) {
    while (__any_sync(0xFFFFFFFFu, heads != 0u)) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t b = heads & (0u - heads);
            heads ^= b;
            const uint32_t e = __popc(chg & (b ^ (b - 1u)));
            copy_u32_if(b, ids + 4 * u, list - 128 + 128 * e);
        }
        ids += 16;
    }
}

// Copies the shards of slots e = lane / 2, lane / 2 + 16, ... below `total`
// into the pool, a lane pair per slot: its two 16-byte copies go out in one
// instruction and make one 32-byte request (a lane that issued both made two,
// and the memory serves requests: 18.5 against 36.9 G shards/s on an 8 GiB
// table).  An L2 miss fills 64 bytes (.L2::64B) instead of 128.
__device__ __forceinline__ void copy_shards(uint32_t total, uint32_t pool, uint32_t ids,
                                            uint32_t shard_mask, const uint64_t* words) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t* half = words + 2 * (lane & 1u);
    uint32_t id = ids + 4 * (lane >> 1), dst = pool + 16 * lane;
    for (uint32_t e = lane >> 1; __any_sync(0xFFFFFFFFu, e < total); e += 64) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            asm volatile(
                "{\n\t.reg .pred p;\n\t.reg .b32 s;\n\t.reg .b64 a;\n\t"
                "setp.lt.u32 p, %0, %1;\n\t"
                "@p ld.shared.u32 s, [%2];\n\t"
                "@p and.b32 s, s, %3;\n\t"
                "@p mad.wide.u32 a, s, 32, %4;\n\t"
                "@p cp.async.cg.shared.global.L2::64B [%5], [a], 16;\n\t}" ::"r"(e + 16 * u),
                "r"(total), "r"(id + 64 * u), "r"(shard_mask), "l"(half), "r"(dst + 512 * u)
                : "memory");
        id += 256;
        dst += 2048;
    }
    cp_async_commit();
}

// Findere test of the window's F s-mers (F = 3 or 4) with byte permutes.  A bit
// address is a byte n (upper three bits) and a bit t in it: for each shard
// word one permute picks the F bytes that the s-mers name and one picks the F
// one-bit masks, and an s-mer is missing when a mask bit is not set in its
// byte.  With four hashes that is 8 permutes and 4 logic operations a window,
// where F * 4 shifts of 64-bit words and their AND took 24; further sets of
// four hashes cost the same again.  n[g][i] holds the n of set g for two words
// in its halves, one nibble per s-mer of the window, t[g][i] the t.
template <int F, int H>
struct ByteTest {
    static constexpr int kSets = H / 4;
    // Nibble 8 reads the sign of mask byte 0, which is 0: no test.
    static constexpr uint32_t kUnused = F == 4 ? 0u : 0x80008000u;
    uint32_t n[kSets][2], t[kSets][2];

    __device__ __forceinline__ ByteTest() {
#pragma unroll
        for (int g = 0; g < kSets; ++g) {
            n[g][0] = n[g][1] = 0;
            t[g][0] = t[g][1] = kUnused;
        }
    }
    // The shard word whose hashes are in half `half` of n[g][i].
    __device__ __forceinline__ static constexpr int word(int i, int half) {
        return H == 8 ? i + 2 * half : 2 * i + half;
    }
    __device__ __forceinline__ void enter(int r, uint64_t h) {
        const uint32_t lo = static_cast<uint32_t>(h), hi = static_cast<uint32_t>(h >> 32);
        const int s = 4 * (r % F);
        const uint32_t m = 0x00070007u << s;
#pragma unroll
        for (int g = 0; g < kSets; ++g) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                // Bit addresses at bits 0-5 and 16-21 (other bits are ignored).
                uint32_t a;
                if constexpr (H == 4)
                    a = i ? hi : lo;
                else if constexpr (H == 8)
                    a = (g ? hi : lo) >> (8 * i);
                else
                    a = bit_address<H>(h, 4 * g + 2 * i) | (bit_address<H>(h, 4 * g + 2 * i + 1) << 16);
                n[g][i] = bit_select(n[g][i], s ? a << (s ? s - 3 : 0) : a >> 3, m);
                t[g][i] = bit_select(t[g][i], a << s, m);
            }
        }
    }
    // Non-zero when an s-mer of the window is missing from shard x.
    __device__ __forceinline__ uint32_t missing(const uint32_t (&x)[8]) const {
        uint32_t bad = 0;
#pragma unroll
        for (int g = 0; g < kSets; ++g) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int q = word(i, half);
                    bad |= prmt(0x08040201u, 0x80402010u, t[g][i] >> (16 * half)) &
                           ~prmt(x[2 * q], x[2 * q + 1], n[g][i] >> (16 * half));
                }
            }
        }
        return bad;
    }
    __device__ __forceinline__ void turn() {
        if constexpr (F == 3) {  // index i takes over from (i + 16) % 3
            auto rotate = [](uint32_t v) {
                return ((v >> 4) & 0x00FF00FFu) | ((v & 0x000F000Fu) << 8);
            };
#pragma unroll
            for (int g = 0; g < kSets; ++g) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    n[g][i] = rotate(n[g][i]);
                    t[g][i] = rotate(t[g][i]) | kUnused;
                }
            }
        }
    }
};

// The word `q` of shard x shifted down by `b`: bit b in bit 0.
__device__ __forceinline__ uint32_t shard_bit(const uint32_t (&x)[8], int q, uint32_t b) {
    return static_cast<uint32_t>(((static_cast<uint64_t>(x[2 * q + 1]) << 32) | x[2 * q]) >> b);
}

// The same test by shifts of 64-bit words, for four hashes and other F.
template <int F>
struct ShiftTest {
    uint32_t b[F][4];

    __device__ __forceinline__ void enter(int r, uint64_t h) {
        const uint32_t lo = static_cast<uint32_t>(h), hi = static_cast<uint32_t>(h >> 32);
        b[r % F][0] = lo & 63u;
        b[r % F][1] = (lo >> 16) & 63u;
        b[r % F][2] = hi & 63u;
        b[r % F][3] = (hi >> 16) & 63u;
    }
    __device__ __forceinline__ uint32_t missing(const uint32_t (&x)[8]) const {
        uint32_t present = 1u;
#pragma unroll
        for (int o = 0; o < F; ++o) {
#pragma unroll
            for (int q = 0; q < 4; ++q) present &= shard_bit(x, q, b[o][q]);
        }
        return ~present & 1u;
    }
    __device__ __forceinline__ void turn() {
        const ShiftTest old = *this;
#pragma unroll
        for (int i = 0; i < F; ++i) {
#pragma unroll
            for (int q = 0; q < 4; ++q) b[i][q] = old.b[(i + kTurn) % F][q];
        }
    }
};

// The same test from a ring of hashes, for H hashes or long rings.
template <int F, int H>
struct HashTest {
    uint64_t h[F];

    __device__ __forceinline__ void enter(int r, uint64_t v) { h[r % F] = v; }
    __device__ __forceinline__ uint32_t missing(const uint32_t (&x)[8]) const {
        uint32_t present = 1u;
#pragma unroll
        for (int o = 0; o < F; ++o) {
#pragma unroll
            for (int j = 0; j < H; ++j) present &= shard_bit(x, j & 3, bit_address<H>(h[o], j));
        }
        return ~present & 1u;
    }
    __device__ __forceinline__ void turn() {
        const HashTest old = *this;
#pragma unroll
        for (int i = 0; i < F; ++i) h[i] = old.h[(i + kTurn) % F];
    }
};

template <class C, int kKind = (C::F == 3 || C::F == 4) ? 0 : (C::H == 4 && C::F <= 8) ? 1 : 2>
struct FindereTest {
    using type = HashTest<C::F, C::H>;
};
template <class C>
struct FindereTest<C, 0> {
    using type = ByteTest<C::F, C::H>;
};
template <class C>
struct FindereTest<C, 1> {
    using type = ShiftTest<C::F>;
};

// The minimizer pass of a strip: lists its runs (one low hash word per run, of
// which kFew keeps the shard id) from shared address `list` on.  Returns the
// windows that start a run (x) and the words of the first and the last window
// (y, z).  A function of its own, so that its registers (two 64-bit arrays of
// W) do not add to the kernel's.
template <class C, bool kFew>
__device__ __noinline__ uint3 list_runs(uint32_t code_mem, uint32_t strip, uint32_t list,
                                        uint32_t shard_mask) {
    uint32_t c[C::kStripWords];
    load_code_words<C>(code_mem, strip, c);
    uint32_t at = list, chg = 1u, first = 0, prev = 0;
    for_each_min<C>(c, [&](int j, uint32_t lo) {
        if constexpr (kFew) lo &= shard_mask;
        if (j == 0) {
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(lo) : "memory");
            at += 128;
            first = lo;
        } else {
            run_list_put(lo, prev, 1u << j, at, chg);
        }
        prev = lo;
    });
    return make_uint3(chg, first, prev);
}

// The runs of a strip.  Windows with different low hash words seldom share a
// shard unless the filter has few; then every run is one more update or copy of
// the same 32 bytes, one after the other, so runs are told apart by shard id.
// 100 Mbp into one shard: 1.61 ms, by hash words 6.08 (17.2 with W = 5); into
// 16 shards 2.88, 3.08.  In larger filters the mask would cost an instruction
// a window (4 Mbp query 20.4 us against 19.9).  Small launches mask always: one
// pass fewer in the instruction cache (one gene 4.9 us, with both 5.5).
template <class C>
__device__ __forceinline__ uint3 strip_runs(uint32_t code_mem, uint32_t strip, uint32_t list,
                                            uint32_t shard_mask) {
    if (C::kStrip < 32 || shard_mask < 16u)
        return list_runs<C, true>(code_mem, strip, list, shard_mask);
    return list_runs<C, false>(code_mem, strip, list, shard_mask);
}

// Query of one strip: the minimizer pass lists the strip's runs, the runs that
// hold a valid window get consecutive slots of the warp's pool (a prefix sum
// over the lanes), the warp copies their shards there, and the test pass
// walks the windows with the current run's shard in registers.  Window 0's
// run reads the left lane's last slot, the one before the lane's own, when
// that lane's last run continues into the strip.  Lanes whose runs do not fit
// the pool any more wait for another round.
//
// Bound: the integer logic pipe (on <31,28,16,4> about 55 of its instructions
// per window, which alone take 4.5 of the 5.11 ms), then the latency of the
// shard copies.  1.51e9 positions of 10 M reads against 8 GiB: 5.11 ms, 29 G
// shards/s; with the copies issued by the thread that finds a run (two
// requests per shard), a copy slot per thread and shifts for the bit tests it
// was 7.82 ms at 19 G shards/s, the rate at which the memory takes two 16-byte
// requests each.  Loading the shards to registers instead keeps the L1 lines
// of all requests in flight and was slower the more shared memory the CTAs
// hold (6.8 ms at 150 KB an SM, 8.6 at 203 KB, before the CTAs had 128
// threads).
template <class C>
__device__ __forceinline__ uint32_t query_strip(uint32_t code_mem, uint32_t strip,
                                                uint32_t vmask, uint32_t shard_mask,
                                                const uint64_t* words, uint32_t run_mem) {
    constexpr int F = C::F;
    constexpr uint32_t kPoolSlots = query_pool_slots(C::W, C::H, C::F);
    static_assert(kPoolSlots * 32 >= 32 * 128, "the run lists fit the pool");
    const uint32_t lane = threadIdx.x & 31;
    uint32_t result = 0;
    while (__any_sync(0xFFFFFFFFu, vmask != 0u)) {
        const uint32_t list = run_mem + 4 * lane;
        const uint3 runs = strip_runs<C>(code_mem, strip, list, shard_mask);
        const uint32_t chg = runs.x, first = runs.y, prev = runs.z;
        // Run heads: a valid window whose predecessor is invalid or of another run.
        uint32_t heads = vmask & (chg | ~(vmask << 1));
        const int n = __popc(heads);
        // A lane lends its last slot when that holds window 31's run and the run
        // is not its window 0's, which may itself be borrowed.
        const bool lend = n > 0 && (vmask >> (C::kStrip - 1)) && !(n == 1 && (vmask & 1u));
        const uint32_t left_lo = __shfl_up_sync(0xFFFFFFFFu, prev, 1);
        const uint32_t lenders = __ballot_sync(0xFFFFFFFFu, lend);
        const bool borrow =
            lane > 0 && (heads & 1u) && (lenders >> (lane - 1) & 1u) && left_lo == first;
        const uint32_t own = n - (borrow ? 1 : 0);
        uint32_t end = own;
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, end, o);
            if (lane >= static_cast<uint32_t>(o)) end += v;
        }
        const uint32_t begin = end - own;
        // The lanes that fit are the first ones, so a lender fits if its borrower does.
        const bool fits = end <= kPoolSlots;
        if (!fits) heads = 0;
        // The shard ids of the lane's slots, from its list: a head's entry is the
        // number of runs that start up to it.
        const uint32_t ids = run_mem + 32 * kPoolSlots;
        uint32_t rest = borrow ? heads & (heads - 1u) : heads;
        list_shard_ids(rest, chg, list, ids + 4 * begin);
        __syncwarp();
        copy_shards(__reduce_max_sync(0xFFFFFFFFu, fits ? end : 0u), run_mem, ids, shard_mask,
                    words);
        uint32_t c[C::kStripWords];
        load_code_words<C>(code_mem, strip, c);
        typename FindereTest<C>::type test;
#pragma unroll
        for (int o = 0; o < F - 1; ++o) test.enter(o, smer_hash(smer_at<C>(c, o)));
        cp_async_wait_all();
        __syncwarp();
        uint32_t x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t at = run_mem + 32 * (borrow ? begin - 1 : begin);
        uint32_t missing = 0;
        // Turns of 16 windows, the code words moving down by one: half the
        // instructions of 32 unrolled windows, which ran out of the instruction
        // cache (10% of the stalls).
#pragma unroll 1
        for (int turn = 0; turn < C::kTurns; ++turn) {
            uint32_t m = 0;
#pragma unroll
            for (int j = 0; j < C::kTurn; ++j) {
                test.enter(j + F - 1, smer_hash(smer_at<C>(c, j + F - 1)));
                next_slot_if(heads & (1u << j), at, x);
                m += min(test.missing(x), 1u) << j;
            }
            if constexpr (C::kTurns == 1) {
                missing = m;
            } else {
                missing = (missing >> 16) | (m << 16);
                test.turn();
                heads >>= 16;
                next_turn_words<C>(c);
            }
        }
        if (fits) {
            result |= vmask & ~missing;
            vmask = 0;
        }
        __syncwarp();  // borrowed slots are read before another round's lists replace them
    }
    return result;
}

// Query of the thread's strip, in parts that fit the pool (Cfg::kPart): as a
// whole it took up to four rounds, each of which goes over the minimizers and
// the windows again.  100 Mbp in 2 MiB, windows of two m-mers (<31,28,30,4>):
// query 0.63 ms, in rounds 0.99; insert 0.77, 1.39.  Of one (<31,28,31,4>):
// insert 1.40, 1.96; query in 256 MiB 1.35, 1.57.  A filter of one shard has one
// run a strip, which parts would only cut up.
template <class C>
__device__ __forceinline__ uint32_t query_parts(uint32_t code_mem, uint32_t vmask,
                                                uint32_t shard_mask, const uint64_t* words,
                                                uint32_t run_mem) {
    if constexpr (C::kParts > 1) {
        if (shard_mask != 0u) {
            using Part = Cfg<C::K, C::S, C::M, C::H, C::kPart, C::kBits>;
            uint32_t result = 0;
#pragma unroll 1
            for (int i = 0; i < C::kParts; ++i)
                result |= query_strip<Part>(code_mem, threadIdx.x * C::kParts + i,
                                            (vmask >> (i * C::kPart)) & Part::kAll, shard_mask,
                                            words, run_mem)
                          << (i * C::kPart);
            return result;
        }
    }
    return query_strip<C>(code_mem, threadIdx.x, vmask, shard_mask, words, run_mem);
}

// Query of one strip without a pool: each run head loads its shard when it is
// reached.  For windows of less than 6 m-mers of at most 8 bases, whose runs
// are so short (a head every second window at W = 3) that a pool would take
// several rounds, and whose m-mers are so few that the shards stay in the
// caches: 100 M windows of <5,4,3,4> took 0.32 ms, two rounds through the pool
// 1.53.  For windows of one m-mer as well while the L2 holds the filter: 100 M
// windows of <31,28,31,4> take 0.75 ms up to 32 MiB (1.29 through the pool in
// parts), at 64 MiB 1.74 (1.26).
template <class C>
__device__ __forceinline__ uint32_t query_strip_direct(uint32_t code_mem, uint32_t strip,
                                                       uint32_t vmask, uint32_t shard_mask,
                                                       const uint64_t* words) {
    constexpr int F = C::F;
    uint32_t c[C::kStripWords];
    load_code_words<C>(code_mem, strip, c);
    typename FindereTest<C>::type test;
#pragma unroll
    for (int o = 0; o < F - 1; ++o) test.enter(o, smer_hash(smer_at<C>(c, o)));
    uint32_t x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint32_t cur = 0, missing = 0;
    bool have = false;
    for_each_shard<C>(c, shard_mask, [&](int j, uint32_t sh) {
        test.enter(j + F - 1, smer_hash(smer_at<C>(c, j + F - 1)));
        if (((vmask >> j) & 1u) && (!have || sh != cur)) {
            uint64_t w[4];
            load_shard(words + static_cast<uint64_t>(sh) * 4, w[0], w[1], w[2], w[3]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                x[2 * q] = static_cast<uint32_t>(w[q]);
                x[2 * q + 1] = static_cast<uint32_t>(w[q] >> 32);
            }
            cur = sh;
            have = true;
        }
        missing |= min(test.missing(x), 1u) << j;
    });
    return vmask & ~missing;
}

// ---------------------------------------------------------------------------
// Insert of one strip
// ---------------------------------------------------------------------------

// acc = a | b | c when `pred` is non-zero.
__device__ __forceinline__ void or3_if(uint32_t pred, uint32_t (&acc)[8], const uint32_t (&a)[8],
                                       const uint32_t (&b)[8], const uint32_t (&c)[8]) {
#pragma unroll
    for (int q = 0; q < 8; q += 4)
        asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %16, 0;\n\t"
            "@p lop3.b32 %0, %4, %8, %12, 0xFE;\n\t@p lop3.b32 %1, %5, %9, %13, 0xFE;\n\t"
            "@p lop3.b32 %2, %6, %10, %14, 0xFE;\n\t@p lop3.b32 %3, %7, %11, %15, 0xFE;\n\t}"
            : "+r"(acc[q]), "+r"(acc[q + 1]), "+r"(acc[q + 2]), "+r"(acc[q + 3])
            : "r"(a[q]), "r"(a[q + 1]), "r"(a[q + 2]), "r"(a[q + 3]), "r"(b[q]), "r"(b[q + 1]),
              "r"(b[q + 2]), "r"(b[q + 3]), "r"(c[q]), "r"(c[q + 1]), "r"(c[q + 2]),
              "r"(c[q + 3]), "r"(pred));
}

// Stores a run's masks at shared address `at` and moves on to the next slot
// (`at` becomes `next`) when `pred` is non-zero.
__device__ __forceinline__ void store_run_if(uint32_t pred, uint32_t& at, uint32_t& next,
                                             const uint32_t (&acc)[8]) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t"
        "@p st.shared.v4.u32 [%0], {%3, %4, %5, %6};\n\t"
        "@p st.shared.v4.u32 [%0+16], {%7, %8, %9, %10};\n\t"
        "@p mov.u32 %0, %1;\n\t@p add.u32 %1, %1, 32;\n\t}"
        : "+r"(at), "+r"(next)
        : "r"(pred), "r"(acc[0]), "r"(acc[1]), "r"(acc[2]), "r"(acc[3]), "r"(acc[4]), "r"(acc[5]),
          "r"(acc[6]), "r"(acc[7])
        : "memory");
}

// *dst |= *src, 32 bytes of shared memory.
__device__ __forceinline__ void or_slot(uint32_t dst, uint32_t src) {
#pragma unroll
    for (int q = 0; q < 32; q += 16)
        asm volatile(
            "{\n\t.reg .b32 a<4>, b<4>;\n\t"
            "ld.shared.v4.u32 {a0, a1, a2, a3}, [%0];\n\t"
            "ld.shared.v4.u32 {b0, b1, b2, b3}, [%1];\n\t"
            "or.b32 a0, a0, b0;\n\tor.b32 a1, a1, b1;\n\t"
            "or.b32 a2, a2, b2;\n\tor.b32 a3, a3, b3;\n\t"
            "st.shared.v4.u32 [%0], {a0, a1, a2, a3};\n\t}" ::"r"(dst + q),
            "r"(src + q)
            : "memory");
}

// ORs the slots below `total` into their shards, four lanes a slot with one
// 8-byte reduction each: the four make one 32-byte request.  (One 32-byte
// bulk reduction per slot takes 72 G slots/s from an L2-resident filter where
// this takes 120, and both 20 to 31 G/s from larger ones.  It also holds the
// slot until it is read.)
__device__ __forceinline__ void flush_pool(uint32_t total, uint32_t pool, uint32_t ids,
                                            uint32_t shard_mask, uint64_t* words) {
    const uint32_t lane = threadIdx.x & 31;
    uint64_t* word = words + (lane & 3u);
    uint32_t id = ids + 4 * (lane >> 2), src = pool + 8 * lane;
    for (uint32_t e = lane >> 2; __any_sync(0xFFFFFFFFu, e < total); e += 32) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            asm volatile(
                "{\n\t.reg .pred p;\n\t.reg .b32 s;\n\t.reg .b64 a, v;\n\t"
                "setp.lt.u32 p, %0, %1;\n\t"
                "@p ld.shared.u32 s, [%2];\n\t"
                "@p ld.shared.u64 v, [%5];\n\t"
                "@p and.b32 s, s, %3;\n\t"
                "@p mad.wide.u32 a, s, 32, %4;\n\t"
                "@p red.relaxed.gpu.global.or.b64 [a], v;\n\t}" ::"r"(e + 8 * u),
                "r"(total), "r"(id + 32 * u), "r"(shard_mask), "l"(word), "r"(src + 256 * u)
                : "memory");
        id += 128;
        src += 1024;
    }
}

// Insert of one strip.  The minimizer pass lists the strip's runs as in a
// query.  The mask pass then walks the windows: the mask of a run is the OR of
// the one-hot masks of all its windows' s-mers, kept in registers and stored
// to a pool slot at the run's last window.  A first run that continues the
// left lane's last one is ORed into that lane's slot.  At the end the warp
// flushes the slots.
//
// Bound: the memory's rate of random read-modify-writes for filters beyond L2
// (20 G shards/s at 8 GiB, 31 at 256 MiB; a genome's repeats raise that by
// what L2 holds of them), else the integer logic pipe.  3.1 Gbp into 8 GiB
// 15.8-16.3 ms (23 G runs/s) and 100 Mbp into 256 MiB 433 us (27 G runs/s); with
// each window issuing the flush of a run that ends there (a predicated 32-byte
// bulk reduction, strips flushing the runs between them twice) it was 21.1 ms
// and 688 us.
template <class C>
__device__ __forceinline__ void insert_strip_runs(uint32_t code_mem, uint32_t strip,
                                                  uint32_t vmask, uint32_t shard_mask,
                                                  uint64_t* words, uint32_t run_mem,
                                                  const uint64_t* onehot) {
    constexpr int F = C::F;
    constexpr uint32_t kPoolSlots = insert_pool_slots(C::W, C::H, C::F);
    static_assert(kPoolSlots * 32 >= 32 * 128, "the run lists fit the pool");
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t ids = run_mem + 32 * kPoolSlots;
    const uint32_t spare = ids + 4 * kPoolSlots + 32 * lane;
    while (__any_sync(0xFFFFFFFFu, vmask != 0u)) {
        const uint32_t list = run_mem + 4 * lane;
        const uint3 runs = strip_runs<C>(code_mem, strip, list, shard_mask);
        const uint32_t chg = runs.x;
        uint32_t heads = vmask & (chg | ~(vmask << 1));
        const int n = __popc(heads);
        const bool lend = n > 0 && (vmask >> (C::kStrip - 1)) && !(n == 1 && (vmask & 1u));
        const uint32_t left_lo = __shfl_up_sync(0xFFFFFFFFu, runs.z, 1);
        const uint32_t lenders = __ballot_sync(0xFFFFFFFFu, lend);
        bool merge =
            lane > 0 && (heads & 1u) && (lenders >> (lane - 1) & 1u) && left_lo == runs.y;
        const uint32_t own = n - (merge ? 1 : 0);
        uint32_t end = own;
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, end, o);
            if (lane >= static_cast<uint32_t>(o)) end += v;
        }
        const uint32_t begin = end - own;
        const bool fits = end <= kPoolSlots;
        // Windows that end a run: the next one is invalid or a head.
        uint32_t ends = vmask & ~((vmask & ~heads) >> 1);
        if (!fits) {
            heads = ends = 0;
            merge = false;
        }
        uint32_t rest = merge ? heads & (heads - 1u) : heads;
        for (uint32_t at = ids + 4 * begin; __any_sync(0xFFFFFFFFu, rest != 0u); at += 4) {
            const uint32_t b = rest & (0u - rest);
            rest ^= b;
            const uint32_t e = __popc(chg & (b ^ (b - 1u))) - 1;
            copy_u32_if(b, at, list + 128 * e);
        }
        __syncwarp();
        uint32_t c[C::kStripWords];
        load_code_words<C>(code_mem, strip, c);
        uint32_t ring[F][8];
        auto enter = [&](int r) {
            uint64_t m[4];
            smer_masks<C>(c, r, m, onehot);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ring[r % F][2 * q] = static_cast<uint32_t>(m[q]);
                ring[r % F][2 * q + 1] = static_cast<uint32_t>(m[q] >> 32);
            }
        };
#pragma unroll
        for (int o = 0; o < F - 1; ++o) enter(o);
        uint32_t acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t at = merge ? spare : run_mem + 32 * begin;
        uint32_t next = run_mem + 32 * (merge ? begin : begin + 1);
#pragma unroll 1
        for (int turn = 0; turn < C::kTurns; ++turn) {
#pragma unroll
            for (int j = 0; j < C::kTurn; ++j) {
                enter(j + F - 1);
                const uint32_t head = heads & (1u << j);
                if constexpr (F == 4) {
                    or3_if(head, acc, ring[j % F], ring[(j + 1) % F], ring[(j + 2) % F]);
                } else {
                    const uint32_t keep = head ? 0u : 0xFFFFFFFFu;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        uint32_t u = acc[q] & keep;
#pragma unroll
                        for (int o = 0; o < F - 1; ++o) u |= ring[(j + o) % F][q];
                        acc[q] = u;
                    }
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[q] |= ring[(j + F - 1) % F][q];
                store_run_if(ends & (1u << j), at, next, acc);
            }
            if constexpr (C::kTurns == 1) break;
            heads >>= kTurn;
            ends >>= kTurn;
            next_turn_words<C>(c);
            if constexpr (kTurn % F != 0) {
                uint32_t old[F][8];
#pragma unroll
                for (int i = 0; i < F; ++i) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) old[i][q] = ring[i][q];
                }
#pragma unroll
                for (int i = 0; i < F; ++i) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) ring[i][q] = old[(i + kTurn) % F][q];
                }
            }
        }
        __syncwarp();
        if (merge) or_slot(run_mem + 32 * (begin - 1), spare);
        __syncwarp();
        flush_pool(__reduce_max_sync(0xFFFFFFFFu, fits ? end : 0u), run_mem, ids, shard_mask,
                    words);
        __syncwarp();  // the slots are read before another round's lists replace them
        if (fits) vmask = 0;
    }
}

// Insert of the thread's strip, in parts as in a query.
template <class C>
__device__ __forceinline__ void insert_parts(uint32_t code_mem, uint32_t vmask,
                                             uint32_t shard_mask, uint64_t* words,
                                             uint32_t run_mem, const uint64_t* onehot) {
    if constexpr (C::kParts > 1) {
        if (shard_mask != 0u) {
            using Part = Cfg<C::K, C::S, C::M, C::H, C::kPart, C::kBits>;
#pragma unroll 1
            for (int i = 0; i < C::kParts; ++i)
                insert_strip_runs<Part>(code_mem, threadIdx.x * C::kParts + i,
                                        (vmask >> (i * C::kPart)) & Part::kAll, shard_mask, words,
                                        run_mem, onehot);
            return;
        }
    }
    insert_strip_runs<C>(code_mem, threadIdx.x, vmask, shard_mask, words, run_mem, onehot);
}

// ---------------------------------------------------------------------------
// The tile kernel
// ---------------------------------------------------------------------------

// Ragged launches: marks the record structure of the staged tile.  brk bit
// r of word q is set when tile position 32q + r starts a record (windows
// that contain it and the byte before it span two records); bytes outside
// every record are added to the invalid bits.  Each thread takes records
// first, first + kThreads, ... of those overlapping the tile.
template <class C>
__device__ __forceinline__ void mark_records(const TileParams& p, int64_t s0, uint32_t first,
                                             DevRange rec, uint32_t* inval, uint32_t* brk) {
    constexpr int64_t kSpan = C::kSpan;
    const int64_t len = static_cast<int64_t>(p.input_bytes);
    const int64_t t_end = s0 + kSpan;
    auto set_bits = [&](uint32_t* arr, int64_t a, int64_t b) {  // dense [a, b)
        a = a > s0 ? a : s0;
        b = b < t_end ? b : t_end;
        for (int64_t x = a; x < b;) {
            const int64_t pos = x - s0;
            const int q = static_cast<int>(pos >> 4), r = static_cast<int>(pos & 15);
            const int64_t n = (16 - r) < (b - x) ? (16 - r) : (b - x);
            atomicOr(arr + (q >> 1), ((1u << n) - 1u) << (r + 16 * (q & 1)));
            x += n;
        }
    };
    const uint64_t n = p.n_ranges;
    if (threadIdx.x == 0) {
        // Bytes before the first overlapping record.
        const int64_t gap0 = first == 0 ? 0
                                        : static_cast<int64_t>(p.ranges[first - 1].offset +
                                                               p.ranges[first - 1].bytes);
        const int64_t until = first < n ? static_cast<int64_t>(p.ranges[first].offset) : len;
        set_bits(inval, gap0, until);
    }
    for (uint64_t r = first + threadIdx.x; r < n; r += kThreads) {
        if (r >= first + kThreads) rec = p.ranges[r];
        const int64_t a = static_cast<int64_t>(rec.offset);
        if (a >= t_end) break;
        const int64_t b = a + static_cast<int64_t>(rec.bytes);
        if (a > s0 && a < t_end) {
            const int64_t pos = a - s0;
            atomicOr(brk + (pos >> 5), 1u << (pos & 31));
        }
        const int64_t next = r + 1 < n ? static_cast<int64_t>(p.ranges[r + 1].offset) : len;
        if (next > b) set_bits(inval, b, next);
    }
}

// Ragged launches: clears windows j of the strip that contain a record start
// other than their own first byte.  Bit r of `bits`: a record starts at base r.
template <class C>
__device__ __forceinline__ uint32_t strip_in_record(uint64_t bits, uint32_t vmask) {
    if constexpr (C::K > 1) {
        if (bits) vmask &= ~static_cast<uint32_t>(any_in_span<C::K - 1>(bits >> 1));
    }
    return vmask;
}

// Ragged launches with per-record tallies: adds the strip's valid windows
// (vmask) and positive windows (hits) to the records they belong to.  Window
// j belongs to the record containing byte x0 + j.  The strip's records are
// found by one binary search (first record ending after its first valid
// window, between the first records of the tile and of the next one: five
// dependent loads for reads, where all of 2 M records took 21 and a sixth of
// the query's time, 2.46 against 2.01 ms) and a walk over the record ends;
// empty records are skipped by the walk.  Across the warp, the record a strip
// starts in is usually the one the previous strip ended in: a strip's last
// record is handed to the next lane when it is that lane's first, and lanes
// holding the same record are summed
// with one match + reduce, so a warp issues about one atomic pair per record
// it touches (count_positive_kmers_per_record_kernel,
// detail/count_positive_kmers.cuh:21-45, fused into the query epilogue).
__device__ __forceinline__ void tally_records(const TileParams& p, uint32_t first, uint32_t last,
                                              int64_t x0, uint32_t vmask, uint32_t hits) {
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t n = p.n_ranges;
    uint32_t kf = kNone, vf = 0, kl = kNone, vl = 0;  // first / last record and (valid << 16 | pos)
    auto add = [&](uint32_t r, uint32_t c) {
        const uint64_t at = static_cast<uint64_t>(r) << p.rec_shift;
        atomicAdd(p.rec_valid + at, static_cast<unsigned long long>(c >> 16));
        if (c & 0xFFFFu) atomicAdd(p.rec_pos + at, static_cast<unsigned long long>(c & 0xFFFFu));
    };
    uint32_t v = vmask;
    const uint32_t h = hits & vmask;
    if (v) {
        int j = __ffs(v) - 1;
        // First record whose end exceeds x0 + j (records before `first` end
        // before the tile, and `last` ends after it).
        uint64_t lo = first, hi = last;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (static_cast<int64_t>(p.ranges[mid].offset + p.ranges[mid].bytes) > x0 + j)
                hi = mid;
            else
                lo = mid + 1;
        }
        uint64_t r = lo;
        for (bool head = true; r < n; head = false) {
            const int64_t lim = static_cast<int64_t>(p.ranges[r].offset + p.ranges[r].bytes) - x0;
            const uint32_t seg = lim >= 32 ? v : (v & ((1u << lim) - 1u));
            const uint32_t c = (static_cast<uint32_t>(__popc(seg)) << 16) |
                               static_cast<uint32_t>(__popc(h & seg));
            v &= ~seg;
            if (head) {
                kf = static_cast<uint32_t>(r);
                vf = c;
            } else if (v) {
                add(static_cast<uint32_t>(r), c);  // a record inside the strip
            } else {
                kl = static_cast<uint32_t>(r);
                vl = c;
            }
            if (!v) break;
            j = __ffs(v) - 1;
            do {
                ++r;
            } while (r < n && static_cast<int64_t>(p.ranges[r].offset + p.ranges[r].bytes) <= x0 + j);
        }
    }
    const uint32_t prev_kl = __shfl_up_sync(0xFFFFFFFFu, kl, 1);
    const uint32_t prev_vl = __shfl_up_sync(0xFFFFFFFFu, vl, 1);
    const uint32_t next_kf = __shfl_down_sync(0xFFFFFFFFu, kf, 1);
    if (lane > 0 && prev_kl != kNone && prev_kl == kf) vf += prev_vl;
    if (kl != kNone && !(lane < 31 && next_kf == kl)) add(kl, vl);
    const uint32_t grp = __match_any_sync(0xFFFFFFFFu, kf);
    const uint32_t tot = __reduce_add_sync(grp, vf);
    if (kf != kNone && lane == static_cast<uint32_t>(__ffs(grp) - 1)) add(kf, tot);
}

// The tile kernel.  A plain launch has a CTA per tile; a smaller grid's CTAs
// walk tiles blockIdx.x + i * gridDim.x, each with the next tile's copy in
// flight.  Six CTAs of 128 threads an SM, with the tiles handed out by the
// hardware, keep all 24 warps busy to the end and cost little at the barriers.
// A persistent grid was slower: its CTAs share an SM's issue slots unevenly,
// so that some finish early and leave 18.5 warps on average (100 Mbp insert
// 488 us against 433, 10 M reads 5.95 ms against 5.12; with a CTA per tile of
// 256 threads 452 and 5.38, of 64 threads 453 and 5.32).
template <class C, bool kQuery, bool kDense, bool kRagged>
__global__ void __launch_bounds__(kThreads, (kQuery ? query_warps(C::W, C::H, C::F)
                                                    : insert_warps(C::W, C::H, C::F)) *
                                                   32 / kThreads)
    tile_kernel(TileParams p) {
    constexpr int kCodeWords = C::kCodeWords;
    __shared__ alignas(128) uint8_t stage[C::kStageBytes];
    __shared__ alignas(8) uint32_t code[kCodeWords + 4];
    // One bit per position: invalid bases, record starts.
    __shared__ alignas(8) uint32_t inval[C::kSpan / 32 + 2];
    __shared__ alignas(8) uint32_t brk[kRagged ? C::kSpan / 32 + 2 : 1];
    __shared__ bool covered;  // the staged tile needs no plain loads
    __shared__ alignas(8) uint64_t bar;
    __shared__ uint64_t onehot[kQuery ? 1 : 64];
    // Dynamic shared memory, a part per warp: the pools of query_strip and
    // insert_strip_runs.
    extern __shared__ __align__(16) uint64_t slots[];

    const int tid = threadIdx.x;
    if constexpr (!kQuery) onehot_init(onehot);
    if constexpr (kRagged) {
        if (p.sizes) {
            const DevSizes z = *p.sizes;
            p.input_bytes = z.input_bytes;
            p.n_kmers = z.n_kmers;
            p.n_tiles = z.n_tiles;
            p.n_ranges = z.n_ranges;
        }
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
        if (blockIdx.x < p.n_tiles) covered = issue_stage<C, kDense>(p, blockIdx.x, stage, &bar);
    }
    __syncthreads();
    unsigned long long n_valid = 0, n_pos = 0;
    const uint32_t origin = stage_origin<C, kDense>(p);
    uint32_t parity = 0;
    for (uint32_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x, parity ^= 1u) {
        uint32_t first_rec = 0;
        DevRange rec{0, 0};  // the thread's first record of the tile
        if constexpr (kRagged) {
            first_rec = p.tile_rec[tile];
            if (first_rec + tid < p.n_ranges) rec = p.ranges[first_rec + tid];
        }
        const bool ok = mbar_wait_bounded(&bar, parity);
        // (Also the barrier behind the last tile's reads of the code words.)
        if (__syncthreads_or(!ok)) {
            // The copy that ran out of time may still be in flight: give it
            // one more bounded wait before the CTA's shared memory is
            // released, so that it does not land in memory a later CTA owns.
            if (tid == 0) {
                atomicExch(p.err, kDevErrStageTimeout);
                (void)mbar_wait_bounded(&bar, parity);
            }
            __syncthreads();
            return;
        }
        if (!covered) {
            fill_ragged<kDense>(p, tile_geom<C, kDense>(p, tile), stage);
            __syncthreads();
        }
        if constexpr (C::kBits != 2) {
            static_assert(!kDense || C::kBits == 2, "dense proteins run the generic kernels");
            for (int t = tid; t <= kThreads; t += kThreads) {
                encode_protein_strip(origin, stage, t, code, inval);
                if constexpr (kRagged) brk[t] = 0u;
            }
        }
        for (int q = tid; C::kBits == 2 && q < kCodeWords; q += kThreads) {
            uint32_t cw, iv;
            encode_word<kDense>(origin, stage, q, cw, iv);
            code[q] = cw;
            reinterpret_cast<uint16_t*>(inval)[q] = static_cast<uint16_t>(iv);
            if constexpr (kRagged) reinterpret_cast<uint16_t*>(brk)[q] = 0;
        }
        if constexpr (kRagged) {
            __syncthreads();
            mark_records<C>(p, tile_first_symbol<C>(p, tile), first_rec, rec, inval, brk);
        }
        __syncthreads();
        // In a limited grid the CTA's next tile lands while this one is hashed.
        if (tid == 0 && tile + gridDim.x < p.n_tiles)
            covered = issue_stage<C, kDense>(p, tile + gridDim.x, stage, &bar);

        auto strip_bits = [&](const uint32_t* a) {
            const uint32_t* w = a + (tid * C::kStrip) / 32;
            if constexpr (C::kStrip == 32) {
                return static_cast<uint64_t>(w[0]) | (static_cast<uint64_t>(w[1]) << 32);
            } else {
                const uint32_t sh = (tid * C::kStrip) & 31;
                return static_cast<uint64_t>(__funnelshift_r(w[0], w[1], sh)) |
                       (static_cast<uint64_t>(__funnelshift_r(w[1], w[2], sh)) << 32);
            }
        };
        // (Made again after the passes over the strip: a live copy spilled.)
        auto first_window = [&] {
            return tile_first_symbol<C>(p, tile) + static_cast<int64_t>(tid) * C::kStrip;
        };
        uint32_t vmask = strip_valid<C>(strip_bits(inval), first_window(), p.n_kmers);
        if constexpr (kRagged) {
            vmask = strip_in_record<C>(strip_bits(brk), vmask);
            n_valid += __popc(vmask);
        }
        uint32_t hits = 0;
        const uint32_t code_mem = smem_addr(code);
        if constexpr (kQuery) {
            if constexpr (C::W < 6 && C::M * C::kBits <= 16) {
                hits = query_strip_direct<C>(code_mem, tid, vmask, p.shard_mask, p.words);
            } else if (C::W == 1 && p.shard_mask < (32u << 20) / 32) {
                hits = query_strip_direct<C>(code_mem, tid, vmask, p.shard_mask, p.words);
            } else {
                constexpr int kWarpBytes = query_warp_bytes(C::W, C::H, C::F);
                hits = query_parts<C>(code_mem, vmask, p.shard_mask, p.words,
                                      smem_addr(slots) + (tid >> 5) * kWarpBytes);
            }
            const int64_t first_kmer = first_window();
            if (p.out) store_strip_bytes<C>(hits, p.out, first_kmer, p.n_kmers);
            if constexpr (kRagged) n_pos += __popc(hits & vmask);
            if (p.out_bits) store_strip_bits<C>(hits, p.out_bits, first_kmer, p.n_kmers);
        } else {
            constexpr int kWarpBytes = insert_warp_bytes(C::W, C::H, C::F);
            insert_parts<C>(code_mem, vmask, p.shard_mask, p.words,
                            smem_addr(slots) + (tid >> 5) * kWarpBytes, onehot);
        }
        if constexpr (kRagged) {
            if (p.rec_valid) {
                const uint32_t last = tile + 1 < p.n_tiles ? p.tile_rec[tile + 1]
                                                           : static_cast<uint32_t>(p.n_ranges);
                tally_records(p, p.tile_rec[tile], last, first_window(), vmask, hits);
            }
        }
    }
    if constexpr (kRagged) {
        // A warp sees at most 2^31 windows of a launch.
        const uint32_t valid = __reduce_add_sync(0xFFFFFFFFu, static_cast<uint32_t>(n_valid));
        const uint32_t pos = __reduce_add_sync(0xFFFFFFFFu, static_cast<uint32_t>(n_pos));
        __shared__ uint32_t tally[kThreads / 32][2];
        if ((tid & 31) == 0) {
            tally[tid >> 5][0] = valid;
            tally[tid >> 5][1] = pos;
        }
        __syncthreads();
        if (tid < 2) {
            unsigned long long sum = 0;
#pragma unroll
            for (int w = 0; w < kThreads / 32; ++w) sum += tally[w][tid];
            if (sum) atomicAdd(p.counts + tid, sum);
        }
    }
}

}  // namespace sbf
