// Zstd entropy stage on the GPU: one Zstd frame per 64 KiB window, built from
// the window's ZSTD_Sequence records, decodable by any conforming decoder
// (stock libzstd).
//
// Frame layout (RFC 8878): magic, a single-segment frame header with the
// content size, and one block.  The block is a compressed block when that is
// smaller than the window, else a raw block.  A compressed block holds
//   - the window's literal bytes, in order, as the smallest of a raw, an RLE
//     or a Huffman-coded literals block;
//   - a sequences section whose literal lengths, offsets and match lengths have
//     a table each (RLE, FSE-compressed or predefined, the cheapest by estimate)
//     and whose bitstream is written by an FSE (tANS) encoder derived from the
//     decoder's state tables: for symbol s and the decoder state D' that
//     follows, the encoder picks the state D of s with
//     baseline(D) <= D' < baseline(D) + 2^nbBits(D) and writes D' - baseline(D).
// Offsets use the format's repeat codes whenever the actual offset equals one
// of the three repeat offsets the decoder holds at that point.
//
// Kernels, per window:
//   zenc_literals_kernel   (one CTA):    window staged by bulk copy, literal
//                                        gather, raw literal section, histogram
//   zenc_huf_plan_kernel   (one warp):   Huffman code and tree description
//   zenc_huf_write_kernel  (one CTA):    RLE or Huffman-coded literal section
//                                        where that is smaller
//   zenc_sequences_kernel  (one CTA):    repeat-code pass, FSE chains, bitstream,
//                                        block header, frame size
//   zenc_compact_kernel    (one CTA):    frames back to back at scanned offsets
// Frames are built in per-window slots of kZencSlot bytes first, because a
// frame's size is known only once its bitstream is written.
#include "gcz_common.cuh"
#include "gcz_kernels.h"

namespace gcz {
namespace {

constexpr uint32_t kErrBadSequences = 4;  // status bit: sequences do not describe their window
constexpr uint32_t kLitThreads = 512;

// Predefined distributions (RFC 8878 3.1.1.3.2.2); -1 = "less than 1".
__constant__ int8_t kLLNorm[36] = {4, 3, 2, 2, 2, 2, 2, 2, 2, 2, 2, 2, 2, 1, 1, 1, 2, 2,
                                   2, 2, 2, 2, 2, 2, 2, 3, 2, 1, 1, 1, 1, 1, -1, -1, -1, -1};
__constant__ int8_t kMLNorm[53] = {1, 4, 3, 2, 2, 2, 2, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1, 1,
                                   1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
                                   1, 1, 1, 1, 1, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1, -1, -1};
__constant__ int8_t kOFNorm[29] = {1, 1, 1, 1, 1, 1, 2, 2, 2, 1, 1, 1, 1, 1, 1,
                                   1, 1, 1, 1, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1};
constexpr uint32_t kLLLog = 6, kMLLog = 6, kOFLog = 5;
constexpr uint32_t kLLSyms = 36, kMLSyms = 53, kOFSyms = 29;

__device__ __forceinline__ uint32_t highbit(uint32_t x) { return 31u - static_cast<uint32_t>(__clz(x)); }

// Codes and extra-bit counts of the small values in shared memory (lanes of a
// warp look up different ones); above those, codes follow the highest set bit.
// Every code's baseline (less 3 for match lengths) is a multiple of 2^(its
// extra bits), so the extra bits are the value's low bits.
struct CodeTables {
    uint16_t ll_lut[64];   // literal length v < 64: code | extra bits << 8
    uint16_t ml_lut[128];  // match length v + 3, v < 128
    __device__ void build() {
        for (uint32_t v = threadIdx.x; v < 128u; v += blockDim.x) {
            uint32_t c, b;
            if (v < 64u) {
                if (v < 16u) c = v, b = 0u;
                else if (v < 24u) c = 16u + ((v - 16u) >> 1), b = 1u;
                else if (v < 32u) c = 20u + ((v - 24u) >> 2), b = 2u;
                else if (v < 48u) c = 22u + ((v - 32u) >> 3), b = 3u;
                else c = 24u, b = 4u;
                ll_lut[v] = static_cast<uint16_t>(c | (b << 8));
            }
            if (v < 32u) c = v, b = 0u;
            else if (v < 40u) c = 32u + ((v - 32u) >> 1), b = 1u;
            else if (v < 48u) c = 36u + ((v - 40u) >> 2), b = 2u;
            else if (v < 64u) c = 38u + ((v - 48u) >> 3), b = 3u;
            else if (v < 96u) c = 40u + ((v - 64u) >> 4), b = 4u;
            else c = 42u, b = 5u;
            ml_lut[v] = static_cast<uint16_t>(c | (b << 8));
        }
    }
    // Literal lengths >= 64 take code 19 + highbit (64 -> 25, ..., 65536 -> 35) with highbit extra bits.
    __device__ __forceinline__ void ll(uint32_t v, uint32_t &code, uint32_t &bits) const {
        const uint32_t e = v < 64u ? ll_lut[v] : 0u, hb = highbit(v | 1u);
        code = v < 64u ? e & 0xFFu : hb + 19u;
        bits = v < 64u ? e >> 8 : hb;
    }
    // Match lengths >= 131 take code 36 + highbit(ml - 3) (131 -> 43, ..., 65539 -> 52) likewise.
    __device__ __forceinline__ void ml(uint32_t m, uint32_t &code, uint32_t &bits) const {
        const uint32_t v = m - 3u, e = v < 128u ? ml_lut[v] : 0u, hb = highbit(v | 1u);
        code = v < 128u ? e & 0xFFu : hb + 36u;
        bits = v < 128u ? e >> 8 : hb;
    }
    // Extra bits by code.
    __device__ __forceinline__ uint32_t ll_bits(uint32_t c) const {
        return c >= 25u ? c - 19u : (c < 16u ? 0u : static_cast<uint32_t>(0x433221111ull >> (4u * (c - 16u))) & 0xFu);
    }
    __device__ __forceinline__ uint32_t ml_bits(uint32_t c) const {
        return c >= 43u ? c - 36u : (c < 32u ? 0u : static_cast<uint32_t>(0x54433221111ull >> (4u * (c - 32u))) & 0xFu);
    }
};

struct ZencArgs {
    const uint8_t *src;
    uint64_t n;
    uint32_t window;
    uint32_t num_windows;
    const uint4 *seqs;         // ZSTD_Sequence records {offset, litLength, matchLength, rep}
    const uint64_t *seq_offsets;  // num_windows + 1
    uint8_t *slots;            // kZencSlot bytes per window
    uint32_t *ovs;             // kZencMaxSeqs per window
    uint32_t *sec_off;         // start of the sequences section in the slot (0 = raw frame)
    uint32_t *fsize;           // frame bytes
    uint8_t *raw;              // 1 = raw block
    uint32_t *hist;            // 256 literal-byte counts per window
    uint8_t *plan;             // kZencPlanBytes per window
    uint32_t *status;
    const WinDesc *wins;       // optional window table (null: windows at b * window)
};

__device__ __forceinline__ uint32_t win_size(const ZencArgs &a, uint32_t b) {
    if (a.wins) return a.wins[b].size;
    const uint64_t s = static_cast<uint64_t>(b) * a.window;
    return static_cast<uint32_t>(a.n - s < a.window ? a.n - s : a.window);
}
// First byte of window b: at b * window, or where the window table puts it.
__device__ __forceinline__ const uint8_t *win_src(const ZencArgs &a, uint32_t b) {
    return a.src + (a.wins ? a.wins[b].offset : static_cast<uint64_t>(b) * a.window);
}
__device__ __forceinline__ uint32_t frame_header_bytes(uint32_t w) { return 4u + 1u + (w < 256u ? 1u : 2u); }

__device__ void write_frame_header(uint8_t *p, uint32_t w) {
    p[0] = 0x28;
    p[1] = 0xB5;
    p[2] = 0x2F;
    p[3] = 0xFD;
    if (w < 256u) {
        p[4] = 0x20;  // Single_Segment, 1-byte Frame_Content_Size
        p[5] = static_cast<uint8_t>(w);
    } else {
        p[4] = 0x60;  // Single_Segment, 2-byte Frame_Content_Size (value - 256)
        p[5] = static_cast<uint8_t>(w - 256u);
        p[6] = static_cast<uint8_t>((w - 256u) >> 8);
    }
}

__device__ __forceinline__ void write_block_header(uint8_t *p, uint32_t type, uint32_t size) {
    const uint32_t h = 1u | (type << 1) | (size << 3);  // Last_Block set: one block per frame
    p[0] = static_cast<uint8_t>(h);
    p[1] = static_cast<uint8_t>(h >> 8);
    p[2] = static_cast<uint8_t>(h >> 16);
}

// 4 bytes at p (any alignment) from global memory: the aligned words that
// hold them, funnel-shifted; the second word is read only when p is unaligned,
// so no word without a wanted byte is touched.
__device__ __forceinline__ uint32_t load4(const uint8_t *p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~static_cast<uintptr_t>(3));
    const uint32_t sh = static_cast<uint32_t>(a & 3u) * 8u;
    const uint32_t lo = __ldg(w);
    return sh ? __funnelshift_r(lo, __ldg(w + 1), sh) : lo;
}

// The CTA copies n bytes from s to d (any alignments): aligned 16-byte stores
// for d, byte stores at its two ends.  The 16 bytes of a store come from the two
// aligned 16-byte blocks of s that hold them (one when s and d are aligned
// alike), so no block is read that holds none of them.
// Bound by memory: 0.22 GB for 3072 windows; with 4-byte stores 4096 windows
// took 104 us, with these 61 (0.3 GB, 4.9 TB/s).
__device__ void cta_copy(uint8_t *d, const uint8_t *s, uint32_t n) {
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    const uint32_t head = min(n, (16u - static_cast<uint32_t>(reinterpret_cast<uintptr_t>(d) & 15u)) & 15u);
    if (tid < head) d[tid] = s[tid];
    const uint32_t nv = (n - head) >> 4;
    uint4 *dv = reinterpret_cast<uint4 *>(d + head);
    const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(s + head) & 15u), sh = 8u * (off & 3u);
    const uint4 *sv = reinterpret_cast<const uint4 *>(s + head - off);
    for (uint32_t k = tid; k < nv; k += nt) {
        const uint4 x = __ldg(sv + k), y = off != 0u ? __ldg(sv + k + 1u) : x;
        uint32_t w[7] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z};
        const uint32_t last = y.w;
        if (off & 8u) {
#pragma unroll
            for (int i = 0; i < 5; i++) w[i] = w[i + 2];
            w[5] = last;
        }
        if (off & 4u) {
#pragma unroll
            for (int i = 0; i < 5; i++) w[i] = w[i + 1];
        }
        dv[k] = make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh),
                           __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
    }
    for (uint32_t k = head + 16u * nv + tid; k < n; k += nt) d[k] = s[k];
}

// ---------------------------------------------------------------- literals
// The literal section is the smallest of: raw; RLE (one distinct byte);
// Huffman-coded (RFC 8878 4.2), one stream below 1024 literals, else four.
// The Huffman code: two-queue construction over the present bytes (leaves
// sorted by count, then byte value; a leaf wins ties), lengths limited to 11
// bits by moving pairs of leaves up the tree (which keeps the code complete),
// the longest codes to the least frequent bytes, canonical code values (the
// longest codes take the smallest values, ties by byte value).  Weights are
// sent directly when there are at most 128 of them, else FSE-compressed with
// accuracy 6: counts normalised by floor(c * 64 / N) (at least 1), the
// largest absorbing the remainder; two interleaved states; the state of the
// second-to-last weight is chosen with at least one update bit, so that the
// decoder's last update runs past the stream start and decoding ends there.
//
// Three kernels: zenc_literals_kernel gathers each window's literals, writes
// the raw literal section (the default) and the byte histogram;
// zenc_huf_plan_kernel builds the code of a window in one warp (many windows
// per SM, so the serial steps of one overlap the others');
// zenc_huf_write_kernel rewrites the section as RLE or Huffman-coded where
// that is smaller.
constexpr uint32_t kHufMaxBits = 11;

// Per-window record from the plan to the write kernel.
struct PlanRec {
    uint8_t len[256];
    uint16_t code[256];
    uint8_t tree[132];  // Huffman_Tree_Description
    uint32_t tree_bytes;
    uint32_t mode;  // 0: keep raw, 1: RLE, 2: Huffman candidate
    uint32_t nlit;
    uint32_t rle;
};
static_assert(sizeof(PlanRec) <= kZencPlanBytes, "plan record");

__device__ __forceinline__ uint32_t raw_lit_header_bytes(uint32_t nlit) {
    return nlit < 32u ? 1u : (nlit < 4096u ? 2u : 3u);
}
__device__ void write_raw_lit_header(uint8_t *h, uint32_t type, uint32_t nlit) {
    const uint32_t hb = raw_lit_header_bytes(nlit);
    if (hb == 1u) {
        h[0] = static_cast<uint8_t>(type | (nlit << 3));
    } else if (hb == 2u) {
        h[0] = static_cast<uint8_t>(type | (1u << 2) | ((nlit << 4) & 0xF0u));
        h[1] = static_cast<uint8_t>(nlit >> 4);
    } else {
        h[0] = static_cast<uint8_t>(type | (3u << 2) | ((nlit << 4) & 0xF0u));
        h[1] = static_cast<uint8_t>(nlit >> 4);
        h[2] = static_cast<uint8_t>(nlit >> 12);
    }
}

// Gathers the literals of each window (one CTA per window), validates the
// sequences, writes frame header + raw literal section into the slot and the
// histogram of the literal bytes.  The window is staged into shared memory
// with 1-D bulk copies and its literals are moved together in place: every
// match toggles a bit at its start and its end, a prefix XOR gives the bytes
// inside matches, a prefix sum of the others each one's place (never behind
// its own), and every thread reads its 8 x 16 bytes before any is written.
// Work is even over the threads whatever the runs' lengths.
//
// What bounds it: latency, two CTAs of 16 warps per SM.  Copying run by run
// from the staged window to a second buffer, one CTA per SM with 64 KiB of
// histograms, took 583 us for 4096 windows and 31 us for 17; this form takes
// 265 and 15 us.
constexpr uint32_t kGatherThreads = 512;
constexpr uint32_t kHistCopies = 16;  // spread the lanes that count the same byte at once

struct GatherSmem {
    uint8_t win[kMaxWindow + 64];          // staged window, then its literals
    uint32_t mask[kMaxWindow / 32 + 1];    // toggles, then one bit per literal byte
    uint16_t before[kMaxWindow / 32];      // literals before each 32-byte word of the window
    uint32_t hist[256 * kHistCopies];      // copies of a count next to each other, in different banks
    uint32_t warp_ll[kGatherThreads / 32], warp_pos[kGatherThreads / 32];
    uint32_t bad, flags;
    alignas(8) uint64_t bar;
};

__global__ void __launch_bounds__(kGatherThreads, 2) zenc_literals_kernel(ZencArgs a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    GatherSmem &S = *reinterpret_cast<GatherSmem *>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5, lt = lanemask_lt();
    uint32_t parity = 0;
    if (tid == 0) {
        mbar_init(&S.bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    for (uint32_t b = blockIdx.x; b < a.num_windows; b += gridDim.x) {
        const uint32_t w = win_size(a, b);
        const uint8_t *src = win_src(a, b);
        const uint64_t s0 = a.seq_offsets[b];
        const uint32_t ns = static_cast<uint32_t>(a.seq_offsets[b + 1] - s0);
        const uint4 *sq = a.seqs + s0;
        uint8_t *slot = a.slots + static_cast<uint64_t>(b) * kZencSlot;
        PlanRec *plan = reinterpret_cast<PlanRec *>(a.plan + static_cast<uint64_t>(b) * kZencPlanBytes);
        const uint32_t fh = frame_header_bytes(w);
        if (ns == 0u) {  // no sequences: the raw block is smaller
            if (tid == 0) {
                write_frame_header(slot, w);
                a.sec_off[b] = 0u;
                plan->nlit = 0u;
            }
            continue;
        }
        if (tid == 0) {
            S.bad = ns > kZencMaxSeqs ? 1u : 0u;
            S.flags = 0u;
        }
        for (uint32_t k = tid; k < 256u * kHistCopies; k += kGatherThreads) S.hist[k] = 0u;
        for (uint32_t k = tid; k <= kMaxWindow / 32; k += kGatherThreads) S.mask[k] = 0u;
        __syncthreads();
        if (wid == 0 && !stage_window(S.win, src, w, &S.bar, parity, a.status) && lane == 0) S.flags = 1u;
        // Each warp owns a contiguous, equal share of the sequences: first the
        // warps' totals, then each sequence's source position by a scan.
        constexpr uint32_t kW32 = kGatherThreads / 32;
        const uint32_t per = (ns + kW32 - 1) / kW32;
        const uint32_t i0 = min(wid * per, ns), i1 = min(i0 + per, ns);
        uint32_t sll = 0, spos = 0;
        for (uint32_t i = i0 + lane; i < i1; i += 32u) {
            const uint4 q = sq[i];
            // lengths bounded by the window, so the sums below cannot wrap
            if (q.x == 0u || q.y > kMaxWindow || q.z < 3u || q.z > kMaxWindow) S.bad = 1u;
            sll += q.y;
            spos += q.y + q.z;
        }
        sll = __reduce_add_sync(kFull, sll);
        spos = __reduce_add_sync(kFull, spos);
        if (lane == 0) {
            S.warp_ll[wid] = sll;
            S.warp_pos[wid] = spos;
        }
        __syncthreads();
        if (S.flags) return;  // the bulk copy never completed: status recorded, every thread leaves
        uint32_t p = 0, TLL = 0, TP = 0;
        for (uint32_t k = 0; k < kW32; ++k) {
            if (k < wid) p += S.warp_pos[k];
            TLL += S.warp_ll[k];
            TP += S.warp_pos[k];
        }
        if (!(TP > w || S.bad)) {  // (S.bad may still be set below; every position stays in the window)
            for (uint32_t ib = i0; ib < i1; ib += 32u) {
                const uint32_t i = ib + lane;
                uint4 q = make_uint4(0u, 0u, 0u, 0u);
                if (i < i1) q = sq[i];
                uint32_t xp = q.y + q.z;  // inclusive scan over the batch
#pragma unroll
                for (uint32_t o = 1; o < 32; o <<= 1) {
                    const uint32_t yp = __shfl_up_sync(kFull, xp, o);
                    if (lane >= o) xp += yp;
                }
                const uint32_t end = p + xp, start = end - q.z;
                if (i < i1) {
                    if (q.x > start) S.bad = 1u;  // match would reach before the window start
                    atomicXor(&S.mask[start >> 5], 1u << (start & 31u));
                    atomicXor(&S.mask[end >> 5], 1u << (end & 31u));
                }
                p += __shfl_sync(kFull, xp, 31);
            }
        } else if (tid == 0) {
            S.bad = 1u;
        }
        __syncthreads();
        if (S.bad) {
            if (tid == 0) {
                atomicOr(a.status, kErrBadSequences);
                write_frame_header(slot, w);
                a.sec_off[b] = 0;  // raw frame
                plan->nlit = 0u;
            }
            __syncthreads();
            continue;
        }
        // toggles -> literal bits, four words per thread
        constexpr uint32_t kWords = kMaxWindow / 32 / kGatherThreads;
        uint32_t m[kWords], odd = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWords; ++k) {
            uint32_t x = S.mask[tid * kWords + k];
#pragma unroll
            for (uint32_t d = 1; d < 32u; d <<= 1) x ^= x << d;
            m[k] = odd ? ~x : x;  // inside a match, counted from this thread's first word
            odd = m[k] >> 31;
        }
        const uint32_t odds = __ballot_sync(kFull, odd != 0u);
        uint32_t flip = static_cast<uint32_t>(__popc(odds & lt)) & 1u;
        if (lane == 0) S.warp_pos[wid] = static_cast<uint32_t>(__popc(odds)) & 1u;
        __syncthreads();
        for (uint32_t k = 0; k < wid; ++k) flip ^= S.warp_pos[k];
        uint32_t cnt = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWords; ++k) {
            const uint32_t q = (tid * kWords + k) * 32u;
            const uint32_t in = q + 32u <= w ? ~0u : (q < w ? (1u << (w - q)) - 1u : 0u);
            m[k] = (flip ? m[k] : ~m[k]) & in;
            cnt += static_cast<uint32_t>(__popc(m[k]));
        }
        uint32_t x = cnt;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31u) S.warp_ll[wid] = x;
        __syncthreads();
        x -= cnt;
        for (uint32_t k = 0; k < wid; ++k) x += S.warp_ll[k];
#pragma unroll
        for (uint32_t k = 0; k < kWords; ++k) {
            S.mask[tid * kWords + k] = m[k];
            S.before[tid * kWords + k] = static_cast<uint16_t>(x);
            x += static_cast<uint32_t>(__popc(m[k]));
        }
        constexpr uint32_t kTiles = kMaxWindow / (16 * kGatherThreads);
        uint4 v[kTiles];
#pragma unroll
        for (uint32_t t = 0; t < kTiles; ++t) v[t] = reinterpret_cast<const uint4 *>(S.win)[t * kGatherThreads + tid];
        __syncthreads();
        const uint32_t copy = lane & (kHistCopies - 1u);
#pragma unroll
        for (uint32_t t = 0; t < kTiles; ++t) {
            const uint32_t word = (t * kGatherThreads + tid) >> 1, mw = S.mask[word];
            const uint32_t m16 = (tid & 1u) ? mw >> 16 : mw & 0xFFFFu;
            if (m16 == 0u) continue;
            uint32_t d = S.before[word] + ((tid & 1u) ? static_cast<uint32_t>(__popc(mw & 0xFFFFu)) : 0u);
#pragma unroll
            for (uint32_t k = 0; k < 16u; ++k) {
                const uint32_t y = k < 4u ? v[t].x : (k < 8u ? v[t].y : (k < 12u ? v[t].z : v[t].w));
                const uint32_t c = (y >> (8u * (k & 3u))) & 0xFFu;
                if ((m16 >> k) & 1u) {
                    S.win[d++] = static_cast<uint8_t>(c);
                    atomicAdd(&S.hist[c * kHistCopies + copy], 1u);
                }
            }
        }
        __syncthreads();
        const uint32_t nlit = TLL + (w - TP);
        const uint32_t rh = raw_lit_header_bytes(nlit);
        // the raw section: whole aligned words of the slot, single bytes at its ends
        uint8_t *dst = slot + fh + 3u + rh;
        const uint32_t head = min(nlit, (4u - static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst) & 3u)) & 3u);
        const uint32_t nw = (nlit - head) >> 2;
        if (tid < head) dst[tid] = S.win[tid];
        const uint32_t *lw = reinterpret_cast<const uint32_t *>(S.win);
        uint32_t *dw = reinterpret_cast<uint32_t *>(dst + head);
        for (uint32_t k = tid; k < nw; k += kGatherThreads) dw[k] = __funnelshift_r(lw[k], lw[k + 1u], 8u * head);
        if (tid < nlit - head - 4u * nw) dst[head + 4u * nw + tid] = S.win[head + 4u * nw + tid];
        if (tid == 0) {
            write_frame_header(slot, w);
            write_raw_lit_header(slot + fh + 3u, 0u, nlit);
            a.sec_off[b] = fh + 3u + rh + nlit;
            plan->nlit = nlit;
        }
        if (tid < 256u) {
            uint32_t c = 0;
#pragma unroll
            for (uint32_t h = 0; h < kHistCopies; ++h) c += S.hist[tid * kHistCopies + ((h + tid) & (kHistCopies - 1u))];
            a.hist[static_cast<uint64_t>(b) * 256u + tid] = c;
        }
        __syncthreads();
    }
}

// Bits into a byte buffer in shared memory, LSB first.
struct SmemBits {
    uint8_t *p;
    uint32_t cap, pos, nbits;
    uint64_t acc;
    bool ovf;
    __device__ void add(uint32_t v, uint32_t nb) {
        acc |= static_cast<uint64_t>(v) << nbits;
        nbits += nb;
        while (nbits >= 8u) {
            if (pos < cap) p[pos] = static_cast<uint8_t>(acc);
            else ovf = true;
            ++pos;
            acc >>= 8;
            nbits -= 8u;
        }
    }
    __device__ void flush() {  // pad the last partial byte with zeros
        if (nbits) add(0u, 8u - nbits);
    }
};

constexpr uint32_t kPlanWarps = 4;

struct PlanSmem {  // one per warp
    uint32_t leafw[258];  // leaf weights ascending, then two sentinels
    uint32_t node[258];   // internal weights in the order they are made, sentinels where none is yet
    uint32_t bl[32];
    uint32_t start[16];
    uint32_t cw[12];
    uint16_t leaf[256];
    uint16_t anc[2][512];
    uint16_t code[256];
    uint16_t fenc[12 * 64];  // weight, next decoder state: state | bit count << 6
    uint8_t dep[2][512];
    uint8_t len[256];
    uint8_t tree[132];
    uint8_t wts[256];
};

// FSE-compressed weights P.wts[0..N) into P.tree + 1 (one warp); returns
// their size, or 0.
__device__ uint32_t plan_fse_weights(PlanSmem &P, uint32_t N) {
    const uint32_t lane = lane_id(), lt = lanemask_lt();
    if (lane < 12u) P.cw[lane] = 0u;
    __syncwarp();
    for (uint32_t i = lane; i < N; i += 32u) atomicAdd(&P.cw[P.wts[i]], 1u);
    __syncwarp();
    int norm[12];
    uint32_t distinct = 0;
    int sum = 0, top = 0, big = 0;
#pragma unroll
    for (uint32_t s2 = 0; s2 < 12; ++s2) {
        const uint32_t c = P.cw[s2];
        distinct += c ? 1u : 0u;
        norm[s2] = c ? max(1, static_cast<int>(c * 64u / N)) : 0;
        sum += norm[s2];
        if (s2 == 0u || norm[s2] > top) {
            top = norm[s2];
            big = static_cast<int>(s2);
        }
    }
    if (distinct < 2u || top + 64 - sum <= 0) return 0;  // warp-uniform
#pragma unroll
    for (uint32_t s2 = 0; s2 < 12; ++s2)
        if (static_cast<int>(s2) == big) norm[s2] += 64 - sum;
    // Decoder table (no "less than 1" entries, so no high threshold): the i-th
    // state in weight order sits at 43 i mod 64 (step (64 >> 1) + (64 >> 3) + 3,
    // whose inverse mod 64 is 3); this lane's states are `lane` and `lane + 32`.
    uint32_t sym[2] = {0, 0}, x[2] = {0, 0}, acc = 0;
    const uint32_t i0 = (3u * lane) & 63u, i1 = (3u * (lane + 32u)) & 63u;
#pragma unroll
    for (uint32_t s2 = 0; s2 < 12; ++s2) {
        acc += static_cast<uint32_t>(norm[s2]);
        if (i0 >= acc) sym[0] = s2 + 1u;
        if (i1 >= acc) sym[1] = s2 + 1u;
    }
#pragma unroll
    for (uint32_t s2 = 0; s2 < 12; ++s2) {
        const uint32_t m0 = __ballot_sync(kFull, sym[0] == s2), m1 = __ballot_sync(kFull, sym[1] == s2);
        const uint32_t nn = static_cast<uint32_t>(norm[s2]);
        if (sym[0] == s2) x[0] = nn + static_cast<uint32_t>(__popc(m0 & lt));
        if (sym[1] == s2) x[1] = nn + static_cast<uint32_t>(__popc(m0) + __popc(m1 & lt));
    }
    uint32_t fnb[2];
#pragma unroll
    for (uint32_t u = 0; u < 2u; ++u) {
        fnb[u] = 6u - highbit(x[u]);
        const uint32_t b0 = (x[u] << fnb[u]) - 64u, st = lane + 32u * u;
        for (uint32_t v = b0; v < b0 + (1u << fnb[u]); ++v)
            P.fenc[sym[u] * 64u + v] = static_cast<uint16_t>(st | (fnb[u] << 6));
    }
    // states: the last two weights pick theirs (the second-to-last one with an
    // update bit), the rest follow the chain
    const uint32_t w1 = P.wts[N - 1], w2 = P.wts[N - 2];
    const uint32_t a0 = __ballot_sync(kFull, sym[0] == w1), a1 = __ballot_sync(kFull, sym[1] == w1);
    const uint32_t p0 = __ballot_sync(kFull, sym[0] == w2 && fnb[0] >= 1u),
                   p1 = __ballot_sync(kFull, sym[1] == w2 && fnb[1] >= 1u);
    const uint32_t s_last = a0 ? static_cast<uint32_t>(__ffs(a0)) - 1u : 31u + static_cast<uint32_t>(__ffs(a1));
    if (!(p0 | p1)) return 0;
    const uint32_t s_prev = p0 ? static_cast<uint32_t>(__ffs(p0)) - 1u : 31u + static_cast<uint32_t>(__ffs(p1));
    __syncwarp();
    uint32_t desc = 0;
    if (lane == 0) {
        // table description (RFC 8878 4.1.1)
        SmemBits wr{P.tree + 1, 127u, 0u, 0u, 0ull, false};
        wr.add(1u, 4u);  // accuracy 6
        int remaining = 65, threshold = 64, lastw = 0;
        uint32_t nb = 7;
#pragma unroll
        for (int s2 = 0; s2 < 12; ++s2)
            if (norm[s2]) lastw = s2;
        int zeros = -1;  // zero counts since the first of a run of them (-1: none)
#pragma unroll
        for (int s2 = 0; s2 < 12; ++s2) {
            if (s2 > lastw) break;
            if (zeros >= 0 && norm[s2] == 0) {
                ++zeros;
                continue;
            }
            if (zeros >= 0) {
                for (; zeros >= 3; zeros -= 3) wr.add(3u, 2u);
                wr.add(static_cast<uint32_t>(zeros), 2u);
                zeros = -1;
            }
            const int v = norm[s2] + 1, mx = (2 * threshold - 1) - remaining;
            if (v < mx) wr.add(static_cast<uint32_t>(v), nb - 1u);
            else if (v < threshold) wr.add(static_cast<uint32_t>(v), nb);
            else wr.add(static_cast<uint32_t>(v + mx), nb);
            remaining -= norm[s2];
            while (remaining < threshold) {
                --nb;
                threshold >>= 1;
            }
            if (norm[s2] == 0) zeros = 0;
        }
        wr.flush();
        desc = wr.pos;
    }
    desc = __shfl_sync(kFull, desc, 0);
    // Entry u of the bitstream: state | bit count << 6, for weights N-3 .. 0,
    // then the states of weights 1 and 0 and the end marker.  The two chains
    // alternate; lanes 0 and 1 run one each, four weights read ahead of it.
    uint16_t *ent = P.anc[0];
    uint32_t *words = reinterpret_cast<uint32_t *>(P.anc[1]);
    const uint32_t M = N - 2u, T = M + 3u;
    if (lane < 2u) {
        uint32_t x = lane ? s_prev : s_last, u = lane;
        for (; u + 6u < M; u += 8u) {
            uint32_t w[4], o[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) w[k] = 64u * P.wts[M - 1u - u - 2u * k];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const uint32_t e = P.fenc[w[k] + x];
                o[k] = x | (e & ~63u);
                x = e & 63u;
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) ent[u + 2u * k] = static_cast<uint16_t>(o[k]);
        }
        for (; u < M; u += 2u) {
            const uint32_t e = P.fenc[64u * P.wts[M - 1u - u] + x];
            ent[u] = static_cast<uint16_t>(x | (e & ~63u));
            x = e & 63u;
        }
        ent[u] = static_cast<uint16_t>(x | (6u << 6));  // u: M or M + 1
    }
    if (lane == 2u) ent[T - 1u] = 1u | (1u << 6);
    for (uint32_t i = lane; i < 52u; i += 32u) words[i] = 0u;
    __syncwarp();
    uint64_t v = 0;  // this lane's eight entries, at most 48 bits
    uint32_t nv = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t u = 8u * lane + k;
        if (u < T) {
            const uint32_t e = ent[u], n = e >> 6;
            v |= static_cast<uint64_t>(e & ((1u << n) - 1u)) << nv;
            nv += n;
        }
    }
    uint32_t end = nv;
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, end, d);
        if (lane >= d) end += y;
    }
    if (nv) {
        const uint32_t at = end - nv, sh = at & 31u;
        const uint64_t lo = v << sh;
        atomicOr(&words[at >> 5], static_cast<uint32_t>(lo));
        atomicOr(&words[(at >> 5) + 1u], static_cast<uint32_t>(lo >> 32));
        if (sh) atomicOr(&words[(at >> 5) + 2u], static_cast<uint32_t>(v >> (64u - sh)));
    }
    const uint32_t bytes = (__shfl_sync(kFull, end, 31) + 7u) >> 3;
    if (desc + bytes > 127u) return 0;
    __syncwarp();
    const uint8_t *wb = reinterpret_cast<const uint8_t *>(words);
    for (uint32_t i = lane; i < bytes; i += 32u) P.tree[1u + desc + i] = wb[i];
    __syncwarp();
    return desc + bytes;
}

// The 256 keys of a warp in ascending order (bitonic network); lane l holds
// elements 8l .. 8l+7.
__device__ __forceinline__ void sort256(uint32_t *v) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (uint32_t k = 2; k <= 256u; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j >= 1u; j >>= 1) {
            if (j >= 8u) {
                const bool keep_min = ((lane & (j >> 3)) == 0u) == (((lane << 3) & k) == 0u);
#pragma unroll
                for (uint32_t r = 0; r < 8u; ++r) {
                    const uint32_t o = __shfl_xor_sync(kFull, v[r], j >> 3);
                    v[r] = keep_min ? min(v[r], o) : max(v[r], o);
                }
            } else {
#pragma unroll
                for (uint32_t r = 0; r < 8u; ++r) {
                    if (r & j) continue;
                    const bool up = (((lane << 3) | r) & k) == 0u;
                    const uint32_t lo = min(v[r], v[r | j]), hi = max(v[r], v[r | j]);
                    v[r] = up ? lo : hi;
                    v[r | j] = up ? hi : lo;
                }
            }
        }
    }
}

// One warp per window: the Huffman code of the window's literals.  One window is
// bound by latency, so what one lane did in order (255 merges, 253 FSE steps with
// their bits, moves of leaves one by one) is done by the warp in few rounds:
// 17 windows 69 -> 36 us, 4096 windows 134 -> 62.
__global__ void __launch_bounds__(32 * kPlanWarps) zenc_huf_plan_kernel(ZencArgs a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
    PlanSmem &P = reinterpret_cast<PlanSmem *>(smem_raw)[wid];
    for (uint32_t b = blockIdx.x * kPlanWarps + wid; b < a.num_windows; b += gridDim.x * kPlanWarps) {
        PlanRec *plan = reinterpret_cast<PlanRec *>(a.plan + static_cast<uint64_t>(b) * kZencPlanBytes);
        const uint32_t nlit = a.sec_off[b] ? plan->nlit : 0u;
        uint32_t mode = 0;
        if (nlit) {
            const uint32_t *hist = a.hist + static_cast<uint64_t>(b) * 256u;
            // present bytes sorted by (count, byte); lane l counts bytes 8l .. 8l+7
            uint32_t key[8];
            uint32_t present = 0, top = 0;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t c = hist[lane * 8u + i];
                key[i] = c ? (c << 8) | (lane * 8u + i) : ~0u;
                if (c) {
                    ++present;
                    top = lane * 8u + i;
                }
            }
            const uint32_t n = __reduce_add_sync(kFull, present), last = __reduce_max_sync(kFull, top);
            if (n == 0u) {
                // nothing counted although the window has literals: keep the raw section
            } else if (n == 1u) {
                mode = 1;
                if (lane == 0) plan->rle = last;
            } else {
                sort256(key);
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    P.leaf[lane * 8u + i] = static_cast<uint16_t>(key[i] & 0xFFu);
                    P.leafw[lane * 8u + i] = key[i] == ~0u ? ~0u : key[i] >> 8;
                    P.node[lane * 8u + i] = ~0u;
                }
                if (lane < 2u) P.leafw[256u + lane] = P.node[256u + lane] = ~0u;
                __syncwarp();
                // Two-queue Huffman construction: the two lightest of the leaves and
                // internal nodes left are merged, a leaf first on equal weights,
                // an older node before a newer one; sentinels stand for what is
                // not there.  No new node is lighter than the first pair's sum,
                // so all items up to that sum pair up in order, at once (an odd
                // last one waits), and the sums at least double every other round.
                uint32_t *srt = reinterpret_cast<uint32_t *>(P.anc[1]);
                for (uint32_t li = 0, ii = 0, m = 0; m + 1u < n;) {
                    const uint32_t l0 = P.leafw[li], l1 = P.leafw[li + 1u], n0 = P.node[ii], n1 = P.node[ii + 1u];
                    const uint32_t sum = l0 <= n0 ? l0 + min(l1, n0) : n0 + min(l0, n1);
                    auto upto = [&](const uint32_t *w, uint32_t from) {  // items from `from` on up to sum
                        for (uint32_t c = 0;;) {
                            const uint32_t k = from + c + lane;
                            const uint32_t bal = __ballot_sync(kFull, k < 256u && w[k] <= sum);
                            c += static_cast<uint32_t>(__popc(bal));
                            if (bal != kFull) return c;
                        }
                    };
                    const uint32_t nl = upto(P.leafw, li), ni = upto(P.node, ii), k = nl + ni, paired = k & ~1u;
                    const bool leaf_last = nl && (!ni || P.leafw[li + nl - 1u] > P.node[ii + ni - 1u]);
                    for (uint32_t j = lane; j < k; j += 32u) {  // to its rank among both
                        const bool lf = j < nl;
                        const uint32_t jj = lf ? j : j - nl, w = lf ? P.leafw[li + jj] : P.node[ii + jj];
                        const uint32_t *other = lf ? P.node + ii : P.leafw + li;
                        const uint32_t cnt = lf ? ni : nl, below = lf ? w : w + 1u;
                        uint32_t r = 0;
                        if (nl && ni)
                            for (uint32_t d = 1u << highbit(max(nl, ni)); d; d >>= 1)
                                if (r + d <= cnt && other[r + d - 1u] < below) r += d;
                        r += jj;
                        srt[r] = w;
                        if (r < paired) P.anc[0][lf ? li + jj : n + ii + jj] = static_cast<uint16_t>(n + m + (r >> 1));
                    }
                    __syncwarp();
                    for (uint32_t j = lane; j < paired / 2u; j += 32u) P.node[m + j] = srt[2u * j] + srt[2u * j + 1u];
                    __syncwarp();
                    m += paired / 2u;
                    li += nl - (k != paired && leaf_last ? 1u : 0u);
                    ii += ni - (k != paired && !leaf_last ? 1u : 0u);
                }
                // depths by pointer jumping (parent links, the root points to itself)
                const uint32_t nn = 2u * n - 1u, root = nn - 1u;
                for (uint32_t k = lane; k < ((nn + 127u) & ~127u); k += 32u) {
                    if (k >= root) P.anc[0][k] = static_cast<uint16_t>(root);
                    P.dep[0][k] = k >= root ? 0u : 1u;
                }
                P.bl[lane] = 0u;
                __syncwarp();
                uint32_t cur = 0;
                for (bool open = true; open; cur ^= 1u) {
                    open = false;
                    for (uint32_t k = lane; k < nn; k += 128u) {
                        uint32_t an[4], a2[4], d[4];
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u) an[u] = P.anc[cur][k + 32u * u];
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u) {
                            a2[u] = P.anc[cur][an[u]];
                            d[u] = P.dep[cur][k + 32u * u] + P.dep[cur][an[u]];
                        }
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u) {
                            P.anc[cur ^ 1u][k + 32u * u] = static_cast<uint16_t>(a2[u]);
                            P.dep[cur ^ 1u][k + 32u * u] = static_cast<uint8_t>(d[u]);
                            open = open || a2[u] != root;
                        }
                    }
                    open = __any_sync(kFull, open);
                    __syncwarp();
                }
                // (65536 literals: no depth above 22)
                for (uint32_t k = lane; k < n; k += 32u) atomicAdd(&P.bl[min(static_cast<uint32_t>(P.dep[cur][k]), 31u)], 1u);
                __syncwarp();
                // Limit to 11 bits, keeping the code complete: two leaves at level i
                // become one at i - 1, and the deepest leaf at most at i - 2 two
                // one level below it.  Lane L holds level L; as long as that leaf
                // is at i - 2 itself, its whole level goes at once.
                uint32_t lv = P.bl[lane];
                for (uint32_t i = highbit(__ballot_sync(kFull, lv != 0u)); i > kHufMaxBits; --i) {
                    for (uint32_t at_i; (at_i = __shfl_sync(kFull, lv, i)) != 0u;) {
                        const uint32_t j = highbit(__ballot_sync(kFull, lv != 0u) & ((1u << (i - 1u)) - 1u));
                        const uint32_t at_j = __shfl_sync(kFull, lv, j);
                        const uint32_t t = j + 2u == i ? min(at_i / 2u, at_j) : 1u;
                        if (lane == i) lv -= 2u * t;
                        if (lane == i - 1u) lv += t;
                        if (lane == j + 1u) lv += 2u * t;
                        if (lane == j) lv -= t;
                    }
                }
                const uint32_t maxb = highbit(__ballot_sync(kFull, lv != 0u));
                uint32_t code0 = 0, mine = 0;  // first code of level L
                for (uint32_t L = maxb - 1u; L >= 1u; --L) {
                    code0 = (code0 + __shfl_sync(kFull, lv, L + 1u)) >> 1;
                    if (lane == L) mine = code0;
                }
                P.bl[lane] = lv;
                if (lane < 16u) P.start[lane] = mine;
                __syncwarp();
                // lengths: the longest codes to the least frequent bytes
                for (uint32_t i = 0; i < 8; ++i) P.len[lane * 8u + i] = 0;
                __syncwarp();
                for (uint32_t k = lane; k < n; k += 32u) {
                    uint32_t cum = 0;
                    for (uint32_t L = kHufMaxBits; L >= 1u; --L) {
                        if (k < cum + P.bl[L]) {
                            P.len[P.leaf[k]] = static_cast<uint8_t>(L);
                            break;
                        }
                        cum += P.bl[L];
                    }
                }
                __syncwarp();
                // canonical codes: start[L] + rank among the bytes of length L
                uint32_t l8[8];
                for (uint32_t i = 0; i < 8; ++i) l8[i] = P.len[lane * 8u + i];
                for (uint32_t L = 1; L <= maxb; ++L) {
                    uint32_t m = 0;
                    for (uint32_t i = 0; i < 8; ++i) m += l8[i] == L ? 1u : 0u;
                    uint32_t x = m;
                    for (uint32_t dd = 1; dd < 32; dd <<= 1) {
                        const uint32_t y = __shfl_up_sync(kFull, x, dd);
                        if (lane >= dd) x += y;
                    }
                    uint32_t code = P.start[L] + x - m;
                    for (uint32_t i = 0; i < 8; ++i)
                        if (l8[i] == L) P.code[lane * 8u + i] = static_cast<uint16_t>(code++);
                }
                // weights of bytes 0 .. last-1 (the last one's is implied)
                const uint32_t N = last;
                for (uint32_t i = 0; i < 8; ++i) {
                    const uint32_t s2 = lane * 8u + i;
                    if (s2 < N) P.wts[s2] = l8[i] ? static_cast<uint8_t>(maxb + 1u - l8[i]) : 0u;
                }
                __syncwarp();
                uint32_t tree_bytes = 0;
                if (N <= 128u) {
                    if (lane == 0) P.tree[0] = static_cast<uint8_t>(127u + N);
                    for (uint32_t m2 = lane; m2 < (N + 1u) / 2u; m2 += 32u) {
                        const uint32_t hi4 = P.wts[2u * m2], lo4 = 2u * m2 + 1u < N ? P.wts[2u * m2 + 1u] : 0u;
                        P.tree[1u + m2] = static_cast<uint8_t>((hi4 << 4) | lo4);
                    }
                    tree_bytes = 1u + (N + 1u) / 2u;
                } else {
                    const uint32_t f = plan_fse_weights(P, N);
                    if (f) {
                        if (lane == 0) P.tree[0] = static_cast<uint8_t>(f);
                        tree_bytes = 1u + f;
                    }
                }
                __syncwarp();
                if (tree_bytes) {
                    mode = 2;
                    for (uint32_t i = lane; i < 256u; i += 32u) {
                        plan->len[i] = P.len[i];
                        plan->code[i] = P.code[i];
                    }
                    for (uint32_t i = lane; i < tree_bytes; i += 32u) plan->tree[i] = P.tree[i];
                    if (lane == 0) plan->tree_bytes = tree_bytes;
                }
            }
        }
        if (lane == 0) plan->mode = mode;
        __syncwarp();
    }
}

// Literal runs for the Huffman streams: with 4 streams, threads 128s .. 128s+127
// split stream s; with one stream all threads split it.  Run j of a stream
// covers [lo + j*size, lo + (j+1)*size); the stream's bits start with its last
// literal, so the highest run comes first.
struct LitRun {
    uint32_t stream, j, group, lo, hi;
};
__device__ __forceinline__ LitRun lit_run(uint32_t tid, uint32_t nlit, uint32_t nstreams, uint32_t seg) {
    LitRun r;
    r.group = nstreams == 4u ? kLitThreads / 4u : kLitThreads;
    r.stream = tid / r.group;
    r.j = tid % r.group;
    const uint32_t s_lo = r.stream * seg, s_hi = r.stream == nstreams - 1u ? nlit : s_lo + seg;
    const uint32_t size = (s_hi - s_lo + r.group - 1u) / r.group;
    r.lo = min(s_lo + r.j * size, s_hi);
    r.hi = min(r.lo + size, s_hi);
    return r;
}

// 32-bit words of `out` from bit `bitpos` on; words shared with a neighbour
// are ORed in, the others stored.
struct RunWriter {
    uint32_t *out;
    uint32_t acc, nb;
    bool first;
    __device__ __forceinline__ RunWriter(uint32_t *o, uint64_t bitpos)
        : out(o + (bitpos >> 5)), acc(0), nb(static_cast<uint32_t>(bitpos & 31u)), first(true) {}
    __device__ __forceinline__ void add(uint32_t v, uint32_t len) {  // len <= 32, v < 2^len
        acc |= v << nb;
        const uint32_t rest = __funnelshift_l(v, 0u, nb);  // v >> (32 - nb), 0 for nb = 0
        nb += len;
        if (nb >= 32u) {
            if (first) atomicOr(out, acc);
            else *out = acc;
            first = false;
            ++out;
            acc = rest;
            nb -= 32u;
        }
    }
    __device__ __forceinline__ void close() {
        if (nb) atomicOr(out, acc);
    }
};

struct WriteSmem {
    uint32_t tab[256];  // length | code << 16 (sums of lengths stay in the low half)
    uint32_t seg_bits[4];
    uint32_t warp_bits[kLitThreads / 32];
    uint32_t stream_off[4], stream_bytes[4];
    uint32_t mode;
};
constexpr uint32_t kWriteSmem = kMaxWindow + sizeof(WriteSmem);

// lit[hi-1] .. lit[lo] in that order: f(byte) or g(byte, next byte), four bytes
// per read inside.
template <class F, class G>
__device__ __forceinline__ void for_run_down(const uint8_t *lit, uint32_t lo, uint32_t hi, F f, G g) {
    const uint32_t *words = reinterpret_cast<const uint32_t *>(lit);
    uint32_t k = hi;
    while (k > lo && (k & 3u)) f(lit[--k]);
    for (; k >= lo + 4u; k -= 4u) {
        const uint32_t w = words[k / 4u - 1u];
        g(w >> 24, (w >> 16) & 0xFFu);
        g((w >> 8) & 0xFFu, w & 0xFFu);
    }
    while (k > lo) f(lit[--k]);
}

// One CTA per window: the RLE or Huffman-coded literal section where it is
// smaller than the raw one already in the slot.
__global__ void __launch_bounds__(kLitThreads, 3) zenc_huf_write_kernel(ZencArgs a) {
    extern __shared__ __align__(16) uint8_t lit[];  // kMaxWindow literal bytes, then WriteSmem
    WriteSmem &H = *reinterpret_cast<WriteSmem *>(lit + kMaxWindow);
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    for (uint32_t b = blockIdx.x; b < a.num_windows; b += gridDim.x) {
        const PlanRec *plan = reinterpret_cast<const PlanRec *>(a.plan + static_cast<uint64_t>(b) * kZencPlanBytes);
        if (a.sec_off[b] == 0u) continue;  // raw frame (uniform over the CTA)
        const uint32_t mode = plan->mode;
        if (mode == 0u) continue;
        const uint32_t w = win_size(a, b);
        const uint32_t fh = frame_header_bytes(w), L0 = fh + 3u;
        const uint32_t nlit = plan->nlit, rh = raw_lit_header_bytes(nlit);
        uint8_t *slot = a.slots + static_cast<uint64_t>(b) * kZencSlot;
        if (mode == 1u) {
            if (tid == 0) {
                write_raw_lit_header(slot + L0, 1u, nlit);
                slot[L0 + rh] = static_cast<uint8_t>(plan->rle);
                a.sec_off[b] = L0 + rh + 1u;
            }
            continue;
        }
        // Huffman: the literals back from the raw section, the code from the plan
        const uint8_t *rawp = slot + L0 + rh;
        uint32_t *lit32 = reinterpret_cast<uint32_t *>(lit);
        for (uint32_t k = tid; k < (nlit >> 2); k += kLitThreads) lit32[k] = load4(rawp + 4u * k);
        for (uint32_t k = (nlit & ~3u) + tid; k < nlit; k += kLitThreads) lit[k] = rawp[k];
        if (tid < 256u) H.tab[tid] = plan->len[tid] | (static_cast<uint32_t>(plan->code[tid]) << 16);
        if (tid < 4u) H.seg_bits[tid] = 0u;
        __syncthreads();
        const uint32_t nst = nlit < 1024u ? 1u : 4u;
        const uint32_t seg = nlit < 1024u ? nlit : (nlit + 3u) / 4u;
        const LitRun run = lit_run(tid, nlit, nst, seg);
        uint32_t v = 0;
        for_run_down(
            lit, run.lo, run.hi, [&](uint32_t x) { v += H.tab[x]; },
            [&](uint32_t x, uint32_t y) { v += H.tab[x] + H.tab[y]; });
        v &= 0xFFFFu;  // a run has at most 128 codes of 11 bits
        // bits of the runs before this one among all (scan of the warps' sums below)
        uint32_t incl = v;
#pragma unroll
        for (uint32_t d = 1; d < 32u; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, incl, d);
            if (lane >= d) incl += y;
        }
        if (lane == 31u) {
            H.warp_bits[tid >> 5] = incl;
            atomicAdd(&H.seg_bits[run.stream], incl);  // a warp's runs are of one stream
        }
        __syncthreads();
        if (tid == 0) {
            const uint32_t tree_bytes = plan->tree_bytes;
            uint32_t streams = 0;
            for (uint32_t s2 = 0; s2 < nst; ++s2) {
                H.stream_bytes[s2] = (H.seg_bits[s2] + 8u) >> 3;  // + end marker, rounded up
                streams += H.stream_bytes[s2];
            }
            const uint32_t body = tree_bytes + (nst == 4u ? 6u : 0u) + streams;
            const uint32_t hdr = nst == 1u ? 3u : (max(nlit, body) < 16384u ? 4u : 5u);
            H.mode = 0;
            if (!((nst == 1u && body >= 1024u) || hdr + body >= rh + nlit)) {
                H.mode = 2;
                uint64_t hv;
                if (hdr == 3u) hv = 2u | (static_cast<uint64_t>(nlit) << 4) | (static_cast<uint64_t>(body) << 14);
                else if (hdr == 4u) hv = 2u | (2u << 2) | (static_cast<uint64_t>(nlit) << 4) | (static_cast<uint64_t>(body) << 18);
                else hv = 2u | (3u << 2) | (static_cast<uint64_t>(nlit) << 4) | (static_cast<uint64_t>(body) << 22);
                uint8_t *h = slot + L0;
                for (uint32_t i = 0; i < hdr; ++i) h[i] = static_cast<uint8_t>(hv >> (8u * i));
                for (uint32_t i = 0; i < tree_bytes; ++i) h[hdr + i] = plan->tree[i];
                uint32_t o = L0 + hdr + tree_bytes;
                if (nst == 4u) {
                    for (uint32_t s2 = 0; s2 < 3; ++s2) {
                        slot[o + 2 * s2] = static_cast<uint8_t>(H.stream_bytes[s2]);
                        slot[o + 2 * s2 + 1] = static_cast<uint8_t>(H.stream_bytes[s2] >> 8);
                    }
                    o += 6u;
                }
                for (uint32_t s2 = 0; s2 < nst; ++s2) {
                    H.stream_off[s2] = o;
                    o += H.stream_bytes[s2];
                }
                a.sec_off[b] = o;
            }
        }
        __syncthreads();
        if (H.mode == 2u) {
            // The streams' bytes start at zero (runs OR their shared words in); the
            // bytes of the headers before them are kept.
            const uint32_t s0b = H.stream_off[0];
            const uint32_t s1b = H.stream_off[nst - 1u] + H.stream_bytes[nst - 1u];
            uint32_t *wslot = reinterpret_cast<uint32_t *>(slot);
            const uint32_t w0 = (s0b + 3u) >> 2, w1 = (s1b + 3u) >> 2;
            for (uint32_t k = s0b + tid; k < min(w0 * 4u, s1b); k += kLitThreads) slot[k] = 0;
            for (uint32_t k = w0 + tid; k < w1; k += kLitThreads) wslot[k] = 0u;
            __syncthreads();
            // bit offset of this run: the runs after it in the stream come first
            uint32_t upto = incl;  // bits of the stream's runs up to this one
            for (uint32_t k = run.stream * (run.group / 32u); k < (tid >> 5); ++k) upto += H.warp_bits[k];
            if (run.hi > run.lo || run.j == 0u) {
                RunWriter wr(wslot, 8ull * H.stream_off[run.stream] + (H.seg_bits[run.stream] - upto));
                for_run_down(
                    lit, run.lo, run.hi,
                    [&](uint32_t x) {
                        const uint32_t t = H.tab[x];
                        wr.add(t >> 16, t & 0xFFFFu);
                    },
                    [&](uint32_t x, uint32_t y) {  // two codes, at most 22 bits
                        const uint32_t t = H.tab[x], u = H.tab[y], l = t & 0xFFFFu;
                        wr.add((t >> 16) | ((u >> 16) << l), l + (u & 0xFFFFu));
                    });
                if (run.j == 0u) wr.add(1u, 1u);  // end of the stream
                wr.close();
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- sequences
// One CTA of kSeqThreads threads per window; each thread owns a run of
// consecutive sequences.  The serial parts of the format are run by all
// threads at once from guessed states, which are then checked against the
// state the thread before left, and run again where they differ:
//   R. ascending: each Offset_Value from the decoder's repeat history.  A
//      thread guesses the history as the three different offsets used last
//      before its run, which is wrong only where an offset repeats without
//      literals; the values go to a per-window global scratch, the LL, ML and
//      OF codes are counted.  (Guessed as the last three offsets, the history
//      of a window that uses one or two distances moved on by one thread per
//      round: 4096 windows of 32-bit counters 15.4 ms against 7.0.)
//   T. one warp each picks and builds the table of LL, ML and OF (RFC 8878
//      3.1.1.3.2.1): RLE_Mode when one code is used, else FSE_Compressed_Mode
//      or Predefined_Mode, whichever costs fewer bits by an integer estimate
//      (below).
//   E. in bitstream order (the last sequence first), kChunk sequences at a time:
//      codes by all threads; one warp per FSE chain, each lane a run of
//      kChunk / 32 symbols; then every thread's bit count, a scan, and every
//      thread writes the bits of its sequences.  An encoder state says little
//      about the states a few symbols on: a lane starts kWarmUp symbols before
//      its run from any state and has mostly met the true chain at its start.
//      Where it has not, its run is repeated from the state before it, round
//      by round (about 30 % of the runs, some over several rounds: runs of one
//      frequent code keep two chains apart).
// What bounds it: latency of the dependent table reads.  With one warp per
// window, the history and the three chains on single lanes, 17 windows took
// 554 us and 4096 windows 978 us; this form takes 75 us and 343 us.
// The cost estimate counts, per code c used k times, k * (A - log2(n_c))
// bits, with log2 taken piecewise linear between powers of two in 1/256 bit
// (lg256 below), plus the table description's bytes.  FSE_Compressed_Mode
// uses accuracy A = max(5, min(Amax, bitlen(ns - 1) - 2)), raised until the
// table has two states per used code (Amax: 9 for LL and ML, 8 for OF), and
// counts normalised to 2^A by rounding k * 2^A / ns (at least 1); the most
// used code takes a positive remainder, a negative one is taken one state at a
// time from the largest count (lowest code first on ties).
// The encoder of any table follows from its decoder (RFC 8878 4.1.1): code c
// with normalised count n owns, in ascending decoder-state order, the states
// numbered x = n .. 2n-1; for the next decoder state D' the encoder takes the
// state x = (D' + 2^A) >> b, with b the bit count that puts x in [n, 2n), and
// writes the low b bits of D' + 2^A.
constexpr uint32_t kSeqThreads = 128;
constexpr uint32_t kChunk = 1024;                        // sequences per pass of step E
constexpr uint32_t kRun = kChunk / 32;                   // symbols per lane of a chain
constexpr uint32_t kWarmUp = 8;                          // symbols before a run that its chain starts at
constexpr uint32_t kOwn = kChunk / kSeqThreads;          // sequences per thread of a chunk
constexpr uint32_t kMaxAl = 9;                           // Accuracy_Log limit of LL and ML (OF: 8)
constexpr uint32_t kTabDesc = 128;                       // bytes of one table description
constexpr uint32_t kOFCodes = 32;                        // offset codes counted (a window's are <= 16)

// One field's (LL, ML or OF) table for one window.
struct FieldTab {
    uint32_t hist[64];           // uses of code c in the window
    // Code c with n states: x = (D' + 2^A) >> nb, nb = (D' + 2^A + enc.x) >> 16
    // (enc.x = (hi << 16) - (n << hi), hi = A - floor(log2(n))), next state
    // stl[x + enc.y] (enc.y: the code's first entry - n).
    uint2 enc[64];
    uint32_t desc[kTabDesc / 4]; // FSE table description, or the RLE code
    uint16_t stl[1u << kMaxAl];  // each code's decoder states, ascending, code after code
    uint16_t cumul[64];          // states of the codes before c
    uint16_t fill[64];           // next stl entry of code c (building only)
    uint16_t norm[64];           // normalised counts (building only)
    uint8_t sym[1u << kMaxAl];   // spread table (building only)
    uint32_t al;                 // accuracy log (0 for RLE_Mode)
    uint32_t mode;               // 0 Predefined_Mode, 1 RLE_Mode, 2 FSE_Compressed_Mode
    uint32_t desc_len;
};

struct SeqSmem {
    CodeTables C;
    FieldTab tab[3];                    // LL, ML, OF
    uint32_t out_state[3][kSeqThreads]; // repeat offsets that each thread's run leaves
    uint32_t state[3];                  // chain states after the chunk
    uint32_t warp_bits[kSeqThreads / 32];
    // Of the chunk's sequences: codes, and update bits (value | count << 12),
    // lane by lane with a gap that spreads the lanes over the banks.
    alignas(4) uint8_t code[3][kChunk + 4 * 32];
    alignas(4) uint16_t upd[3][kChunk + 2 * 32];
};

// log2(x) * 256, piecewise linear between powers of two (x >= 1).
__device__ __forceinline__ uint32_t lg256(uint32_t x) {
    const uint32_t h = highbit(x);
    return 256u * h + ((x << 8) >> h) - 256u;
}

__device__ __forceinline__ void or_desc(uint32_t *d, uint32_t bitpos, uint64_t v, uint32_t nb) {
    if (nb == 0u) return;
    const uint32_t w = bitpos >> 5, sh = bitpos & 31u;
    const uint64_t lo = v << sh;  // nb <= 48, so v << sh spans at most 80 bits: three words
    atomicOr(d + w, static_cast<uint32_t>(lo));
    if (sh + nb > 32u) atomicOr(d + w + 1, static_cast<uint32_t>(lo >> 32));
    if (sh + nb > 64u) atomicOr(d + w + 2, static_cast<uint32_t>(v >> (64u - sh)));
}

__device__ __forceinline__ uint32_t scan_incl(uint32_t x) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, d);
        if (lane >= d) x += y;
    }
    return x;
}

// Picks and builds a field's table from its code histogram (one warp; lane l
// holds codes l and l + 32).  pre: the predefined distribution (-1 = "less
// than 1"), pre_n codes.
__device__ void build_field_table(FieldTab &T, uint32_t ns, uint32_t ncodes, uint32_t amax, const int8_t *pre,
                                  uint32_t pre_n, uint32_t pre_al) {
    const uint32_t lane = lane_id(), lt = lanemask_lt();
    uint32_t h[2], n[2];
    int32_t pn[2];
    bool no_pre = false;
#pragma unroll
    for (uint32_t u = 0; u < 2u; ++u) {
        const uint32_t c = lane + 32u * u;
        h[u] = c < ncodes ? T.hist[c] : 0u;
        pn[u] = c < pre_n ? pre[c] : 0;
        no_pre = no_pre || (h[u] && pn[u] == 0);  // a used code without a predefined state
    }
    const uint32_t m0 = __ballot_sync(kFull, h[0] != 0u), m1 = __ballot_sync(kFull, h[1] != 0u);
    const uint32_t used = static_cast<uint32_t>(__popc(m0) + __popc(m1));
    const uint32_t last = m1 ? 32u + highbit(m1) : highbit(m0);
    if (lane < kTabDesc / 4u) T.desc[lane] = 0u;
    __syncwarp();
    if (used == 1u) {  // RLE_Mode: one code, no state
        if (lane == 0) {
            T.mode = 1;
            T.al = 0;
            T.desc[0] = last;
            T.desc_len = 1;
            T.enc[last] = make_uint2(0u - 1u, 0u - 1u);
            T.stl[0] = 0;
        }
        return;
    }
    const bool pre_ok = !__any_sync(kFull, no_pre);
    // FSE_Compressed_Mode: accuracy, normalised counts.
    uint32_t al = 32u - static_cast<uint32_t>(__clz(ns - 1u));  // bit length of ns - 1
    al = al > 2u ? al - 2u : 0u;
    al = al < amax ? al : amax;
    al = al > 5u ? al : 5u;
    while ((1u << al) < 2u * used && al < amax) ++al;
    const uint32_t size = 1u << al;
#pragma unroll
    for (uint32_t u = 0; u < 2u; ++u) n[u] = h[u] ? max((h[u] * size + ns / 2u) / ns, 1u) : 0u;
    int32_t d = static_cast<int32_t>(size) - static_cast<int32_t>(__reduce_add_sync(kFull, n[0] + n[1]));
    // the lowest code among those with the largest key
    auto top_of = [&](uint32_t k0, uint32_t k1) {
        const uint32_t a = (k0 << 6) | (63u - lane), b = (k1 << 6) | (31u - lane);
        return 63u - (__reduce_max_sync(kFull, a > b ? a : b) & 63u);
    };
    if (d > 0) {
        const uint32_t top = top_of(h[0], h[1]);
        if (top == lane) n[0] += static_cast<uint32_t>(d);
        if (top == lane + 32u) n[1] += static_cast<uint32_t>(d);
    }
    for (; d < 0; ++d) {
        const uint32_t big = top_of(n[0], n[1]);
        if (big == lane) --n[0];
        if (big == lane + 32u) --n[1];
    }
    // Table description (RFC 8878 4.1.1).  The width of a count's field follows
    // from the counts before it; of a run of zeros the first is a count, the
    // others are two-bit repeat flags.
    const uint32_t s0 = scan_incl(n[0]), sum0 = __shfl_sync(kFull, s0, 31), s1 = scan_incl(n[1]) + sum0;
    const uint64_t zeros = ~((static_cast<uint64_t>(m1) << 32) | m0);  // codes with no uses
    uint64_t fv[2];
    uint32_t fb[2];
#pragma unroll
    for (uint32_t u = 0; u < 2u; ++u) {
        const uint32_t c = lane + 32u * u;
        fv[u] = 0;
        fb[u] = 0;
        const bool follows = c > 0u && ((zeros >> (c - 1u)) & 1u) != 0u && n[u] == 0u;  // inside a run of zeros
        if (c > last || follows) continue;
        const uint32_t before = (u ? s1 : s0) - n[u];
        const uint32_t remaining = size + 1u - before;
        // the threshold halves while it is above `remaining`, from 2^al on
        const uint32_t tlog = min(highbit(remaining), al), threshold = 1u << tlog;
        const uint32_t v = n[u] + 1u, mx = 2u * threshold - 1u - remaining;
        if (v < mx) {
            fv[u] = v;
            fb[u] = tlog;
        } else {
            fv[u] = v < threshold ? v : v + mx;
            fb[u] = tlog + 1u;
        }
        if (n[u] == 0u) {
            const uint64_t rest = ~(zeros >> (c + 1u));  // c < last < 63
            const uint32_t z = static_cast<uint32_t>(__ffsll(static_cast<long long>(rest))) - 1u;  // zeros after c
            uint32_t b = fb[u];
            for (uint32_t k = 0; k < z / 3u; ++k, b += 2u) fv[u] |= 3ull << b;
            fv[u] |= static_cast<uint64_t>(z % 3u) << b;
            fb[u] = b + 2u;
        }
    }
    const uint32_t b0 = scan_incl(fb[0]), bsum0 = __shfl_sync(kFull, b0, 31), b1 = scan_incl(fb[1]);
    const uint32_t bits = 4u + bsum0 + __shfl_sync(kFull, b1, 31), bytes = (bits + 7u) >> 3;
    uint32_t cp = 0, cf = 0;
#pragma unroll
    for (uint32_t u = 0; u < 2u; ++u) {
        if (!h[u]) continue;
        if (pre_ok) cp += h[u] * (256u * pre_al - lg256(pn[u] < 0 ? 1u : static_cast<uint32_t>(pn[u])));
        cf += h[u] * (256u * al - lg256(n[u]));
    }
    // (sums of at most 21845 * 9 * 256)
    const uint32_t cost_pre = __reduce_add_sync(kFull, cp), cost_fse = __reduce_add_sync(kFull, cf) + 2048u * bytes;
    const bool fse = bytes <= kTabDesc && (!pre_ok || cost_fse < cost_pre);
    uint32_t high, tal;
    if (fse) {
        if (lane == 0) or_desc(T.desc, 0u, al - 5u, 4u);
        or_desc(T.desc, 4u + b0 - fb[0], fv[0], fb[0]);
        or_desc(T.desc, 4u + bsum0 + b1 - fb[1], fv[1], fb[1]);
        tal = al;
        high = size - 1u;
    } else {  // Predefined_Mode; "less than 1" codes take the top states, one each
        const uint32_t l0 = __ballot_sync(kFull, pn[0] < 0), l1 = __ballot_sync(kFull, pn[1] < 0);
        tal = pre_al;
        const uint32_t top = (1u << pre_al) - 1u;
        high = top - static_cast<uint32_t>(__popc(l0) + __popc(l1));
        if (pn[0] < 0) T.sym[top - static_cast<uint32_t>(__popc(l0 & lt))] = static_cast<uint8_t>(lane);
        if (pn[1] < 0) T.sym[top - static_cast<uint32_t>(__popc(l0) + __popc(l1 & lt))] = static_cast<uint8_t>(lane + 32u);
#pragma unroll
        for (uint32_t u = 0; u < 2u; ++u) n[u] = pn[u] < 0 ? 1u : static_cast<uint32_t>(pn[u]);
    }
    const uint32_t tsize = 1u << tal, mask = tsize - 1u, step = (tsize >> 1) + (tsize >> 3) + 3u;
    // states before each code: all of them (cumul), and those that are spread (fill, for the search below)
    const bool sp0 = fse || pn[0] > 0, sp1 = fse || pn[1] > 0;
    const uint32_t a0 = scan_incl(n[0]), asum = __shfl_sync(kFull, a0, 31), a1 = scan_incl(n[1]) + asum;
    const uint32_t q0 = scan_incl(sp0 ? n[0] : 0u), qsum = __shfl_sync(kFull, q0, 31), q1 = scan_incl(sp1 ? n[1] : 0u) + qsum;
    T.cumul[lane] = static_cast<uint16_t>(a0 - n[0]);
    T.cumul[lane + 32u] = static_cast<uint16_t>(a1 - n[1]);
    T.fill[lane] = static_cast<uint16_t>(q0 - (sp0 ? n[0] : 0u));
    T.fill[lane + 32u] = static_cast<uint16_t>(q1 - (sp1 ? n[1] : 0u));
#pragma unroll
    for (uint32_t u = 0; u < 2u; ++u) {
        const uint32_t c = lane + 32u * u, before = (u ? a1 : a0) - n[u];
        const uint32_t hi = n[u] ? tal - highbit(n[u]) : 0u;
        T.enc[c] = make_uint2((hi << 16) - (n[u] << hi), before - n[u]);
    }
    __syncwarp();
    // Spread (RFC 8878 4.1.1): the codes' states in order, stepped through the
    // table, past the positions above `high`.  The k-th state placed belongs to
    // the last code with at most k spread states before it.
    // Four steps of 32 states at a time, here and below: their searches and
    // groups do not depend on one another (17 windows 79 -> 75 us; groups by one
    // ballot per bit of the code instead: 4096 windows 368 us against 343).
    uint32_t placed = 0;
    for (uint32_t i0 = 0; i0 < tsize; i0 += 128u) {
        uint32_t pos[4], k[4], c[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (uint32_t v = 0; v < 4u; ++v) {
            pos[v] = ((i0 + 32u * v + lane) * step) & mask;
            if (i0 + 32u * v >= tsize) pos[v] = tsize;
            const uint32_t ok = __ballot_sync(kFull, pos[v] <= high);
            k[v] = placed + static_cast<uint32_t>(__popc(ok & lt));
            placed += static_cast<uint32_t>(__popc(ok));
        }
#pragma unroll
        for (uint32_t dd = 32; dd >= 1u; dd >>= 1)
#pragma unroll
            for (uint32_t v = 0; v < 4u; ++v)
                if (T.fill[c[v] + dd] <= k[v]) c[v] += dd;  // c + dd <= 63
#pragma unroll
        for (uint32_t v = 0; v < 4u; ++v)
            if (pos[v] <= high) T.sym[pos[v]] = static_cast<uint8_t>(c[v]);
    }
    __syncwarp();
    T.fill[lane] = T.cumul[lane];
    T.fill[lane + 32u] = T.cumul[lane + 32u];
    __syncwarp();
    // Each code's states in ascending order.
    for (uint32_t u0 = 0; u0 < tsize; u0 += 128u) {
        uint32_t sy[4], g[4];
#pragma unroll
        for (uint32_t v = 0; v < 4u; ++v) sy[v] = u0 + 32u * v < tsize ? T.sym[u0 + 32u * v + lane] : 0u;
#pragma unroll
        for (uint32_t v = 0; v < 4u; ++v) g[v] = __match_any_sync(kFull, sy[v]);
#pragma unroll
        for (uint32_t v = 0; v < 4u; ++v) {
            if (u0 + 32u * v >= tsize) break;
            const uint32_t base = T.fill[sy[v]];
            T.stl[base + static_cast<uint32_t>(__popc(g[v] & lt))] = static_cast<uint16_t>(u0 + 32u * v + lane);
            __syncwarp();
            if (!(g[v] & ~lt & ~(1u << lane))) T.fill[sy[v]] = static_cast<uint16_t>(base + static_cast<uint32_t>(__popc(g[v])));
            __syncwarp();
        }
    }
    if (lane == 0) {
        T.mode = fse ? 2u : 0u;
        T.al = tal;
        T.desc_len = fse ? bytes : 0u;
    }
}

// Places of chunk sequence j in SeqSmem::code and ::upd.
__device__ __forceinline__ uint32_t code_at(uint32_t j) { return j + 4u * (j / kRun); }
__device__ __forceinline__ uint32_t upd_at(uint32_t j) { return j + 2u * (j / kRun); }

// One FSE chain over a chunk of len symbols (one warp): update bits of every
// symbol into up; D: the state before the chunk, then the one after it.
// fresh: the chunk's first symbol takes any state of its code, without bits.
__device__ void fse_chain(const FieldTab &T, const uint8_t *cd, uint16_t *up, uint32_t len, bool fresh, uint32_t &D) {
    const uint32_t lane = lane_id(), size = 1u << T.al;
    const uint32_t j0 = lane * kRun, n = len > j0 ? min(kRun, len - j0) : 0u;
    const uint32_t *cw = reinterpret_cast<const uint32_t *>(cd + code_at(j0));  // (rounded up to four codes)
    uint32_t *uw = reinterpret_cast<uint32_t *>(up + upd_at(j0));
    uint32_t in = D;
    if (lane > 0u && n) {  // a guess: the state kWarmUp symbols on from any state
        in = 0u;
        for (uint32_t j = j0 - kWarmUp; j < j0; ++j) {
            const uint2 e = T.enc[cd[code_at(j)]];
            const uint32_t v = in + size, nb = (v + e.x) >> 16;
            in = T.stl[(v >> nb) + e.y];
        }
    }
    uint32_t out = in;
    for (bool again = n > 0u; __any_sync(kFull, again);) {
        if (again) {
            out = in;
            // Four symbols at a time; the codes' entries, which do not depend
            // on the state, are read one group ahead of the chain.
            uint32_t w = cw[0];
            uint2 e[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) e[k] = T.enc[(w >> (8u * k)) & 0xFFu];
#pragma unroll 1
            for (uint32_t j = 0; j < n; j += 4u) {
                uint2 f[4];
                const bool more = j + 4u < n;
                if (more) w = cw[j / 4u + 1u];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) f[k] = T.enc[(w >> (8u * k)) & 0xFFu];
                uint32_t u[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint32_t v = out + size, nb = (v + e[k].x) >> 16, x = v >> nb;
                    u[k] = (v - (x << nb)) | (nb << 12);
                    if (j + k < n) out = T.stl[x + e[k].y];
                }
                uw[j / 2u] = u[0] | (u[1] << 16);
                uw[j / 2u + 1u] = u[2] | (u[3] << 16);
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) e[k] = f[k];
            }
            if (fresh && lane == 0u) up[0] = 0;
        }
        const uint32_t p = __shfl_up_sync(kFull, out, 1);
        again = lane > 0u && n && p != in;
        if (again) in = p;
    }
    D = __shfl_sync(kFull, out, (len - 1u) / kRun);
}

// Step R for one thread's run [i0, i1): Offset_Values from the repeat history
// r1, r2, r3, which it leaves as it is after the run.
__device__ __forceinline__ void offset_values(const uint4 *sq, uint32_t *ovg, uint32_t i0, uint32_t i1, uint32_t &r1,
                                              uint32_t &r2, uint32_t &r3) {
    uint4 q = i0 < i1 ? sq[i0] : make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t i = i0; i < i1; ++i) {
        const uint32_t o = q.x, z = q.y == 0u ? 1u : 0u;
        if (i + 1u < i1) q = sq[i + 1u];
        uint32_t v;
        if (!z) v = o == r1 ? 1u : (o == r2 ? 2u : (o == r3 ? 3u : o + 3u));
        else v = o == r2 ? 1u : (o == r3 ? 2u : (o == r1 - 1u ? 3u : o + 3u));
        const uint32_t idx = v > 3u ? 3u : v - 1u + z;
        // idx 0: rep1 kept; 1: rep2 swapped to the front; else: o in front, the rest shift
        if (idx >= 2u) r3 = r2;
        if (idx >= 1u) {
            r2 = r1;
            r1 = o;
        }
        ovg[i] = v;
    }
}

// Offset o (0: none) into a list of up to three different ones, behind those there.
__device__ __forceinline__ void recent(uint32_t &a, uint32_t &b, uint32_t &c, uint32_t o) {
    if (o == 0u || o == a || o == b || c != 0u) return;
    if (a == 0u) a = o;
    else if (b == 0u) b = o;
    else c = o;
}

// The frame's block content size, or 0 when a raw block is smaller (the whole
// CTA gets it).
__device__ uint32_t encode_sequences(const ZencArgs &a, SeqSmem &G, uint32_t b, uint32_t w, uint32_t fh,
                                     uint8_t *slot, uint32_t sec) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint64_t s0 = a.seq_offsets[b];
    const uint32_t ns = static_cast<uint32_t>(a.seq_offsets[b + 1] - s0);
    const uint4 *sq = a.seqs + s0;
    uint32_t *ovg = a.ovs + static_cast<uint64_t>(b) * kZencMaxSeqs;
    const uint32_t per = (ns + kSeqThreads - 1u) / kSeqThreads;
    const uint32_t i0 = min(tid * per, ns), i1 = min(i0 + per, ns);

    for (uint32_t k = tid; k < 64u; k += kSeqThreads) G.tab[0].hist[k] = G.tab[1].hist[k] = G.tab[2].hist[k] = 0u;
    __syncthreads();
    // ---- R: Offset_Values and code counts
    // The guessed history: the three different offsets used last before the run,
    // by a scan of each thread's own (0: none).
    uint32_t l1 = 0, l2 = 0, l3 = 0;
    for (uint32_t i = i1; i > i0 && l3 == 0u; --i) recent(l1, l2, l3, sq[i - 1u].x);
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1) {  // with those of the lanes before it
        const uint32_t a1 = __shfl_up_sync(kFull, l1, d), a2 = __shfl_up_sync(kFull, l2, d),
                       a3 = __shfl_up_sync(kFull, l3, d);
        if (lane >= d) {
            recent(l1, l2, l3, a1);
            recent(l1, l2, l3, a2);
            recent(l1, l2, l3, a3);
        }
    }
    if (lane == 31u) {
        G.out_state[0][warp] = l1;
        G.out_state[1][warp] = l2;
        G.out_state[2][warp] = l3;
    }
    uint32_t in1 = __shfl_up_sync(kFull, l1, 1), in2 = __shfl_up_sync(kFull, l2, 1), in3 = __shfl_up_sync(kFull, l3, 1);
    if (lane == 0u) in1 = in2 = in3 = 0u;
    __syncthreads();
    for (uint32_t v = warp; v > 0u; --v) {  // and of the warps before it
        recent(in1, in2, in3, G.out_state[0][v - 1u]);
        recent(in1, in2, in3, G.out_state[1][v - 1u]);
        recent(in1, in2, in3, G.out_state[2][v - 1u]);
    }
    recent(in1, in2, in3, 1u);
    recent(in1, in2, in3, 4u);
    recent(in1, in2, in3, 8u);
    __syncthreads();
    for (uint32_t i = tid; i < ns; i += kSeqThreads) {
        const uint4 q = sq[i];
        uint32_t c, nb;
        G.C.ll(q.y, c, nb);
        atomicAdd(&G.tab[0].hist[c], 1u);
        G.C.ml(q.z, c, nb);
        atomicAdd(&G.tab[1].hist[c], 1u);
    }
    for (bool again = true;;) {
        if (again) {
            uint32_t r1 = in1, r2 = in2, r3 = in3;
            offset_values(sq, ovg, i0, i1, r1, r2, r3);
            G.out_state[0][tid] = r1;
            G.out_state[1][tid] = r2;
            G.out_state[2][tid] = r3;
        }
        __syncthreads();
        again = false;
        if (tid > 0u && i0 < i1) {
            const uint32_t p1 = G.out_state[0][tid - 1u], p2 = G.out_state[1][tid - 1u], p3 = G.out_state[2][tid - 1u];
            again = p1 != in1 || p2 != in2 || p3 != in3;
            in1 = p1;
            in2 = p2;
            in3 = p3;
        }
        if (!__syncthreads_or(again)) break;  // (a thread's history is right once the one before it is)
    }
    for (uint32_t i = i0; i < i1; ++i) atomicAdd(&G.tab[2].hist[highbit(ovg[i])], 1u);
    __syncthreads();

    // ---- T: the three tables
    if (warp == 0) build_field_table(G.tab[0], ns, kLLSyms, kMaxAl, kLLNorm, kLLSyms, kLLLog);
    else if (warp == 1) build_field_table(G.tab[1], ns, kMLSyms, kMaxAl, kMLNorm, kMLSyms, kMLLog);
    else if (warp == 2) build_field_table(G.tab[2], ns, kOFCodes, 8u, kOFNorm, kOFSyms, kOFLog);
    __syncthreads();

    // header: Number_of_Sequences, modes, table descriptions (LL, OF, ML)
    uint8_t *hp = slot + sec;
    const uint32_t nsb = ns < 128u ? 1u : 2u;
    const uint32_t d_ll = G.tab[0].desc_len, d_of = G.tab[2].desc_len, d_ml = G.tab[1].desc_len;
    const uint32_t hl = nsb + 1u + d_ll + d_of + d_ml;
    if (sec + hl >= fh + 3u + w) return 0u;  // the literals alone fill the window
    if (tid == 0) {
        if (ns < 128u) {
            hp[0] = static_cast<uint8_t>(ns);
        } else {
            hp[0] = static_cast<uint8_t>((ns >> 8) + 0x80u);
            hp[1] = static_cast<uint8_t>(ns);
        }
        hp[nsb] = static_cast<uint8_t>((G.tab[0].mode << 6) | (G.tab[2].mode << 4) | (G.tab[1].mode << 2));
    }
    for (uint32_t k = tid; k < d_ll + d_of + d_ml; k += kSeqThreads) {
        const uint8_t *t0 = reinterpret_cast<const uint8_t *>(G.tab[0].desc);
        const uint8_t *t1 = reinterpret_cast<const uint8_t *>(G.tab[1].desc);
        const uint8_t *t2 = reinterpret_cast<const uint8_t *>(G.tab[2].desc);
        hp[nsb + 1u + k] = k < d_ll ? t0[k] : (k < d_ll + d_of ? t2[k - d_ll] : t1[k - d_ll - d_of]);
    }
    // ---- E: chunks in bitstream order (sequence ns - 1 - j)
    uint32_t *wslot = reinterpret_cast<uint32_t *>(slot);
    const uint32_t sb = sec + hl;                 // first byte of the stream
    const uint32_t room = 8u * (fh + 3u + w - sb);  // stream bits at which the block stops paying
    if (tid < ((4u - (sb & 3u)) & 3u)) slot[sb + tid] = 0;  // to the first whole word; the words follow chunk by chunk
    uint32_t zeroed = (sb + 3u) >> 2;             // words below are zero or written (runs OR their shared words in)
    uint32_t pos = 8u * sb, D = 0;
    for (uint32_t c0 = 0; c0 < ns; c0 += kChunk) {
        const uint32_t len = min(kChunk, ns - c0);
        for (uint32_t j = tid; j < len; j += kSeqThreads) {
            const uint32_t i = ns - 1u - c0 - j;
            const uint4 q = sq[i];
            uint32_t lc, mc, nb;
            G.C.ll(q.y, lc, nb);
            G.C.ml(q.z, mc, nb);
            G.code[0][code_at(j)] = static_cast<uint8_t>(lc);
            G.code[1][code_at(j)] = static_cast<uint8_t>(mc);
            G.code[2][code_at(j)] = static_cast<uint8_t>(highbit(ovg[i]));
        }
        if (tid < 3u)  // the chains read four codes at a time
            for (uint32_t j = len; j & 3u; ++j) G.code[tid][code_at(j)] = 0;
        __syncthreads();
        if (warp < 3u) {
            fse_chain(G.tab[warp], G.code[warp], G.upd[warp], len, c0 == 0u, D);
            if (lane == 0) G.state[warp] = D;
        }
        __syncthreads();
        const uint32_t j0 = min(tid * kOwn, len), j1 = min(j0 + kOwn, len);
        uint32_t bits = 0;
        for (uint32_t j = j0; j < j1; ++j) {
            const uint32_t u = upd_at(j), c = code_at(j);
            bits += (G.upd[0][u] >> 12) + (G.upd[1][u] >> 12) + (G.upd[2][u] >> 12) + G.C.ll_bits(G.code[0][c]) +
                    G.C.ml_bits(G.code[1][c]) + G.code[2][c];
        }
        const uint32_t incl = scan_incl(bits);
        if (lane == 31u) G.warp_bits[warp] = incl;
        __syncthreads();
        uint32_t before = incl - bits, total = 0;
#pragma unroll
        for (uint32_t k = 0; k < kSeqThreads / 32u; ++k) {
            const uint32_t x = G.warp_bits[k];
            if (k < warp) before += x;
            total += x;
        }
        if (pos + total - 8u * sb >= room) return 0u;
        // this chunk's words (and room for the final states), then its bits
        const uint32_t wend = ((pos + total + 31u) >> 5) + 1u;
        for (uint32_t k = zeroed + tid; k < wend; k += kSeqThreads) wslot[k] = 0u;
        __syncthreads();
        if (j0 < j1) {
            RunWriter wr(wslot, pos + before);
            for (uint32_t j = j0; j < j1; ++j) {
                const uint32_t u = upd_at(j), c = code_at(j), i = ns - 1u - c0 - j;
                const uint4 q = sq[i];
                const uint32_t uo = G.upd[2][u], um = G.upd[1][u], ul = G.upd[0][u];
                const uint32_t no = uo >> 12, nm = um >> 12, nl = ul >> 12;
                const uint32_t lb = G.C.ll_bits(G.code[0][c]), mb = G.C.ml_bits(G.code[1][c]), oc = G.code[2][c];
                // updates: OF, ML, LL (the decoder, reading backwards, takes LL, ML, OF); extra bits: LL, ML, OF
                wr.add((uo & 0xFFFu) | ((um & 0xFFFu) << no) | ((ul & 0xFFFu) << (no + nm)), no + nm + nl);
                wr.add((q.y & ((1u << lb) - 1u)) | (((q.z - 3u) & ((1u << mb) - 1u)) << lb), lb + mb);
                wr.add(ovg[i] - (1u << oc), oc);
            }
            wr.close();
        }
        zeroed = wend;
        pos += total;
        __syncthreads();
    }
    // the final states ML, OF, LL and the end marker
    const uint32_t al0 = G.tab[0].al, al1 = G.tab[1].al, al2 = G.tab[2].al;
    const uint32_t stream = (pos - 8u * sb + al0 + al1 + al2 + 1u + 7u) >> 3;
    const uint32_t content = sb + stream - (fh + 3u);
    if (content >= w) return 0u;
    if (tid == 0) {
        RunWriter wr(wslot, pos);
        wr.add(G.state[1], al1);
        wr.add(G.state[2], al2);
        wr.add(G.state[0], al0);
        wr.add(1u, 1u);
        wr.close();
    }
    return content;
}

__global__ void __launch_bounds__(kSeqThreads, 8) zenc_sequences_kernel(ZencArgs a) {
    __shared__ SeqSmem G;
    const uint32_t tid = threadIdx.x;
    G.C.build();
    __syncthreads();
    for (uint32_t b = blockIdx.x; b < a.num_windows; b += gridDim.x) {
        const uint32_t w = win_size(a, b);
        const uint32_t fh = frame_header_bytes(w);
        uint8_t *slot = a.slots + static_cast<uint64_t>(b) * kZencSlot;
        const uint32_t sec = a.sec_off[b];
        const uint32_t content = sec != 0u ? encode_sequences(a, G, b, w, fh, slot, sec) : 0u;
        if (tid == 0) {
            if (content) {
                write_block_header(slot + fh, 2u, content);
                a.fsize[b] = fh + 3u + content;
                a.raw[b] = 0;
            } else {
                write_block_header(slot + fh, 0u, w);
                a.fsize[b] = fh + 3u + w;
                a.raw[b] = 1;
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- compaction
// blockIdx.y of gridDim.y parts of a frame (multiples of 16 bytes): few
// windows are copied by several CTAs each.
// kScan: the frame offsets are computed here too (few windows).
template <bool kScan>
__global__ void __launch_bounds__(256) zenc_compact_kernel(ZencArgs a, uint64_t *foff, uint8_t *out,
                                                           uint64_t capacity) {
    const uint32_t tid = threadIdx.x;
    // the part [lo, hi) of n bytes
    auto copy_part = [&](uint8_t *d, const uint8_t *s, uint32_t n) {
        const uint32_t per = ((n + gridDim.y - 1u) / gridDim.y + 15u) & ~15u, lo = blockIdx.y * per;
        if (lo < n) cta_copy(d + lo, s + lo, n - lo < per ? n - lo : per);
    };
    for (uint32_t b = blockIdx.x; b < a.num_windows; b += gridDim.x) {
        uint64_t o, size;
        if constexpr (kScan) {
            o = cta_sum_before(a.fsize, b);
            size = a.fsize[b];
            if (tid == 0 && blockIdx.y == 0u) {
                foff[b] = o;
                if (b + 1u == a.num_windows) foff[b + 1u] = o + size;
            }
        } else {
            o = foff[b];
            size = foff[b + 1] - o;
        }
        if (o + size > capacity) {
            if (tid == 0) atomicOr(a.status, kErrCapacity);
            continue;
        }
        const uint8_t *slot = a.slots + static_cast<uint64_t>(b) * kZencSlot;
        uint8_t *dst = out + o;
        if (!a.raw[b]) {
            copy_part(dst, slot, static_cast<uint32_t>(size));
        } else {
            const uint32_t w = win_size(a, b);
            const uint32_t hl = frame_header_bytes(w) + 3u;
            if (blockIdx.y == 0u) cta_copy(dst, slot, hl);
            copy_part(dst + hl, win_src(a, b), w);
        }
    }
}

ZencArgs args_of(const ZencLaunch &l) {
    ZencArgs a{};
    a.src = l.src;
    a.n = l.n;
    a.window = l.window;
    a.num_windows = l.num_windows;
    a.seqs = reinterpret_cast<const uint4 *>(l.seqs);
    a.seq_offsets = l.seq_offsets;
    a.slots = l.slots;
    a.ovs = l.ovs;
    a.sec_off = l.sec_off;
    a.fsize = l.fsize;
    a.raw = l.raw;
    a.hist = l.hist;
    a.plan = l.plan;
    a.status = l.status;
    a.wins = l.wins;
    return a;
}

SmemOnce g_lit_smem_set{0}, g_plan_smem_set{0}, g_write_smem_set{0};

}  // namespace

cudaError_t launch_zenc(const ZencLaunch &l, cudaStream_t st) {
    if (l.num_windows == 0) return cudaSuccess;
    const ZencArgs a = args_of(l);
    cudaError_t e = set_smem_once(zenc_literals_kernel, sizeof(GatherSmem), g_lit_smem_set);
    if (e != cudaSuccess) return e;
    if ((e = set_smem_once(zenc_huf_plan_kernel, sizeof(PlanSmem) * kPlanWarps, g_plan_smem_set)) != cudaSuccess)
        return e;
    if ((e = set_smem_once(zenc_huf_write_kernel, kWriteSmem, g_write_smem_set)) != cudaSuccess) return e;
    int grid = l.num_sms * 2;  // two 512-thread CTAs per SM
    if (static_cast<uint32_t>(grid) > l.num_windows) grid = static_cast<int>(l.num_windows);
    zenc_literals_kernel<<<grid, kGatherThreads, sizeof(GatherSmem), st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    grid = l.num_sms * 3;
    if (static_cast<uint32_t>(grid) > l.num_windows) grid = static_cast<int>(l.num_windows);
    uint32_t pgrid = (l.num_windows + kPlanWarps - 1) / kPlanWarps;
    if (pgrid > static_cast<uint32_t>(l.num_sms * 5)) pgrid = static_cast<uint32_t>(l.num_sms * 5);
    zenc_huf_plan_kernel<<<pgrid, 32 * kPlanWarps, sizeof(PlanSmem) * kPlanWarps, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    zenc_huf_write_kernel<<<grid, kLitThreads, kWriteSmem, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    grid = l.num_sms * 8;  // 64 registers per thread
    if (static_cast<uint32_t>(grid) > l.num_windows) grid = static_cast<int>(l.num_windows);
    zenc_sequences_kernel<<<grid, kSeqThreads, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_zenc_compact(const ZencLaunch &l, uint64_t *frame_offsets, uint8_t *out, uint64_t capacity,
                                cudaStream_t st) {
    if (l.num_windows == 0) return cudaSuccess;
    const uint32_t most = static_cast<uint32_t>(l.num_sms) * 8u;
    const uint32_t grid = most < l.num_windows ? most : l.num_windows;
    // up to 16 parts of a frame (about 4 KiB each) while CTAs are left
    const uint32_t parts = grid * 16u <= most ? 16u : most / grid;
    if (l.num_windows <= kFusedScan) {
        zenc_compact_kernel<true><<<dim3(grid, parts), 256, 0, st>>>(args_of(l), frame_offsets, out, capacity);
    } else {
        const cudaError_t e = launch_scan_counts(l.fsize, l.num_windows, frame_offsets, st);
        if (e != cudaSuccess) return e;
        zenc_compact_kernel<false><<<dim3(grid, parts), 256, 0, st>>>(args_of(l), frame_offsets, out, capacity);
    }
    return cudaGetLastError();
}

}  // namespace gcz
