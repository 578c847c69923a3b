// LZMA2 L1+ match finder for sm_100a.
//
// Reproduces lzma2_match_find (lzma2_match_find.cu:54-194) bit for bit.  The
// reference walks each 64 KiB window with one thread: a one-entry 14-bit table
// (empty == 0xFFFF), the "chain" loop stops after its first candidate
// (:157-160), so every position gets at most one match:
//   - candidate = table entry for hash(q) (q+3 < size), verified on 4 bytes
//     (len 4, extended to <= min(size-q, 273)) or else on 2 bytes (len 2,
//     extended the same way, which stops at 3 at most);
//   - if there is none, a distance-1 run when src[q-1]==src[q]==src[q+1]
//     (:164-181).
// Every position with q+3 < size is inserted right after its own lookup, so
// the candidate at q is cand(q) = max{p < q : hash(p) == hash(q)} (or none):
// one warp per window computes it 32 positions per step (__match_any_sync for
// in-step predecessors, shared-memory table for earlier steps) and then every
// lane verifies and extends its own position independently.
#include <type_traits>

#include "gcz_common.cuh"
#include "gcz_kernels.h"

namespace gcz {
namespace {

constexpr uint32_t kLzmaMaxMatch = 273;  // MAX_MATCH_LEN, lzma2_match_find.cu:21
constexpr uint32_t kNone = 0xFFFFu;      // empty sentinel, :73

// First index in [len, lim) where the bytes at c+i and q+i differ, else lim.
template <class Win>
__device__ __forceinline__ uint32_t extend_lane(const Win &win, uint32_t c, uint32_t q, uint32_t len, uint32_t lim) {
    while (len < lim) {
        const uint32_t d = win.u32(q + len) ^ win.u32(c + len);
        if (d) {
            len += (static_cast<uint32_t>(__ffs(d)) - 1u) >> 3;
            return len < lim ? len : lim;
        }
        len += 4u;
    }
    return lim;
}

// First index in [len, lim) where byte q+i differs from `b`, else lim.
template <class Win>
__device__ __forceinline__ uint32_t run_lane(const Win &win, uint32_t q, uint32_t b, uint32_t len, uint32_t lim) {
    const uint32_t pat = b * 0x01010101u;
    while (len < lim) {
        const uint32_t d = win.u32(q + len) ^ pat;
        if (d) {
            len += (static_cast<uint32_t>(__ffs(d)) - 1u) >> 3;
            return len < lim ? len : lim;
        }
        len += 4u;
    }
    return lim;
}

struct LzmaArgs {
    const uint8_t *src;
    uint64_t n;
    uint32_t window;
    uint32_t num_windows;
    uint32_t search_depth;   // 0 disables the hash candidate (chain loop never runs)
    uint32_t max_matches;    // slot stride of the reference layout
    uint32_t *packed;        // compact: len<<16 | dist per position (or null)
    uint8_t *has_matches;    // per window (or null)
    uint32_t *ref_matches;   // reference layout LzmaMatch pairs (or null)
    uint32_t *ref_counts;    // reference layout counts (or null)
    uint32_t *status;
};

template <class Win>
__device__ void lzma_window(const Win &win, uint16_t *T, uint32_t size, const LzmaArgs &a, uint32_t w) {
    const uint32_t lane = lane_id();
    const uint32_t lt = lanemask_lt(), gt = lanemask_gt();
    {
        uint32_t *t32 = reinterpret_cast<uint32_t *>(T);
        for (uint32_t i = lane; i < kHashSize / 2; i += 32) t32[i] = 0xFFFFFFFFu;  // :72-74
    }
    __syncwarp();
    const uint64_t wbase = static_cast<uint64_t>(w) * a.window;
    uint32_t *packed = a.packed ? a.packed + wbase : nullptr;
    uint32_t *rc = a.ref_counts ? a.ref_counts + wbase : nullptr;
    uint32_t *rm = a.ref_matches ? a.ref_matches + wbase * a.max_matches * 2u : nullptr;
    uint32_t any = 0;
    const uint32_t nsteps = (size + 31u) >> 5;
    for (uint32_t s = 0; s < nsteps; ++s) {
        const uint32_t q = (s << 5) + lane;
        const bool valid4 = q + 3u < size;
        const uint32_t x = win.u32(q);
        const uint32_t h = hash4(x);
        const uint32_t g = __match_any_sync(kFull, valid4 ? h : (0x80000000u | lane));
        const uint32_t lower = g & lt;
        const uint32_t tv = valid4 ? static_cast<uint32_t>(T[h]) : kNone;
        const uint32_t cand = lower ? ((s << 5) + 31u - static_cast<uint32_t>(__clz(lower))) : tv;
        __syncwarp();
        if (valid4 && !(g & gt)) T[h] = static_cast<uint16_t>(q);  // :108
        __syncwarp();

        uint32_t dist = 0, len = 0;
        if (q + 1u < size) {
            if (valid4 && a.search_depth > 0 && cand != kNone) {
                const uint32_t lim = size - q < kLzmaMaxMatch ? size - q : kLzmaMaxMatch;
                const uint32_t y = win.u32(cand);
                uint32_t l = 0;
                if (y == x) {
                    l = extend_lane(win, cand, q, 4u, lim);             // :127-133
                } else if (((y ^ x) & 0xFFFFu) == 0u) {
                    l = ((y ^ x) & 0xFF0000u) == 0u ? 3u : 2u;          // :134-139 (byte 3 differs)
                }
                if (l >= 2u) {
                    dist = q - cand;
                    len = l;
                }
            }
            if (len == 0 && q > 0) {  // distance-1 run (:164-181)
                const uint32_t b0 = x & 0xFFu, b1 = (x >> 8) & 0xFFu;
                if (b1 == b0 && win.byte(q - 1u) == b0) {
                    const uint32_t lim = size - q < kLzmaMaxMatch ? size - q : kLzmaMaxMatch;
                    len = run_lane(win, q, b0, 2u, lim);
                    dist = 1;
                }
            }
        }
        if (q < size) {
            if (packed) packed[q] = len ? ((len << 16) | dist) : 0u;
            if (rc) rc[q] = len ? 1u : 0u;
            if (rm && len) {
                uint32_t *slot = rm + static_cast<uint64_t>(q) * a.max_matches * 2u;
                slot[0] = dist;
                slot[1] = len;
            }
        }
        any |= len;
    }
    if (rc)
        for (uint32_t q = size + lane; q < a.window; q += 32) rc[q] = 0u;  // :188-190
    any = __any_sync(kFull, any != 0);
    if (a.has_matches && lane == 0) a.has_matches[w] = any ? 1 : 0;
}

constexpr uint32_t kSmemData = kMaxWindow + 64;
constexpr uint32_t kSmemTable = kHashSize * sizeof(uint16_t);
constexpr uint32_t kSmemStaged = kSmemData + kSmemTable + 16;

template <bool kStaged>
__global__ void __launch_bounds__(32) lzma_match_kernel(LzmaArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint16_t *T = reinterpret_cast<uint16_t *>(smem + (kStaged ? kSmemData : 0u));
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kSmemData + kSmemTable);
    uint32_t parity = 0;
    if (kStaged) {
        if (lane_id() == 0) {
            mbar_init(bar, 1);
            fence_mbar_init();
        }
        __syncwarp();
    }
    for (uint32_t w = blockIdx.x; w < a.num_windows; w += gridDim.x) {
        const uint64_t start = static_cast<uint64_t>(w) * a.window;
        const uint32_t size = static_cast<uint32_t>(a.n - start < a.window ? a.n - start : a.window);
        if constexpr (kStaged) {
            if (!stage_window(smem, a.src + start, size, bar, parity, a.status)) return;
            SmemWin win{reinterpret_cast<const uint32_t *>(smem)};
            lzma_window(win, T, size, a, w);
        } else {
            GlobalWin win{reinterpret_cast<const uint32_t *>(a.src + start), (size + 3u) >> 2};
            lzma_window(win, T, size, a, w);
        }
    }
}

// Packed -> GpuMatchData layout (compress_lzma2_custom.rs:539-549): counts,
// and de-interleaved distance / length arrays with max_matches slots per
// position, unused slots zero (the reference allocates them with alloc_zeros).
__global__ void __launch_bounds__(256) lzma_unpack_kernel(const uint32_t *packed, uint64_t n, uint32_t window,
                                                          uint32_t num_windows, uint32_t max_matches,
                                                          uint32_t *dists, uint32_t *lens, uint32_t *counts) {
    const uint64_t total = static_cast<uint64_t>(num_windows) * window;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        // positions past n inside the last window have count 0
        const uint32_t v = i < n ? packed[i] : 0u;
        if (counts) counts[i] = v ? 1u : 0u;
        const uint64_t base = i * max_matches;
        for (uint32_t k = 0; k < max_matches; ++k) {
            if (dists) dists[base + k] = (k == 0) ? (v & 0xFFFFu) : 0u;
            if (lens) lens[base + k] = (k == 0) ? (v >> 16) : 0u;
        }
    }
}

// ---------------------------------------------------------------------------
// Second stage after the candidate sweep (gcz_sweep.cu): the window is staged
// into shared memory, cand(q) streams in from global memory, and every lane
// verifies four consecutive positions, 128 per warp iteration.
//
// Lengths come from the ends of match runs.  Where q and q+1 both match on 4
// bytes and cand(q+1) == cand(q) + 1, both matches end at the same byte, so
// only a run's last position needs a comparison (about five of 128 positions
// on the synthetic data, gathered and shared out to the lanes).  Each warp goes through its part of the window from
// the back, so that a run's end is known when its earlier positions come up:
// inside a lane, from the next lane that holds a run's end (one ballot, one
// shuffle), or carried over from the block after it.  The cap of 273 bytes is
// applied to the end of each run and again per position.
//
// Two cases need no comparison loop.  A candidate that fails on 4 bytes
// matches on 2 at most: it has the same 14 upper bits of v * K (K odd), and
// two values v that agree in their low 24 bits and differ above differ in the
// upper 8 bits of the product.  A distance-1 run (lzma2_match_find.cu:164-181)
// is looked for only where the candidate fails; four equal bytes after an
// equal one would have made q-1 a candidate that matches, so it is 2 or 3 long
// (with search_depth 0 there are no candidates, and it is measured).
//
// What bounds it: instruction issue.  One lane per position and one warp-wide
// extension per run head took 378 K warp instructions per window, 6.55 ms per
// GiB of the synthetic data; this form takes 199 K and 4.1 ms (the memory's own
// time for cand, input and output would be 1.2 ms).
constexpr uint32_t kL2Pre = 64;
constexpr uint32_t kL2DataBytes = kL2Pre + kMaxWindow + 64;

struct L2Smem {
    uint8_t data[kL2DataBytes];
    uint32_t any;
    uint32_t flags;
    alignas(16) uint64_t bar;
};

struct L2Args {
    const uint8_t *src;
    const uint16_t *cand;
    uint64_t n;
    uint32_t window;
    uint32_t num_windows;
    uint32_t search_depth;
    uint32_t max_matches;
    uint32_t *packed;
    uint8_t *has_matches;
    uint32_t *ref_matches;
    uint32_t *ref_counts;
    uint32_t *status;
    const WinDesc *wins;
    uint32_t parts;  // CTAs that share a window (a cluster), 1, 2, 4 or 8
};

// Cluster barrier: every thread of the window's CTAs; shared-memory writes
// before it are visible to them after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The 32-bit word at `p`'s place in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_read(const uint32_t *p, uint32_t rank) {
    uint32_t a, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// The candidates of positions q .. q+3 (none past the window).
__device__ __forceinline__ uint2 load_cand4(const uint16_t *cand, uint32_t q, uint32_t size) {
    if (q + 4u <= size) return *reinterpret_cast<const uint2 *>(cand + q);
    uint32_t e[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) e[k] = q + k < size ? static_cast<uint32_t>(cand[q + k]) : kNone;
    return make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
}

// Lanes with `open` have k equal bytes at (c, q) and compare on, up to lim
// (left: bytes to the window's end): one lane at a time, the whole warp 128
// bytes per iteration.  Open lanes inside the same stretch of equal bytes at
// the same distance share its end.
__device__ __forceinline__ uint32_t finish_long(const SmemWin &win, uint32_t c, uint32_t q, uint32_t k, uint32_t lim,
                                                uint32_t left, bool open) {
    const uint32_t lane = lane_id();
    for (uint32_t pend; (pend = __ballot_sync(kFull, open)) != 0u;) {
        const uint32_t hl = static_cast<uint32_t>(__ffs(pend)) - 1u;
        const uint32_t hc = __shfl_sync(kFull, c, hl), hq = __shfl_sync(kFull, q, hl);
        const uint32_t hb = __shfl_sync(kFull, lim, hl);
        const uint32_t h0 = __shfl_sync(kFull, k, hl);
        uint32_t len = h0;
        for (;;) {
            const uint32_t i = len + 4u * lane;
            uint32_t res = i;
            if (i < hb) {
                const uint32_t d = win.u32(hq + i) ^ win.u32(hc + i);
                const uint32_t fb = d ? (static_cast<uint32_t>(__ffs(d)) - 1u) >> 3 : 4u;
                res = i + (fb < hb - i ? fb : hb - i);
            }
            const uint32_t sb = __ballot_sync(kFull, res < i + 4u);
            if (sb) {
                len = __shfl_sync(kFull, res, static_cast<uint32_t>(__ffs(sb)) - 1u);
                break;
            }
            len += 128u;
        }
        const uint32_t end = hq + len;  // a mismatch or the window's end, unless the cap of lane hl came first
        const bool real = len < hb || hb == __shfl_sync(kFull, left, hl);
        if (lane == hl) {
            k = len;
            open = false;
        } else if (open && real && q - c == hq - hc && q + k >= hq + h0 && q + k <= end) {
            k = end - q < lim ? end - q : lim;
            open = false;
        }
    }
    return k;
}

// Two rare cases of positions q .. q+3, whose packed results so far are `out`:
// a candidate that fails on 4 bytes but matches on 2 comes before a run, and
// with search_depth 0 a run is measured.  A call of its own, so that the step
// loop holds no registers for it.
__device__ __noinline__ uint4 short_matches(SmemWin win, uint2 cc, uint32_t q, uint32_t size, uint32_t depth,
                                            uint4 out) {
#pragma unroll 1
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t p = q + k;
        const uint32_t c = ((k & 2u ? cc.y : cc.x) >> (16u * (k & 1u))) & 0xFFFFu;
        uint32_t o = k == 0u ? out.x : (k == 1u ? out.y : (k == 2u ? out.z : out.w));
        if (c != kNone) {
            const uint32_t d = win.u32(c) ^ win.u32(p);
            if (d != 0u && (d & 0xFFFFu) == 0u) o = (2u << 16) | (p - c);
        } else if (o && depth == 0) {
            const uint32_t lim = size - p < kLzmaMaxMatch ? size - p : kLzmaMaxMatch;
            o = (run_lane(win, p, win.byte(p), 2u, lim) << 16) | 1u;
        }
        if (k == 0u) out.x = o;
        else if (k == 1u) out.y = o;
        else if (k == 2u) out.z = o;
        else out.w = o;
    }
    return out;
}

// kL2Threads (256, 512 or 1024) is a schedule knob: the window's 128-position
// blocks are split into kL2Threads / 32 contiguous ranges, one per warp.
// kRefOut: the reference layout's per-position counts and match slots are
// written too (the parity entry points); without it the loop carries no code
// for them.  Few windows: a.parts CTAs share each one, their warps' ranges side
// by side (every CTA stages the whole window).
template <uint32_t kL2Threads, bool kRefOut>
__global__ void __launch_bounds__(kL2Threads, kL2Threads == 1024 ? 2 : 3) lzma_verify_kernel(L2Args a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    L2Smem &S = *reinterpret_cast<L2Smem *>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t lt = lanemask_lt(), gt = lanemask_gt();
    uint32_t *ends = reinterpret_cast<uint32_t *>(smem_raw + sizeof(L2Smem)) + warp * 128u;  // of one block's tails
    uint32_t parity = 0;
    if (tid == 0) {
        mbar_init(&S.bar, 1);
        fence_mbar_init();
    }
    for (uint32_t i = tid; i < kL2Pre / 4; i += kL2Threads) reinterpret_cast<uint32_t *>(S.data)[i] = 0u;
    __syncthreads();
    const uint32_t *W = reinterpret_cast<const uint32_t *>(S.data + kL2Pre);
    const SmemWin win{W};
    constexpr bool kSplit = kL2Threads == 1024;
    const uint32_t parts = kSplit ? a.parts : 1u, part = kSplit ? blockIdx.x % parts : 0u;  // rank in the cluster
    for (uint32_t wi = blockIdx.x / parts; wi < a.num_windows; wi += gridDim.x / parts) {
        const uint64_t start = a.wins ? a.wins[wi].offset : static_cast<uint64_t>(wi) * a.window;
        const uint32_t size =
            a.wins ? a.wins[wi].size : static_cast<uint32_t>(a.n - start < a.window ? a.n - start : a.window);
        __syncthreads();
        if (tid == 0) {
            S.any = 0;
            S.flags = 0;
        }
        __syncthreads();
        if (warp == 0) {
            if (!stage_window(S.data + kL2Pre, a.src + start, size, &S.bar, parity, a.status) && lane == 0)
                S.flags = 1u;
        }
        __syncthreads();
        const bool failed = S.flags != 0u;  // the bulk copy never completed: status recorded, every thread leaves below
        const uint16_t *cand = a.cand + start;
        uint32_t *packed = a.packed ? a.packed + start : nullptr;
        const bool al16 = (reinterpret_cast<uintptr_t>(packed) & 15u) == 0u;
        uint32_t *rc = kRefOut && a.ref_counts ? a.ref_counts + start : nullptr;
        uint32_t *rm = kRefOut && a.ref_matches ? a.ref_matches + start * a.max_matches * 2u : nullptr;
        uint32_t any = 0;
        const uint32_t nblk = failed ? 0u : (size + 127u) >> 7;
        constexpr uint32_t kL2Warps = kL2Threads / 32;
        const uint32_t warps = parts * kL2Warps, gw = part * kL2Warps + warp;
        const uint32_t per = (nblk + warps - 1u) / warps;
        const uint32_t b0 = gw * per < nblk ? gw * per : nblk, b1 = b0 + per < nblk ? b0 + per : nblk;
        // Of the position after the block: candidate, 4-byte match (bit 16)
        // and the end of its run.  Not known after a warp's last block.
        constexpr uint32_t kUnknown = ~0u;
        uint32_t after = kUnknown, after_end = 0;
        uint2 cn = b1 > b0 ? load_cand4(cand, (b1 - 1u) * 128u + 4u * lane, size) : make_uint2(~0u, ~0u);
        for (uint32_t blk = b1; blk-- > b0;) {
            const uint32_t q = blk * 128u + 4u * lane, i = q >> 2;
            // (search_depth 0: the chain loop never runs)
            const uint2 cc = a.search_depth ? cn : make_uint2(~0u, ~0u);
            const uint32_t c[4] = {cc.x & 0xFFFFu, cc.x >> 16, cc.y & 0xFFFFu, cc.y >> 16};
            if (blk > b0) cn = load_cand4(cand, q - 128u, size);  // arrives while this block is worked on
            const uint32_t x0 = W[i], x1 = W[i + 1u];
            const uint32_t xm = W[static_cast<int>(i) - 1];
            bool eq[4], rare = false;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                // none: word 16383, inside the window's buffer (the shift counts modulo 32)
                const uint32_t *y = reinterpret_cast<const uint32_t *>(S.data + kL2Pre + (c[k] & 0xFFFCu));
                const uint32_t d = __funnelshift_r(y[0], y[1], c[k] << 3) ^ (k ? __funnelshift_r(x0, x1, 8u * k) : x0);
                eq[k] = d == 0u && c[k] != kNone;
                rare = rare || ((d & 0xFFFFu) == 0u && !eq[k]);  // fails on 4 bytes, may match on 2
            }
            // What follows each position: the next one's candidate and 4-byte
            // match; the run goes on when that is this one's candidate plus 0x10001.
            uint32_t v[5];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) v[k] = eq[k] ? c[k] + 0x10000u : c[k];
            v[4] = __shfl_down_sync(kFull, v[0], 1);
            if (lane == 31u) v[4] = after;
            uint32_t E[4];      // end of the run at a run's last position
            bool tail[4];
            uint32_t rank[4], ntail = 0;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                tail[k] = eq[k] && v[k + 1u] - c[k] != 0x10001u;
                const uint32_t m = __ballot_sync(kFull, tail[k]);
                rank[k] = ntail + static_cast<uint32_t>(__popc(m & lt));
                ntail += static_cast<uint32_t>(__popc(m));
            }
            if (ntail) {
                // Five positions of the 128 on average: spread over the lanes through shared memory.
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k)
                    if (tail[k]) ends[rank[k]] = (q + k) | (c[k] << 16);
                __syncwarp();
                for (uint32_t t0 = 0; t0 < ntail; t0 += 32u) {
                    const uint32_t t = t0 + lane;
                    const uint32_t e = t < ntail ? ends[t] : 0u;
                    const uint32_t tq = e & 0xFFFFu, tc = e >> 16;
                    const uint32_t left = size - tq, lim = left < kLzmaMaxMatch ? left : kLzmaMaxMatch;
                    uint32_t len = 4u;
                    bool open = false;
                    if (t < ntail) {
                        uint32_t ql, qh, cl, ch;
                        win.u64(tq + 4u, ql, qh);
                        win.u64(tc + 4u, cl, ch);
                        const uint32_t dl = ql ^ cl, dh = qh ^ ch;
                        const uint32_t fb = dl ? (static_cast<uint32_t>(__ffs(dl)) - 1u) >> 3
                                               : (dh ? 4u + ((static_cast<uint32_t>(__ffs(dh)) - 1u) >> 3) : 8u);
                        len = 4u + fb < lim ? 4u + fb : lim;
                        open = fb == 8u && lim > 12u;
                    }
                    if (__any_sync(kFull, open)) len = finish_long(win, tc, tq, len, lim, left, open);
                    if (t < ntail) ends[t] = tq + len;
                }
                __syncwarp();
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) E[k] = tail[k] ? ends[rank[k]] : 0u;
            if (ntail) __syncwarp();
            // ends of the runs that go on past their lane
            const bool has_tail = tail[0] || tail[1] || tail[2] || tail[3];
            const uint32_t first = tail[0] ? E[0] : (tail[1] ? E[1] : (tail[2] ? E[2] : E[3]));
            const uint32_t later = __ballot_sync(kFull, has_tail) & gt;
            const uint32_t fl = __shfl_sync(kFull, first, later ? static_cast<uint32_t>(__ffs(later)) - 1u : 0u);
            uint32_t run_end = later ? fl : after_end;
            // distance-1 runs: byte t of D is zero where bytes q-1+t and q+t are equal;
            // flags at bit 8k + 7 of two (f2) and three (f3) equal bytes from q + k
            const uint32_t D0 = __funnelshift_r(xm, x0, 24) ^ x0, D1 = __funnelshift_r(x0, x1, 24) ^ x1;
            const uint32_t z0 = ~(((D0 & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | D0 | 0x7F7F7F7Fu);
            const uint32_t z1 = ~(((D1 & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | D1 | 0x7F7F7F7Fu);
            uint32_t f2 = z0 & __funnelshift_r(z0, z1, 8), f3 = f2 & __funnelshift_r(z0, z1, 16);
            if (blk == 0u && lane == 0u) f2 &= ~0x80u;  // position 0 has no byte before it
            if (blk + 2u >= nblk) {                     // bytes past the window are not equal to anything
                const uint32_t n2 = size - 1u > q ? size - 1u - q : 0u, n3 = n2 ? n2 - 1u : 0u;
                f2 = n2 < 4u ? f2 & ((1u << (8u * n2)) - 1u) : f2;
                f3 = n3 < 4u ? f3 & ((1u << (8u * n3)) - 1u) : f3;
            }
            uint32_t out[4];
#pragma unroll
            for (int k = 3; k >= 0; --k) {
                const uint32_t p = q + static_cast<uint32_t>(k), bit = 0x80u << (8 * k);
                if (tail[k]) run_end = E[k];
                const uint32_t e = run_end - p;
                const uint32_t run = (f2 & bit) ? ((f3 & bit) ? 0x30001u : 0x20001u) : 0u;
                out[k] = eq[k] ? min(e, kLzmaMaxMatch) * 65536u + (p - c[k]) : run;
            }
            if (rare || a.search_depth == 0) {
                const uint4 o = short_matches(win, cc, q, size, a.search_depth, make_uint4(out[0], out[1], out[2], out[3]));
                out[0] = o.x;
                out[1] = o.y;
                out[2] = o.z;
                out[3] = o.w;
            }
            any |= out[0] | out[1] | out[2] | out[3];
            if constexpr (kRefOut) {
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint32_t p = q + k;
                    if (p >= size) continue;
                    if (rc) rc[p] = out[k] ? 1u : 0u;
                    if (rm && out[k]) {
                        uint32_t *slot = rm + static_cast<uint64_t>(p) * a.max_matches * 2u;
                        slot[0] = out[k] & 0xFFFFu;
                        slot[1] = out[k] >> 16;
                    }
                }
            }
            // of position q of lane 0, for the block before this one (a position
            // past the window has no match, so out[] and any need no guard)
            after = __shfl_sync(kFull, v[0], 0);
            after_end = __shfl_sync(kFull, run_end, 0);
            if (packed) {
                if (al16 && q + 4u <= size) {
                    *reinterpret_cast<uint4 *>(packed + q) = make_uint4(out[0], out[1], out[2], out[3]);
                } else {
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k)
                        if (q + k < size) packed[q + k] = out[k];
                }
            }
        }
        if (kRefOut && rc && part == 0u && !failed)
            for (uint32_t q = size + tid; q < a.window; q += kL2Threads) rc[q] = 0u;  // :188-190
        if (__any_sync(kFull, any != 0) && lane == 0) S.any = 1u;
        if (parts == 1u) {
            __syncthreads();
            if (tid == 0 && a.has_matches && !failed) a.has_matches[wi] = S.any ? 1 : 0;
        } else {
            cluster_sync();
            if (tid == 0 && part == 0u && a.has_matches) {
                uint32_t m = 0;
                for (uint32_t r = 0; r < parts; ++r) m |= cluster_read(&S.any, r);
                a.has_matches[wi] = m ? 1 : 0;
            }
            cluster_sync();  // no CTA leaves while its word is read
        }
        if (failed) return;
    }
}

}  // namespace

cudaError_t launch_lzma_match(const LzmaLaunch &l, cudaStream_t st) {
    LzmaArgs a{};
    a.src = l.src;
    a.n = l.n;
    a.window = l.window;
    a.num_windows = l.num_windows;
    a.search_depth = l.search_depth;
    a.max_matches = l.max_matches;
    a.packed = l.packed;
    a.has_matches = l.has_matches;
    a.ref_matches = l.ref_matches;
    a.ref_counts = l.ref_counts;
    a.status = l.status;
    if (a.num_windows == 0) return cudaSuccess;
    const bool staged = l.staged != 0;
    int grid = l.num_sms * (staged ? 2 : 6);
    if (static_cast<uint32_t>(grid) > a.num_windows) grid = static_cast<int>(a.num_windows);
    const uint32_t smem = staged ? kSmemStaged : kSmemTable;
    cudaError_t e;
    if (staged) {
        { static SmemOnce smem_set_1{0}; e = set_smem_once(lzma_match_kernel<true>, smem, smem_set_1); }
        if (e != cudaSuccess) return e;
        lzma_match_kernel<true><<<grid, 32, smem, st>>>(a);
    } else {
        { static SmemOnce smem_set_2{0}; e = set_smem_once(lzma_match_kernel<false>, smem, smem_set_2); }
        if (e != cudaSuccess) return e;
        lzma_match_kernel<false><<<grid, 32, smem, st>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t launch_lzma_unpack(const uint32_t *packed, uint64_t n, uint32_t window, uint32_t num_windows,
                               uint32_t max_matches, uint32_t *dists, uint32_t *lens, uint32_t *counts, int num_sms,
                               cudaStream_t st) {
    if (num_windows == 0) return cudaSuccess;
    lzma_unpack_kernel<<<num_sms * 8, 256, 0, st>>>(packed, n, window, num_windows, max_matches, dists, lens, counts);
    return cudaGetLastError();
}

namespace {
template <uint32_t kThreads, bool kRefOut>
cudaError_t launch_verify_variant(const L2Args &args, const LzmaLaunch &l, cudaStream_t st) {
    const uint32_t smem = sizeof(L2Smem) + kThreads / 32 * 128 * sizeof(uint32_t);
    static_assert((sizeof(L2Smem) + kThreads * 16 + 1024) * (kThreads == 1024 ? 2 : 3) <= 233472, "CTAs of one wave must fit");
    static SmemOnce smem_set{0};
    cudaError_t e = set_smem_once(lzma_verify_kernel<kThreads, kRefOut>, smem, smem_set);
    if (e != cudaSuccess) return e;
    // no more CTAs than fit on the SMs at once, so that no CTA waits for a second wave
    const int fit = kThreads == 1024 ? 2 : 3;
    int grid = l.num_sms * (l.ctas_per_sm > 0 && l.ctas_per_sm < fit ? l.ctas_per_sm : fit);
    // Windows for at most half of the CTAs that fit: 2, 4 or 8 CTAs each, of at
    // least 8 KiB on average (48 windows: 74 -> 58 us, 1 window: 64 -> 35
    // us, sweep included; a 4 KiB window gains nothing).
    L2Args a = args;
    a.parts = 1;
    while (kThreads == 1024 && a.parts < 8u && a.parts * 2u * l.num_windows <= static_cast<uint32_t>(l.num_sms * fit) &&
           l.n / l.num_windows >= a.parts * 2u * 8192u)
        a.parts *= 2u;
    if (static_cast<uint32_t>(grid) > l.num_windows) grid = static_cast<int>(l.num_windows);
    if (a.parts == 1u) {
        lzma_verify_kernel<kThreads, kRefOut><<<grid, kThreads, smem, st>>>(a);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(l.num_windows * a.parts);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = a.parts;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, lzma_verify_kernel<kThreads, kRefOut>, a);
}
}  // namespace

cudaError_t launch_lzma_verify(const LzmaLaunch &l, const uint16_t *cand, cudaStream_t st) {
    if (l.num_windows == 0) return cudaSuccess;
    L2Args a{};
    a.src = l.src;
    a.cand = cand;
    a.n = l.n;
    a.window = l.window;
    a.num_windows = l.num_windows;
    a.search_depth = l.search_depth;
    a.max_matches = l.max_matches;
    a.packed = l.packed;
    a.has_matches = l.has_matches;
    a.ref_matches = l.ref_matches;
    a.ref_counts = l.ref_counts;
    a.status = l.status;
    a.wins = l.wins;
    if (a.ref_counts || a.ref_matches) {
        if (l.threads == 256) return launch_verify_variant<256, true>(a, l, st);
        if (l.threads == 512) return launch_verify_variant<512, true>(a, l, st);
        return launch_verify_variant<1024, true>(a, l, st);
    }
    // 1024 threads finish a window soonest (1 window: 64 us against 90 for 256
    // threads, 256 windows 115 against 124); once there are several windows per
    // CTA, 256 threads with their 64 registers have the higher throughput
    // (1036 windows 390 us against 407, 16384 windows 5.11 ms against 5.25).
    const bool many = l.num_windows > 6u * static_cast<uint32_t>(l.num_sms);
    if (l.threads == 256 || (l.threads != 512 && many)) return launch_verify_variant<256, false>(a, l, st);
    if (l.threads == 512) return launch_verify_variant<512, false>(a, l, st);
    return launch_verify_variant<1024, false>(a, l, st);
}

}  // namespace gcz
