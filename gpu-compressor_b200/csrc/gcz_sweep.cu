// Candidate sweep shared by the Zstd and LZMA2 match finders.
//
// Both reference kernels keep a one-entry 14-bit table per 64 KiB window and
// write every position p with p+3 < size into it exactly once, in increasing
// order, each lookup at q happening after all p < q were written
// (zstd_compress.cu:231-235,280,303,328-331; lzma2_match_find.cu:104-108).  The
// candidate either of them sees at q is therefore
//     cand(q) = max{ p < q : hash4(p) == hash4(q) }       (none: 0xFFFF, the
// LZMA2 table's empty entry; or 0, the Zstd one's, which stands for position 0)
// which this kernel computes for every position of every window; the match
// finders then verify, extend and parse from it.
//
// Lookup and insertion are one shared-memory exchange per position: the entry
// is {window epoch, position}, and what the exchange returns is the position
// that was there.  One warp instruction covers 32 positions, lane l the l-th.
// The lanes of one instruction that hit the same bucket are applied in some
// order; on sm_100a that order is ascending, which makes every returned value
// the candidate, equal hashes inside the step included.  Nothing rests on it:
// the exchanges of a bucket form one chain, and if every one of them returns
// an entry below its own, the chain ascends and each value is the highest
// position before it.  A single returned entry that is not below its own makes
// the CTA sweep its windows again with the lanes grouped first
// (__match_any_sync), which is exact whatever the order.
//
// One window per CTA at a time, three CTAs (64 KiB tables) per SM.  The CTA's
// warps take turns, 512 positions each, in window order: a warp hashes its
// chunk before its turn and writes its candidates after it, so that the turn
// is sixteen exchanges and a named-barrier handover.  The epoch in the entries
// marks earlier windows' positions as empty, so that the table is cleared once
// per launch (and every 65535 windows) and the turns run on from one window to
// the next.
#include "gcz_common.cuh"
#include "gcz_kernels.h"

namespace gcz {
namespace {

struct SweepArgs {
    const uint8_t *src;
    uint64_t n;
    uint32_t window;
    uint32_t num_windows;
    uint16_t *cand;  // one entry per input byte, same offsets as src
    const WinDesc *wins;
    uint32_t zero_windows;  // windows whose positions without a candidate get 0 (0xFFFF in the others)
};

constexpr uint32_t kChunkSteps = 16;                 // exchanges of one turn
constexpr uint32_t kChunkPos = 32u * kChunkSteps;    // positions of one turn
constexpr uint32_t kSweepCtas = 3;                   // per SM: 3 x (64 KiB table + hash buffers)

template <int kWarps>
struct SweepSmem {
    uint32_t T[kHashSize];
    uint16_t h[kWarps][kChunkPos];  // a warp's chunk: byte offsets of its positions' buckets in T
    uint32_t redo;
};

__device__ __forceinline__ void window_of(const SweepArgs &a, uint32_t w, uint64_t &start, uint32_t &size) {
    start = a.wins ? a.wins[w].offset : static_cast<uint64_t>(w) * a.window;
    size = a.wins ? a.wins[w].size : static_cast<uint32_t>(a.n - start < a.window ? a.n - start : a.window);
}

// The words of one chunk: lane l holds words 2l, 2l+1 of each half (256
// positions), lane 31 also the first word after the chunk.  0 past the window.
struct ChunkWords {
    uint2 a, b;
    uint32_t next;
};
__device__ __forceinline__ uint2 load_words(const uint32_t *src32, uint32_t nwords, uint32_t i) {
    if (i + 1u < nwords) return __ldg(reinterpret_cast<const uint2 *>(src32 + i));
    return make_uint2(i < nwords ? __ldg(src32 + i) : 0u, 0u);
}
__device__ __forceinline__ ChunkWords load_chunk(const uint32_t *src32, uint32_t nwords, uint32_t ch) {
    const uint32_t lane = lane_id(), i = ch * (kChunkPos / 4u) + 2u * lane, e = (ch + 1u) * (kChunkPos / 4u);
    ChunkWords w;
    w.a = load_words(src32, nwords, i);
    w.b = load_words(src32, nwords, i + 64u);
    w.next = lane == 31u && e < nwords ? __ldg(src32 + e) : 0u;
    return w;
}

// The bucket offsets (4 * hash4) of the eight positions whose bytes start in
// w, packed in pairs; nx: the word after w.
__device__ __forceinline__ uint4 bucket_offsets(uint2 w, uint32_t nx) {
    uint32_t p[8];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        p[k] = (k ? __funnelshift_r(w.x, w.y, 8u * k) : w.x) * kHashMul;
        p[4 + k] = (k ? __funnelshift_r(w.y, nx, 8u * k) : w.y) * kHashMul;
    }
    // hash4 = product >> 18, so 4 * hash4 is the product's upper half without its two low bits
    uint4 r;
    r.x = __byte_perm(p[0], p[1], 0x7632) & 0xFFFCFFFCu;
    r.y = __byte_perm(p[2], p[3], 0x7632) & 0xFFFCFFFCu;
    r.z = __byte_perm(p[4], p[5], 0x7632) & 0xFFFCFFFCu;
    r.w = __byte_perm(p[6], p[7], 0x7632) & 0xFFFCFFFCu;
    return r;
}

// Named barrier between the warp whose turn ends (arrive) and the next (sync).
__device__ __forceinline__ void turn_wait(uint32_t id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void turn_pass(uint32_t id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }

// Candidates of one window by one warp, 32 positions per step with the lanes
// grouped by hash first: exact for any order of colliding lanes.  T: a table
// of kHashSize entries (one warp at a time).
__device__ void sweep_window_grouped(uint32_t *T, uint16_t *out, const uint32_t *src32, uint32_t size,
                                     uint32_t none) {
    const uint32_t lane = lane_id(), lt = lanemask_lt(), gt = lanemask_gt();
    const uint32_t nwords = (size + 3u) >> 2;
    for (uint32_t i = lane; i < kHashSize; i += 32u) T[i] = none;
    __syncwarp();
    for (uint32_t q = lane; q - lane < size; q += 32u) {
        const bool v = q + 3u < size;
        const uint32_t i = q >> 2;
        const uint32_t x = i < nwords ? __ldg(src32 + i) : 0u, y = i + 1u < nwords ? __ldg(src32 + i + 1u) : 0u;
        const uint32_t h = hash4(__funnelshift_r(x, y, (q & 3u) * 8u));
        const uint32_t g = __match_any_sync(kFull, v ? h : (0x80000000u | lane));
        const uint32_t lower = g & lt;
        uint32_t c = v ? T[h] : none;
        if (lower) c = q - lane + 31u - static_cast<uint32_t>(__clz(lower));
        __syncwarp();
        if (v && !(g & gt)) T[h] = q;
        __syncwarp();
        if (q < size) out[q] = static_cast<uint16_t>(c);
    }
}

// kWarps warps take turns on a window (a schedule knob, 4-7).  kDescending: the
// steps of a turn are exchanged last to first, an order that the check finds
// wherever two of a turn's positions share a bucket (selftest).
template <int kWarps, bool kDescending>
__global__ void __launch_bounds__(32 * kWarps, kSweepCtas) cand_sweep_kernel(SweepArgs a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    SweepSmem<kWarps> &S = *reinterpret_cast<SweepSmem<kWarps> *>(smem_raw);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    constexpr uint32_t kThreads = 32u * kWarps;
    auto clear = [&] {
        uint4 *T4 = reinterpret_cast<uint4 *>(S.T);
        for (uint32_t i = tid; i < kHashSize / 4; i += kThreads) T4[i] = make_uint4(0u, 0u, 0u, 0u);
    };
    if (tid == 0) S.redo = 0u;
    clear();
    __syncthreads();
    bool bad = false;
    uint32_t first = 0;  // warp whose turn the window's first chunk is
    uint32_t epoch = 0;
    bool begun = false;  // some chunk of this CTA has been handed out
    for (uint32_t w = blockIdx.x; w < a.num_windows; w += gridDim.x) {
        if (++epoch == 0x10000u) {
            __syncthreads();
            clear();
            __syncthreads();
            epoch = 1u;
        }
        uint64_t start;
        uint32_t size;
        window_of(a, w, start, size);
        const uint32_t *src32 = reinterpret_cast<const uint32_t *>(a.src + start);
        uint16_t *out = a.cand + start;
        const uint32_t nwords = (size + 3u) >> 2;
        const uint32_t nch = (size + kChunkPos - 1u) / kChunkPos;
        const bool last_window = a.num_windows - w <= gridDim.x;
        const uint32_t none = w < a.zero_windows ? 0u : 0xFFFFu;
        uint32_t ch = warp >= first ? warp - first : warp + kWarps - first;  // this warp's first chunk
        ChunkWords cw = load_chunk(src32, nwords, ch);
        for (; ch < nch; ch += kWarps) {
            uint32_t nx = __shfl_down_sync(kFull, cw.a.x, 1);
            const uint32_t b0 = __shfl_sync(kFull, cw.b.x, 0);
            if (lane == 31u) nx = b0;
            uint32_t ny = __shfl_down_sync(kFull, cw.b.x, 1);
            if (lane == 31u) ny = cw.next;
            uint4 *hb = reinterpret_cast<uint4 *>(S.h[warp]);
            hb[lane] = bucket_offsets(cw.a, nx);
            hb[32u + lane] = bucket_offsets(cw.b, ny);
            __syncwarp();
            cw = load_chunk(src32, nwords, ch + kWarps);  // the next chunk's words arrive while others take turns
            uint32_t h[kChunkSteps], old[kChunkSteps];
#pragma unroll
            for (uint32_t j = 0; j < kChunkSteps; ++j) h[j] = S.h[warp][32u * j + lane];
            const uint32_t q0 = ch * kChunkPos + lane, e0 = epoch << 16;
            uint8_t *T = reinterpret_cast<uint8_t *>(S.T);
            if (begun || ch > 0u) turn_wait(1u + warp);
            const bool full = (ch + 1u) * kChunkPos + 3u <= size;  // every position has its four bytes
            if (full) {
#pragma unroll
                for (uint32_t i = 0; i < kChunkSteps; ++i) {
                    const uint32_t j = kDescending ? kChunkSteps - 1u - i : i;
                    old[j] = atomicExch(reinterpret_cast<uint32_t *>(T + h[j]), e0 + q0 + 32u * j);
                }
            } else {
#pragma unroll
                for (uint32_t i = 0; i < kChunkSteps; ++i) {
                    const uint32_t j = kDescending ? kChunkSteps - 1u - i : i;
                    old[j] = 0u;
                    if (q0 + 32u * j + 3u < size)
                        old[j] = atomicExch(reinterpret_cast<uint32_t *>(T + h[j]), e0 + q0 + 32u * j);
                }
            }
            if (!(last_window && ch + 1u == nch)) turn_pass(1u + (warp + 1u == kWarps ? 0u : warp + 1u));
#pragma unroll
            for (uint32_t j = 0; j < kChunkSteps; ++j) {
                const uint32_t q = q0 + 32u * j;
                bad = bad || old[j] >= e0 + q;
                const uint32_t c = old[j] - e0;  // an earlier epoch's entry is below e0: none
                if (full || q < size) out[q] = static_cast<uint16_t>(c < 0x10000u ? c : none);
            }
        }
        if (nch) begun = true;
        first = (first + nch) % kWarps;
    }
    if (bad) S.redo = 1u;
    __syncthreads();
    if (S.redo && warp == 0) {
        for (uint32_t w = blockIdx.x; w < a.num_windows; w += gridDim.x) {
            uint64_t start;
            uint32_t size;
            window_of(a, w, start, size);
            sweep_window_grouped(S.T, a.cand + start, reinterpret_cast<const uint32_t *>(a.src + start), size,
                                 w < a.zero_windows ? 0u : 0xFFFFu);
            __syncwarp();
        }
    }
}

template <int kWarps, bool kDescending>
cudaError_t launch_sweep_variant(const SweepArgs &a, int num_sms, cudaStream_t st) {
    const uint32_t smem = sizeof(SweepSmem<kWarps>);
    static_assert((sizeof(SweepSmem<kWarps>) + 1024) * kSweepCtas <= 233472, "three CTAs per SM must fit");
    static SmemOnce smem_set{0};
    cudaError_t e = set_smem_once(cand_sweep_kernel<kWarps, kDescending>, smem, smem_set);
    if (e != cudaSuccess) return e;
    uint32_t ctas = static_cast<uint32_t>(num_sms) * kSweepCtas;
    if (ctas > a.num_windows) ctas = a.num_windows;
    cand_sweep_kernel<kWarps, kDescending><<<ctas, 32 * kWarps, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_cand_sweep(const uint8_t *src, uint64_t n, uint32_t window, uint32_t num_windows, uint16_t *cand,
                              uint32_t zero_windows, int num_sms, cudaStream_t st, const WinDesc *wins,
                              int sweep_warps, bool descending) {
    if (num_windows == 0) return cudaSuccess;
    SweepArgs a{src, n, window, num_windows, cand, wins, zero_windows};
    if (descending) return launch_sweep_variant<7, true>(a, num_sms, st);
    switch (sweep_warps) {
    case 4: return launch_sweep_variant<4, false>(a, num_sms, st);
    case 5: return launch_sweep_variant<5, false>(a, num_sms, st);
    case 6: return launch_sweep_variant<6, false>(a, num_sms, st);
    default: return launch_sweep_variant<7, false>(a, num_sms, st);
    }
}

}  // namespace gcz
