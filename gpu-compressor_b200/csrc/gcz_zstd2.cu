// Zstd L1/L2 match finder, second stage: verification and parse.
//
// Input: the window bytes and cand(q) from the candidate sweep
// (gcz_sweep.cu).  Output: the exact sequence list of zstd_match_find
// (zstd_compress.cu:179-355) for every window.
//
// The window is staged into shared memory with 1-D bulk copies, and every
// position's hash candidate (empty == position 0, :195-200) is verified on 3
// bytes (:241-246); the results form a bitmap.  Two parses work from it.
//
// Lane parse (zstd_lane_parse_kernel, the default).  The reference parse is a
// state machine over (pos, rep0, rep1, rep2), but its repeat offsets
// (:259-275) decide a match only a few times per window.  So:
// 1. Parse without repeat offsets.  Its state is the position alone.  The
//    window is cut into 132-byte segments; every lane parses one at a time
//    from the segment's start and pulls the next of its warp's when done.
// 2. Link.  Where a segment's parse ends, it joins the list of the segment
//    that holds that position: at once when that list has no match across it
//    (the state is the position, so both parses go on alike), else after a few
//    more matches.  The links from segment 0 pick the list of the whole parse.
// 3. Check.  The repeat offsets of every literal run are those of the three
//    matches before it, so all runs are tested at once, 16 positions and three
//    offsets per lane task, tasks of 32 runs spread evenly over the lanes.
// 4. Mend.  A run with a repeat-offset match is parsed again from its start,
//    with repeat offsets, by one warp, until it emits a match of the list with
//    the list's repeat offsets after it: from there on the list is right.
//    Mends lie side by side; one that starts inside an earlier one is dropped.
//    Every literal run is then either checked or parsed exactly, so the
//    sequences are the reference's by induction over the runs.
// 5. Give up.  A window with more than kMostFixes such runs, with runs that
//    have such matches all over them, with a mend that finds no end soon, or
//    with no room for a list is parsed again after the CTA's other windows, and
//    some windows after it are given up at once.  How depends on how close to
//    one another the matches lie, by the entries or by a few mends tried out:
//    - close (counters, records with a fixed stride, 4-letter text): steps 1 and
//      2 with repeat offsets.  A segment's parse starts from {1,4,8} and joins a
//      later segment's list at a match that both have with the same repeat
//      offsets after it, nearly always its third;
//    - far apart (samples, floating-point numbers): the segment parse by warps;
//    - else (pixels, sorted numbers), and where a segment does not join a list
//      soon: the segment parse by 8-lane groups.
//    Per 256 MiB, with the segment parse by warps as the only way out and now:
//    32-bit counters 33.7 -> 4.3 ms, sorted numbers 23.5 -> 3.5, 20-byte records
//    11.1 -> 3.6, 8-byte records 12.2 -> 3.5, 3-byte pixels 5.8 -> 2.9, 4-letter
//    text (long continuations, step 2) 15.6 -> 3.9.
//
// Segment parse (zstd_seg_parse_kernel, and ways out of the lane parse).  Each
// warp parses one segment of 2-8 KiB, or each 8-lane group one of 1 KiB, from a
// guessed state (the segment start, repeat offsets {1,4,8}), then goes on past
// its end until one of its matches
// equals a match of a later warp's list -- same start, length and offset, and
// the same repeat offsets afterwards.  A chain walk from warp 0 picks the
// lists; every list on the chain is exact by induction.  A warp step takes the
// hash-match bits of the next positions from the bitmap, and the lanes test
// the three repeat offsets on the positions before the first hash match -- one
// (position, offset) pair per lane when there are at most 10 of them, one
// position per lane up to 32, and four positions per lane (8-byte compares)
// over up to 128 positions that hold no hash match; a ballot finds the first
// event, matches are extended 128 bytes per warp iteration, and one lazy step
// (:278-307) follows.  If a continuation does not meet a later list within
// kContCap matches, one warp parses the whole window exactly.
//
// Output: packed {ll | (ml-3) << 16, off} (or the reference's {ll, ml-3, off}
// triples) at the per-window stride, each literal length taken from the entry
// before it, capped at max_seqs exactly like the reference's
// `num_seqs < max_sequences_per_chunk` test (:309): the capped parse emits the
// first max_seqs matches of the uncapped one and nothing after them.
#include <type_traits>

#include "gcz_common.cuh"
#include "gcz_kernels.h"

namespace gcz {
namespace {

constexpr uint32_t kMinMatch = 3;                 // MIN_MATCH_LEN, zstd_compress.cu:28

// Segment parse: segment width (a schedule knob: 2, 4 or 8 KiB, one warp each;
// it never changes the sequences), or 1 KiB, one 8-lane group each.
template <uint32_t SegW, uint32_t GL = 32>
struct SegCfg {
    static constexpr uint32_t kSegW = SegW;
    static constexpr uint32_t kSegs = kMaxWindow / SegW;
    static constexpr uint32_t kThreads = kSegs * GL;
    // A segment's own parse ends with a step that starts before seg_end and
    // looks at most kLook positions ahead (a warp's wide scan 128, a group's
    // scan 32), the lazy step one more; matches do not overlap and are >= 3
    // bytes, so a list holds at most (SegW + kLook) / 3 + 1 entries; lists are
    // written in 32-entry blocks.
    static constexpr uint32_t kLook = GL == 32 ? 128 : 32;
    static constexpr uint32_t kSpecCap = ((SegW + kLook) / 3 + 1 + 31) / 32 * 32;
    // continuation matches before giving up (three meet nearly always)
    static constexpr uint32_t kContCap = GL == 32 ? 256 : 128;
    static constexpr uint32_t kLaneCap = kSpecCap + kContCap;
    static constexpr uint32_t kMinBlocks = kThreads >= 1024 ? 1 : 3;
};
constexpr uint32_t kNoWarp = 0xFFFFu;
constexpr uint32_t kNoEntry = 0xFFFFu;

constexpr uint32_t kPre = 32;                           // zero bytes before the window
constexpr uint32_t kDataBytes = kPre + kMaxWindow + 64; // + zero pad after it
constexpr uint32_t kBmWords = kMaxWindow / 32 + 8;  // the wide scan reads up to 4 words past a step's first

// Shared-memory fields of the segment parse (list lengths, indices and output
// offsets of a window are below 2^15).
template <uint32_t kSegs>
struct SegSmem {
    uint16_t spec_count[kSegs];
    uint16_t cont_count[kSegs];
    uint16_t sync_warp[kSegs];
    uint16_t sync_idx[kSegs];
    uint16_t chain_from[kSegs];
    uint16_t out_off[kSegs];
    uint16_t on_chain[kSegs];
    uint16_t prev_last[kSegs];  // seg index of the entry before a chain segment's first copied one (kNoEntry: none)
};

struct ParseScalars {
    uint32_t flags;    // 1: the segment parse gives up, 2: staging failed, 4: the lane parse gives up, 16: at once
    uint32_t total;
    uint32_t covered;
    uint32_t count;    // literal runs with a repeat-offset match found
    uint32_t mends;    // mends of the window
    uint32_t chunks;   // chunks of continuations in use
    uint32_t probe[2]; // matches and bytes of the window's mends
    uint32_t again;    // 1 + the last window given up (0: none); each leads to the one before it
    uint32_t how;      // how to parse the windows given up: 1 lanes, 0 groups, 2 warps
    uint32_t skip, streak;  // windows to give up at once; of the last time
    uint32_t warp_sum[32];
    alignas(8) uint64_t bar;
};

// Lane parse.
// 33 words, so that the lanes of a warp start in different banks, and stay there
// where the data has a short period (128 bytes: 32-bit counters 10.4 ms per 256
// MiB against 5.8, 64-byte records 2.3 against 1.7, the benchmark's data alike).
constexpr uint32_t kLSegW = 132, kLists = (kMaxWindow + kLSegW - 1) / kLSegW;
constexpr uint32_t kLSegs = 512;                                // kLists, up to whole warps
constexpr uint32_t kLCap = (kLSegW + 2) / 3;                    // matches that start their search in a segment
constexpr uint32_t kLCont = 12;                                 // continuation: 11 matches, then a chunk's number ...
constexpr uint32_t kLChunks = 224, kLChunk = 16;                // ... chunks of 15 more matches and the next one's number
constexpr uint32_t kLMost = 255;                                // most matches before a segment's parse joins a list
constexpr uint32_t kFixes = 256, kFixCap = 255;                 // runs recorded per window, most matches per mend
constexpr uint32_t kMostFixes = 192;                            // most runs that are mended
// Bytes per match of a window given up: lanes below kDense (kTryDense by the
// few matches tried out), warps from kSparse on, groups between.  64 MiB of 16-bit
// samples: with a match every 31 bytes 1.8 ms with lanes tried first, 1.04 by
// groups, 1.30 by warps; every 47 bytes 2.7 by groups, 1.2 by warps.
constexpr uint32_t kDense = 16, kTryDense = 12, kSparse = 44;
constexpr uint32_t kDenseCap = 48, kTryCap = 4;                 // most matches of a dense mend, and of one only tried out
constexpr uint32_t kMostSteps = 128;                            // most steps before a parse with repeat offsets joins a list
// Entries in a window's scratch: the segments' lists, then the continuations;
// once the list of the whole parse is known it takes the lists' place, and
// the mends that of the continuations.
constexpr uint32_t kLContBase = kLists * kLCap;
constexpr uint32_t kLChunkBase = kLContBase + kLists * kLCont;
constexpr uint32_t kLEntries = kLChunkBase + kLChunks * kLChunk;
constexpr uint32_t kFixEntries = kLEntries - kLContBase;        // shared by a window's mends
static_assert(kLContBase >= 21846, "the whole parse fits where the lists were");
static_assert(kLists <= kLSegs && kLSegs % 32 == 0, "whole warps of segments");
static_assert(kLMost <= 255, "8-bit counts");

template <uint32_t kWarps>
struct LaneSmem {
    union {
        struct {
            uint16_t link[kLSegs];   // parse end past the segment, then the segment joined, then the output offset
            uint8_t count[kLSegs];   // list entries
            uint8_t from[kLSegs];    // entry joined at, then the first entry on the chain
            uint8_t cont[kLSegs];    // continuation entries
            uint32_t chain[kLSegs / 32];  // segments on the chain
        };
        struct {
            uint16_t run[kFixes];    // literal runs with a repeat-offset match
            uint16_t pos[kFixes];    // position at or less than 16 before the run's first one
            uint16_t meet[kFixes];   // entry a mend ends at
            int16_t shift[kFixes];   // output index minus list index from there on
            uint8_t len[kFixes];     // entries of the mend
            uint8_t list[kFixes];    // the mend's list in the scratch
        } fix;
        SegSmem<64> seg;
        SegSmem<kWarps> segw;
    };
};

template <class P>
struct SmemLayout {
    uint8_t data[kDataBytes];
    uint32_t bm[kBmWords];
    P p;
    ParseScalars s;
};

struct Zstd2Args {
    const uint8_t *src;
    const uint16_t *cand;
    uint64_t n;
    uint32_t window;
    uint32_t num_windows;
    uint32_t lazy;
    uint32_t max_seqs;
    uint2 *seg;          // per window: seg_stride entries {start | (ml-3)<<16, off}
    uint2 *packed;       // packed output at stride max_seqs (or null)
    uint32_t *ref_seqs;  // reference triples at stride max_seqs (or null)
    uint32_t *seq_counts;
    uint32_t *lit_counts;
    uint32_t *status;
    const WinDesc *wins;
    uint32_t seg_stride;  // seg entries per window
};

// ---------------------------------------------------------------- helpers
struct Win {
    const uint8_t *d;  // window byte 0 (kPre zero bytes before it in shared memory)
    __device__ __forceinline__ uint32_t u32(int q) const {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(d - kPre);
        const uint32_t a = static_cast<uint32_t>(q + static_cast<int>(kPre));
        return __funnelshift_r(w[a >> 2], w[(a >> 2) + 1], a << 3);  // the shift counts modulo 32
    }
    // The 4 bytes at q, q a multiple of 4.
    __device__ __forceinline__ uint32_t w32(uint32_t q) const { return reinterpret_cast<const uint32_t *>(d)[q >> 2]; }
    // The 8 bytes at q: three aligned words, two funnel shifts.
    __device__ __forceinline__ void u64(int q, uint32_t &lo, uint32_t &hi) const {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(d - kPre);
        const uint32_t a = static_cast<uint32_t>(q + static_cast<int>(kPre));
        const uint32_t i = a >> 2, sh = a << 3;
        const uint32_t w1 = w[i + 1];
        lo = __funnelshift_r(w[i], w1, sh);
        hi = __funnelshift_r(w1, w[i + 2], sh);
    }
};

// First index in [0, lim) where bytes c+i and q+i differ, else lim.
// Warp-cooperative (all lanes call it with the same arguments): each lane
// compares 4 bytes, 128 bytes per iteration.
__device__ __forceinline__ uint32_t extend_warp(const Win &w, uint32_t c, uint32_t q, uint32_t lim) {
    const uint32_t lane = lane_id();
    uint32_t len = 0;
    for (;;) {
        const uint32_t k = len + 4u * lane;
        uint32_t res = k;
        if (k < lim) {
            const uint32_t d = w.u32(static_cast<int>(q + k)) ^ w.u32(static_cast<int>(c + k));
            const uint32_t fb = d ? (static_cast<uint32_t>(__ffs(d)) - 1u) >> 3 : 4u;
            const uint32_t rem = lim - k;
            res = k + (fb < rem ? fb : rem);
        }
        const uint32_t sb = __ballot_sync(kFull, res < k + 4u);
        if (sb) return __shfl_sync(kFull, res, __ffs(sb) - 1);
        len += 128u;
    }
}

// Two extensions at once: lanes 0-15 extend (ca, qa) up to la, lanes 16-31
// extend (cb, qb) up to lb, 64 bytes per half per iteration.
__device__ __forceinline__ void extend_pair(const Win &w, uint32_t ca, uint32_t qa, uint32_t la, uint32_t cb,
                                            uint32_t qb, uint32_t lb, uint32_t &ra, uint32_t &rb) {
    const uint32_t lane = lane_id(), half = lane >> 4, hl = lane & 15u;
    const uint32_t c = half ? cb : ca, q = half ? qb : qa, lim = half ? lb : la;
    bool da = false, db = false;
    ra = 0;
    rb = 0;
    for (uint32_t len = 0;; len += 64u) {
        const uint32_t k = len + 4u * hl;
        uint32_t res = k;
        if (k < lim) {
            const uint32_t d = w.u32(static_cast<int>(q + k)) ^ w.u32(static_cast<int>(c + k));
            const uint32_t fb = d ? (static_cast<uint32_t>(__ffs(d)) - 1u) >> 3 : 4u;
            const uint32_t rem = lim - k;
            res = k + (fb < rem ? fb : rem);
        }
        const uint32_t sb = __ballot_sync(kFull, res < k + 4u);
        const uint32_t sa = sb & 0xFFFFu, sbb = sb >> 16;
        const uint32_t va = __shfl_sync(kFull, res, sa ? __ffs(sa) - 1 : 0);
        const uint32_t vb = __shfl_sync(kFull, res, sbb ? 16 + __ffs(sbb) - 1 : 16);
        if (!da && sa) {
            ra = va;
            da = true;
        }
        if (!db && sbb) {
            rb = vb;
            db = true;
        }
        if (da && db) return;
    }
}

// Rolling register buffer of candidates for one warp: lane l holds
// cand[base + l], cand[base + 32 + l] and cand[base + 64 + l] (the third block
// is a prefetch), base 32-aligned.
struct CandBuf {
    const uint16_t *cand;
    uint32_t size, base, c0, c1, c2;
    __device__ __forceinline__ uint32_t ld(uint32_t pos) const {
        return pos < size ? static_cast<uint32_t>(cand[pos]) : 0u;
    }
    __device__ __forceinline__ void init(uint32_t p) {
        const uint32_t lane = lane_id();
        base = p & ~31u;
        c0 = ld(base + lane);
        c1 = ld(base + 32u + lane);
        c2 = ld(base + 64u + lane);
    }
    // Make positions [p, p+33) available (p uniform).
    __device__ __forceinline__ void advance(uint32_t p) {
        const uint32_t nb = p & ~31u, lane = lane_id();
        if (nb == base) return;
        if (nb == base + 32u) {
            c0 = c1;
            c1 = c2;
            c2 = ld(nb + 64u + lane);
        } else if (nb == base + 64u) {
            c0 = c2;
            c1 = ld(nb + 32u + lane);
            c2 = ld(nb + 64u + lane);
        } else {
            init(p);
            return;
        }
        base = nb;
    }
    // cand[pos] for pos in [base, base+96) (pos uniform).
    __device__ __forceinline__ uint32_t get(uint32_t pos) const {
        const uint32_t k = pos - base;
        const uint32_t r = k < 32u ? c0 : (k < 64u ? c1 : c2);
        return __shfl_sync(kFull, r, k & 31u);
    }
};

__device__ __forceinline__ bool eq3(const Win &w, uint32_t a, uint32_t b) {
    return ((w.u32(static_cast<int>(a)) ^ w.u32(static_cast<int>(b))) & 0xFFFFFFu) == 0u;
}

__device__ __forceinline__ uint32_t bm_bit(const uint32_t *bm, uint32_t q) { return (bm[q >> 5] >> (q & 31u)) & 1u; }

struct PState {
    uint32_t p, r0, r1, r2;
};

struct Match {
    uint32_t start, len, off;
};

// One warp-uniform step of the exact parse from state s (s.p + 3 < size):
// either finds the next match (returns true, s advanced past it, repeat
// offsets updated) or moves s.p over up to 32 literal positions.
__device__ __forceinline__ bool warp_step(const Win &w, const uint32_t *bm, CandBuf &cb, uint32_t size, bool lazy,
                                          PState &s, Match &m) {
    const uint32_t lane = lane_id();
    const uint32_t p = s.p;
    const uint32_t lim = size - 3u - p;
    const uint32_t nscan = lim < 32u ? lim : 32u;
    uint32_t H = __funnelshift_r(bm[p >> 5], bm[(p >> 5) + 1], p & 31u);
    if (nscan < 32u) H &= (1u << nscan) - 1u;
    const uint32_t q = p + lane;
    cb.advance(p);  // candidates of p .. p+32 (and the next block in flight)
    uint32_t f, r = 0;  // event position; for a repeat-offset match, which repeat offset (0-2)
    bool hash;
    if (H & 1u) {
        f = p;
        hash = true;
    } else {
        // Repeat offsets are tried only at positions without a hash match, in
        // order r0, r1, r2, and the first position with a hit wins
        // (zstd_compress.cu:259-275).  How the lanes share the tests depends
        // on how many positions come before the first hash match.
        const uint32_t n = H ? static_cast<uint32_t>(__ffs(H)) - 1u : nscan;  // positions without a hash match
        if (n <= 10u) {
            // Few positions: one (position, repeat offset) pair per lane, in
            // position-major order, so the first set ballot bit is the event.
            const uint32_t i = lane / 3u, k = lane - 3u * i;
            const uint32_t rv = k == 0u ? s.r0 : (k == 1u ? s.r1 : s.r2);
            const uint32_t qq = p + i;
            const bool hit = i < n && rv <= qq && eq3(w, qq, rv <= qq ? qq - rv : qq);
            const uint32_t rb = __ballot_sync(kFull, hit);
            if (rb) {
                const uint32_t l = static_cast<uint32_t>(__ffs(rb)) - 1u;
                f = p + l / 3u;
                r = l % 3u;
                hash = false;
            } else if (H) {
                f = p + n;
                hash = true;
            } else {
                s.p = p + nscan;
                return false;
            }
        } else if (H == 0u && lim > 32u) {
            // No hash match in 32 positions: scan up to 128, four positions
            // per lane, each repeat offset tested on 8-byte words.
            const uint32_t n4s = lim < 128u ? lim : 128u;
            const uint32_t wi = p >> 5, sh = p & 31u;
            uint32_t n4 = n4s;
#pragma unroll
            for (uint32_t k = 3; k >= 1; --k) {
                const uint32_t hk = __funnelshift_r(bm[wi + k], bm[wi + k + 1u], sh);
                if (hk) n4 = 32u * k + static_cast<uint32_t>(__ffs(hk)) - 1u;
            }
            if (n4 > n4s) n4 = n4s;
            const uint32_t j0 = 4u * lane;  // this lane's first position index
            const uint32_t q0 = j0 < n4 ? p + j0 : p;
            const uint32_t vlim = j0 < n4 ? (n4 - j0 < 4u ? n4 - j0 : 4u) : 0u;  // positions of this lane to test
            const uint32_t xlo = w.u32(static_cast<int>(q0)), xhi = w.u32(static_cast<int>(q0 + 4u));
            uint32_t mk[3];
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k) {
                const uint32_t rv = k == 0u ? s.r0 : (k == 1u ? s.r1 : s.r2);
                // positions q0 + t with t < vlim and q0 + t >= rv; their source bytes start at q0 - rv + t >= 0
                const uint32_t tmin = rv > q0 ? rv - q0 : 0u;
                uint32_t valid = tmin < vlim ? ((1u << vlim) - 1u) & ~((1u << tmin) - 1u) : 0u;
                const int yb = valid ? static_cast<int>(q0) - static_cast<int>(rv) : static_cast<int>(q0);
                const uint32_t dlo = xlo ^ w.u32(yb), dhi = xhi ^ w.u32(yb + 4);
                const uint32_t e = ((dlo & 0xFFFFFFu) == 0u ? 1u : 0u) | ((dlo >> 8) == 0u ? 2u : 0u) |
                                   ((__funnelshift_r(dlo, dhi, 16) & 0xFFFFFFu) == 0u ? 4u : 0u) |
                                   ((__funnelshift_r(dlo, dhi, 24) & 0xFFFFFFu) == 0u ? 8u : 0u);
                mk[k] = e & valid;
            }
            const uint32_t any = mk[0] | mk[1] | mk[2];
            const uint32_t rb = __ballot_sync(kFull, any != 0u);
            if (rb) {
                const uint32_t l = static_cast<uint32_t>(__ffs(rb)) - 1u;
                const uint32_t al = __shfl_sync(kFull, any, l), m0 = __shfl_sync(kFull, mk[0], l),
                               m1 = __shfl_sync(kFull, mk[1], l);
                const uint32_t t = static_cast<uint32_t>(__ffs(al)) - 1u;
                f = p + 4u * l + t;
                r = (m0 >> t) & 1u ? 0u : ((m1 >> t) & 1u ? 1u : 2u);
                hash = false;
            } else if (n4 < n4s) {
                f = p + n4;
                hash = true;
            } else {
                s.p = p + n4s;
                return false;
            }
        } else {
            const bool need = lane < n;
            const uint32_t x = w.u32(static_cast<int>(q));
            const bool a0 =
                need && s.r0 <= q && ((x ^ w.u32(static_cast<int>(s.r0 <= q ? q - s.r0 : 0u))) & 0xFFFFFFu) == 0u;
            const bool a1 = need && !a0 && s.r1 <= q &&
                            ((x ^ w.u32(static_cast<int>(s.r1 <= q ? q - s.r1 : 0u))) & 0xFFFFFFu) == 0u;
            const bool a2 = need && !a0 && !a1 && s.r2 <= q &&
                            ((x ^ w.u32(static_cast<int>(s.r2 <= q ? q - s.r2 : 0u))) & 0xFFFFFFu) == 0u;
            const uint32_t rsel = a0 ? 0u : (a1 ? 1u : 2u);
            const uint32_t rb = __ballot_sync(kFull, a0 || a1 || a2);
            if (rb) {
                const uint32_t l = static_cast<uint32_t>(__ffs(rb)) - 1u;
                f = p + l;
                r = __shfl_sync(kFull, rsel, l);
                hash = false;
            } else if (H) {
                f = p + n;
                hash = true;
            } else {
                s.p = p + nscan;
                return false;
            }
        }
    }
    cb.advance(f);  // a wide scan's event can lie past the buffer
    const uint32_t cf = cb.get(f);
    const uint32_t cf1 = cb.get(f + 1u);
    uint32_t off, c0;
    if (hash) {
        off = f - cf;
        c0 = cf;
    } else {  // first repeat offset with 3 equal bytes wins
        off = r == 0u ? s.r0 : (r == 1u ? s.r1 : s.r2);
        c0 = f - off;
    }
    uint32_t len;
    // The lazy candidate at f+1 (zstd_compress.cu:278-307) is taken only when
    // len2 > len + 1.  When it is the same match one byte on (cand(f+1) ==
    // c0 + 1) it is exactly one byte shorter -- its 3 verified bytes include
    // byte f+3 == c0+3, so the main match extends past 3 -- and is never taken.
    if (lazy && f + 4u < size && bm_bit(bm, f + 1u) && cf1 != c0 + 1u) {  // main match and lazy candidate together
        uint32_t l1, l2;
        extend_pair(w, c0 + kMinMatch, f + kMinMatch, size - f - kMinMatch, cf1 + kMinMatch, f + 1u + kMinMatch,
                    size - f - 1u - kMinMatch, l1, l2);
        len = l1 + kMinMatch;
        const uint32_t len2 = l2 + kMinMatch;
        if (len2 > len + 1u) {
            f += 1u;
            len = len2;
            off = f - cf1;
        }
    } else {
        len = extend_warp(w, c0 + kMinMatch, f + kMinMatch, size - f - kMinMatch) + kMinMatch;
    }
    m.start = f;
    m.len = len;
    m.off = off;
    s.r2 = s.r1;
    s.r1 = s.r0;
    s.r0 = off;
    s.p = f + len;
    return true;
}

// Bit t (t < 16) set when bytes q+t .. q+t+2 equal bytes q-r+t .. q-r+t+2
// (zstd_compress.cu:259-275 tests one position at a time).  Both 18-byte
// ranges are read as aligned words; a byte of x ^ y is zero exactly when its
// 0x80 flag survives ~(((d & 0x7F..) + 0x7F..) | d | 0x7F..), three flags in
// a row mark a 3-byte match, and a multiply gathers each word's four flags.
template <uint32_t kWords>
__device__ __forceinline__ uint32_t rep3_scan(const Win &w, uint32_t q, uint32_t r) {
    const uint32_t *wd = reinterpret_cast<const uint32_t *>(w.d - kPre);
    const uint32_t ax = q + kPre, ay = q - r + kPre;
    const uint32_t *px = wd + (ax >> 2), *py = wd + (ay >> 2);
    const uint32_t sx = (ax & 3u) * 8u, sy = (ay & 3u) * 8u;
    uint32_t z[kWords + 1u];
    uint32_t xp = px[0], yp = py[0];
#pragma unroll
    for (uint32_t j = 0; j <= kWords; ++j) {
        const uint32_t xn = px[j + 1], yn = py[j + 1];
        const uint32_t d = __funnelshift_r(xp, xn, sx) ^ __funnelshift_r(yp, yn, sy);
        z[j] = ~(((d & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | d | 0x7F7F7F7Fu);
        xp = xn;
        yp = yn;
    }
    uint32_t m = 0;
#pragma unroll
    for (uint32_t j = 0; j < kWords; ++j) {
        const uint32_t e = z[j] & __funnelshift_r(z[j], z[j + 1], 8) & __funnelshift_r(z[j], z[j + 1], 16);
        m |= ((e * 0x00204081u) >> 28) << (4u * j);
    }
    return m;
}

// Whether any position of q .. q+min(n,16)-1 (n >= 1) has its three bytes equal
// to those at one of the three distances ro (all <= q).  Per word of positions
// and distance: y = OR of the difference bytes at t, t+1 and t+2, which is zero
// at a match; (y - 0x01..) & ~y has 0x80 at the lowest zero byte (and maybe
// above it, which does not change whether there is one).
__device__ __forceinline__ bool rep3_any16(const Win &w, uint32_t q, const uint32_t *ro, uint32_t n) {
    const uint32_t *wd = reinterpret_cast<const uint32_t *>(w.d - kPre);
    const uint32_t ax = q + kPre;
    const uint32_t *px = wd + (ax >> 2);
    uint32_t x[5], a[4] = {0u, 0u, 0u, 0u}, xp = px[0];
#pragma unroll
    for (uint32_t j = 0; j < 5; ++j) {
        const uint32_t xn = px[j + 1];
        x[j] = __funnelshift_r(xp, xn, ax << 3);
        xp = xn;
    }
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k) {
        const uint32_t ay = ax - ro[k];
        const uint32_t *py = wd + (ay >> 2);
        uint32_t yp = py[0], yn = py[1], d = x[0] ^ __funnelshift_r(yp, yn, ay << 3);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            yp = yn;
            yn = py[j + 2];
            const uint32_t dn = x[j + 1] ^ __funnelshift_r(yp, yn, ay << 3);
            const uint32_t y = d | __funnelshift_r(d, dn, 8) | __funnelshift_r(d, dn, 16);
            a[j] |= (y - 0x01010101u) & ~y;
            d = dn;
        }
    }
    if (n < 16u) {
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t t = n > 4u * j ? n - 4u * j : 0u;  // positions of word j that count
            if (t < 4u) a[j] &= (1u << (8u * t)) - 1u;
        }
    }
    return ((a[0] | a[1] | a[2] | a[3]) & 0x80808080u) != 0u;
}

// Group-wide extension: the lanes of each GL-lane group compare 4 bytes each
// (4 * GL per iteration) of their group's own (c, q, lim) and get the first
// index in [0, lim) where bytes c+i and q+i differ, else lim; groups with
// act == false get 0.  All 32 lanes call it (the loop runs while any group
// is still extending).
template <uint32_t GL>
__device__ __forceinline__ uint32_t extend_group(const Win &w, uint32_t c, uint32_t q, uint32_t lim, bool act) {
    const uint32_t lane = lane_id(), gl = lane & (GL - 1u), gb = lane & ~(GL - 1u);
    uint32_t len = 0, out = 0;
    bool done = !act;
    while (__any_sync(kFull, !done)) {
        const uint32_t k = len + 8u * gl;  // 8 bytes per lane
        uint32_t res = k;
        if (!done && k < lim) {
            uint32_t ql, qh, cl, ch;
            w.u64(static_cast<int>(q + k), ql, qh);
            w.u64(static_cast<int>(c + k), cl, ch);
            const uint32_t dl = ql ^ cl, dh = qh ^ ch;
            const uint32_t fb = dl ? (static_cast<uint32_t>(__ffs(dl)) - 1u) >> 3
                                   : (dh ? 4u + ((static_cast<uint32_t>(__ffs(dh)) - 1u) >> 3) : 8u);
            const uint32_t rem = lim - k;
            res = k + (fb < rem ? fb : rem);
        }
        const uint32_t sb = (__ballot_sync(kFull, !done && res < k + 8u) >> gb) & ((1u << GL) - 1u);
        const uint32_t v = __shfl_sync(kFull, res, gb + (sb ? static_cast<uint32_t>(__ffs(sb)) - 1u : 0u));
        if (!done && sb) {
            out = v;
            done = true;
        }
        len += 8u * GL;
    }
    return out;
}

// One step of the exact parse for every 8-lane group of the warp at once, each
// from its own state s (group-uniform); groups with run == false keep theirs.
// A group looks at the 32 positions from s.p: the hash-match bits come from the
// bitmap, and six lanes test the three repeat offsets among the positions
// before the first hash match (zstd_compress.cu:259-275), 16 positions each.
// The first event is the match, extended 64 bytes per group iteration, with the
// lazy step (:278-307) at f+1; with no event the group moves over the 32
// positions.  Returns whether the group found a match (m set, s advanced past
// it, repeat offsets updated).
template <uint32_t GL>
__device__ __forceinline__ bool group_step(const Win &w, const uint32_t *bm, const uint16_t *cand, uint32_t size,
                                           bool lazy, bool run, PState &s, Match &m) {
    static_assert(GL == 8, "8-lane groups");
    const uint32_t lane = lane_id(), gl = lane & (GL - 1u), gb = lane & ~(GL - 1u);
    const uint32_t p = run ? s.p : 0u;
    const uint32_t lim = run ? size - 3u - p : 0u;
    const uint32_t n32 = lim < 32u ? lim : 32u;
    uint32_t H = __funnelshift_r(bm[p >> 5], bm[(p >> 5) + 1], p & 31u);
    if (n32 < 32u) H &= (1u << n32) - 1u;
    const uint32_t nh = H ? static_cast<uint32_t>(__ffs(H)) - 1u : n32;  // positions without a hash match
    // The candidates at the first hash match and the position after it are
    // loaded before the repeat-offset test, so that their latency overlaps
    // it: the event is that hash match unless a repeat offset hits earlier
    // (a few times per window), and only then is cand(f+1) loaded again.
    const uint32_t fh = nh < n32 ? p + nh : 0u;
    const uint32_t ch0 = cand[fh], ch1 = cand[fh + 1u];
    uint32_t m0, m1, m2;  // per repeat offset: hits among the 32 positions
    {
        // Lane 2k+h (k < 3) tests repeat offset k on the 16 positions from
        // p + 16h that come before the first hash match and whose source lies
        // in the window; lanes 6 and 7 test nothing.
        const uint32_t rk = gl >> 1, hh = gl & 1u;
        const uint32_t q0 = p + 16u * hh;
        const uint32_t rv = rk == 0u ? s.r0 : (rk == 1u ? s.r1 : s.r2);
        const uint32_t lo = rv > q0 ? (rv - q0 < 16u ? rv - q0 : 16u) : 0u;
        const uint32_t hi = (rk < 3u && nh > 16u * hh) ? (nh - 16u * hh < 16u ? nh - 16u * hh : 16u) : 0u;
        const uint32_t vm = ((1u << hi) - 1u) & ~((1u << lo) - 1u);
        const uint32_t mk = rep3_scan<4>(w, q0, rv <= q0 + 16u ? rv : 0u) & vm;
        const uint32_t mo = __shfl_xor_sync(kFull, mk, 1);
        const uint32_t mf = hh ? (mo | (mk << 16)) : (mk | (mo << 16));  // offset rk over all 32 positions
        m0 = __shfl_sync(kFull, mf, gb);
        m1 = __shfl_sync(kFull, mf, gb + 2u);
        m2 = __shfl_sync(kFull, mf, gb + 4u);
    }
    const uint32_t al = m0 | m1 | m2;
    const bool rep = al != 0u;
    const bool ev = run && (rep || nh < n32);
    uint32_t f = p + nh, r = 0;
    if (rep) {
        const uint32_t t = static_cast<uint32_t>(__ffs(al)) - 1u;
        f = p + t;
        r = (m0 >> t) & 1u ? 0u : ((m1 >> t) & 1u ? 1u : 2u);
    }
    const uint32_t fc = ev ? f : 0u;
    const uint32_t cf = ch0;
    uint32_t cf1 = ch1;
    if (rep) cf1 = cand[fc + 1u];
    uint32_t off, c0;
    if (!rep) {
        off = fc - cf;
        c0 = cf;
    } else {  // first repeat offset with 3 equal bytes wins
        off = r == 0u ? s.r0 : (r == 1u ? s.r1 : s.r2);
        c0 = fc - off;
    }
    // The lazy candidate at f+1 is skipped when it is the same match one byte on
    // (cand(f+1) == c0 + 1): it is exactly one byte shorter, never taken.
    const bool ltry = ev && lazy && fc + 4u < size && bm_bit(bm, fc + 1u) && cf1 != c0 + 1u;
    const uint32_t e1 = extend_group<GL>(w, c0 + kMinMatch, fc + kMinMatch, ev ? size - fc - kMinMatch : 0u, ev);
    const uint32_t e2 =
        extend_group<GL>(w, cf1 + kMinMatch, fc + 1u + kMinMatch, ltry ? size - fc - 1u - kMinMatch : 0u, ltry);
    uint32_t len = e1 + kMinMatch;
    f = fc;
    if (ltry && e2 + kMinMatch > len + 1u) {
        f = fc + 1u;
        len = e2 + kMinMatch;
        off = f - cf1;
    }
    if (ev) {
        m.start = f;
        m.len = len;
        m.off = off;
        s.r2 = s.r1;
        s.r1 = s.r0;
        s.r0 = off;
        s.p = f + len;
    } else if (run) {
        s.p = p + n32;
    }
    return ev;
}

__device__ __forceinline__ uint2 pack_entry(const Match &m) {
    return make_uint2(m.start | ((m.len - kMinMatch) << 16), m.off);
}

// Repeat offsets after entry j of a list whose parse started from {1,4,8}.
__device__ __forceinline__ void reps_after(const uint2 *list, uint32_t j, uint32_t &a, uint32_t &b, uint32_t &c) {
    a = list[j].y;
    b = j >= 1 ? list[j - 1].y : 1u;
    c = j >= 2 ? list[j - 2].y : (j == 1 ? 1u : 4u);
}

// Warp-buffered list writer: entry i is held by lane i%32 until 32 are ready.
struct ListWriter {
    uint2 *out;
    uint32_t n;
    uint2 v;
    __device__ __forceinline__ explicit ListWriter(uint2 *o) : out(o), n(0), v(make_uint2(0u, 0u)) {}
    __device__ __forceinline__ void put(const uint2 &e) {
        if (lane_id() == (n & 31u)) v = e;
        if ((n & 31u) == 31u) out[(n & ~31u) + lane_id()] = v;
        ++n;
    }
    __device__ __forceinline__ void flush() {
        if (lane_id() < (n & 31u)) out[(n & ~31u) + lane_id()] = v;
    }
};

// ---------------------------------------------------------------- shared parts of the kernels
// First byte and size of window wi.
__device__ __forceinline__ void window_of(const Zstd2Args &a, uint32_t wi, uint64_t &start, uint32_t &size) {
    start = a.wins ? a.wins[wi].offset : static_cast<uint64_t>(wi) * a.window;
    size = a.wins ? a.wins[wi].size : static_cast<uint32_t>(a.n - start < a.window ? a.n - start : a.window);
}

// Verification bitmap of a staged window, by all kW warps of the CTA: bit q
// set when q can start a match and its candidate matches on 3 bytes.
template <uint32_t kW>
__device__ __forceinline__ void verify_window(const Win &win, uint32_t *bm, const uint16_t *cand, uint32_t size) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    // Lane l covers positions 4l .. 4l+3 of a 128-position chunk: one
    // 8-byte load brings its four candidates, one aligned 8-byte read its own
    // bytes, and the 8 lanes of each bitmap word gather their four bits with
    // three shuffles.  kVC chunks per batch: their candidate loads are all
    // issued first.  Words up to four past the window's last are set.
    constexpr uint32_t kVC = 4;
    static_assert(kBmWords % 4u == 0u, "bitmap words come in 128-position chunks");
    const uint32_t nch = (size >> 7) + 2u, lim_pos = size > 3u ? size - 3u : 0u;
    for (uint32_t c0 = warp * kVC; c0 < nch; c0 += kW * kVC) {
        uint2 cv[kVC];
#pragma unroll
        for (uint32_t u = 0; u < kVC; ++u) {
            const uint32_t q = (c0 + u) * 128u + 4u * lane;
            cv[u] = make_uint2(0u, 0u);
            if (q + 4u <= size) {
                cv[u] = *reinterpret_cast<const uint2 *>(cand + q);
            } else if (q < lim_pos) {
                uint32_t e[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) e[k] = q + k < size ? static_cast<uint32_t>(cand[q + k]) : 0u;
                cv[u] = make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < kVC; ++u) {
            const uint32_t ch = c0 + u;
            if (ch >= nch) break;
            const uint32_t q = min(ch * 128u + 4u * lane, kMaxWindow);
            const uint32_t x0 = win.w32(q), x1 = win.w32(q + 4u);
            uint32_t v = 0;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const uint32_t cw = k < 2u ? cv[u].x : cv[u].y;
                const uint32_t c = (k & 1u) ? cw >> 16 : cw & 0xFFFFu;
                const uint32_t xk = k ? __funnelshift_r(x0, x1, 8u * k) : x0;
                if (((xk ^ win.u32(static_cast<int>(c))) & 0xFFFFFFu) == 0u) v |= 1u << k;
            }
            v <<= 4u * (lane & 7u);
            v |= __shfl_xor_sync(kFull, v, 1);
            v |= __shfl_xor_sync(kFull, v, 2);
            v |= __shfl_xor_sync(kFull, v, 4);
            if (ch == 0u && lane == 0u) v &= ~1u;  // position 0 has nothing before it
            if (ch * 128u + 128u > lim_pos) {      // positions from lim_pos on start no match
                const uint32_t p = ch * 128u + 32u * (lane >> 3), in = lim_pos > p ? lim_pos - p : 0u;
                if (in < 32u) v &= (1u << in) - 1u;
            }
            if ((lane & 7u) == 0u) bm[ch * 4u + (lane >> 3)] = v;
        }
    }
}

// Output entry o of window wi.
template <bool kRef>
__device__ __forceinline__ void write_seq(const Zstd2Args &a, uint32_t wi, uint32_t o, uint32_t ll, uint32_t mlm3,
                                          uint32_t off) {
    if constexpr (kRef) {
        uint32_t *r = a.ref_seqs + (static_cast<uint64_t>(wi) * a.max_seqs + o) * 3u;
        r[0] = ll;
        r[1] = mlm3;
        r[2] = off;
    } else {
        a.packed[static_cast<uint64_t>(wi) * a.max_seqs + o] = make_uint2(ll | (mlm3 << 16), off);
    }
}

// ---------------------------------------------------------------- segment parse
// All threads of the CTA (SegCfg<SegW>::kThreads) call it with the window
// staged and verified, S.flags & 1 clear and S.covered zero.
template <bool kRef, uint32_t SegW, uint32_t GL = 32>
__device__ __forceinline__ void parse_segments(const Zstd2Args &a, SegSmem<SegCfg<SegW, GL>::kSegs> &G, ParseScalars &S,
                                               const Win &win, const uint32_t *bm, const uint16_t *cand, uint2 *seg,
                                               uint32_t wi, uint32_t size, bool lazy) {
    using C = SegCfg<SegW, GL>;
    constexpr uint32_t kSegW = C::kSegW, kSegs = C::kSegs;
    constexpr uint32_t kSpecCap = C::kSpecCap, kLaneCap = C::kLaneCap, kContCap = C::kContCap;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t lim_pos = size > 3u ? size - 3u : 0u;  // positions q < lim_pos can start a match
    if constexpr (GL == 32) {
        // ---- 2a. speculative parse of each segment (one warp each)
        const uint32_t seg_start = warp * kSegW, seg_end = seg_start + kSegW;
        const bool active = seg_start < lim_pos;
        const bool last_active = !(seg_end < lim_pos);
        ListWriter lw(seg + warp * kLaneCap);
        PState s{seg_start, 1u, 4u, 8u};
        CandBuf cb{cand, size, 0u, 0u, 0u, 0u};
        if (active) cb.init(seg_start);
        if (active) {
            const uint32_t stop = last_active ? size : seg_end;
            Match m;
            while (s.p < stop && s.p + 3u < size) {
                if (warp_step(win, bm, cb, size, lazy, s, m)) lw.put(pack_entry(m));
            }
            lw.flush();
        }
        if (lane == 0) {
            G.spec_count[warp] = lw.n;
            G.cont_count[warp] = 0;
            G.sync_warp[warp] = kNoWarp;
            G.sync_idx[warp] = 0;
        }
        __syncthreads();

        // ---- 2b. continue each warp's parse until it meets a later warp's list
        if (active && !last_active) {
            ListWriter cw(seg + warp * kLaneCap + kSpecCap);
            uint32_t t = kNoWarp, j = 0;
            Match m;
            while (s.p + 3u < size) {
                if (!warp_step(win, bm, cb, size, lazy, s, m)) continue;
                const uint32_t tw = m.start / kSegW;  // warp whose segment holds this match start
                if (tw != t) {
                    t = tw;
                    j = 0;
                }
                const uint32_t tcount = G.spec_count[t];
                const uint2 *tl = seg + t * kLaneCap;
                // first entry of t's list with start >= m.start (lists are sorted by start)
                for (;;) {
                    const uint32_t idx = j + lane;
                    const bool ge = idx >= tcount || (tl[idx].x & 0xFFFFu) >= m.start;
                    const uint32_t b = __ballot_sync(kFull, ge);
                    if (b) {
                        j += static_cast<uint32_t>(__ffs(b)) - 1u;
                        break;
                    }
                    j += 32u;
                }
                bool met = false;
                if (j < tcount) {
                    const uint2 e = tl[j];
                    if (e.x == pack_entry(m).x && e.y == m.off) {
                        uint32_t e0, e1, e2;
                        reps_after(tl, j, e0, e1, e2);
                        met = e0 == s.r0 && e1 == s.r1 && e2 == s.r2;
                    }
                }
                if (met) {
                    if (lane == 0) {
                        G.sync_warp[warp] = t;
                        G.sync_idx[warp] = j;
                    }
                    break;
                }
                if (cw.n == kContCap) {
                    if (lane == 0) atomicOr(&S.flags, 1u);  // give up: exact fallback below
                    break;
                }
                cw.put(pack_entry(m));
            }
            cw.flush();
            if (lane == 0) G.cont_count[warp] = cw.n;
        }
        __syncthreads();
    } else {
        // ---- 2a. speculative parse of each segment (one 8-lane group each)
        const uint32_t sg = tid / GL, gl = lane & (GL - 1u), gb = lane & ~(GL - 1u);
        const uint32_t seg_start = sg * kSegW, seg_end = seg_start + kSegW;
        const bool active = sg < kSegs && seg_start < lim_pos;
        const bool last_active = !(seg_end < lim_pos);
        const uint32_t stop = last_active ? size : seg_end;
        uint2 *lst = seg + sg * kLaneCap;
        PState s{seg_start, 1u, 4u, 8u};
        uint32_t n = 0;
        for (;;) {
            const bool run = active && s.p < stop && s.p + 3u < size;
            if (!__any_sync(kFull, run)) break;
            Match m;
            if (group_step<GL>(win, bm, cand, size, lazy, run, s, m)) {
                if (gl == 0) lst[n] = pack_entry(m);
                ++n;
            }
        }
        if (gl == 0 && sg < kSegs) {
            G.spec_count[sg] = n;
            G.cont_count[sg] = 0;
            G.sync_warp[sg] = kNoWarp;
            G.sync_idx[sg] = 0;
        }
        __syncthreads();

        // ---- 2b. continue each group's parse until it meets a later segment's list
        bool crun = active && !last_active;
        uint32_t t = kNoWarp, j = 0, cn = 0;
        uint2 *cl = lst + kSpecCap;
        for (;;) {
            const bool run = crun && s.p + 3u < size;
            const uint32_t runners = __ballot_sync(kFull, run && gl == 0u);
            if (!runners) break;
            if ((runners & (runners - 1u)) == 0u) {
                // Only one group of the warp still runs (the slow tail of the
                // phase): the whole warp takes over its parse with warp-wide
                // steps (up to 128 positions scanned, 128 bytes extended per
                // iteration), same meeting test, then the loop ends.
                const uint32_t L = static_cast<uint32_t>(__ffs(runners)) - 1u;
                PState ws{__shfl_sync(kFull, s.p, L), __shfl_sync(kFull, s.r0, L), __shfl_sync(kFull, s.r1, L),
                          __shfl_sync(kFull, s.r2, L)};
                const uint32_t wsg = __shfl_sync(kFull, sg, L);
                uint32_t wt = __shfl_sync(kFull, t, L), wj = __shfl_sync(kFull, j, L),
                         wcn = __shfl_sync(kFull, cn, L);
                uint2 *wcl = seg + wsg * kLaneCap + kSpecCap;
                CandBuf wcb{cand, size, 0u, 0u, 0u, 0u};
                wcb.init(ws.p);
                while (ws.p + 3u < size) {
                    Match m;
                    if (!warp_step(win, bm, wcb, size, lazy, ws, m)) continue;
                    const uint32_t tw = m.start / kSegW;  // segment that holds this match start
                    if (tw != wt) {
                        wt = tw;
                        wj = 0;
                    }
                    const uint32_t tcount = G.spec_count[wt];
                    const uint2 *tl = seg + wt * kLaneCap;
                    // first entry of wt's list with start >= m.start, 32 per step
                    for (;;) {
                        const uint32_t idx = wj + lane;
                        const bool ge = idx >= tcount || (tl[idx].x & 0xFFFFu) >= m.start;
                        const uint32_t b = __ballot_sync(kFull, ge);
                        if (b) {
                            wj += static_cast<uint32_t>(__ffs(b)) - 1u;
                            break;
                        }
                        wj += 32u;
                    }
                    bool met = false;
                    if (wj < tcount) {
                        const uint2 e = tl[wj];
                        if (e.x == pack_entry(m).x && e.y == m.off) {
                            uint32_t e0, e1, e2;
                            reps_after(tl, wj, e0, e1, e2);
                            met = e0 == ws.r0 && e1 == ws.r1 && e2 == ws.r2;
                        }
                    }
                    if (met) {
                        if (lane == 0) {
                            G.sync_warp[wsg] = wt;
                            G.sync_idx[wsg] = wj;
                        }
                        break;
                    }
                    if (wcn == kContCap) {
                        if (lane == 0) atomicOr(&S.flags, 1u);  // give up: exact fallback below
                        break;
                    }
                    if (lane == 0) wcl[wcn] = pack_entry(m);
                    ++wcn;
                }
                if (lane >= L && lane < L + GL) {
                    cn = wcn;
                    crun = false;
                }
                break;
            }
            Match m;
            const bool ev = group_step<GL>(win, bm, cand, size, lazy, run, s, m);
            uint32_t tcount = 0;
            const uint2 *tl = seg;
            if (ev) {
                const uint32_t tw = m.start / kSegW;  // segment that holds this match start
                if (tw != t) {
                    t = tw;
                    j = 0;
                }
                tcount = G.spec_count[t];
                tl = seg + t * kLaneCap;
            }
            // first entry of t's list with start >= m.start (lists are sorted by start), 8 per step
            bool found = !ev;
            while (__any_sync(kFull, !found)) {
                const uint32_t idx = j + gl;
                const bool ge = !found && (idx >= tcount || (tl[idx].x & 0xFFFFu) >= m.start);
                const uint32_t b = (__ballot_sync(kFull, ge) >> gb) & ((1u << GL) - 1u);
                if (!found) {
                    if (b) {
                        j += static_cast<uint32_t>(__ffs(b)) - 1u;
                        found = true;
                    } else {
                        j += GL;
                    }
                }
            }
            if (!ev) {
                if (!run) crun = false;
                continue;
            }
            bool met = false;
            if (j < tcount) {
                const uint2 e = tl[j];
                if (e.x == pack_entry(m).x && e.y == m.off) {
                    uint32_t e0, e1, e2;
                    reps_after(tl, j, e0, e1, e2);
                    met = e0 == s.r0 && e1 == s.r1 && e2 == s.r2;
                }
            }
            if (met) {
                if (gl == 0) {
                    G.sync_warp[sg] = t;
                    G.sync_idx[sg] = j;
                }
                crun = false;
            } else if (cn == kContCap) {
                if (gl == 0) atomicOr(&S.flags, 1u);  // give up: exact fallback below
                crun = false;
            } else {
                if (gl == 0) cl[cn] = pack_entry(m);
                ++cn;
            }
        }
        if (gl == 0 && sg < kSegs) G.cont_count[sg] = cn;
        __syncthreads();
    }

    if (!(S.flags & 1u)) {
        // ---- 3. chain walk, then copy in chain order.  Nearly always every
        // continuation meets the next segment's list, so the chain is
        // segments 0..K in order (K: the first segment with no link): warp
        // 0 then sets it up at once -- output offsets by a scan of the
        // segments' contributions, each segment's preceding entry by a max
        // scan (entry indices grow with the segment).  Otherwise one
        // thread walks the links.
        bool chained = false;
        if (warp == 0 && lim_pos > 0) {
            constexpr uint32_t kPer = (kSegs + 31u) / 32u;  // segments per lane, contiguous
            uint32_t kf = kSegs;
            bool gap = false;
#pragma unroll
            for (uint32_t u = 0; u < kPer; ++u) {
                const uint32_t i = lane * kPer + u;
                if (i < kSegs && G.sync_warp[i] == kNoWarp && i < kf) kf = i;
            }
            const uint32_t K = __reduce_min_sync(kFull, kf);  // segment 0 always parses, so K < kSegs
#pragma unroll
            for (uint32_t u = 0; u < kPer; ++u) {
                const uint32_t i = lane * kPer + u;
                if (i < K && G.sync_warp[i] != i + 1u) gap = true;
            }
            chained = !__any_sync(kFull, gap);
            if (chained) {
                uint32_t con[kPer], lst1[kPer], sum = 0, lmax = 0;
#pragma unroll
                for (uint32_t u = 0; u < kPer; ++u) {
                    const uint32_t i = lane * kPer + u;
                    con[u] = 0;
                    lst1[u] = 0;
                    if (i <= K) {
                        const uint32_t from = i ? static_cast<uint32_t>(G.sync_idx[i - 1u]) : 0u;
                        const uint32_t ns = G.spec_count[i], nc = G.cont_count[i];
                        con[u] = ns - from + nc;
                        if (con[u]) lst1[u] = 1u + i * kLaneCap + (nc ? kSpecCap + nc - 1u : ns - 1u);
                    }
                    sum += con[u];
                    lmax = lst1[u] > lmax ? lst1[u] : lmax;
                }
                // exclusive scans over the lanes: sum of contributions, max of last entries (+1)
                uint32_t incl = sum, mx = lmax;
#pragma unroll
                for (uint32_t d = 1; d < 32u; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(kFull, incl, d), om = __shfl_up_sync(kFull, mx, d);
                    if (lane >= d) {
                        incl += o;
                        mx = om > mx ? om : mx;
                    }
                }
                uint32_t acc = incl - sum, last1 = __shfl_up_sync(kFull, mx, 1);
                if (lane == 0) last1 = 0;
#pragma unroll
                for (uint32_t u = 0; u < kPer; ++u) {
                    const uint32_t i = lane * kPer + u;
                    if (i >= kSegs) continue;
                    const bool on = i <= K;
                    G.on_chain[i] = on ? 1u : 0u;
                    if (on) {
                        G.chain_from[i] = i ? G.sync_idx[i - 1u] : 0u;
                        G.out_off[i] = acc;
                        G.prev_last[i] = last1 ? last1 - 1u : kNoEntry;
                    }
                    acc += con[u];
                    last1 = lst1[u] > last1 ? lst1[u] : last1;
                }
                if (lane == 31u) S.total = incl;
            }
        }
        chained = __syncthreads_or(chained);
        if (tid == 0 && !chained) {
            for (uint32_t i = 0; i < kSegs; ++i) G.on_chain[i] = 0;
            uint32_t cur = 0, from = 0, acc = 0, last = kNoEntry;
            if (lim_pos > 0) {
                for (;;) {
                    G.on_chain[cur] = 1;
                    G.chain_from[cur] = from;
                    G.out_off[cur] = acc;
                    G.prev_last[cur] = last;
                    const uint32_t ns = G.spec_count[cur], nc = G.cont_count[cur];
                    acc += (ns - from) + nc;
                    if (ns + nc > from) last = cur * kLaneCap + (nc ? kSpecCap + nc - 1u : ns - 1u);
                    const uint32_t nx = G.sync_warp[cur];
                    if (nx == kNoWarp) break;
                    from = G.sync_idx[cur];
                    cur = nx;
                }
            }
            S.total = acc;
        }
        __syncthreads();
        const uint32_t total = S.total;
        const uint32_t keep = total < a.max_seqs ? total : a.max_seqs;
        // Write {ll, ml-3, off} in chain order: an entry's literal length is
        // its start minus the end of the entry before it -- the previous
        // entry of the same list, or for a segment's first copied entry the
        // last entry contributed before it, which the chain walk located.
        const uint32_t csg = tid / GL, csl = tid % GL;  // segment whose list this thread copies
        if (csg < kSegs && G.on_chain[csg]) {
            const uint32_t from = G.chain_from[csg], ns = G.spec_count[csg], nc = G.cont_count[csg];
            const uint32_t base = G.out_off[csg];
            const uint2 *mine = seg + csg * kLaneCap;
            uint32_t cov = 0;
            for (uint32_t i = from + csl; i < ns + nc; i += GL) {
                const uint32_t o = base + (i - from);
                if (o >= keep) break;
                const uint2 e = mine[i < ns ? i : kSpecCap + (i - ns)];
                const uint32_t pi =
                    i > from ? csg * kLaneCap + (i - 1u < ns ? i - 1u : kSpecCap + (i - 1u - ns)) : G.prev_last[csg];
                uint32_t pe = 0;
                if (pi != kNoEntry) {
                    const uint32_t px = seg[pi].x;
                    pe = (px & 0xFFFFu) + (px >> 16) + kMinMatch;
                }
                const uint32_t st0 = e.x & 0xFFFFu, mlm3 = e.x >> 16;
                const uint32_t ll = st0 - pe;
                cov += mlm3 + kMinMatch;
                if constexpr (kRef) {
                    uint32_t *r = a.ref_seqs + (static_cast<uint64_t>(wi) * a.max_seqs + o) * 3u;
                    r[0] = ll;
                    r[1] = mlm3;
                    r[2] = e.y;
                } else {
                    a.packed[static_cast<uint64_t>(wi) * a.max_seqs + o] = make_uint2(ll | (mlm3 << 16), e.y);
                }
            }
            if (cov) atomicAdd(&S.covered, cov);
        }
        __syncthreads();
        if (tid == 0) {
            a.seq_counts[wi] = keep;
            if (a.lit_counts) a.lit_counts[wi] = size - S.covered;
        }
    } else if (warp == 0) {
        // ---- exact warp-wide parse of the whole window
        PState fs{0u, 1u, 4u, 8u};
        CandBuf fcb{cand, size, 0u, 0u, 0u, 0u};
        fcb.init(0u);
        uint32_t idx = 0, cov = 0, prev_end = 0;
        Match m;
        while (fs.p + 3u < size) {
            if (!warp_step(win, bm, fcb, size, lazy, fs, m)) continue;
            if (idx < a.max_seqs && lane == 0) {
                const uint32_t ll = m.start - prev_end;
                if constexpr (kRef) {
                    uint32_t *r = a.ref_seqs + (static_cast<uint64_t>(wi) * a.max_seqs + idx) * 3u;
                    r[0] = ll;
                    r[1] = m.len - kMinMatch;
                    r[2] = m.off;
                } else {
                    a.packed[static_cast<uint64_t>(wi) * a.max_seqs + idx] =
                        make_uint2(ll | ((m.len - kMinMatch) << 16), m.off);
                }
            }
            if (idx < a.max_seqs) cov += m.len;
            ++idx;
            prev_end = m.start + m.len;
        }
        if (lane == 0) {
            a.seq_counts[wi] = idx < a.max_seqs ? idx : a.max_seqs;
            if (a.lit_counts) a.lit_counts[wi] = size - cov;
            atomicAdd(a.status + 1, 1u);  // fallback counter (diagnostics)
        }
    }
}

template <bool kRef, uint32_t SegW>
__global__ void __launch_bounds__(SegCfg<SegW>::kThreads, SegCfg<SegW>::kMinBlocks)
    zstd_seg_parse_kernel(Zstd2Args a) {
    using C = SegCfg<SegW>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    SmemLayout<SegSmem<C::kSegs>> &M = *reinterpret_cast<SmemLayout<SegSmem<C::kSegs>> *>(smem_raw);
    ParseScalars &S = M.s;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t parity = 0;
    if (tid == 0) {
        mbar_init(&S.bar, 1);
        fence_mbar_init();
    }
    for (uint32_t i = tid; i < kPre / 4; i += C::kThreads) reinterpret_cast<uint32_t *>(M.data)[i] = 0u;
    Win win{M.data + kPre};
    for (uint32_t wi = blockIdx.x; wi < a.num_windows; wi += gridDim.x) {
        uint64_t start;
        uint32_t size;
        window_of(a, wi, start, size);
        __syncthreads();  // previous window fully consumed
        if (tid == 0) {
            S.flags = 0;
            S.covered = 0;
        }
        __syncthreads();
        if (warp == 0) {
            if (!stage_window(M.data + kPre, a.src + start, size, &S.bar, parity, a.status) && lane == 0)
                S.flags = 2u;
        }
        __syncthreads();
        if (S.flags & 2u) return;  // bulk copy never completed: status already recorded, all threads leave
        verify_window<C::kThreads / 32>(win, M.bm, a.cand + start, size);
        __syncthreads();
        parse_segments<kRef, SegW>(a, M.p, S, win, M.bm, a.cand + start,
                                   a.seg + static_cast<uint64_t>(wi) * a.seg_stride, wi, size, a.lazy != 0);
    }
}

// ---------------------------------------------------------------- lane parse
// First set bit of bm in [p, stop), else stop.
__device__ __forceinline__ uint32_t next_bit(const uint32_t *bm, uint32_t p, uint32_t stop) {
    if (p >= stop) return stop;
    uint32_t i = p >> 5, b = bm[i] & (~0u << (p & 31u));
    while (!b) {
        if ((++i << 5) >= stop) return stop;
        b = bm[i];
    }
    const uint32_t f = (i << 5) + static_cast<uint32_t>(__ffs(b)) - 1u;
    return f < stop ? f : stop;
}

// Equal bytes (0-8) at the start of two 8-byte reads.
__device__ __forceinline__ uint32_t equal8(const Win &w, uint32_t c, uint32_t q) {
    uint32_t ql, qh, cl, ch;
    w.u64(static_cast<int>(q), ql, qh);
    w.u64(static_cast<int>(c), cl, ch);
    const uint32_t dl = ql ^ cl, dh = qh ^ ch;
    return dl ? (static_cast<uint32_t>(__ffs(dl)) - 1u) >> 3
              : (dh ? 4u + ((static_cast<uint32_t>(__ffs(dh)) - 1u) >> 3) : 8u);
}

// Per lane: first index in [0, lim) where bytes c+i and q+i differ, else lim
// (0 for lanes without act).  All lanes call it.  Three matches in four end in
// the first 8 bytes, which each lane compares alone, as it does the next 32;
// the lanes still open then are finished one by one by the whole warp, 128
// bytes per iteration, so that a long match does not hold 31 lanes for long.
__device__ __forceinline__ uint32_t extend_lanes(const Win &w, uint32_t c, uint32_t q, uint32_t lim, bool act) {
    const uint32_t lane = lane_id();
    uint32_t k = 0;
    bool open = act && lim > 0u;
    if (open) {
        const uint32_t e = equal8(w, c, q);
        k = e < lim ? e : lim;
        open = e == 8u && lim > 8u;
    }
#pragma unroll 1
    for (uint32_t r = 0; r < 2u; ++r) {
        if (!__any_sync(kFull, open)) return k;
        if (open) {
            uint32_t e = equal8(w, c + k, q + k);
            if (e == 8u) e += equal8(w, c + k + 8u, q + k + 8u);
            open = e == 16u && lim > k + 16u;
            k = k + e < lim ? k + e : lim;
        }
    }
    for (uint32_t pend; (pend = __ballot_sync(kFull, open)) != 0u;) {
        const uint32_t hl = static_cast<uint32_t>(__ffs(pend)) - 1u;
        const uint32_t hk = __shfl_sync(kFull, k, hl);
        const uint32_t hc = __shfl_sync(kFull, c, hl) + hk, hq = __shfl_sync(kFull, q, hl) + hk;
        const uint32_t end = hq + extend_warp(w, hc, hq, __shfl_sync(kFull, lim, hl) - hk);
        // lanes inside the same match at the same distance end there too
        if (open && q - c == hq - hc && q + k >= hq && q + k <= end) {
            k = end - q;
            open = false;
        }
    }
    return k;
}

// The match a parse takes at its event position f (lanes with act): a hash
// match, or with kRep one at repeat offset rep (0: hash match), extended, with
// the lazy step (:278-307).
template <bool kRep>
__device__ __forceinline__ void lane_match(const Win &w, const uint32_t *bm, const uint16_t *cand, uint32_t size,
                                           bool lazy, bool act, uint32_t f, uint32_t rep, Match &m) {
    const uint32_t fc = act ? f : 0u;
    const uint32_t c0 = kRep && act && rep ? fc - rep : cand[fc], c1 = cand[fc + 1u];
    // skipped when it is the same match one byte on, which is never longer (warp_step)
    const bool ltry = act && lazy && fc + 4u < size && bm_bit(bm, fc + 1u) && c1 != c0 + 1u;
    m.start = fc;
    m.len = kMinMatch + extend_lanes(w, c0 + kMinMatch, fc + kMinMatch, act ? size - fc - kMinMatch : 0u, act);
    m.off = fc - c0;
    if (__any_sync(kFull, ltry)) {
        const uint32_t l2 = kMinMatch + extend_lanes(w, c1 + kMinMatch, fc + 1u + kMinMatch,
                                                     ltry ? size - fc - 1u - kMinMatch : 0u, ltry);
        if (ltry && l2 > m.len + 1u) {
            m.start = fc + 1u;
            m.len = l2;
            m.off = fc + 1u - c1;
        }
    }
}

// List entry of a match found at position f: {start | (ml-3) << 16,
// offset | lazy << 16}, lazy: the match starts at f + 1.
__device__ __forceinline__ uint2 lane_entry(const Match &m, uint32_t f) {
    return make_uint2(m.start | ((m.len - kMinMatch) << 16), m.off | ((m.start - f) << 16));
}
__device__ __forceinline__ uint32_t entry_end(uint2 e) { return (e.x & 0xFFFFu) + (e.x >> 16) + kMinMatch; }

// Repeat offsets before entry i of the list of a whole window.
__device__ __forceinline__ void reps_before(const uint2 *list, uint32_t i, uint32_t &a, uint32_t &b, uint32_t &c) {
    a = i >= 1u ? list[i - 1u].y & 0xFFFFu : 1u;
    b = i >= 2u ? list[i - 2u].y & 0xFFFFu : (i == 1u ? 1u : 4u);
    c = i >= 3u ? list[i - 3u].y & 0xFFFFu : (i == 2u ? 1u : (i == 1u ? 4u : 8u));
}

// The next positions of a parse with repeat offsets r0, r1, r2, from p on (below
// stop): ev, the position of the first event among p .. p+7 and its repeat
// offset (0: a hash match); else a position reached, up to 64 further on.
__device__ __forceinline__ uint32_t rep_event(const Win &w, const uint32_t *bm, uint32_t p, uint32_t stop, uint32_t r0,
                                              uint32_t r1, uint32_t r2, uint32_t &rep, bool &ev) {
    const uint32_t n = min(stop - p, 8u), valid = (1u << n) - 1u;
    const uint32_t H = __funnelshift_r(bm[p >> 5], bm[(p >> 5) + 1u], p) & valid;  // (the shift counts modulo 32)
    uint32_t hit[3];
#pragma unroll
    for (uint32_t k = 0; k < 3u; ++k) {
        const uint32_t r = k == 0u ? r0 : (k == 1u ? r1 : r2);
        const uint32_t skip = r > p ? r - p : 0u;  // positions whose source is before the window
        hit[k] = skip < 8u ? rep3_scan<2>(w, p, r) & (valid << skip) : 0u;
    }
    const uint32_t any = H | ((hit[0] | hit[1] | hit[2]) & valid);
    ev = any != 0u;
    rep = 0;
    if (ev) {
        const uint32_t k = static_cast<uint32_t>(__ffs(any)) - 1u;
        if (!((H >> k) & 1u)) rep = (hit[0] >> k) & 1u ? r0 : ((hit[1] >> k) & 1u ? r1 : r2);
        return p + k;
    }
    p += n;
    const uint32_t ro[3] = {r0, r1, r2};
#pragma unroll 1
    for (uint32_t i = 0; i < 4u && p + 16u <= stop && max(max(r0, r1), r2) <= p; ++i) {
        if ((__funnelshift_r(bm[p >> 5], bm[(p >> 5) + 1u], p) & 0xFFFFu) || rep3_any16(w, p, ro, 16u)) break;
        p += 16u;
    }
    return p;
}

// Step 1: every lane parses segments of its warp's pool, without repeat offsets
// or (kRep) with them, from {1,4,8}.
template <bool kRep, uint32_t kWarps>
__device__ __forceinline__ void lane_parse(LaneSmem<kWarps> &N, const Win &win, const uint32_t *bm, const uint16_t *cand,
                                           uint2 *seg, uint32_t size, uint32_t nact, bool lazy) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, lt = lanemask_lt();
    // A short window's segments are spread over all warps: fewer lanes of a warp
    // wait for one another.
    const uint32_t pool = (nact + kWarps - 1u) / kWarps;
    uint32_t next = warp * pool;
    const uint32_t end = next + pool < nact ? next + pool : nact;
    bool has = false;
    uint32_t s = 0, p = 0, n = 0, r0 = 0, r1 = 0, r2 = 0;
    for (;;) {
        const uint32_t need = __ballot_sync(kFull, !has);
        if (need && next < end) {
            const uint32_t mine = next + static_cast<uint32_t>(__popc(need & lt));
            if (!has && mine < end) {
                has = true;
                s = mine;
                p = s * kLSegW;
                n = 0;
                if constexpr (kRep) r0 = 1u, r1 = 4u, r2 = 8u;
            }
            next += static_cast<uint32_t>(__popc(need));
        }
        if (!__any_sync(kFull, has)) break;
        const uint32_t seg_end = (s + 1u) * kLSegW;
        uint32_t f, rep = 0;
        bool ev = false;
        if constexpr (kRep) {
            f = has ? rep_event(win, bm, p, min(seg_end, size - 3u), r0, r1, r2, rep, ev) : 0u;
        } else {
            f = has ? next_bit(bm, p, seg_end) : seg_end;
            ev = has && f < seg_end;
        }
        if (__any_sync(kFull, ev)) {
            Match m;
            lane_match<kRep>(win, bm, cand, size, lazy, ev, f, rep, m);
            if (ev) {
                seg[s * kLCap + n] = lane_entry(m, f);
                ++n;
                p = m.start + m.len;
                if constexpr (kRep) r2 = r1, r1 = r0, r0 = m.off;
            }
        }
        if constexpr (kRep) {
            if (has && !ev) p = f;
            if (has && p >= min(seg_end, size - 3u)) {
                N.count[s] = static_cast<uint8_t>(n);
                N.link[s] = static_cast<uint16_t>(p > seg_end ? p - seg_end : 0u);
                has = false;
            }
        } else if (has && (!ev || p >= seg_end)) {  // no match left, or the last one ends past the segment
            N.count[s] = static_cast<uint8_t>(n);
            N.link[s] = static_cast<uint16_t>(ev ? p - seg_end : 0u);
            has = false;
        }
    }
}

// Where a segment's continuation puts its next match.
struct ContSlot {
    uint32_t cur, end;  // next slot, the slot of its block's last entry (which leads to the next chunk)
    __device__ __forceinline__ explicit ContSlot(uint32_t s) : cur(kLContBase + s * kLCont), end(cur + kLCont - 1u) {}
    // false when there is no room for it
    __device__ __forceinline__ bool put(ParseScalars &S, uint2 *seg, const uint2 &e) {
        if (cur == end) {
            const uint32_t c = atomicAdd(&S.chunks, 1u);
            if (c >= kLChunks) return false;
            seg[end].x = c;
            cur = kLChunkBase + c * kLChunk;
            end = cur + kLChunk - 1u;
        }
        seg[cur++] = e;
        return true;
    }
};
// Slot of match i of segment s's continuation.
__device__ __forceinline__ uint32_t cont_slot(const uint2 *seg, uint32_t s, uint32_t i) {
    uint32_t at = kLContBase + s * kLCont, n = kLCont - 1u;  // block and the matches it holds
    for (; i >= n; n = kLChunk - 1u) {
        i -= n;
        at = kLChunkBase + seg[at + n].x * kLChunk;
    }
    return at + i;
}

// Step 2, first half: where each segment's parse joins a later segment's list.
template <uint32_t kWarps>
__device__ __forceinline__ void lane_link(LaneSmem<kWarps> &N, ParseScalars &S, const Win &win, const uint32_t *bm,
                                          const uint16_t *cand, uint2 *seg, uint32_t size, uint32_t nact,
                                          uint32_t lim_pos, bool lazy) {
    const uint32_t tid = threadIdx.x;
#pragma unroll 1
    for (uint32_t s = tid; s < kLSegs; s += 32u * kWarps) {
        uint32_t E = (s + 1u) * kLSegW + (s < nact ? N.link[s] : 0u);  // position the parse has reached
        uint32_t t = kNoWarp, j = 0, cn = 0;
        ContSlot slot(s);
        bool run = s < nact;
        for (;;) {
            if (run && E >= lim_pos) run = false;  // the parse is over: no link
            if (run) {
                t = E / kLSegW;
                j = 0;
                uint32_t pe = t * kLSegW;  // end of the list's match before E
                if (E != pe) {
                    const uint32_t tc = N.count[t];
                    for (; j < tc; ++j) {
                        const uint2 e = seg[t * kLCap + j];
                        if ((e.x & 0xFFFFu) - (e.y >> 16) >= E) break;  // found at or after E
                        pe = entry_end(e);
                    }
                }
                if (pe <= E) run = false;  // both go on from E without a match in between
                else t = kNoWarp;
            }
            if (!__any_sync(kFull, run)) break;
            const uint32_t f = run ? next_bit(bm, E, lim_pos) : lim_pos;
            const bool ev = run && f < lim_pos;
            if (run && !ev) run = false;
            Match m;
            lane_match<false>(win, bm, cand, size, lazy, ev, f, 0u, m);
            if (ev) {
                if (cn == kLMost || !slot.put(S, seg, lane_entry(m, f))) {
                    atomicOr(&S.flags, 4u);
                    run = false;
                } else {
                    ++cn;
                    E = m.start + m.len;
                }
            }
        }
        N.link[s] = static_cast<uint16_t>(t);
        N.from[s] = static_cast<uint8_t>(j);
        N.cont[s] = static_cast<uint8_t>(cn);
        if (s >= nact) N.count[s] = 0;
    }
}

// The same with repeat offsets: a segment's parse joins a later segment's list
// at a match that both have, with the same repeat offsets after it.
template <uint32_t kWarps>
__device__ __forceinline__ void lane_link_reps(LaneSmem<kWarps> &N, ParseScalars &S, const Win &win, const uint32_t *bm,
                                               const uint16_t *cand, uint2 *seg, uint32_t size, uint32_t nact,
                                               uint32_t lim_pos, bool lazy) {
#pragma unroll 1
    for (uint32_t s = threadIdx.x; s < kLSegs; s += 32u * kWarps) {
        bool run = s < nact;
        uint32_t p = (s + 1u) * kLSegW, r0 = 0, r1 = 0, r2 = 0;
        if (run) {
            p += N.link[s];
            reps_before(seg + s * kLCap, N.count[s], r0, r1, r2);
        }
        uint32_t link = kNoWarp, t = kNoWarp, j = 0, cn = 0, steps = 0, rep = 0, f = 0;
        bool ev = false;
        ContSlot slot(s);
        for (;;) {
            // (the parse is over, or some segment has found no place to join)
            if (p >= lim_pos || (*const_cast<volatile uint32_t *>(&S.flags) & 4u)) run = false;
            const uint32_t runs = __ballot_sync(kFull, run);
            if (!runs) break;
            if (run && !ev) {
                f = rep_event(win, bm, p, lim_pos, r0, r1, r2, rep, ev);
                if (!ev) p = f;
                if (++steps > kMostSteps) atomicOr(&S.flags, 4u);
            }
            ev = ev && run;
            // (a match takes several times as long as a step)
            if (2u * __popc(__ballot_sync(kFull, ev)) < __popc(runs)) continue;
            Match m;
            lane_match<true>(win, bm, cand, size, lazy, ev, f, rep, m);
            if (ev) {
                ev = false;
                const uint2 e = lane_entry(m, f);
                if (f / kLSegW != t) {
                    t = f / kLSegW;
                    j = 0;
                }
                const uint2 *tl = seg + t * kLCap;
                const uint32_t tc = N.count[t];
                while (j < tc && (tl[j].x & 0xFFFFu) < m.start) ++j;
                if (j < tc && tl[j].x == e.x && (tl[j].y & 0xFFFFu) == m.off) {
                    uint32_t a, b, c;
                    reps_before(tl, j, a, b, c);
                    if (a == r0 && b == r1) {
                        link = t;
                        run = false;
                    }
                }
                if (run) {
                    if (cn == kLMost || !slot.put(S, seg, e)) {
                        atomicOr(&S.flags, 4u);
                        run = false;
                    } else {
                        ++cn;
                        p = m.start + m.len;
                        r2 = r1, r1 = r0, r0 = m.off;
                    }
                }
            }
        }
        N.link[s] = static_cast<uint16_t>(link);
        N.from[s] = static_cast<uint8_t>(j);
        N.cont[s] = static_cast<uint8_t>(cn);
        if (s >= nact) N.count[s] = 0;
    }
}

// Step 2, second half (whole CTA): the segments on the chain from segment 0,
// the entry each is joined at and its output offset; the chain's entries.
// Marking doubles: when the marked segments are those fewer than 2^r links
// from segment 0 and `link` leads 2^r links on, the marked ones mark theirs.
template <uint32_t kWarps>
__device__ __forceinline__ uint32_t lane_chain(LaneSmem<kWarps> &N, ParseScalars &S, bool any) {
    static_assert(32u * kWarps >= kLSegs, "a thread for every segment");
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const bool mine = tid < kLSegs;  // thread s keeps segment s
    uint32_t n = mine ? N.link[tid] : kNoWarp, l = n, j = mine ? N.from[tid] : 0u;
    bool on = any && tid == 0u;
    if (tid < kLSegs / 32u) N.chain[tid] = any && tid == 0 ? 1u : 0u;
    __syncthreads();
    for (;;) {
        bool go = false;
        if (n != kNoWarp) {
            if (on) atomicOr(&N.chain[n >> 5], 1u << (n & 31u));
            n = N.link[n];
            go = n != kNoWarp;
        }
        go = __syncthreads_or(go);
        if (mine) on = (N.chain[tid >> 5] >> (tid & 31u)) & 1u;
        if (!go) break;
        if (mine) N.link[tid] = static_cast<uint16_t>(n);
        __syncthreads();
    }
    if (on && l != kNoWarp) N.from[l] = static_cast<uint8_t>(j);
    if (tid == 0) N.from[0] = 0;
    __syncthreads();
    const uint32_t sum = on ? N.count[tid] - N.from[tid] + N.cont[tid] : 0u;
    uint32_t x = sum;
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31u) S.warp_sum[warp] = x;
    __syncthreads();
    uint32_t base = 0, total = 0;
    for (uint32_t w = 0; w < kWarps; ++w) {
        const uint32_t v = S.warp_sum[w];
        if (w < warp) base += v;
        total += v;
    }
    if (mine) N.link[tid] = static_cast<uint16_t>(base + x - sum);
    return total;
}

// The chain's entries (the first `total`) in order into the output slots, then
// from there to the front of the scratch, over the lists.
template <bool kRef, uint32_t kWarps>
__device__ __forceinline__ void lane_gather(const Zstd2Args &a, const LaneSmem<kWarps> &N, uint2 *seg, uint32_t wi,
                                            uint32_t total) {
    const uint32_t tid = threadIdx.x;
    constexpr uint32_t kThreads = 32u * kWarps;
    uint2 *pk = kRef ? nullptr : a.packed + static_cast<uint64_t>(wi) * a.max_seqs;
    uint32_t *rk = kRef ? a.ref_seqs + static_cast<uint64_t>(wi) * a.max_seqs * 3u : nullptr;
    for (uint32_t s = tid >> 2; s < kLSegs; s += kThreads / 4u) {
        if (!((N.chain[s >> 5] >> (s & 31u)) & 1u)) continue;
        const uint32_t from = N.from[s], ns = N.count[s], nc = N.cont[s];
        for (uint32_t i = from + (tid & 3u); i < ns + nc; i += 4u) {
            const uint32_t o = N.link[s] + (i - from);
            if (o >= total) break;
            const uint2 e = seg[i < ns ? s * kLCap + i : cont_slot(seg, s, i - ns)];
            if constexpr (kRef) {
                rk[3u * o] = e.x;
                rk[3u * o + 1u] = e.y;
            } else {
                pk[o] = e;
            }
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < total; i += kThreads) {
        if constexpr (kRef) seg[i] = make_uint2(rk[3u * i], rk[3u * i + 1u]);
        else seg[i] = pk[i];
    }
    __syncthreads();
}

// Step 3: runs of literals in which a repeat offset matches on 3 bytes
// (zstd_compress.cu:259-275), into N.fix.run (unsorted, repeats possible);
// S.count counts them.  Run i lies before entry i of the list, the last one
// after it.
template <uint32_t kWarps>
__device__ __forceinline__ void lane_check(LaneSmem<kWarps> &N, ParseScalars &S, const Win &win, const uint2 *list,
                                           uint32_t total, uint32_t lim_pos) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    // Few groups of 32 runs (long runs, so many tasks each) are shared by
    // several warps, each of which repeats the group's scan: 16 warps up to 8
    // groups, 4 up to 16 (a window of random bytes is one run of 4096 tasks).
    const uint32_t groups = total / 32u + 1u;
    const uint32_t team = groups <= 8u ? kWarps : (groups <= kWarps ? 4u : 1u);
    for (uint32_t g = warp / team * 32u; g <= total; g += kWarps / team * 32u) {
        const uint32_t i = g + lane;
        uint32_t lo = 0, hi = 0, r1 = 1, r2 = 4, r3 = 8;
        if (i <= total) {
            if (i) lo = entry_end(list[i - 1u]);
            hi = lim_pos;
            if (i < total) {  // up to the hash match (the byte before a lazy match's start)
                const uint2 e = list[i];
                hi = (e.x & 0xFFFFu) - (e.y >> 16);
            }
            reps_before(list, i, r1, r2, r3);
        }
        const uint32_t nt = hi > lo ? (hi - lo + 15u) >> 4 : 0u;  // tasks of 16 positions
        uint32_t x = nt;
#pragma unroll
        for (uint32_t d = 1; d < 32u; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, d);
            if (lane >= d) x += y;
        }
        const uint32_t T = __shfl_sync(kFull, x, 31), before = x - nt;
        const uint32_t span = lo | (hi << 16), r12 = r1 | (r2 << 16);  // hi <= 65533
        bool found = false;
        for (uint32_t b = warp % team * 32u; b < T; b += team * 32u) {
            const uint32_t t = b + lane;
            uint32_t o = 0;  // the run of task t: the first lane whose inclusive count is above t
#pragma unroll
            for (uint32_t d = 16; d >= 1u; d >>= 1)
                if (__shfl_sync(kFull, x, o + d - 1u) <= t) o += d;
            o &= 31u;  // t >= T: any
            const uint32_t k = t - __shfl_sync(kFull, before, o);
            const uint32_t sp = __shfl_sync(kFull, span, o), ra = __shfl_sync(kFull, r12, o),
                           rc = __shfl_sync(kFull, r3, o);
            bool hit = false;
            if (t < T) {
                const uint32_t q0 = (sp & 0xFFFFu) + 16u * k, left = (sp >> 16) - q0;
                const uint32_t ro[3] = {ra & 0xFFFFu, ra >> 16, rc};
                if (max(max(ro[0], ro[1]), ro[2]) <= q0) {
                    hit = rep3_any16(win, q0, ro, left);
                } else {  // sources before the window start do not count
                    const uint32_t upto = left < 16u ? (1u << left) - 1u : 0xFFFFu;
                    uint32_t any = 0;
#pragma unroll 1
                    for (uint32_t v = 0; v < 3u; ++v) {
                        const uint32_t r = v == 0u ? ro[0] : (v == 1u ? ro[1] : ro[2]);
                        const uint32_t skip = r > q0 ? r - q0 : 0u;
                        if (skip < 16u) any |= rep3_scan<4>(win, q0, r) & (0xFFFFu << skip);
                    }
                    hit = (any & upto) != 0u;
                }
            }
            if (__any_sync(kFull, hit)) {
                const uint32_t po = __shfl_up_sync(kFull, o, 1);
                const bool ph = __shfl_up_sync(kFull, hit ? 1u : 0u, 1) != 0u;
                found = true;
                if (hit && !(lane > 0u && ph && po == o)) {
                    const uint32_t at = atomicAdd(&S.count, 1u);
                    if (at < kFixes) {
                        N.fix.run[at] = static_cast<uint16_t>(g + o);
                        N.fix.pos[at] = static_cast<uint16_t>((sp & 0xFFFFu) + 16u * k);
                    }
                }
            }
        }
        // too many to mend
        if (found && __any_sync(kFull, *const_cast<volatile uint32_t *>(&S.count) > kMostFixes)) return;
    }
}

// Step 4, first part (warp 0): the n recorded runs sorted, each once, with its
// lowest recorded position; returns how many.
template <uint32_t kWarps>
__device__ __forceinline__ uint32_t sort_runs(LaneSmem<kWarps> &N, uint32_t n) {
    const uint32_t lane = lane_id(), lt = lanemask_lt();
    auto key = [&](uint32_t i) { return (static_cast<uint32_t>(N.fix.run[i]) << 16) | N.fix.pos[i]; };
    uint32_t m = 0;
    for (uint32_t i = lane; i < n; i += 32u) {  // each to its rank, through meet and shift
        const uint32_t v = key(i);
        uint32_t rank = 0;
        for (uint32_t k = 0; k < n; ++k) {
            const uint32_t o = key(k);
            rank += o < v || (o == v && k < i) ? 1u : 0u;
        }
        N.fix.meet[rank] = static_cast<uint16_t>(v >> 16);
        N.fix.shift[rank] = static_cast<int16_t>(v & 0xFFFFu);
    }
    __syncwarp();
    for (uint32_t i0 = 0; i0 < n; i0 += 32u) {  // the first of each run, moved together
        const uint32_t i = i0 + lane;
        const bool first = i < n && (i == 0u || N.fix.meet[i] != N.fix.meet[i - 1u]);
        const uint32_t f = __ballot_sync(kFull, first), at = m + static_cast<uint32_t>(__popc(f & lt));
        if (first) {
            N.fix.run[at] = N.fix.meet[i];
            N.fix.pos[at] = static_cast<uint16_t>(N.fix.shift[i]);
        }
        m += static_cast<uint32_t>(__popc(f));
    }
    __syncwarp();
    return m;
}

// Past literals that start no match, 512 at a time (16 per lane), for long
// stretches without a hash match (a window of random bytes is one): a position
// from which on the state is the same.
__device__ __noinline__ uint32_t skip_literals(Win win, const uint32_t *bm, uint32_t lim_pos, PState st) {
    const uint32_t lane = lane_id();
    const uint32_t ro[3] = {st.r0, st.r1, st.r2};
    while (st.p + 512u <= lim_pos && max(max(ro[0], ro[1]), ro[2]) <= st.p) {
        const uint32_t sh = st.p & 31u;
        uint32_t b = lane <= 16u ? bm[(st.p >> 5) + lane] : 0u;
        if (lane == 0u) b &= ~0u << sh;
        if (lane == 16u) b &= (1u << sh) - 1u;
        if (__any_sync(kFull, b != 0u)) break;
        const uint32_t hit = __ballot_sync(kFull, rep3_any16(win, st.p + 16u * lane, ro, 16u));
        if (hit) return st.p + 16u * (static_cast<uint32_t>(__ffs(hit)) - 1u);
        st.p += 512u;
    }
    return st.p;
}

// Step 4, second part: mend r (one warp) parses run i exactly from its first
// repeat-offset match (less than 16 positions before it; the literals up to
// there are checked) until it emits entry `meet` of the list with the same
// repeat offsets.
template <uint32_t kWarps>
__device__ __noinline__ void mend_run(LaneSmem<kWarps> &N, ParseScalars &S, Win win, const uint32_t *bm, const uint16_t *cand,
                                      uint2 *seg, uint32_t size, bool lazy, uint32_t total, uint32_t r,
                                      uint32_t cap) {
    const uint32_t lane = lane_id();
    const uint32_t i = N.fix.run[r];
    const uint2 *list = seg;
    uint2 *out = seg + kLContBase + r * cap;
    const uint32_t lim_pos = size - 3u;  // a window with a run to mend has more than 3 bytes
    PState st;
    st.p = N.fix.pos[r];
    reps_before(list, i, st.r0, st.r1, st.r2);
    CandBuf cb{cand, size, 0u, 0u, 0u, 0u};
    cb.init(st.p);
    uint32_t j = i, n = 0, meet = total;
    while (st.p + 3u < size) {
        const uint32_t *ahead = bm + (st.p >> 5);
        if ((ahead[1] | ahead[2] | ahead[3]) == 0u) st.p = skip_literals(win, bm, lim_pos, st);
        if (__any_sync(kFull, *const_cast<volatile uint32_t *>(&S.flags) & 4u)) break;  // another one gave up
        Match m;
        if (!warp_step(win, bm, cb, size, lazy, st, m)) continue;
        for (;;) {  // first entry with start >= m.start
            const uint32_t idx = j + lane;
            const uint32_t b = __ballot_sync(kFull, idx >= total || (list[idx].x & 0xFFFFu) >= m.start);
            if (b) {
                j += static_cast<uint32_t>(__ffs(b)) - 1u;
                break;
            }
            j += 32u;
        }
        if (j < total && list[j].x == pack_entry(m).x) {
            uint32_t e0, e1, e2;
            reps_before(list, j + 1u, e0, e1, e2);
            if (e0 == st.r0 && e1 == st.r1 && e2 == st.r2) {
                meet = j;
                break;
            }
        }
        if (n == cap || (n == kDenseCap && m.start - N.fix.pos[r] < kDenseCap * kDense)) {
            if (lane == 0) atomicOr(&S.flags, 4u);
            break;
        }
        if (lane == 0) out[n] = pack_entry(m);
        ++n;
    }
    if (lane == 0) {
        N.fix.meet[r] = static_cast<uint16_t>(meet);
        N.fix.len[r] = static_cast<uint8_t>(n);
        atomicAdd(&S.probe[0], n);
        atomicAdd(&S.probe[1], st.p - N.fix.pos[r]);
    }
}

template <bool kRef, uint32_t kWarps>
__device__ __noinline__ void parse_segments_out(Zstd2Args a, SegSmem<kWarps> &G, ParseScalars &S, Win win,
                                                const uint32_t *bm, const uint16_t *cand, uint2 *seg, uint32_t wi,
                                                uint32_t size, bool lazy) {
    parse_segments<kRef, kMaxWindow / kWarps>(a, G, S, win, bm, cand, seg, wi, size, lazy);
}

// The segment parse by 8-lane groups, 64 of them whatever the CTA's warps.
template <bool kRef>
__device__ __noinline__ void parse_groups_out(Zstd2Args a, SegSmem<64> &G, ParseScalars &S, Win win, const uint32_t *bm,
                                              const uint16_t *cand, uint2 *seg, uint32_t wi, uint32_t size, bool lazy) {
    using C = SegCfg<1024, 8>;
    static_assert(C::kThreads == 512 && C::kMinBlocks == 3, "what the smallest form of the lane parse has");
    parse_segments<kRef, 1024, 8>(a, G, S, win, bm, cand, seg, wi, size, lazy);
}

// Steps 1 and 2 with repeat offsets, and the output (whole CTA, S.flags clear):
// a segment's parse starts from {1,4,8} and has the state of the parse before
// it after a few matches.  False, with S.flags clear, where a segment does not
// join a list soon.
template <bool kRef, uint32_t kWarps>
__device__ __noinline__ bool parse_lanes_reps(Zstd2Args a, LaneSmem<kWarps> &N, ParseScalars &S, Win win,
                                              const uint32_t *bm, const uint16_t *cand, uint2 *seg, uint32_t wi,
                                              uint32_t size, bool lazy) {
    const uint32_t tid = threadIdx.x;
    const uint32_t lim_pos = size - 3u, nact = (lim_pos + kLSegW - 1u) / kLSegW;  // (no window of up to 3 bytes is given up)
    lane_parse<true>(N, win, bm, cand, seg, size, nact, lazy);
    __syncthreads();
    lane_link_reps(N, S, win, bm, cand, seg, size, nact, lim_pos, lazy);
    __syncthreads();
    if (S.flags & 4u) {
        __syncthreads();
        if (tid == 0) S.flags = 0;
        __syncthreads();
        return false;
    }
    uint32_t total = lane_chain(N, S, true);
    __syncthreads();
    if (total > a.max_seqs) total = a.max_seqs;
    lane_gather<kRef>(a, N, seg, wi, total);
    uint32_t cov = 0;
    for (uint32_t x = tid; x < total; x += 32u * kWarps) {
        const uint2 e = seg[x];
        cov += (e.x >> 16) + kMinMatch;
        write_seq<kRef>(a, wi, x, (e.x & 0xFFFFu) - (x ? entry_end(seg[x - 1u]) : 0u), e.x >> 16, e.y & 0xFFFFu);
    }
    if (kRef && cov) atomicAdd(&S.covered, cov);
    if (tid == 0) a.seq_counts[wi] = total;
    if (a.lit_counts) {
        __syncthreads();
        if (tid == 0) a.lit_counts[wi] = size - S.covered;
    }
    return true;
}

// Window wi to be parsed again in the way S.how (one thread).
__device__ __forceinline__ void give_up(const Zstd2Args &a, ParseScalars &S, uint32_t wi) {
    a.seg[static_cast<uint64_t>(wi + 1u) * a.seg_stride - 1u] = make_uint2(S.again, S.how);
    S.again = wi + 1u;
    a.seq_counts[wi] = 0u;
}

// kCtas: CTAs of an SM.
template <bool kRef, uint32_t kWarps, int kCtas>
__global__ void __launch_bounds__(32 * kWarps, kCtas) zstd_lane_parse_kernel(Zstd2Args a) {
    constexpr uint32_t kThreads = 32u * kWarps;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    SmemLayout<LaneSmem<kWarps>> &M = *reinterpret_cast<SmemLayout<LaneSmem<kWarps>> *>(smem_raw);
    ParseScalars &S = M.s;
    LaneSmem<kWarps> &N = M.p;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t parity = 0;
    if (tid == 0) {
        mbar_init(&S.bar, 1);
        fence_mbar_init();
        S.again = S.skip = S.streak = 0;
    }
    for (uint32_t i = tid; i < kPre / 4; i += kThreads) reinterpret_cast<uint32_t *>(M.data)[i] = 0u;
    const Win win{M.data + kPre};
    const bool lazy = a.lazy != 0;
    for (uint32_t wi = blockIdx.x; wi < a.num_windows; wi += gridDim.x) {
        uint64_t start;
        uint32_t size;
        window_of(a, wi, start, size);
        const uint16_t *cand = a.cand + start;
        uint2 *seg = a.seg + static_cast<uint64_t>(wi) * a.seg_stride;
        __syncthreads();  // previous window fully consumed
        if (tid == 0) {
            S.flags = 0;
            S.covered = 0;
            S.count = 0;
            S.chunks = 0;
            S.probe[0] = S.probe[1] = 0;
            if (S.skip && size > 3u) {
                --S.skip;
                S.flags = 16u;
                give_up(a, S, wi);
            }
        }
        __syncthreads();
        if (S.flags & 16u) continue;
        if (warp == 0) {
            if (!stage_window(M.data + kPre, a.src + start, size, &S.bar, parity, a.status) && lane == 0)
                S.flags = 2u;
        }
        __syncthreads();
        if (S.flags & 2u) return;  // bulk copy never completed: status already recorded, all threads leave
        verify_window<kWarps>(win, M.bm, cand, size);
        __syncthreads();

        const uint32_t lim_pos = size > 3u ? size - 3u : 0u;  // positions q < lim_pos can start a match
        const uint32_t nact = (lim_pos + kLSegW - 1u) / kLSegW;
        lane_parse<false>(N, win, M.bm, cand, seg, size, nact, lazy);
        __syncthreads();
        lane_link(N, S, win, M.bm, cand, seg, size, nact, lim_pos, lazy);
        __syncthreads();
        uint32_t total = lane_chain(N, S, lim_pos > 0u);
        __syncthreads();
        const bool capped = total > a.max_seqs;
        if (capped) total = a.max_seqs;
        lane_gather<kRef>(a, N, seg, wi, total);
        lane_check(N, S, win, seg, total, capped ? 0u : lim_pos);
        __syncthreads();
        uint32_t nfix = S.count, fcap = 0;
        if (nfix > 0u) {
            bool many = capped || nfix > kMostFixes;  // (uniform over the CTA)
            uint32_t n = kWarps;
            if (!many) {
                const uint32_t found = nfix;
                if (warp == 0) {
                    nfix = sort_runs(N, nfix);
                    if (lane == 0) S.mends = nfix;
                }
                __syncthreads();
                nfix = S.mends;
                many = found * 512u >= size && found >= 8u * nfix;  // few runs with matches all over them
                if (!many || nfix < n) n = nfix;
            }
            fcap = kFixEntries / nfix < kFixCap ? kFixEntries / nfix : kFixCap;
            if (many) {  // a few are tried out, unless the entries tell how dense the window is
                fcap = kTryCap;
                if (capped || (total && entry_end(seg[total - 1u]) < total * kDense)) n = 0;
            }
            for (uint32_t r = warp; r < n; r += kWarps)
                mend_run(N, S, win, M.bm, cand, seg, size, lazy, total, r, fcap);
            __syncthreads();
            if (many) {
                if (tid == 0) S.flags |= 4u;
            } else {
                if (tid == 0) {  // drop the mends that start inside an earlier one
                    uint32_t kept = 0;
                    int32_t shift = 0;
                    for (uint32_t r = 0; r < nfix; ++r) {
                        const uint32_t i = N.fix.run[r], j = N.fix.meet[r], n = N.fix.len[r];
                        if (kept && i <= N.fix.meet[kept - 1u]) continue;
                        shift += static_cast<int32_t>(n) - static_cast<int32_t>(j - i);
                        N.fix.run[kept] = static_cast<uint16_t>(i);
                        N.fix.meet[kept] = static_cast<uint16_t>(j);
                        N.fix.shift[kept] = static_cast<int16_t>(shift);
                        N.fix.len[kept] = static_cast<uint8_t>(n);
                        N.fix.list[kept] = static_cast<uint8_t>(r);
                        ++kept;
                    }
                    S.mends = kept;
                    S.total = static_cast<uint32_t>(static_cast<int32_t>(total) + shift);
                }
            }
            __syncthreads();
            nfix = S.mends;
        }
        if (S.flags & 4u) {
            if (tid == 0) {  // parsed again at the end, as are 3 windows after it at once, later 7
                const uint32_t end = total ? entry_end(seg[total - 1u]) : 0u;
                const bool dense = S.probe[1] < S.probe[0] * kTryDense || end < total * kDense;
                const bool sparse = S.probe[1] >= S.probe[0] * kSparse && end >= total * kSparse;
                S.how = dense ? 1u : (sparse ? 2u : 0u);
                S.streak = S.streak ? 7u : 3u;
                S.skip = S.streak;
                give_up(a, S, wi);
            }
            continue;
        }
        const uint32_t out_n = nfix ? S.total : total;
        const uint32_t keep = out_n < a.max_seqs ? out_n : a.max_seqs;
        uint32_t cov = 0;
        for (uint32_t x = tid; x < total; x += kThreads) {
            uint32_t o = x, pi = x;  // output index; the entry before x is prev[pi - 1]
            const uint2 *prev = seg;
            bool skip = false;
            uint32_t z = 0;  // mends that start at or before x
            for (uint32_t d = kFixes; d >= 1u; d >>= 1)
                if (z + d <= nfix && N.fix.run[z + d - 1u] <= x) z += d;
            if (z) {
                --z;
                const uint32_t j = N.fix.meet[z];
                skip = x < j;
                o = x + static_cast<uint32_t>(static_cast<int32_t>(N.fix.shift[z]));
                if (x == j && N.fix.len[z]) {
                    prev = seg + kLContBase + N.fix.list[z] * fcap;
                    pi = N.fix.len[z];
                }
            }
            if (skip || o >= keep) continue;
            const uint2 e = seg[x];
            const uint32_t pe = pi ? entry_end(prev[pi - 1u]) : 0u;
            cov += (e.x >> 16) + kMinMatch;
            write_seq<kRef>(a, wi, o, (e.x & 0xFFFFu) - pe, e.x >> 16, e.y & 0xFFFFu);
        }
        for (uint32_t z = warp; z < nfix; z += kWarps) {
            const uint32_t i = N.fix.run[z], n = N.fix.len[z];
            const uint32_t base = i + (z ? static_cast<uint32_t>(static_cast<int32_t>(N.fix.shift[z - 1u])) : 0u);
            const uint2 *fl = seg + kLContBase + N.fix.list[z] * fcap;
            for (uint32_t k = lane; k < n && base + k < keep; k += 32u) {
                const uint2 e = fl[k];
                const uint32_t pe = k ? entry_end(fl[k - 1u]) : (i ? entry_end(seg[i - 1u]) : 0u);
                cov += (e.x >> 16) + kMinMatch;
                write_seq<kRef>(a, wi, base + k, (e.x & 0xFFFFu) - pe, e.x >> 16, e.y);
            }
        }
        if (kRef && cov) atomicAdd(&S.covered, cov);
        if (tid == 0) {
            a.seq_counts[wi] = keep;
            S.streak = 0;
        }
        if (a.lit_counts) {
            __syncthreads();
            if (tid == 0) a.lit_counts[wi] = size - S.covered;
        }
    }
    // The windows given up, here and not above: a call in that loop costs every
    // window registers (256 MiB of the benchmark's data 1.36 ms against 1.31).
    __syncthreads();
    for (uint32_t w = S.again; w;) {
        const uint32_t wi = w - 1u;
        uint64_t start;
        uint32_t size;
        window_of(a, wi, start, size);
        const uint16_t *cand = a.cand + start;
        uint2 *seg = a.seg + static_cast<uint64_t>(wi) * a.seg_stride;
        const uint2 l = seg[a.seg_stride - 1u];
        __syncthreads();
        if (tid == 0) {
            S.flags = 0;
            S.covered = 0;
            S.chunks = 0;
        }
        __syncthreads();
        if (warp == 0) {
            if (!stage_window(M.data + kPre, a.src + start, size, &S.bar, parity, a.status) && lane == 0)
                S.flags = 2u;
        }
        __syncthreads();
        if (S.flags & 2u) return;
        verify_window<kWarps>(win, M.bm, cand, size);
        __syncthreads();
        if (l.y == 2u)
            parse_segments_out<kRef, kWarps>(a, N.segw, S, win, M.bm, cand, seg, wi, size, lazy);
        else if (l.y == 0u || !parse_lanes_reps<kRef, kWarps>(a, N, S, win, M.bm, cand, seg, wi, size, lazy))
            parse_groups_out<kRef>(a, N.seg, S, win, M.bm, cand, seg, wi, size, lazy);
        w = l.x;
    }
}

}  // namespace

// Scratch entries per window: the largest of the layouts, so that a buffer
// sized once serves every segment width.
template <uint32_t SegW, uint32_t GL = 32>
constexpr uint32_t seg_entries() { return SegCfg<SegW, GL>::kSegs * SegCfg<SegW, GL>::kLaneCap; }
constexpr uint32_t kSegStride = []() constexpr {
    uint32_t m = kLEntries + 1;  // (the last one leads from a window given up to the one before it)
    if (seg_entries<1024, 8>() > m) m = seg_entries<1024, 8>();
    if (seg_entries<2048>() > m) m = seg_entries<2048>();
    if (seg_entries<4096>() > m) m = seg_entries<4096>();
    if (seg_entries<8192>() > m) m = seg_entries<8192>();
    return m;
}();

size_t zstd2_seg_scratch_entries(uint32_t num_windows) { return static_cast<size_t>(num_windows) * kSegStride; }

namespace {
template <class Kernel>
cudaError_t launch_parse_kernel(Kernel kernel, uint32_t smem, uint32_t threads, SmemOnce &smem_set,
                                const Zstd2Args &a, int num_sms, int ctas_per_sm, cudaStream_t st) {
    cudaError_t e = set_smem_once(kernel, smem, smem_set);
    if (e != cudaSuccess) return e;
    int grid = num_sms * ctas_per_sm;
    if (static_cast<uint32_t>(grid) > a.num_windows) grid = static_cast<int>(a.num_windows);
    kernel<<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <bool kRef, uint32_t SegW>
cudaError_t launch_seg_parse(const Zstd2Args &a, int num_sms, int ctas_per_sm, cudaStream_t st) {
    using C = SegCfg<SegW>;
    constexpr uint32_t smem = sizeof(SmemLayout<SegSmem<C::kSegs>>);
    static_assert(smem + 1024 <= 233472 / 3, "three CTAs per SM must fit");
    static SmemOnce smem_set{0};
    return launch_parse_kernel(zstd_seg_parse_kernel<kRef, SegW>, smem, C::kThreads, smem_set, a, num_sms, ctas_per_sm,
                               st);
}

template <bool kRef, uint32_t kWarps, int kCtas>
cudaError_t launch_lane_parse(const Zstd2Args &a, int num_sms, int ctas_per_sm, cudaStream_t st) {
    constexpr uint32_t smem = sizeof(SmemLayout<LaneSmem<kWarps>>);
    static_assert(smem + 1024 <= 233472 / 3, "three CTAs per SM must fit");
    static SmemOnce smem_set{0};
    return launch_parse_kernel(zstd_lane_parse_kernel<kRef, kWarps, kCtas>, smem, 32 * kWarps, smem_set, a, num_sms,
                               ctas_per_sm < kCtas ? ctas_per_sm : kCtas, st);
}

template <bool kRef>
cudaError_t launch_parse_ref(const Zstd2Args &a, uint32_t seg_width, int num_sms, int ctas_per_sm, cudaStream_t st) {
    if (seg_width == 2048) return launch_seg_parse<kRef, 2048>(a, num_sms, ctas_per_sm, st);
    if (seg_width == 4096) return launch_seg_parse<kRef, 4096>(a, num_sms, ctas_per_sm, st);
    if (seg_width == 8192) return launch_seg_parse<kRef, 8192>(a, num_sms, ctas_per_sm, st);
    // At most one window per SM: 32 warps share it instead of 16, with all of
    // the SM's registers.  Sweep to records, 1 window 100.3 -> 89.3 us, 148
    // windows 109.6 -> 96.6; a 4 KiB window takes the same 26.7.  At most two:
    // 16 warps each, 64 registers instead of 40 and no spills, 256 windows
    // 127.7 -> 120.4.  More: three CTAs per SM (4096 windows 1.31 ms, two 1.72).
    const uint32_t sms = static_cast<uint32_t>(num_sms);
    if (a.num_windows <= sms) return launch_lane_parse<kRef, 32, 1>(a, num_sms, ctas_per_sm, st);
    if (a.num_windows <= 2u * sms) return launch_lane_parse<kRef, 16, 2>(a, num_sms, ctas_per_sm, st);
    return launch_lane_parse<kRef, 16, 3>(a, num_sms, ctas_per_sm, st);
}
}  // namespace

cudaError_t launch_zstd_parse(const Zstd2Launch &l, cudaStream_t st) {
    if (l.num_windows == 0) return cudaSuccess;
    Zstd2Args a{};
    a.src = l.src;
    a.cand = l.cand;
    a.n = l.n;
    a.window = l.window;
    a.num_windows = l.num_windows;
    a.lazy = l.search_depth > 1 ? 1u : 0u;
    a.max_seqs = l.max_seqs;
    a.seg = reinterpret_cast<uint2 *>(l.seg);
    a.packed = reinterpret_cast<uint2 *>(l.packed);
    a.ref_seqs = l.ref_seqs;
    a.seq_counts = l.seq_counts;
    a.lit_counts = l.lit_counts;
    a.status = l.status;
    a.wins = l.wins;
    a.seg_stride = kSegStride;
    return l.ref_seqs ? launch_parse_ref<true>(a, l.seg_width, l.num_sms, l.ctas_per_sm, st)
                      : launch_parse_ref<false>(a, l.seg_width, l.num_sms, l.ctas_per_sm, st);
}

}  // namespace gcz
