// gxy_device.cuh -- device data layout and the x-drop extenders.
//
// Sequences live in HBM in the reference's PackedSeq bit layout
// (src/sequences.rs:53-66) behind a 64-position leading pad, read as
// little-endian words: a u64 of `codes` holds 32 positions (2 bits each,
// position 32*i+k at bits 2k), a u32 of `valid`/`mask` holds 32 positions.
// Global position gp = kPad + local position, so a 32-position load at any
// gp >= 0 is in bounds; the tail carries kTailPad positions of zeros.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gxy {

constexpr uint32_t kPad = 64;         // leading pad (positions)
constexpr uint32_t kTailPad = 1536;   // trailing pad (positions); covers one warp stage
constexpr int kMaxWeight = 15;        // 4^15 buckets; starts[] is u32 x (2^30 + 1)
constexpr uint32_t kFull = 0xffffffffu;

// Process-wide count of kernels this library launched (gxy_kernel_launches).
void count_launch(uint64_t n = 1);

// One sequence segment as the kernels see it.  `base` is the global position
// of local position 0 (a chunk view of a target starts at kPad + chunk_lo);
// `key_base` places the segment on a private axis of the candidate sort key
// so that units never share a (target, query) coordinate pair.
struct SeqView {
    const uint64_t* codes;
    const uint32_t* valid;
    const uint32_t* mask;
    uint64_t base;
    uint32_t len;
    uint32_t key_base;
    // Optional window records (a table's target): record i - rec_first holds the
    // codes of the 32-position words i - 1 .. i + 2 in 32 bytes, so that the
    // surroundings of a position in word i (32 positions before it to 32 after a
    // seed of up to 32) take one sector.  The last of its 128 positions is never
    // among them: its two bits are set when any of the 128 is invalid, else clear.
    const uint32_t* rec = nullptr;
    uint64_t rec_first = 0;
};

// Codes and valid bits of the 32 positions from global position gp.
__device__ __forceinline__ void load_window32(const SeqView& S, uint64_t gp, uint64_t& codes, uint32_t& valid) {
    const uint64_t i = gp >> 5;
    const uint32_t s = (uint32_t)(gp & 31);
    const uint64_t lo = __ldg(S.codes + i), hi = __ldg(S.codes + i + 1);
    codes = s ? ((lo >> (2 * s)) | (hi << (64 - 2 * s))) : lo;
    valid = __funnelshift_r(__ldg(S.valid + i), __ldg(S.valid + i + 1), s);
}

// One reference search() call: a (target segment, query segment) pair with
// the target's position table (src/seed_search.rs:45-51).
struct UnitDev {
    uint32_t tseg;
    uint32_t qseg;
    const uint32_t* starts;
    const uint32_t* positions;
    const uint32_t* occ;  // bucket occupancy bitmap (bit w & 31 of occ[w >> 5])
    const uint16_t* nbr;  // neighbour masks, or null (see launch_neighbours)
    const uint2* packed;  // bounds of eight buckets each (see pack_buckets), with nbr
    uint32_t nwin;        // query windows 0, step, ... <= len - L
    uint32_t tile_base;   // first screen tile of this unit
    uint32_t primary_lo;  // driver primary-region filter, src/driver.rs:250-256
    uint32_t primary_hi;  // (lo == hi disables it)
};

// A hit that survived the screen: it either reaches hspthresh within the
// column cap (its extension result is exact and stored), or it is still
// extending at the cap (kCandLong) and is re-extended in full by the walk.
struct Cand {
    uint32_t unit;
    uint32_t t;
    uint32_t q;
    uint32_t flags;
    uint32_t lext;
    uint32_t rext;
    int32_t score;
    uint32_t pad_;
};
constexpr uint32_t kCandLong = 1u;

// Output record, layout-identical to gxy_hsp / the reference's Hsp.
struct Hsp {
    uint32_t t_start;
    uint32_t q_start;
    uint32_t length;
    int32_t score;
};

// Scoring parameters the extenders read (src/scoring.rs:32-40, src/hsp.rs:46-49).
struct Score {
    int32_t sub[16];
    int32_t ambig;
    int32_t xdrop;
    int32_t hspthresh;
};

// The hits of a tile's group: bucket sizes summed by 16-bit halves, which 32 bits
// hold for up to 65,536 buckets of any size (32 windows over one repeat of 140 M
// positions have more than 2^32 hits).  The halves can be reduced across a warp
// before they are joined.
struct HitSum {
    uint32_t lo = 0, hi = 0;
    __host__ __device__ __forceinline__ void add(uint32_t bucket) {
        lo += bucket & 0xffffu;
        hi += bucket >> 16;
    }
    __host__ __device__ __forceinline__ uint64_t total() const { return ((uint64_t)hi << 16) + lo; }
};
// The windows that start in positions [p0, p0 + span), counted from p0: first, first +
// stride .. below stop.  Windows start at multiples of step up to `last`, which is
// not below p0.  (A stride of a whole span ends the loop; step itself could wrap.)
struct SpanWindows {
    uint32_t first, stop, stride;
    __host__ __device__ __forceinline__ SpanWindows(uint64_t p0, uint64_t last, uint32_t step, uint32_t span) {
        const uint64_t f = step == 1 ? 0 : (p0 + step - 1) / step * step - p0, n = last - p0 + 1;
        first = f < span ? (uint32_t)f : span;
        stop = n < span ? (uint32_t)n : span;
        stride = step < span ? step : span;
    }
};
// Whether slots [base, base + hits) lie in a buffer of cap slots.
__host__ __device__ __forceinline__ bool hits_fit(uint64_t base, uint64_t hits, uint64_t cap) {
    return hits <= cap && base <= cap - hits;
}

// The blocks of a launch that take part when n items came, `per` a block: counts are
// only known on the device, and inputs of repeats have hundreds of times the hits
// that the sizes let one expect.  Grids are launched whole; the blocks past
// these return at once.  The 8 spread what is little over SMs.
__device__ __forceinline__ uint32_t live_blocks(uint64_t n, uint32_t per) {
    return (uint32_t)min((uint64_t)gridDim.x, n / per + 8);
}

__device__ __forceinline__ uint64_t load_codes32(const uint64_t* __restrict__ codes, uint64_t gp) {
    const uint64_t i = gp >> 5;
    const uint32_t s = (uint32_t)(gp & 31) * 2;
    const uint64_t lo = __ldg(codes + i);
    const uint64_t hi = __ldg(codes + i + 1);
    return s ? ((lo >> s) | (hi << (64 - s))) : lo;
}

__device__ __forceinline__ uint32_t load_bits32(const uint32_t* __restrict__ bits, uint64_t gp) {
    const uint64_t i = gp >> 5;
    const uint32_t s = (uint32_t)(gp & 31);
    return __funnelshift_r(__ldg(bits + i), __ldg(bits + i + 1), s);
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Each set bit of x becomes a set 2-bit pair (bit k -> bits 2k, 2k+1).
__device__ __forceinline__ uint64_t spread_bits_to_pairs(uint32_t x) {
    uint64_t v = x;
    v = (v | (v << 16)) & 0x0000FFFF0000FFFFull;
    v = (v | (v << 8)) & 0x00FF00FF00FF00FFull;
    v = (v | (v << 4)) & 0x0F0F0F0F0F0F0F0Full;
    v = (v | (v << 2)) & 0x3333333333333333ull;
    v = (v | (v << 1)) & 0x5555555555555555ull;
    return v * 3;   // each set bit -> a set 2-bit pair
}

// Reverses the order of the 32 two-bit codes of a word (a left-side chunk
// read upwards becomes column 0 = the position next to the seed).
__device__ __forceinline__ uint64_t rev_pairs64(uint64_t c) {
    c = __brevll(c);
    return ((c >> 1) & 0x5555555555555555ull) | ((c & 0x5555555555555555ull) << 1);
}

// Column score (src/hsp.rs:198-211): ambig when either base is invalid.
__device__ __forceinline__ int32_t col_score(uint64_t tc, uint64_t qc, uint32_t vv, int sh,
                                             const int32_t* lut, int32_t ambig) {
    const uint32_t idx = (((uint32_t)(tc >> (2 * sh)) & 3u) << 2) | ((uint32_t)(qc >> (2 * sh)) & 3u);
    return ((vv >> sh) & 1u) ? lut[idx] : ambig;
}

// One side of extend_one_side (src/hsp.rs:160-195), one lane, 32 columns per
// pair of loads.  t0/q0 are the local positions of the first column; forward
// walks up, backward walks down.  Returns true when the side ended (x-drop
// break or sequence bound) within `cap` columns, false when it is still
// running after `cap` columns (the caller then defers the hit to the walk).
// The arithmetic is plain i32: the host admits a search only when no partial
// sum can leave i32, so the reference's saturating adds never saturate.
template <bool kForward>
__device__ __forceinline__ bool side_lane(const SeqView& T, const SeqView& Q, uint32_t t0,
                                          uint32_t q0, uint32_t maxext, uint32_t cap,
                                          int32_t xdrop, const int32_t* lut, int32_t ambig,
                                          int32_t& best_out, uint32_t& bext_out) {
    int32_t run = 0, best = 0;
    uint32_t bext = 0, ext = 0;
    while (ext < maxext) {
        const uint64_t tg = kForward ? T.base + t0 + ext : T.base + t0 - ext - 31;
        const uint64_t qg = kForward ? Q.base + q0 + ext : Q.base + q0 - ext - 31;
        const uint64_t tc = load_codes32(T.codes, tg);
        const uint64_t qc = load_codes32(Q.codes, qg);
        const uint32_t vv = load_bits32(T.valid, tg) & load_bits32(Q.valid, qg);
        const uint32_t n = min(32u, maxext - ext);
#pragma unroll
        for (int i = 0; i < 32; i++) {
            if ((uint32_t)i >= n) break;
            const int sh = kForward ? i : 31 - i;
            run += col_score(tc, qc, vv, sh, lut, ambig);
            if (run > best) {
                best = run;
                bext = ext + i + 1;
            } else if (best - run > xdrop) {
                best_out = best;
                bext_out = bext;
                return true;
            }
        }
        ext += n;
        if (ext >= cap && ext < maxext) {
            best_out = best;
            bext_out = bext;
            return false;
        }
    }
    best_out = best;
    bext_out = bext;
    return true;
}

struct LaneExt {
    int32_t score;
    uint32_t lext;
    uint32_t rext;
    bool done;   // both sides ended within the cap: the result is exact
};

// extend_hit_scalar (src/hsp.rs:98-148) for one lane with a column cap per
// side.  Requires t + L <= T.len and q + L <= Q.len (the caller checks).
__device__ __forceinline__ LaneExt extend_lane(const SeqView& T, const SeqView& Q, uint32_t t,
                                               uint32_t q, uint32_t L, uint32_t cap,
                                               int32_t xdrop, const int32_t* lut, int32_t ambig) {
    LaneExt r;
    // Seed footprint: all L columns, care and don't-care (src/hsp.rs:119-123).
    const uint64_t tc = load_codes32(T.codes, T.base + t);
    const uint64_t qc = load_codes32(Q.codes, Q.base + q);
    const uint32_t vv = load_bits32(T.valid, T.base + t) & load_bits32(Q.valid, Q.base + q);
    int32_t seed = 0;
#pragma unroll
    for (int k = 0; k < 32; k++) {
        if ((uint32_t)k >= L) break;
        seed += col_score(tc, qc, vv, k, lut, ambig);
    }
    int32_t rb, lb = 0;
    uint32_t re, le = 0;
    const uint32_t rmax = min(T.len - t - L, Q.len - q - L);
    r.done = side_lane<true>(T, Q, t + L, q + L, rmax, cap, xdrop, lut, ambig, rb, re);
    if (r.done) {
        const uint32_t lmax = min(t, q);
        if (lmax) r.done = side_lane<false>(T, Q, t - 1, q - 1, lmax, cap, xdrop, lut, ambig, lb, le);
    }
    r.score = seed + lb + rb;
    r.lext = le;
    r.rext = re;
    return r;
}

// ---------------------------------------------------------------------------
// Warp-cooperative x-drop: one warp per hit, half a warp per side, 128 columns
// per step (eight per lane), the x-drop cut found with shuffle scans.
// Column k of a step breaks the reference's
// loop iff run_k <= PM_{k-1} and PM_{k-1} - run_k > xdrop, where
// PM_{k-1} = max(best, run_0..run_{k-1}); the best extent is the first column
// whose running score equals the step's maximum (the reference updates only
// on a strict increase).  Sequence bytes are staged through shared memory in
// 16-byte vector loads: kStageSpan positions per side and refill.
//
// What bounds it is latency -- the step's chain of shuffles, the refills, and in a
// short kernel the fetch of its own code: one side after the other, 64 columns a
// step in two unrolled copies, took 13,000 cycles for sides of a few hundred
// columns.  The walk of 10 Mbp (its launch of one strand) went from 81 to 65 us,
// that of 1 Mbp with entropy gates from 95 to 79 us.
// ---------------------------------------------------------------------------
constexpr uint32_t kStageCols = 512;                       // columns a refill is good for
constexpr uint32_t kStageSpan = 768;                       // positions per refill (+ 127 to the boundary, + a funnel read)
struct WarpStage {   // [0]: the right side, [1]: the left one
    uint64_t tcodes[2][kStageSpan / 32];
    uint64_t qcodes[2][kStageSpan / 32];
    uint32_t tvalid[2][kStageSpan / 32];
    uint32_t qvalid[2][kStageSpan / 32];
};

// Copies positions [a, a + kStageSpan) (a a multiple of 128) of one sequence
// into a side's stage with 16-byte loads by its 16 lanes: codes 192 bytes, valid 96.
__device__ __forceinline__ void stage_fill(const uint64_t* codes, const uint32_t* valid, uint64_t a,
                                           uint64_t* scodes, uint32_t* svalid, int hl) {
    const uint4* c4 = reinterpret_cast<const uint4*>(codes + (a >> 5));
    const uint4* v4 = reinterpret_cast<const uint4*>(valid + (a >> 5));
    constexpr int kC4 = kStageSpan / 32 * 8 / 16;   // 12
    constexpr int kV4 = kStageSpan / 32 * 4 / 16;   // 6
    if (hl < kC4) reinterpret_cast<uint4*>(scodes)[hl] = __ldg(c4 + hl);
    if (hl < kV4) reinterpret_cast<uint4*>(svalid)[hl] = __ldg(v4 + hl);
}

__device__ __forceinline__ uint64_t stage_codes32(const uint64_t* s, uint32_t off) {
    const uint32_t i = off >> 5, sh = (off & 31) * 2;
    const uint64_t lo = s[i], hi = s[i + 1];
    return sh ? ((lo >> sh) | (hi << (64 - sh))) : lo;
}
__device__ __forceinline__ uint32_t stage_bits32(const uint32_t* s, uint32_t off) {
    return __funnelshift_r(s[off >> 5], s[(off >> 5) + 1], off & 31);
}

// The 8 columns in the low 16 bits in reverse order.
__device__ __forceinline__ uint32_t rev_pairs16(uint32_t x) {
    x = __brev(x) >> 16;
    return ((x >> 1) & 0x5555u) | ((x & 0x5555u) << 1);
}

// extend_hit_scalar (src/hsp.rs:98-148) with one warp; every lane returns the
// same result.
__device__ __forceinline__ LaneExt extend_warp(const SeqView& T, const SeqView& Q, uint32_t t,
                                               uint32_t q, uint32_t L, int32_t xdrop,
                                               const int32_t* lut, int32_t ambig, WarpStage* st) {
    const int lane = threadIdx.x & 31, hl = lane & 15;
    const bool left = lane >= 16;
    const uint32_t half = left ? 16u : 0u;   // the side's first lane
    const uint64_t stc = load_codes32(T.codes, T.base + t);
    const uint64_t sqc = load_codes32(Q.codes, Q.base + q);
    const uint32_t svv = load_bits32(T.valid, T.base + t) & load_bits32(Q.valid, Q.base + q);
    // The side's column 0 and columns; it runs up or (left) down from there.
    const uint64_t t0 = left ? T.base + t - 1 : T.base + t + L, q0 = left ? Q.base + q - 1 : Q.base + q + L;
    const uint32_t maxext = left ? min(t, q) : min(T.len - t - L, Q.len - q - L);
    uint64_t* const tcodes = st->tcodes[left];
    uint64_t* const qcodes = st->qcodes[left];
    uint32_t* const tvalid = st->tvalid[left];
    uint32_t* const qvalid = st->qvalid[left];
    int32_t run = 0, best = 0;
    uint32_t bext = 0, ext = 0;
    uint64_t ta = 0, qa = 0;   // staged windows' first global positions
    uint32_t staged = 0;       // columns left in the current stage
    bool live = maxext > 0;
    while (__any_sync(kFull, live)) {
        const uint64_t tg = left ? t0 - ext : t0 + ext, qg = left ? q0 - ext : q0 + ext;
        const bool refill = live && staged < 128;
        if (__any_sync(kFull, refill)) {
            __syncwarp();
            if (refill) {
                ta = (left ? (tg >= kStageCols ? tg - (kStageCols - 1) : 0) : tg) & ~127ull;
                qa = (left ? (qg >= kStageCols ? qg - (kStageCols - 1) : 0) : qg) & ~127ull;
                stage_fill(T.codes, T.valid, ta, tcodes, tvalid, hl);
                stage_fill(Q.codes, Q.valid, qa, qcodes, qvalid, hl);
                staged = kStageCols;
            }
            __syncwarp();
        }
        // Eight columns by one funnel read from the lowest position (a lane whose
        // columns do not exist may lie before the stage).
        const uint32_t c0 = 8u * (uint32_t)hl;
        const int32_t lo = left ? -(int32_t)(c0 + 7) : (int32_t)c0;
        const uint32_t to = live ? (uint32_t)max(0, (int32_t)(tg - ta) + lo) : 0u;
        const uint32_t qo = live ? (uint32_t)max(0, (int32_t)(qg - qa) + lo) : 0u;
        uint32_t tc = (uint32_t)stage_codes32(tcodes, to) & 0xffffu;
        uint32_t qc = (uint32_t)stage_codes32(qcodes, qo) & 0xffffu;
        uint32_t vv = stage_bits32(tvalid, to) & stage_bits32(qvalid, qo) & 0xffu;
        if (left) {
            tc = rev_pairs16(tc);
            qc = rev_pairs16(qc);
            vv = __brev(vv) >> 24;
        }
        const uint32_t n = live ? min(128u, maxext - ext) : 0u, mine = c0 < n ? min(8u, n - c0) : 0u;
        // The lane's running sums and their maximum, then both before the lane.
        int32_t p[8], sum = 0, top = INT32_MIN;
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            const int32_t x = (vv >> k) & 1u ? lut[((tc >> (2 * k)) & 3u) << 2 | ((qc >> (2 * k)) & 3u)] : ambig;
            if (k < mine) {
                sum += x;
                top = max(top, sum);
            }
            p[k] = sum;
        }
        int32_t S = sum, M = top;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int32_t ys = __shfl_up_sync(kFull, S, o, 16), ym = __shfl_up_sync(kFull, M, o, 16);
            if (hl >= o) {
                M = M == INT32_MIN ? ym : max(ym, ys + M);
                S += ys;
            }
        }
        int32_t pm = __shfl_up_sync(kFull, M, 1, 16);
        pm = hl == 0 || pm == INT32_MIN ? best : max(best, run + pm);   // before the lane's first column
        const int32_t r = run + S - sum;
        // Its columns up to the first break, their maximum and where it is first.
        uint32_t upto = mine, at = 0;
        int32_t c = INT32_MIN;
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            const int32_t rk = r + p[k];
            if (k < upto) {
                if (rk <= pm && pm - rk > xdrop) {
                    upto = k;
                } else {
                    pm = max(pm, rk);
                    if (rk > c) {
                        c = rk;
                        at = k;
                    }
                }
            }
        }
        const uint32_t bm = (__ballot_sync(kFull, upto < mine) >> half) & 0xffffu;
        if (bm && hl > __ffs(bm) - 1) c = INT32_MIN;
        const int32_t high0 = __reduce_max_sync(kFull, left ? INT32_MIN : c);
        const int32_t high1 = __reduce_max_sync(kFull, left ? c : INT32_MIN);
        const int32_t high = left ? high1 : high0;
        const uint32_t eq = (__ballot_sync(kFull, c == high) >> half) & 0xffffu;   // (never empty)
        const int el = __ffs(eq) - 1;
        const uint32_t at_el = __shfl_sync(kFull, at, el, 16);
        if (high > best) {
            bext = ext + 8u * (uint32_t)el + at_el + 1;
            best = high;
        }
        run = __shfl_sync(kFull, run + S, 15, 16);
        ext += n;
        staged -= live ? 128u : 0u;
        live = live && bm == 0 && ext < maxext;
    }
    int32_t s = ((uint32_t)lane < L) ? col_score(stc, sqc, svv, lane, lut, ambig) : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    LaneExt r;
    r.score = s + __shfl_sync(kFull, best, 0) + __shfl_sync(kFull, best, 16);
    r.rext = __shfl_sync(kFull, bext, 0);
    r.lext = __shfl_sync(kFull, bext, 16);
    r.done = true;
    return r;
}

}  // namespace gxy
