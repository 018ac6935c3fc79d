// gxy_filter.cu -- the upper-bound x-drop filter between seed-hit
// enumeration and the exact screen, for sm_100a.
//
// search() (src/seed_search.rs:92-116) extends every admitted seed hit, but
// only a hit whose HSP reaches hspthresh changes the output: the diagonal
// filter records cover for passing HSPs only (src/seed_search.rs:113).  So a
// hit that provably cannot reach hspthresh can be dropped before the exact
// screen looks at it.  k_filter_hits proves it cheaply, one lane per raw hit
// of the hit array that k_enumerate wrote:
//
//  - it runs extend_one_side (src/hsp.rs:160-195) on both sides with every
//    column score replaced by an upper bound -- the largest score of the
//    column's class x = t_code ^ q_code (match, transition, and the two
//    transversion classes); invalid columns take a class whose bound is
//    >= the ambiguous score.  With scores raised, every running sum and best
//    is raised and the drop best - run can only shrink, so a bounded side
//    breaks no earlier and its best is an upper bound of the exact best.  The
//    break is tested every 32 columns only, which again can only raise the
//    best;
//  - four columns are scored per step through a 256-entry table of
//    (sum, maximum prefix) indexed by the four columns' classes: one byte
//    permute, one shared-memory load and three integer operations per four
//    columns, against five operations per column in the exact screen;
//  - a hit survives when the bounded seed footprint + both sides' bests reach
//    hspthresh, or when a side is still running after f_cap columns;
//  - nearly every hit is decided by the first 32 columns of both sides, so
//    these are scored for 32 hits at a time from one 32-byte record of the
//    target (SeqView::rec) and the query's words around the window; the few
//    hits that run on, or whose columns hold an invalid base or a sequence end,
//    go through a queue of the warp's own, 32 at a time.
//
// Survivors (about 1 % of the raw hits on chromosome-scale inputs) go to a
// second hit array, where the exact screen (k_screen) takes them.  The
// dropped hits are exactly hits whose exact score is below hspthresh, so the
// pipeline's output does not change.
#include "gxy_kernels.cuh"

#include <algorithm>

namespace gxy {

namespace {

constexpr int kLutBytes = 256 * 32 * 8;         // (sum, max prefix) x 32 lane copies; one table a direction
constexpr int kFilterWarps = 32;                // warps per block, one block per SM (the tables fill it)
constexpr uint32_t kQueue = 64;                 // hits a warp's queue holds, eight words each
constexpr int kFilterSmem = 2 * kLutBytes + kFilterWarps * kQueue * 32;

// Columns whose bit in `keep` is clear take the classes of `pat`.
__device__ __forceinline__ uint64_t fold_cols(uint64_t x, uint32_t keep, uint64_t pat) {
    const uint64_t m = spread_bits_to_pairs(keep);
    return (x & m) | (pat & ~m);
}

struct FSide {
    int32_t run;
    int32_t best;
};

// Four columns (byte g of w, column k at bits 2k..2k+1): the table entry of
// the byte gives their bounded sum and the maximum of their four prefix sums.
// The entry of byte b for lane l sits at b * 256 + l * 8, so the 16 lanes of
// each half-warp read distinct banks; one byte permute forms that address.
__device__ __forceinline__ void f_group(FSide& S, uint32_t w, uint32_t lane8, int g, const unsigned char* lut) {
    const uint32_t ad = __byte_perm(w, lane8, 0x5504u | ((uint32_t)g << 4));
    const int2 e = *reinterpret_cast<const int2*>(lut + ad);
    S.best = max(S.best, S.run + e.y);
    S.run += e.x;
}

// 32 columns of each side, interleaved so that the two serial chains issue
// side by side.  R runs up from column 0 of (r0, r1); L runs down from column
// 31 of (l0, l1), through the table of prefix sums taken from a byte's high end.
__device__ __forceinline__ void f_scan2(FSide& R, uint32_t r0, uint32_t r1, FSide& Lf, uint32_t l0, uint32_t l1,
                                        uint32_t lane8, const unsigned char* lut) {
#pragma unroll
    for (int g = 0; g < 4; g++) {
        f_group(R, r0, lane8, g, lut);
        f_group(Lf, l1, lane8, 3 - g, lut + kLutBytes);
    }
#pragma unroll
    for (int g = 0; g < 4; g++) {
        f_group(R, r1, lane8, g, lut);
        f_group(Lf, l0, lane8, 3 - g, lut + kLutBytes);
    }
}

__device__ __forceinline__ void lut_fill(unsigned char* lut, const int32_t* fub) {
    // Sixteen entries a warp, one a lane, then each to all 32 copies.  (With every
    // lane forming the entry it stored, this took 12 us of a block.)
    static_assert(kFilterWarps * 16 == 512, "two tables of 256 entries");
    const uint32_t lane = threadIdx.x & 31, e0 = (threadIdx.x >> 5) * 16;
    const uint32_t b = (e0 + (lane & 15)) & 255u;
    const bool down = e0 >> 8;
    int32_t p = 0, mp = INT32_MIN;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        p += fub[(b >> (2 * (down ? 3 - c : c))) & 3u];
        mp = max(mp, p);
    }
#pragma unroll
    for (uint32_t k = 0; k < 16; k++)
        reinterpret_cast<int2*>(lut)[(e0 + k) * 32 + lane] = make_int2(__shfl_sync(kFull, p, k), __shfl_sync(kFull, mp, k));
}

// The seed footprint's bound: all L columns from column 0 of x (src/hsp.rs:119-123).
__device__ __forceinline__ int32_t seed_sum(uint64_t x, uint32_t L, int32_t ub0, uint32_t lane8, const unsigned char* lut) {
    int32_t sd = 0;
#pragma unroll
    for (int g = 0; g < 8; g++) {
        if (4u * g >= L) break;
        const uint32_t w = g < 4 ? (uint32_t)x : (uint32_t)(x >> 32);
        const uint32_t r = min(4u, L - 4u * g);
        uint32_t byte = (w >> (8 * (g & 3))) & 0xFFu;
        if (r < 4) byte &= (1u << (2 * r)) - 1u;   // columns past L: class 0, taken off below
        const int2 e = *reinterpret_cast<const int2*>(lut + (byte << 8) + lane8);
        sd += e.x - (int32_t)(4u - r) * ub0;
    }
    return sd;
}

// 256 bits from a 32-byte boundary.
__device__ __forceinline__ void load_rec(const uint32_t* p, uint32_t (&w)[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "l"(p));
}

// The 96 positions from position s (0 .. 31) of 128: 16 a word.
__device__ __forceinline__ void align96(const uint32_t (&w)[8], uint32_t s, uint32_t (&o)[6]) {
    const bool up = s & 16;
    const uint32_t sh = 2 * (s & 15);
    uint32_t v[7];
#pragma unroll
    for (int i = 0; i < 7; i++) v[i] = up ? w[i + 1] : w[i];
#pragma unroll
    for (int i = 0; i < 6; i++) o[i] = __funnelshift_r(v[i], v[i + 1], sh);
}

// The bounded x-drop over the raw-hit array written by k_enumerate.  Warps
// claim hits in chunks from a cursor and take 32 at a time, one a lane: both
// sides' first 32 columns, from which nearly every hit is dropped.  The rest is
// queued and taken 32 at a time, a further 32 columns a step.  Survivors go to
// a.hits.
//
// What bounds it: the integer pipe and the L1's one tag a cycle.  A form with a
// persistent hit a lane, a window of its own for each side (two 16-byte records
// and four query words) and a reversal of the left one took 601 instructions
// and 6.6 sectors a hit, 0.70 ms for 26.1 M hits (10 Mbp x 10 Mbp); this one
// 404 and 2.2, 0.48 ms.
__global__ __launch_bounds__(kFilterWarps * 32, 1) void k_filter_hits(const __grid_constant__ ScreenArgs a,
                                                                       const __grid_constant__ FilterIO io) {
    extern __shared__ __align__(16) unsigned char smem[];
    // Past the buffer's end the pass did not write (those tiles went to the
    // next pass).
    const uint32_t n_hits = (uint32_t)min(*io.raw_count, (unsigned long long)io.raw_cap);
    // A hit a lane at most: small launches leave the rest of the GPU alone (each
    // block fills its two 64 KB tables, each warp claims from the cursor).
    const uint32_t n_blocks = live_blocks(n_hits, kFilterWarps * 32);
    if (blockIdx.x >= n_blocks) return;
    unsigned char* lut = smem;
    lut_fill(lut, a.fub);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    // Word k of queued hit s at k * kQueue + s: t, q, unit, the right run and best,
    // the left ones, and the columns scanned << 2 | the sides that run (whose columns
    // scanned are the same number).
    uint32_t* const queue = reinterpret_cast<uint32_t*>(smem + 2 * kLutBytes) + (threadIdx.x >> 5) * (kQueue * 8);
    const uint32_t lane8 = (uint32_t)lane * 8u, lt = lanemask_lt();
    const uint32_t L = a.pat.len;
    const int32_t X = a.sc.xdrop, thresh = a.sc.hspthresh;
    const int32_t need = thresh - a.f_seed_max;
    const int32_t ub0 = a.fub[0];
    const uint32_t n_warps = n_blocks * kFilterWarps;
    const uint32_t chunk = a.f_claim ? a.f_claim : max(32u, min(512u, n_hits / max(1u, n_warps * 8u)) & ~31u);
    uint32_t wcur = 0, wend = 0, qn = 0;
    bool exhausted = false;
    unsigned long long n_cols = 0;
    uint32_t cur_unit = kNoUnit;
    // The current unit's target records and query.
    const uint32_t* rec = nullptr;
    uint64_t t_base = 0, q_base = 0;   // t_base counts from the first record
    uint32_t t_len = 0, q_len = 0;
    const uint64_t* qc = nullptr;
    const uint32_t* qv = nullptr;
    auto take_unit = [&](uint32_t u) {
        cur_unit = u;
        const UnitDev U = a.units[u];
        const SeqView& T = a.tsegs[U.tseg];
        const SeqView& Q = a.qsegs[U.qseg];
        rec = T.rec;
        t_base = T.base - 32 * T.rec_first;
        t_len = T.len;
        qc = Q.codes;
        qv = Q.valid;
        q_base = Q.base;
        q_len = Q.len;
    };
    auto emit = [&](bool surv, uint32_t t, uint32_t q, uint32_t u) {
        const uint32_t sm = __ballot_sync(kFull, surv);
        if (!sm) return;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.hit_count, (unsigned long long)__popc(sm));
        base = __shfl_sync(kFull, base, 0);
        const unsigned long long slot = base + __popc(sm & lt);
        if (surv && slot < a.hit_cap) {
            a.hits[slot] = t;
            a.hits[a.hit_cap + slot] = q;
            if (a.n_units > 1) a.hits[2 * a.hit_cap + slot] = u;
        }
    };
    auto enqueue = [&](bool on, uint32_t t, uint32_t q, uint32_t u, const FSide& R, const FSide& Lf, uint32_t state) {
        const uint32_t m = __ballot_sync(kFull, on);
        if (on) {
            uint32_t* e = queue + qn + __popc(m & lt);
            e[0] = t;
            e[kQueue] = q;
            e[2 * kQueue] = u;
            e[3 * kQueue] = (uint32_t)R.run;
            e[4 * kQueue] = (uint32_t)R.best;
            e[5 * kQueue] = (uint32_t)Lf.run;
            e[6 * kQueue] = (uint32_t)Lf.best;
            e[7 * kQueue] = state;
        }
        qn += __popc(m);
        __syncwarp();
    };
    for (;;) {
        if (wcur == wend && !exhausted) {
            uint32_t nb = 0;
            if (lane == 0) nb = atomicAdd(io.cursor, chunk);
            nb = __shfl_sync(kFull, nb, 0);
            wcur = min(nb, n_hits);
            wend = min(nb + chunk, n_hits);
            exhausted = nb + chunk >= n_hits;
        }
        if (qn < 32 && wcur < wend) {
            // ---- 32 new hits: both sides' first 32 columns.
            const uint32_t idx = wcur + lane;
            wcur = min(wcur + 32, wend);
            uint32_t t = 0, q = 0, u = kNoUnit;
            if (idx < wend) {
                t = __ldg(io.raw + idx);
                q = __ldg(io.raw + io.raw_cap + idx);
                u = q == kNoHit ? kNoUnit : (a.n_units > 1 ? __ldg(io.raw + 2 * io.raw_cap + idx) : 0u);
            }
            const bool on = u != kNoUnit;   // else an unused slot of a failed reservation
            if (on && u != cur_unit) take_unit(u);
            const uint32_t rrem = on ? min(t_len - t - L, q_len - q - L) : 0u, lrem = on ? min(t, q) : 0u;
            bool plain = on && rec && rrem >= 32 && lrem >= 32;
            uint32_t x[6] = {0, 0, 0, 0, 0, 0};
            if (plain) {
                const uint64_t gt = t_base + t, gq = q_base + q;
                uint32_t w[8], o[6];
                load_rec(rec + (gt >> 5) * 8, w);
                const uint64_t* c = qc + (gq >> 5) - 1;
                const uint32_t* v = qv + (gq >> 5) - 1;
                uint32_t y[8];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint64_t z = __ldg(c + k);
                    y[2 * k] = (uint32_t)z;
                    y[2 * k + 1] = (uint32_t)(z >> 32);
                }
                const uint32_t ok = __ldg(v) & __ldg(v + 1) & __ldg(v + 2) & __ldg(v + 3);
                plain = ok == kFull && !(w[7] >> 31);
                align96(w, (uint32_t)gt & 31, x);
                align96(y, (uint32_t)gq & 31, o);
#pragma unroll
                for (int k = 0; k < 6; k++) x[k] ^= o[k];
            }
            // Classes: the 32 columns left of the seed in x[0..1], 32 from its start
            // in x[2..3], the next 32 in x[4..5]; the right side starts L further.
            const uint32_t s = 2 * (L & 15);
            const uint32_t a0 = L >= 32 ? x[4] : (L >= 16 ? x[3] : x[2]), a1 = L >= 32 ? x[5] : (L >= 16 ? x[4] : x[3]),
                           a2 = L >= 16 ? x[5] : x[4];
            FSide R{0, 0}, Lf{0, 0};
            f_scan2(R, __funnelshift_r(a0, a1, s), __funnelshift_r(a1, a2, s), Lf, x[0], x[1], lane8, lut);
            const bool ra = plain && rrem > 32 && R.best - R.run <= X, la = plain && lrem > 32 && Lf.best - Lf.run <= X;
            bool surv = plain && !ra && !la && R.best + Lf.best >= need;
            if (__any_sync(kFull, surv)) {
                if (surv)
                    surv = seed_sum(((uint64_t)x[3] << 32) | x[2], L, ub0, lane8, lut) + R.best + Lf.best >= thresh;
                emit(surv, t, q, u);
            }
            if (plain) n_cols += 64;
            if (on && !plain) R = Lf = FSide{0, 0};
            const bool more = ra || la || (on && !plain);
            if (__any_sync(kFull, more))
                enqueue(more, t, q, u, R, Lf,
                        plain ? (32u << 2) | (ra ? 1u : 0u) | (la ? 2u : 0u) : (rrem ? 1u : 0u) | (lrem ? 2u : 0u));
            continue;
        }
        if (qn == 0) {
            if (exhausted) break;
            continue;
        }
        // ---- up to 32 queued hits: 32 more columns of each side that runs.
        const uint32_t take = min(qn, 32u);
        qn -= take;
        const bool on = (uint32_t)lane < take;
        uint32_t t = 0, q = 0, u = kNoUnit, state = 0;
        FSide R{0, 0}, Lf{0, 0};
        if (on) {
            const uint32_t* e = queue + qn + lane;
            t = e[0];
            q = e[kQueue];
            u = e[2 * kQueue];
            R.run = (int32_t)e[3 * kQueue];
            R.best = (int32_t)e[4 * kQueue];
            Lf.run = (int32_t)e[5 * kQueue];
            Lf.best = (int32_t)e[6 * kQueue];
            state = e[7 * kQueue];
            if (u != cur_unit) take_unit(u);
        }
        __syncwarp();
        const uint32_t ext = state >> 2;
        const uint32_t rrem = on ? min(t_len - t - L, q_len - q - L) - ext : 0u, lrem = on ? min(t, q) - ext : 0u;
        const uint32_t nr = (state & 1u) ? min(32u, rrem) : 0u, nl = (state & 2u) ? min(32u, lrem) : 0u;
        // The classes of the 32 columns from target position tp and query position
        // qp (tp may lie up to 32 before the view); n columns count, from the low
        // end or (top) the high one.
        auto classes = [&](int64_t tp, int64_t qp, uint32_t n, bool top) {
            const uint64_t gq = (uint64_t)((int64_t)q_base + qp);
            uint64_t tcod, qcod;
            uint32_t ok, w[8];
            qcod = load_codes32(qc, gq);
            ok = load_bits32(qv, gq);
            bool exact = true;   // the record tells that all is valid
            if (rec) {
                const uint64_t gt = (uint64_t)((int64_t)t_base + tp);
                load_rec(rec + (gt >> 5) * 8, w);
                const bool up = gt & 16;
                const uint32_t sh = 2 * ((uint32_t)gt & 15);
                const uint32_t v0 = up ? w[3] : w[2], v1 = up ? w[4] : w[3], v2 = up ? w[5] : w[4];
                tcod = ((uint64_t)__funnelshift_r(v1, v2, sh) << 32) | __funnelshift_r(v0, v1, sh);
                exact = !(w[7] >> 31);
            }
            if (!rec || !exact) {
                const SeqView& T = a.tsegs[a.units[u].tseg];
                uint32_t tv;
                load_window32(T, (uint64_t)((int64_t)T.base + tp), tcod, tv);
                ok &= tv;
            }
            uint64_t x = tcod ^ qcod;
            if (n < 32 || ok != kFull)
                x = fold_cols(fold_cols(x, ok, a.f_inv), n >= 32 ? kFull : (top ? kFull << (32 - n) : (1u << n) - 1u), a.f_end);
            return x;
        };
        uint64_t xr = 0, xl = 0;
        if (nr) xr = classes((int64_t)t + L + ext, (int64_t)q + L + ext, nr, false);
        if (nl) xl = classes((int64_t)t - ext - 32, (int64_t)q - ext - 32, nl, true);
        const FSide R0 = R, L0 = Lf;
        f_scan2(R, (uint32_t)xr, (uint32_t)(xr >> 32), Lf, (uint32_t)xl, (uint32_t)(xl >> 32), lane8, lut);
        n_cols += nr + nl;
        bool ra = false, la = false;
        if (nr) {
            ra = rrem > nr && R.best - R.run <= X;
        } else {
            R = R0;
        }
        if (nl) {
            la = lrem > nl && Lf.best - Lf.run <= X;
        } else {
            Lf = L0;
        }
        const bool capped = on && (ra || la) && ext + 32 >= a.f_cap;
        const bool done = on && (capped || (!ra && !la));
        bool surv = done && (capped || R.best + Lf.best >= need);
        if (__any_sync(kFull, surv && !capped)) {
            if (surv && !capped) {
                surv = seed_sum(classes(t, q, 32, false), L, ub0, lane8, lut) + R.best + Lf.best >= thresh;
            }
        }
        emit(surv, t, q, u);
        if (__any_sync(kFull, on && !done))
            enqueue(on && !done, t, q, u, R, Lf, (ext + 32) << 2 | (ra ? 1u : 0u) | (la ? 2u : 0u));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_cols += __shfl_xor_sync(kFull, n_cols, o);
    if (lane == 0 && n_cols) atomicAdd(&a.stats[3], n_cols);
}

__global__ void k_occupancy(const uint32_t* __restrict__ starts, uint64_t nw, uint32_t* __restrict__ occ,
                            uint2* __restrict__ packed) {
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    const uint64_t w0 = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t base = w0 * 32; base < nw; base += warps * 32) {
        const uint64_t w = base + lane;
        const uint32_t b = w < nw ? __ldg(starts + w) : 0u, c = w < nw ? __ldg(starts + w + 1) - b : 0u;
        const uint32_t m = __ballot_sync(kFull, c != 0);
        if (lane == 0) occ[base >> 5] = m;
        if (packed) {
            uint32_t y = c < 15 ? c << (4 * (lane & 7)) : 0xffffffffu;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) y |= __shfl_xor_sync(kFull, y, o);
            if ((lane & 7) == 0 && w < nw) packed[w >> 3] = make_uint2(b, y);
        }
    }
}

// One thread per 32 buckets: the occupancy words of the bucket's own and its
// neighbours' 32 (a transition flips the high bit of a care position: inside
// the word for the last two positions, in another word for the rest), as 16
// rows, transposed into 32 masks.
__global__ void k_neighbours(const uint32_t* __restrict__ occ, uint64_t n_words, uint32_t words_per_view, uint32_t weight,
                             uint16_t* __restrict__ nbr) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n_words; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t view = i & ~(uint64_t)(words_per_view - 1);   // 4^weight / 32 words, a power of two
        const uint32_t x = (uint32_t)(i - view);
        const uint32_t w0 = __ldg(occ + i);
        uint32_t r[16];
        r[0] = w0;
#pragma unroll
        for (uint32_t v = 1; v < 16; v++) {
            r[v] = 0;
            if (v <= weight) {
                const uint32_t bit = 2 * (weight - v) + 1;
                if (bit == 1) r[v] = ((w0 >> 2) & 0x33333333u) | ((w0 & 0x33333333u) << 2);
                else if (bit == 3) r[v] = ((w0 >> 8) & 0x00ff00ffu) | ((w0 & 0x00ff00ffu) << 8);
                else r[v] = __ldg(occ + view + (x ^ (1u << (bit - 5))));
            }
        }
        // Both 16 x 16 halves at once, by the recursive block swap of Warren, Hacker's
        // Delight, section 7-3.
        uint32_t m = 0x00ff00ffu;
#pragma unroll
        for (int j = 8; j; j >>= 1, m ^= m << j) {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                if (k & j) continue;
                const uint32_t t = ((r[k] >> j) ^ r[k + j]) & m;
                r[k + j] ^= t;
                r[k] ^= t << j;
            }
        }
        uint4* o = reinterpret_cast<uint4*>(nbr + 32 * i);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                lo[c] = __byte_perm(r[8 * k + 2 * c], r[8 * k + 2 * c + 1], 0x5410);
                hi[c] = __byte_perm(r[8 * k + 2 * c], r[8 * k + 2 * c + 1], 0x7632);
            }
            o[k] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            o[2 + k] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
}

}  // namespace

bool filter_bounds(ScreenArgs& a) {
    // Per class x = t ^ q: the largest score among the four (t, q) pairs of
    // that class.  sub is indexed (t << 2) | q (src/scoring.rs:32-40).
    int32_t ub[4];
    for (int x = 0; x < 4; x++) {
        int32_t m = INT32_MIN;
        for (int t = 0; t < 4; t++) m = std::max(m, a.sc.sub[(t << 2) | (t ^ x)]);
        ub[x] = m;
    }
    // Invalid columns score `ambig`: they take the class with the smallest
    // bound that is still >= ambig.  Past-the-end columns take the lowest
    // class, whose bound must be <= 0 (else a bounded side would never
    // break and the filter keeps nothing).
    int inv = -1, end = 0;
    for (int x = 0; x < 4; x++) {
        if (ub[x] >= a.sc.ambig && (inv < 0 || ub[x] < ub[inv])) inv = x;
        if (ub[x] < ub[end]) end = x;
    }
    if (inv < 0 || ub[end] > 0) return false;
    int64_t top = ub[0];
    for (int x = 1; x < 4; x++) top = std::max<int64_t>(top, ub[x]);
    // The bounded sums stay in i32: 4-column sums and prefixes are small,
    // and a side's run over f_cap columns is within the exact envelope the
    // host already checked for the scores' magnitude.
    for (int x = 0; x < 4; x++) a.fub[x] = ub[x];
    auto repeat = [](int x) {
        uint64_t p = 0;
        for (int k = 0; k < 32; k++) p |= (uint64_t)x << (2 * k);
        return p;
    };
    a.f_inv = repeat(inv);
    a.f_end = repeat(end);
    a.f_seed_max = (int32_t)(top * (int64_t)a.pat.len);
    return true;
}

void filter_init() {
    cudaFuncSetAttribute(k_filter_hits, cudaFuncAttributeMaxDynamicSharedMemorySize, kFilterSmem);
}

void launch_filter_hits(const ScreenArgs& a, const FilterIO& io, int sm_count, cudaStream_t st) {
    count_launch();
    k_filter_hits<<<sm_count, kFilterWarps * 32, kFilterSmem, st>>>(a, io);
}

void launch_occupancy(const uint32_t* starts, uint64_t num_words, uint32_t* occ, uint2* packed, cudaStream_t st) {
    const uint64_t words = (num_words + 31) / 32;
    const int blocks = (int)std::min<uint64_t>((words + 7) / 8, 148 * 16);
    count_launch();
    k_occupancy<<<std::max(blocks, 1), 256, 0, st>>>(starts, num_words, occ, packed);
}

void launch_neighbours(const uint32_t* occ, uint32_t n_views, uint32_t weight, uint16_t* nbr, cudaStream_t st) {
    const uint32_t per_view = 1u << (2 * weight - 5);
    const uint64_t words = (uint64_t)n_views * per_view;
    count_launch();
    k_neighbours<<<(int)std::min<uint64_t>((words + 255) / 256, 148 * 16), 256, 0, st>>>(occ, words, per_view, weight, nbr);
}

}  // namespace gxy
