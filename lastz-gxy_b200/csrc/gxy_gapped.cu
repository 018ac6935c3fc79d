// gxy_gapped.cu -- gapped extension (src/gapped_extend.rs:78-460) on the device.
//
// extend() runs a banded 3-state affine x-drop DP (Gotoh M/X/Y) to the right
// of an anchor and, on reversed inputs, to its left, then traces the best
// cell back into a run-length edit script.  The DP is row by row: row i's
// band is [lo - R, hi + R] around the previous row's surviving cells, capped
// at band_width = min(4R + 4, m + 1) cells; after a row, the cells whose best
// state is more than y_drop below the best score so far are killed.  These
// rules (the band, the row-major first maximum, the kill) decide the result,
// so the device keeps the row order.  One warp runs one side of one anchor
// (k_gapped_sides):
//
//  - The row's best states and the next row's X sit in shared memory, a ring
//    over the columns; a row is worked in chunks of 32 S columns, S consecutive
//    columns a lane, only where cells live.  While they stay in one chunk the
//    rows run in registers.
//  - X and M of a cell need the previous row only.  Y is a max-plus recurrence
//    along the row, Y[j] = max(M[j-1] - (O+E), Y[j-1] - E): each lane reduces its
//    cells to what they give the cell after them, and a warp shuffle scan
//    composes the lanes.  The arithmetic is the reference's i32 arithmetic:
//    max-plus composition is exact.
//  - The rows' best states go to global memory (pool blocks of kRows rows kept
//    by the warp across its tasks, a chain it grows from a shared pool as its
//    longest side needs).  After the last row the warp walks from the best cell
//    to (0, 0), finding each cell's source by value, and writes the runs.  Sides
//    whose rows did not fit the pool run again with exactly sized storage.
//
// A last kernel joins the two sides per anchor: total = anchor column + left
// best + right best (saturating), the left runs in walk order, the anchor's
// Match merged with its neighbours, the right runs reversed
// (src/gapped_extend.rs:99-131, src/edit_script.rs:63-92).
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "gxy_engine.cuh"

using namespace gxy;

namespace {

constexpr int32_t kNegInf = INT32_MIN / 4;   // NEG_INF (src/gapped_extend.rs:44)
constexpr int kMaxCells = 2048;               // band_width at most (the ring of a row's columns holds it)
constexpr int kRows = 32;                     // DP rows, and units of a row's chunks, a pool block holds at most
constexpr int kHdr = 4;                       // block header words: previous block, next block, first row (64 bits)
constexpr uint32_t kNone = 0xffffffffu;

// Side flags.
constexpr uint32_t kFlagPool = 1;    // the traceback pool ran out: rerun with a larger one
constexpr uint32_t kFlagRuns = 2;    // the run buffer ran out: the first pass reruns with a larger one
constexpr uint32_t kFlagState = 4;   // inconsistent traceback (a bug; reported as an error)
constexpr uint32_t kFlagScratch = 8; // more runs than the warp's scratch holds: the second pass
constexpr uint32_t kScratchWords = 16384;   // first pass: run scratch per warp (64 KB)
constexpr uint32_t kSideRuns2 = 1u << 8;   // the side's runs are in the second run buffer

// Counters (u64): task cursor, pool blocks claimed, run words reserved, rows,
// cells, flags, the most rows of one side.
enum { kCtrTask = 0, kCtrBlocks, kCtrRuns, kCtrRows, kCtrCells, kCtrFlags, kCtrMaxRows, kCtrWords = 8 };

constexpr int kMaxLaneCells = 16;
// Words of a unit (a chunk of 32 S cells of one row, 16 or 32 bits each) and of
// a pool block (a header, {thr, first column, units, first unit} of each row,
// the units).
__host__ __device__ constexpr uint32_t unit_words(int S, bool k16) { return k16 ? 16 * S : 32 * S; }
__host__ __device__ constexpr uint32_t pool_block_words(int S, bool k16) {
    return kHdr + 4 * kRows + kRows * unit_words(S, k16);
}

struct GapSide {
    int32_t score;
    uint32_t t_span;
    uint32_t q_span;
    uint32_t n_runs;
    uint64_t run_off;
    uint32_t flags;   // kFlag* | kSideRuns2
    uint32_t blocks;  // pool blocks its rows took, or would have taken
};

struct GapArgs {
    SeqView T, Q;
    const uint32_t* t_pos;
    const uint32_t* q_pos;
    uint32_t n_anchors;
    int32_t sub[16];
    int32_t ambig;
    int32_t goe;      // gap_open + gap_extend
    int32_t ge;       // gap_extend
    int32_t ydrop;
    int32_t rows[5][4];      // column scores of a row by target code (4: an invalid base) and query code
    uint32_t row_bytes[5];   // the same as bytes, query code 0 lowest (when every score fits one)
    int32_t nge[kMaxLaneCells]; // -c gap_extend
    int64_t radius;   // band radius; < 0: m + 1 (gap_extend <= 0)
    uint32_t* pool;
    uint64_t pool_blocks;
    uint32_t block_words;
    int32_t ring_blocks;  // lane blocks (S columns) of a warp's ring
    uint32_t* runs;       // where this pass's tracebacks write
    uint64_t runs_cap;
    const uint32_t* runs2;   // the second pass's runs (for the join)
    unsigned long long* ctr;
    GapSide* sides;   // [2a] left, [2a + 1] right
    // list: only the listed sides (nullptr: every side).  base (the second
    // pass): side list[k]'s rows go to the pool blocks base[k], base[k] + 1, ...
    // and its runs to the second run buffer; nullptr: blocks in chains.
    const uint32_t* list;
    const uint64_t* base;
    uint64_t n_list;
    // First pass: each warp walks its sides' tracebacks into its own
    // scratch of scratch_words words, then copies the runs out to a range of
    // exactly their number.
    uint32_t* scratch;
    uint32_t scratch_words;
};

__device__ __forceinline__ int32_t sat_add32(int32_t a, int32_t b) {
    const int64_t r = (int64_t)a + b;
    return r > INT32_MAX ? INT32_MAX : (r < INT32_MIN ? INT32_MIN : (int32_t)r);
}

// Swaps the two bits of every 2-bit field (undoes __brevll's swap inside a code).
__device__ __forceinline__ uint64_t swap_pairs(uint64_t x) {
    return ((x >> 1) & 0x5555555555555555ull) | ((x & 0x5555555555555555ull) << 1);
}

__device__ __forceinline__ uint32_t code_at(const SeqView& S, uint64_t gp) {
    return (uint32_t)(__ldg(S.codes + (gp >> 5)) >> (2 * (gp & 31))) & 3u;
}
__device__ __forceinline__ uint32_t valid_at(const SeqView& S, uint64_t gp) {
    return (__ldg(S.valid + (gp >> 5)) >> (gp & 31)) & 1u;
}

// One side of one anchor per warp, tasks claimed from a cursor.
//
// The row's state lives in shared memory, a ring over the columns: the best
// state H and the next row's X of a cell, and its query base.  A row is worked
// in chunks of 32 S columns, S consecutive columns a lane, from the first
// column that can be alive (cb) on: a chunk is read (which kills the previous
// row's cells below its threshold, finds its survivors and files it), and if
// it has a survivor or something enters it from the left, computed.  So a row
// costs the chunks its live cells touch -- one or two -- whatever the band, and
// chunks a row leaves out hold only dead cells: a value below a threshold stays
// below the later ones.
//
// Instead of back-pointers a row files its H, 16 bits a cell (k16): the
// survivors lie in [thr, thr + y_drop], so with the row's thr the low half of H
// gives it back, and thr - 1 marks a dead cell.  The traceback finds the
// sources by value (below).  X is not cleared in a dead cell: there it is below
// thr, and an X that once fell below only falls further behind, so it can never
// be a survivor's best state.
//
// What bounds it: a side's rows are a dependent chain, so a row's latency --
// here mostly the instructions one warp issues for it.  Additions issue every
// cycle, but maxima, selects, byte permutes and compares every other, so the
// form of a cell counts: its M is one dot product of the row's four score bytes
// with the query base's one-hot byte (on the multiplier pipe), the rest about
// eight half-rate instructions.
// Rows in one chunk (all but a few) stay in registers between two events --
// the rows' bases or the pool block running out, a cell about to leave the
// chunk -- and what only checks or counts is computed beside the scan.
// A 40 kbp alignment's three anchors: 17.1 ms, 0.42 us a row of the longest side
// (38,379 rows); all rows through shared memory 36 ms; a block of warps a side
// with 4 cells a thread, two reductions and three barriers a row 104 ms.  400
// anchors of 1.5 Mbp sequences: 6.3 ms against 33.
template <int S, bool kByte, bool k16, typename I>
__global__ void __launch_bounds__(32) k_gapped_sides(const __grid_constant__ GapArgs a) {
    constexpr int32_t kCols = 32 * S;
    constexpr uint32_t kUnit = unit_words(S, k16);
    extern __shared__ __align__(16) int4 g_ring[];
    const int lane = threadIdx.x;
    const int32_t goe = a.goe, ge = a.ge;
    const int32_t nblk = a.ring_blocks;        // lane blocks (S columns) of the ring
    int4* const rH = g_ring;                   // piece p of block b at p * nblk + b
    int4* const rX = rH + (S / 4) * nblk;
    int4* const rQ = rX + (S / 4) * nblk;
    const int32_t lane_ge = lane * S * ge;
    const uint64_t ntasks = a.list ? a.n_list : 2ull * a.n_anchors;
    // This warp's chain of pool blocks (kept across tasks), and the blocks it
    // claimed but has not linked yet.
    uint32_t chain_head = kNone, claim = 0, claim_end = 0;
    for (;;) {
        unsigned long long task = 0;
        if (lane == 0) task = atomicAdd(a.ctr + kCtrTask, 1ull);
        task = __shfl_sync(kFull, task, 0);
        if (task >= ntasks) break;
        const uint64_t fixed_base = a.base ? a.base[task] : 0;
        if (a.list) task = a.list[task];
        const uint32_t an = (uint32_t)(task >> 1);
        const bool right = task & 1;
        const uint32_t t0 = a.t_pos[an], q0 = a.q_pos[an];
        const I n = (I)(right ? a.T.len - t0 - 1 : t0);
        const I m = (I)(right ? a.Q.len - q0 - 1 : q0);
        GapSide res{};
        if (n == 0 || m == 0) {
            if (lane == 0) a.sides[task] = res;
            continue;
        }
        const I R = a.radius >= 0 ? (I)a.radius : m + 1;
        const I reach = a.radius >= 0 ? (I)min((int64_t)(4 * R + 3), (int64_t)m) : m;   // band_width - 1
        // The ring holds no survivor.
        for (int k = lane; k < (S / 4) * nblk; k += 32) rH[k] = rX[k] = make_int4(kNegInf, kNegInf, kNegInf, kNegInf);
        // Columns [.., q_end) of the query are in the ring: a one-hot byte of the
        // code, 0 for an invalid base (kByte), or the code, 4 for an invalid one.
        // (Columns past the query's end are dead whatever they score.)
        I q_end = 0, inv_end = 0;      // chunks from below inv_end on may hold invalid bases
        auto load_query = [&]() {
            const I col = q_end + lane * S;
            uint64_t qc = 0;
            uint32_t qv = 0;
            if (col <= m) {
                if (right) {
                    load_window32(a.Q, a.Q.base + q0 + (uint64_t)col, qc, qv);
                } else {
                    load_window32(a.Q, a.Q.base + q0 - (uint64_t)col - 31, qc, qv);
                    qc = swap_pairs(__brevll(qc));
                    qv = __brev(qv);
                }
            }
            const int32_t b = (int32_t)(((uint32_t)(q_end / S) + lane) % (uint32_t)nblk);
#pragma unroll
            for (int p = 0; p < S / 4; p++) {
                int32_t w[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t code = (uint32_t)(qc >> (2 * (4 * p + c))) & 3u, ok = (qv >> (4 * p + c)) & 1u;
                    w[c] = (int32_t)(kByte ? ok << (8 * code) : (ok ? code : 4u));
                }
                rQ[p * nblk + b] = make_int4(w[0], w[1], w[2], w[3]);
            }
            q_end += kCols;
            if (__any_sync(kFull, (~qv & ((1u << S) - 1u)) != 0 && col <= m)) inv_end = q_end;
            __syncwarp();
        };
        // Lane r's target base of row 32 k + r: its score bytes (kByte) or code;
        // the next rows' bases are loaded ahead.
        uint32_t rows_l = 0;
        uint64_t tw_next = 0;
        uint32_t tv_next = 0;
        auto target_load = [&](I r0) {
            if (r0 > n) return;
            if (right) {
                load_window32(a.T, a.T.base + t0 + (uint64_t)r0, tw_next, tv_next);
            } else {
                load_window32(a.T, a.T.base + t0 - (uint64_t)r0 - 31, tw_next, tv_next);
                tw_next = swap_pairs(__brevll(tw_next));
                tv_next = __brev(tv_next);
            }
        };
        target_load(0);
        __syncwarp();
        int32_t best = 0, thr = -a.ydrop;    // the best score of the rows so far, their threshold
        I bi = 0;                            // the best's row
        uint32_t flags = 0;
        // The pool block being filled: kRows rows and kRows units of kCols cells at
        // most; blocks of the chain in order, n_blk of them for this side.
        uint32_t blk = kNone, nxt = kNone, n_blk = 0;
        int32_t blk_rows = kRows, blk_units = 0;
        uint32_t* bp = nullptr;
        bool store = true;
        uint64_t cells = (uint64_t)min(R, reach) + 1;   // row 0's band
        I cb = 0;                            // the row's first column that can be alive, a multiple of S
        int32_t cbb = 0;                     // its block in the ring
        I e_prev = 0;                        // the previous row's cells are in columns [cb, e_prev)
        // The first and the last chunk with survivors of a row: the lanes that have
        // some, this lane's, and the chunk's first column.
        struct Ends {
            uint32_t f_live, f_alive, l_live, l_alive;
            I f_c0, l_c0;
        };
        Ends pe{};                           // of row i - 2
        I i = 0, rows = 0;
        // Pass i reads row i - 1 and computes row i; the band of row i - 1 is
        // counted and cb moved on then too, from the survivors of row i - 2, so
        // that nothing in the row waits for them.
        for (;; i++) {
            const int32_t r = (int32_t)(i & 31);
            if (r == 0) {
                const uint32_t tc = ((tv_next >> lane) & 1u) ? (uint32_t)(tw_next >> (2 * lane)) & 3u : 4u;
                rows_l = kByte ? a.row_bytes[tc] : tc;
                target_load(i + 32);
            }
            uint32_t* unit = nullptr;        // where row i - 1's chunks go
            if (i) {
                const int32_t ns = (int32_t)((uint32_t)(e_prev - cb + kCols - 1) / (uint32_t)kCols);
                if (blk_rows == kRows || blk_units + ns > kRows) {
                    // The next pool block: the chain's next one, or one of four
                    // claimed at a time (second pass: consecutive ones).
                    uint32_t nb = kNone;
                    if (a.base) {
                        nb = (uint32_t)fixed_base + n_blk;
                    } else if (store) {
                        nb = n_blk == 0 ? chain_head : __shfl_sync(kFull, nxt, 0);
                        if (nb == kNone) {
                            if (claim == claim_end) {
                                unsigned long long b = 0;
                                if (lane == 0) b = atomicAdd(a.ctr + kCtrBlocks, 4ull);
                                b = __shfl_sync(kFull, b, 0);
                                claim = (uint32_t)min(b, (unsigned long long)a.pool_blocks);
                                claim_end = (uint32_t)min(b + 4, (unsigned long long)a.pool_blocks);
                            }
                            if (claim < claim_end) {
                                nb = claim++;
                                if (lane == 0) {
                                    a.pool[(uint64_t)nb * a.block_words + 1] = kNone;
                                    if (blk != kNone) a.pool[(uint64_t)blk * a.block_words + 1] = nb;
                                }
                                if (chain_head == kNone) chain_head = nb;
                                nxt = kNone;
                            }
                        } else {
                            if (lane == 0) nxt = a.pool[(uint64_t)nb * a.block_words + 1];   // looked at a block later
                        }
                    }
                    if (nb == kNone) {
                        if (store) flags |= kFlagPool;   // the DP goes on: score, best row and rows stay exact
                        store = false;
                    } else {
                        bp = a.pool + (uint64_t)nb * a.block_words;
                        if (lane == 0) {
                            bp[0] = n_blk == 0 ? kNone : blk;
                            *reinterpret_cast<uint64_t*>(bp + 2) = (uint64_t)(i - 1);
                        }
                        blk = nb;
                    }
                    n_blk++;
                    blk_rows = blk_units = 0;
                }
                if (store) {
                    if (lane == 0)
                        *reinterpret_cast<uint4*>(bp + kHdr + 4 * blk_rows) =
                            make_uint4((uint32_t)thr, (uint32_t)cb, (uint32_t)ns, (uint32_t)blk_units);
                    unit = bp + kHdr + 4 * kRows + (uint32_t)blk_units * kUnit;
                }
                blk_rows++;
                blk_units += ns;
            }
            const int32_t thr_p = thr;       // the previous row's threshold
            // A dead cell's value: far below every threshold, its low half thr - 1.
            const int32_t dead = k16 ? (kNegInf & ~0xffff) | ((thr_p - 1) & 0xffff) : kNegInf;
            const uint32_t rw = __shfl_sync(kFull, rows_l, r);
            int32_t carry = kNegInf;         // H of the previous row left of the chunk
            int32_t T = kNegInf;             // Y entering the chunk
            int32_t rv = kNegInf;            // the largest M
            Ends ne{};                       // of row i - 1
            I lo2 = 0, hi2 = 0;              // row i - 2's first survivor, last + 1
            I e_new = cb;
            // The last column the row can have (from cb on; from the first survivor
            // on once a chunk needs it).
            I limit = min(m, max(cb - R, (I)0) + reach);
            for (I c0 = cb;; c0 += kCols) {
                int32_t b = cbb + (int32_t)((uint32_t)(c0 - cb) / S) + lane;
                while (b >= nblk) b -= nblk;
                int32_t H[S];
#pragma unroll
                for (int p = 0; p < S / 4; p++) {
                    const int4 v = rH[p * nblk + b];
                    H[4 * p] = v.x; H[4 * p + 1] = v.y; H[4 * p + 2] = v.z; H[4 * p + 3] = v.w;
                }
                // ---- the previous row's cells: kill, file, find the survivors.
                uint32_t alive = 0;
#pragma unroll
                for (int c = 0; c < S; c++) {
                    const bool ok = H[c] >= thr_p;
                    if (ok) alive |= 1u << c;
                    H[c] = ok ? H[c] : dead;
                }
                const uint32_t live = __ballot_sync(kFull, alive != 0);   // none in pass 0
                if (unit && c0 < e_prev) {
                    uint2* o = reinterpret_cast<uint2*>(unit) + lane;
                    if (k16) {
#pragma unroll
                        for (int p = 0; p < S / 4; p++)
                            o[32 * p] = make_uint2(__byte_perm((uint32_t)H[4 * p], (uint32_t)H[4 * p + 1], 0x5410),
                                                   __byte_perm((uint32_t)H[4 * p + 2], (uint32_t)H[4 * p + 3], 0x5410));
                    } else {
#pragma unroll
                        for (int p = 0; p < S / 2; p++) o[32 * p] = make_uint2((uint32_t)H[2 * p], (uint32_t)H[2 * p + 1]);
                    }
                    unit += kUnit;
                }
                // The first chunk is computed in any case (its row is dead if nothing
                // is alive), a later one if it has a survivor or one can enter it.
                bool work = i <= n;
                if (c0 != cb) work = work && (live || carry >= thr_p || T >= thr_p);
                if (work && c0 + kCols > limit) {
                    // The band's cap from its exact start.
                    const uint32_t fl = ne.f_live ? ne.f_live : live, fa = ne.f_live ? ne.f_alive : alive;
                    const I fc = ne.f_live ? ne.f_c0 : c0;
                    if (fl) {
                        const int lf = __ffs(fl) - 1;
                        const I lo = fc + lf * S + __ffs(__shfl_sync(kFull, fa, lf)) - 1;
                        limit = min(m, max(lo - R, (I)0) + reach);
                    }
                    work = c0 <= limit;
                }
                if (live) {
                    if (!ne.f_live) {
                        ne.f_live = live;
                        ne.f_alive = alive;
                        ne.f_c0 = c0;
                    }
                    ne.l_live = live;
                    ne.l_alive = alive;
                    ne.l_c0 = c0;
                }
                if (work) {
                    while (q_end < c0 + kCols) load_query();
                    int32_t X[S];
                    uint32_t sel[S];
#pragma unroll
                    for (int p = 0; p < S / 4; p++) {
                        const int4 x = rX[p * nblk + b], q = rQ[p * nblk + b];
                        X[4 * p] = x.x; X[4 * p + 1] = x.y; X[4 * p + 2] = x.z; X[4 * p + 3] = x.w;
                        sel[4 * p] = (uint32_t)q.x; sel[4 * p + 1] = (uint32_t)q.y;
                        sel[4 * p + 2] = (uint32_t)q.z; sel[4 * p + 3] = (uint32_t)q.w;
                    }
                    int32_t hl = __shfl_up_sync(kFull, H[S - 1], 1);
                    if (lane == 0) hl = carry;
                    carry = __shfl_sync(kFull, H[S - 1], 31);
                    int32_t M[S];
                    if (kByte) {
#pragma unroll
                        for (int c = 0; c < S; c++) M[c] = __dp4a((int32_t)rw, (int32_t)sel[c], c ? H[c - 1] : hl);
                        if (c0 < inv_end) {
#pragma unroll
                            for (int c = 0; c < S; c++)
                                if (!sel[c]) M[c] += a.ambig;
                        }
                    } else {
                        const int32_t s0 = a.rows[rw][0], s1 = a.rows[rw][1], s2 = a.rows[rw][2], s3 = a.rows[rw][3];
#pragma unroll
                        for (int c = 0; c < S; c++) {
                            const uint32_t q = sel[c];
                            const int32_t s = q > 3 ? a.ambig : ((q & 2) ? ((q & 1) ? s3 : s2) : ((q & 1) ? s1 : s0));
                            M[c] = (c ? H[c - 1] : hl) + s;
                        }
                    }
                    if (i == 0 && c0 == 0 && lane == 0) M[0] = 0;   // everything else is dead
                    const bool cut = c0 + kCols - 1 > limit;
                    const int32_t last = (int32_t)max(min(limit - c0 - lane * S, (I)S), (I)-1);
                    if (cut) {
#pragma unroll
                        for (int c = 0; c < S; c++)
                            if (c > last) M[c] = kNegInf;
                    }
                    int32_t lm[2] = {M[0], M[1]};
#pragma unroll
                    for (int c = 2; c < S; c += 2) lm[(c >> 1) & 1] = __vimax3_s32(lm[(c >> 1) & 1], M[c], M[c + 1]);
                    rv = max(rv, __reduce_max_sync(kFull, max(lm[0], lm[1])));
                    // Y inside the lane's cells (h[c]: what cells before c give cell
                    // c), composed over the lanes: an inclusive max-plus scan (a lane
                    // without a lane o below gets its own value back: no change).
                    int32_t fm[S], h[S];
#pragma unroll
                    for (int c = 0; c < S; c++) fm[c] = M[c] - goe;
                    h[0] = kNegInf;
                    h[1] = fm[0];
#pragma unroll
                    for (int c = 2; c < S; c++) h[c] = __viaddmax_s32(h[c - 1], -ge, fm[c - 1]);
                    int32_t A = __viaddmax_s32(h[S - 1], -ge, fm[S - 1]);
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int32_t p = __shfl_up_sync(kFull, A, o);
                        A = __viaddmax_s32(p, -o * S * ge, A);
                    }
                    {
                        // Row i - 2's survivors (beside the scan; any chunk gives the same).
                        const int lf = __ffs(pe.f_live) - 1, ll = 31 - __clz(pe.l_live);
                        lo2 = pe.f_c0 + lf * S + __ffs(__shfl_sync(kFull, pe.f_alive, lf & 31)) - 1;
                        hi2 = pe.l_c0 + ll * S + 32 - __clz(__shfl_sync(kFull, pe.l_alive, ll & 31));
                    }
                    int32_t yin = __shfl_up_sync(kFull, A, 1);
                    const int32_t tl = __shfl_sync(kFull, A, 31);
                    if (lane == 0) yin = kNegInf;
                    yin = __viaddmax_s32(T, -lane_ge, yin);
                    T = __viaddmax_s32(T, -kCols * ge, tl);
#pragma unroll
                    for (int c = 0; c < S; c++) {
                        const int32_t Y = c ? __viaddmax_s32(yin, a.nge[c], h[c]) : yin;
                        h[c] = __vimax3_s32(M[c], X[c], Y);
                        X[c] = __viaddmax_s32(X[c], -ge, fm[c]);
                    }
                    if (cut) {
#pragma unroll
                        for (int c = 0; c < S; c++)
                            if (c > last) h[c] = X[c] = kNegInf;
                    }
#pragma unroll
                    for (int p = 0; p < S / 4; p++) {
                        rH[p * nblk + b] = make_int4(h[4 * p], h[4 * p + 1], h[4 * p + 2], h[4 * p + 3]);
                        rX[p * nblk + b] = make_int4(X[4 * p], X[4 * p + 1], X[4 * p + 2], X[4 * p + 3]);
                    }
                    e_new = c0 + kCols;
                } else {
                    if (live && i <= n) {   // past the cap: no cells of this row, whatever lies above them
#pragma unroll
                        for (int p = 0; p < S / 4; p++)
                            rH[p * nblk + b] = rX[p * nblk + b] = make_int4(kNegInf, kNegInf, kNegInf, kNegInf);
                    }
                    carry = __shfl_sync(kFull, H[S - 1], 31);
                    T = kNegInf;
                }
                // On to the next chunk while the previous row has cells there, or
                // some can be entered from this one.
                const I next = c0 + kCols;
                if (next < e_prev) continue;
                if (i > n || !(carry >= thr_p || T >= thr_p)) break;
                if (next > limit) {
                    // The limit from cb may fall short of the one from the survivors.
                    if (!ne.f_live) break;
                    const int lf = __ffs(ne.f_live) - 1;
                    const I lo = ne.f_c0 + lf * S + __ffs(__shfl_sync(kFull, ne.f_alive, lf)) - 1;
                    limit = min(m, max(lo - R, (I)0) + reach);
                    if (next > limit) break;
                }
            }
            if (i > n && pe.f_live) {
                const int lf = __ffs(pe.f_live) - 1, ll = 31 - __clz(pe.l_live);
                lo2 = pe.f_c0 + lf * S + __ffs(__shfl_sync(kFull, pe.f_alive, lf & 31)) - 1;
                hi2 = pe.l_c0 + ll * S + 32 - __clz(__shfl_sync(kFull, pe.l_alive, ll & 31));
            }
            if (i > 1 && pe.f_live) {   // row i - 1's band
                const I jl = max(lo2 - R, (I)0);
                cells += (uint64_t)(min(min(hi2 - 1 + R, m), jl + reach) - jl + 1);
            }
            if (i && (!ne.f_live || i > n)) {   // row i - 1 is dead, or the target's last one
                rows = i;
                break;
            }
            // Only an M can exceed the best: Y stays below an M of its row, X
            // below an M of an earlier one.
            if (rv > best) bi = i;
            best = max(best, rv);
            thr = best - a.ydrop;
            e_prev = e_new;
            if (i > 1 && pe.f_live) {
                const int32_t k = (int32_t)((uint32_t)(lo2 - cb) / S);   // lane blocks that are dead for good
                cb += k * S;
                cbb += k;
                while (cbb >= nblk) cbb -= nblk;
            }
            pe = ne;
            // ---- rows whose cells stay in the first chunk, all of it in the band and
            // with valid query bases: the chunk in registers, until the rows'
            // bases or the pool block run out or a cell could leave the chunk on
            // the right (that row is then worked above, from its start).
            int32_t left = (int32_t)min((I)(31 - r), n - i);
            left = min(left, kRows - max(blk_rows, blk_units));
            if (left <= 0 || i < 2 || e_prev > cb + kCols || cb + kCols - 1 > min(m, max(cb - R, (I)0) + reach) ||
                q_end < cb + kCols || (kByte && cb < inv_end))
                continue;
            int32_t b = cbb + lane;
            while (b >= nblk) b -= nblk;
            int32_t H[S], X[S];
            uint32_t sel[S];
#pragma unroll
            for (int p = 0; p < S / 4; p++) {
                const int4 v = rH[p * nblk + b], x = rX[p * nblk + b], q = rQ[p * nblk + b];
                H[4 * p] = v.x; H[4 * p + 1] = v.y; H[4 * p + 2] = v.z; H[4 * p + 3] = v.w;
                X[4 * p] = x.x; X[4 * p + 1] = x.y; X[4 * p + 2] = x.z; X[4 * p + 3] = x.w;
                sel[4 * p] = (uint32_t)q.x; sel[4 * p + 1] = (uint32_t)q.y;
                sel[4 * p + 2] = (uint32_t)q.z; sel[4 * p + 3] = (uint32_t)q.w;
            }
            {   // row i's band, from row i - 1's survivors
                const int lf = __ffs(pe.f_live) - 1, ll = 31 - __clz(pe.l_live);
                const I lo = pe.f_c0 + lf * S + __ffs(__shfl_sync(kFull, pe.f_alive, lf)) - 1;
                const I hi = pe.l_c0 + ll * S + 32 - __clz(__shfl_sync(kFull, pe.l_alive, ll));
                const I jl = max(lo - R, (I)0);
                cells += (uint64_t)(min(min(hi - 1 + R, m), jl + reach) - jl + 1);
                pe.f_live = 0;   // counted
            }
            // (Without a pool block -- store is off -- nothing is filed.)
            uint4* mt = store ? reinterpret_cast<uint4*>(bp + kHdr + 4 * blk_rows) : nullptr;
            uint2* o = store ? reinterpret_cast<uint2*>(bp + kHdr + 4 * kRows + (uint32_t)blk_units * kUnit) + lane : nullptr;
            const I i0 = i;
            // Relative to cb: the first column (as far as a band from here reaches
            // left), the query's last one (as far as it reaches right), R.
            const int32_t Rc = (int32_t)min(R, (I)(1 << 20)), left0 = -(int32_t)min(cb, (I)(1 << 20)),
                          right0 = (int32_t)min(m - cb, (I)(1 << 22)), reach_c = (int32_t)min(reach, (I)(1 << 22));
            for (; left; left--) {
                uint32_t alive = 0;
                const int32_t dead1 = k16 ? (kNegInf & ~0xffff) | ((thr - 1) & 0xffff) : kNegInf;
#pragma unroll
                for (int c = 0; c < S; c++) {
                    const bool ok = H[c] >= thr;
                    if (ok) alive |= 1u << c;
                    H[c] = ok ? H[c] : dead1;
                }
                const uint32_t live = __ballot_sync(kFull, alive != 0);
                int32_t hl = __shfl_up_sync(kFull, H[S - 1], 1);
                const uint32_t rw1 = __shfl_sync(kFull, rows_l, (int)((i + 1) & 31));
                if (lane == 0) hl = kNegInf;
                int32_t M[S];
                if (kByte) {
#pragma unroll
                    for (int c = 0; c < S; c++) M[c] = __dp4a((int32_t)rw1, (int32_t)sel[c], c ? H[c - 1] : hl);
                } else {
                    const int32_t s0 = a.rows[rw1][0], s1 = a.rows[rw1][1], s2 = a.rows[rw1][2], s3 = a.rows[rw1][3];
#pragma unroll
                    for (int c = 0; c < S; c++) {
                        const uint32_t q = sel[c];
                        const int32_t s = q > 3 ? a.ambig : ((q & 2) ? ((q & 1) ? s3 : s2) : ((q & 1) ? s1 : s0));
                        M[c] = (c ? H[c - 1] : hl) + s;
                    }
                }
                int32_t lm[2] = {M[0], M[1]};
#pragma unroll
                for (int c = 2; c < S; c += 2) lm[(c >> 1) & 1] = __vimax3_s32(lm[(c >> 1) & 1], M[c], M[c + 1]);
                const int32_t rv1 = __reduce_max_sync(kFull, max(lm[0], lm[1]));
                int32_t fm[S], h[S];
#pragma unroll
                for (int c = 0; c < S; c++) fm[c] = M[c] - goe;
                h[0] = kNegInf;
                h[1] = fm[0];
#pragma unroll
                for (int c = 2; c < S; c++) h[c] = __viaddmax_s32(h[c - 1], -ge, fm[c - 1]);
                int32_t A = __viaddmax_s32(h[S - 1], -ge, fm[S - 1]);
#pragma unroll
                for (int q = 1; q < 32; q <<= 1) {
                    const int32_t w = __shfl_up_sync(kFull, A, q);
                    A = __viaddmax_s32(w, -q * S * ge, A);
                }
                const int lf = __ffs(live) - 1, ll = 31 - __clz(live);
                const int32_t lo = lf * S + __ffs(__shfl_sync(kFull, alive, lf & 31)) - 1;
                const int32_t hi = ll * S + 31 - __clz(__shfl_sync(kFull, alive, ll & 31));
                int32_t yin = __shfl_up_sync(kFull, A, 1);
                const int32_t tl = __shfl_sync(kFull, A, 31);
                if (lane == 0) yin = kNegInf;
                // (From the threshold before this row: it only rises.)
                if (tl >= thr - ge || live == 0 || (live >> 31)) break;
                if (store) {
#pragma unroll
                    for (int p = 0; p < S / 4; p++) {
                        if (k16) {
                            o[32 * p] = make_uint2(__byte_perm((uint32_t)H[4 * p], (uint32_t)H[4 * p + 1], 0x5410),
                                                   __byte_perm((uint32_t)H[4 * p + 2], (uint32_t)H[4 * p + 3], 0x5410));
                        } else {
                            o[64 * p] = make_uint2((uint32_t)H[4 * p], (uint32_t)H[4 * p + 1]);
                            o[64 * p + 32] = make_uint2((uint32_t)H[4 * p + 2], (uint32_t)H[4 * p + 3]);
                        }
                    }
                    if (lane == 0) *mt = make_uint4((uint32_t)thr, (uint32_t)cb, 1u, (uint32_t)blk_units);
                    o += kUnit / 2;
                    mt++;
                }
                blk_units++;
#pragma unroll
                for (int c = 0; c < S; c++) {
                    const int32_t Y = c ? __viaddmax_s32(yin, a.nge[c], h[c]) : yin;
                    H[c] = __vimax3_s32(M[c], X[c], Y);
                    X[c] = __viaddmax_s32(X[c], -ge, fm[c]);
                }
                i++;
                const int32_t jl = max(lo - Rc, left0);   // row i's band
                cells += (uint32_t)(min(min(hi + Rc, right0), jl + reach_c) - jl + 1);
                if (rv1 > best) bi = i;
                best = max(best, rv1);
                thr = best - a.ydrop;
            }
            blk_rows += (int32_t)(i - i0);
            if (i != i0) e_prev = cb + kCols;
#pragma unroll
            for (int p = 0; p < S / 4; p++) {
                rH[p * nblk + b] = make_int4(H[4 * p], H[4 * p + 1], H[4 * p + 2], H[4 * p + 3]);
                rX[p * nblk + b] = make_int4(X[4 * p], X[4 * p + 1], X[4 * p + 2], X[4 * p + 3]);
            }
        }
        __threadfence_block();
        __syncwarp();
        bool walk = !(flags & kFlagPool);
        // Row x in the pool: its block, given that of a row at or below it.
        auto first_row = [&](uint32_t b) { return *reinterpret_cast<const int64_t*>(a.pool + (uint64_t)b * a.block_words + 2); };
        auto block_of = [&](int64_t x, uint32_t b) {
            while (first_row(b) > x) b = a.pool[(uint64_t)b * a.block_words];
            return b;
        };
        // H of cell (x, c) in row x's block, whose first row is f; kNegInf: dead.
        auto h_at = [&](int64_t x, int64_t c, uint32_t b, int64_t f) {
            const uint32_t* p = a.pool + (uint64_t)b * a.block_words + kHdr;
            const uint4 mt = *reinterpret_cast<const uint4*>(p + 4 * (uint32_t)(x - f));
            const uint32_t rel = (uint32_t)c - mt.y;
            if (c < 0 || rel >= mt.z * (uint32_t)kCols) return kNegInf;
            const uint32_t ln = rel % (uint32_t)kCols / S, cc = rel % S;
            p += 4 * kRows + (mt.w + rel / (uint32_t)kCols) * kUnit;
            if (!k16) return (int32_t)p[((cc >> 1) * 32 + ln) * 2 + (cc & 1u)];
            const uint32_t d = ((uint32_t) reinterpret_cast<const uint16_t*>(p)[((cc >> 2) * 32 + ln) * 4 + (cc & 3u)] - mt.x) & 0xffffu;
            return d == 0xffffu ? kNegInf : (int32_t)(mt.x + d);
        };
        // The best's column: the first one of its row that holds it.
        int64_t bj = 0;
        uint32_t b = kNone;   // the pool block of the traceback's row, and its first row
        int64_t b0 = 0;
        if (bi && walk) {
            b = block_of((int64_t)bi, blk);
            b0 = first_row(b);
            const uint4 mt = *reinterpret_cast<const uint4*>(a.pool + (uint64_t)b * a.block_words + kHdr + 4 * (uint32_t)((int64_t)bi - b0));
            uint32_t at = kNone;
            for (uint32_t rel = lane; rel < mt.z * (uint32_t)kCols && at == kNone; rel += 32)
                if (h_at((int64_t)bi, (int64_t)mt.y + rel, b, b0) == best) at = mt.y + rel;
            bj = (int64_t)__reduce_min_sync(kFull, at);
        } else if (bi) {
            // An estimate: the second pass finds the column, and its host makes room for
            // the runs of one further right (the last row's cells can all lie to the left
            // of it).  Kept exactly, the end of the best row's chunks took 1 to 2 % of
            // every call's time.
            bj = (int64_t)min(m, e_prev);
        }
        res.score = best;
        res.t_span = (uint32_t)bi;
        res.q_span = (uint32_t)bj;
        // ---- traceback from the best cell (src/gapped_extend.rs:404-437), runs
        // in walk order (tip to root), from the rows' H alone.  With v = H(i, j):
        //  - the best state is M when H(i-1, j-1) + s(i, j) = v (a diagonal run
        //    is followed 32 cells at a time);
        //  - else it is X when some M(i-k, j) = v + (O+E) + (k-1) E, and the gap's
        //    length is the smallest such k: at each cell of the gap X comes from M
        //    exactly when M - (O+E) reaches its value, and the cells between are
        //    alive, their X being above v.  M is at most the row's best, which
        //    bounds k (E > 0); a cell between with H < v + its E's ends the
        //    search as well;
        //  - else it is Y, in the same way along the row.
        // The first pass walks into its scratch and reserves exactly the runs
        // written; the second pass reserves best_i + best_j words (the longest
        // possible script) and writes in place, if they fit: the counter has the
        // reservations of all sides in any case.
        int64_t ti = (int64_t)bi, tj = bj;
        int32_t v = best;
        uint32_t op = 3, cnt = 0, nr = 0;
        uint64_t off = 0, wcap = 0;
        const uint64_t cap = (uint64_t)((int64_t)bi + bj);
        uint32_t* wr = nullptr;
        if (walk && a.base) {
            if (lane == 0 && cap) off = atomicAdd(a.ctr + kCtrRuns, (unsigned long long)cap);
            off = __shfl_sync(kFull, off, 0);
            flags |= kSideRuns2;
            if (off + cap > a.runs_cap) {
                flags |= kFlagRuns;
                walk = false;
            }
            wr = a.runs + off;
            wcap = cap;
        } else if (walk) {
            wr = a.scratch + (uint64_t)blockIdx.x * a.scratch_words;
            wcap = a.scratch_words;
        }
        auto col_score = [&](int64_t x, int64_t c) {   // s(x, c), x and c at least 1
            const uint64_t tg = a.T.base + (uint64_t)((int64_t)t0 + (right ? x : -x));
            const uint64_t qg = a.Q.base + (uint64_t)((int64_t)q0 + (right ? c : -c));
            const uint32_t tc = code_at(a.T, tg), qc = code_at(a.Q, qg), ok = valid_at(a.T, tg) & valid_at(a.Q, qg);
            const int32_t s = a.rows[tc][qc];
            return ok ? s : a.ambig;
        };
        // M(x, c), row x - 1 in some block at or before b1: row 0 and column 0
        // hold one, at the origin.
        auto m_at = [&](int64_t x, int64_t c, uint32_t b1) {
            if (x == 0 || c == 0) return (x | c) ? kNegInf : 0;
            const uint32_t bb = block_of(x - 1, b1);
            const int32_t h = h_at(x - 1, c - 1, bb, first_row(bb));
            return h == kNegInf ? kNegInf : h + col_score(x, c);
        };
        if (walk && cap) {
            // pb: the block before b, from row p0 on.
            uint32_t pb = b0 ? block_of(b0 - 1, b) : b;
            int64_t p0 = b0 ? first_row(pb) : 0;
            while (ti | tj) {
                if (ti < b0) {
                    b = block_of(ti, pb);
                    b0 = first_row(b);
                    pb = b0 ? block_of(b0 - 1, b) : b;
                    p0 = b0 ? first_row(pb) : 0;
                }
                uint32_t eop, k;
                // Diagonal steps: lane l the one from (ti - l, tj - l).
                int32_t hm = kNegInf;
                bool diag = false;
                {
                    const int64_t x = ti - lane - 1;
                    const bool in = x >= p0 && lane < tj;
                    int32_t s = 0;
                    if (in) {
                        hm = h_at(x, tj - lane - 1, x >= b0 ? b : pb, x >= b0 ? b0 : p0);
                        s = col_score(x + 1, tj - lane);
                    }
                    int32_t h = __shfl_up_sync(kFull, hm, 1);
                    if (lane == 0) h = v;
                    diag = in && hm != kNegInf && hm + s == h;
                }
                const uint32_t stop = ~__ballot_sync(kFull, diag);
                k = stop ? (uint32_t)__ffs(stop) - 1 : 32u;
                if (k) {
                    v = __shfl_sync(kFull, hm, (int)k - 1);
                    ti -= (int64_t)k;
                    tj -= (int64_t)k;
                    eop = 0;
                } else {
                    // A gap: X (DeleteQuery) if one fits, else Y (InsertQuery).
                    const int32_t thr_i = (int32_t)a.pool[(uint64_t)b * a.block_words + kHdr + 4 * (uint32_t)(ti - b0)];
                    const int32_t room = thr_i + a.ydrop - v - goe;   // (k - 1) E at most
                    const int64_t kmax = room < 0 ? 0 : (ge ? room / ge + 1 : INT64_MAX);
                    eop = 3;
                    bool broken = false;
                    for (int64_t k0 = 1; k0 <= min(kmax, ti) && eop == 3 && !broken; k0 += 32) {
                        const int64_t kk = k0 + lane;
                        const bool in = kk <= min(kmax, ti);
                        bool hit = false, low = false;
                        if (in) {
                            // (A cell past its row's cap has no M: its H is dead.)
                            const uint32_t bb = block_of(ti - kk, b);
                            const int32_t h = h_at(ti - kk, tj, bb, first_row(bb)), want = v + goe + ((int32_t)kk - 1) * ge;
                            low = ge == 0 && h < v;
                            hit = h >= want && m_at(ti - kk, tj, bb) == want;
                        }
                        const uint32_t hb = __ballot_sync(kFull, hit), lb = __ballot_sync(kFull, low);
                        broken = lb != 0;
                        if (hb && (!lb || __ffs(hb) <= __ffs(lb))) {
                            k = (uint32_t)(k0 + __ffs(hb) - 1);
                            eop = 2;
                        }
                    }
                    for (int64_t k0 = 1; k0 <= min(kmax, tj) && eop == 3; k0 += 32) {
                        const int64_t kk = k0 + lane;
                        const bool hit = kk <= min(kmax, tj) && m_at(ti, tj - kk, b) == v + goe + ((int32_t)kk - 1) * ge;
                        const uint32_t hb = __ballot_sync(kFull, hit);
                        if (hb) {
                            k = (uint32_t)(k0 + __ffs(hb) - 1);
                            eop = 1;
                        }
                    }
                    if (eop == 3) {
                        flags |= kFlagState;
                        break;
                    }
                    v += goe + ((int32_t)k - 1) * ge;   // M at the gap's start
                    if (eop == 2) ti -= (int64_t)k;
                    else tj -= (int64_t)k;
                }
                if (eop == op) {
                    cnt += k;
                    continue;
                }
                if (cnt) {
                    if (nr >= wcap) {   // more runs than the scratch holds: the second pass
                        flags |= kFlagScratch;
                        break;
                    }
                    if (lane == 0) wr[nr] = (cnt << 2) | op;
                    nr++;
                }
                op = eop;
                cnt = k;
            }
            if (!(flags & (kFlagState | kFlagScratch)) && cnt) {
                if (nr >= wcap) {
                    flags |= kFlagScratch;
                } else {
                    if (lane == 0) wr[nr] = (cnt << 2) | op;
                    nr++;
                }
            }
        }
        __syncwarp();
        if (walk && !(flags & (kFlagState | kFlagScratch))) {
            res.n_runs = nr;
            res.run_off = off;
            if (!a.base) {   // the runs' range in the run buffer, exactly nr words
                if (lane == 0 && nr) off = atomicAdd(a.ctr + kCtrRuns, (unsigned long long)nr);
                off = __shfl_sync(kFull, off, 0);
                if (off + nr > a.runs_cap) {
                    flags |= kFlagRuns;
                } else {
                    res.run_off = off;
                    for (uint32_t k = lane; k < nr; k += 32) a.runs[off + k] = wr[k];
                }
            }
        }
        if (lane == 0) {
            res.flags = flags;
            res.blocks = n_blk;
            a.sides[task] = res;
            atomicAdd(a.ctr + kCtrRows, (unsigned long long)rows);
            atomicAdd(a.ctr + kCtrCells, (unsigned long long)cells);
            atomicMax(a.ctr + kCtrMaxRows, (unsigned long long)rows);
            if (flags) atomicOr(a.ctr + kCtrFlags, (unsigned long long)flags);
        }
        __syncwarp();
    }
}

__device__ __forceinline__ const uint32_t* side_runs(const GapArgs& a, const GapSide& s) {
    return ((s.flags & kSideRuns2) ? a.runs2 : a.runs) + s.run_off;
}

// Per anchor: the total, pass or fail, the joined run count.
__global__ void k_gapped_join(GapArgs a, int32_t threshold, gxy_gapped_aln* out, uint32_t* counts) {
    const uint32_t an = blockIdx.x * blockDim.x + threadIdx.x;
    if (an >= a.n_anchors) return;
    const GapSide L = a.sides[2 * an], R = a.sides[2 * an + 1];
    const uint32_t t0 = a.t_pos[an], q0 = a.q_pos[an];
    const uint64_t tg = a.T.base + t0, qg = a.Q.base + q0;
    const int32_t col = (valid_at(a.T, tg) && valid_at(a.Q, qg)) ? a.sub[code_at(a.T, tg) * 4 + code_at(a.Q, qg)]
                                                                  : a.ambig;
    const int32_t total = sat_add32(sat_add32(col, L.score), R.score);
    gxy_gapped_aln o{};
    o.score = total;
    uint32_t cnt = 0;
    if (total >= threshold) {
        o.passed = 1;
        o.t_start = t0 - L.t_span;
        o.q_start = q0 - L.q_span;
        o.t_len = L.t_span + 1 + R.t_span;
        o.q_len = L.q_span + 1 + R.q_span;
        const uint32_t* lr = side_runs(a, L), * rr = side_runs(a, R);
        const uint32_t lm = L.n_runs && (lr[L.n_runs - 1] & 3u) == 0;
        const uint32_t rm = R.n_runs && (rr[R.n_runs - 1] & 3u) == 0;
        cnt = L.n_runs + R.n_runs + 1 - lm - rm;
    }
    o.script_len = cnt;
    out[an] = o;
    counts[an] = cnt;
}

// Per anchor (one warp): the joined runs at offs[an].
__global__ void k_gapped_emit(GapArgs a, const gxy_gapped_aln* alns, const uint32_t* offs, uint32_t* out) {
    const int lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t an = blockIdx.x * (uint64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); an < a.n_anchors; an += nw) {
        if (!alns[an].passed) continue;
        const GapSide L = a.sides[2 * an], R = a.sides[2 * an + 1];
        const uint32_t* lr = side_runs(a, L);
        const uint32_t* rr = side_runs(a, R);
        const uint32_t lm = L.n_runs && (lr[L.n_runs - 1] & 3u) == 0;
        const uint32_t rm = R.n_runs && (rr[R.n_runs - 1] & 3u) == 0;
        const uint32_t nl = L.n_runs - lm, nr = R.n_runs - rm;
        uint32_t* o = out + offs[an];
        for (uint32_t k = lane; k < nl; k += 32) o[k] = lr[k];
        if (lane == 0) {
            const uint32_t mid = 1 + (lm ? lr[L.n_runs - 1] >> 2 : 0) + (rm ? rr[R.n_runs - 1] >> 2 : 0);
            o[nl] = mid << 2;
        }
        for (uint32_t k = lane; k < nr; k += 32) o[nl + 1 + k] = rr[nr - 1 - k];
    }
}

// The launch of the DP: S cells a lane, the ring, the pool layout.
struct SidesPlan {
    int S;
    bool bytes;           // every column score fits a byte
    bool k16;             // a survivor's distance from the threshold fits 16 bits
    bool wide;            // positions need more than 31 bits
    int32_t ring_blocks;
    uint32_t block_words; // words of a pool block
    size_t smem;
    int blocks;           // resident blocks
};

using SidesKernel = void (*)(GapArgs);
SidesKernel sides_kernel(const SidesPlan& p) {
    if (p.wide) return k_gapped_sides<16, false, false, int64_t>;
    if (!p.k16) return k_gapped_sides<16, false, false, int32_t>;
    if (!p.bytes) return k_gapped_sides<16, false, true, int32_t>;
    if (p.S == 16) return k_gapped_sides<16, true, true, int32_t>;
    return p.S == 8 ? k_gapped_sides<8, true, true, int32_t> : k_gapped_sides<4, true, true, int32_t>;
}

// Sizes the persistent grid.  Eight warps an SM (two a scheduler) fill the
// issue slots; more would only take pool and scratch.
cudaError_t plan_sides(SidesPlan& p, int sm_count) {
    int per_sm = 0;
    cudaError_t e = cudaFuncSetAttribute(sides_kernel(p), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sides_kernel(p), 32, p.smem);
    p.blocks = sm_count * std::max(std::min(per_sm, 8), 1);
    return e;
}

cudaError_t launch_sides(const GapArgs& a, const SidesPlan& p, cudaStream_t st) {
    count_launch();
    sides_kernel(p)<<<p.blocks, 32, p.smem, st>>>(a);
    return cudaGetLastError();
}

struct WorkerLease {
    gxy_ctx* ctx;
    Worker* w;
    gxy_status err;
    explicit WorkerLease(gxy_ctx* c) : ctx(c), w(nullptr), err(GXY_OK) { w = checkout(c, &err); }
    ~WorkerLease() {
        if (w) checkin(ctx, w);
    }
};

gxy_status fail(gxy_status s, const std::string& m) {
    set_error(m);
    return s;
}

}  // namespace

extern "C" {

gxy_status gxy_gapped_extend(gxy_ctx* ctx, const gxy_dseq* target, uint64_t t_lo, uint64_t t_hi,
                             const gxy_dseq* query, const gxy_search_params* params, const gxy_gapped_params* gp,
                             const uint32_t* t_pos, const uint32_t* q_pos, uint64_t n, gxy_gapped_result* out,
                             gxy_gapped_stats* stats) {
    if (!ctx || !target || !query || !params || !gp || !out || (n && (!t_pos || !q_pos)))
        return fail(GXY_EINVAL, "null argument");
    memset(out, 0, sizeof(*out));
    if (stats) memset(stats, 0, sizeof(*stats));
    if (t_lo == 0 && t_hi == 0) t_hi = target->len;
    if (t_lo > t_hi || t_hi > target->len) return fail(GXY_EINVAL, "target view outside the target");
    const uint64_t lt = t_hi - t_lo, lq = query->len;
    if (lt >= (1ull << 32) || lq >= (1ull << 32)) return fail(GXY_EUNSUPPORTED, "sequences of 2^32 bases or more");
    if (n >= (1ull << 31)) return fail(GXY_EUNSUPPORTED, "2^31 anchors or more");
    for (uint64_t k = 0; k < n; k++)
        if (t_pos[k] >= lt || q_pos[k] >= lq) return fail(GXY_EINVAL, "anchor outside its sequence");
    // The exact envelope: every DP value formed stays far from i32 limits, and
    // values formed from NEG_INF stay below every threshold.
    int64_t smax = std::abs((int64_t)params->ambig);
    for (int k = 0; k < 16; k++) smax = std::max<int64_t>(smax, std::abs((int64_t)params->sub[k]));
    if (smax > (1 << 16)) return fail(GXY_EUNSUPPORTED, "substitution scores beyond +-65536");
    if (gp->gap_open < 0 || gp->gap_open > (1 << 20) || gp->gap_extend < 0 || gp->gap_extend > (1 << 16))
        return fail(GXY_EUNSUPPORTED, "gap costs outside [0, 2^20] (open) / [0, 2^16] (extend)");
    if (gp->y_drop < 0 || gp->y_drop > (1 << 27)) return fail(GXY_EUNSUPPORTED, "y_drop outside [0, 2^27]");
    // A cell's score is at most the largest positive column score times the
    // columns of the shorter sequence.
    int64_t spos = std::max<int64_t>(0, params->ambig);
    for (int k = 0; k < 16; k++) spos = std::max<int64_t>(spos, params->sub[k]);
    if ((double)spos * (double)(std::min(lt, lq) + 2) >= 2147483648.0 - 1048576.0)
        return fail(GXY_EUNSUPPORTED, "scores could exceed 2^31 - 2^20 on sequences this long");
    const int32_t goe = gp->gap_open + gp->gap_extend, ge = gp->gap_extend;
    int64_t radius = -1;
    if (ge > 0) {
        const int64_t r = ((int64_t)gp->y_drop - goe) / ge;   // truncates toward zero, as Rust's i32 `/`
        radius = std::max<int64_t>(r, 0) + 2;
    }
    // Band width bound over all sides: min(4R + 4, m + 1) with m < lq.
    const int64_t bw_max = radius >= 0 ? std::min<int64_t>(4 * radius + 4, (int64_t)lq) : (int64_t)lq;
    int Sc = 4;
    {
        std::lock_guard<std::mutex> g(ctx->mu);
        if (ctx->tuning.gapped_cells == 8) Sc = 8;
    }
    if (bw_max > kMaxCells)
        return fail(GXY_EUNSUPPORTED, "band wider than 2048 cells (y_drop / gap_extend too large for the device DP)");
    // S: a row's live cells span the gaps to the right of the best cell (R
    // columns) and shorter ones to its left, about 1.3 R while the best still
    // grows (379 columns for R = 301 on a 40 kbp alignment at 90 % identity) and
    // 2 R and more after it, so that most rows take one chunk of 32 S columns.
    // gapped_cells = 8 asks for chunks of 256 columns.
    const int64_t span = std::min<int64_t>(radius >= 0 ? radius + radius * 3 / 10 : (int64_t)lq, (int64_t)lq);
    SidesPlan plan{};
    plan.wide = std::max(lt, lq) >= (1ull << 31) - 16384;
    plan.bytes = smax <= 127;
    plan.k16 = gp->y_drop < 65535 && !plan.wide;
    plan.S = !plan.k16 || !plan.bytes ? 16 : (Sc == 8 ? 8 : (span <= 112 ? 4 : (span <= 240 ? 8 : 16)));
    // The ring: a row's band (at most 4R + 4 columns, or the query), the alignment
    // of its first column, a last chunk that overhangs it, and one of query bases
    // loaded ahead.
    const int64_t chunk = 32 * plan.S, cols = std::min<int64_t>(radius >= 0 ? 4 * radius + 4 : (int64_t)lq, (int64_t)lq);
    plan.ring_blocks = (int32_t)((cols + plan.S + 2 * chunk + chunk - 1) / chunk * 32);
    plan.block_words = pool_block_words(plan.S, plan.k16);
    plan.smem = (size_t)plan.ring_blocks * plan.S * 12;
    out->n_alns = n;
    out->alns = n ? (gxy_gapped_aln*)calloc(n, sizeof(gxy_gapped_aln)) : nullptr;
    if (n && !out->alns) return fail(GXY_ENOMEM, "host allocation");
    if (n == 0) return GXY_OK;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return fail(GXY_ECUDA, "cudaSetDevice");
    WorkerLease Lw(ctx);
    if (!Lw.w) {
        gxy_gapped_result_free(out);
        return Lw.err;
    }
    Worker* W = Lw.w;
    cudaStream_t st = W->st;
    // Per-anchor arrays: anchors (2 x u32), sides (2 x 32 B), joined records,
    // run counts and offsets (+1), counters.
    const size_t off_t = 0, off_q = off_t + n * 4, off_side = (off_q + n * 4 + 255) & ~(size_t)255,
                 off_aln = off_side + 2 * n * sizeof(GapSide), off_cnt = off_aln + n * sizeof(gxy_gapped_aln),
                 off_offs = off_cnt + n * 4, off_ctr = (off_offs + (n + 1) * 4 + 255) & ~(size_t)255,
                 aux_bytes = off_ctr + kCtrWords * 8;
    cudaError_t e = W->gaux.ensure(aux_bytes);
    if (e != cudaSuccess) {
        gxy_gapped_result_free(out);
        return fail(GXY_ENOMEM, std::string("gapped buffers: ") + cudaGetErrorString(e));
    }
    unsigned char* aux = W->gaux.as<unsigned char>();
    GapArgs A{};
    A.T = view_of(target, t_lo, t_hi);
    A.Q = view_of(query, 0, lq);
    A.t_pos = reinterpret_cast<uint32_t*>(aux + off_t);
    A.q_pos = reinterpret_cast<uint32_t*>(aux + off_q);
    A.n_anchors = (uint32_t)n;
    memcpy(A.sub, params->sub, sizeof(A.sub));
    A.ambig = params->ambig;
    A.goe = goe;
    A.ge = ge;
    A.ydrop = gp->y_drop;
    A.radius = radius;
    for (int c = 0; c < kMaxLaneCells; c++) A.nge[c] = -c * ge;
    for (int t = 0; t < 5; t++) {
        A.row_bytes[t] = 0;
        for (int q = 0; q < 4; q++) {
            A.rows[t][q] = t < 4 ? params->sub[t * 4 + q] : params->ambig;
            A.row_bytes[t] |= ((uint32_t)A.rows[t][q] & 0xffu) << (8 * q);
        }
    }
    A.ctr = reinterpret_cast<unsigned long long*>(aux + off_ctr);
    A.sides = reinterpret_cast<GapSide*>(aux + off_side);
    gxy_gapped_aln* d_aln = reinterpret_cast<gxy_gapped_aln*>(aux + off_aln);
    uint32_t* d_cnt = reinterpret_cast<uint32_t*>(aux + off_cnt);
    uint32_t* d_offs = reinterpret_cast<uint32_t*>(aux + off_offs);
    e = cudaMemcpyAsync(aux + off_t, t_pos, n * 4, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(aux + off_q, q_pos, n * 4, cudaMemcpyHostToDevice, st);
    // Pass 1: every side, its rows in chains of pool blocks.  The pool is sized
    // for 32 pool blocks per warp and grows toward what earlier calls needed,
    // within a quarter of the free device memory.
    if (e == cudaSuccess) e = plan_sides(plan, ctx->sm_count);
    A.ring_blocks = plan.ring_blocks;
    A.block_words = plan.block_words;
    const uint64_t block_bytes = (uint64_t)plan.block_words * 4;
    size_t free_b = 0, total_b = 0;
    uint32_t pool_limit = 0;
    {
        std::lock_guard<std::mutex> g(ctx->mu);
        pool_limit = ctx->tuning.gapped_pool_blocks;
    }
    uint64_t want_pool = std::max<uint64_t>((uint64_t)plan.blocks * 32 * block_bytes, W->gpool_want);
    if (want_pool > W->gpool.bytes) {   // growing: at most a quarter of the free memory
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) free_b = 0;
        const uint64_t pool_cap = std::max<uint64_t>((uint64_t)plan.blocks * 4 * block_bytes, free_b / 4);
        want_pool = std::max<uint64_t>(std::min(want_pool, pool_cap), W->gpool.bytes);
    } else {
        want_pool = W->gpool.bytes;
    }
    // Runs: a first-pass side reserves exactly the runs it wrote (the second
    // pass reserves best_i + best_j words in a buffer of its own).
    uint64_t want_runs = std::max<uint64_t>(std::max<uint64_t>(n * 512, std::min<uint64_t>(n * 4096, 1ull << 28)),
                                            W->gruns.bytes / 4);
    cudaEvent_t e0 = W->ev[0], e1 = W->ev[2];
    unsigned long long ctr[kCtrWords] = {};
    uint32_t reruns = 0;
    A.list = nullptr;
    A.base = nullptr;
    A.n_list = 0;
    A.runs2 = nullptr;
    // First pass: a run scratch per resident CUDA block.
    A.scratch_words = kScratchWords;
    if (e == cudaSuccess) e = W->gscr.ensure((size_t)plan.blocks * kScratchWords * 4);
    A.scratch = W->gscr.as<uint32_t>();
    float ms = 0.f;
    // One launch between the two events; its counters come back.
    auto launch = [&](const GapArgs& a, unsigned long long* c) {
        cudaError_t r = cudaEventRecord(e0, st);
        if (r == cudaSuccess) r = launch_sides(a, plan, st);
        if (r == cudaSuccess) r = cudaEventRecord(e1, st);
        if (r == cudaSuccess) r = cudaMemcpyAsync(c, a.ctr, kCtrWords * 8, cudaMemcpyDeviceToHost, st);
        if (r == cudaSuccess) r = cudaStreamSynchronize(st);
        float t = 0.f;
        if (r == cudaSuccess) cudaEventElapsedTime(&t, e0, e1);
        ms += t;
        return r;
    };
    for (int attempt = 0; e == cudaSuccess; attempt++) {
        e = W->gpool.ensure(want_pool);
        if (e == cudaSuccess) e = W->gruns.ensure(want_runs * 4);
        if (e != cudaSuccess) break;
        A.pool = W->gpool.as<uint32_t>();
        A.pool_blocks = W->gpool.bytes / block_bytes;
        if (pool_limit) A.pool_blocks = std::min<uint64_t>(A.pool_blocks, pool_limit);
        A.runs = W->gruns.as<uint32_t>();
        A.runs_cap = W->gruns.bytes / 4;
        ms = 0.f;
        e = cudaMemsetAsync(A.ctr, 0, kCtrWords * 8, st);
        if (e == cudaSuccess) e = launch(A, ctr);
        if (e != cudaSuccess) break;
        // Only a short run buffer reruns the whole pass (the pool's shortfall
        // goes to pass 2): grow it to what the sides reserved.
        if (!(ctr[kCtrFlags] & kFlagRuns) || attempt >= 2) break;
        want_runs = std::max<uint64_t>(want_runs * 2, ctr[kCtrRuns] * 5 / 4 + 1024);
        reruns++;
    }
    constexpr unsigned long long kShort = kFlagPool | kFlagRuns | kFlagScratch;
    if (e == cudaSuccess && (ctr[kCtrFlags] & kFlagState)) {
        gxy_gapped_result_free(out);
        return fail(GXY_ECUDA, "gapped extension: inconsistent traceback state");
    }
    // Pass 2: the sides pass 1 could not store, each with exactly the blocks
    // its rows need (pass 1 counted them), in groups that fit half the free
    // memory; their runs go to a second buffer of exactly their reservations.
    uint32_t* d_pool2 = nullptr;
    uint32_t* d_runs2 = nullptr;
    void* d_list = nullptr;
    uint64_t pass2_sides = 0, pass2_cells = 0;
    if (e == cudaSuccess && (ctr[kCtrFlags] & kShort)) {
        std::vector<GapSide> sides(2 * n);
        e = cudaMemcpyAsync(sides.data(), A.sides, 2 * n * sizeof(GapSide), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        std::vector<uint32_t> list;
        std::vector<uint64_t> need;
        uint64_t runs2 = 0, max_need = 0, tot_need = 0;
        for (uint64_t k = 0; e == cudaSuccess && k < 2 * n; k++) {
            if (!(sides[k].flags & kShort)) continue;
            list.push_back((uint32_t)k);
            const uint64_t nb = sides[k].blocks;
            need.push_back(nb);
            max_need = std::max(max_need, nb);
            tot_need += nb;
            runs2 += (uint64_t)sides[k].t_span + sides[k].q_span;
        }
        pass2_sides = list.size();
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) free_b = 0;
        const uint64_t group_blocks = std::min<uint64_t>(std::max<uint64_t>(max_need, free_b / 2 / block_bytes), tot_need);
        if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_runs2, std::max<uint64_t>(runs2, 1) * 4, st);
        if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_pool2, group_blocks * block_bytes, st);
        if (e == cudaSuccess) e = cudaMallocAsync(&d_list, list.size() * 16, st);
        // Later calls start with a pass-1 pool closer to this need.
        W->gpool_want = (A.pool_blocks + tot_need) * block_bytes;
        GapArgs B = A;
        B.pool = d_pool2;
        B.pool_blocks = group_blocks;
        B.runs = d_runs2;
        B.runs_cap = std::max<uint64_t>(runs2, 1);
        uint32_t* dl = reinterpret_cast<uint32_t*>(d_list);
        uint64_t* dbase = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(d_list) + list.size() * 8);
        std::vector<uint64_t> base(list.size());
        uint64_t k0 = 0;
        unsigned long long c2[kCtrWords] = {};
        uint64_t reserved = 0;   // run words of the groups done
        bool more_room = false;
        while (e == cudaSuccess && k0 < list.size()) {
            uint64_t k1 = k0, used = 0;
            while (k1 < list.size() && used + need[k1] <= group_blocks) {
                base[k1] = used;
                used += need[k1];
                k1++;
            }
            B.list = dl + k0;
            B.base = dbase + k0;
            B.n_list = k1 - k0;
            e = cudaMemcpyAsync(dl + k0, list.data() + k0, (k1 - k0) * 4, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(dbase + k0, base.data() + k0, (k1 - k0) * 8, cudaMemcpyHostToDevice, st);
            // The task cursor restarts; the run counter goes on from the groups done.
            if (e == cudaSuccess) e = cudaMemsetAsync(B.ctr + kCtrTask, 0, 8, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(B.ctr + kCtrRuns, &reserved, 8, cudaMemcpyHostToDevice, st);
            // Rows and cells count this group's sides only.
            if (e == cudaSuccess) e = cudaMemsetAsync(B.ctr + kCtrRows, 0, 16, st);
            if (e == cudaSuccess) e = cudaMemsetAsync(B.ctr + kCtrFlags, 0, 8, st);
            if (e == cudaSuccess) e = launch(B, c2);
            if (e == cudaSuccess && !(c2[kCtrFlags] & (kFlagPool | kFlagState)) && (c2[kCtrFlags] & kFlagRuns) && !more_room) {
                // The columns were estimates; now all that this group's sides need is
                // known.  The groups done keep their runs.
                uint32_t* bigger = nullptr;
                B.runs_cap += c2[kCtrRuns] - reserved;
                e = cudaMallocAsync((void**)&bigger, B.runs_cap * 4, st);
                if (e == cudaSuccess && reserved) e = cudaMemcpyAsync(bigger, d_runs2, reserved * 4, cudaMemcpyDeviceToDevice, st);
                if (e == cudaSuccess) std::swap(d_runs2, bigger);
                if (bigger) cudaFreeAsync(bigger, st);
                B.runs = d_runs2;
                more_room = true;
                pass2_cells += c2[kCtrCells];
                continue;
            }
            if (e == cudaSuccess && (c2[kCtrFlags] & (kFlagPool | kFlagRuns | kFlagState))) {
                cudaFreeAsync(d_pool2, st);
                cudaFreeAsync(d_runs2, st);
                cudaFreeAsync(d_list, st);
                cudaStreamSynchronize(st);
                gxy_gapped_result_free(out);
                return fail(GXY_ECUDA, "gapped extension: the exactly sized second pass fell short");
            }
            pass2_cells += c2[kCtrCells];
            reserved = c2[kCtrRuns];
            more_room = false;
            k0 = k1;
        }
        A.runs2 = d_runs2;
    }
    uint32_t total_runs = 0;
    if (e == cudaSuccess) {
        count_launch();
        k_gapped_join<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(A, gp->gapped_threshold, d_aln, d_cnt);
        scan_u32(d_cnt, d_offs, nullptr, n, n, true, nullptr, W->ps, st);
        e = cudaMemcpyAsync(&total_runs, d_offs + n, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(out->alns, d_aln, n * sizeof(gxy_gapped_aln), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    uint32_t* d_final = nullptr;
    if (e == cudaSuccess && total_runs) {
        out->runs = (uint32_t*)malloc((size_t)total_runs * 4);
        if (!out->runs) {
            gxy_gapped_result_free(out);
            return fail(GXY_ENOMEM, "host allocation");
        }
        e = cudaMallocAsync((void**)&d_final, (size_t)total_runs * 4, st);
        if (e == cudaSuccess) {
            const uint64_t blocks = std::min<uint64_t>((n + 7) / 8, (uint64_t)ctx->sm_count * 16);
            count_launch();
            k_gapped_emit<<<(unsigned)blocks, 256, 0, st>>>(A, d_aln, d_offs, d_final);
            e = cudaMemcpyAsync(out->runs, d_final, (size_t)total_runs * 4, cudaMemcpyDeviceToHost, st);
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (d_final) cudaFreeAsync(d_final, st);
    }
    if (d_pool2) cudaFreeAsync(d_pool2, st);
    if (d_runs2) cudaFreeAsync(d_runs2, st);
    if (d_list) cudaFreeAsync(d_list, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        gxy_gapped_result_free(out);
        return fail(e == cudaErrorMemoryAllocation ? GXY_ENOMEM : GXY_ECUDA,
                    std::string("gapped extension: ") + cudaGetErrorString(e));
    }
    out->n_runs = total_runs;
    // Offsets of the passing anchors' scripts: the scan's output, on the host.
    uint64_t acc = 0;
    for (uint64_t k = 0; k < n; k++) {
        out->alns[k].script_off = acc;
        acc += out->alns[k].script_len;
    }
    if (stats) {
        stats->rows = ctr[kCtrRows];
        stats->cells = ctr[kCtrCells];
        stats->device_ms = ms;
        stats->reruns = reruns;
        stats->second_pass_sides = pass2_sides;
        stats->second_pass_cells = pass2_cells;
        stats->warps_per_side = 1;
        stats->cells_per_thread = (uint32_t)plan.S;
        stats->max_side_rows = ctr[kCtrMaxRows];
    }
    return GXY_OK;
}

void gxy_gapped_result_free(gxy_gapped_result* r) {
    if (!r) return;
    free(r->alns);
    free(r->runs);
    r->alns = nullptr;
    r->runs = nullptr;
    r->n_alns = r->n_runs = 0;
}

}  // extern "C"
