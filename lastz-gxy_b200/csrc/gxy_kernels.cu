// gxy_kernels.cu -- the seed->HSP kernels for sm_100a.
//
// Work is integer and byte work bounded by HBM/L2, so there are no tensor
// cores here.  Shapes: grids are persistent (a multiple of the SM count) or
// grid-stride; every sequence access goes through the padded layout of
// gxy_device.cuh.
#include "gxy_kernels.cuh"

namespace gxy {

__host__ __device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

// ---------------------------------------------------------------------------
// Packing
// ---------------------------------------------------------------------------

// encode_base (src/dna.rs:12-20) on one byte: code, valid, soft-masked.
__device__ __forceinline__ void encode(uint8_t b, uint32_t& code, uint32_t& valid, uint32_t& masked) {
    const uint8_t u = b & 0xDF;   // ASCII upper case
    code = 0;
    valid = 1;
    if (u == 'A') code = 0;
    else if (u == 'C') code = 1;
    else if (u == 'G') code = 2;
    else if (u == 'T' || u == 'U') code = 3;
    else valid = 0;
    masked = valid && (b >= 'a' && b <= 'z');
}

// One thread per 32 positions: reads 32 ASCII bytes (two 16-byte loads when
// aligned), writes one u64 of codes and one u32 each of valid and mask.
__global__ void k_pack_ascii(const uint8_t* __restrict__ ascii, uint64_t n, uint64_t* codes, uint32_t* valid,
                             uint32_t* mask) {
    const uint64_t nw = (n + 31) / 32;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t p0 = w * 32;
        uint64_t c = 0;
        uint32_t v = 0, m = 0;
#pragma unroll 8
        for (int k = 0; k < 32; k++) {
            const uint64_t p = p0 + k;
            if (p >= n) break;
            uint32_t code, val, msk;
            encode(ascii[p], code, val, msk);
            c |= (uint64_t)code << (2 * k);
            v |= val << k;
            m |= msk << k;
        }
        // Local position p lives at global kPad + p; kPad is a multiple of 32.
        codes[kPad / 32 + w] = c;
        valid[kPad / 32 + w] = v;
        mask[kPad / 32 + w] = m;
    }
}

void launch_pack_ascii(const uint8_t* ascii, uint64_t n, uint64_t* codes, uint32_t* valid, uint32_t* mask,
                       cudaStream_t st) {
    const uint64_t nw = (n + 31) / 32;
    if (!nw) return;
    const int blocks = (int)umin64((nw + 255) / 256, 148 * 16);
    count_launch();
    k_pack_ascii<<<blocks, 256, 0, st>>>(ascii, n, codes, valid, mask);
}

// Reverse complement: output position o takes input position n-1-o; a valid
// base becomes its complement (3 - c), an invalid one code 0 and unmasked,
// and the mask bit moves with the base (src/sequences.rs:303-318).  One thread
// per 32 output positions; the 32 input positions are one unaligned load.
struct RcWord {
    uint64_t c;
    uint32_t v, m;
};

// Output positions [32w, 32w+32) <- input positions n-1-32w down to n-32-32w.
__device__ __forceinline__ RcWord rc_word(const uint64_t* ic, const uint32_t* iv, const uint32_t* im, uint64_t n, uint64_t w) {
    // Load the 32 input positions ending at n-1-32w: start gp = kPad + n - 32 - 32w
    // (never below 32 because kPad = 64).
    const uint64_t gp = kPad + n - 32 - 32 * w;
    uint64_t c = load_codes32(ic, gp);
    uint32_t v = load_bits32(iv, gp);
    uint32_t m = load_bits32(im, gp);
    // Input lane j (position gp + j) maps to output lane 31 - j.
    v = __brev(v);
    m = __brev(m) & v;
    c = __brevll(c);
    // __brevll reverses bits; swap the two bits of each pair back.
    c = ((c >> 1) & 0x5555555555555555ull) | ((c & 0x5555555555555555ull) << 1);
    c = (~c) & spread_bits_to_pairs(v);
    const uint32_t nvalid = (uint32_t)umin64(32, n - 32 * w);
    if (nvalid < 32) {
        const uint32_t keep = (1u << nvalid) - 1;
        v &= keep;
        m &= keep;
        c &= spread_bits_to_pairs(keep);
    }
    return RcWord{c, v, m};
}

__global__ void k_reverse_complement(const uint64_t* __restrict__ ic, const uint32_t* __restrict__ iv,
                                     const uint32_t* __restrict__ im, uint64_t n, uint64_t* oc, uint32_t* ov,
                                     uint32_t* om) {
    const uint64_t nw = (n + 31) / 32;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x) {
        const RcWord r = rc_word(ic, iv, im, n, w);
        oc[kPad / 32 + w] = r.c;
        ov[kPad / 32 + w] = r.v;
        om[kPad / 32 + w] = r.m;
    }
}

// Many sequences at once, pads included: a block takes 256 words of one.  What
// bounds it is the launch: 300 contigs of 20 kbp, with a launch, an allocation
// and a fill for each, took 3.0 us of device time and 8 us of host time a
// contig; together 11 us of device time
// for all (cold caches) and 0.1 us of host time each.
__global__ __launch_bounds__(256) void k_reverse_complement_many(const RcItem* __restrict__ items, uint32_t n_items) {
    uint32_t lo = 0, hi = n_items;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (items[mid].block_base <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    const RcItem it = items[lo];
    const uint64_t i = (uint64_t)(blockIdx.x - it.block_base) * 256 + threadIdx.x;
    if (i >= it.nwords) return;
    RcWord r{0, 0, 0};
    const uint64_t w = i - kPad / 32;   // (wraps below the first one)
    if (i >= kPad / 32 && w < (it.n + 31) / 32) r = rc_word(it.icodes, it.ivalid, it.imask, it.n, w);
    it.ocodes[i] = r.c;
    it.ovalid[i] = r.v;
    it.omask[i] = r.m;
}

void launch_reverse_complement(const uint64_t* icodes, const uint32_t* ivalid, const uint32_t* imask, uint64_t n,
                               uint64_t* ocodes, uint32_t* ovalid, uint32_t* omask, cudaStream_t st) {
    const uint64_t nw = (n + 31) / 32;
    if (!nw) return;
    const int blocks = (int)umin64((nw + 255) / 256, 148 * 16);
    count_launch();
    k_reverse_complement<<<blocks, 256, 0, st>>>(icodes, ivalid, imask, n, ocodes, ovalid, omask);
}

void launch_reverse_complement_many(const RcItem* items, uint32_t n_items, uint32_t n_blocks, cudaStream_t st) {
    count_launch();
    k_reverse_complement_many<<<n_blocks, 256, 0, st>>>(items, n_items);
}

// ---------------------------------------------------------------------------
// Seed words and the table build
// ---------------------------------------------------------------------------

__global__ void k_seed_words(SeqView view, Pattern pat, uint32_t step, uint32_t nwin, uint32_t sentinel,
                             uint32_t* keys, uint32_t* vals, uint32_t* counts) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nwin; k += gridDim.x * blockDim.x) {
        const uint32_t p = k * step;
        uint32_t w;
        if (word_at(view, pat, p, w)) {
            keys[k] = w;
            atomicAdd(&counts[w], 1u);
        } else {
            keys[k] = sentinel;
        }
        vals[k] = p;
    }
}

void launch_seed_words(SeqView view, Pattern pat, uint32_t step, uint32_t nwin, uint32_t sentinel, uint32_t* keys,
                       uint32_t* vals, uint32_t* counts, cudaStream_t st) {
    if (!nwin) return;
    const int blocks = (int)umin64((nwin + 255) / 256, 148 * 16);
    count_launch();
    k_seed_words<<<blocks, 256, 0, st>>>(view, pat, step, nwin, sentinel, keys, vals, counts);
}


__global__ void k_prune_counts(const uint32_t* starts, uint64_t nw, uint32_t limit, uint32_t* counts2) {
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = starts[w + 1] - starts[w];
        counts2[w] = c <= limit ? c : 0u;
    }
}

void launch_prune_counts(const uint32_t* starts, uint64_t num_words, uint32_t limit, uint32_t* counts2,
                         cudaStream_t st) {
    count_launch();
    k_prune_counts<<<148 * 8, 256, 0, st>>>(starts, num_words, limit, counts2);
}

__global__ void k_prune_copy(const uint32_t* pos, const uint32_t* starts, uint64_t nw, const uint32_t* new_starts,
                             uint32_t limit, uint32_t* new_pos) {
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = starts[w], e = starts[w + 1];
        if (e - s > limit) continue;
        const uint32_t o = new_starts[w];
        for (uint32_t i = s; i < e; i++) new_pos[o + (i - s)] = pos[i];
    }
}

void launch_prune_copy(const uint32_t* positions, const uint32_t* starts, uint64_t num_words,
                       const uint32_t* new_starts, uint32_t limit, uint32_t* new_positions, cudaStream_t st) {
    count_launch();
    k_prune_copy<<<148 * 8, 256, 0, st>>>(positions, starts, num_words, new_starts, limit, new_positions);
}

// ---------------------------------------------------------------------------
// Scan helpers of the exact lane-per-hit screens below (k_screen_wide and
// the packed k_screen).  The screens read hits from a global array written
// either by k_enumerate (every raw hit) or by k_seed_filter in gxy_filter.cu
// (only the hits whose upper-bound x-drop might reach hspthresh).
// ---------------------------------------------------------------------------

// 32 positions starting at offset o of a 4-word window (o <= 96).
__device__ __forceinline__ uint64_t win_codes(const uint64_t (&w)[4], uint32_t o) {
    const uint32_t i = o >> 5, s = (o & 31) * 2;
    const uint64_t lo = i == 0 ? w[0] : (i == 1 ? w[1] : w[2]);
    const uint64_t hi = i == 0 ? w[1] : (i == 1 ? w[2] : w[3]);
    return s ? ((lo >> s) | (hi << (64 - s))) : lo;
}
__device__ __forceinline__ uint32_t win_bits(const uint32_t (&w)[4], uint32_t o) {
    const uint32_t i = o >> 5;
    const uint32_t lo = i == 0 ? w[0] : (i == 1 ? w[1] : w[2]);
    const uint32_t hi = i == 0 ? w[1] : (i == 1 ? w[2] : w[3]);
    return __funnelshift_r(lo, hi, o & 31);
}

// Spreads the 2-bit codes of 16 columns (32 bits) into 16 nibbles (64 bits).
__device__ __forceinline__ uint64_t spread16(uint32_t x) {
    uint64_t v = x;
    v = (v | (v << 16)) & 0x0000FFFF0000FFFFull;
    v = (v | (v << 8)) & 0x00FF00FF00FF00FFull;
    v = (v | (v << 4)) & 0x0F0F0F0F0F0F0F0Full;
    v = (v | (v << 2)) & 0x3333333333333333ull;
    return v;
}

// The x-drop scan of extend_one_side (src/hsp.rs:179-193) over up to 32
// columns whose codes and validity are in registers (column k at bits 2k /
// bit k).  Continues a side from (run, best, bext) after ext0 columns; n = 0
// is a no-op.  Sets ended when the x-drop break fired; used = columns consumed.
template <bool kCheckValid>
__device__ __forceinline__ void scan32(uint64_t tc, uint64_t qc, uint32_t vv, uint32_t n, int32_t xd,
                                       const int32_t* lut, int32_t ambig, uint32_t ext0, int32_t& run,
                                       int32_t& best, uint32_t& bext, bool& ended, uint32_t& used) {
    // idx_k = (t_k << 2) | q_k as nibble k of nib[k / 16].
    const uint64_t nib0 = (spread16((uint32_t)tc) << 2) | spread16((uint32_t)qc);
    const uint64_t nib1 = (spread16((uint32_t)(tc >> 32)) << 2) | spread16((uint32_t)(qc >> 32));
    int32_t r = run, b = best;
    uint32_t be = bext, lim = n, brk = n;
#pragma unroll
    for (int g = 0; g < 4; g++) {
        if (!__any_sync(kFull, (uint32_t)(g * 8) < lim)) break;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int k = g * 8 + i;
            if ((uint32_t)k < lim) {
                const uint32_t idx = (uint32_t)(((k < 16 ? nib0 : nib1) >> (4 * (k & 15))) & 15u);
                int32_t sc = lut[idx];
                if (kCheckValid) sc = ((vv >> k) & 1u) ? sc : ambig;
                r += sc;
                if (r > b) {
                    b = r;
                    be = ext0 + k + 1;
                } else if (b - r > xd) {
                    brk = k;
                    lim = 0;
                }
            }
        }
    }
    ended = brk < n;
    used = ended ? brk + 1 : n;
    run = r;
    best = b;
    bext = be;
}

// One side's scan state for the interleaved scans below.
struct SideScan {
    uint64_t nib0, nib1;   // (t << 2 | q) nibbles of columns 0-15 and 16-31
    uint32_t vv;           // column validity
    uint32_t lim;          // columns still to scan (0 once the side broke)
    uint32_t brk;          // break column, or n when the side did not break
    uint32_t ext0;         // columns of this side already scanned
    int32_t r, b;          // running score, best
    uint32_t be;           // best extent
};

__device__ __forceinline__ void side_init(SideScan& S, uint64_t tc, uint64_t qc, uint32_t vv, uint32_t n,
                                          uint32_t ext0, int32_t run, int32_t best, uint32_t bext) {
    S.nib0 = (spread16((uint32_t)tc) << 2) | spread16((uint32_t)qc);
    S.nib1 = (spread16((uint32_t)(tc >> 32)) << 2) | spread16((uint32_t)(qc >> 32));
    S.vv = vv;
    S.lim = n;
    S.brk = n;
    S.ext0 = ext0;
    S.r = run;
    S.b = best;
    S.be = bext;
}

template <bool kCheckValid, int k>
__device__ __forceinline__ void side_step(SideScan& S, int32_t xd, const int32_t* lut, int32_t ambig) {
    if ((uint32_t)k < S.lim) {
        const uint32_t idx = (uint32_t)(((k < 16 ? S.nib0 : S.nib1) >> (4 * (k & 15))) & 15u);
        int32_t sc = lut[idx];
        if (kCheckValid) sc = ((S.vv >> k) & 1u) ? sc : ambig;
        S.r += sc;
        if (S.r > S.b) {
            S.b = S.r;
            S.be = S.ext0 + k + 1;
        } else if (S.b - S.r > xd) {
            S.brk = k;
            S.lim = 0;
        }
    }
}

// Two independent sides scanned column by column in lockstep: the x-drop
// recurrence of each side is a serial chain, and interleaving two chains
// lets the scheduler issue from both.
template <bool kCheckValid>
__device__ __forceinline__ void scan_pair(SideScan& A, SideScan& B, int32_t xd, const int32_t* lut,
                                          int32_t ambig) {
#define GXY_STEP8(g)                                                             \
    side_step<kCheckValid, g * 8 + 0>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 0>(B, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 1>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 1>(B, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 2>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 2>(B, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 3>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 3>(B, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 4>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 4>(B, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 5>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 5>(B, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 6>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 6>(B, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 7>(A, xd, lut, ambig);                        \
    side_step<kCheckValid, g * 8 + 7>(B, xd, lut, ambig);
    if (!__any_sync(kFull, A.lim > 0 || B.lim > 0)) return;
    GXY_STEP8(0)
    if (!__any_sync(kFull, A.lim > 8 || B.lim > 8)) return;
    GXY_STEP8(1)
    if (!__any_sync(kFull, A.lim > 16 || B.lim > 16)) return;
    GXY_STEP8(2)
    if (!__any_sync(kFull, A.lim > 24 || B.lim > 24)) return;
    GXY_STEP8(3)
#undef GXY_STEP8
}

__device__ __forceinline__ void scan_pair_any(SideScan& A, SideScan& B, uint32_t na, uint32_t nb, int32_t xd,
                                              const int32_t* lut, int32_t ambig) {
    const uint32_t need_a = na >= 32 ? 0xffffffffu : ((1u << na) - 1u);
    const uint32_t need_b = nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u);
    if (__any_sync(kFull, (A.vv & need_a) != need_a || (B.vv & need_b) != need_b))
        scan_pair<true>(A, B, xd, lut, ambig);
    else
        scan_pair<false>(A, B, xd, lut, ambig);
}

// ---------------------------------------------------------------------------
// Enumeration: one warp per item -- a tile of 32 consecutive query windows of
// one unit and a group of word variants.  Each lane forms its window's seed word
// (src/seed_search.rs:76-90) by table, and a mask of the variants whose bucket
// is not empty: with transitions, bit 1 + i stands for the word with care
// position i's transition.  The table's neighbour masks give it in one read
// (13 occupancy bits, one read each, took most of the L2 traffic before).  Two
// transitions take a group for every first one: the masks of the words one
// transition away, less the pairs other groups hold; a group is an item of its own while the items can be counted in
// 32 bits (n_split), else a tile is.
//
// The masks' bits -- a tenth to half of the variants -- are listed across the
// warp, so that the bucket bounds and the positions are read 32 entries at a
// time with every lane at work; the warp reserves room for all hits of the item
// with one atomic and writes (t, q[, unit]) for every position of every listed
// bucket (src/pos_table.rs:102-108), neighbouring lanes to neighbouring slots.
//
// What bounds it: the latency of dependent reads (words, mask, bounds,
// position) and the L2 sectors of the last two.  10 Mbp x 10 Mbp, one
// transition, 26.1 M hits: 0.36 ms, 101 M L2 sectors and
// 0.60 GB of DRAM traffic (with 13 occupancy bits and the plain starts read per
// window 0.74 ms; with the masks and the plain starts, 64 MB that push the masks
// and positions out of L2, 0.59 ms and 1.7 GB; four entries a lane at a time
// instead of two spill registers, 0.42 ms).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void store_hit(const ScreenArgs& a, uint64_t i, uint32_t t, uint32_t q, uint32_t u) {
    a.hits[i] = t;
    a.hits[a.hit_cap + i] = q;
    if (a.n_units > 1) a.hits[2 * a.hit_cap + i] = u;
}

constexpr int kEnumWarps = 8, kEnumBlocks = 4;   // 31 KB of shared memory a block, 35 with a lane a byte
constexpr uint32_t kWordBits = (1u << 27) - 1;   // of an entry; the lane above
constexpr uint32_t kBigReads = 5;               // of a lane in a large bucket

// kMode 0: the words themselves only; 1: neighbour masks; 2: masks formed from
// the occupancy bitmap (tables without neighbour masks).
template <int kMode>
__global__ __launch_bounds__(kEnumWarps * 32, kEnumBlocks) void k_enumerate(const __grid_constant__ ScreenArgs a) {
    constexpr uint32_t kEntries = kMode == 0 ? 32 : 512;   // 32 masks of at most 16 bits
    constexpr int K = kMode == 0 ? 1 : 2;                  // entries a lane holds at a time
    __shared__ unsigned long long s_stats[2];              // windows, raw hits
    __shared__ uint32_t s_ent[kEnumWarps][kEntries];       // the entries' words, then their buckets' starts
    __shared__ uint32_t s_cnt[kEnumWarps][kMode == 0 ? 1 : kEntries - 64];   // lane and size from entry 64 on
    __shared__ uint8_t s_who[kMode == 1 ? 1 : kEnumWarps][kEntries];          // the entries' lanes
    const int lane = threadIdx.x & 31;
    const uint32_t weight = a.pat.weight;
    if (threadIdx.x < 2) s_stats[threadIdx.x] = 0;
    __syncthreads();
    uint32_t* const ent = s_ent[threadIdx.x >> 5];
    uint32_t* const cnt = s_cnt[threadIdx.x >> 5];
    uint8_t* const who = s_who[kMode == 1 ? 0 : threadIdx.x >> 5];
    const uint32_t n_items = a.n_items, n_groups = a.n_groups, n_split = a.n_split;
    uint32_t windows = 0, n_raw = 0;   // of the lane, of the warp: fewer than the tiles and the buffer's slots
    uint32_t* const ctl = a.ctl;
    unsigned long long* const max_fail = reinterpret_cast<unsigned long long*>(ctl + kCMaxFail);
    // This pass takes the items the previous pass could not fit first (its
    // redo list), then fresh items until the hit buffer is full.
    const uint32_t pass = ctl[kCPass];
    const uint2* redo_in = a.redo + ((pass - 1) & 1u) * kRedoCap;
    uint2* redo_out = a.redo + (pass & 1u) * kRedoCap;
    const uint32_t n_redo = ctl[kCRedoN + ((pass - 1) & 1u)];
    uint32_t* const n_redo_out = ctl + kCRedoN + (pass & 1u);
    // A tile's group that did not fit this pass goes to the next pass's list.
    auto defer = [&](uint32_t tile, uint32_t group, unsigned long long wtot) {
        atomicExch(ctl + kCStop, 1u);
        const uint32_t i = atomicAdd(n_redo_out, 1u);
        if (i < kRedoCap) redo_out[i] = make_uint2(tile, group);
        else atomicExch(ctl + kCRedoOver, 1u);
        atomicMax(max_fail, wtot);
    };
    bool redo_done = n_redo == 0;
    // Fresh items are claimed kClaim at a time, and the next claim is made
    // while the current items are processed: one atomic per kClaim items
    // (all warps hit that counter), its round trip off the critical path.
    // (Measured on the 10 Mbp plain launch: 2 beats 4 by 2 % and 8 is slower.)
    constexpr uint32_t kClaim = 2;
    uint32_t next = 0xffffffffu;   // a claimed batch not yet started (warp-uniform)
    uint32_t u = 0, u_lo = 1, u_hi = 0;   // the current unit and its tiles (none yet)
    const UnitDev* U = a.units;   // (read where used: kept in registers, they spilled others)
    for (;;) {
      uint32_t batch, batch_end, group, group_end;   // items (or one listed tile), their groups
      if (!redo_done) {
          uint32_t i = 0;
          if (lane == 0) i = atomicAdd(ctl + kCRedoTake, 1u);
          i = __shfl_sync(kFull, i, 0);
          if (i < n_redo) {
              const uint2 r = redo_in[i];
              batch = r.x;
              batch_end = r.x + 1;
              group = r.y;
              group_end = n_split > 1 ? r.y + 1 : n_groups;
          } else {
              redo_done = true;
              continue;
          }
      } else {
          if (next == 0xffffffffu) {
              // Stop claiming once the buffer is full; the items not claimed
              // yet wait for the next pass behind the cursor.
              if (*reinterpret_cast<volatile uint32_t*>(ctl + kCStop)) break;
              uint32_t c = 0;
              if (lane == 0) c = atomicAdd(a.tile_counter, kClaim);
              next = __shfl_sync(kFull, c, 0);
          }
          batch = next;
          if (batch >= n_items) break;
          next = 0xffffffffu;
          if (!*reinterpret_cast<volatile uint32_t*>(ctl + kCStop)) {
              uint32_t c = 0;
              if (lane == 0) c = atomicAdd(a.tile_counter, kClaim);
              next = __shfl_sync(kFull, c, 0);
          }
          batch_end = min(n_items, batch + kClaim);
          group = 0;
          group_end = n_groups;
      }
      for (uint32_t item = batch; item < batch_end; item++) {
        uint32_t tile = item, g = group, g_end = group_end;
        if (n_split > 1 && redo_done) {   // an item is one group of a tile
            tile = item / n_split;
            g = item - tile * n_split;
            g_end = g + 1;
        }
        if (tile < u_lo || tile >= u_hi) {
            uint32_t lo = 0, hi = a.n_units;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (a.units[mid].tile_base <= tile) lo = mid;
                else hi = mid;
            }
            u = lo;
            U = a.units + u;
            u_lo = U->tile_base;
            u_hi = u_lo + (U->nwin + 31) / 32;
        }
        const uint32_t k = (tile - u_lo) * 32 + lane;
        // The window's word.
        uint32_t word0 = 0;
        bool wv = false;
        if (k < U->nwin) {
            const SeqView& Q = a.qsegs[U->qseg];
            const uint64_t gq = Q.base + (uint64_t)k * a.step;
            const uint32_t ok = load_bits32(Q.valid, gq) & ~load_bits32(Q.mask, gq);
            wv = (ok & a.pat.care_mask) == a.pat.care_mask;
            word0 = word_of(a.pat, load_codes32(Q.codes, gq));
        }
        for (; g < g_end; g++) {
            if (g == 0) windows += wv ? 1 : 0;
            // Group g > 0: the words one transition (of care position g - 1) away, with
            // a second one at a later position.
            const uint32_t word = kMode != 0 && g ? word0 ^ (2u << (2 * (weight - g))) : word0;
            uint32_t mask = 0;
            if (wv) {
                if (kMode == 0) {
                    mask = (__ldg(U->occ + (word >> 5)) >> (word & 31u)) & 1u;
                } else if (kMode == 1) {
                    mask = __ldg(U->nbr + word);
                } else {
                    for (uint32_t i = 0; i <= weight; i++) {
                        const uint32_t w = i ? word ^ (2u << (2 * (weight - i))) : word;
                        mask |= ((__ldg(U->occ + (w >> 5)) >> (w & 31u)) & 1u) << i;
                    }
                }
                if (kMode != 0 && g) mask &= ~((2u << g) - 1u);
            }
            // ---- the masks' bits, listed: bucket word and lane of each.
            const uint32_t mine = __popc(mask);
            uint32_t pos = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, pos, o);
                if (lane >= o) pos += y;
            }
            const uint32_t n_ent = __shfl_sync(kFull, pos, 31);
            if (n_ent == 0) continue;
            pos -= mine;
            __syncwarp();
            if (kMode == 1) {   // (bit by bit: finding the next one set has a longer latency)
                const uint32_t tagged = word | (uint32_t)lane << 27;
                if (mask & 1u) ent[pos++] = tagged;
                uint32_t flip = 2u << (2 * (weight - 1));
#pragma unroll
                for (uint32_t v = 1; v <= kNbrMaxWeight; v++, flip >>= 2)
                    if ((mask >> v) & 1u) ent[pos++] = tagged ^ flip;
            } else {
                while (mask) {
                    const uint32_t v = __ffs(mask) - 1;
                    mask &= mask - 1;
                    ent[pos] = v ? word ^ (2u << (2 * (weight - v))) : word;
                    who[pos] = (uint8_t)lane;
                    pos++;
                }
            }
            __syncwarp();
            // ---- their bounds: start, and size with the lane in the top bits, the first 64 entries' in
            // registers, the others' in place of the words; and the item's hits.
            uint32_t rb[K], rc[K];
            HitSum sum;
            auto bounds = [&](uint32_t e0) {
                uint32_t w[K];
#pragma unroll
                for (int k = 0; k < K; k++) {
                    w[k] = 0;
                    rc[k] = 0;
                    if (e0 + 32 * k + lane < n_ent) w[k] = ent[e0 + 32 * k + lane];
                }
                if (kMode == 1) {
                    uint2 p[K];
#pragma unroll
                    for (int k = 0; k < K; k++)
                        if (e0 + 32 * k + lane < n_ent) p[k] = __ldg(U->packed + ((w[k] & kWordBits) >> 3));
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        if (e0 + 32 * k + lane < n_ent) {
                            const uint32_t sh = 4 * (w[k] & 7u), below = p[k].y & ((1u << sh) - 1u);
                            rb[k] = p[k].x + __dp4a((below & 0x0f0f0f0fu) + ((below >> 4) & 0x0f0f0f0fu), 0x01010101u, 0u);
                            uint32_t c = (p[k].y >> sh) & 15u;
                            if (p[k].y == 0xffffffffu) {   // a bucket of 15 or more among the eight
                                rb[k] = __ldg(U->starts + (w[k] & kWordBits));
                                c = __ldg(U->starts + (w[k] & kWordBits) + 1) - rb[k];
                            }
                            sum.add(c);
                            rc[k] = min(c, kWordBits) | (w[k] & ~kWordBits);
                        }
                    }
                } else {
                    uint32_t h[K];
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        if (e0 + 32 * k + lane < n_ent) {
                            rb[k] = __ldg(U->starts + w[k]);
                            h[k] = __ldg(U->starts + w[k] + 1);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        if (e0 + 32 * k + lane < n_ent) {
                            sum.add(h[k] - rb[k]);
                            rc[k] = min(h[k] - rb[k], kWordBits) | (uint32_t)who[e0 + 32 * k + lane] << 27;
                        }
                    }
                }
            };
            for (uint32_t e0 = (n_ent - 1) & ~63u; e0; e0 -= 64) {
                bounds(e0);
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (e0 + 32 * k + lane < n_ent) {
                        ent[e0 + 32 * k + lane] = rb[k];
                        cnt[e0 - 64 + 32 * k + lane] = rc[k];
                    }
                }
            }
            bounds(0);
            sum.lo = __reduce_add_sync(kFull, sum.lo);
            sum.hi = __reduce_add_sync(kFull, sum.hi);
            const unsigned long long wtot = sum.total();
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(a.hit_count, wtot);
            // ---- entry e's first hit takes slot e, the second hits of the larger buckets
            // come behind those, and so on: both 32 consecutive slots at a time.  The
            // hits' order in the buffer is free (candidates are sorted by a unique
            // (diagonal, t) key later).
            uint32_t first[K];
#pragma unroll
            for (int k = 0; k < K; k++)   // on their way while the reservation comes back
                if (32 * k + lane < n_ent) first[k] = __ldg(U->positions + rb[k]);
            base = __shfl_sync(kFull, base, 0);
            if (!hits_fit(base, wtot, a.hit_cap)) {
                // The buffer is full: this item goes to the next pass, and the
                // part of its reservation inside the buffer is marked unused.
                if (lane == 0) defer(tile, g, wtot);
                for (uint64_t j = base + lane; j < min((unsigned long long)a.hit_cap, base + wtot); j += 32)
                    a.hits[a.hit_cap + j] = kNoHit;
                if (g == 0) windows -= wv ? 1 : 0;
                break;   // with the groups after it
            }
            n_raw += lane == 0 ? (uint32_t)wtot : 0;   // (no more than the buffer's slots)
            const uint32_t q0 = (tile - u_lo) * 32;
            uint64_t more = base + n_ent;   // where the next further hits go
            for (uint32_t e0 = 0;;) {
#pragma unroll
                for (int k = 0; k < K; k++)
                    if (e0 + 32 * k + lane < n_ent)
                        store_hit(a, base + e0 + 32 * k + lane, first[k], (q0 + (rc[k] >> 27)) * a.step, u);
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (e0 + 32 * k >= n_ent) break;
                    const uint32_t c = rc[k] & kWordBits, q = (q0 + (rc[k] >> 27)) * a.step;
                    const bool big = c > 16;
                    for (uint32_t j = 1;; j++) {
                        const uint32_t m = __ballot_sync(kFull, c > j && !big);
                        if (m == 0) break;
                        if (c > j && !big)
                            store_hit(a, more + __popc(m & ((1u << lane) - 1u)), __ldg(U->positions + rb[k] + j), q, u);
                        more += __popc(m);
                    }
                    uint32_t bm = __ballot_sync(kFull, big);
                    while (bm) {   // a large bucket is copied by the whole warp
                        const int src = __ffs(bm) - 1;
                        bm &= bm - 1;
                        const uint32_t bb = __shfl_sync(kFull, rb[k], src);
                        uint32_t cc = __shfl_sync(kFull, c, src);
                        const uint32_t qq = __shfl_sync(kFull, q, src);
                        if (cc == kWordBits) {   // its size did not fit: the next larger start ends it
                            uint32_t lo = 0, hi = 1u << (2 * weight);
                            while (lo < hi) {
                                const uint32_t mid = lo + (hi - lo) / 2;
                                if (U->starts[mid] > bb) hi = mid;
                                else lo = mid + 1;
                            }
                            cc = U->starts[lo] - bb;
                        }
                        // Several reads on their way at a time: a run of one base (or another
                        // short unit) in the query is one warp's millions of hits (29 M hits of
                        // runs of A: 7.5 ms, one read at a time 34.5; four 7.1, six 7.1 and
                        // eight 5.8, but with spills that ordinary tiles pay for, 1 % with six;
                        // in a function of its own 12 %).
                        const uint32_t* from = U->positions + bb + 1 + lane;
                        uint32_t* to = a.hits + more + lane;
                        uint32_t left = cc - 1;
                        for (; left >= 32 * kBigReads; left -= 32 * kBigReads) {
                            uint32_t p[kBigReads];
#pragma unroll
                            for (uint32_t x = 0; x < kBigReads; x++) p[x] = __ldg(from + 32 * x);
#pragma unroll
                            for (uint32_t x = 0; x < kBigReads; x++) {
                                to[32 * x] = p[x];
                                to[a.hit_cap + 32 * x] = qq;
                                if (a.n_units > 1) to[2 * a.hit_cap + 32 * x] = u;
                            }
                            from += 32 * kBigReads;
                            to += 32 * kBigReads;
                        }
                        for (uint32_t j = lane; j < left; j += 32, from += 32, to += 32) {
                            to[0] = __ldg(from);
                            to[a.hit_cap] = qq;
                            if (a.n_units > 1) to[2 * a.hit_cap] = u;
                        }
                        more += cc - 1;
                    }
                }
                e0 += 64;
                if (e0 >= n_ent) break;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    rc[k] = 0;
                    if (e0 + 32 * k + lane < n_ent) {
                        rb[k] = ent[e0 + 32 * k + lane];
                        rc[k] = cnt[e0 - 64 + 32 * k + lane];
                        first[k] = __ldg(U->positions + rb[k]);
                    }
                }
            }
        }
      }
    }
    // A batch claimed ahead but not started: the next pass takes it.
    if (next != 0xffffffffu && lane == 0)
        for (uint32_t item = next; item < min(n_items, next + kClaim); item++) defer(item / n_split, item % n_split, 0);
    unsigned long long n_windows = windows;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_windows += __shfl_xor_sync(kFull, n_windows, o);
    // One pair of global atomics a block: every warp's own took longer than the
    // work of a small launch.
    if (lane == 0 && n_windows) atomicAdd(&s_stats[0], n_windows);
    if (lane == 0 && n_raw) atomicAdd(&s_stats[1], (unsigned long long)n_raw);
    __syncthreads();
    if (threadIdx.x < 2 && s_stats[threadIdx.x]) atomicAdd(&a.stats[threadIdx.x], s_stats[threadIdx.x]);
}

__global__ void k_pass_reset(uint32_t* ctl, uint64_t surv_cap) {
    if (threadIdx.x != 0) return;
    unsigned long long* hits = reinterpret_cast<unsigned long long*>(ctl + kCHits);
    unsigned long long* surv = reinterpret_cast<unsigned long long*>(ctl + kCSurv);
    if (*surv > surv_cap) ctl[kCSurvOver] = 1u;   // the previous pass lost survivors
    if (*hits) ctl[kCWorkPasses]++;
    reinterpret_cast<unsigned long long*>(ctl + kCStats)[4] += *surv;   // survivors of the launch
    const uint32_t p = ctl[kCPass] + 1;
    ctl[kCPass] = p;
    ctl[kCRedoN + (p & 1u)] = 0;
    ctl[kCRedoTake] = 0;
    ctl[kCStop] = 0;
    ctl[kCHitNext] = 0;
    ctl[kCFiltNext] = 0;
    *hits = 0;
    *surv = 0;
}

void launch_pass_reset(uint32_t* ctl, uint64_t surv_cap, cudaStream_t st) {
    count_launch();
    k_pass_reset<<<1, 32, 0, st>>>(ctl, surv_cap);
}

void launch_enumerate(const ScreenArgs& a, int sm_count, cudaStream_t st) {
    count_launch();
    // A warp per item at most (those that claim first take several): the idle warps
    // of a full grid took 30 us to claim nothing on a 30 kbp query (938 tiles).
    const int blocks = (int)std::max<uint64_t>(1, umin64(((uint64_t)a.n_items + kEnumWarps - 1) / kEnumWarps, (uint64_t)sm_count * kEnumBlocks));
    if (a.enum_mode == 0) k_enumerate<0><<<blocks, kEnumWarps * 32, 0, st>>>(a);
    else if (a.enum_mode == 1) k_enumerate<1><<<blocks, kEnumWarps * 32, 0, st>>>(a);
    else k_enumerate<2><<<blocks, kEnumWarps * 32, 0, st>>>(a);
}

// ---------------------------------------------------------------------------
// Screen: capped lane-per-hit x-drop over the enumerated hits.
//
// Each idle lane takes the next hit from the pass's hit array and loads one
// 128-position window of the target and of the query around it; from those
// registers it scores the seed footprint and the first 32 columns of both
// sides of extend_hit (src/hsp.rs:98-195) -- the sides are independent and
// are scanned in lockstep.  A side still running after 32 columns continues
// one chunk per iteration with fresh loads while the other lanes take new
// hits.  A hit is extended up to `cap` columns per side:
//  - ended below hspthresh: dropped.  Such a hit can never change the output:
//    search() only records diagonal cover for a hit whose HSP passes
//    (src/seed_search.rs:95-114), so whether it was admitted is irrelevant.
//  - ended at or above hspthresh, or still running at the cap: kept as a
//    candidate for the walk, which applies the diagonal rule in order.
// ---------------------------------------------------------------------------
template <int WARPS, int MINB>
__global__ __launch_bounds__(WARPS * 32, MINB) void k_screen_wide(const __grid_constant__ ScreenArgs a) {
    // Past the buffer's end the pass did not write (those tiles went to the
    // next pass).
    const uint32_t n_hits = (uint32_t)min(*a.hit_count, (unsigned long long)a.hit_cap);
    if (blockIdx.x >= live_blocks(n_hits, WARPS * 32)) return;
    __shared__ int32_t s_lut[16];
    if (threadIdx.x < 16) s_lut[threadIdx.x] = a.sc.sub[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t lt = lanemask_lt();
    const uint32_t L = a.pat.len;
    const int32_t ambig = a.sc.ambig, xdrop = a.sc.xdrop, thresh = a.sc.hspthresh;
    unsigned long long n_cols = 0;
    bool exhausted = false;

    bool busy = false, rdone = true, ldone = true;
    uint32_t ht = 0, hq = 0, hu = 0xffffffffu;
    int32_t seed = 0;
    int32_t rrun = 0, rbest = 0, lrun = 0, lbest = 0;
    uint32_t rbext = 0, lbext = 0, rext = 0, lext = 0, rrem = 0, lrem = 0;
    SeqView T{}, Q{};
    uint32_t cur_unit = 0xffffffffu;

    for (;;) {
        // ---------------- assign ----------------
        const uint32_t im = __ballot_sync(kFull, !busy);
        uint32_t base = 0, take = 0;
        if (!exhausted && im) {
            if (lane == 0) base = atomicAdd(a.hit_next, (uint32_t)__popc(im));
            base = __shfl_sync(kFull, base, 0);
            take = base < n_hits ? min((uint32_t)__popc(im), n_hits - base) : 0u;
            if (base + (uint32_t)__popc(im) >= n_hits) exhausted = true;
        }
        bool fresh = false;
        if (!busy) {
            const uint32_t rk = __popc(im & lt);
            if (rk < take) {
                ht = a.hits[base + rk];
                hq = a.hits[a.hit_cap + base + rk];
                hu = hq == kNoHit ? kNoUnit : (a.n_units > 1 ? a.hits[2 * a.hit_cap + base + rk] : 0u);
                if (hu != kNoUnit && hu != cur_unit) {
                    cur_unit = hu;
                    const UnitDev U = a.units[hu];
                    T = a.tsegs[U.tseg];
                    Q = a.qsegs[U.qseg];
                }
                fresh = hu != kNoUnit;   // an unused slot of a failed reservation
                busy = fresh;
            }
        }
        if (!__any_sync(kFull, busy)) {
            if (exhausted) break;
            continue;
        }

        // ---------------- chunk data ----------------
        // Scan A: a fresh hit's first right chunk, or a continuing side's next chunk.
        // Scan B: a fresh hit's first left chunk.
        uint64_t atc = 0, aqc = 0, btc = 0, bqc = 0;
        uint32_t avv = 0, bvv = 0, an = 0, bn = 0;
        const bool a_right = fresh || !rdone;   // which side scan A advances
        if (fresh) {
            const uint64_t tb = T.base + ht, qb = Q.base + hq;
            const uint64_t tw = (tb - 32) & ~31ull, qw = (qb - 32) & ~31ull;
            uint64_t twc[4], qwc[4];
            uint32_t twv[4], qwv[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                twc[j] = __ldg(T.codes + (tw >> 5) + j);
                qwc[j] = __ldg(Q.codes + (qw >> 5) + j);
                twv[j] = __ldg(T.valid + (tw >> 5) + j);
                qwv[j] = __ldg(Q.valid + (qw >> 5) + j);
            }
            const uint32_t ot = (uint32_t)(tb - tw), oq = (uint32_t)(qb - qw);   // both in [32, 63]
            // Seed footprint: all L columns (src/hsp.rs:119-123).
            {
                const uint64_t tc = win_codes(twc, ot), qc = win_codes(qwc, oq);
                const uint32_t vv = win_bits(twv, ot) & win_bits(qwv, oq);
                int32_t sd = 0;
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    if ((uint32_t)k >= L) break;
                    sd += col_score(tc, qc, vv, k, s_lut, ambig);
                }
                seed = sd;
            }
            rrem = min(T.len - ht - L, Q.len - hq - L);
            lrem = min(ht, hq);
            rrun = rbest = lrun = lbest = 0;
            rbext = lbext = rext = lext = 0;
            rdone = rrem == 0;
            ldone = lrem == 0;
            an = min(32u, rrem);
            atc = win_codes(twc, ot + L);
            aqc = win_codes(qwc, oq + L);
            avv = win_bits(twv, ot + L) & win_bits(qwv, oq + L);
            bn = min(32u, lrem);
            btc = rev_pairs64(win_codes(twc, ot - 32));
            bqc = rev_pairs64(win_codes(qwc, oq - 32));
            bvv = __brev(win_bits(twv, ot - 32) & win_bits(qwv, oq - 32));
        } else if (busy) {
            if (!rdone) {
                const uint64_t tg = T.base + ht + L + rext, qg = Q.base + hq + L + rext;
                atc = load_codes32(T.codes, tg);
                aqc = load_codes32(Q.codes, qg);
                avv = load_bits32(T.valid, tg) & load_bits32(Q.valid, qg);
                an = min(32u, rrem);
            } else {
                // Left side continues below position ht - 1 - lext.
                const uint64_t tg = T.base + ht - lext - 32, qg = Q.base + hq - lext - 32;
                atc = rev_pairs64(load_codes32(T.codes, tg));
                aqc = rev_pairs64(load_codes32(Q.codes, qg));
                avv = __brev(load_bits32(T.valid, tg) & load_bits32(Q.valid, qg));
                an = min(32u, lrem);
            }
        }

        // ---------------- scans ----------------
        {
            if (!busy) an = 0;
            if (!fresh) bn = 0;
            SideScan A, B;
            side_init(A, atc, aqc, avv, an, a_right ? rext : lext, a_right ? rrun : lrun, a_right ? rbest : lbest,
                      a_right ? rbext : lbext);
            side_init(B, btc, bqc, bvv, bn, 0, lrun, lbest, lbext);
            scan_pair_any(A, B, an, bn, xdrop, s_lut, ambig);
            const bool aend = A.brk < an, bend = B.brk < bn;
            const uint32_t aused = aend ? A.brk + 1 : an, bused = bend ? B.brk + 1 : bn;
            n_cols += aused + bused;
            if (busy) {
                if (a_right) {
                    rrun = A.r; rbest = A.b; rbext = A.be; rext += aused; rrem -= aused;
                    rdone = rdone || aend || rrem == 0;
                } else {
                    lrun = A.r; lbest = A.b; lbext = A.be; lext += aused; lrem -= aused;
                    ldone = ldone || aend || lrem == 0;
                }
            }
            if (fresh) {
                lrun = B.r; lbest = B.b; lbext = B.be; lext += bused; lrem -= bused;
                ldone = ldone || bend || lrem == 0;
            }
        }

        // ---------------- bookkeeping ----------------
        bool finish = false, cand = false, is_long = false;
        int32_t score = 0;
        if (busy) {
            if (rdone && ldone) {
                finish = true;
                score = seed + rbest + lbest;
                cand = score >= thresh;
            } else if ((!rdone && rext >= a.cap) || (!ldone && lext >= a.cap)) {
                finish = true;      // still extending at the cap: defer to the walk
                cand = true;
                is_long = true;
            }
        }
        const uint32_t m = __ballot_sync(kFull, finish && cand);
        if (m) {
            uint32_t slot0 = 0;
            if (lane == 0) slot0 = atomicAdd(a.cand_count, (uint32_t)__popc(m));
            slot0 = __shfl_sync(kFull, slot0, 0);
            if (finish && cand) {
                const uint32_t slot = slot0 + __popc(m & lt);
                if (slot < a.cand_cap) {
                    const uint32_t tk = T.key_base + ht, qk = Q.key_base + hq;
                    a.cand_keys[slot] = ((uint64_t)(tk - qk + a.qkey_total) << 32) | tk;
                    a.cand_vals[slot] = slot;
                    Cand c;
                    c.unit = hu; c.t = ht; c.q = hq;
                    c.flags = is_long ? kCandLong : 0u;
                    c.lext = lbext; c.rext = rbext; c.score = score; c.pad_ = 0;
                    a.cands[slot] = c;
                }
            }
        }
        if (finish) busy = false;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_cols += __shfl_xor_sync(kFull, n_cols, o);
    if (lane == 0) atomicAdd(&a.stats[2], n_cols);
}

// ---------------------------------------------------------------------------
// Screen, packed form.  The same lane-per-hit screen as k_screen_wide, with
// the x-drop state of a side packed into two integers:
//     P = 256 * run  + (255 - columns scanned)
//     B = 256 * best + (255 - best extent)
// One column of extend_one_side (src/hsp.rs:179-193) is then
//     P += 256 * score - 1;  B = max(B, P);  break when B - P >= 256 (xdrop + 1)
// and this is exact:
//  - run > best: P exceeds B by at least 1, so B takes P -- best and its
//    extent move together, as in the reference.
//  - run <= best: P < B (a later column has a smaller low byte), so B keeps the
//    first extent that reached the best, as the reference's strict `>` does.
//  - then B - P = 256 (best - run) + d with 1 <= d <= 255, and
//    B - P >= 256 (xdrop + 1)  <=>  best - run > xdrop.
// It needs at most 255 columns per side in the screen (cap <= 192), xdrop in
// [0, 2^22] and |scores| <= 16383, so that no packed value leaves i32; the
// host uses k_screen_wide outside that envelope.
// ---------------------------------------------------------------------------
struct PkSide {
    uint64_t e, o;         // nibble j of e: column 2j, of o: column 2j+1; nibble = q << 2 | t
    uint32_t vv;           // column validity
    uint32_t n;            // columns present in this chunk
    int32_t p, b;          // packed run and best
};

// A side with no columns starts dead (b - p = T) so that no column moves it.
__device__ __forceinline__ void pk_init(PkSide& S, uint64_t tc, uint64_t qc, uint32_t vv, uint32_t n, int32_t p,
                                        int32_t b, int32_t T) {
    constexpr uint64_t m = 0x3333333333333333ull;
    S.e = (tc & m) | ((qc << 2) & ~m);
    S.o = ((tc >> 2) & m) | (qc & ~m);
    S.vv = vv;
    S.n = n;
    S.b = b;
    S.p = n ? p : b - T;
}

// Column k of a side, branch-free.  A side is alive while b - p < T; once the
// x-drop break fires its later columns add 0, so p and b (and b - p >= T)
// stay as the break left them.  kSlow: the chunk may hold invalid bases
// (scored `ambig`) or end before column 32 (absent columns add 0 and keep
// the side alive).  plut is indexed by (q << 2) | t.
template <bool kSlow, int k>
__device__ __forceinline__ void pk_step(PkSide& S, int32_t T, const int32_t* plut, int32_t pamb) {
    const uint32_t idx = (uint32_t)(((k & 1) ? S.o : S.e) >> (4 * (k >> 1))) & 15u;
    int32_t s = plut[idx];
    bool go = S.b - S.p < T;
    if (kSlow) {
        s = ((S.vv >> k) & 1u) ? s : pamb;
        go = go && (uint32_t)k < S.n;
    }
    s = go ? s : 0;
    S.p += s;
    S.b = max(S.b, S.p);
}

// Both sides column by column in lockstep: two independent serial chains.
template <bool kSlow>
__device__ __forceinline__ void pk_scan_pair(PkSide& A, PkSide& B, int32_t T, const int32_t* plut, int32_t pamb) {
#define GXY_PK4(g)                                                         \
    pk_step<kSlow, g * 4 + 0>(A, T, plut, pamb);                           \
    pk_step<kSlow, g * 4 + 0>(B, T, plut, pamb);                           \
    pk_step<kSlow, g * 4 + 1>(A, T, plut, pamb);                           \
    pk_step<kSlow, g * 4 + 1>(B, T, plut, pamb);                           \
    pk_step<kSlow, g * 4 + 2>(A, T, plut, pamb);                           \
    pk_step<kSlow, g * 4 + 2>(B, T, plut, pamb);                           \
    pk_step<kSlow, g * 4 + 3>(A, T, plut, pamb);                           \
    pk_step<kSlow, g * 4 + 3>(B, T, plut, pamb);
    GXY_PK4(0) GXY_PK4(1) GXY_PK4(2) GXY_PK4(3) GXY_PK4(4) GXY_PK4(5) GXY_PK4(6) GXY_PK4(7)
#undef GXY_PK4
}

__device__ __forceinline__ int32_t pk_run(int32_t p) { return p >> 8; }            // arithmetic shift
__device__ __forceinline__ uint32_t pk_ext(int32_t p) { return 255u - ((uint32_t)p & 255u); }
constexpr int32_t kPkStart = 255;   // run 0, no columns

// 64 bits from the 128-bit pair (hi:lo) starting at bit s (0 <= s < 64).
__device__ __forceinline__ uint64_t funnel64(uint64_t lo, uint64_t hi, uint32_t s) {
    return s ? ((lo >> s) | (hi << (64 - s))) : lo;
}

// Seed footprint score, all L columns at t / q (src/hsp.rs:119-123): two
// columns per table read, an odd last one singly, invalid columns re-scored ambig.
__device__ __forceinline__ int32_t seed_score(const SeqView& T, const SeqView& Q, uint32_t t, uint32_t q,
                                              uint32_t L, uint32_t seed_mask, const int32_t* s_duo,
                                              const int32_t* s_lut, int32_t ambig) {
    const uint64_t tc = load_codes32(T.codes, T.base + t), qc = load_codes32(Q.codes, Q.base + q);
    const uint32_t vv = load_bits32(T.valid, T.base + t) & load_bits32(Q.valid, Q.base + q);
    int32_t sd = 0;
#pragma unroll
    for (int k = 0; k < 32; k += 2) {
        if ((uint32_t)k + 2 > L) break;
        sd += s_duo[((((uint32_t)(tc >> (2 * k))) & 15u) << 4) | ((uint32_t)(qc >> (2 * k)) & 15u)];
    }
    for (uint32_t k = L & ~1u; k < L; k++)
        sd += s_lut[((((uint32_t)(tc >> (2 * k))) & 3u) << 2) | ((uint32_t)(qc >> (2 * k)) & 3u)];
    uint32_t bad = ~vv & seed_mask;
    while (bad) {
        const uint32_t k = __ffs(bad) - 1;
        bad &= bad - 1;
        sd += ambig - s_lut[((((uint32_t)(tc >> (2 * k))) & 3u) << 2) | ((uint32_t)(qc >> (2 * k)) & 3u)];
    }
    return sd;
}

template <int WARPS, int MINB>
__global__ __launch_bounds__(WARPS * 32, MINB) void k_screen(const __grid_constant__ ScreenArgs a) {
    // Past the buffer's end the pass did not write (those hits went to the
    // next pass, or were lost with a survivor overflow, which reruns the launch).
    const uint32_t n_hits = (uint32_t)min(*a.hit_count, (unsigned long long)a.hit_cap);
    const uint32_t n_blocks = live_blocks(n_hits, WARPS * 32);
    if (blockIdx.x >= n_blocks) return;
    __shared__ int32_t s_lut[16];     // raw column scores, index (t << 2) | q
    __shared__ int32_t s_plut[16];    // 256 * score - 1, index (q << 2) | t
    __shared__ int32_t s_duo[256];    // sum of two columns' scores, index (t2 << 4) | q2
    for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x)
        s_duo[i] = a.sc.sub[((i >> 4 & 3u) << 2) | (i & 3u)] + a.sc.sub[((i >> 6 & 3u) << 2) | (i >> 2 & 3u)];
    if (threadIdx.x < 16) {
        s_lut[threadIdx.x] = a.sc.sub[threadIdx.x];
        s_plut[threadIdx.x] = a.sc.sub[((threadIdx.x & 3u) << 2) | (threadIdx.x >> 2)] * 256 - 1;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t lt = lanemask_lt();
    const uint32_t L = a.pat.len;
    const int32_t ambig = a.sc.ambig, thresh = a.sc.hspthresh;
    const int32_t pamb = ambig * 256 - 1;
    const int32_t T = (a.sc.xdrop + 1) * 256;
    const uint32_t seed_mask = L >= 32 ? 0xffffffffu : ((1u << L) - 1u);
    // No seed footprint scores above this: a hit whose two sides' bests stay
    // below thresh - seed_ub can never pass, whatever its seed scores.
    int32_t top = ambig;
    for (int i = 0; i < 16; i++) top = max(top, a.sc.sub[i]);
    const int32_t seed_ub = top * (int32_t)L;
    // Each warp claims hits in chunks (one atomic per chunk) and deals them
    // to its idle lanes; chunks shrink for small launches so that every warp
    // still gets work.
    const uint32_t n_warps = n_blocks * WARPS;
    const uint32_t chunk = max(32u, min(256u, n_hits / max(1u, n_warps * 8u)));
    uint32_t wcur = 0, wend = 0;   // this warp's claimed, not yet dealt hits
    uint32_t n_cols = 0;
    unsigned long long n_cols_all = 0;
    bool exhausted = false;

    bool busy = false, rdone = true, ldone = true;
    uint32_t ht = 0, hq = 0, hu = 0xffffffffu;
    int32_t rp = kPkStart, rb = kPkStart, lp = kPkStart, lb = kPkStart;
    uint32_t rrem = 0, lrem = 0;
    SeqView T_{}, Q_{};
    uint32_t cur_unit = 0xffffffffu;

    for (;;) {
        // ---------------- assign ----------------
        const uint32_t im = __ballot_sync(kFull, !busy);
        const uint32_t need = __popc(im);
        const uint32_t avail = wend - wcur;
        uint32_t nb = 0, ncount = 0;
        if (need > avail && !exhausted) {
            if (lane == 0) nb = atomicAdd(a.hit_next, chunk);
            nb = __shfl_sync(kFull, nb, 0);
            ncount = nb < n_hits ? min(chunk, n_hits - nb) : 0u;
            if (nb + chunk >= n_hits) exhausted = true;
        }
        bool fresh = false;
        if (!busy) {
            const uint32_t rk = __popc(im & lt);
            uint32_t hidx = 0xffffffffu;
            if (rk < avail) hidx = wcur + rk;
            else if (rk - avail < ncount) hidx = nb + (rk - avail);
            if (hidx != 0xffffffffu) {
                ht = a.hits[hidx];
                hq = a.hits[a.hit_cap + hidx];
                hu = hq == kNoHit ? kNoUnit : (a.n_units > 1 ? a.hits[2 * a.hit_cap + hidx] : 0u);
                if (hu != kNoUnit && hu != cur_unit) {
                    cur_unit = hu;
                    const UnitDev U = a.units[hu];
                    T_ = a.tsegs[U.tseg];
                    Q_ = a.qsegs[U.qseg];
                }
                fresh = hu != kNoUnit;   // an unused slot of a failed reservation
                busy = fresh;
            }
        }
        {
            const uint32_t from_old = min(need, avail);
            if (ncount) {
                wcur = nb + min(need - from_old, ncount);
                wend = nb + ncount;
            } else {
                wcur += from_old;
            }
        }
        if (!__any_sync(kFull, busy)) {
            if (exhausted && wcur == wend) break;
            continue;
        }

        // ---------------- chunk data ----------------
        // The next chunk of each side that still runs: A right, forward from the
        // column after the last one scanned, B left, the 32 positions below it,
        // reversed.
        uint64_t atc = 0, aqc = 0, btc = 0, bqc = 0;
        uint32_t avv = 0, bvv = 0, an = 0, bn = 0;
        if (fresh) {
            rrem = min(T_.len - ht - L, Q_.len - hq - L);
            lrem = min(ht, hq);
            rp = rb = lp = lb = kPkStart;
            rdone = rrem == 0;
            ldone = lrem == 0;
        }
        if (busy && !rdone) {
            const uint32_t ext = pk_ext(rp);
            const uint64_t ta = T_.base + ht + L + ext, qa = Q_.base + hq + L + ext;
            atc = load_codes32(T_.codes, ta);
            aqc = load_codes32(Q_.codes, qa);
            avv = load_bits32(T_.valid, ta) & load_bits32(Q_.valid, qa);
            an = min(32u, rrem);
        }
        if (busy && !ldone) {
            const uint32_t ext = pk_ext(lp);
            const uint64_t tb = T_.base + ht - ext - 32, qb = Q_.base + hq - ext - 32;
            btc = rev_pairs64(load_codes32(T_.codes, tb));
            bqc = rev_pairs64(load_codes32(Q_.codes, qb));
            bvv = __brev(load_bits32(T_.valid, tb) & load_bits32(Q_.valid, qb));
            bn = min(32u, lrem);
        }

        // ---------------- scans ----------------
        {
            PkSide A, B;
            pk_init(A, atc, aqc, avv, an, rp, rb, T);
            pk_init(B, btc, bqc, bvv, bn, lp, lb, T);
            const bool slow = (an != 0 && (an < 32 || avv != 0xffffffffu)) ||
                              (bn != 0 && (bn < 32 || bvv != 0xffffffffu));
            if (__any_sync(kFull, slow)) pk_scan_pair<true>(A, B, T, s_plut, pamb);
            else pk_scan_pair<false>(A, B, T, s_plut, pamb);
            if (an) {
                const uint32_t used = ((uint32_t)rp & 255u) - ((uint32_t)A.p & 255u);
                const bool end = A.b - A.p >= T;
                n_cols += used;
                rp = A.p; rb = A.b; rrem -= used;
                rdone = end || rrem == 0;
            }
            if (bn) {
                const uint32_t used = ((uint32_t)lp & 255u) - ((uint32_t)B.p & 255u);
                const bool end = B.b - B.p >= T;
                n_cols += used;
                lp = B.p; lb = B.b; lrem -= used;
                ldone = end || lrem == 0;
            }
        }
        if (n_cols >= (1u << 30)) {
            n_cols_all += n_cols;
            n_cols = 0;
        }

        // ---------------- bookkeeping ----------------
        bool finish = false, cand = false, is_long = false;
        int32_t score = 0;
        if (busy) {
            if (rdone && ldone) {
                finish = true;
                score = pk_run(rb) + pk_run(lb);
                cand = score >= thresh - seed_ub;   // else the seed cannot lift it to thresh
            } else if ((!rdone && pk_ext(rp) >= a.cap) || (!ldone && pk_ext(lp) >= a.cap)) {
                finish = true;      // still extending at the cap: defer to the walk
                cand = true;
                is_long = true;
            }
        }
        if (__any_sync(kFull, finish && cand && !is_long)) {
            if (finish && cand && !is_long) {
                score += seed_score(T_, Q_, ht, hq, L, seed_mask, s_duo, s_lut, ambig);
                cand = score >= thresh;
            }
        }
        const uint32_t m = __ballot_sync(kFull, finish && cand);
        if (m) {
            uint32_t slot0 = 0;
            if (lane == 0) slot0 = atomicAdd(a.cand_count, (uint32_t)__popc(m));
            slot0 = __shfl_sync(kFull, slot0, 0);
            if (finish && cand) {
                const uint32_t slot = slot0 + __popc(m & lt);
                if (slot < a.cand_cap) {
                    const uint32_t tk = T_.key_base + ht, qk = Q_.key_base + hq;
                    a.cand_keys[slot] = ((uint64_t)(tk - qk + a.qkey_total) << 32) | tk;
                    a.cand_vals[slot] = slot;
                    Cand c;
                    c.unit = hu; c.t = ht; c.q = hq;
                    c.flags = is_long ? kCandLong : 0u;
                    c.lext = pk_ext(lb); c.rext = pk_ext(rb); c.score = is_long ? 0 : score; c.pad_ = 0;
                    a.cands[slot] = c;
                }
            }
        }
        if (finish) busy = false;
    }
    n_cols_all += n_cols;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_cols_all += __shfl_xor_sync(kFull, n_cols_all, o);
    if (lane == 0) atomicAdd(&a.stats[2], n_cols_all);
}

// The packed screen's envelope (see above).
static bool packed_ok(const ScreenArgs& a) {
    int64_t m = a.sc.ambig < 0 ? -(int64_t)a.sc.ambig : a.sc.ambig;
    for (int i = 0; i < 16; i++) m = std::max<int64_t>(m, a.sc.sub[i] < 0 ? -(int64_t)a.sc.sub[i] : a.sc.sub[i]);
    return a.cap <= 192 && m <= 16383 && a.sc.xdrop >= 0 && a.sc.xdrop <= (1 << 22);
}

void launch_screen(const ScreenArgs& a, int warps, int per_sm, int blocks, cudaStream_t st) {
    // For 8-warp blocks the register budget follows the requested blocks per SM
    // (2: 128, 3: 85, 4: 64 registers).
    count_launch();
    if (packed_ok(a)) {
        switch (warps) {
            case 4: k_screen<4, 4><<<blocks, 128, 0, st>>>(a); break;
            case 16: k_screen<16, 1><<<blocks, 512, 0, st>>>(a); break;
            default:
                if (per_sm >= 4) k_screen<8, 4><<<blocks, 256, 0, st>>>(a);
                else if (per_sm == 3) k_screen<8, 3><<<blocks, 256, 0, st>>>(a);
                else k_screen<8, 2><<<blocks, 256, 0, st>>>(a);
                break;
        }
        return;
    }
    switch (warps) {
        case 4: k_screen_wide<4, 4><<<blocks, 128, 0, st>>>(a); break;
        case 16: k_screen_wide<16, 1><<<blocks, 512, 0, st>>>(a); break;
        default:
            if (per_sm >= 4) k_screen_wide<8, 4><<<blocks, 256, 0, st>>>(a);
            else if (per_sm == 3) k_screen_wide<8, 3><<<blocks, 256, 0, st>>>(a);
            else k_screen_wide<8, 2><<<blocks, 256, 0, st>>>(a);
            break;
    }
}

// ---------------------------------------------------------------------------
// Walk: diagonal suppression over the sorted candidates.
//
// Along one diagonal the reference visits hits in ascending t (query windows
// ascend, and one window meets a diagonal once).  A hit is admitted iff
// t >= cover, cover being the t_end of the last HSP emitted on the diagonal
// (src/diag_hash.rs:34-53); only a passing HSP moves cover.  The walk replays
// exactly that over the candidates of one (unit, diagonal) segment, which
// are the only hits that can pass.  Deferred (long) candidates are extended
// in full here with the warp x-drop when they are admitted.
// ---------------------------------------------------------------------------
// Entropy gate (src/entropy.rs:27-67) over target [ts, te), one warp, f64.
__device__ bool entropy_gate_warp(const SeqView& T, uint32_t ts, uint32_t te, int32_t score, int32_t thr) {
    const int lane = threadIdx.x & 31;
    const uint32_t e = min(te, T.len);
    uint32_t cnt[4] = {0, 0, 0, 0};
    for (uint32_t p = ts + 32 * lane; p < e; p += 32 * 32) {
        const uint64_t c = load_codes32(T.codes, T.base + p);
        uint32_t v = load_bits32(T.valid, T.base + p);
        const uint32_t nn = min(32u, e - p);
        if (nn < 32) v &= (1u << nn) - 1;
        // Split codes into low/high bit planes and count each code.
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int k = 0; k < 32; k++) {
            lo |= (uint32_t)((c >> (2 * k)) & 1u) << k;
            hi |= (uint32_t)((c >> (2 * k + 1)) & 1u) << k;
        }
        cnt[0] += __popc(v & ~hi & ~lo);
        cnt[1] += __popc(v & ~hi & lo);
        cnt[2] += __popc(v & hi & ~lo);
        cnt[3] += __popc(v & hi & lo);
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt[k] += __shfl_xor_sync(kFull, cnt[k], o);
    const uint32_t total = cnt[0] + cnt[1] + cnt[2] + cnt[3];
    double h = 0.0;
    if (total) {
        const double tt = (double)total;
        for (int k = 0; k < 4; k++) {
            if (cnt[k] == 0) continue;
            const double p = (double)cnt[k] / tt;
            h -= p * log2(p);
        }
    }
    const double scaled = (double)score * (h / 2.0);
    return scaled >= (double)thr;
}

template <int WARPS>
__global__ __launch_bounds__(WARPS * 32) void k_walk(const __grid_constant__ WalkArgs a) {
    const uint32_t n = min(*a.n_dev, a.n_cap), n_blocks = live_blocks(n, 32);
    if (blockIdx.x >= n_blocks || *a.gave_up) return;
    __shared__ int32_t s_lut[16];
    __shared__ WarpStage s_stage[WARPS];
    if (threadIdx.x < 16) s_lut[threadIdx.x] = a.sc.sub[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t L = a.seed_len;
    // Chunks of sorted positions are claimed dynamically: a segment with
    // long candidates (full re-extension) can take far longer than the rest.  A
    // chunk is 32 positions where that leaves every warp four of them, and down to
    // one position in a small launch, whose time is that of the warp with the most
    // segments.
    const uint32_t chunk = max(1u, min(32u, n / (n_blocks * WARPS * 4u)));
    for (;;) {
        uint32_t r = 0;
        if (lane == 0) r = atomicAdd(a.chunk_next, 1u);
        r = __shfl_sync(kFull, r, 0);
        if ((uint64_t)r * chunk >= n) break;
        const uint32_t i = r * chunk + lane;
        bool head = false;
        uint32_t key_hi = 0;
        if (i < n && (uint32_t)lane < chunk) {
            key_hi = (uint32_t)(a.keys[i] >> 32);
            head = (i == 0) || (key_hi != (uint32_t)(a.keys[i - 1] >> 32));
        }
        // A diagonal segment of one candidate needs no walk: nothing can
        // cover it, so it is kept when it passes.  Its own lane settles it
        // when its extension is already exact (not a long candidate, and no
        // entropy gate, which takes the whole warp).
        bool alone = false;
        if (head && !a.has_entropy) {
            const bool tail = (i + 1 >= n) || (key_hi != (uint32_t)(a.keys[i + 1] >> 32));
            if (tail) {
                const Cand c = a.cands[a.idx[i]];
                if (!(c.flags & kCandLong)) {
                    alone = true;
                    if (c.score >= a.sc.hspthresh) {
                        const UnitDev U = a.units[c.unit];
                        const uint32_t ts = c.t - c.lext, len = a.seed_len + c.lext + c.rext;
                        Hsp o;
                        o.t_start = ts; o.q_start = c.q - c.lext; o.length = len; o.score = c.score;
                        a.out_hsp[i] = o;
                        a.out_flag[i] = (U.primary_hi <= U.primary_lo || (ts >= U.primary_lo && ts < U.primary_hi))
                                            ? 1 : 0;
                    }
                }
            }
        }
        uint32_t hb = __ballot_sync(kFull, head && !alone);
        while (hb) {
            const uint32_t h = r * chunk + (uint32_t)(__ffs(hb) - 1);
            hb &= hb - 1;
            const uint32_t segkey = (uint32_t)(a.keys[h] >> 32);
            // A segment (one diagonal key) can hold the candidates of several
            // units that share a target segment, interleaved in t.  Each unit
            // is walked by its own pass with its own cover: first the unit of
            // the segment's first candidate (u0), then the other units in
            // ascending order -- those above u0, then those below it.  Each
            // pass finds the next unit as the smallest one above the current
            // one (and below `ceil`); a segment of one unit takes one pass.
            const uint32_t u0 = a.cands[a.idx[h]].unit;
            uint32_t cur_unit = u0, ceil = 0xffffffffu, below = 0xffffffffu;
            for (;;) {
            uint32_t j = h;
            uint32_t cover = 0;
            uint32_t next = 0xffffffffu;
            for (;;) {
                const uint32_t jj = j + lane;
                const bool inseg = jj < n && (uint32_t)(a.keys[jj] >> 32) == segkey;
                Cand c;
                c.unit = 0xffffffffu; c.t = 0;
                if (inseg) c = a.cands[a.idx[jj]];
                const uint32_t be = __ballot_sync(kFull, !inseg);
                const uint32_t stop = be ? (uint32_t)(__ffs(be) - 1) : 32u;
                // The candidates of these 32 positions that cover admits, one by one.
                for (uint32_t from = 0;;) {
                    const bool elig = inseg && c.unit == cur_unit && c.t >= cover && (uint32_t)lane >= from;
                    const uint32_t bc = __ballot_sync(kFull, elig);
                    const uint32_t first = bc ? (uint32_t)(__ffs(bc) - 1) : 32u;
                    // Other units among the positions this step passes over.
                    if (a.n_units > 1) {
                        const uint32_t upto = min(first, stop);
                        const bool seen = (uint32_t)lane <= upto && inseg;
                        next = min(next, __reduce_min_sync(kFull, (seen && c.unit > cur_unit && c.unit < ceil)
                                                                      ? c.unit : 0xffffffffu));
                        below = min(below, __reduce_min_sync(kFull, (seen && c.unit < u0) ? c.unit : 0xffffffffu));
                    }
                    if (first >= stop) break;
                    const uint32_t unit = cur_unit;
                    const uint32_t t = __shfl_sync(kFull, c.t, first);
                    const uint32_t q = __shfl_sync(kFull, c.q, first);
                    const uint32_t flags = __shfl_sync(kFull, c.flags, first);
                    int32_t score = __shfl_sync(kFull, c.score, first);
                    uint32_t lext = __shfl_sync(kFull, c.lext, first);
                    uint32_t rext = __shfl_sync(kFull, c.rext, first);
                    const UnitDev U = a.units[unit];
                    const SeqView T = a.tsegs[U.tseg];
                    if (flags & kCandLong) {
                        const SeqView Q = a.qsegs[U.qseg];
                        const LaneExt r = extend_warp(T, Q, t, q, L, a.sc.xdrop, s_lut, a.sc.ambig, &s_stage[w]);
                        score = r.score;
                        lext = r.lext;
                        rext = r.rext;
                    }
                    bool pass = score >= a.sc.hspthresh;
                    const uint32_t ts = t - lext, len = L + lext + rext;
                    if (pass && a.has_entropy) pass = entropy_gate_warp(T, ts, ts + len, score, a.entropy_thr);
                    if (pass) {
                        cover = ts + len;   // mark_covered(t_end) (src/diag_hash.rs:43-53)
                        if (lane == 0) {
                            const bool keep = U.primary_hi <= U.primary_lo ||
                                              (ts >= U.primary_lo && ts < U.primary_hi);
                            const uint32_t pos = j + first;
                            Hsp o;
                            o.t_start = ts; o.q_start = q - lext; o.length = len; o.score = score;
                            a.out_hsp[pos] = o;
                            a.out_flag[pos] = keep ? 1 : 0;
                        }
                    }
                    from = first + 1;
                }
                if (stop < 32) break;
                j += 32;
                if (a.n_units == 1) {
                    // Past the 32-position steps whose last key is still covered (with several
                    // units every position is looked at: another one may hide there).
                    const uint64_t uncovered = (uint64_t)segkey << 32 | (a.tsegs[a.units[0].tseg].key_base + cover);
                    uint32_t skip = 32;
                    while (skip == 32) {
                        const uint64_t last = (uint64_t)j + 32u * (uint32_t)lane + 31;
                        const uint32_t go = __ballot_sync(kFull, last >= n || a.keys[last] >= uncovered);
                        skip = go ? (uint32_t)(__ffs(go) - 1) : 32u;
                        j += 32 * skip;
                    }
                }
            }
            if (next != 0xffffffffu) {
                cur_unit = next;                      // the next unit above
            } else if (ceil == 0xffffffffu && below != 0xffffffffu) {
                cur_unit = below;                     // then the units below u0, ascending
                ceil = u0;
            } else {
                break;
            }
            }
        }
    }
}

void launch_walk(const WalkArgs& a, int warps, int blocks, cudaStream_t st) {
    switch (warps) {
        case 4: count_launch(); k_walk<4><<<blocks, 128, 0, st>>>(a); break;
        default: count_launch(); k_walk<8><<<blocks, 256, 0, st>>>(a); break;
    }
}

// ---------------------------------------------------------------------------
// Driver records: global coordinates, per-group order and dedup
// (build_ungapped_record src/driver.rs:437-468; sort and dedup_by :371-391).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t shl64(uint64_t x, int s) { return s >= 64 ? 0ull : x << s; }

__global__ void k_record_keys(const Hsp* hsp, const uint32_t* unit, const Place* place, const uint32_t* perm,
                              const uint32_t* n_dev, uint32_t n_cap, int mode, int sh_g, int sh_t, int sh_q,
                              uint64_t* key, uint32_t* val, const uint32_t* gave_up) {
    if (*gave_up) return;
    const uint32_t n = min(*n_dev, n_cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t p = perm ? perm[i] : i;
        const Hsp h = hsp[p];
        const Place pl = place[unit[p]];
        const uint32_t t = h.t_start + pl.t_offset;
        uint64_t k;
        if (mode == 0)
            k = shl64(pl.group, sh_g) | shl64(t, sh_t) | shl64(h.q_start, sh_q) | h.length;
        else if (mode == 1)
            k = ((uint64_t)h.q_start << 32) | h.length;
        else
            k = ((uint64_t)pl.group << 32) | t;
        key[i] = k;
        val[i] = p;
    }
}

void launch_record_keys(const Hsp* hsp, const uint32_t* unit, const Place* place, const uint32_t* perm,
                        const uint32_t* n_dev, uint32_t n_cap, int mode, int sh_g, int sh_t, int sh_q, uint64_t* key,
                        uint32_t* val, const uint32_t* gave_up, int blocks, cudaStream_t st) {
    count_launch();
    k_record_keys<<<blocks, 256, 0, st>>>(hsp, unit, place, perm, n_dev, n_cap, mode, sh_g, sh_t, sh_q, key, val,
                                            gave_up);
}

__device__ __forceinline__ Record make_record(const Hsp* hsp, const uint32_t* unit, const Place* place,
                                              uint32_t p) {
    const Hsp h = hsp[p];
    const uint32_t u = unit[p];
    const Place pl = place[u];
    Record r;
    r.group = pl.group;
    r.t_start = h.t_start + pl.t_offset;
    r.q_start = h.q_start;
    r.span = h.length;
    r.score = h.score;
    r.unit = u;
    return r;
}

__global__ void k_record_heads(const Hsp* hsp, const uint32_t* unit, const Place* place, const uint32_t* perm,
                               const uint32_t* n_dev, uint32_t n_cap, uint8_t* flag, const uint32_t* gave_up) {
    if (*gave_up) return;
    const uint32_t n = min(*n_dev, n_cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint8_t head = 1;
        if (i > 0) {
            const Record a = make_record(hsp, unit, place, perm[i - 1]);
            const Record b = make_record(hsp, unit, place, perm[i]);
            head = (a.group != b.group || a.t_start != b.t_start || a.q_start != b.q_start || a.span != b.span);
        }
        flag[i] = head;
    }
}

void launch_record_heads(const Hsp* hsp, const uint32_t* unit, const Place* place, const uint32_t* perm,
                         const uint32_t* n_dev, uint32_t n_cap, uint8_t* flag, const uint32_t* gave_up, int blocks,
                         cudaStream_t st) {
    count_launch();
    k_record_heads<<<blocks, 256, 0, st>>>(hsp, unit, place, perm, n_dev, n_cap, flag, gave_up);
}

__global__ void k_record_emit(const Hsp* hsp, const uint32_t* unit, const Place* place, const uint32_t* perm,
                              const uint8_t* flag, const uint32_t* offsets, const uint32_t* n_dev, uint32_t n_cap,
                              Record* out, const uint32_t* gave_up) {
    if (*gave_up) return;
    const uint32_t n = min(*n_dev, n_cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (flag[i]) out[offsets[i]] = make_record(hsp, unit, place, perm[i]);
}

void launch_record_emit(const Hsp* hsp, const uint32_t* unit, const Place* place, const uint32_t* perm,
                        const uint8_t* flag, const uint32_t* offsets, const uint32_t* n_dev, uint32_t n_cap,
                        Record* out, const uint32_t* gave_up, int blocks, cudaStream_t st) {
    count_launch();
    k_record_emit<<<blocks, 256, 0, st>>>(hsp, unit, place, perm, flag, offsets, n_dev, n_cap, out,
                                            gave_up);
}

// ---------------------------------------------------------------------------
// x-drop of given hits (extend_hit, src/hsp.rs:66-148): mode 0 one lane per
// hit (uncapped), mode 1 one warp per hit.
// ---------------------------------------------------------------------------
__global__ void k_extend_lane(SeqView T, SeqView Q, Score sc, const uint32_t* tp, const uint32_t* qp, uint64_t n,
                              uint32_t L, Hsp* out, uint8_t* ok) {
    __shared__ int32_t s_lut[16];
    if (threadIdx.x < 16) s_lut[threadIdx.x] = sc.sub[threadIdx.x];
    __syncthreads();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t t = tp[i], q = qp[i];
        if ((uint64_t)t + L > T.len || (uint64_t)q + L > Q.len) {   // src/hsp.rs:113-115
            ok[i] = 0;
            continue;
        }
        const LaneExt r = extend_lane(T, Q, t, q, L, 0xffffffffu, sc.xdrop, s_lut, sc.ambig);
        const bool pass = r.score >= sc.hspthresh;
        ok[i] = pass ? 1 : 0;
        Hsp o;
        o.t_start = t - r.lext; o.q_start = q - r.lext; o.length = L + r.lext + r.rext; o.score = r.score;
        out[i] = o;
    }
}

__global__ void k_extend_warp(SeqView T, SeqView Q, Score sc, const uint32_t* tp, const uint32_t* qp, uint64_t n,
                              uint32_t L, Hsp* out, uint8_t* ok) {
    __shared__ int32_t s_lut[16];
    __shared__ WarpStage s_stage[8];
    if (threadIdx.x < 16) s_lut[threadIdx.x] = sc.sub[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint64_t i = blockIdx.x * 8ull + w; i < n; i += (uint64_t)gridDim.x * 8) {
        const uint32_t t = tp[i], q = qp[i];
        if ((uint64_t)t + L > T.len || (uint64_t)q + L > Q.len) {
            if (lane == 0) ok[i] = 0;
            continue;
        }
        const LaneExt r = extend_warp(T, Q, t, q, L, sc.xdrop, s_lut, sc.ambig, &s_stage[w]);
        if (lane == 0) {
            ok[i] = r.score >= sc.hspthresh ? 1 : 0;
            Hsp o;
            o.t_start = t - r.lext; o.q_start = q - r.lext; o.length = L + r.lext + r.rext; o.score = r.score;
            out[i] = o;
        }
    }
}

void launch_extend_hits(SeqView T, SeqView Q, Score sc, const uint32_t* tpos, const uint32_t* qpos, uint64_t n,
                        uint32_t seed_len, uint32_t mode, Hsp* out, uint8_t* ok, cudaStream_t st) {
    if (!n) return;
    if (mode == 1) {
        const int blocks = (int)umin64((n + 7) / 8, 148 * 8);
        count_launch();
        k_extend_warp<<<blocks, 256, 0, st>>>(T, Q, sc, tpos, qpos, n, seed_len, out, ok);
    } else {
        const int blocks = (int)umin64((n + 255) / 256, 148 * 8);
        count_launch();
        k_extend_lane<<<blocks, 256, 0, st>>>(T, Q, sc, tpos, qpos, n, seed_len, out, ok);
    }
}

}  // namespace gxy
