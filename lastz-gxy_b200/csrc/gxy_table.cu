// gxy_table.cu -- PosTable::build (src/pos_table.rs:35-83) on the device, for
// one view of a sequence or for many views at once (the driver's chunk
// tables, src/driver.rs:156-210).
//
// The reference counts every seedable window's word, scans the counts into
// bucket starts and drops the positions into their buckets in ascending order
// through per-word cursors (src/pos_table.rs:42-75).  Here the views share
// one bucket space, view v's word w being bucket g = v * 4^w + w:
//
// Weights 6 to 13 (kPartBuckets and more words, at most kMaxParts partitions of
// kPartBuckets a view), from kMinParts partitions in all on, are built by
// partition, a group of views at a time:
//
//  1. k_part_count: every block counts its share of the windows by partition, in
//     shared memory;  k_part_prefix and a scan turn the counts into every block's
//     first slot in every partition;
//  2. k_part_scatter writes each window's position and low word bits to its slot;
//  3. k_part_build, a block a partition: counts, starts, occupancy, packed bounds
//     and the positions of its 4,096 buckets in shared memory, buckets of up to 8
//     positions put in order there, all written once and in order.
//
// What bounds it: the scattered 8-byte writes of step 2 (73 us for a 10 Mbp target),
// in step 3 the instructions for the buckets, empty or not (47 us for 16.7 M of
// them, 88 us with a 10 Mbp target's positions); step 1 takes 26 us.  Bucket by bucket the same
// table took 256 us (random atomics on 64 MB of counts, twice, a three-pass scan
// and a copy of them), an all but empty one 95 us against 63.  Three and four
// blocks an SM instead of two spill step 3's registers: 103 and 117 us.
//
// The others, bucket by bucket:
//
//  1. k_count_words counts the windows of every bucket (atomics on an array
//     that stays in L2 for a chromosome-sized view);
//  2. one exclusive scan turns the counts into global bucket starts, and
//     leaves a copy in the counts array: the cursors;
//  3. k_fill_buckets drops every window's position into its bucket through
//     an atomic cursor -- in an arbitrary order inside the bucket;
//  4. k_sort_small_buckets writes the occupancy bitmap and orders every
//     bucket of 2 or 3 positions on the spot, k_sort_warp_buckets those up to
//     32 a warp each, k_sort_block_buckets those up to kBlockBucket in shared
//     memory, and the radix sort the few larger ones, so every bucket holds
//     the reference's order when the build returns.
//
// View v's table is a window onto the shared arrays: its starts are the
// global starts g = v * 4^w .. v * 4^w + 4^w (global indices into the shared
// positions array, which the searches use as they are; the download
// subtracts the view's first index), and its occupancy bitmap is the shared
// bitmap's words from v * 4^w / 32 on.
#include "gxy_engine.cuh"
#include "gxy_kernels.cuh"
#include "gxy_radix.cuh"

#include <algorithm>
#include <vector>

namespace gxy {

namespace {

constexpr uint32_t kBlockBucket = 4096;   // the largest bucket sorted in shared memory

// Each thread takes four windows at a time (stride apart, so a warp's loads
// stay coalesced): four independent word loads and atomics in flight instead
// of one dependent chain per window.
__global__ void k_count_words(SeqView view, Pattern pat, uint32_t step, uint32_t nwin, uint32_t* counts) {
    const uint32_t S = gridDim.x * blockDim.x;
    for (uint32_t k0 = blockIdx.x * blockDim.x + threadIdx.x; k0 < nwin; k0 += 4 * S) {
        uint32_t w[4];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t k = k0 + u * S;
            ok[u] = k < nwin && word_at(view, pat, k * step, w[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (ok[u]) atomicAdd(&counts[w[u]], 1u);
    }
}

__global__ void k_fill_buckets(SeqView view, Pattern pat, uint32_t step, uint32_t nwin, uint32_t* cursor,
                               uint32_t* positions) {
    const uint32_t S = gridDim.x * blockDim.x;
    for (uint32_t k0 = blockIdx.x * blockDim.x + threadIdx.x; k0 < nwin; k0 += 4 * S) {
        uint32_t w[4], slot[4];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t k = k0 + u * S;
            ok[u] = k < nwin && word_at(view, pat, k * step, w[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (ok[u]) slot[u] = atomicAdd(&cursor[w[u]], 1u);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (ok[u]) positions[slot[u]] = (k0 + u * S) * step;
    }
}

__device__ __forceinline__ void cswap(uint32_t& x, uint32_t& y) {
    const uint32_t lo = min(x, y), hi = max(x, y);
    x = lo;
    y = hi;
}

// Files bucket g (first index b, n positions) for the sort that fits it.
__device__ __forceinline__ void order_bucket(uint32_t* __restrict__ pos, uint32_t b, uint32_t n, uint2* mid,
                                             uint32_t* n_mid, uint2* big, uint32_t* n_big, uint2* huge,
                                             uint32_t* n_huge) {
    if (n <= 1) return;
    if (n > 3) {
        if (n > kBlockBucket) huge[atomicAdd(n_huge, 1u)] = make_uint2(b, n);
        else if (n > 32) big[atomicAdd(n_big, 1u)] = make_uint2(b, n);
        else mid[atomicAdd(n_mid, 1u)] = make_uint2(b, n);
        return;
    }
    uint32_t x = pos[b], y = pos[b + 1];
    if (n == 2) {
        if (x > y) {
            pos[b] = y;
            pos[b + 1] = x;
        }
        return;
    }
    uint32_t z = pos[b + 2];
    cswap(x, y);
    cswap(y, z);
    cswap(x, y);
    pos[b] = x;
    pos[b + 1] = y;
    pos[b + 2] = z;
}

// One pass over the bucket starts, four buckets a thread (one 16-byte load;
// the fifth start comes from the next lane): each group of eight lanes
// assembles one 32-bucket occupancy word; buckets of 2 or 3 positions --
// nearly all the buckets that need it at chromosome scale -- are put in
// order on the spot, larger ones listed for the warp sort (mid, <= 32), the
// block sort (big, <= kBlockBucket) or the radix sort (huge), as (first
// index, size) pairs.  The lists hold every such bucket: at most n / 4 + 1,
// n / 33 + 1 and n / (kBlockBucket + 1) + 1 of them for n positions.
__global__ void k_sort_small_buckets(const uint32_t* __restrict__ starts, uint64_t nb, uint32_t* __restrict__ pos,
                                     uint32_t* __restrict__ occ, uint2* __restrict__ packed,
                                     uint2* __restrict__ mid, uint32_t* n_mid,
                                     uint2* __restrict__ big, uint32_t* n_big, uint2* __restrict__ huge,
                                     uint32_t* n_huge) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nb128 = (nb + 127) & ~(uint64_t)127;   // whole warps: every lane reaches the shuffles
    for (uint64_t g0 = 4 * (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x); g0 < nb128;
         g0 += 4 * (uint64_t)gridDim.x * blockDim.x) {
        uint32_t s[4] = {0, 0, 0, 0};
        if (g0 + 3 < nb) {
            const uint4 v = *reinterpret_cast<const uint4*>(starts + g0);
            s[0] = v.x;
            s[1] = v.y;
            s[2] = v.z;
            s[3] = v.w;
        } else {
            // starts has nb + 1 entries: the next lane's first may be starts[nb].
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (g0 + k <= nb) s[k] = starts[g0 + k];
        }
        uint32_t next = __shfl_down_sync(kFull, s[0], 1);
        if (lane == 31 && g0 + 4 <= nb) next = starts[g0 + 4];
        uint32_t n[4], nib = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t e = k < 3 ? s[k + 1] : next;
            n[k] = g0 + k < nb ? e - s[k] : 0u;
            nib |= (n[k] != 0 ? 1u : 0u) << k;
        }
        // Eight lanes cover 32 buckets: OR their nibbles into one word.
        uint32_t word = nib << (4 * (lane & 7));
        word |= __shfl_xor_sync(kFull, word, 1);
        word |= __shfl_xor_sync(kFull, word, 2);
        word |= __shfl_xor_sync(kFull, word, 4);
        if ((lane & 7) == 0 && g0 < nb) occ[g0 >> 5] = word;
        if (packed) {   // two lanes cover eight buckets
            uint32_t sizes = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) sizes |= n[k] < 15 ? n[k] << (4 * (4 * (lane & 1) + k)) : 0xffffffffu;
            sizes |= __shfl_xor_sync(kFull, sizes, 1);
            if ((lane & 1) == 0 && g0 < nb) packed[g0 >> 3] = make_uint2(s[0], sizes);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) order_bucket(pos, s[k], n[k], mid, n_mid, big, n_big, huge, n_huge);
    }
}

// ---- The build by partition ------------------------------------------------
constexpr uint32_t kPartBuckets = 4096;
constexpr uint32_t kMaxParts = 16384;      // partitions of a group of views: their counts fit a block's shared memory
// Fewer partitions than this leave step 3 too few blocks.  By partition and by bucket,
// ms: weight 6, 2 Mbp (1 partition) 1.91 and 0.39; weight 8, 10 Mbp (16) 1.87 and 1.50;
// weight 9, 40 Mbp (64) 6.12 and 5.76, 2 Mbp 0.16 and 0.17; 40 views of 100 kbp at
// weight 7 (160) 0.43 and 0.63; weight 10, 2 Mbp (256) 0.12 and 0.18.
constexpr uint32_t kMinParts = 128;
constexpr int kPartThreads = 1024;
constexpr int kBuildThreads = 512;
constexpr uint32_t kStagedPositions = 7936;
constexpr int kHeldWindows = 6;            // a thread holds in registers
static_assert(kPartBuckets == 8 * kBuildThreads, "eight buckets a thread");

struct PartView {
    uint64_t base;   // of its first position, pad included
    uint32_t n;      // windows
    uint32_t pad_;
};

struct PartArgs {
    const uint64_t* codes;
    const uint32_t* valid;
    const uint32_t* mask;
    Pattern pat;
    uint32_t step;
    uint32_t n_views;           // of the group
    const PartView* views;
    uint32_t parts_per_view;
    uint32_t parts;             // n_views * parts_per_view
    uint32_t* hist;             // block x partition
    uint32_t* part_start;       // totals, then starts
    uint2* win;                 // the group's windows by partition: position, low word bits
};

// Calls f(partition, low word bits, position) for the block's share of the
// windows.  A thread takes those that start in 16 positions from one read of 64
// (read and reversed for each window alone they took 95 instructions apiece).
template <typename F>
__device__ __forceinline__ void for_windows(const PartArgs& a, F f) {
    constexpr uint32_t kSpan = 16;
    for (uint32_t v = 0; v < a.n_views; v++) {
        const PartView view = a.views[v];
        if (!view.n) continue;
        const uint64_t last = (uint64_t)(view.n - 1) * a.step;   // the last window's position
        const uint64_t spans = last / kSpan + 1, per = (spans + gridDim.x - 1) / gridDim.x;
        const uint64_t beg = min(spans, per * blockIdx.x), end = min(spans, beg + per);
        for (uint64_t x = beg + threadIdx.x; x < end; x += kPartThreads) {
            const uint64_t p0 = x * kSpan, g = view.base + p0;
            const SpanWindows at(p0, last, a.step, kSpan);
            if (at.first >= kSpan) continue;
            const uint64_t hi = rev_pairs64(load_codes32(a.codes, g)), lo = rev_pairs64(load_codes32(a.codes, g + 32));
            const uint32_t ok0 = load_bits32(a.valid, g) & ~load_bits32(a.mask, g);
            const uint32_t ok1 = load_bits32(a.valid, g + 32) & ~load_bits32(a.mask, g + 32);
#pragma unroll 4
            for (uint32_t j = at.first; j < at.stop; j += at.stride) {
                if ((__funnelshift_r(ok0, ok1, j) & a.pat.care_mask) != a.pat.care_mask) continue;
                const uint32_t w = word_of_reversed(a.pat, j ? hi << (2 * j) | lo >> (64 - 2 * j) : hi);
                f(v * a.parts_per_view + w / kPartBuckets, w % kPartBuckets, (uint32_t)p0 + j);
            }
        }
    }
}

__global__ __launch_bounds__(kPartThreads, 1) void k_part_count(const __grid_constant__ PartArgs a) {
    extern __shared__ uint32_t s_cnt[];
    for (uint32_t i = threadIdx.x; i < a.parts; i += kPartThreads) s_cnt[i] = 0;
    __syncthreads();
    for_windows(a, [&](uint32_t p, uint32_t, uint32_t) { atomicAdd(&s_cnt[p], 1u); });
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < a.parts; i += kPartThreads) a.hist[(uint64_t)blockIdx.x * a.parts + i] = s_cnt[i];
}

// hist's columns become exclusive prefixes over the blocks, part_start the totals.
__global__ void k_part_prefix(uint32_t* hist, uint32_t parts, uint32_t n_blocks, uint32_t* part_start) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= parts) return;
    uint32_t run = 0;
    for (uint32_t b0 = 0; b0 < n_blocks; b0 += 16) {
        uint32_t c[16];
#pragma unroll
        for (uint32_t k = 0; k < 16; k++) c[k] = b0 + k < n_blocks ? hist[(uint64_t)(b0 + k) * parts + p] : 0u;
#pragma unroll
        for (uint32_t k = 0; k < 16; k++) {
            if (b0 + k < n_blocks) hist[(uint64_t)(b0 + k) * parts + p] = run;
            run += c[k];
        }
    }
    part_start[p] = run;
}

__global__ __launch_bounds__(kPartThreads, 1) void k_part_scatter(const __grid_constant__ PartArgs a) {
    extern __shared__ uint32_t s_cnt[];
    for (uint32_t i = threadIdx.x; i < a.parts; i += kPartThreads)
        s_cnt[i] = a.part_start[i] + a.hist[(uint64_t)blockIdx.x * a.parts + i];
    __syncthreads();
    for_windows(a, [&](uint32_t p, uint32_t low, uint32_t position) {
        const uint32_t slot = atomicAdd(&s_cnt[p], 1u);
        a.win[slot] = make_uint2(position, low);
    });
}

// Partition p's buckets are first_bucket + p * kPartBuckets ..; their positions
// start where the buckets before them end.  A partition of more positions than the
// stage holds (a long repeat's) writes them to memory as they come.
__global__ __launch_bounds__(kBuildThreads, 2) void k_part_build(const uint32_t* __restrict__ part_start, uint32_t parts,
                                                                  const uint2* __restrict__ win, uint64_t first_bucket,
                                                                  uint32_t* starts, uint32_t* positions,
                                                                  uint32_t* __restrict__ occ, uint2* __restrict__ packed,
                                                                  uint2* __restrict__ mid, uint32_t* n_mid,
                                                                  uint2* __restrict__ big, uint32_t* n_big,
                                                                  uint2* __restrict__ huge, uint32_t* n_huge) {
    __shared__ __align__(16) uint32_t s_cnt[kPartBuckets];   // sizes, then cursors
    __shared__ uint32_t s_pos[kStagedPositions];
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_total;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    // (the group before this one left its end here; written again with the same value)
    const uint32_t base = first_bucket ? *reinterpret_cast<volatile uint32_t*>(starts + first_bucket) : 0u;
    uint4* const mine = reinterpret_cast<uint4*>(s_cnt) + 2 * tid;
    // A partition of up to 3,072 windows (at 10 M in 16.7 M buckets 2,441 on average)
    // is read once, into registers, while the one before it is built; the count's
    // atomics give each window its place in its bucket.
    uint2 win_next[kHeldWindows];
    uint32_t e0_next = 0, n_next = 0;
    auto fetch = [&](uint32_t p) {
        n_next = 0;
        if (p >= parts) return;
        e0_next = part_start[p];
        n_next = part_start[p + 1] - e0_next;
#pragma unroll
        for (int k = 0; k < kHeldWindows; k++)
            if (tid + k * kBuildThreads < n_next) win_next[k] = win[e0_next + tid + k * kBuildThreads];
    };
    fetch(blockIdx.x);
    for (uint32_t p = blockIdx.x; p < parts; p += gridDim.x) {
        const uint32_t e0 = e0_next, n = n_next;
        const bool held = n <= kHeldWindows * kBuildThreads;
        mine[0] = mine[1] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        uint2 w[kHeldWindows];
        uint32_t rank[kHeldWindows];
#pragma unroll
        for (int k = 0; k < kHeldWindows; k++) {
            w[k] = win_next[k];
            if (tid + k * kBuildThreads < n) rank[k] = atomicAdd(&s_cnt[w[k].y], 1u);
        }
        if (!held) {
#pragma unroll 4
            for (uint32_t i = tid + kHeldWindows * kBuildThreads; i < n; i += kBuildThreads) atomicAdd(&s_cnt[win[e0 + i].y], 1u);
        }
        fetch(p + gridDim.x);
        __syncthreads();
        uint32_t c[8], at[8], sum = 0;
        {
            const uint4 x = mine[0], y = mine[1];
            c[0] = x.x; c[1] = x.y; c[2] = x.z; c[3] = x.w;
            c[4] = y.x; c[5] = y.y; c[6] = y.z; c[7] = y.w;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) sum += c[k];
        uint32_t run = block_excl_scan<kBuildThreads>(sum, s_warp, &s_total);
        uint32_t sizes = 0, some = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            at[k] = run;
            run += c[k];
            sizes |= c[k] < 15 ? c[k] << (4 * k) : 0xffffffffu;
            some |= (c[k] ? 1u : 0u) << k;
        }
        mine[0] = make_uint4(at[0], at[1], at[2], at[3]);
        mine[1] = make_uint4(at[4], at[5], at[6], at[7]);
        const uint64_t g = first_bucket + (uint64_t)p * kPartBuckets + 8 * tid;
        const uint32_t b = base + e0;
        *reinterpret_cast<uint4*>(starts + g) = make_uint4(b + at[0], b + at[1], b + at[2], b + at[3]);
        *reinterpret_cast<uint4*>(starts + g + 4) = make_uint4(b + at[4], b + at[5], b + at[6], b + at[7]);
        if (packed) packed[g >> 3] = make_uint2(b + at[0], sizes);
        some <<= 8 * (lane & 3);
        some |= __shfl_xor_sync(kFull, some, 1);
        some |= __shfl_xor_sync(kFull, some, 2);
        if ((lane & 3) == 0) occ[g >> 5] = some;
        if (p == parts - 1 && tid == 0) starts[first_bucket + (uint64_t)parts * kPartBuckets] = b + n;
        __syncthreads();
        const bool staged = n <= kStagedPositions;
        auto place = [&](uint32_t* to) {
            if (held) {
#pragma unroll
                for (int k = 0; k < kHeldWindows; k++)
                    if (tid + k * kBuildThreads < n) to[s_cnt[w[k].y] + rank[k]] = w[k].x;
            } else {
#pragma unroll 4
                for (uint32_t i = tid; i < n; i += kBuildThreads) {
                    const uint2 x = win[e0 + i];
                    to[atomicAdd(&s_cnt[x.y], 1u)] = x.x;
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (c[k] < 2) continue;
                if (c[k] > 8) {
                    const uint2 e = make_uint2(b + at[k], c[k]);
                    if (c[k] > kBlockBucket) huge[atomicAdd(n_huge, 1u)] = e;
                    else if (c[k] > 32) big[atomicAdd(n_big, 1u)] = e;
                    else mid[atomicAdd(n_mid, 1u)] = e;
                    continue;
                }
                uint32_t* const x = to + at[k];
                for (uint32_t i = 1; i < c[k]; i++) {
                    const uint32_t y = x[i];
                    uint32_t j = i;
                    for (; j && x[j - 1] > y; j--) x[j] = x[j - 1];
                    x[j] = y;
                }
            }
        };
        if (!staged) {
            place(positions + b);
        } else {
            place(s_pos);
            __syncthreads();
            for (uint32_t i = tid; i < n; i += kBuildThreads) positions[b + i] = s_pos[i];
        }
        __syncthreads();
    }
}

// Listed buckets of 4..32 positions, a warp each: a bitonic sort across the
// lanes by shuffles.
__global__ void k_sort_warp_buckets(const uint2* __restrict__ mid, const uint32_t* n_mid, uint32_t* __restrict__ pos) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nl = *n_mid;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); e < nl; e += warps) {
        const uint32_t b = mid[e].x, n = mid[e].y;
        uint32_t x = lane < n ? pos[b + lane] : 0xffffffffu;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const uint32_t y = __shfl_xor_sync(kFull, x, j);
                const bool up = (lane & k) == 0;
                const bool low = (lane & j) == 0;
                // the lower lane of a pair keeps the smaller in an ascending run
                x = (low == up) ? min(x, y) : max(x, y);
            }
        }
        if (lane < n) pos[b + lane] = x;
    }
}

// Bitonic sort of listed buckets (33 .. kBlockBucket positions) in shared
// memory, a block each.
__global__ __launch_bounds__(256) void k_sort_block_buckets(const uint2* __restrict__ big, const uint32_t* n_big,
                                                             uint32_t* __restrict__ pos) {
    __shared__ uint32_t s[kBlockBucket];
    const uint32_t nl = *n_big;
    for (uint32_t e = blockIdx.x; e < nl; e += gridDim.x) {
        const uint32_t b = big[e].x, n = big[e].y;
        uint32_t m = 1;
        while (m < n) m <<= 1;
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) s[i] = i < n ? pos[b + i] : 0xffffffffu;
        __syncthreads();
        for (uint32_t k = 2; k <= m; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                    const uint32_t l = i ^ j;
                    if (l > i) {
                        const uint32_t x = s[i], y = s[l];
                        const bool up = (i & k) == 0;
                        if (up ? x > y : x < y) {
                            s[i] = y;
                            s[l] = x;
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) pos[b + i] = s[i];
        __syncthreads();
    }
}

// first[v] = global start of view v's buckets; first[n] = all positions.
__global__ void k_view_firsts(const uint32_t* __restrict__ starts, uint64_t nw, uint32_t n_views, uint32_t* first) {
    for (uint32_t v = threadIdx.x; v <= n_views; v += blockDim.x) first[v] = starts[(uint64_t)v * nw];
}

// rec[8 j ..]: the codes of words first + j - 1 .. first + j + 2; the last
// position's two bits set when any of the 128 positions is invalid, else clear.
__global__ void k_window_records(const uint64_t* __restrict__ codes, const uint32_t* __restrict__ valid, uint64_t first,
                                 uint64_t n, uint4* __restrict__ rec) {
    for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t w = first + j - 1;
        const uint64_t a = codes[w], b = codes[w + 1], c = codes[w + 2], d = codes[w + 3];
        const bool ok = (valid[w] & valid[w + 1] & valid[w + 2] & valid[w + 3]) == 0xffffffffu;
        rec[2 * j] = make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
        rec[2 * j + 1] = make_uint4((uint32_t)c, (uint32_t)(c >> 32), (uint32_t)d,
                                    ((uint32_t)(d >> 32) & 0x3fffffffu) | (ok ? 0u : 0xc0000000u));
    }
}

}  // namespace

void table_init() {
    cudaFuncSetAttribute(k_part_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxParts * 4);
    cudaFuncSetAttribute(k_part_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxParts * 4);
}

void launch_window_records(const uint64_t* codes, const uint32_t* valid, uint64_t first, uint64_t n, uint32_t* rec,
                           cudaStream_t st) {
    if (!n) return;
    count_launch();
    k_window_records<<<(int)std::min<uint64_t>((n + 255) / 256, 148 * 16), 256, 0, st>>>(codes, valid, first, n,
                                                                                         reinterpret_cast<uint4*>(rec));
}

gxy_status atomic_build_views(const gxy_dseq* seq, uint32_t n_views, const uint64_t* lo, const uint64_t* hi,
                              const Pattern& pat, uint32_t step, uint32_t* starts, uint32_t* positions,
                              uint32_t* occ, uint2* packed, uint32_t* first_host, Worker* W) {
    cudaStream_t st = W->st;
    const uint64_t nw = 1ull << (2 * pat.weight);
    const uint64_t G = (uint64_t)n_views * nw;
    if (n_views == 0 || (n_views > 1 && nw < 32)) {
        set_error("a multi-view build needs at least 32 buckets per view");
        return GXY_EUNSUPPORTED;
    }
    uint64_t total = 0;
    std::vector<uint32_t> nwin(n_views);
    for (uint32_t v = 0; v < n_views; v++) {
        nwin[v] = n_windows(hi[v] - lo[v], pat.len, step);
        total += nwin[v];
    }
    if (total >= (1ull << 32)) {
        set_error("more than 2^32 windows in one table build");
        return GXY_EUNSUPPORTED;
    }
    const uint64_t n_mid_cap = total / 4 + 1, n_big_cap = total / 33 + 1,
                   n_huge_cap = total / (kBlockBucket + 1) + 1;
    GXY_CK(W->tv0.ensure((n_mid_cap + n_big_cap + n_huge_cap) * 8));
    GXY_CK(W->tv1.ensure(64 + ((size_t)n_views + 1) * 4));
    uint2* mid = W->tv0.as<uint2>();
    uint2* big = mid + n_mid_cap;
    uint2* huge = big + n_big_cap;
    uint32_t* ctr = W->tv1.as<uint32_t>();   // [0] big buckets, [1] huge buckets, [2] mid buckets
    uint32_t* first = ctr + 16;
    GXY_CK(cudaMemsetAsync(ctr, 0, 12, st));
    uint32_t ppv = 1, per_group = 1, max_blocks = 1;
    bool by_partition = nw >= kPartBuckets && nw / kPartBuckets <= kMaxParts;
    if (by_partition) {
        ppv = (uint32_t)(nw / kPartBuckets);
        per_group = kMaxParts / ppv;
        by_partition = (uint64_t)std::min(n_views, per_group) * ppv >= kMinParts;
    }
    if (by_partition) {
        uint64_t most = 0;   // windows of a group
        for (uint32_t v0 = 0; v0 < n_views; v0 += per_group) {
            uint64_t t = 0;
            for (uint32_t v = v0; v < std::min(n_views, v0 + per_group); v++) t += nwin[v];
            most = std::max(most, t);
        }
        // A block's share is 2,048 windows at least: below that its counts outweigh them.
        max_blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(148, most / 2048));
        const uint32_t max_parts = std::min(n_views, per_group) * ppv;
        // Eight bytes a window: where they do not fit, the table is built bucket by
        // bucket, from four bytes a bucket.
        by_partition = W->tk0.ensure(n_views * sizeof(PartView) + ((uint64_t)max_blocks * max_parts + max_parts + 8) * 4) ==
                           cudaSuccess &&
                       W->tk1.ensure(most * 8 + 64) == cudaSuccess;
        if (!by_partition) {
            cudaGetLastError();
            W->tk1.release();
        }
    }
    if (by_partition) {
        std::vector<PartView> spans(n_views);
        for (uint32_t v = 0; v < n_views; v++) spans[v] = PartView{kPad + lo[v], nwin[v], 0};
        PartView* dspans = W->tk0.as<PartView>();
        uint32_t* part_start = reinterpret_cast<uint32_t*>(dspans + n_views);   // (16-byte aligned)
        GXY_CK(cudaMemcpyAsync(dspans, spans.data(), n_views * sizeof(PartView), cudaMemcpyHostToDevice, st));
        for (uint32_t v0 = 0; v0 < n_views; v0 += per_group) {
            PartArgs a;
            a.codes = seq->codes;
            a.valid = seq->valid;
            a.mask = seq->mask;
            a.pat = pat;
            a.step = step;
            a.n_views = std::min(per_group, n_views - v0);
            a.views = dspans + v0;
            a.parts_per_view = ppv;
            a.parts = a.n_views * ppv;
            a.part_start = part_start;
            a.hist = part_start + ((a.parts + 1 + 3) & ~3u);
            a.win = W->tk1.as<uint2>();
            uint64_t t = 0;
            for (uint32_t v = v0; v < v0 + a.n_views; v++) t += nwin[v];
            const uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(max_blocks, t / 2048));
            count_launch(4);
            k_part_count<<<blocks, kPartThreads, a.parts * 4, st>>>(a);
            k_part_prefix<<<(a.parts + 63) / 64, 64, 0, st>>>(a.hist, a.parts, blocks, part_start);
            scan_small(part_start, (int)a.parts, st);
            k_part_scatter<<<blocks, kPartThreads, a.parts * 4, st>>>(a);
            k_part_build<<<(int)std::min<uint32_t>(a.parts, 148 * 2), kBuildThreads, 0, st>>>(
                part_start, a.parts, a.win, (uint64_t)v0 * nw, starts, positions, occ, packed, mid, ctr + 2, big, ctr, huge,
                ctr + 1);
        }
    } else {
        GXY_CK(W->tk0.ensure((G + 1) * 4));
        uint32_t* counts = W->tk0.as<uint32_t>();
        GXY_CK(cudaMemsetAsync(counts, 0, (G + 1) * 4, st));
        std::vector<SeqView> views(n_views);
        for (uint32_t v = 0; v < n_views; v++) views[v] = view_of(seq, lo[v], hi[v]);
        const int cblocks = 148 * 16;
        for (uint32_t v = 0; v < n_views; v++) {
            if (!nwin[v]) continue;
            count_launch();
            k_count_words<<<(int)std::min<uint64_t>((nwin[v] + 255) / 256, cblocks), 256, 0, st>>>(
                views[v], pat, step, nwin[v], counts + (uint64_t)v * nw);
        }
        // Global starts, and their copy back in counts: the fill's cursors (a
        // fill that decremented the counts and read the start instead measured
        // 169 us against 96 us: one more random load per window).
        scan_u32(counts, starts, nullptr, G, G, true, nullptr, W->ps, st, counts);
        for (uint32_t v = 0; v < n_views; v++) {
            if (!nwin[v]) continue;
            count_launch();
            k_fill_buckets<<<(int)std::min<uint64_t>((nwin[v] + 255) / 256, cblocks), 256, 0, st>>>(
                views[v], pat, step, nwin[v], counts + (uint64_t)v * nw, positions);
        }
        count_launch();
        k_sort_small_buckets<<<148 * 16, 256, 0, st>>>(starts, G, positions, occ, packed, mid, ctr + 2, big, ctr, huge, ctr + 1);
    }
    count_launch(3);
    k_sort_warp_buckets<<<148 * 4, 256, 0, st>>>(mid, ctr + 2, positions);
    k_sort_block_buckets<<<148 * 2, 256, 0, st>>>(big, ctr, positions);
    k_view_firsts<<<1, 256, 0, st>>>(starts, nw, n_views, first);
    GXY_CK(cudaGetLastError());
    std::vector<uint32_t> h(16 + (size_t)n_views + 1);
    GXY_CK(cudaMemcpyAsync(h.data(), ctr, h.size() * 4, cudaMemcpyDeviceToHost, st));
    GXY_CK(cudaStreamSynchronize(st));
    const uint32_t n_huge = h[1];
    if (n_huge) {
        // Buckets past kBlockBucket (long repeats): the radix sort, one at a time.
        std::vector<uint2> hb(n_huge);
        GXY_CK(cudaMemcpyAsync(hb.data(), huge, (size_t)n_huge * 8, cudaMemcpyDeviceToHost, st));
        GXY_CK(cudaStreamSynchronize(st));
        int bits = 1;
        uint64_t span = 0;
        for (uint32_t v = 0; v < n_views; v++) span = std::max<uint64_t>(span, hi[v] - lo[v]);
        while (bits < 32 && (1ull << bits) < span) bits++;
        RadixPass passes[8];
        const int np = plan_radix(0, bits, 0, 0, passes, 8);
        for (const uint2& e : hb) {
            GXY_CK(W->tk1.ensure((size_t)e.y * 4));
            GXY_CK(W->tv0.ensure((size_t)e.y * 4));
            GXY_CK(W->tk0.ensure((size_t)e.y * 4));
            const int which = radix_sort_u32(positions + e.x, W->tv0.as<uint32_t>(), W->tk1.as<uint32_t>(),
                                             W->tk0.as<uint32_t>(), nullptr, e.y, e.y, passes, np, W->ps, st);
            if (which)
                GXY_CK(cudaMemcpyAsync(positions + e.x, W->tk1.p, (size_t)e.y * 4, cudaMemcpyDeviceToDevice, st));
        }
        GXY_CK(cudaStreamSynchronize(st));
        GXY_CK(cudaGetLastError());
    }
    if (first_host) memcpy(first_host, h.data() + 16, ((size_t)n_views + 1) * 4);
    return GXY_OK;
}

}  // namespace gxy
