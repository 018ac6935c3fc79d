// gxy_epilogue.cu -- what follows the passes of a launch, each in one kernel
// for sm_100a: the candidates' sort by (diagonal, t), and after the walk the
// kept HSPs' compaction, grouping by unit and order within a diagonal.
//
// The element counts are only known on the device (the screen's candidates,
// the walk's HSPs) and range from a handful to tens of millions.  Both kernels
// are cooperative launches of a block an SM that use as many of their blocks as
// the count needs -- one, without any grid barrier, up to 512 candidates (the
// sort) or a tile of 4,096 (the finish) -- so a small search does not pay for
// empty launches (a three-kernel pass per digit took 60 us for a few hundred
// candidates), and a large one crosses the device a few times per digit.
//
// What bounds them: barriers and launch latency for small counts; for large
// ones the scatter's read and write of 12 B an item and digit.
#include "gxy_engine.cuh"
#include "gxy_kernels.cuh"
#include "gxy_radix.cuh"

#include <algorithm>

namespace gxy {

namespace {

constexpr int kEpiThreads = 512;
constexpr int kEpiWarps = kEpiThreads / 32;
// A cooperative launch starts when all of its blocks fit the device at once, so a
// block must fit an SM beside what other streams run there: two a SM hold its
// registers (64 a thread) and its 68 KB to half of one or less.  With 125 registers
// a block took a whole SM, and a search waited for every SM to be empty: 4 streams
// with a 2 Mbp request beside 40 small ones each took 140 ms and 85 ms a request on
// average, against 70 and 10 now (same figures for three a SM, which spills).
constexpr int kEpiPerSm = 2;
constexpr int kEpiItems = 8;
constexpr uint32_t kEpiTile = kEpiThreads * kEpiItems;

struct EpiSmem {
    uint64_t keys[kEpiTile];
    uint32_t vals[kEpiTile];
    uint32_t wcnt[kEpiWarps][kRadixMax];
    uint32_t tile_excl[kRadixMax];
    uint32_t tile_tot[kRadixMax];
    uint32_t off[kRadixMax];
    uint32_t hist[kRadixMax];
    uint32_t warp_tmp[32];
    uint32_t total;
    uint32_t ok;
};

// Barrier of the first n blocks of a cooperative launch.  False: some block gave
// up; the caller returns.
struct GridBarrier {
    uint32_t* bar;       // arrivals, zero before the launch
    uint32_t* gave_up;
    uint32_t polls;      // of a wait
    uint32_t phase = 0;
    __device__ GridBarrier(uint32_t* b, uint32_t* g, uint32_t p) : bar(b), gave_up(g), polls(p) {}
    __device__ __forceinline__ bool wait(uint32_t n, uint32_t* s_ok) {
        if (n == 1) {
            __syncthreads();
            return true;
        }
        __syncthreads();
        phase++;
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(bar, 1u);
            const uint32_t target = phase * n;
            uint32_t seen = 0, ok = 1;
            for (uint32_t p = 0;; p++) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
                if (seen >= target) break;
                if (p >= polls) {
                    atomicExch(gave_up, 1u);
                    ok = 0;
                    break;
                }
            }
            *s_ok = ok;
        }
        __syncthreads();
        return *s_ok != 0;
    }
};

// The contiguous range of block b of nb when n items are split into whole tiles.
__device__ __forceinline__ void epi_range(uint32_t n, uint32_t nb, uint32_t b, uint32_t& beg, uint32_t& end) {
    const uint32_t tiles = (n + kEpiTile - 1) / kEpiTile, per = (tiles + nb - 1) / nb;
    beg = (uint32_t)min((uint64_t)n, (uint64_t)b * per * kEpiTile);
    end = (uint32_t)min((uint64_t)n, (uint64_t)beg + (uint64_t)per * kEpiTile);
}

// The buffers are read with plain loads: other blocks wrote them in this launch.
// One stable pass over a digit of (key, value) pairs by blocks 0 .. nb - 1.
// hist: nb x 256 counts.  False: a barrier gave up.
template <typename K>
__device__ bool epi_radix_pass(EpiSmem& S, const K* kin, const uint32_t* vin, K* kout, uint32_t* vout,
                               uint32_t n, uint32_t nb, int shift, int bits, uint32_t* hist,
                               GridBarrier& barrier) {
    const uint32_t dmask = (1u << bits) - 1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t lt = lanemask_lt();
    uint32_t beg, end;
    epi_range(n, nb, blockIdx.x, beg, end);
    // The block's counts, then the output offsets: all smaller digits, and
    // this digit in the blocks before this one.
    if (threadIdx.x < kRadixMax) S.hist[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = beg + threadIdx.x; i < end; i += kEpiThreads)
        atomicAdd(&S.hist[(uint32_t)(kin[i] >> shift) & dmask], 1u);
    __syncthreads();
    uint32_t before = 0, all = 0;
    if (nb == 1) {
        if (threadIdx.x < kRadixMax) all = S.hist[threadIdx.x];
    } else {
        if (threadIdx.x < kRadixMax) hist[blockIdx.x * kRadixMax + threadIdx.x] = S.hist[threadIdx.x];
        if (!barrier.wait(nb, &S.ok)) return false;
        if (threadIdx.x < kRadixMax) {
#pragma unroll 8
            for (uint32_t b = 0; b < nb; b++) {
                const uint32_t c = __ldcg(hist + b * kRadixMax + threadIdx.x);
                before += b < blockIdx.x ? c : 0u;
                all += c;
            }
        }
    }
    const uint32_t g = block_excl_scan<kEpiThreads>(all, S.warp_tmp, &S.total);
    if (threadIdx.x < kRadixMax) S.off[threadIdx.x] = g + before;
    for (uint32_t tb = beg; tb < end; tb += kEpiTile) {
        for (int i = threadIdx.x; i < kEpiWarps * kRadixMax; i += kEpiThreads) (&S.wcnt[0][0])[i] = 0;
        __syncthreads();
        K k[kEpiItems];
        uint32_t v[kEpiItems], d[kEpiItems], rk[kEpiItems];
#pragma unroll
        for (int it = 0; it < kEpiItems; it++) {
            const uint32_t idx = tb + (uint32_t)w * 32 * kEpiItems + (uint32_t)it * 32 + lane;
            const bool ok = idx < end;
            k[it] = ok ? kin[idx] : (K)0;
            v[it] = ok ? vin[idx] : 0u;
            d[it] = ok ? ((uint32_t)(k[it] >> shift) & dmask) : (uint32_t)kRadixMax;
        }
#pragma unroll
        for (int it = 0; it < kEpiItems; it++) {
            const uint32_t peers = __match_any_sync(kFull, d[it]);
            uint32_t base = 0;
            if (d[it] < (uint32_t)kRadixMax) base = S.wcnt[w][d[it]];
            __syncwarp();
            if (d[it] < (uint32_t)kRadixMax && (peers & lt) == 0) S.wcnt[w][d[it]] = base + __popc(peers);
            __syncwarp();
            rk[it] = base + __popc(peers & lt);
        }
        __syncthreads();
        // Per digit: exclusive prefix over warps and the tile total.
        uint32_t run = 0;
        if (threadIdx.x < kRadixMax) {
#pragma unroll
            for (int ww = 0; ww < kEpiWarps; ww++) {
                const uint32_t c = S.wcnt[ww][threadIdx.x];
                S.wcnt[ww][threadIdx.x] = run;
                run += c;
            }
            S.tile_tot[threadIdx.x] = run;
        }
        const uint32_t ex = block_excl_scan<kEpiThreads>(run, S.warp_tmp, &S.total);
        if (threadIdx.x < kRadixMax) S.tile_excl[threadIdx.x] = ex;
        __syncthreads();
#pragma unroll
        for (int it = 0; it < kEpiItems; it++) {
            if (d[it] < (uint32_t)kRadixMax) {
                const uint32_t p = S.tile_excl[d[it]] + S.wcnt[w][d[it]] + rk[it];
                S.keys[p] = k[it];
                S.vals[p] = v[it];
            }
        }
        __syncthreads();
        const uint32_t cnt = min(kEpiTile, end - tb);
        for (uint32_t j = threadIdx.x; j < cnt; j += kEpiThreads) {
            const K key = (K)S.keys[j];
            const uint32_t dd = (uint32_t)(key >> shift) & dmask;
            const uint32_t o = S.off[dd] + (j - S.tile_excl[dd]);
            kout[o] = key;
            vout[o] = S.vals[j];
        }
        __syncthreads();
        if (threadIdx.x < kRadixMax) S.off[threadIdx.x] += S.tile_tot[threadIdx.x];
        __syncthreads();
    }
    return barrier.wait(nb, &S.ok);
}

// Blocks that share n items: one per tile, as far as the grid has them.
__device__ __forceinline__ uint32_t epi_blocks(uint32_t n) {
    return min(gridDim.x, max(1u, (n + kEpiTile - 1) / kEpiTile));
}

// ---- Up to kMergeMax candidates: tiles sorted in registers, then each item's
// place from its rank in every other tile.  A digit pass costs two grid barriers
// and a scan whatever the count, some 4 us; 30 to 40 key bits took five of them.

// Keys of E x 512 items, item threadIdx.x * E + e in k[e] and v[e], in ascending
// order (bitonic: strides inside a thread, then lanes, then the block).
template <int E>
__device__ void sort_tile(EpiSmem& S, uint64_t (&k)[E], uint32_t (&v)[E]) {
    const uint32_t tid = threadIdx.x;
    auto keep = [&](int e, uint64_t pk, uint32_t pv, bool lower) {   // the smaller of the two, or the larger
        const bool take = lower ? pk < k[e] : pk > k[e];
        k[e] = take ? pk : k[e];
        v[e] = take ? pv : v[e];
    };
    for (uint32_t size = 2; size <= E * kEpiThreads; size <<= 1) {
        const bool asc = !((tid * E) & size);   // (of strides from E on; inside a thread it may depend on e)
        for (uint32_t stride = size >> 1; stride >= E; stride >>= 1) {
            const uint32_t d = stride / E;
            const bool lower = !(tid & d) == asc;
            if (d >= 32) {
                __syncthreads();
#pragma unroll
                for (int e = 0; e < E; e++) {
                    S.keys[e * kEpiThreads + tid] = k[e];
                    S.vals[e * kEpiThreads + tid] = v[e];
                }
                __syncthreads();
#pragma unroll
                for (int e = 0; e < E; e++) keep(e, S.keys[e * kEpiThreads + (tid ^ d)], S.vals[e * kEpiThreads + (tid ^ d)], lower);
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const uint64_t pk = __shfl_xor_sync(kFull, k[e], d);
                    const uint32_t pv = __shfl_xor_sync(kFull, v[e], d);
                    keep(e, pk, pv, lower);
                }
            }
        }
#pragma unroll
        for (uint32_t stride = E / 2; stride; stride >>= 1) {
            if (stride >= size) continue;
#pragma unroll
            for (uint32_t e = 0; e < E; e++) {
                if (e & stride) continue;
                const bool up = !((tid * E + e) & size);
                if (up ? k[e + stride] < k[e] : k[e + stride] > k[e]) {
                    const uint64_t tk = k[e];
                    k[e] = k[e + stride];
                    k[e + stride] = tk;
                    const uint32_t tv = v[e];
                    v[e] = v[e + stride];
                    v[e + stride] = tv;
                }
            }
        }
    }
}

constexpr uint32_t kMergeTiles = 32;
constexpr uint32_t kMergeMax = kMergeTiles * 2 * kEpiThreads;

template <int E>
__device__ void sort_by_ranks(EpiSmem& S, const EpiSort& a, uint32_t n, uint32_t nb, GridBarrier& barrier) {
    constexpr uint32_t kTile = E * kEpiThreads;
    const uint32_t nt = (n + kTile - 1) / kTile, tid = threadIdx.x;
    const bool odd = a.npass & 1;
    uint64_t* const kout = odd ? a.k1 : a.k0;
    uint32_t* const vout = odd ? a.v1 : a.v0;
    // The sorted tiles: the result itself when there is one, else the buffer
    // that the result does not take.
    uint64_t* const kt = nt == 1 ? kout : (odd ? a.k0 : a.k1);
    uint32_t* const vt = nt == 1 ? vout : (odd ? a.v0 : a.v1);
    for (uint32_t t = blockIdx.x; t < nt; t += nb) {
        uint64_t k[E];
        uint32_t v[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const uint32_t i = t * kTile + tid * E + e;
            k[e] = i < n ? a.k0[i] : ~0ull;
            v[e] = i < n ? a.v0[i] : 0xffffffffu;
        }
        __syncthreads();   // all of the tile is read: it may be written in place
        sort_tile<E>(S, k, v);
#pragma unroll
        for (int e = 0; e < E; e++) {
            const uint32_t i = t * kTile + tid * E + e;
            if (i < n) {
                kt[i] = k[e];
                vt[i] = v[e];
            }
        }
    }
    if (nt == 1) return;
    if (!barrier.wait(nb, &S.ok)) return;
    // 128 neighbours of one tile a turn (their searches take almost the same
    // path), a quarter of the tiles by each four warps, four searches at a time.
    const uint32_t mine = tid & 127u, part = tid >> 7;
    for (uint32_t i0 = blockIdx.x * 128; i0 < n; i0 += nb * 128) {
        __syncthreads();
        if (tid < 128) S.off[tid] = 0;
        __syncthreads();
        const uint32_t i = i0 + mine, own = i0 / kTile;
        const uint64_t key = i < n ? kt[i] : ~0ull;
        uint32_t rank = 0;
        for (uint32_t t0 = part; t0 < nt; t0 += 16) {
            uint32_t pos[4] = {0, 0, 0, 0}, cnt[4];
#pragma unroll
            for (uint32_t x = 0; x < 4; x++) {
                const uint32_t t = t0 + 4 * x;
                cnt[x] = t < nt && t != own ? min(kTile, n - t * kTile) : 0u;
            }
#pragma unroll
            for (uint32_t s = kTile; s; s >>= 1) {
#pragma unroll
                for (uint32_t x = 0; x < 4; x++) {
                    if (pos[x] + s <= cnt[x]) {
                        const uint32_t t = t0 + 4 * x;
                        const uint64_t other = kt[t * kTile + pos[x] + s - 1];
                        if (other < key || (t < own && other == key)) pos[x] += s;
                    }
                }
            }
            rank += pos[0] + pos[1] + pos[2] + pos[3];
        }
        if (rank) atomicAdd(&S.off[mine], rank);
        __syncthreads();
        if (tid < 128 && i < n) {
            const uint32_t o = i - own * kTile + S.off[tid];
            kout[o] = key;
            vout[o] = vt[i];
        }
    }
}

// What bounds it: up to 32,768 candidates the latency of the sorting network and
// of the searches; above, two crossings of the buffers a digit.  By ranks and by
// five digits: 721 candidates 10 and 22 us, 4,639 14 and 61, 15,346 22 and 68,
// 32,187 48 and 69; with tiles of 2,048, 46,590 take 71 and 70, 64,123 96 and 68.
__global__ __launch_bounds__(kEpiThreads, kEpiPerSm) void k_sort_candidates(const __grid_constant__ EpiSort a) {
    extern __shared__ __align__(16) unsigned char epi_smem[];
    EpiSmem& S = *reinterpret_cast<EpiSmem*>(epi_smem);
    const uint32_t n = min(*a.n_dev, a.n_cap);
    GridBarrier barrier(a.bar, a.gave_up, a.polls);
    if (n <= kMergeMax && a.npass > 0) {
        // The smallest tiles of which there are at most kMergeTiles; as many blocks
        // as have 128 items to place.
        const uint32_t nb = n <= kEpiThreads ? 1u : min(gridDim.x, (n + 127) / 128);
        if (blockIdx.x >= nb) return;
        if (a.clear)
            for (uint32_t i = blockIdx.x * kEpiThreads + threadIdx.x; i < n; i += nb * kEpiThreads) a.clear[i] = 0;
        if (n <= kMergeMax / 2) sort_by_ranks<1>(S, a, n, nb, barrier);
        else sort_by_ranks<2>(S, a, n, nb, barrier);
        return;
    }
    const uint32_t nb = epi_blocks(n);
    if (blockIdx.x >= nb) return;
    if (a.clear)
        for (uint32_t i = blockIdx.x * kEpiThreads + threadIdx.x; i < n; i += nb * kEpiThreads) a.clear[i] = 0;
    for (int p = 0; p < a.npass; p++) {
        const bool odd = p & 1;
        if (!epi_radix_pass<uint64_t>(S, odd ? a.k1 : a.k0, odd ? a.v1 : a.v0, odd ? a.k0 : a.k1, odd ? a.v0 : a.v1, n, nb,
                                      a.passes[p].shift, a.passes[p].bits, a.hist, barrier))
            return;
    }
}

__device__ __forceinline__ int64_t diag_of(const Hsp& h) { return (int64_t)h.t_start - (int64_t)h.q_start; }
__device__ __forceinline__ bool hsp_less(const Hsp& x, const Hsp& y) {
    if (x.t_start != y.t_start) return x.t_start < y.t_start;
    if (x.length != y.length) return x.length < y.length;
    return x.score < y.score;
}

// The walk's flagged HSPs in candidate order, grouped by unit (stably), each
// (unit, diagonal) run in (t_start, length, score) order.
__global__ __launch_bounds__(kEpiThreads, kEpiPerSm) void k_finish_hsps(const __grid_constant__ EpiFinish a) {
    extern __shared__ __align__(16) unsigned char epi_smem[];
    EpiSmem& S = *reinterpret_cast<EpiSmem*>(epi_smem);
    const uint32_t n = min(*a.n_dev, a.n_cap), nb = epi_blocks(n);
    if (*a.sort_gave_up) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *a.gave_up = 1;
        return;
    }
    if (blockIdx.x >= nb) return;
    GridBarrier barrier(a.bar, a.gave_up, a.polls);
    uint32_t beg, end;
    epi_range(n, nb, blockIdx.x, beg, end);
    // Kept HSPs of the block's range, and of the ranges before it.
    uint32_t mine = 0;
    for (uint32_t i = beg + threadIdx.x; i < end; i += kEpiThreads) mine += a.flag[i];
    block_excl_scan<kEpiThreads>(mine, S.warp_tmp, &S.total);
    uint32_t base = 0, m = S.total;
    if (nb > 1) {
        if (threadIdx.x == 0) a.hist[blockIdx.x] = S.total;
        if (!barrier.wait(nb, &S.ok)) return;
        uint32_t c0 = 0, c1 = 0;
        for (uint32_t b = threadIdx.x; b < nb; b += kEpiThreads) {
            const uint32_t c = __ldcg(a.hist + b);
            c0 += b < blockIdx.x ? c : 0u;
            c1 += c;
        }
        block_excl_scan<kEpiThreads>(c0, S.warp_tmp, &S.total);
        base = S.total;
        __syncthreads();
        block_excl_scan<kEpiThreads>(c1, S.warp_tmp, &S.total);
        m = S.total;
        __syncthreads();
    }
    for (uint32_t tb = beg; tb < end; tb += kEpiThreads) {
        const uint32_t i = tb + threadIdx.x;
        const bool keep = i < end && a.flag[i];
        const uint32_t o = base + block_excl_scan<kEpiThreads>(keep ? 1u : 0u, S.warp_tmp, &S.total);
        if (keep) {
            a.hsp0[o] = a.ohsp[i];
            const uint32_t u = a.n_units > 1 ? a.cands[a.idx[i]].unit : 0u;
            a.unit0[o] = u;
            if (a.n_units > 1) {
                a.key0[o] = u;
                a.perm0[o] = o;
            }
        }
        base += S.total;
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.n_hsps = m;
    if (!barrier.wait(nb, &S.ok)) return;
    Hsp* hsp = a.hsp0;
    uint32_t* unit = a.unit0;
    const uint32_t stride = nb * kEpiThreads, first = blockIdx.x * kEpiThreads + threadIdx.x;
    if (a.n_units > 1) {
        // Stable sort of the positions by unit, then the gather.
        for (int p = 0; p < a.npass; p++) {
            const bool odd = p & 1;
            if (!epi_radix_pass<uint32_t>(S, odd ? a.key1 : a.key0, odd ? a.perm1 : a.perm0, odd ? a.key0 : a.key1,
                                          odd ? a.perm0 : a.perm1, m, nb, a.passes[p].shift, a.passes[p].bits, a.hist,
                                          barrier))
                return;
        }
        const uint32_t* perm = (a.npass & 1) ? a.perm1 : a.perm0;
        const uint32_t* key = (a.npass & 1) ? a.key1 : a.key0;
        for (uint32_t i = first; i < m; i += stride) {
            a.hsp1[i] = a.hsp0[__ldcg(perm + i)];
            a.unit1[i] = __ldcg(key + i);
        }
        hsp = a.hsp1;
        unit = a.unit1;
        if (!barrier.wait(nb, &S.ok)) return;
    }
    // Run heads from the unmodified array, then one thread per run sorts it;
    // runs are short and almost always in order already.
    for (uint32_t i = first; i < m; i += stride)
        a.head[i] = (i == 0 || unit[i - 1] != unit[i] || diag_of(hsp[i - 1]) != diag_of(hsp[i])) ? 1 : 0;
    if (!barrier.wait(nb, &S.ok)) return;
    for (uint32_t i = first; i < m; i += stride) {
        if (!a.head[i]) continue;
        uint32_t e = i + 1;
        bool sorted = true;
        while (e < m && !a.head[e]) {
            if (hsp_less(hsp[e], hsp[e - 1])) sorted = false;
            e++;
        }
        if (sorted) continue;
        for (uint32_t x = i + 1; x < e; x++) {
            const Hsp key = hsp[x];
            uint32_t y = x;
            while (y > i && hsp_less(key, hsp[y - 1])) {
                hsp[y] = hsp[y - 1];
                y--;
            }
            hsp[y] = key;
        }
    }
}

}  // namespace

void epilogue_init() {
    cudaFuncSetAttribute(k_sort_candidates, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EpiSmem));
    cudaFuncSetAttribute(k_finish_hsps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EpiSmem));
}

cudaError_t launch_sort_candidates(const EpiSort& a, int sm_count, cudaStream_t st) {
    EpiSort arg = a;
    void* args[] = {&arg};
    count_launch();
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_sort_candidates), dim3(sm_count), dim3(kEpiThreads),
                                       args, sizeof(EpiSmem), st);
}

cudaError_t launch_finish_hsps(const EpiFinish& a, int sm_count, cudaStream_t st) {
    EpiFinish arg = a;
    void* args[] = {&arg};
    count_launch();
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_finish_hsps), dim3(sm_count), dim3(kEpiThreads), args,
                                       sizeof(EpiSmem), st);
}

}  // namespace gxy
