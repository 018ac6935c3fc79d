// gxy_input.cu -- FASTA and 2bit input straight into device sequences.
//
// The reference parses on the host byte by byte and packs with
// PackedSeq::push_ascii (src/sequences.rs:338-377, src/bit2.rs:73-163).
// Here the host only walks the structure (FASTA header lines; 2bit index,
// N-block and mask-block lists) and the per-base work runs on the device:
//  - FASTA: the file goes to the device once; a pass over tiles of 4 KB counts
//    the bytes that are neither ASCII whitespace nor of a header line, a second one
//    gathers them, and the ASCII packer encodes each record's (codes, valid, soft
//    mask).
//  - 2bit: each record's packed DNA goes to the device as is; one thread per
//    32 positions reverses the 2bit byte order, remaps T/C/A/G = 0/1/2/3 to
//    the PackedSeq codes A/C/G/T = 0/1/2/3, and applies the N and mask blocks
//    (N: invalid, code 0, never masked; mask: soft-masked).
// The results equal the reference's parse followed by PackedSeq::from_ascii,
// bit for bit (the ASCII the reference decodes 2bit into only ever holds
// T/C/A/G/N/t/c/a/g).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "gxy_engine.cuh"
#include "gxy_radix.cuh"

using namespace gxy;

namespace gxy {
gxy_status dseq_alloc(gxy_ctx* ctx, uint64_t len, gxy_dseq** out, cudaStream_t st);
void dseq_destroy(gxy_dseq* s);
}

namespace gxy {

namespace {

// u8::is_ascii_whitespace: space, tab, LF, FF, CR.
__device__ __forceinline__ bool ascii_ws(uint8_t b) {
    return b == ' ' || b == '\t' || b == '\n' || b == '\f' || b == '\r';
}

constexpr uint32_t kFastaTile = 4096;
constexpr int kFastaThreads = 256;
static_assert(kFastaTile == 16 * kFastaThreads, "16 bytes a thread");

// First header pair with end > p, of pairs [lo, hi) (sorted, disjoint).
__device__ __forceinline__ uint32_t header_after(const uint64_t* hdr, uint32_t lo, uint32_t hi, uint64_t p) {
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (hdr[2 * mid + 1] > p) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Bit k: byte i0 + k (i0 a multiple of 16, the buffer padded to one) is a base.
// [first, last): the headers that may lie there.
__device__ __forceinline__ uint32_t fasta_bases(const uint8_t* bytes, uint64_t n, uint64_t i0, const uint64_t* hdr,
                                                uint32_t first, uint32_t last, uint4& v) {
    if (i0 >= n) return 0;
    v = *reinterpret_cast<const uint4*>(bytes + i0);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t keep = 0;
#pragma unroll
    for (uint32_t k = 0; k < 16; k++) keep |= (ascii_ws((uint8_t)(w[k >> 2] >> (8 * (k & 3)))) ? 0u : 1u) << k;
    if (n - i0 < 16) keep &= (1u << (n - i0)) - 1;
    for (uint32_t h = header_after(hdr, first, last, i0); h < last && hdr[2 * h] < i0 + 16; h++) {
        const uint32_t a = hdr[2 * h] > i0 ? (uint32_t)(hdr[2 * h] - i0) : 0u;
        const uint32_t b = hdr[2 * h + 1] < i0 + 16 ? (uint32_t)(hdr[2 * h + 1] - i0) : 16u;
        keep &= ~(((1u << b) - 1) & ~((1u << a) - 1));
    }
    return keep;
}

// The bases of every tile: counted (out null), or gathered from offset[tile] on.
// What bounds it is the bytes, read twice (from L2 the second time) and written
// once.  A keep flag and a 4-byte offset for each byte took 11 bytes of traffic a
// byte and five times its memory: 0.21 ms for 20 MB, against 0.06 (both passes, the
// scan of the tile counts and the records' bounds).
__global__ __launch_bounds__(kFastaThreads) void k_fasta_tiles(const uint8_t* __restrict__ bytes, uint64_t n,
                                                               const uint64_t* __restrict__ hdr, uint32_t n_hdr,
                                                               uint32_t* count, const uint32_t* offset, uint8_t* out) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_total, s_first, s_last;
    __shared__ uint8_t s_out[kFastaTile];
    const uint64_t tiles = (n + kFastaTile - 1) / kFastaTile;
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint64_t t0 = t * kFastaTile;
        if (threadIdx.x == 0) s_first = header_after(hdr, 0, n_hdr, t0);
        if (threadIdx.x == 32) {   // the first that starts past the tile
            uint32_t lo = 0, hi = n_hdr;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (hdr[2 * mid] >= t0 + kFastaTile) hi = mid;
                else lo = mid + 1;
            }
            s_last = lo;
        }
        __syncthreads();
        uint4 v = make_uint4(0, 0, 0, 0);
        const uint32_t keep = fasta_bases(bytes, n, t0 + 16 * threadIdx.x, hdr, s_first, s_last, v);
        uint32_t at = block_excl_scan<kFastaThreads>(__popc(keep), s_warp, &s_total);
        if (!out) {
            if (threadIdx.x == 0) count[t] = s_total;
        } else {
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (uint32_t k = 0; k < 16; k++)
                if ((keep >> k) & 1u) s_out[at++] = (uint8_t)(w[k >> 2] >> (8 * (k & 3)));
            __syncthreads();
            uint8_t* const o = out + offset[t];
            for (uint32_t i = threadIdx.x; i < s_total; i += kFastaThreads) o[i] = s_out[i];
        }
        __syncthreads();
    }
}

// Bases before position at[i], one warp each.
__global__ void k_fasta_offsets_at(const uint8_t* __restrict__ bytes, uint64_t n, const uint64_t* __restrict__ hdr,
                                   uint32_t n_hdr, const uint32_t* __restrict__ offset, const uint64_t* __restrict__ at,
                                   uint32_t n_at, uint32_t* out) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n_at; i += (gridDim.x * blockDim.x) >> 5) {
        const uint64_t p = at[i], t = p / kFastaTile;
        uint32_t c = 0;
        for (uint64_t x = t * kFastaTile + 16 * lane; x < p; x += 512) {
            uint4 v;
            uint32_t keep = fasta_bases(bytes, n, x, hdr, 0, n_hdr, v);
            if (p - x < 16) keep &= (1u << (p - x)) - 1;
            c += __popc(keep);
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) out[i] = offset[t] + c;
    }
}

// Positions [32w, 32w + 32) of one 2bit record.  Blocks are sorted, disjoint
// (start, end) pairs; the ones that meet this word are found by binary search.
__device__ __forceinline__ uint32_t range_bits(const uint32_t* r, uint32_t nr, uint64_t p0) {
    uint32_t lo = 0, hi = nr;   // first range with end > p0
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (r[2 * mid + 1] > p0) hi = mid;
        else lo = mid + 1;
    }
    uint32_t bits = 0;
    for (uint32_t k = lo; k < nr && r[2 * k] < p0 + 32; k++) {
        const uint64_t a = r[2 * k] > p0 ? r[2 * k] - p0 : 0;
        const uint64_t b = r[2 * k + 1] - p0 < 32 ? r[2 * k + 1] - p0 : 32;
        if (b > a) bits |= (uint32_t)((b - a >= 32 ? 0xffffffffull : ((1ull << (b - a)) - 1)) << a);
    }
    return bits;
}

__global__ void k_2bit_decode(const uint8_t* __restrict__ packed, uint64_t len, const uint32_t* nblk, uint32_t n_n,
                              const uint32_t* mblk, uint32_t n_m, uint64_t* codes, uint32_t* valid,
                              uint32_t* mask) {
    // 2bit byte -> PackedSeq byte: four bases, first base in the high bits
    // there and in the low bits here; T C A G (0 1 2 3) -> 3 1 0 2.
    __shared__ uint8_t s_lut[256];
    for (int b = threadIdx.x; b < 256; b += blockDim.x) {
        const uint8_t remap[4] = {3, 1, 0, 2};
        uint8_t o = 0;
        for (int k = 0; k < 4; k++) o |= (uint8_t)(remap[(b >> (6 - 2 * k)) & 3] << (2 * k));
        s_lut[b] = o;
    }
    __syncthreads();
    const uint64_t nw = (len + 31) / 32;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t p0 = w * 32;
        const uint32_t present = len - p0 >= 32 ? 0xffffffffu : (uint32_t)((1ull << (len - p0)) - 1);
        const uint32_t nbits = range_bits(nblk, n_n, p0);
        const uint32_t v = present & ~nbits;
        const uint32_t m = range_bits(mblk, n_m, p0) & v;
        uint64_t c = 0;
        const uint64_t nbytes = (len + 3) / 4;
        for (int k = 0; k < 8; k++) {
            const uint64_t j = w * 8 + k;
            if (j < nbytes) c |= (uint64_t)s_lut[packed[j]] << (8 * k);
        }
        // Invalid positions (N, and past the end) carry code 0 (encode_base).
        uint64_t keepc = 0;
        for (int k = 0; k < 32; k++)
            if ((v >> k) & 1u) keepc |= 3ull << (2 * k);
        codes[kPad / 32 + w] = c & keepc;
        valid[kPad / 32 + w] = v;
        mask[kPad / 32 + w] = m;
    }
}

struct Reader {   // the reference's Cursor (src/bit2.rs:166-215)
    const uint8_t* b;
    uint64_t n, pos;
    bool be;
    bool ok = true;
    uint64_t need_at = 0, need = 0;
    bool take(uint64_t k) {
        if (!ok) return false;
        if (pos + k > n) {
            ok = false;
            need_at = pos;
            need = k;
            return false;
        }
        return true;
    }
    uint32_t u32() {
        if (!take(4)) return 0;
        uint32_t x;
        memcpy(&x, b + pos, 4);
        pos += 4;
        if (be) x = __builtin_bswap32(x);
        return x;
    }
    uint8_t u8() {
        if (!take(1)) return 0;
        return b[pos++];
    }
};

gxy_status fail_set(gxy_seq_set* out, const std::string& msg, gxy_status s) {
    gxy_seq_set_free(out);
    set_error(msg);
    return s;
}

gxy_status alloc_set(gxy_seq_set* out, uint64_t n) {
    out->n = n;
    out->seqs = static_cast<gxy_dseq**>(calloc(std::max<uint64_t>(n, 1), sizeof(gxy_dseq*)));
    out->names = static_cast<char**>(calloc(std::max<uint64_t>(n, 1), sizeof(char*)));
    if (!out->seqs || !out->names) return GXY_ENOMEM;
    return GXY_OK;
}

char* dup_name(const uint8_t* p, uint64_t k) {
    char* s = static_cast<char*>(malloc(k + 1));
    if (s) {
        memcpy(s, p, k);
        s[k] = 0;
    }
    return s;
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

}  // namespace

}  // namespace gxy

extern "C" {

void gxy_seq_set_free(gxy_seq_set* set) {
    if (!set) return;
    for (uint64_t i = 0; i < set->n; i++) {
        if (set->seqs && set->seqs[i]) dseq_destroy(set->seqs[i]);
        if (set->names) free(set->names[i]);
    }
    free(set->seqs);
    free(set->names);
    set->seqs = nullptr;
    set->names = nullptr;
    set->n = 0;
}

gxy_status gxy_parse_fasta(gxy_ctx* ctx, const uint8_t* bytes, uint64_t n, gxy_seq_set* out) {
    if (!ctx || (!bytes && n) || !out) return GXY_EINVAL;
    memset(out, 0, sizeof(*out));
    if (n >= (1ull << 32)) {
        set_error("FASTA input of 4 GiB or more is not supported");
        return GXY_EUNSUPPORTED;
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess) return GXY_ECUDA;
    // Header lines: a line (split at LF) whose first byte is '>' (src/sequences.rs:354).
    // Line i starts after the i-th LF.  Empty lines are skipped by the
    // reference; they hold no bytes here either.
    // Line starts with a '>' are looked for while the bytes go to the device.
    uint8_t* dbytes = nullptr;
    WorkerLease L(ctx);
    if (!L.w) return L.err;
    Worker* W = L.w;
    cudaStream_t st = W->st;
    auto failed = [&](gxy_status s) {
        if (dbytes) cudaFreeAsync(dbytes, st);
        cudaStreamSynchronize(st);
        return s;
    };
    std::vector<uint64_t> at;
    std::mutex at_mu;
    auto scan = [&](size_t lo, size_t hi) {
        std::vector<uint64_t> mine;
        for (uint64_t pos = lo; pos < hi;) {
            const void* gt = memchr(bytes + pos, '>', hi - pos);
            if (!gt) break;
            const uint64_t i = static_cast<const uint8_t*>(gt) - bytes;
            if (i == 0 || bytes[i - 1] == '\n') mine.push_back(i);
            pos = i + 1;
        }
        std::lock_guard<std::mutex> g(at_mu);
        at.insert(at.end(), mine.begin(), mine.end());
    };
    cudaError_t e = cudaMallocAsync((void**)&dbytes, (n + 31) & ~(uint64_t)15, st);
    const CopyPiece piece{const_cast<uint8_t*>(bytes), dbytes, n};
    if (e == cudaSuccess) e = host_copy(ctx, &piece, 1, false, st, scan);
    if (e != cudaSuccess) {
        set_error(std::string("FASTA bytes to the device: ") + cudaGetErrorString(e));
        return failed(e == cudaErrorMemoryAllocation ? GXY_ENOMEM : GXY_ECUDA);
    }
    std::sort(at.begin(), at.end());
    std::vector<uint64_t> hdr;          // header line [start, end) pairs, end excludes the LF
    std::vector<std::string> names;
    for (const uint64_t i : at) {
        const void* lf = memchr(bytes + i, '\n', n - i);
        const uint64_t end = lf ? (uint64_t)(static_cast<const uint8_t*>(lf) - bytes) : n;
        // The name: the first whitespace-delimited token after '>'.
        uint64_t a = i + 1;
        auto ws = [](uint8_t c) { return c == ' ' || c == '\t' || c == '\n' || c == '\f' || c == '\r'; };
        while (a < end && ws(bytes[a])) a++;
        uint64_t b = a;
        while (b < end && !ws(bytes[b])) b++;
        if (b == a) {
            uint64_t line = 1;
            for (uint64_t k = 0; k < i; k++) line += bytes[k] == '\n';
            set_error("empty FASTA header at line " + std::to_string(line) + " (src/sequences.rs:357-361)");
            return failed(GXY_EINVAL);
        }
        names.emplace_back(reinterpret_cast<const char*>(bytes + a), b - a);
        hdr.push_back(i);
        hdr.push_back(end);
    }
    const uint64_t nrec = names.size();
    if (alloc_set(out, nrec) != GXY_OK) return failed(fail_set(out, "host allocation of the sequence set", GXY_ENOMEM));
    for (uint64_t r = 0; r < nrec; r++) {
        out->names[r] = dup_name(reinterpret_cast<const uint8_t*>(names[r].data()), names[r].size());
        if (!out->names[r]) return failed(fail_set(out, "host allocation of FASTA names", GXY_ENOMEM));
    }
    if (nrec == 0) return failed(GXY_OK);   // no header: the reference returns no sequences
    // Device buffers: file bytes, tile counts and offsets, gathered bases.
    const uint64_t tiles = (n + kFastaTile - 1) / kFastaTile;
    uint8_t* dcomp = nullptr;
    uint32_t *dcnt = nullptr, *doff = nullptr;
    uint64_t* dhdr = nullptr;
    uint64_t* dat = nullptr;
    uint32_t* dbound = nullptr;
    auto release = [&]() {
        cudaFreeAsync(dbytes, st);
        cudaFreeAsync(dcnt, st);
        cudaFreeAsync(dcomp, st);
        cudaFreeAsync(doff, st);
        cudaFreeAsync(dhdr, st);
        cudaFreeAsync(dat, st);
        cudaFreeAsync(dbound, st);
        cudaStreamSynchronize(st);
    };
    e = cudaMallocAsync((void**)&dcnt, (tiles + 1) * 4, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&dcomp, n, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&doff, (tiles + 1) * 4, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&dhdr, hdr.size() * 8, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&dat, (nrec + 1) * 8, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&dbound, (nrec + 1) * 4, st);
    if (e != cudaSuccess) {
        release();
        return fail_set(out, std::string("FASTA device buffers: ") + cudaGetErrorString(e), GXY_ENOMEM);
    }
    // Record r's bases are those kept in [boundary r, boundary r + 1): record
    // 0 also takes bases before the first header, as the reference does.
    at.assign(nrec + 1, 0);
    for (uint64_t r = 1; r < nrec; r++) at[r] = hdr[2 * r];
    at[nrec] = n;
    e = cudaMemcpyAsync(dhdr, hdr.data(), hdr.size() * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dat, at.data(), at.size() * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        const int grid = (int)std::min<uint64_t>(tiles, (uint64_t)ctx->sm_count * 8);
        count_launch(3);
        k_fasta_tiles<<<grid, kFastaThreads, 0, st>>>(dbytes, n, dhdr, (uint32_t)nrec, dcnt, nullptr, nullptr);
        scan_u32(dcnt, doff, nullptr, tiles, tiles, true, nullptr, W->ps, st);
        k_fasta_tiles<<<grid, kFastaThreads, 0, st>>>(dbytes, n, dhdr, (uint32_t)nrec, nullptr, doff, dcomp);
        k_fasta_offsets_at<<<(int)std::min<uint64_t>((nrec + 8) / 8, 148 * 8), 256, 0, st>>>(
            dbytes, n, dhdr, (uint32_t)nrec, doff, dat, (uint32_t)(nrec + 1), dbound);
    }
    std::vector<uint32_t> bound(nrec + 1);
    if (e == cudaSuccess) e = cudaMemcpyAsync(bound.data(), dbound, (nrec + 1) * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    for (uint64_t r = 0; r < nrec && e == cudaSuccess; r++) {
        const uint64_t len = bound[r + 1] - bound[r];
        gxy_status s = dseq_alloc(ctx, len, &out->seqs[r], st);
        if (s != GXY_OK) {
            release();
            gxy_seq_set_free(out);
            return s;
        }
        launch_pack_ascii(dcomp + bound[r], len, out->seqs[r]->codes, out->seqs[r]->valid, out->seqs[r]->mask, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    release();
    if (e != cudaSuccess) return fail_set(out, std::string("FASTA parse: ") + cudaGetErrorString(e), GXY_ECUDA);
    return GXY_OK;
}

gxy_status gxy_parse_2bit(gxy_ctx* ctx, const uint8_t* bytes, uint64_t n, gxy_seq_set* out) {
    if (!ctx || (!bytes && n) || !out) return GXY_EINVAL;
    memset(out, 0, sizeof(*out));
    auto truncated = [&](const Reader& r) {
        return fail_set(out, "truncated 2bit file (needed " + std::to_string(r.need) + " bytes at offset " +
                                 std::to_string(r.need_at) + ", src/bit2.rs:51-52)",
                        GXY_EINVAL);
    };
    if (n < 4) {
        Reader r{bytes, n, 0, false};
        r.take(4);
        return truncated(r);
    }
    uint32_t m0;
    memcpy(&m0, bytes, 4);
    bool be;
    if (m0 == 0x1A412743u) be = false;
    else if (m0 == 0x4327411Au) be = true;
    else {
        char buf[64];
        snprintf(buf, sizeof buf, "not a 2bit file (magic = 0x%08x)", m0);
        set_error(buf);
        return GXY_EINVAL;
    }
    Reader r{bytes, n, 0, be};
    r.u32();
    const uint32_t version = r.u32();
    if (r.ok && version != 0) {
        set_error("unsupported 2bit version " + std::to_string(version));
        return GXY_EINVAL;
    }
    const uint32_t count = r.u32();
    r.u32();
    if (!r.ok) return truncated(r);
    std::vector<std::pair<std::string, uint32_t>> index;
    for (uint32_t i = 0; i < count; i++) {
        const uint32_t ns = r.u8();
        if (!r.take(ns)) return truncated(r);
        std::string name(reinterpret_cast<const char*>(bytes + r.pos), ns);
        r.pos += ns;
        const uint32_t off = r.u32();
        if (!r.ok) return truncated(r);
        index.emplace_back(std::move(name), off);
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess) return GXY_ECUDA;
    if (alloc_set(out, count) != GXY_OK) return fail_set(out, "host allocation of the sequence set", GXY_ENOMEM);
    for (uint32_t i = 0; i < count; i++) {
        out->names[i] = dup_name(reinterpret_cast<const uint8_t*>(index[i].first.data()), index[i].first.size());
        if (!out->names[i]) return fail_set(out, "host allocation of 2bit names", GXY_ENOMEM);
    }
    WorkerLease L(ctx);
    if (!L.w) return fail_set(out, "no worker", L.err);
    cudaStream_t st = L.w->st;
    // The structure of all records first; their packed bases go to the device together.
    struct Rec {
        uint32_t i;
        const uint8_t* packed;
        uint64_t pb, pk_at, rng_at, nn, nm;
    };
    std::vector<Rec> recs;
    std::vector<uint32_t> rng;
    uint64_t pk_bytes = 0;
    for (uint32_t i = 0; i < count; i++) {
        Reader q{bytes, n, 0, be};
        if (index[i].second > n) {
            q.need_at = 0;
            q.need = index[i].second;
            return truncated(q);
        }
        q.pos = index[i].second;
        const uint32_t dna = q.u32();
        auto blocks = [&](std::vector<uint32_t>& out_ranges) {
            const uint32_t k = q.u32();
            std::vector<uint32_t> s(k), z(k);
            for (uint32_t j = 0; j < k; j++) s[j] = q.u32();
            for (uint32_t j = 0; j < k; j++) z[j] = q.u32();
            // Sorted, merged [start, end) ranges clamped to the record.
            std::vector<std::pair<uint64_t, uint64_t>> v;
            for (uint32_t j = 0; j < k; j++) {
                const uint64_t a = std::min<uint64_t>(s[j], dna), b = std::min<uint64_t>((uint64_t)s[j] + z[j], dna);
                if (b > a) v.emplace_back(a, b);
            }
            std::sort(v.begin(), v.end());
            for (auto& x : v) {
                if (!out_ranges.empty() && x.first <= out_ranges.back()) {
                    out_ranges.back() = std::max<uint32_t>(out_ranges.back(), (uint32_t)x.second);
                } else {
                    out_ranges.push_back((uint32_t)x.first);
                    out_ranges.push_back((uint32_t)x.second);
                }
            }
        };
        std::vector<uint32_t> nr, mr;
        blocks(nr);
        blocks(mr);
        q.u32();
        const uint64_t pb = (uint64_t)(dna + 3) / 4;
        if (!q.take(pb)) return truncated(q);
        const uint8_t* packed = bytes + q.pos;
        gxy_status s = dseq_alloc(ctx, dna, &out->seqs[i], st);
        if (s != GXY_OK) {
            gxy_seq_set_free(out);
            return s;
        }
        if (dna == 0) continue;
        recs.push_back(Rec{i, packed, pb, pk_bytes, rng.size(), nr.size(), mr.size()});
        pk_bytes += (pb + 255) & ~(uint64_t)255;
        rng.insert(rng.end(), nr.begin(), nr.end());
        rng.insert(rng.end(), mr.begin(), mr.end());
    }
    if (recs.empty()) return cudaStreamSynchronize(st) == cudaSuccess ? GXY_OK : fail_set(out, "2bit decode", GXY_ECUDA);
    uint8_t* dpk = nullptr;
    uint32_t* drng = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&drng, (rng.size() + 2) * 4, st);
    if (e == cudaSuccess && !rng.empty()) e = cudaMemcpyAsync(drng, rng.data(), rng.size() * 4, cudaMemcpyHostToDevice, st);
    // All records at once, or as many at a time as the device has room for.
    uint64_t room = pk_bytes;
    for (size_t k0 = 0; e == cudaSuccess && k0 < recs.size();) {
        const uint64_t at0 = recs[k0].pk_at;
        size_t k1 = k0 + 1;
        while (k1 < recs.size() && recs[k1].pk_at + recs[k1].pb - at0 <= room) k1++;
        const uint64_t bytes_n = recs[k1 - 1].pk_at + recs[k1 - 1].pb - at0;
        e = cudaMallocAsync((void**)&dpk, bytes_n, st);
        if (e == cudaErrorMemoryAllocation && k1 - k0 > 1) {
            e = cudaSuccess;
            cudaGetLastError();
            room = bytes_n / 2;
            continue;
        }
        std::vector<CopyPiece> pieces;
        for (size_t k = k0; k < k1; k++)
            pieces.push_back({const_cast<uint8_t*>(recs[k].packed), dpk + (recs[k].pk_at - at0), recs[k].pb});
        if (e == cudaSuccess) e = host_copy(ctx, pieces.data(), (int)pieces.size(), false, st);
        for (size_t k = k0; e == cudaSuccess && k < k1; k++) {
            const Rec& x = recs[k];
            gxy_dseq* d = out->seqs[x.i];
            const uint64_t nw = (d->len + 31) / 32;
            count_launch();
            k_2bit_decode<<<(unsigned)std::min<uint64_t>((nw + 255) / 256, (uint64_t)ctx->sm_count * 16), 256, 0, st>>>(
                dpk + (x.pk_at - at0), d->len, drng + x.rng_at, (uint32_t)(x.nn / 2), drng + x.rng_at + x.nn,
                (uint32_t)(x.nm / 2), d->codes, d->valid, d->mask);
        }
        if (dpk) cudaFreeAsync(dpk, st);
        dpk = nullptr;
        k0 = k1;
    }
    const cudaError_t synced = cudaStreamSynchronize(st);   // the host buffers die here
    if (e == cudaSuccess) e = synced;
    if (drng) cudaFreeAsync(drng, st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail_set(out, std::string("2bit decode: ") + cudaGetErrorString(e), GXY_ECUDA);
    if (cudaStreamSynchronize(st) != cudaSuccess) return fail_set(out, "2bit decode", GXY_ECUDA);
    return GXY_OK;
}

}  // extern "C"
