// grg_format.cu -- the reference's compressed edge stream on the device.
//
// The reference spills partitions as a CSR byte stream (storeElements_c /
// elements2Edges, src/main.cpp:510-596) and reads them back with
// readElements_c / edges2Elements (src/main.cpp:335-445): per source vertex in
// order, per label 1..L, the row's destinations ascending, 5 bytes each
// (little-endian uint32 destination, uint8 label id), with the row lengths kept
// in a separate degree array. Here both directions run on the device:
//   records -> stream: sort the element records by (row, label, base) with a
//     64-bit radix sort, prefix-sum their popcounts into edge offsets, then
//     a warp per 32 elements gathers their edges' bytes and stores them whole;
//   stream -> edges: prefix-sum the row lengths, then each thread expands a
//     run of 16 consecutive edges, finding its first row by binary search.
// Both are HBM-streaming passes over the records / the stream.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <vector>

#include "grg_format.h"

namespace {

constexpr uint32_t KEY_BITS = 32;          // word 6: label << 25 | base
constexpr uint32_t EIDS = 192;
constexpr uint32_t BASE_MASK = (1u << 25) - 1;
constexpr uint32_t EXPAND_RUN = 16;        // edges per thread in the expansion

int grid_of(uint64_t n, int block)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t g = (n + block - 1) / block, cap = (uint64_t)(sms > 0 ? sms : 1) * 16;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

__global__ void k_fmt_keys(const uint4 *__restrict__ rec, uint64_t n, uint32_t v_begin, uint64_t *key, uint32_t *idx)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 b = rec[2 * i + 1];
        key[i] = ((uint64_t)(b.w - v_begin) << KEY_BITS) | b.z;
        idx[i] = (uint32_t)i;
    }
}

__device__ __forceinline__ uint32_t popc6(uint4 a, uint4 b)
{
    return __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w) + __popc(b.x) + __popc(b.y);
}

// Edge count of each sorted element (for the offsets) and of each row.
__global__ void k_fmt_count(const uint4 *__restrict__ rec, const uint32_t *__restrict__ idx, uint64_t n,
                            uint32_t v_begin, uint64_t *cnt, uint32_t *degree)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t j = idx[i];
        const uint4 a = rec[2 * j], b = rec[2 * j + 1];
        const uint32_t c = popc6(a, b);
        cnt[i] = c;
        if (c) atomicAdd(&degree[b.w - v_begin], c);
    }
}

// The edge bytes of 32 consecutive sorted elements a warp: 5 bytes an edge, ids ascending.
//
// Bound: the stream's own bytes. The elements' edges are contiguous in the stream, so a warp gathers
// them in shared memory, at the stream's alignment, and stores whole 16-byte vectors; the bytes of the
// first and the last vector, which neighbours share, go out singly. Groups with many edges (16 an
// element in the mean) go one element at a time, a lane a bit of each bitmap word; sparser ones a lane
// an element. A thread per bitmap word that stored its bytes one by one, 5 stores an edge, scattered,
// took 6.4 ms for 160.7M edges in 1.0M elements (0.13 TB/s); this takes 0.30 ms (2.7 TB/s).
constexpr int WRITE_WARPS = 8;
constexpr uint32_t WRITE_EDGES = 640;      // edges a warp gathers before it stores them
constexpr uint32_t WRITE_DENSE = 32 * 16;  // edges of a group from which elements go one at a time
static_assert(WRITE_DENSE <= WRITE_EDGES && EIDS <= WRITE_EDGES, "a sparse group, or an element, fits the buffer");

__device__ __forceinline__ void put_edge(uint8_t *q, uint32_t dst, uint32_t lab)
{
    q[0] = (uint8_t)dst;
    q[1] = (uint8_t)(dst >> 8);
    q[2] = (uint8_t)(dst >> 16);
    q[3] = (uint8_t)(dst >> 24);
    q[4] = (uint8_t)lab;
}

// The warp's n bytes at buf + (dst mod 16) go to dst.
__device__ __forceinline__ void store_bytes(const uint8_t *buf, uint8_t *dst, uint32_t n, uint32_t lane)
{
    const uint32_t pad = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 15u);
    uint8_t *base = dst - pad;                       // 16-byte aligned; [pad, pad + n) is ours
    const uint32_t end = pad + n, v0 = (pad + 15u) >> 4, v1 = end >> 4;
    for (uint32_t v = v0 + lane; v < v1; v += 32)
        reinterpret_cast<uint4 *>(base)[v] = reinterpret_cast<const uint4 *>(buf)[v];
    const uint32_t h = min(end, v0 * 16u);           // bytes before the first whole vector
    if (pad + lane < h) base[pad + lane] = buf[pad + lane];
    const uint32_t u = max(h, v1 * 16u);             // and after the last
    if (u + lane < end) base[u + lane] = buf[u + lane];
}

__global__ void __launch_bounds__(WRITE_WARPS * 32) k_fmt_write(const uint4 *__restrict__ rec,
                                                                const uint32_t *__restrict__ idx,
                                                                const uint64_t *__restrict__ off, uint64_t n,
                                                                uint8_t *out)
{
    __shared__ __align__(16) uint8_t sbuf[WRITE_WARPS][WRITE_EDGES * 5 + 16];
    const uint32_t lane = threadIdx.x & 31;
    uint8_t *buf = sbuf[threadIdx.x >> 5];
    const uint64_t groups = (n + 31) / 32, step = (uint64_t)gridDim.x * WRITE_WARPS;
    for (uint64_t gi = blockIdx.x * (uint64_t)WRITE_WARPS + (threadIdx.x >> 5); gi < groups; gi += step) {
        const uint64_t i = gi * 32 + lane;
        uint4 a = make_uint4(0, 0, 0, 0), b = a;
        uint64_t o = 0;
        if (i < n) {
            const uint32_t j = idx[i];
            a = rec[2 * (uint64_t)j];
            b = rec[2 * (uint64_t)j + 1];
            o = off[i];
        }
        const uint32_t c = popc6(a, b), total = __reduce_add_sync(0xffffffffu, c);
        const uint32_t lab = b.z >> 25, first = (b.z & BASE_MASK) * EIDS;
        const uint32_t words[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
        uint8_t *at = out + __shfl_sync(0xffffffffu, o, 0) * 5;      // where the buffer's bytes go
        uint32_t pad = (uint32_t)(reinterpret_cast<uintptr_t>(at) & 15u);
        if (total < WRITE_DENSE) {
            uint8_t *q = buf + pad + (uint32_t)(o - __shfl_sync(0xffffffffu, o, 0)) * 5;
#pragma unroll
            for (int w = 0; w < 6; w++)
                for (uint32_t bits = words[w]; bits; bits &= bits - 1, q += 5)
                    put_edge(q, first + w * 32 + (__ffs(bits) - 1), lab);
            __syncwarp();
            store_bytes(buf, at, total * 5, lane);
            __syncwarp();
            continue;
        }
        uint32_t held = 0;                                           // edges in the buffer
        for (uint32_t e = 0; e < 32; e++) {
            const uint32_t ce = __shfl_sync(0xffffffffu, c, e);
            if (held + ce > WRITE_EDGES) {
                __syncwarp();
                store_bytes(buf, at, held * 5, lane);
                __syncwarp();
                at += (uint64_t)held * 5;
                pad = (uint32_t)(reinterpret_cast<uintptr_t>(at) & 15u);
                held = 0;
            }
            const uint32_t le = __shfl_sync(0xffffffffu, lab, e), fe = __shfl_sync(0xffffffffu, first, e) + lane;
#pragma unroll
            for (int w = 0; w < 6; w++) {
                const uint32_t bits = __shfl_sync(0xffffffffu, words[w], e);
                if ((bits >> lane) & 1u)
                    put_edge(buf + pad + (held + __popc(bits & ((1u << lane) - 1u))) * 5, fe + w * 32, le);
                held += __popc(bits);
            }
        }
        __syncwarp();
        store_bytes(buf, at, held * 5, lane);
        __syncwarp();
    }
}

// roff[r] = degree[r] widened (roff[nrows] = 0), for the exclusive scan.
__global__ void k_fmt_widen(const uint32_t *__restrict__ degree, uint32_t nrows, uint64_t *roff)
{
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r <= nrows; r += (uint64_t)gridDim.x * blockDim.x)
        roff[r] = r < nrows ? degree[r] : 0;
}

// A block's tile of EXPAND_TILE runs: the stream's bytes in shared memory, a run's 20 words at a stride
// of 21 (so that a warp's reads of word w of 32 runs hit 32 banks), and the rows that the tile spans.
constexpr uint32_t EXPAND_TILE = 256;                    // runs (threads) a block
constexpr uint32_t RUN_WORDS = EXPAND_RUN * 5 / 4;       // 20
static_assert(EXPAND_RUN % 4 == 0, "4 edges are 5 words");
struct RunTile {
    uint32_t word[EXPAND_TILE * (RUN_WORDS + 1)];
    uint32_t row[2];                                     // of the tile's first and last edge
};

// Last row with start[row] <= e among [lo, hi): start[lo] <= e < start[hi].
__device__ __forceinline__ uint32_t row_of(const uint64_t *__restrict__ start, uint32_t lo, uint32_t hi, uint64_t e)
{
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (start[mid] <= e) lo = mid; else hi = mid;
    }
    return lo;
}

// Brings in the tile whose first edge is e0 < m. The whole block calls it.
__device__ void load_runs(RunTile &s, const uint8_t *__restrict__ bytes, const uint64_t *__restrict__ start,
                          uint32_t nrows, uint64_t m, uint64_t e0)
{
    const uint64_t e1 = min(m, e0 + (uint64_t)EXPAND_TILE * EXPAND_RUN);
    const uint32_t n = (uint32_t)(e1 - e0) * 5;
    const uint8_t *src = bytes + e0 * 5;                 // e0 * 5: a multiple of 80
    auto put = [&](uint32_t w, uint32_t v) { s.word[w / RUN_WORDS * (RUN_WORDS + 1) + w % RUN_WORDS] = v; };
    uint32_t done = 0;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        for (uint32_t v = threadIdx.x; v < n / 16; v += EXPAND_TILE) {
            const uint4 x = reinterpret_cast<const uint4 *>(src)[v];
            put(4 * v, x.x);
            put(4 * v + 1, x.y);
            put(4 * v + 2, x.z);
            put(4 * v + 3, x.w);
        }
        done = n / 16 * 4;
    }
    for (uint32_t w = done + threadIdx.x; 4 * w < n; w += EXPAND_TILE) {   // the tail, or a stream at an odd address
        uint32_t x = 0;
        for (uint32_t k = 0; k < 4 && 4 * w + k < n; k++) x |= (uint32_t)src[4 * w + k] << (8 * k);
        put(w, x);
    }
    if (threadIdx.x == 0) s.row[0] = row_of(start, 0, nrows, e0);
    if (threadIdx.x == 32) s.row[1] = row_of(start, 0, nrows, e1 - 1);
    __syncthreads();
}

// Walks the consecutive edges of the tile's run threadIdx.x: f(row, label, dst,
// starts) per edge, where `starts` says the edge begins a new element -- the
// first edge of a row, or one whose label or 192-id base differs from the edge
// before it (the stream is sorted by label, then destination, within a row).
// The run's first row is the last r with start[r] <= its first edge (rows of
// length 0 share their start with the next row).
//
// Bound: the stream's bytes, read once a pass, and about 20 instructions an edge. Bytes come in as
// 16-byte vectors and are taken as 5 words per 4 edges; a run's row is searched among the tile's rows.
// 160.7M edges of 200,000 rows: 0.40 ms the first pass, 0.50 ms the second (0.61 and 1.09 ms with byte
// loads at a stride of 80 and a search over all rows by every run).
template <class F>
__device__ __forceinline__ void walk_run(const RunTile &s, const uint8_t *__restrict__ bytes,
                                         const uint64_t *__restrict__ start, uint64_t m, uint64_t tile_e0, F f)
{
    const uint64_t e0 = tile_e0 + threadIdx.x * EXPAND_RUN;
    if (e0 >= m) return;
    const uint32_t *wd = s.word + threadIdx.x * (RUN_WORDS + 1);
    uint32_t r = row_of(start, s.row[0], s.row[1] + 1, e0), plab = 0, pbase = 0;
    uint64_t next = start[r + 1];                // start[nrows] = m is beyond every edge
    bool have_prev = false;
    if (e0 > start[r]) {                         // the edge before e0 is in the same row
        uint32_t dst;
        if (threadIdx.x) {                       // the run before ends in its words 18 and 19
            const uint32_t *pw = wd - (RUN_WORDS + 1) + RUN_WORDS - 2;
            dst = (pw[0] >> 24) | (pw[1] << 8);
            plab = pw[1] >> 24;
        } else {
            const uint8_t *q = bytes + (e0 - 1) * 5;
            dst = (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16) | ((uint32_t)q[3] << 24);
            plab = q[4];
        }
        pbase = dst / EIDS;
        have_prev = true;
    }
    const uint32_t ne = (uint32_t)min((uint64_t)EXPAND_RUN, m - e0);
    for (uint32_t g = 0; g < ne; g += 4) {
        uint32_t x[5];
#pragma unroll
        for (int k = 0; k < 5; k++) x[k] = wd[g / 4 * 5 + k];   // beyond the stream's end: read, not used
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (g + k >= ne) break;
            const uint32_t dst = k ? __funnelshift_r(x[k], x[k + 1], 8 * k) : x[0];
            const uint32_t lab = (x[k + 1] >> (8 * k)) & 0xFFu, base = dst / EIDS;
            while (next <= e0 + g + k) {
                r++;
                next = start[r + 1];
                have_prev = false;
            }
            f(r, lab, dst, !have_prev || lab != plab || base != pbase);
            have_prev = true;
            plab = lab;
            pbase = base;
        }
    }
}

// Pass 1: elements starting in each run; labels outside 1..L and destinations
// >= num_vars set bits 1 and 2 of *bad.
__global__ void __launch_bounds__(EXPAND_TILE) k_fmt_starts(const uint8_t *__restrict__ bytes,
                                                            const uint64_t *__restrict__ start, uint32_t nrows,
                                                            uint64_t m, uint32_t num_vars, uint32_t L,
                                                            uint64_t *run_cnt, unsigned *bad)
{
    __shared__ RunTile s;
    const uint64_t runs = (m + EXPAND_RUN - 1) / EXPAND_RUN;
    for (uint64_t u0 = blockIdx.x * (uint64_t)EXPAND_TILE; u0 < runs; u0 += (uint64_t)gridDim.x * EXPAND_TILE) {
        load_runs(s, bytes, start, nrows, m, u0 * EXPAND_RUN);
        uint32_t c = 0;
        unsigned b = 0;
        walk_run(s, bytes, start, m, u0 * EXPAND_RUN, [&](uint32_t, uint32_t lab, uint32_t dst, bool starts) {
            if (lab - 1u >= L) b |= 1u;
            if (dst >= num_vars) b |= 2u;
            c += starts;
        });
        if (u0 + threadIdx.x < runs) run_cnt[u0 + threadIdx.x] = c;
        if (b) atomicOr(bad, b);
        __syncthreads();
    }
}

// Pass 2: ORs each edge's bit into its element (id = elements started before
// it); the element's first edge writes its key and row. Bits gather in a
// register while consecutive edges share a word.
__global__ void __launch_bounds__(EXPAND_TILE) k_fmt_build(const uint8_t *__restrict__ bytes,
                                                           const uint64_t *__restrict__ start, uint32_t nrows,
                                                           uint64_t m, uint32_t v_begin,
                                                           const uint64_t *__restrict__ run_off, uint32_t *rec)
{
    __shared__ RunTile s;
    const uint64_t runs = (m + EXPAND_RUN - 1) / EXPAND_RUN;
    for (uint64_t u0 = blockIdx.x * (uint64_t)EXPAND_TILE; u0 < runs; u0 += (uint64_t)gridDim.x * EXPAND_TILE) {
        load_runs(s, bytes, start, nrows, m, u0 * EXPAND_RUN);
        // the element the run's first edge continues, if it does
        uint64_t id = (u0 + threadIdx.x < runs ? run_off[u0 + threadIdx.x] : 0) - 1;
        uint64_t at = 0;                         // the word of rec that `bits` goes to
        uint32_t bits = 0;
        walk_run(s, bytes, start, m, u0 * EXPAND_RUN, [&](uint32_t r, uint32_t lab, uint32_t dst, bool starts) {
            if (starts) {
                id++;
                rec[id * 8 + 6] = (lab << 25) | (dst / EIDS);
                rec[id * 8 + 7] = v_begin + r;
            }
            const uint32_t o = dst % EIDS;
            const uint64_t w = id * 8 + (o >> 5);
            if (w != at) {
                if (bits) atomicOr(&rec[at], bits);
                at = w;
                bits = 0;
            }
            bits |= 1u << (o & 31);
        });
        if (bits) atomicOr(&rec[at], bits);
        __syncthreads();
    }
}

__global__ void k_fmt_fill(uint32_t *p, uint64_t n, uint32_t v)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

int bit_width(uint64_t x)
{
    int b = 0;
    while (x) { b++; x >>= 1; }
    return b;
}

}  // namespace

#define FMT_CHECK(x)                      \
    do {                                  \
        cudaError_t e_ = (x);             \
        if (e_ != cudaSuccess) {          \
            err = e_;                     \
            goto done;                    \
        }                                 \
    } while (0)

cudaError_t grg_fmt_records_to_csr5(const uint4 *rec, uint64_t n, uint32_t v_begin, uint32_t nrows,
                                    uint64_t total_edges, uint8_t *out_bytes, uint32_t *degree, cudaStream_t s)
{
    cudaError_t err = cudaSuccess;
    uint64_t *key = nullptr, *cnt = nullptr;
    uint32_t *idx = nullptr;
    void *tmp = nullptr;
    size_t tsort = 0, tscan = 0;
    const int end_bit = (int)KEY_BITS + (nrows > 1 ? bit_width(nrows - 1) : 0);
    FMT_CHECK(cudaMemsetAsync(degree, 0, (size_t)nrows * 4, s));
    if (!n) return cudaStreamSynchronize(s);
    // key[0..n) / key[n..2n): radix sort input and output; idx the same; cnt then offsets
    FMT_CHECK(cudaMalloc(&key, n * 16));
    FMT_CHECK(cudaMalloc(&idx, n * 8));
    FMT_CHECK(cudaMalloc(&cnt, n * 16));
    FMT_CHECK(cub::DeviceRadixSort::SortPairs(nullptr, tsort, key, key + n, idx, idx + n, n, 0, end_bit, s));
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, tscan, cnt, cnt + n, n, s));
    FMT_CHECK(cudaMalloc(&tmp, tsort > tscan ? tsort : tscan));
    k_fmt_keys<<<grid_of(n, 256), 256, 0, s>>>(rec, n, v_begin, key, idx);
    FMT_CHECK(cub::DeviceRadixSort::SortPairs(tmp, tsort, key, key + n, idx, idx + n, n, 0, end_bit, s));
    k_fmt_count<<<grid_of(n, 256), 256, 0, s>>>(rec, idx + n, n, v_begin, cnt, degree);
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(tmp, tscan, cnt, cnt + n, n, s));
    // the stream is written only when the records' popcount is the length the caller sized it for
    {
        uint64_t last[2] = {0, 0};
        FMT_CHECK(cudaMemcpyAsync(&last[0], cnt + n - 1, 8, cudaMemcpyDeviceToHost, s));
        FMT_CHECK(cudaMemcpyAsync(&last[1], cnt + 2 * n - 1, 8, cudaMemcpyDeviceToHost, s));
        FMT_CHECK(cudaStreamSynchronize(s));
        if (last[0] + last[1] != total_edges) {
            err = cudaErrorInvalidValue;
            goto done;
        }
    }
    if (total_edges) k_fmt_write<<<grid_of((n + 31) / 32, WRITE_WARPS), WRITE_WARPS * 32, 0, s>>>(rec, idx + n, cnt + n, n, out_bytes);
    FMT_CHECK(cudaGetLastError());
    FMT_CHECK(cudaStreamSynchronize(s));
done:
    cudaFree(tmp);
    cudaFree(cnt);
    cudaFree(idx);
    cudaFree(key);
    return err;
}

cudaError_t grg_fmt_csr5_to_records(const uint8_t *bytes, uint64_t num_edges, const uint32_t *degree,
                                    uint32_t v_begin, uint32_t nrows, uint32_t num_vars, uint32_t L, uint4 *into,
                                    uint32_t *into_st, uint64_t into_cap, uint4 **recs, uint32_t **stamps,
                                    uint64_t *n_elems, uint64_t *sum, unsigned *bad, cudaStream_t s)
{
    cudaError_t err = cudaSuccess;
    uint64_t *roff = nullptr, *start = nullptr, *rcnt = nullptr, *roffs = nullptr;
    unsigned *dbad = nullptr;
    void *tmp = nullptr;
    size_t tscan = 0, tscan2 = 0;
    const uint64_t runs = (num_edges + EXPAND_RUN - 1) / EXPAND_RUN;
    uint32_t *rec = nullptr, *st = nullptr;
    if (recs) *recs = nullptr;
    if (stamps) *stamps = nullptr;
    *n_elems = 0;
    *sum = 0;
    *bad = 0;
    if (!nrows) return cudaSuccess;
    FMT_CHECK(cudaMalloc(&roff, ((uint64_t)nrows + 1) * 16));
    start = roff + nrows + 1;
    FMT_CHECK(cudaMalloc(&rcnt, (runs + 1) * 16 + 16));
    roffs = rcnt + runs + 1;
    dbad = (unsigned *)(roffs + runs + 1);
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, tscan, roff, start, (uint64_t)nrows + 1, s));
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, tscan2, rcnt, roffs, runs + 1, s));
    FMT_CHECK(cudaMalloc(&tmp, tscan > tscan2 ? tscan : tscan2));
    k_fmt_widen<<<grid_of((uint64_t)nrows + 1, 256), 256, 0, s>>>(degree, nrows, roff);
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(tmp, tscan, roff, start, (uint64_t)nrows + 1, s));
    FMT_CHECK(cudaMemcpyAsync(sum, start + nrows, 8, cudaMemcpyDeviceToHost, s));
    FMT_CHECK(cudaStreamSynchronize(s));
    if (*sum != num_edges || !num_edges) goto done;
    FMT_CHECK(cudaMemsetAsync(rcnt, 0, (runs + 1) * 8, s));
    FMT_CHECK(cudaMemsetAsync(dbad, 0, 4, s));
    k_fmt_starts<<<grid_of(runs, EXPAND_TILE), EXPAND_TILE, 0, s>>>(bytes, start, nrows, num_edges, num_vars, L, rcnt, dbad);
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(tmp, tscan2, rcnt, roffs, runs + 1, s));
    FMT_CHECK(cudaMemcpyAsync(bad, dbad, 4, cudaMemcpyDeviceToHost, s));
    FMT_CHECK(cudaMemcpyAsync(n_elems, roffs + runs, 8, cudaMemcpyDeviceToHost, s));
    FMT_CHECK(cudaStreamSynchronize(s));
    if (*bad || !*n_elems || (!into && !recs)) goto done;
    if (into) {
        if (*n_elems > into_cap) {
            err = cudaErrorInvalidValue;
            goto done;
        }
        rec = reinterpret_cast<uint32_t *>(into);
        st = into_st;
    } else {
        FMT_CHECK(cudaMalloc(&rec, *n_elems * 32));
        FMT_CHECK(cudaMalloc(&st, *n_elems * 4));
    }
    FMT_CHECK(cudaMemsetAsync(rec, 0, *n_elems * 32, s));
    k_fmt_fill<<<grid_of(*n_elems, 256), 256, 0, s>>>(st, *n_elems, 1u);
    // run u's edges belong to elements run_off[u] - 1 (continued) and run_off[u] .. run_off[u+1] - 1
    k_fmt_build<<<grid_of(runs, EXPAND_TILE), EXPAND_TILE, 0, s>>>(bytes, start, nrows, num_edges, v_begin, roffs, rec);
    FMT_CHECK(cudaGetLastError());
    FMT_CHECK(cudaStreamSynchronize(s));
    if (!into) {
        *recs = reinterpret_cast<uint4 *>(rec);
        *stamps = st;
    }
    rec = nullptr;
    st = nullptr;
done:
    if (!into) {
        cudaFree(rec);
        cudaFree(st);
    }
    cudaFree(tmp);
    cudaFree(rcnt);
    cudaFree(roff);
    return err;
}

// ------------------------------------------------------------------ columns -> rows
//
// Labels stored by destination keep, per (label, destination j), elements over
// the sources i. Their records are turned into records by source here, 192 x 192
// tiles at a time: the records of one label whose destinations share a 192-id
// block jb and whose source elements share a base ib form one tile (at most 192
// records, one per destination of the block); a warp loads the tile into shared
// memory and transposes it one 32 x 32 bit block at a time with warp ballots.

namespace {

constexpr int TILE_WARPS = 4;
constexpr uint64_t NOT_COLUMN = 1ull << 56;   // sort key of records that are copied as they are

__global__ void k_col_keys(const uint4 *__restrict__ rec, uint64_t n, unsigned long long tmask, uint64_t *key,
                           uint32_t *idx)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 b = rec[2 * i + 1];
        const uint32_t lab = b.z >> 25;
        const bool col = lab >= 1 && lab <= 63 && ((tmask >> (lab - 1)) & 1ull);
        key[i] = col ? ((uint64_t)lab << 50) | ((uint64_t)(b.w / EIDS) << 25) | (b.z & BASE_MASK) : NOT_COLUMN;
        idx[i] = (uint32_t)i;
    }
}

// head[i] = 1 where a tile starts among the first nt (column) sorted keys
__global__ void k_col_heads(const uint64_t *__restrict__ key, uint64_t nt, uint32_t *head)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nt; i += (uint64_t)gridDim.x * blockDim.x)
        head[i] = (i == 0 || key[i] != key[i - 1]) ? 1u : 0u;
}

__global__ void k_col_starts(const uint32_t *__restrict__ head, const uint32_t *__restrict__ pos, uint64_t nt,
                             uint32_t *start)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nt; i += (uint64_t)gridDim.x * blockDim.x)
        if (head[i]) start[pos[i]] = (uint32_t)i;
}

// One warp per tile. EMIT = false: cnt[t] = records the tile yields; true: they
// are written at off[t] (sources ascending within a tile).
template <bool EMIT>
__global__ void __launch_bounds__(TILE_WARPS * 32) k_col_tiles(const uint4 *__restrict__ rec, const uint64_t *__restrict__ key,
                                                            const uint32_t *__restrict__ idx,
                                                            const uint32_t *__restrict__ start, uint64_t ntiles,
                                                            uint64_t nt, uint32_t *cnt, const uint64_t *__restrict__ off,
                                                            uint4 *out)
{
    __shared__ uint32_t M[TILE_WARPS][EIDS][7];   // 7 words a row: conflict-free column reads
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t(*m)[7] = M[w];
    for (uint64_t t = blockIdx.x * (uint64_t)TILE_WARPS + w; t < ntiles; t += (uint64_t)gridDim.x * TILE_WARPS) {
        const uint64_t a = start[t], z = t + 1 < ntiles ? start[t + 1] : nt;
        for (uint32_t u = lane; u < EIDS * 7; u += 32) (&m[0][0])[u] = 0;
        __syncwarp();
        const uint64_t k = key[a];
        const uint32_t lab = (uint32_t)(k >> 50), jb = (uint32_t)(k >> 25) & BASE_MASK, ib = (uint32_t)k & BASE_MASK;
        for (uint64_t r = a + lane; r < z; r += 32) {
            const uint32_t j = idx[r];
            const uint4 e0 = rec[2 * j], e1 = rec[2 * j + 1];
            const uint32_t jo = e1.w - jb * EIDS;      // < 192: the tile's destinations share block jb
            if (jo < EIDS) {
                m[jo][0] = e0.x; m[jo][1] = e0.y; m[jo][2] = e0.z; m[jo][3] = e0.w; m[jo][4] = e1.x; m[jo][5] = e1.y;
            }
        }
        __syncwarp();
        uint64_t made = 0;
        for (int iw = 0; iw < 6; iw++) {
            uint32_t o[6];
#pragma unroll
            for (int jw = 0; jw < 6; jw++) {
                const uint32_t v = m[jw * 32 + lane][iw];   // lane = destination jw*32+lane, bits over 32 sources
                uint32_t res = 0;
                if (__any_sync(0xffffffffu, v != 0)) {
#pragma unroll 4
                    for (int b = 0; b < 32; b++) {
                        const uint32_t col = __ballot_sync(0xffffffffu, (v >> b) & 1u);
                        if ((int)lane == b) res = col;   // source iw*32+b: its destinations in word jw
                    }
                }
                o[jw] = res;
            }
            const bool any = (o[0] | o[1] | o[2] | o[3] | o[4] | o[5]) != 0;
            const unsigned msk = __ballot_sync(0xffffffffu, any);
            if (EMIT && any) {
                const uint64_t p = off[t] + made + __popc(msk & ((1u << lane) - 1u));
                out[2 * p] = make_uint4(o[0], o[1], o[2], o[3]);
                out[2 * p + 1] = make_uint4(o[4], o[5], (lab << 25) | jb, ib * EIDS + iw * 32 + lane);
            }
            made += __popc(msk);
        }
        if (!EMIT && lane == 0) cnt[t] = (uint32_t)made;
        __syncwarp();
    }
}

// sorted records [from, n) copied as they are to out[dst0 + (i - from)]
__global__ void k_col_copy(const uint4 *__restrict__ rec, const uint32_t *__restrict__ idx, uint64_t from, uint64_t n,
                           uint4 *out, uint64_t dst0)
{
    for (uint64_t i = from + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t j = idx[i];
        const uint64_t o = dst0 + (i - from);
        out[2 * o] = rec[2 * j];
        out[2 * o + 1] = rec[2 * j + 1];
    }
}

__global__ void k_widen32(const uint32_t *in, uint64_t n, uint64_t *out)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = in[i];
}

}  // namespace

cudaError_t grg_fmt_columns_to_rows(const uint4 *rec, uint64_t n, uint64_t tmask, uint4 **out, uint64_t *n_out,
                                    cudaStream_t s)
{
    cudaError_t err = cudaSuccess;
    uint64_t *key = nullptr, *toff = nullptr;
    uint32_t *idx = nullptr, *head = nullptr, *tcnt = nullptr;
    void *tmp = nullptr;
    uint4 *res = nullptr;
    size_t tsort = 0, tscan = 0, tscan2 = 0;
    uint64_t nt = 0, ntiles = 0, made = 0;
    *out = nullptr;
    *n_out = 0;
    if (!n) return cudaSuccess;
    FMT_CHECK(cudaMalloc(&key, n * 16));
    FMT_CHECK(cudaMalloc(&idx, n * 8));
    FMT_CHECK(cub::DeviceRadixSort::SortPairs(nullptr, tsort, key, key + n, idx, idx + n, n, 0, 57, s));
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, tscan, idx, idx, n + 1, s));
    FMT_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, tscan2, key, key, n + 1, s));
    if (tscan2 > tscan) tscan = tscan2;
    FMT_CHECK(cudaMalloc(&tmp, tsort > tscan ? tsort : tscan));
    k_col_keys<<<grid_of(n, 256), 256, 0, s>>>(rec, n, tmask, key, idx);
    FMT_CHECK(cub::DeviceRadixSort::SortPairs(tmp, tsort, key, key + n, idx, idx + n, n, 0, 57, s));
    {
        // column records come first; nt = their number (the first key >= NOT_COLUMN)
        uint64_t lo = 0, hi = n;
        std::vector<uint64_t> probe(1);
        while (lo < hi) {          // binary search on the sorted keys, one 8-byte read a step
            const uint64_t mid = (lo + hi) / 2;
            FMT_CHECK(cudaMemcpyAsync(probe.data(), key + n + mid, 8, cudaMemcpyDeviceToHost, s));
            FMT_CHECK(cudaStreamSynchronize(s));
            if (probe[0] >= NOT_COLUMN) hi = mid; else lo = mid + 1;
        }
        nt = lo;
    }
    if (nt) {
        // tile starts: heads -> their positions -> start[]
        FMT_CHECK(cudaMalloc(&head, (nt + 1) * 12));
        uint32_t *pos = head + nt + 1, *start = pos + nt + 1;
        FMT_CHECK(cudaMemsetAsync(head + nt, 0, 4, s));
        k_col_heads<<<grid_of(nt, 256), 256, 0, s>>>(key + n, nt, head);
        FMT_CHECK(cub::DeviceScan::ExclusiveSum(tmp, tscan, head, pos, nt + 1, s));
        uint32_t nt32 = 0;
        FMT_CHECK(cudaMemcpyAsync(&nt32, pos + nt, 4, cudaMemcpyDeviceToHost, s));
        FMT_CHECK(cudaStreamSynchronize(s));
        ntiles = nt32;
        k_col_starts<<<grid_of(nt, 256), 256, 0, s>>>(head, pos, nt, start);
        // records per tile, their offsets, then the records
        FMT_CHECK(cudaMalloc(&tcnt, (ntiles + 1) * 4));
        FMT_CHECK(cudaMalloc(&toff, (ntiles + 1) * 16));
        FMT_CHECK(cudaMemsetAsync(tcnt + ntiles, 0, 4, s));
        const int tg = grid_of((ntiles + TILE_WARPS - 1) / TILE_WARPS, 1);
        k_col_tiles<false><<<tg, TILE_WARPS * 32, 0, s>>>(rec, key + n, idx + n, start, ntiles, nt, tcnt, nullptr,
                                                           nullptr);
        k_widen32<<<grid_of(ntiles + 1, 256), 256, 0, s>>>(tcnt, ntiles + 1, toff + ntiles + 1);
        FMT_CHECK(cub::DeviceScan::ExclusiveSum(tmp, tscan, toff + ntiles + 1, toff, ntiles + 1, s));
        FMT_CHECK(cudaMemcpyAsync(&made, toff + ntiles, 8, cudaMemcpyDeviceToHost, s));
        FMT_CHECK(cudaStreamSynchronize(s));
        FMT_CHECK(cudaMalloc(&res, (made + (n - nt)) * 32 + 32));
        k_col_tiles<true><<<tg, TILE_WARPS * 32, 0, s>>>(rec, key + n, idx + n, start, ntiles, nt, nullptr, toff, res);
    } else {
        FMT_CHECK(cudaMalloc(&res, n * 32 + 32));
    }
    // records stored by source follow, as they are (out index made + (i - nt))
    if (n > nt) k_col_copy<<<grid_of(n - nt, 256), 256, 0, s>>>(rec, idx + n, nt, n, res, made);
    FMT_CHECK(cudaGetLastError());
    FMT_CHECK(cudaStreamSynchronize(s));
    *out = res;
    *n_out = made + (n - nt);
    res = nullptr;
done:
    cudaFree(res);
    cudaFree(toff);
    cudaFree(tcnt);
    cudaFree(head);
    cudaFree(tmp);
    cudaFree(idx);
    cudaFree(key);
    return err;
}
