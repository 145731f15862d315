// pbf_cell_sort_noalloc: the neighbour-search sort (cell hash, stable
// counting sort, cell ranges) for callers that cannot allocate device
// memory.
//
// Some callers cannot call cudaMalloc at the point where they need the
// sort: code that runs while a stream is being captured into a CUDA graph,
// plug-ins whose host application owns every device allocation through its
// own pool, or real-time paths where an allocation (and the device-wide
// synchronisation it may cause) is not allowed.  This entry point needs no
// handle and allocates nothing: its scratch (keys, slots, bucket scratch,
// cell counts and offsets) lives in one file-scope __device__ array of fixed
// size, which every GPU that loads the library holds until the process exits.
//
// Limits: n <= PBF_NOALLOC_MAX_PARTICLES particles and
// Gx*Gy*Gz <= PBF_NOALLOC_MAX_CELLS cells (7.3 MB of device memory).
//
// The first call on a device looks up the array's device address (with that
// device current) and caches it; make that first call before any stream
// capture.  All calls share the one array: calls whose work overlaps on the
// GPU (different streams, or different host threads on one device) race on it
// and must be serialised by the caller.  Each call clears the cell counts it
// uses before the histogram, so a call never sees the previous call's data.
#include <mutex>

#include "pbf103.h"
#include "pbf_internal.h"
#include "pbf_scan.cuh"
#include "pbf_sort.cuh"

namespace pbf103 {
void set_last_error(const char *what, cudaError_t e);
}

namespace {

constexpr uint32_t kMaxN = PBF_NOALLOC_MAX_PARTICLES;
constexpr uint32_t kMaxC = PBF_NOALLOC_MAX_CELLS;
constexpr uint32_t kTile = 4096;                            // cells per scan tile
constexpr uint32_t kMaxTiles = (kMaxC + 1 + kTile - 1) / kTile;
// buckets of more than kRankMax entries are sorted by a block each
// (block_radix_stable); at most kMaxBig of them fit in kMaxN particles
constexpr uint32_t kRankMax = 4096;
constexpr uint32_t kMaxBig = kMaxN / (kRankMax + 1) + 1;
// words: keys, slots, tmp (n each); counts, offsets (C + 2 each); tile sums;
// the queue of large buckets (count, then cells)
constexpr size_t kWords = 3ull * kMaxN + 2ull * (kMaxC + 2) + kMaxTiles + 4 + 1 + kMaxBig;

static __device__ __align__(256) uint32_t g_noalloc_scratch[kWords];

struct Scratch {
    uint32_t *keys, *slots, *tmp, *counts, *offsets, *tsum, *big;
};

Scratch carve(uint32_t *base)
{
    Scratch s;
    s.keys = base;
    s.slots = s.keys + kMaxN;
    s.tmp = s.slots + kMaxN;
    s.counts = s.tmp + kMaxN;
    s.offsets = s.counts + (kMaxC + 2);
    s.tsum = s.offsets + (kMaxC + 2);
    s.big = s.tsum + kMaxTiles + 4;
    return s;
}

// device address of the scratch array, per device, looked up once
std::mutex g_mu;
uint32_t *g_ptr[256];
uint32_t g_blocks[256];  // blocks the scan's cluster may have there

__device__ __forceinline__ uint32_t hash_of(float x, float y, float z, float cw, uint3 g)
{
    const uint32_t gx = (uint32_t)__float2int_rd(__fdiv_rn(x, cw)) & (g.x - 1u);
    const uint32_t gy = (uint32_t)__float2int_rd(__fdiv_rn(y, cw)) & (g.y - 1u);
    const uint32_t gz = (uint32_t)__float2int_rd(__fdiv_rn(z, cw)) & (g.z - 1u);
    return gz * g.x * g.y + gy * g.x + gx;
}

__global__ void na_hash_count(const float *__restrict__ x, uint32_t n, float cw, uint3 g, Scratch s)
{
    pbf103::release_next();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t k = hash_of(x[3 * i], x[3 * i + 1], x[3 * i + 2], cw, g);
    s.keys[i] = k;
    s.slots[i] = atomicAdd(s.counts + k, 1u);
}

__global__ void na_tile_sums(uint32_t C, Scratch s)
{
    __shared__ uint32_t part[256];
    const uint32_t t = blockIdx.x, base = t * kTile;
    uint32_t v = 0;
    for (uint32_t c = base + threadIdx.x; c < base + kTile && c < C; c += 256) v += s.counts[c];
    part[threadIdx.x] = v;
    __syncthreads();
    for (uint32_t o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) s.tsum[t] = part[0];
}

// A cell's range for the caller.
__device__ __forceinline__ void put_range(uint32_t c, uint32_t st, uint32_t count, uint32_t *__restrict__ cs,
                                          uint32_t *__restrict__ ce)
{
    cs[c] = count ? st : 0xFFFFFFFFu;
    ce[c] = count ? st + count : 0xFFFFFFFFu;
}

// The whole scan in one cluster launch, for tables of up to
// kScanClusterMax * 1024 * kScanRoundsMax cells; also the caller's ranges, and
// empties the large-bucket queue that na_rank fills next.  The sort is bound
// by its launches: 250,007 particles in 32,768 cells took 49 us with the scan
// in three launches (one of them one thread over the tile sums) and the
// ranges in another, 35 with this one, 27 with each launch set up while the
// one before runs (launch_after; 100,000 particles 29 -> 21, 1,000 18 -> 15).
template <uint32_t R>
__global__ void __launch_bounds__(1024) na_scan_cluster(uint32_t C, Scratch s, uint32_t *__restrict__ cs,
                                                        uint32_t *__restrict__ ce)
{
    pbf103::after_previous();
    pbf103::release_next();
    if (blockIdx.x == 0 && threadIdx.x == 0) s.big[0] = 0;
    const uint32_t all = pbf103::cluster_scan<R>([&](uint32_t c) { return s.counts[c]; }, C, [&](uint32_t c, uint32_t offset, uint32_t count) {
        s.offsets[c] = offset;
        put_range(c, offset, count, cs, ce);
    });
    if (blockIdx.x == 0 && threadIdx.x == 0) s.offsets[C] = all;
}

using ScanFn = void (*)(uint32_t, Scratch, uint32_t *, uint32_t *);
ScanFn scan_fn(uint32_t rounds)
{
    switch (rounds) {
    case 1: return na_scan_cluster<1>;
    case 2: return na_scan_cluster<2>;
    case 4: return na_scan_cluster<4>;
    case 8: return na_scan_cluster<8>;
    case 16: return na_scan_cluster<16>;
    default: return na_scan_cluster<pbf103::kScanRoundsMax>;
    }
}

// one block: exclusive scan of the (at most kMaxTiles) tile sums; empties
// the large-bucket queue that na_rank fills next
static_assert(kMaxTiles <= 256, "na_tile_scan's threads take a tile sum each");
__global__ void __launch_bounds__(256) na_tile_scan(uint32_t ntiles, uint32_t C, Scratch s)
{
    __shared__ uint32_t tot[8];
    const uint32_t t = threadIdx.x, warp = t >> 5;
    const uint32_t v = t < ntiles ? s.tsum[t] : 0u, inc = pbf103::warp_incl_scan(v);
    if ((t & 31u) == 31u) tot[warp] = inc;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < warp; ++w) before += tot[w];
    if (t < ntiles) s.tsum[t] = before + inc - v;
    if (t == 255) s.offsets[C] = before + inc;
    if (t == 0) s.big[0] = 0;
}

__global__ void na_scan_tiles(uint32_t C, Scratch s, uint32_t *__restrict__ cs, uint32_t *__restrict__ ce)
{
    __shared__ uint32_t buf[kTile];
    __shared__ uint32_t warp_tot[8];
    const uint32_t t = blockIdx.x, base = t * kTile;
    for (uint32_t c = threadIdx.x; c < kTile; c += 256) buf[c] = (base + c < C) ? s.counts[base + c] : 0u;
    __syncthreads();
    // each of the 256 threads scans 16 consecutive cells
    uint32_t loc[16], sum = 0;
    for (int k = 0; k < 16; ++k) {
        loc[k] = sum;
        sum += buf[threadIdx.x * 16 + k];
    }
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc = sum;
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    uint32_t wpre = 0;
    for (uint32_t w = 0; w < warp; ++w) wpre += warp_tot[w];
    const uint32_t pre = s.tsum[t] + wpre + inc - sum;
    for (int k = 0; k < 16; ++k) {
        const uint32_t c = base + threadIdx.x * 16 + k;
        if (c < C) {
            s.offsets[c] = pre + loc[k];
            put_range(c, pre + loc[k], buf[threadIdx.x * 16 + k], cs, ce);
        }
    }
}

__global__ void na_scatter(uint32_t n, Scratch s)
{
    pbf103::after_previous();
    pbf103::release_next();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) s.tmp[s.offsets[s.keys[i]] + s.slots[i]] = i;
}

// stable position = bucket start + number of smaller indices in the bucket;
// a bucket above kRankMax entries is queued (by its member of atomic slot 0)
// for na_big instead
constexpr uint32_t kRankLong = 1024;  // one by one above: 2,048 members 34 us against 45
__global__ void na_rank(uint32_t n, Scratch s, uint32_t *__restrict__ perm)
{
    pbf103::after_previous();
    pbf103::release_next();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t k = s.keys[i];
    const uint32_t st = s.offsets[k], en = s.offsets[k + 1];
    if (en - st > kRankMax) {
        if (s.slots[i] == 0) s.big[1 + atomicAdd(s.big, 1u)] = k;
        return;
    }
    uint32_t r = 0, t = st;
    if (en - st > kRankLong)
        for (; t < en; ++t) r += s.tmp[t] < i ? 1u : 0u;
    for (; t < en; t += 8) {  // 8 members requested together
        uint32_t m[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) m[k] = t + k < en ? s.tmp[t + k] : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) r += m[k] < i ? 1u : 0u;
    }
    perm[st + r] = i;
}

// the queued large buckets, a block each: stable order by input index
__global__ void __launch_bounds__(pbf103::kRadixThreads) na_big(uint32_t n, Scratch s, uint32_t *__restrict__ perm)
{
    __shared__ pbf103::RadixSmem sm;
    __shared__ uint32_t base[16], tot[16];
    pbf103::after_previous();
    pbf103::release_next();
    const uint32_t nb = s.big[0];
    for (uint32_t q = blockIdx.x; q < nb; q += gridDim.x) {
        const uint32_t k = s.big[1 + q];
        const uint32_t st = s.offsets[k], en = s.offsets[k + 1];
        pbf103::block_radix_stable(s.tmp + st, perm + st, en - st, 0xFFFFFFFFu, pbf103::radix_bits(n), sm, base,
                                   tot, pbf103::BlockSync());
    }
}

bool pow2(uint32_t v) { return v && !(v & (v - 1)); }

}  // namespace

extern "C" pbf_status pbf_cell_sort_noalloc(const float *x_dev, uint32_t n, float cell_width,
                                            const uint32_t grid[3], uint32_t *perm_dev, uint32_t *cell_start_dev,
                                            uint32_t *cell_end_dev, void *stream)
{
    if (!grid || !(cell_width > 0.f) || (n && (!x_dev || !perm_dev)) || !cell_start_dev || !cell_end_dev)
        return PBF_ERROR_INVALID_ARGUMENT;
    if (!pow2(grid[0]) || !pow2(grid[1]) || !pow2(grid[2])) return PBF_ERROR_INVALID_ARGUMENT;
    const uint64_t C64 = (uint64_t)grid[0] * grid[1] * grid[2];
    if (n > kMaxN || C64 > kMaxC) return PBF_ERROR_CAPACITY;  // beyond the fixed scratch
    const uint32_t C = (uint32_t)C64;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 256) {
        pbf103::set_last_error("cudaGetDevice", e);
        return PBF_ERROR_CUDA;
    }
    uint32_t *base, blocks;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_ptr[dev]) {
            void *p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess) {
                pbf103::set_last_error("cudaGetSymbolAddress", e);
                return PBF_ERROR_CUDA;
            }
            bool ok = true;
            for (uint32_t r : {1u, 2u, 4u, 8u, 16u, pbf103::kScanRoundsMax}) ok = pbf103::allows_cluster(scan_fn(r)) && ok;
            g_blocks[dev] = ok ? pbf103::kScanClusterMax : 8u;
            g_ptr[dev] = static_cast<uint32_t *>(p);
        }
        base = g_ptr[dev];
        blocks = g_blocks[dev];
    }
    const Scratch s = carve(base);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uint3 g = make_uint3(grid[0], grid[1], grid[2]);
    const uint32_t ntiles = (C + kTile - 1) / kTile, rounds = pbf103::cluster_scan_rounds(C, blocks);
    // the histogram must start from zero: clear this call's cells
    e = cudaMemsetAsync(s.counts, 0, 4ull * (C + 1), st);
    if (e != cudaSuccess) {
        pbf103::set_last_error("cudaMemsetAsync", e);
        return PBF_ERROR_CUDA;
    }
    if (n) na_hash_count<<<(n + 255) / 256, 256, 0, st>>>(x_dev, n, cell_width, g, s);
    if (rounds) {
        pbf103::launch_cluster<true>(scan_fn(rounds), blocks, st, C, s, cell_start_dev, cell_end_dev);
    } else {
        na_tile_sums<<<ntiles, 256, 0, st>>>(C, s);
        na_tile_scan<<<1, 256, 0, st>>>(ntiles, C, s);
        na_scan_tiles<<<ntiles, 256, 0, st>>>(C, s, cell_start_dev, cell_end_dev);
    }
    if (n) {
        pbf103::launch_after(na_scatter, (n + 255) / 256, 256, st, n, s);
        // Crowded cells: the rank re-reads its buckets through L1, which is
        // smaller beside early-started blocks.  100,000 particles of 195 a cell
        // 55 us by a plain launch, 77 set up early, of 49 a cell 29 and 35; of 24 a
        // cell 25 both ways, 250,007 of 8 a cell 29 and 27.
        if (n / 48u >= C)
            na_rank<<<(n + 255) / 256, 256, 0, st>>>(n, s, perm_dev);
        else
            pbf103::launch_after(na_rank, (n + 255) / 256, 256, st, n, s, perm_dev);
        if (n > kRankMax) pbf103::launch_after(na_big, kMaxBig, pbf103::kRadixThreads, st, n, s, perm_dev);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        pbf103::set_last_error("pbf_cell_sort_noalloc launch", e);
        return PBF_ERROR_CUDA;
    }
    return PBF_SUCCESS;
}
