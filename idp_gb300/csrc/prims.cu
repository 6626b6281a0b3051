// Sort, scan and fixed-order sum kernels (see prims.cuh).
#include "prims.cuh"

namespace idp {

namespace {
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_WARPS = RS_THREADS / 32;

__global__ void rs_histogram(const uint64_t* __restrict__ keys, long n, int shift, uint32_t* __restrict__ counts,
                             int ntiles) {
    __shared__ uint32_t h[256];
    int t = threadIdx.x;
    h[t] = 0;
    __syncthreads();
    long base = (long)blockIdx.x * RS_TILE;
    for (int r = 0; r < RS_ITEMS; ++r) {
        long i = base + r * RS_THREADS + t;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    counts[(long)t * ntiles + blockIdx.x] = h[t];
}

__global__ void rs_scatter(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals, long n, int shift,
                           const uint32_t* __restrict__ offsets, int ntiles, uint64_t* __restrict__ okeys,
                           uint32_t* __restrict__ ovals) {
    __shared__ uint32_t wc[RS_WARPS][256];
    __shared__ uint32_t running[256];
    __shared__ uint32_t gbase[256];
    int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    running[t] = 0;
    gbase[t] = offsets[(long)t * ntiles + blockIdx.x];
    for (int w = 0; w < RS_WARPS; ++w) wc[w][t] = 0;
    __syncthreads();
    long base = (long)blockIdx.x * RS_TILE;
    for (int r = 0; r < RS_ITEMS; ++r) {
        long i = base + r * RS_THREADS + t;
        bool valid = i < n;
        uint64_t k = valid ? keys[i] : 0;
        uint32_t v = valid ? vals[i] : 0;
        uint32_t d = valid ? (uint32_t)((k >> shift) & 255u) : (256u + lane);
        uint32_t peers = __match_any_sync(0xffffffffu, d);
        uint32_t lt = (1u << lane) - 1u;
        uint32_t rank_w = __popc(peers & lt);
        if (valid && (peers & lt) == 0) wc[warp][d] = __popc(peers);
        __syncthreads();
        // exclusive prefix over warps for digit t, in place
        {
            uint32_t run = 0;
            for (int w = 0; w < RS_WARPS; ++w) {
                uint32_t c = wc[w][t];
                wc[w][t] = run;
                run += c;
            }
            // this pass's total stays in a register (the prefix overwrote the slots)
            __syncthreads();
            if (valid) {
                uint32_t pos = gbase[d] + running[d] + wc[warp][d] + rank_w;
                okeys[pos] = k;
                ovals[pos] = v;
            }
            __syncthreads();
            running[t] += run;
            for (int w = 0; w < RS_WARPS; ++w) wc[w][t] = 0;
            __syncthreads();
        }
    }
}

// ---- sort of up to kMergeMax items in two launches: tiles of 1024 sorted in
// registers, then every item's rank is its place in its tile plus the number of
// smaller items of the other tiles (equal ones count from earlier tiles only: the
// order of the radix sort). The radix sort is bound by its four or five launches
// per 8 bits of the key; the ranks by the n^2 / 1024 binary searches. 18-bit /
// 42-bit keys, radix passes -> tiles: 1,000 items 48 / 89 -> 7.6 us, 8,192 items
// 58 / 98 -> 14 us, 32,768 items 74 / 134 -> 28 us, 50,000 items 77 / 136 -> 57 us,
// 100,000 items 78 / 139 against 167 us. kMergeMax stays below the crossing of both
// widths, which was not looked for between 50,000 and 100,000 items (by these figures
// near 60,000 at 18 bits and 90,000 at 42).
constexpr int MS_TILE = 1024;
constexpr int MS_LANES = 8;  // per item, each with every 8th tile
constexpr int MS_IDX = 10;   // bits of a place in a tile
constexpr long kMergeMax = 49152;

__device__ __forceinline__ uint64_t ms_exchange(uint64_t a, uint64_t b, bool low) { return (a < b) == low ? a : b; }

__global__ void __launch_bounds__(MS_TILE) ms_tiles(const uint64_t* keys, const uint32_t* vals, long n, uint64_t mask,
                                                    uint64_t* okeys, uint32_t* ovals) {
    __shared__ uint64_t sh[MS_TILE];
    const int t = threadIdx.x;
    const long base = (long)blockIdx.x * MS_TILE, i = base + t;
    // key and place in one word: no two are equal
    uint64_t a = i < n ? (keys[i] & mask) << MS_IDX | (uint64_t)t : ~0ull - (MS_TILE - 1 - t);
    for (int size = 2; size <= MS_TILE; size <<= 1)
        for (int st = size >> 1; st > 0; st >>= 1) {
            uint64_t b;
            if (st >= 32) {
                __syncthreads();
                sh[t] = a;
                __syncthreads();
                b = sh[t ^ st];
            } else {
                b = __shfl_xor_sync(0xffffffffu, a, st);
            }
            a = ms_exchange(a, b, ((t & size) == 0) == ((t & st) == 0));
        }
    uint64_t k = 0;
    uint32_t v = 0;
    if (i < n) {
        const long from = base + (long)(a & (MS_TILE - 1));
        k = keys[from];
        v = vals[from];
    }
    __syncthreads();  // one tile may be sorted in place
    if (i < n) {
        okeys[i] = k;
        ovals[i] = v;
    }
}

__global__ void ms_ranks(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals, long n, uint64_t mask,
                         int ntiles, uint64_t* __restrict__ okeys, uint32_t* __restrict__ ovals) {
    const long g = (long)blockIdx.x * blockDim.x + threadIdx.x, i = g / MS_LANES;
    const int lane = (int)(g % MS_LANES);
    const bool valid = i < n;
    const uint64_t key = valid ? keys[i] : 0, k = key & mask;
    const int own = (int)(i / MS_TILE);
    uint32_t rank = 0;
    for (int t = lane; valid && t < ntiles; t += MS_LANES) {
        if (t == own) {
            rank += (uint32_t)(i % MS_TILE);
            continue;
        }
        const uint64_t* p = keys + (long)t * MS_TILE;
        const uint64_t lim = t < own ? k + 1 : k;  // counts keys below it (mask < 2^63)
        int lo = 0, hi = (int)min((long)MS_TILE, n - (long)t * MS_TILE);
        while (lo < hi) {
            const int m = (lo + hi) >> 1;
            if ((__ldg(p + m) & mask) < lim) lo = m + 1;
            else hi = m;
        }
        rank += (uint32_t)lo;
    }
    for (int o = 1; o < MS_LANES; o <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (valid && lane == 0) {
        okeys[rank] = key;
        ovals[rank] = vals[i];
    }
}

// ---- scan
constexpr int SC_THREADS = 256;
constexpr int SC_ITEMS = 8;
constexpr int SC_TILE = SC_THREADS * SC_ITEMS;
constexpr long kScanTiles = 2048;  // up to these a CTA sums the tiles before its own: 8 loads a thread, no third launch

__device__ uint32_t block_excl_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t ws[SC_THREADS / 32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = (lane < SC_THREADS / 32) ? ws[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < SC_THREADS / 32) ws[lane] = w;
    }
    __syncthreads();
    uint32_t prefix = (warp > 0 ? ws[warp - 1] : 0) + x - v;
    if (total) *total = ws[SC_THREADS / 32 - 1];
    __syncthreads();
    return prefix;
}

__global__ void scan_tile_sums(const uint32_t* __restrict__ in, long n, uint32_t* __restrict__ sums) {
    long base = (long)blockIdx.x * SC_TILE + (long)threadIdx.x * SC_ITEMS;
    uint32_t s = 0;
    for (int k = 0; k < SC_ITEMS; ++k)
        if (base + k < n) s += in[base + k];
    uint32_t tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// sums (tile sums) or tile_off (their scan) give a tile's first value; neither
// with a single tile
__global__ void scan_tiles(const uint32_t* in, uint32_t* out, long n, const uint32_t* __restrict__ sums,
                           const uint32_t* __restrict__ tile_off, uint32_t* total) {
    long base = (long)blockIdx.x * SC_TILE + (long)threadIdx.x * SC_ITEMS;
    uint32_t loc[SC_ITEMS];
    uint32_t s = 0;
    for (int k = 0; k < SC_ITEMS; ++k) {
        loc[k] = (base + k < n) ? in[base + k] : 0;
        s += loc[k];
    }
    uint32_t tot, first = tile_off ? tile_off[blockIdx.x] : 0;
    if (sums) {
        uint32_t p = 0;
        for (int t = threadIdx.x; t < blockIdx.x; t += SC_THREADS) p += sums[t];
        block_excl_scan(p, &first);
    }
    uint32_t pre = block_excl_scan(s, &tot);
    uint32_t off = first + pre;
    for (int k = 0; k < SC_ITEMS; ++k) {
        if (base + k < n) out[base + k] = off;
        off += loc[k];
    }
    if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == SC_THREADS - 1) *total = off;
}

// ---- fixed-order double sum
constexpr int DS_THREADS = 256;
constexpr int DS_ITEMS = 8;
constexpr int DS_TILE = DS_THREADS * DS_ITEMS;

__global__ void det_sum_tiles(const double* __restrict__ x, long n, double* __restrict__ out) {
    __shared__ double a[DS_THREADS];
    long base = (long)blockIdx.x * DS_TILE;
    double s = 0.0;
    for (int k = 0; k < DS_ITEMS; ++k) {
        long i = base + k * DS_THREADS + threadIdx.x;
        if (i < n) s += x[i];
    }
    a[threadIdx.x] = s;
    __syncthreads();
    for (int st = DS_THREADS / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st) a[threadIdx.x] += a[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = a[0];
}
}  // namespace

int bits_for(uint64_t m) {
    int b = 0;
    while (b < 64 && (m >> b) != 0) ++b;
    return b < 1 ? 1 : b;
}

size_t radix_sort_scratch_bytes(long n) {
    long tiles = (n + RS_TILE - 1) / RS_TILE;
    if (tiles < 1) tiles = 1;
    return 256 * tiles * sizeof(uint32_t) + scan_scratch_bytes(256 * tiles) + 256;
}

size_t scan_scratch_bytes(long n) {
    // level sizes: n/2048, n/2048^2, ... each level needs sums + offsets
    size_t bytes = 0;
    long m = n;
    while (m > SC_TILE) {
        long t = (m + SC_TILE - 1) / SC_TILE;
        bytes += 2 * ((t + 63) / 64 * 64) * sizeof(uint32_t);
        m = t;
    }
    return bytes + 256;
}

cudaError_t scan_exclusive(const uint32_t* in, uint32_t* out, long n, uint32_t* total, void* scratch,
                           cudaStream_t s) {
    if (n <= 0) {
        if (total) return cudaMemsetAsync(total, 0, sizeof(uint32_t), s);
        return cudaSuccess;
    }
    long tiles = (n + SC_TILE - 1) / SC_TILE;
    if (tiles == 1) {
        (::idp::count_launch(), scan_tiles<<<1, SC_THREADS, 0, s>>>(in, out, n, nullptr, nullptr, total));
        return cudaGetLastError();
    }
    uint32_t* sums = reinterpret_cast<uint32_t*>(scratch);
    long padded = (tiles + 63) / 64 * 64;
    uint32_t* offs = sums + padded;
    void* rest = offs + padded;
    (::idp::count_launch(), scan_tile_sums<<<(int)tiles, SC_THREADS, 0, s>>>(in, n, sums));
    if (tiles <= kScanTiles) {
        (::idp::count_launch(), scan_tiles<<<(int)tiles, SC_THREADS, 0, s>>>(in, out, n, sums, nullptr, total));
        return cudaGetLastError();
    }
    cudaError_t e = scan_exclusive(sums, offs, tiles, nullptr, rest, s);
    if (e != cudaSuccess) return e;
    (::idp::count_launch(), scan_tiles<<<(int)tiles, SC_THREADS, 0, s>>>(in, out, n, nullptr, offs, total));
    return cudaGetLastError();
}

cudaError_t radix_sort_pairs(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt, long n,
                             int bits, void* scratch, cudaStream_t s) {
    if (n <= 1) return cudaSuccess;
    if (n <= kMergeMax && bits + MS_IDX <= 64) {
        const uint64_t mask = (1ull << bits) - 1;  // bits <= 54
        const int nt = (int)((n + MS_TILE - 1) / MS_TILE);
        uint64_t* k1 = nt > 1 ? keys_alt : keys;
        uint32_t* v1 = nt > 1 ? vals_alt : vals;
        (::idp::count_launch(), ms_tiles<<<nt, MS_TILE, 0, s>>>(keys, vals, n, mask, k1, v1));
        if (nt > 1)
            (::idp::count_launch(), ms_ranks<<<grid_for(MS_LANES * n), kBlock, 0, s>>>(k1, v1, n, mask, nt, keys, vals));
        return cudaGetLastError();
    }
    long tiles = (n + RS_TILE - 1) / RS_TILE;
    uint32_t* counts = reinterpret_cast<uint32_t*>(scratch);
    void* scan_scratch = counts + 256 * tiles;
    uint64_t* kin = keys;
    uint32_t* vin = vals;
    uint64_t* kout = keys_alt;
    uint32_t* vout = vals_alt;
    int passes = (bits + 7) / 8;
    for (int p = 0; p < passes; ++p) {
        int shift = 8 * p;
        (::idp::count_launch(), rs_histogram<<<(int)tiles, RS_THREADS, 0, s>>>(kin, n, shift, counts, (int)tiles));
        cudaError_t e = scan_exclusive(counts, counts, 256 * tiles, nullptr, scan_scratch, s);
        if (e != cudaSuccess) return e;
        (::idp::count_launch(), rs_scatter<<<(int)tiles, RS_THREADS, 0, s>>>(kin, vin, n, shift, counts, (int)tiles, kout, vout));
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    if (kin != keys) {
        cudaMemcpyAsync(keys, kin, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(vals, vin, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
    }
    return cudaGetLastError();
}

cudaError_t det_sum(const double* x, long n, double* result, double* scratch, cudaStream_t s) {
    if (n <= 0) return cudaMemsetAsync(result, 0, sizeof(double), s);
    const double* in = x;
    long m = n;
    double* buf[2] = {scratch, scratch + (n / DS_TILE + 2)};
    int which = 0;
    while (true) {
        long tiles = (m + DS_TILE - 1) / DS_TILE;
        double* out = (tiles == 1) ? result : buf[which];
        (::idp::count_launch(), det_sum_tiles<<<(int)tiles, DS_THREADS, 0, s>>>(in, m, out));
        if (tiles == 1) break;
        in = out;
        m = tiles;
        which ^= 1;
    }
    return cudaGetLastError();
}

}  // namespace idp
