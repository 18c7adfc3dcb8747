// prims.cuh -- data-parallel building blocks used by the routing kernels:
// exclusive scan, order-preserving compaction and a stable LSD radix sort.
// All are written for one GPU and one stream, sized in multiples of the SM
// count by the caller's grid choice, and allocate nothing: the caller passes
// a workspace (Scratch) carved from the engine's pool.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace lsdtt_gb300
{

// Bump allocator over one device buffer owned by an engine. Reset per build.
struct Scratch
{
    char* base = nullptr;
    std::size_t cap = 0;
    std::size_t used = 0;
    template <class T>
    T* take(std::size_t count)
    {
        std::size_t off = (used + 255) & ~std::size_t(255);
        std::size_t bytes = count * sizeof(T);
        if (off + bytes > cap) return nullptr;
        used = off + bytes;
        return reinterpret_cast<T*>(base + off);
    }
};

constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;                       // per thread
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096

template <class T>
__device__ inline T block_exclusive_scan(T v, T* smem_warp, T& total)
{
    // Warp-level inclusive scan then a scan of warp totals.
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (warp == 0)
    {
        T w = (lane < nw) ? smem_warp[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            T y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) smem_warp[lane] = w;
    }
    __syncthreads();
    T warp_prefix = (warp > 0) ? smem_warp[warp - 1] : T(0);
    total = smem_warp[nw - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// Per-tile sums (each block reduces one tile of kScanTile inputs).
template <class TIn, class T>
__global__ void scan_tile_sums(const TIn* __restrict__ in, std::int64_t n, T* __restrict__ sums)
{
    LSDTT_COUNT();
    __shared__ T sw[32];
    const std::int64_t base = static_cast<std::int64_t>(blockIdx.x) * kScanTile;
    T acc = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
    {
        const std::int64_t k = base + static_cast<std::int64_t>(i) * kScanThreads + threadIdx.x;
        if (k < n) acc += static_cast<T>(in[k]);
    }
    T total;
    block_exclusive_scan<T>(acc, sw, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Exclusive scan of each tile plus the tile's offset. Each thread owns
// kScanItems consecutive elements so the output order is the input order.
template <class TIn, class T>
__global__ void scan_tile_apply(const TIn* __restrict__ in, std::int64_t n, const T* __restrict__ offs,
                                T* __restrict__ out)
{
    LSDTT_COUNT();
    __shared__ T sw[32];
    const std::int64_t base = static_cast<std::int64_t>(blockIdx.x) * kScanTile +
                              static_cast<std::int64_t>(threadIdx.x) * kScanItems;
    T v[kScanItems];
    T acc = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
    {
        const std::int64_t k = base + i;
        v[i] = (k < n) ? static_cast<T>(in[k]) : T(0);
        acc += v[i];
    }
    T total;
    T pre = block_exclusive_scan<T>(acc, sw, total) + offs[blockIdx.x];
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
    {
        const std::int64_t k = base + i;
        if (k < n) out[k] = pre;
        pre += v[i];
    }
}

// A short scan by one block, kScanTile * 2 values a step with the running sum
// carried over: sums, their own scan and the application are four launches and
// a memset for a few thousand values (a digit's histogram of a small grid).
// Routing 129 x 203 cells 583 us, now 554; a 512 x 512 LEM step 4.01 ms, now
// 3.92. Past four steps (32768 values) the chip's width pays again.
constexpr std::int64_t kScanShort = 32768;

template <class TIn, class T>
__global__ void __launch_bounds__(1024) scan_short(const TIn* __restrict__ in, std::int64_t n, T* __restrict__ out,
                                                   T* __restrict__ total_out)
{
    LSDTT_COUNT();
    __shared__ T sw[32];
    T carry = 0;
    for (std::int64_t b = 0; b < n; b += 1024 * kScanItems)
    {
        const std::int64_t base = b + static_cast<std::int64_t>(threadIdx.x) * kScanItems;
        T v[kScanItems];
        T acc = 0;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i)
        {
            v[i] = base + i < n ? static_cast<T>(in[base + i]) : T(0);
            acc += v[i];
        }
        T total;
        T pre = carry + block_exclusive_scan<T>(acc, sw, total);
#pragma unroll
        for (int i = 0; i < kScanItems; ++i)
        {
            if (base + i < n) out[base + i] = pre;
            pre += v[i];
        }
        carry += total;
    }
    if (threadIdx.x == 0 && total_out) *total_out = carry;
}

// Host: exclusive scan of n values into out (out may alias nothing), and the
// grand total written to *total_dev (device). Workspace: ~n/4096*2 T.
template <class TIn, class T>
inline cudaError_t exclusive_scan(const TIn* in, std::int64_t n, T* out, T* total_dev, Scratch& ws,
                                  cudaStream_t st)
{
    const std::int64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (n == 0)
    {
        if (total_dev) return cudaMemsetAsync(total_dev, 0, sizeof(T), st);
        return cudaSuccess;
    }
    if (n <= kScanShort)
    {
        scan_short<TIn, T><<<1, 1024, 0, st>>>(in, n, out, total_dev);
        return cudaGetLastError();
    }
    const std::size_t mark = ws.used;
    T* sums = ws.take<T>(static_cast<std::size_t>(tiles) + 1);
    T* offs = ws.take<T>(static_cast<std::size_t>(tiles) + 1);
    if (!sums || !offs) return cudaErrorMemoryAllocation;
    scan_tile_sums<TIn, T><<<static_cast<unsigned>(tiles), kScanThreads, 0, st>>>(in, n, sums);
    const cudaError_t e = exclusive_scan<T, T>(sums, tiles, offs, total_dev, ws, st);
    if (e != cudaSuccess) return e;
    scan_tile_apply<TIn, T><<<static_cast<unsigned>(tiles), kScanThreads, 0, st>>>(in, n, offs, out);
    ws.used = mark;
    return cudaGetLastError();
}

// The flagged (1; others 0) indices of a tile, in order, from the tile's offset.
static __global__ void compact_tile(const std::uint8_t* __restrict__ flag, std::int64_t n,
                                    const std::int64_t* __restrict__ offs, std::int64_t* __restrict__ out)
{
    LSDTT_COUNT();
    __shared__ int sw[32];
    const std::int64_t base = static_cast<std::int64_t>(blockIdx.x) * kScanTile +
                              static_cast<std::int64_t>(threadIdx.x) * kScanItems;
    static_assert(kScanItems == 8, "a thread's flags are one 8-byte word");
    std::uint64_t w = 0;
    if (base + kScanItems <= n)
        w = *reinterpret_cast<const std::uint64_t*>(flag + base);
    else
        for (int i = 0; i < kScanItems; ++i)
            if (base + i < n) w |= static_cast<std::uint64_t>(flag[base + i]) << (8 * i);
    int total;
    std::int64_t at = offs[blockIdx.x] + block_exclusive_scan<int>(__popcll(w), sw, total);
    for (; w; w &= w - 1) out[at++] = base + ((__ffsll(static_cast<long long>(w)) - 1) >> 3);
}

// Host: the flagged indices of n flags (0 or 1; 8-byte aligned) into out, in
// order, their number to *total_dev. The positions stay in registers (writing
// and reading one per flag took 137 us of 16.4 M flags, this 32).
inline cudaError_t compact_flagged(const std::uint8_t* flag, std::int64_t n, std::int64_t* out,
                                   std::int64_t* total_dev, Scratch& ws, cudaStream_t st)
{
    if (n == 0) return cudaMemsetAsync(total_dev, 0, sizeof(std::int64_t), st);
    const std::int64_t tiles = (n + kScanTile - 1) / kScanTile;
    const std::size_t mark = ws.used;
    std::int64_t* sums = ws.take<std::int64_t>(static_cast<std::size_t>(tiles));
    std::int64_t* offs = ws.take<std::int64_t>(static_cast<std::size_t>(tiles));
    if (!sums || !offs) return cudaErrorMemoryAllocation;
    scan_tile_sums<std::uint8_t, std::int64_t><<<static_cast<unsigned>(tiles), kScanThreads, 0, st>>>(flag, n, sums);
    const cudaError_t e = exclusive_scan<std::int64_t, std::int64_t>(sums, tiles, offs, total_dev, ws, st);
    if (e != cudaSuccess) return e;
    compact_tile<<<static_cast<unsigned>(tiles), kScanThreads, 0, st>>>(flag, n, offs, out);
    ws.used = mark;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (uint64 key, uint32 value) pairs over the low
// `bits` bits of the key, 8 bits per pass. Ping-pongs between (k0,v0) and
// (k1,v1); returns the buffer index (0 or 1) holding the result. With a
// device count `dn`, only the first min(n, *dn) pairs are sorted (the
// launches stay sized for n; tiles past the count do nothing).
// ---------------------------------------------------------------------------
constexpr int kSortThreads = 256;  // 8 warps
constexpr int kSortWarpItems = 512;  // per warp: 16 rounds of 32
constexpr int kSortTile = kSortWarpItems * (kSortThreads / 32);  // 4096

static __global__ void __launch_bounds__(kSortThreads)
radix_hist(const std::uint64_t* __restrict__ keys, std::int64_t n, int shift, std::uint32_t* __restrict__ hist,
           int n_tiles, const unsigned* __restrict__ dn)
{
    LSDTT_COUNT();
    if (dn && static_cast<std::int64_t>(*dn) < n) n = static_cast<std::int64_t>(*dn);
    __shared__ std::uint32_t h[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const std::int64_t base = static_cast<std::int64_t>(blockIdx.x) * kSortTile;
    std::uint64_t key[kSortTile / kSortThreads];  // all of a thread's loads in flight at once
#pragma unroll
    for (int r = 0; r < kSortTile / kSortThreads; ++r)
    {
        const std::int64_t k = base + r * kSortThreads + threadIdx.x;
        if (k < n) key[r] = keys[k];
    }
#pragma unroll
    for (int r = 0; r < kSortTile / kSortThreads; ++r)
        if (base + r * kSortThreads + threadIdx.x < n) atomicAdd(&h[(key[r] >> shift) & 255u], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
        hist[static_cast<std::int64_t>(i) * n_tiles + blockIdx.x] = h[i];  // digit-major
}

// A tile's pairs are ranked by warp, put in order in shared memory and then
// written: neighbouring threads write a digit's run to neighbouring addresses
// (a pair at a time from the rank straight to its place is one sector a lane,
// keys and values both). Four passes over 16.4 M pairs: 0.93 ms, now 0.67; the
// ten of a 256-member ensemble step: 13.1 ms, now 4.3.
static __global__ void __launch_bounds__(kSortThreads, 3)
radix_scatter(const std::uint64_t* __restrict__ kin, const std::uint32_t* __restrict__ vin, std::int64_t n, int shift,
              const std::uint32_t* __restrict__ offs, int n_tiles, std::uint64_t* __restrict__ kout,
              std::uint32_t* __restrict__ vout, const unsigned* __restrict__ dn)
{
    LSDTT_COUNT();
    if (dn && static_cast<std::int64_t>(*dn) < n) n = static_cast<std::int64_t>(*dn);
    constexpr int kWarps = kSortThreads / 32, kRounds = kSortWarpItems / 32;
    static_assert(kSortThreads == 256, "a thread per digit");
    __shared__ std::uint64_t stage[kSortTile];          // the keys in order, then the values
    __shared__ std::uint32_t wcount[kWarps][256];       // counts, then local bases by warp and digit
    __shared__ std::uint32_t delta[256];                // global place - local place of a digit's pairs
    __shared__ std::uint32_t wsum[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const std::int64_t base = static_cast<std::int64_t>(blockIdx.x) * kSortTile;
    if (base >= n) return;
    for (int i = lane; i < 256; i += 32) wcount[warp][i] = 0;
    __syncwarp();
    const std::int64_t wbase = base + static_cast<std::int64_t>(warp) * kSortWarpItems;
    std::uint64_t key[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        const std::int64_t k = wbase + r * 32 + lane;
        if (k < n) key[r] = kin[k];
    }
    const std::uint32_t goff = offs[static_cast<std::int64_t>(threadIdx.x) * n_tiles + blockIdx.x];
    std::uint32_t place[kRounds];  // digit << 16 | rank in the warp, then the local place
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        const bool ok = wbase + r * 32 + lane < n;
        const std::uint32_t d = ok ? static_cast<std::uint32_t>((key[r] >> shift) & 255u) : 256u + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        std::uint32_t before = 0;
        if (ok) before = wcount[warp][d];
        place[r] = (d << 16) | (before + __popc(peers & ((1u << lane) - 1u)));
        __syncwarp();
        // The highest lane of each peer group bumps the shared counter.
        if (ok && (peers >> lane) == 1u) wcount[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Thread d: exclusive prefix of digit d over the warps, of the digits over
    // the tile.
    {
        const int d = threadIdx.x;
        std::uint32_t acc = 0;
        for (int w = 0; w < kWarps; ++w)
        {
            const std::uint32_t c = wcount[w][d];
            wcount[w][d] = acc;
            acc += c;
        }
        std::uint32_t inc = acc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const std::uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        std::uint32_t first = inc - acc;
        for (int w = 0; w < warp; ++w) first += wsum[w];
        for (int w = 0; w < kWarps; ++w) wcount[w][d] += first;
        delta[d] = goff - first;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        if (wbase + r * 32 + lane < n)
        {
            place[r] = wcount[warp][place[r] >> 16] + (place[r] & 0xffffu);
            stage[place[r]] = key[r];
        }
    }
    std::uint32_t val[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        const std::int64_t k = wbase + r * 32 + lane;
        if (k < n) val[r] = vin[k];
    }
    __syncthreads();
    const int m = n - base < kSortTile ? static_cast<int>(n - base) : kSortTile;
    std::uint32_t dst[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        const int i = r * kSortThreads + threadIdx.x;
        if (i < m)
        {
            const std::uint64_t v = stage[i];
            dst[r] = delta[(v >> shift) & 255u] + static_cast<std::uint32_t>(i);
            kout[dst[r]] = v;
        }
    }
    __syncthreads();
    std::uint32_t* vs = reinterpret_cast<std::uint32_t*>(stage);
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
        if (wbase + r * 32 + lane < n) vs[place[r]] = val[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        const int i = r * kSortThreads + threadIdx.x;
        if (i < m) vout[dst[r]] = vs[i];
    }
}

inline int radix_sort_pairs(std::uint64_t* k0, std::uint32_t* v0, std::uint64_t* k1, std::uint32_t* v1,
                            std::int64_t n, int bits, Scratch& ws, cudaStream_t st, cudaError_t* err,
                            const unsigned* dn = nullptr)
{
    *err = cudaSuccess;
    if (n <= 1) return 0;
    const int tiles = static_cast<int>((n + kSortTile - 1) / kSortTile);
    const std::size_t mark = ws.used;
    std::uint32_t* hist = ws.take<std::uint32_t>(static_cast<std::size_t>(tiles) * 256);
    std::uint32_t* offs = ws.take<std::uint32_t>(static_cast<std::size_t>(tiles) * 256);
    if (!hist || !offs) { *err = cudaErrorMemoryAllocation; return 0; }
    int cur = 0;
    for (int shift = 0; shift < bits; shift += 8)
    {
        std::uint64_t* ki = cur ? k1 : k0;
        std::uint32_t* vi = cur ? v1 : v0;
        std::uint64_t* ko = cur ? k0 : k1;
        std::uint32_t* vo = cur ? v0 : v1;
        radix_hist<<<tiles, kSortThreads, 0, st>>>(ki, n, shift, hist, tiles, dn);
        *err = exclusive_scan<std::uint32_t, std::uint32_t>(hist, static_cast<std::int64_t>(tiles) * 256, offs,
                                                            static_cast<std::uint32_t*>(nullptr), ws, st);
        if (*err != cudaSuccess) return cur;
        radix_scatter<<<tiles, kSortThreads, 0, st>>>(ki, vi, n, shift, offs, tiles, ko, vo, dn);
        cur ^= 1;
    }
    ws.used = mark;
    *err = cudaGetLastError();
    return cur;
}

}  // namespace lsdtt_gb300
