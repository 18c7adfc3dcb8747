// stream_power.cu -- implicit D8 stream-power incision (Braun & Willett 2013).
//
// Reference: compute_d8_stream_power_incision (src/cpu/lsdtt_stream_power_cpu.
// cpp:159-326). The reference sweeps the reverse topological order; each
// cell reads only its own old elevation and its receiver's NEW elevation, so
// any order that finalises a receiver before its donors gives the same bits.
// Here cells are grouped by depth below their outlet (from the Euler tour)
// and each depth level is one parallel step. The arithmetic keeps the
// reference's operand types: float elevations, double kam = K*w*A^m,
// float dt/dx_eff, the n = 1 closed form in double rounded to float, and for
// n != 1 the same Newton iteration (double epsilon, float updates, at most
// 100 iterations, then the rise guard and the over-excavation clamp).

#include <cmath>
#include <cstdlib>
#include <vector>

#include "engine.cuh"
#include "sp_node.cuh"

namespace lsdtt_gb300
{
namespace
{

// Depth histogram and scatter with warp-aggregated atomics (lanes of a warp
// holding the same depth, as neighbouring cells mostly do, share one). The
// deepest level takes one atomic a block: one a warp and depth on its single
// address took 0.66 of the 0.73 ms of a 2048 x 2048 histogram.
__global__ void __launch_bounds__(256) depth_hist(const std::uint8_t* __restrict__ mask,
                                                  const std::int32_t* __restrict__ depth, std::int64_t n,
                                                  std::uint32_t* __restrict__ count,
                                                  unsigned long long* __restrict__ maxd)
{
    LSDTT_COUNT();
    __shared__ int sh_max[8];
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int key = (i < n && mask[i]) ? depth[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && static_cast<int>(threadIdx.x & 31) == __ffs(peers) - 1)
        atomicAdd(&count[key], static_cast<unsigned>(__popc(peers)));
    const int top = __reduce_max_sync(0xffffffffu, key);
    if ((threadIdx.x & 31) == 0) sh_max[threadIdx.x >> 5] = top;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int m = sh_max[0];
        for (int k = 1; k < 8; ++k) m = max(m, sh_max[k]);
        if (m > 0) atomicMax(maxd, static_cast<unsigned long long>(m));
    }
}

// (with each cell's position in the order)
__global__ void depth_scatter(const std::uint8_t* __restrict__ mask, const std::int32_t* __restrict__ depth,
                              std::int64_t n, const std::uint32_t* __restrict__ start, std::uint32_t* __restrict__ fillc,
                              std::uint32_t* __restrict__ order, std::uint32_t* __restrict__ pos)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int key = (i < n && mask[i]) ? depth[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    std::uint32_t base = 0;
    if (key >= 0 && lane == leader) base = atomicAdd(&fillc[key], static_cast<unsigned>(__popc(peers)));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (key >= 0)
    {
        const std::uint32_t k = start[key] + base + __popc(peers & ((1u << lane) - 1u));
        order[k] = static_cast<std::uint32_t>(i);
        pos[i] = k;
    }
}

// K * A^m per node ahead of the sweep (fully parallel), in place over the
// accumulated area. With the exact accumulation path (area = count * dx^2)
// and a uniform K, counts below kKamTab take a table built with the same
// arithmetic.
constexpr int kKamTab = 4096;

__global__ void sp_kam_table(SpParams P, double dw, double* __restrict__ tab)
{
    LSDTT_COUNT();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < kKamTab) tab[c] = sp_kam(P, static_cast<double>(c) * dw, P.K);
}

__global__ void sp_kam_pass(std::int64_t n, SpParams P, const std::uint8_t* __restrict__ mask,
                            const std::int64_t* __restrict__ receiver, const std::uint64_t* __restrict__ size,
                            const double* __restrict__ tab, const float* __restrict__ kfield, double* __restrict__ area)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n || !mask[i] || receiver[i] < 0) return;
    if (tab && size[i] < static_cast<std::uint64_t>(kKamTab))
        area[i] = tab[size[i]];
    else
        area[i] = sp_kam(P, area[i], kfield ? kfield[i] : P.K);
}

// The sweep works on records in depth order, so that a level's inputs are one
// coalesced read that can be issued ahead and only the receiver's new
// elevation is a dependent one. A record is 16 bytes:
//   x, y  n = 1: w = 1 / (1 + K A^m dt / dx) in two FP32 words (1, 0 where the
//         cell is not eroded; y NaN where w has no such form), else not used
//   z     the old elevation
//   w     the receiver's position in the order (bit 31: a diagonal step)
// a[k] = K A^m (n = 1: K A^m dt / dx), negative where the cell is not eroded;
// z[k] = the new elevation.
struct SpRecords
{
    SpParams P;
    float tol[2];  // rise guard of a cardinal and a diagonal step
    const std::uint32_t* start;  // device level offsets
    uint4* q;
    double* a;
    float* z;
};

__global__ void __launch_bounds__(256) sp_records(SpRecords R, std::uint32_t n_valid, std::int64_t n,
                                                  const std::uint32_t* __restrict__ order,
                                                  const std::uint32_t* __restrict__ pos,
                                                  const std::int64_t* __restrict__ receiver,
                                                  const std::uint8_t* __restrict__ dir, const double* __restrict__ kam,
                                                  const float* __restrict__ z_old)
{
    LSDTT_COUNT();
    const std::uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_valid) return;
    const std::uint32_t flat = order[k];
    const std::int64_t recv = receiver[flat];
    const float zo = z_old[flat];
    double a = -1.0;
    float wh = 1.0f, wl = 0.0f;
    std::uint32_t rp = 0;
    if (recv >= 0 && recv < n)
    {
        const bool diag = (dir[flat] & 1u) != 0;
        rp = pos[recv] | (diag ? 0x80000000u : 0u);
        a = kam[flat];
        if (R.P.n_is_one && !(a < 0.0))
        {
            a = __dmul_rn(a, static_cast<double>(__fdiv_rn(R.P.dt, diag ? R.P.dx_diag : R.P.dx)));
            const double w = __drcp_rn(__dadd_rn(1.0, a));
            wh = static_cast<float>(w);
            wl = a < 1e15 ? static_cast<float>(w - static_cast<double>(wh)) : NAN;
        }
    }
    R.a[k] = a;
    R.q[k] = make_uint4(__float_as_uint(wh), __float_as_uint(wl), __float_as_uint(zo), rp);
    R.z[k] = zo;
}

// The n = 1 update of sp_solve_tol from the record (sp_linear_pair; FP64 where
// that cannot decide). The 13 FP64 instructions a cell took one SM, on which
// the tail of a 512 x 512 grid's sweep runs, most of 1.5 ms.
__device__ __forceinline__ float sp_linear(const SpRecords& R, std::uint32_t k, float wh, float wl, float zo, float zr,
                                           bool diag)
{
    if (zr >= zo) return zo;
    float zn;
    if (!sp_linear_pair(wh, wl, zo, zr, zn))
    {
        const double spf = R.a[k];
        if (spf < 0.0) return zo;
        zn = static_cast<float>(__ddiv_rn(
            __dadd_rn(static_cast<double>(zo), __dmul_rn(static_cast<double>(zr), spf)), __dadd_rn(1.0, spf)));
    }
    return (__fsub_rn(zn, zo) > R.tol[diag ? 1 : 0] || isnan(zn)) ? zo : zn;
}

template <bool kLinear>
__device__ __forceinline__ float sp_record(const SpRecords& R, std::uint32_t k, uint4 q, float zr)
{
    const bool diag = (q.w & 0x80000000u) != 0;
    const float zo = __uint_as_float(q.z);
    if (kLinear) return sp_linear(R, k, __uint_as_float(q.x), __uint_as_float(q.y), zo, zr, diag);
    const double kam = R.a[k];
    return kam < 0.0 ? zo : sp_solve(R.P, diag, kam, zo, zr);
}

template <bool kLinear>
__global__ void __launch_bounds__(128) sp_level(SpRecords R, std::uint32_t lo, std::uint32_t hi)
{
    LSDTT_COUNT();
    const std::uint32_t k = lo + blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= hi) return;
    const uint4 q = R.q[k];
    R.z[k] = sp_record<kLinear>(R, k, q, R.z[q.w & 0x7fffffffu]);
}

// Levels k0 .. kmax in one block, one cell a thread (the long tail of small
// levels). The tail's records are one contiguous run: they stream through a
// ring of four batches in shared memory (asynchronous copies, two to three
// batches ahead), and the level before is there too, so a level is a few
// shared reads, the update and a barrier. With the records behind four
// dependent loads (offset, order, receiver, elevation) the tail of a 512 x 512
// timestep took 2.14 ms, read one level ahead into registers 1.65 ms, and with
// the n = 1 update in FP32 pairs as well 0.25 ms.
constexpr int kSpBatch = 1024;  // records of a batch; a level of the tail has at most as many
struct SpRing
{
    uint4 q[4 * kSpBatch];
    float zb[2][kSpBatch];
    std::uint32_t st[kSpBatch + 3];
};

template <bool kLinear, int NT>
__global__ void __launch_bounds__(NT) sp_tail(SpRecords R, int k0, int kmax)
{
    LSDTT_COUNT();
    extern __shared__ __align__(16) unsigned char sp_smem[];
    SpRing& S = *reinterpret_cast<SpRing*>(sp_smem);
    const int tid = threadIdx.x;
    const std::uint32_t base = R.start[k0], end = R.start[kmax + 1];
    // batch b: records base + b * kSpBatch on (one group even when empty)
    auto load = [&](std::uint32_t b) {
#pragma unroll
        for (int q = 0; q < kSpBatch / NT; ++q)
        {
            const std::uint32_t o = b * kSpBatch + q * NT + tid, k = base + o, s = o & (4 * kSpBatch - 1);
            if (k < end)
            {
                const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(&S.q[s]));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(R.q + k) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (std::uint32_t b = 0; b < 4; ++b) load(b);
    std::uint32_t cur = 0, prev = 0;  // the batch that the level starts in; the last level's first record
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    for (int c0 = k0; c0 <= kmax; c0 += kSpBatch)
    {
        __syncthreads();
        for (int k = tid; k <= kSpBatch; k += NT) S.st[k] = R.start[min(c0 + k, kmax + 1)] - base;
        __syncthreads();
        const int c1 = min(kmax + 1, c0 + kSpBatch);
        for (int k = c0; k < c1; ++k)
        {
            const std::uint32_t lo = S.st[k - c0], hi = S.st[k - c0 + 1];
            while (lo / kSpBatch > cur)
            {
                // the batch behind has been read by every thread (the last
                // level's barrier): its place takes the next one
                load(cur + 4);
                ++cur;
                asm volatile("cp.async.wait_group 2;" ::: "memory");
                __syncthreads();
            }
            const std::uint32_t j = lo + tid;
            if (j < hi)
            {
                const uint4 q = S.q[j & (4 * kSpBatch - 1)];
                const std::uint32_t r = q.w & 0x7fffffffu;
                const float zr = k == k0 ? R.z[r] : S.zb[(k - 1) & 1][r - base - prev];
                const float zn = sp_record<kLinear>(R, base + j, q, zr);
                S.zb[k & 1][tid] = zn;
                R.z[base + j] = zn;
            }
            prev = lo;
            __syncthreads();
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Valid cells take their new elevation, the others keep the old one.
__global__ void __launch_bounds__(256) sp_store(std::int64_t n, const std::uint8_t* __restrict__ mask,
                                                const std::uint32_t* __restrict__ pos, const float* __restrict__ z,
                                                const float* z_old, float* z_out)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) z_out[i] = mask[i] ? z[pos[i]] : z_old[i];
}

}  // namespace

// Device order of valid cells by depth below the outlet and the host copy of
// the level offsets; reused by every sweep of the same build.
struct DepthLevels
{
    std::uint32_t* order = nullptr;
    std::uint32_t* pos = nullptr;  // [n] position of each valid cell in the order
    std::uint32_t* start_dev = nullptr;
    std::vector<std::uint32_t> start;  // [maxdepth + 2]
};

cudaError_t depth_levels(lsdtt_gpu_flow* f, DepthLevels& L, cudaStream_t st)
{
    const std::int64_t n = f->g.n;
    Scratch& ws = f->ws;
    std::uint32_t* count = ws.take<std::uint32_t>(static_cast<std::size_t>(n) + 2);
    std::uint32_t* start = ws.take<std::uint32_t>(static_cast<std::size_t>(n) + 2);
    std::uint32_t* fillc = ws.take<std::uint32_t>(static_cast<std::size_t>(n) + 2);
    L.order = ws.take<std::uint32_t>(static_cast<std::size_t>(n));
    L.pos = ws.take<std::uint32_t>(static_cast<std::size_t>(n));
    unsigned long long* maxd = ws.take<unsigned long long>(1);
    if (!count || !start || !fillc || !L.order || !L.pos || !maxd) return cudaErrorMemoryAllocation;
    cudaMemsetAsync(count, 0, sizeof(std::uint32_t) * (n + 2), st);
    cudaMemsetAsync(fillc, 0, sizeof(std::uint32_t) * (n + 2), st);
    cudaMemsetAsync(maxd, 0, sizeof(unsigned long long), st);
    depth_hist<<<grid_blocks(n, 256), 256, 0, st>>>(f->mask, f->depth, n, count, maxd);
    unsigned long long hmax = 0;
    cudaMemcpyAsync(&hmax, maxd, sizeof(hmax), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    const std::int64_t nlev = static_cast<std::int64_t>(hmax) + 1;
    e = exclusive_scan<std::uint32_t, std::uint32_t>(count, nlev + 1, start, static_cast<std::uint32_t*>(nullptr), ws,
                                                     st);
    if (e != cudaSuccess) return e;
    depth_scatter<<<grid_blocks(n, 256), 256, 0, st>>>(f->mask, f->depth, n, start, fillc, L.order, L.pos);
    L.start_dev = start;
    L.start.resize(static_cast<std::size_t>(nlev) + 1);
    cudaMemcpyAsync(L.start.data(), start, sizeof(std::uint32_t) * (nlev + 1), cudaMemcpyDeviceToHost, st);
    return cudaStreamSynchronize(st);
}

}  // namespace lsdtt_gb300

using namespace lsdtt_gb300;

extern "C" int lsdtt_gpu_stream_power_d8(lsdtt_gpu_flow* f, const float* z_dev, const float* k_field_dev, float K,
                                         float m, float n, float dt, float incision_threshold_area,
                                         std::int32_t divide_area_by_dx, float slope_clamp, float* z_out_dev,
                                         void* stream)
{
    if (!f || !z_dev || !z_out_dev) return fail(LSDTT_GPU_EINVAL, "lsdtt_gpu_stream_power_d8: null argument");
    if (!f->built || !(f->has_topo || f->has_sv) || f->n_valid < 0)
        return fail(LSDTT_GPU_ESTATE, "compute_d8_stream_power_incision: the flow engine has no topological order");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Grid& g = f->g;
    f->ws.used = 0;
    double* area = f->ws.take<double>(static_cast<std::size_t>(g.n));
    if (!area) return cuda_fail(cudaErrorMemoryAllocation, "lsdtt_gpu_stream_power_d8");
    bool exact = false;
    cudaError_t e = accumulate(f, nullptr, area, st, &exact);
    if (e != cudaSuccess) return cuda_fail(e, "lsdtt_gpu_stream_power_d8");
    DepthLevels L;
    e = depth_levels(f, L, st);
    if (e != cudaSuccess) return cuda_fail(e, "lsdtt_gpu_stream_power_d8");
    SpParams P{};
    P.K = K;
    P.m = m;
    P.n = n;
    P.dt = dt;
    P.threshold = incision_threshold_area;
    P.slope_clamp = slope_clamp;
    P.dx = static_cast<float>(g.cell);
    P.dx_diag = P.dx * static_cast<float>(1.4142135623730950488);
    P.divide_by_dx = divide_area_by_dx;
    P.n_is_one = std::fabs(n - 1.0f) < 1e-6f ? 1 : 0;
    // K * A^m per node, then the records in depth order, then the sweep
    double* tab = nullptr;
    if (exact && !k_field_dev)
    {
        tab = f->ws.take<double>(kKamTab);
        if (!tab) return cuda_fail(cudaErrorMemoryAllocation, "lsdtt_gpu_stream_power_d8");
        sp_kam_table<<<grid_blocks(kKamTab, 256), 256, 0, st>>>(P, g.cell * g.cell, tab);
    }
    sp_kam_pass<<<grid_blocks(g.n, 256), 256, 0, st>>>(g.n, P, f->mask, f->receiver, f->sv_size, tab, k_field_dev,
                                                       area);
    const int nlev = static_cast<int>(L.start.size()) - 1;  // levels 0 .. nlev-1
    const std::uint32_t nv = L.start.back();
    SpRecords R{};
    R.P = P;
    R.tol[0] = static_cast<float>(static_cast<double>(P.slope_clamp) * static_cast<double>(P.dx));
    R.tol[1] = static_cast<float>(static_cast<double>(P.slope_clamp) * static_cast<double>(P.dx_diag));
    R.start = L.start_dev;
    R.q = f->ws.take<uint4>(nv + 1);
    R.a = f->ws.take<double>(nv + 1);
    R.z = f->ws.take<float>(nv + 1);
    if (!R.a || !R.q || !R.z) return cuda_fail(cudaErrorMemoryAllocation, "lsdtt_gpu_stream_power_d8");
    if (nv)
        sp_records<<<grid_blocks(nv, 256), 256, 0, st>>>(R, nv, g.n, L.order, L.pos, f->receiver, f->dir, area, z_dev);
    // Levels too small for a launch of their own go to one block. With n = 1 a
    // level of 1024 cells is a few dozen FP32 instructions a warp, less than a
    // launch; otherwise it is a Newton solve of a few hundred a cell, and past
    // eight warps the launch is the shorter.
    const std::uint32_t tail = P.n_is_one ? 1024u : 256u;
    int split = nlev;
    while (split > 1 && L.start[split] - L.start[split - 1] <= tail) --split;
    for (int k = 1; k < split; ++k)
    {
        const std::uint32_t lo = L.start[k], hi = L.start[k + 1];
        if (hi <= lo) continue;
        if (P.n_is_one) sp_level<true><<<grid_blocks(hi - lo, 128), 128, 0, st>>>(R, lo, hi);
        else sp_level<false><<<grid_blocks(hi - lo, 128), 128, 0, st>>>(R, lo, hi);
    }
    if (split < nlev)
    {
        const void* fn = P.n_is_one ? reinterpret_cast<const void*>(sp_tail<true, 1024>)
                                    : reinterpret_cast<const void*>(sp_tail<false, 256>);
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(SpRing)));
        if (e != cudaSuccess) return cuda_fail(e, "lsdtt_gpu_stream_power_d8");
        if (P.n_is_one) sp_tail<true, 1024><<<1, 1024, sizeof(SpRing), st>>>(R, std::max(split, 1), nlev - 1);
        else sp_tail<false, 256><<<1, 256, sizeof(SpRing), st>>>(R, std::max(split, 1), nlev - 1);
    }
    sp_store<<<grid_blocks(g.n, 256), 256, 0, st>>>(g.n, f->mask, L.pos, R.z, z_dev, z_out_dev);
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "lsdtt_gpu_stream_power_d8");
    return LSDTT_GPU_OK;
}

namespace lsdtt_gb300
{
LSDTT_DEFINE_LAUNCH_READER(stream_power)
}  // namespace lsdtt_gb300
