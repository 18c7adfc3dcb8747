// hillslope.cu -- implicit (backward-Euler) hillslope diffusion on the GPU.
//
// Reference: compute_hillslope_newton / _transient (src/cpu/lsdtt_hillslope_
// newton_cpu.cpp:196-675, 690-788) on the shared operator of
// src/cpu/lsdtt_hillslope_operator_cpu.hpp:83-322. The residual on every
// degree of freedom (valid, not a channel, not on an 'o' edge) is
//     F_P = inv_dt (z_P - z_P^n) - U - (D/h^2) sum_f alpha_f (z_nb,f - z_P)
// with faces N, E, S, W; 'p' wraps, every other edge and every masked
// neighbour resolves to the cell itself (zero flux); Dirichlet cells keep
// their value. For the linear law (alpha = 1) the Jacobian is constant and
// symmetric positive definite:
//     (J x)_P = inv_dt x_P + (D/h^2) sum_{f: nb != P} (x_P - [nb is DOF] x_nb)
// One Newton step J dz = -F from z^n solves the backward-Euler step; it is
// solved here matrix-free by Jacobi-preconditioned CG to a relative residual
// ||r||_2 <= tol * ||b||_2 (1e-8 on the benchmark configurations), with FP32
// vectors and FP64 dot products. The step is added in double and rounded to
// float, as the reference rounds its double working field.

#include <cmath>
#include <string>
#include <vector>

#include "engine.cuh"
#include "hs_stencil.cuh"

namespace lsdtt_gb300
{
namespace
{

// ---- grid-wide sums --------------------------------------------------------
// Each block writes one FP64 partial per quantity; the block that finishes
// last adds them in index order and forms the solver's next coefficient
// there. Against one FP64 atomic a block on a single address (0.76 ns each at
// the L2) or a one-block kernel after every pass (4.5 us of its own) this
// leaves about a microsecond, and the sums are the same on every run.
// Within a block an iteration's FP32 products are summed in two FP32 words (the
// high words without error, the errors in plain FP32: about 40 bits over a
// block's 2048 or 4096 cells, where FP32 within a warp and FP64 beyond would
// hold about 22): a warp's FP64 addition holds this part's FP64 pipe for 16
// cycles, and ten of them a warp and quantity cost 6 us of a 16 us pass over a
// million cells. The set-up, once a solve, sums in FP64.
struct Sum2
{
    float h = 0.0f, l = 0.0f;
    __device__ __forceinline__ void add(float v)
    {
        const float t = h + v, q = t - h;
        l += (h - (t - q)) + (v - q);
        h = t;
    }
};

template <int K>
__device__ __forceinline__ void block_partials(Sum2 (&v)[K], double* __restrict__ part, unsigned nblk)
{
    __shared__ Sum2 sh_part[K][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto fold = [&](Sum2& a, int from) {
#pragma unroll
        for (int o = from; o > 0; o >>= 1)
        {
            const float h = __shfl_down_sync(0xffffffffu, a.h, o), l = __shfl_down_sync(0xffffffffu, a.l, o);
            a.add(h);
            a.l += l;
        }
    };
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        fold(v[k], 16);
        if (lane == 0) sh_part[k][w] = v[k];
    }
    __syncthreads();
    if (w < K)
    {
        Sum2 a;
        if (lane < 8) a = sh_part[w][lane];
        fold(a, 4);
        if (lane == 0)
        {
            part[static_cast<std::size_t>(w) * nblk + blockIdx.x] = static_cast<double>(a.h) + static_cast<double>(a.l);
            __threadfence();
        }
    }
}

// After block_partials: true in the last block to arrive (every thread of it).
__device__ __forceinline__ bool last_block(unsigned* __restrict__ arrived, unsigned nblk)
{
    __shared__ bool sh_last;
    __syncthreads();
    if (threadIdx.x == 0) sh_last = atomicInc(arrived, nblk - 1) == nblk - 1;  // wraps to 0 for the next pass
    __syncthreads();
    if (sh_last) __threadfence();
    return sh_last;
}

// The last block's totals of K quantities (thread 0 holds them).
template <int K>
__device__ __forceinline__ void total_partials(const double* __restrict__ part, unsigned nblk, double (&out)[K])
{
    __shared__ double sh_tot[K][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        double s = 0.0;
        for (unsigned b = threadIdx.x; b < nblk; b += blockDim.x)
            s += __ldcg(part + static_cast<std::size_t>(k) * nblk + b);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) sh_tot[k][w] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            out[k] = sh_tot[k][0];
            for (int j = 1; j < static_cast<int>(blockDim.x >> 5); ++j) out[k] += sh_tot[k][j];
        }
}

// A cell's class: 0 not a degree of freedom; else bit 0 set, bit 1 "fast"
// (interior, its four neighbours in the grid and DOFs themselves), bits 2-5
// the faces N, E, S, W that lead to another cell.
__device__ __forceinline__ unsigned hs_class(const Hs& H, const std::uint8_t* __restrict__ mask,
                                             const std::uint8_t* __restrict__ chan, int r, int c)
{
    auto is_dof = [&](int rr, int cc) {
        const std::int64_t j = static_cast<std::int64_t>(rr) * H.nc + cc;
        return mask[j] && !(chan && chan[j]) && !hs_dirichlet_edge(H, rr, cc);
    };
    if (!is_dof(r, c)) return 0u;
    const std::int64_t i = static_cast<std::int64_t>(r) * H.nc + c;
    const bool fast = r > 0 && r < H.nr - 1 && c > 0 && c < H.nc - 1 && is_dof(r - 1, c) && is_dof(r, c + 1) &&
                      is_dof(r + 1, c) && is_dof(r, c - 1);
    if (fast) return 1u | 2u | (15u << 2);
    unsigned faces = 0;
#pragma unroll
    for (int f = 0; f < 4; ++f) faces |= (hs_nb(H, mask, r, c, kDr[f], kDc[f]) != i ? 4u : 0u) << f;
    return 1u | faces;
}

// The class plane for the Roering solver.
__global__ void hs_dofs(Hs H, const std::uint8_t* __restrict__ mask, const std::uint8_t* __restrict__ chan,
                        std::uint8_t* __restrict__ dof)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<std::int64_t>(H.nr) * H.nc) return;
    const int r = static_cast<int>(i / H.nc), c = static_cast<int>(i - static_cast<std::int64_t>(r) * H.nc);
    dof[i] = static_cast<std::uint8_t>(hs_class(H, mask, chan, r, c));
}

// ---- linear step -------------------------------------------------------------
// Jacobi-PCG in two passes an iteration:
//   hsl_direction  p = D^-1 r + beta p_old, stored; sum p.(A p), then alpha
//   hsl_update     A p again from p; x += alpha p, r -= alpha A p; sums
//                  r.D^-1 r and r.r, then beta and the convergence test
// D^-1 is one of five values (a cell's class says how many faces it has), so
// neither it nor D^-1 r nor A p is an array: 34 bytes a cell and iteration.
//
// A warp walks a strip 32 columns wide (30 of them its own, the outer lanes
// the halo) down RW rows: north and south neighbours are its registers, east
// and west a shuffle, and all loads of the strip are issued before the first
// is used. The halo wraps where the edge does, a cell's class says which of
// its faces lead to another cell, and p is 0 at a cell that is not a DOF, so
// every cell takes the same path: resolving an edge cell's neighbours one by
// one (mask, class, values: three dependent loads each) made the warps of the
// east and west edges the longest by far, 47 us of a pass on 2048 x 2051. The
// passes now take 24 and 33 us there (about 8 of each the grid-wide sum's
// chain of fence, arrival and last block) where the three untiled passes they
// replace took 162: a solve of 80 iterations 14.3 -> 5.4 ms.
constexpr int kHslTC = 128;  // columns of a set-up block

struct Strip
{
    int r0, c;     // first own row, this lane's column
    bool own;      // the lane's column is the warp's own (and on the grid)
    bool any;      // the strip exists
    int nr, up, dn;  // rows read as row -1 and row nr (-1: none)
    __device__ Strip(const Hs& H, int rw)
    {
        const int nc = H.nc;
        nr = H.nr;
        up = H.bn == 'p' ? nr - 1 : -1;
        dn = H.bs == 'p' ? 0 : -1;
        const int ns = (nc + 29) / 30;
        const int g = static_cast<int>(blockIdx.x) * 8 + static_cast<int>(threadIdx.x >> 5);
        const int lane = threadIdx.x & 31;
        r0 = g / ns * rw;
        c = g % ns * 30 - 1 + lane;
        any = r0 < nr;
        own = any && lane >= 1 && lane <= 30 && c < nc;
        // the halo column a wrapped edge reads
        if (c == -1) c = H.bw == 'p' ? nc - 1 : -1;
        else if (c == nc) c = H.be == 'p' ? 0 : -1;
        else if (c > nc) c = -1;
    }
    // Row k - 1 of the strip as it is read (-1: none).
    __device__ __forceinline__ int row(int k) const
    {
        const int r = r0 - 1 + k;
        return !any || c < 0 ? -1 : (r < 0 ? up : (r < nr ? r : (r == nr ? dn : -1)));
    }
};

struct HsState
{
    double bb, rz, rr, rel, finf;
    float alpha, beta;
    int iters, done;
    unsigned arrived, pad;
};

struct HslArgs
{
    Hs H;
    float inv_dt, DA;
    float invd[5];  // 1 / (1/dt + faces * D/h^2)
    const std::uint8_t* mask;
    const std::uint8_t* cls;
    HsState* S;
    double* part;
    double rel_tol;
    int max_iter;
};

__device__ __forceinline__ float hsl_invd(const HslArgs& A, unsigned cl)
{
    const int f = __popc(cl >> 2);
    return !(cl & 1u) ? 0.0f : (f == 4 ? A.invd[4] : (f == 3 ? A.invd[3] : (f == 2 ? A.invd[2] : (f == 1 ? A.invd[1] : A.invd[0]))));
}

// Classes, b = -F (F = -(D/h^2) sum_f (z_nb - z_P)), r = b, x = 0; ||b||^2,
// r.D^-1 r, max |F|. All in FP64, b rounded once: this runs once a solve, and
// the squares decide when the solve stops (in FP32 they leave its range from
// |F| = 1.8e19 on). It takes 0.16 of the 5.44 ms of a 2048 x 2051 solve more than
// with b in two FP32 words and FP32 squares.
__global__ void __launch_bounds__(256) hsl_setup(HslArgs A, const std::uint8_t* __restrict__ chan,
                                                 const float* __restrict__ z, std::uint8_t* __restrict__ cls,
                                                 float* __restrict__ r, float* __restrict__ x)
{
    LSDTT_COUNT();
    const Hs& H = A.H;
    const int ntx = (H.nc + kHslTC - 1) / kHslTC;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int row = static_cast<int>(blockIdx.x / ntx) * 8 + w, c0 = static_cast<int>(blockIdx.x % ntx) * kHslTC;
    double bb = 0.0, rz = 0.0, fin = 0.0;
    if (row < H.nr)
    {
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const int c = c0 + 32 * k + lane;
            if (c >= H.nc) continue;
            const std::int64_t i = static_cast<std::int64_t>(row) * H.nc + c;
            const unsigned cl = hs_class(H, A.mask, chan, row, c);
            cls[i] = static_cast<std::uint8_t>(cl);
            x[i] = 0.0f;
            float b = 0.0f;
            if (cl)
            {
                const double zp = z[i];
                double flux = 0.0;
#pragma unroll
                for (int f = 0; f < 4; ++f)
                {
                    const std::int64_t j = (cl & 2u) ? i + static_cast<std::int64_t>(kDr[f]) * H.nc + kDc[f]
                                                     : hs_nb(H, A.mask, row, c, kDr[f], kDc[f]);
                    flux += static_cast<double>(z[j]) - zp;
                }
                const double F = -H.DA * flux;
                b = static_cast<float>(-F);
                bb += F * F;
                rz += static_cast<double>(b) * (b * hsl_invd(A, cl));
                fin = fmax(fin, fabs(F));
            }
            r[i] = b;
        }
    }
    const unsigned nblk = gridDim.x;
    block_atomic_max_nonneg(&A.S->finf, fin);
    bb = block_reduce_d(bb, false);
    rz = block_reduce_d(rz, false);
    if (threadIdx.x == 0)
    {
        A.part[blockIdx.x] = bb;
        A.part[nblk + blockIdx.x] = rz;
        __threadfence();
    }
    if (!last_block(&A.S->arrived, nblk)) return;
    double t[2];
    total_partials<2>(A.part, nblk, t);
    if (threadIdx.x == 0)
    {
        A.S->bb = t[0];
        A.S->rz = t[1];
        A.S->beta = 0.0f;
        A.S->done = t[0] == 0.0 ? 1 : 0;
    }
}

// A p at a cell from its own and its neighbours' p (faces in the order N, E,
// S, W).
__device__ __forceinline__ float hsl_op(const HslArgs& A, float pi, float pn, float pe, float ps, float pw, unsigned cl)
{
    float s = 0.0f;
    s += (cl & 4u) ? pi - pn : 0.0f;
    s += (cl & 8u) ? pi - pe : 0.0f;
    s += (cl & 16u) ? pi - ps : 0.0f;
    s += (cl & 32u) ? pi - pw : 0.0f;
    return A.inv_dt * pi + A.DA * s;
}

template <int RW, bool kFirst>
__global__ void __launch_bounds__(256) hsl_direction(HslArgs A, const float* __restrict__ r,
                                                     const float* __restrict__ p_old, float* __restrict__ p)
{
    LSDTT_COUNT();
    if (A.S->done) return;
    const int nr = A.H.nr, nc = A.H.nc;
    const Strip t(A.H, RW);
    const float beta = A.S->beta;
    float rv[RW + 2], pv[RW + 2];
    unsigned cl[RW + 2];
#pragma unroll
    for (int k = 0; k < RW + 2; ++k)
    {
        const int row = t.row(k);
        const bool in = row >= 0;
        const std::int64_t i = static_cast<std::int64_t>(row) * nc + t.c;
        cl[k] = in ? A.cls[i] : 0u;
        rv[k] = in ? r[i] : 0.0f;
        pv[k] = (in && !kFirst) ? p_old[i] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < RW + 2; ++k)
    {
        const float d = hsl_invd(A, cl[k]) * rv[k];
        pv[k] = kFirst ? d : d + beta * pv[k];
    }
    Sum2 v[1];
#pragma unroll
    for (int k = 1; k <= RW; ++k)
    {
        const float pe = __shfl_down_sync(0xffffffffu, pv[k], 1), pw = __shfl_up_sync(0xffffffffu, pv[k], 1);
        if (t.own && t.r0 - 1 + k < nr)
        {
            p[static_cast<std::int64_t>(t.r0 - 1 + k) * nc + t.c] = pv[k];
            if (cl[k]) v[0].add(pv[k] * hsl_op(A, pv[k], pv[k - 1], pe, pv[k + 1], pw, cl[k]));
        }
    }
    const unsigned nblk = gridDim.x;
    block_partials<1>(v, A.part, nblk);
    if (!last_block(&A.S->arrived, nblk)) return;
    double s[1];
    total_partials<1>(A.part, nblk, s);
    if (threadIdx.x == 0) A.S->alpha = s[0] > 0.0 ? static_cast<float>(A.S->rz / s[0]) : 0.0f;
}

template <int RW>
__global__ void __launch_bounds__(256) hsl_update(HslArgs A, const float* __restrict__ p, float* __restrict__ x,
                                                  float* __restrict__ r)
{
    LSDTT_COUNT();
    if (A.S->done) return;
    const int nr = A.H.nr, nc = A.H.nc;
    const Strip t(A.H, RW);
    const float alpha = A.S->alpha;
    float pv[RW + 2], xv[RW], rv[RW];
    unsigned cl[RW];
#pragma unroll
    for (int k = 0; k < RW + 2; ++k)
    {
        const int row = t.row(k);
        const std::int64_t i = static_cast<std::int64_t>(row) * nc + t.c;
        pv[k] = row >= 0 ? p[i] : 0.0f;
        if (k >= 1 && k <= RW)
        {
            const bool in = t.own && t.r0 - 1 + k < nr;
            cl[k - 1] = in ? A.cls[i] : 0u;
            xv[k - 1] = in ? x[i] : 0.0f;
            rv[k - 1] = in ? r[i] : 0.0f;
        }
    }
    Sum2 v[2];
#pragma unroll
    for (int k = 1; k <= RW; ++k)
    {
        const float pe = __shfl_down_sync(0xffffffffu, pv[k], 1), pw = __shfl_up_sync(0xffffffffu, pv[k], 1);
        const unsigned c1 = cl[k - 1];
        if (c1)
        {
            const std::int64_t i = static_cast<std::int64_t>(t.r0 - 1 + k) * nc + t.c;
            x[i] = xv[k - 1] + alpha * pv[k];
            const float ri = rv[k - 1] - alpha * hsl_op(A, pv[k], pv[k - 1], pe, pv[k + 1], pw, c1);
            r[i] = ri;
            v[0].add(ri * (ri * hsl_invd(A, c1)));
            v[1].add(ri * ri);
        }
    }
    const unsigned nblk = gridDim.x;
    block_partials<2>(v, A.part, nblk);
    if (!last_block(&A.S->arrived, nblk)) return;
    double s[2];
    total_partials<2>(A.part, nblk, s);
    if (threadIdx.x == 0)
    {
        HsState& S = *A.S;
        S.beta = S.rz > 0.0 ? static_cast<float>(s[0] / S.rz) : 0.0f;
        S.rz = s[0];
        S.rr = s[1];
        const int it = ++S.iters;
        if (it % 4 == 0 || it >= A.max_iter)
        {
            S.rel = sqrt(s[1]) / sqrt(S.bb);
            if (S.rel <= A.rel_tol || it >= A.max_iter) S.done = 1;
        }
    }
}

__global__ void hs_finish(std::int64_t n, const std::uint8_t* __restrict__ dof, const float* __restrict__ z,
                          const float* __restrict__ x, float* __restrict__ out)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = dof[i] ? __fadd_rn(z[i], x[i]) : z[i];  // the exact sum, rounded once
}

}  // namespace
}  // namespace lsdtt_gb300

using namespace lsdtt_gb300;

extern "C" int lsdtt_gpu_hillslope_linear_implicit(const lsdtt_gpu_grid* grid, const float* z_dev,
                                                   const std::uint8_t* mask_dev, const std::uint8_t* is_channel_dev,
                                                   float D, float dt, double rel_tol, int32_t max_iter,
                                                   float* z_out_dev, lsdtt_gpu_solve_report* report, void* stream)
{
    if (!grid || !z_dev || !mask_dev || !z_out_dev)
        return fail(LSDTT_GPU_EINVAL, "lsdtt_gpu_hillslope_linear_implicit: null argument");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        return fail(LSDTT_GPU_ENODEV, "lsdtt_gpu_hillslope_linear_implicit: no CUDA device");
    if (!(grid->n_rows > 0 && grid->n_cols > 0 && grid->cell_size > 0.0))
        return fail(LSDTT_GPU_EINVAL, "lsdtt_gpu_hillslope_linear_implicit: raster metadata is invalid");
    if (!(dt > 0.0f)) return fail(LSDTT_GPU_EINVAL, "lsdtt_gpu_hillslope_linear_implicit: dt must be positive");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const std::int64_t n = static_cast<std::int64_t>(grid->n_rows) * grid->n_cols;
    Hs H{};
    H.nr = grid->n_rows;
    H.nc = grid->n_cols;
    const char* b = grid->boundary_conditions;
    H.bn = b[0]; H.be = b[1]; H.bs = b[2]; H.bw = b[3];
    const double h = grid->cell_size;
    H.DA = static_cast<double>(D) / (h * h);
    H.inv_dt = 1.0 / static_cast<double>(dt);
    H.U = 0.0;
    // Scratch: x, r, two directions (f32), classes u8, partials, state.
    const int kMaxIt = max_iter > 0 ? max_iter : 1000;
    const std::size_t fbytes = (sizeof(float) * static_cast<std::size_t>(n) + 255) & ~std::size_t(255);
    const std::size_t cbytes = (static_cast<std::size_t>(n) + 255) & ~std::size_t(255);
    const int ntx = (H.nc + kHslTC - 1) / kHslTC;
    const unsigned tiles8 = static_cast<unsigned>(ntx) * static_cast<unsigned>((H.nr + 7) / 8);
    const bool tall = strip_long(H.nr, H.nc);
    const unsigned tiles = strip_blocks(H.nr, H.nc, tall ? 16 : 8);
    const std::size_t need = 4 * fbytes + cbytes + sizeof(double) * 2 * static_cast<std::size_t>(std::max(tiles8, tiles)) + 1024;
    char* base = nullptr;
    cudaError_t e = cudaMallocAsync(&base, need, st);
    if (e != cudaSuccess) return cuda_fail(e, "lsdtt_gpu_hillslope_linear_implicit");
    float* x = reinterpret_cast<float*>(base);
    float* r = reinterpret_cast<float*>(base + fbytes);
    float* pbuf[2] = {reinterpret_cast<float*>(base + 2 * fbytes), reinterpret_cast<float*>(base + 3 * fbytes)};
    std::uint8_t* cls = reinterpret_cast<std::uint8_t*>(base + 4 * fbytes);
    HslArgs A{};
    A.S = reinterpret_cast<HsState*>(base + 4 * fbytes + cbytes);
    A.part = reinterpret_cast<double*>(base + 4 * fbytes + cbytes + 512);
    A.H = H;
    A.inv_dt = static_cast<float>(H.inv_dt);
    A.DA = static_cast<float>(H.DA);
    for (int f = 0; f < 5; ++f) A.invd[f] = static_cast<float>(1.0 / (H.inv_dt + H.DA * f));
    A.mask = mask_dev;
    A.cls = cls;
    A.rel_tol = rel_tol;
    A.max_iter = kMaxIt;
    cudaMemsetAsync(A.S, 0, sizeof(HsState), st);
    const unsigned nb = grid_blocks(n, 256);
    hsl_setup<<<tiles8, 256, 0, st>>>(A, is_channel_dev, z_dev, cls, r, x);
    // Iterations in batches, each followed by one read of the state; a batch
    // launched past convergence returns at once.
    HsState S{};
    int queued = 0, batch = 4;
    while (e == cudaSuccess)
    {
        for (int k = 0; k < batch && queued < kMaxIt; ++k, ++queued)
        {
            const float* po = pbuf[(queued + 1) & 1];
            float* p = pbuf[queued & 1];
            // Algorithmic bytes: residual 4, class 1, old direction 4 in, direction 4 out.
            LSDTT_TIMED("hillslope_apply", 13.0 * static_cast<double>(n), st, ({
                            if (tall)
                            {
                                if (queued == 0) hsl_direction<16, true><<<tiles, 256, 0, st>>>(A, r, po, p);
                                else hsl_direction<16, false><<<tiles, 256, 0, st>>>(A, r, po, p);
                            }
                            else if (queued == 0) hsl_direction<8, true><<<tiles, 256, 0, st>>>(A, r, po, p);
                            else hsl_direction<8, false><<<tiles, 256, 0, st>>>(A, r, po, p);
                        }));
            if (tall) hsl_update<16><<<tiles, 256, 0, st>>>(A, p, x, r);
            else hsl_update<8><<<tiles, 256, 0, st>>>(A, p, x, r);
        }
        cudaMemcpyAsync(&S, A.S, sizeof(S), cudaMemcpyDeviceToHost, st);
        e = cudaStreamSynchronize(st);
        if (S.done || queued >= kMaxIt) break;
        batch = std::min(16, batch + 4);
    }
    const int it = S.iters;
    const double rel = S.rel, finf0 = S.finf;
    const bool converged = S.bb == 0.0 || (it > 0 && rel <= rel_tol);
    if (e == cudaSuccess)
    {
        hs_finish<<<nb, 256, 0, st>>>(n, cls, z_dev, x, z_out_dev);
        e = cudaStreamSynchronize(st);
    }
    cudaFreeAsync(base, st);
    if (e != cudaSuccess) return cuda_fail(e, "lsdtt_gpu_hillslope_linear_implicit");
    if (report)
    {
        *report = lsdtt_gpu_solve_report{};
        report->iterations = it;
        report->relative_residual = rel;
        report->initial_residual_inf = finf0;
        report->converged = converged ? 1 : 0;
        report->linear_solves = 1;
        report->explicit_relative_residual = -1.0;  // not computed on this path
    }
    if (!converged)
        return fail(LSDTT_GPU_ENOCONV, "lsdtt_gpu_hillslope_linear_implicit: Jacobi-PCG did not reach the relative "
                                       "residual within max_iter iterations");
    return LSDTT_GPU_OK;
}

namespace lsdtt_gb300
{
LSDTT_DEFINE_LAUNCH_READER(hillslope)
}  // namespace lsdtt_gb300

// ===========================================================================
// Nonlinear (Roering) implicit step.
//
// compute_hillslope_newton_transient with nonlinear = true: the face
// coefficient alpha_f = 1/(1 - min((S_n^2 + S_t^2)/Sc^2, cap)) with the
// tangential slope averaged across the face (operator_cpu.hpp:229-321), so
// alpha is a property of the face and the lagged-coefficient (Picard)
// operator
//     (A x)_P = inv_dt x_P + (D/h^2) sum_f alpha_f (x_P - [nb DOF] x_nb)
// is symmetric positive definite. Each outer iteration evaluates F(z) in
// FP64 on an FP64 working field, solves A(alpha(z)) dz = -F by Jacobi-PCG
// (FP32 vectors, FP64 dot products, relative residual rel_tol) and takes the
// largest step lambda = 1, 1/2, ... that keeps every face sub-critical and
// lowers ||F||_inf, restoring feasibility first when the iterate starts
// super-critical (newton_cpu.cpp:553-641). Converged when ||F||_inf <=
// residual_tol (1e-12 m/yr, the reference's default). Sub-steps follow the
// reference controller (newton_cpu.cpp:690-788): start with the whole dt,
// halve on failure, grow x1.7 after an easy step. The outer iteration is a
// fixed point on the symmetric operator rather than the reference's Newton
// on the 9-point Jacobian, so iteration counts differ; the converged field
// is the same root of F.
// ===========================================================================
namespace lsdtt_gb300
{
namespace
{

struct HsN
{
    Hs H;
    double Sc2;
    double cap;
    double h;
    int nonlinear;
    // reciprocals formed once on the host (hsn_reciprocals): FP64 division
    // is a long instruction sequence on this part, and the evaluation would
    // otherwise divide ~18 times per cell
    double inv_h, inv_2h, inv_Sc2, inv_Sc;
};

inline void hsn_reciprocals(HsN& P)
{
    P.inv_h = 1.0 / P.h;
    P.inv_2h = 1.0 / (2.0 * P.h);
    P.inv_Sc2 = 1.0 / P.Sc2;
    P.inv_Sc = 1.0 / std::sqrt(P.Sc2);
}

// Neighbour (rr, cc) of (r, c) in direction (dr, dc) by the boundary rules
// of hs_nb (wrap on 'p', else the cell itself; a masked neighbour is the
// cell itself), without forming the flat index.
__device__ __forceinline__ void hs_nb_rc(const Hs& H, const std::uint8_t* mask, int r, int c, int dr, int dc, int& rr,
                                         int& cc)
{
    rr = r + dr;
    cc = c + dc;
    if (rr < 0) rr = (H.bn == 'p') ? H.nr - 1 : r;
    else if (rr >= H.nr) rr = (H.bs == 'p') ? 0 : r;
    if (cc < 0) cc = (H.bw == 'p') ? H.nc - 1 : c;
    else if (cc >= H.nc) cc = (H.be == 'p') ? 0 : c;
    if (!hs_valid(mask, H.nc, rr, cc))
    {
        rr = r;
        cc = c;
    }
}

__device__ __forceinline__ double hs_slope_x(const HsN& P, const std::uint8_t* mask, const double* z, int r, int c)
{
    const std::int64_t e = hs_nb(P.H, mask, r, c, 0, 1), w = hs_nb(P.H, mask, r, c, 0, -1);
    return (z[e] - z[w]) * P.inv_2h;
}

__device__ __forceinline__ double hs_slope_y(const HsN& P, const std::uint8_t* mask, const double* z, int r, int c)
{
    const std::int64_t s = hs_nb(P.H, mask, r, c, 1, 0), n = hs_nb(P.H, mask, r, c, -1, 0);
    return (z[s] - z[n]) * P.inv_2h;
}

// Per DOF: face alphas (float4 N,E,S,W), residual F (double), and the
// reductions ||F||_inf, ||F||_2^2, max |grad z|/Sc (feasibility).
__global__ void hsn_eval(HsN P, const std::uint8_t* __restrict__ mask, const std::uint8_t* __restrict__ dof,
                         const double* __restrict__ z, const double* __restrict__ zn, float4* __restrict__ alpha,
                         double* __restrict__ F, double* __restrict__ acc)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const std::int64_t n = static_cast<std::int64_t>(P.H.nr) * P.H.nc;
    double finf = 0.0, f2 = 0.0, ratio = 0.0;
    if (i < n && dof[i])
    {
        const int r = static_cast<int>(i / P.H.nc), c = static_cast<int>(i % P.H.nc);
        const double zc = z[i];
        const double sxc = P.nonlinear ? hs_slope_x(P, mask, z, r, c) : 0.0;
        const double syc = P.nonlinear ? hs_slope_y(P, mask, z, r, c) : 0.0;
        double a[4];
        double flux = 0.0;
#pragma unroll
        for (int f = 0; f < 4; ++f)
        {
            int jr, jc;
            hs_nb_rc(P.H, mask, r, c, kDr[f], kDc[f], jr, jc);
            const std::int64_t j = static_cast<std::int64_t>(jr) * P.H.nc + jc;
            const double sn = (z[j] - zc) * P.inv_h;
            double al = 1.0;
            if (P.nonlinear)
            {
                const double st = (f == 0 || f == 2) ? 0.5 * (sxc + hs_slope_x(P, mask, z, jr, jc))
                                                     : 0.5 * (syc + hs_slope_y(P, mask, z, jr, jc));
                const double s2 = fmin((sn * sn + st * st) * P.inv_Sc2, P.cap);
                al = 1.0 / (1.0 - s2);
            }
            a[f] = al;
            flux += al * sn * P.h;
        }
        alpha[i] = make_float4(static_cast<float>(a[0]), static_cast<float>(a[1]), static_cast<float>(a[2]),
                               static_cast<float>(a[3]));
        double Fv = -P.H.U - P.H.DA * flux;
        if (P.H.inv_dt > 0.0) Fv += P.H.inv_dt * (zc - zn[i]);
        F[i] = Fv;
        finf = fabs(Fv);
        f2 = Fv * Fv;
        if (P.nonlinear) ratio = sqrt(sxc * sxc + syc * syc) * P.inv_Sc;
    }
    else if (i < n)
    {
        F[i] = 0.0;
        alpha[i] = make_float4(1.f, 1.f, 1.f, 1.f);
    }
    block_atomic_max_nonneg(&acc[0], finf);
    block_atomic_add(&acc[1], f2);
    block_atomic_max_nonneg(&acc[2], ratio);
}

// PCG set-up for A(alpha) x = -F: inverse diagonal, b, x = 0, r = b,
// p = M^-1 r, acc[0] = r.z, acc[1] = ||b||^2.
__global__ void hsn_pcg_init(HsN P, const std::uint8_t* __restrict__ mask, const std::uint8_t* __restrict__ dof,
                             const float4* __restrict__ alpha, const double* __restrict__ F,
                             float* __restrict__ invd, float* __restrict__ b, float* __restrict__ x,
                             float* __restrict__ r, float* __restrict__ p, double* __restrict__ acc)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const std::int64_t n = static_cast<std::int64_t>(P.H.nr) * P.H.nc;
    double rz = 0.0, bb = 0.0;
    if (i < n)
    {
        float id = 0.0f, bi = 0.0f;
        if (dof[i])
        {
            const int rr = static_cast<int>(i / P.H.nc), cc = static_cast<int>(i % P.H.nc);
            const float4 a = alpha[i];
            const float av[4] = {a.x, a.y, a.z, a.w};
            double diag = P.H.inv_dt;
#pragma unroll
            for (int f = 0; f < 4; ++f)
                if (hs_nb(P.H, mask, rr, cc, kDr[f], kDc[f]) != i) diag += P.H.DA * av[f];
            id = static_cast<float>(1.0 / diag);
            bi = static_cast<float>(-F[i]);
        }
        invd[i] = id;
        b[i] = bi;
        x[i] = 0.0f;
        r[i] = bi;
        const float zi = bi * id;
        p[i] = zi;
        rz = static_cast<double>(bi) * zi;
        bb = static_cast<double>(bi) * bi;
    }
    block_atomic_add(&acc[0], rz);
    block_atomic_add(&acc[1], bb);
}

// ---- operator and fixed-order reductions of the PCG loops -------------------
// The loops below run the operator over strips and the learned
// preconditioner's smoothing over 128 x 32 tiles (the network's output staged
// in shared memory with a one-cell halo), write one partial per block (HsParts)
// instead of atomics on a single address, and add the partials in a fixed
// order in one block, which also forms alpha or beta once (FP64 on this part is
// a narrow pipe: one division per block stalled every block behind its thread 0).

// FP32 sum over the warp (lane 0 gets it; 32 terms, as block_atomic_add_f).
__device__ __forceinline__ float warp_sum_f(float v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Block total of per-warp FP64 sums (lane 0 of each warp holds one), in warp
// order, stored by thread 0 at dst.
__device__ __forceinline__ void block_store_d(double v, double* dst)
{
    __shared__ double sh_store_d[32];
    __syncthreads();  // a previous call may still be reading
    if ((threadIdx.x & 31) == 0) sh_store_d[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = sh_store_d[0];
        for (int k = 1; k < static_cast<int>(blockDim.x >> 5); ++k) t += sh_store_d[k];
        *dst = t;
    }
}

// Operator value at a cell of the tile: inv_dt x_P + (D/h^2) sum_f alpha_f
// (x_P - [nb DOF] x_nb) in FP32 (the difference form keeps the operator
// symmetric: alpha is a property of the face), the faces summed in the order
// N, E, S, W on both paths. Fast cells (class bit 1: interior, all four neighbours
// DOFs) read the neighbours from the tile; other DOFs resolve them by the
// boundary rules and `xg` (the global value of a cell).
template <class XG>
__device__ __forceinline__ float hs_op_cell(const HsN& P, float inv_dt, float DA, const std::uint8_t* __restrict__ mask,
                                            const std::uint8_t* __restrict__ dof, const float4* __restrict__ alpha,
                                            const float (&sx)[kHsTR + 2][132], int lr, int lc, int r, int c,
                                            std::int64_t i, std::uint8_t kd, XG xg)
{
    const float xi = sx[lr][lc];
    if (kd == 0) return 0.0f;
    const float4 a = alpha[i];
    float s = 0.0f;
    if (kd & 2)
    {
        s += a.x * (xi - sx[lr - 1][lc]);
        s += a.y * (xi - sx[lr][lc + 1]);
        s += a.z * (xi - sx[lr + 1][lc]);
        s += a.w * (xi - sx[lr][lc - 1]);
    }
    else
    {
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int f = 0; f < 4; ++f)
        {
            const std::int64_t j = hs_nb(P.H, mask, r, c, kDr[f], kDc[f]);
            if (j == i) continue;
            s += av[f] * (xi - (dof[j] ? xg(j) : 0.0f));
        }
    }
    return inv_dt * xi + DA * s;
}

// Stage x over the tile and its one-cell halo (0 outside the grid): warp w
// loads rows w, w + 8, ...; each lane columns lane, lane + 32, ...
template <class XG>
__device__ __forceinline__ void hs_stage_tile(float (&sx)[kHsTR + 2][132], int nr, int nc, int r0, int c0, XG xg)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int lr = w; lr < kHsTR + 2; lr += 8)
    {
        const int r = r0 - 1 + lr;
        const bool row_in = r >= 0 && r < nr;
        const std::int64_t rb = static_cast<std::int64_t>(r) * nc;
#pragma unroll
        for (int k = 0; k < 5; ++k)
        {
            const int col = 32 * k + lane;
            if (col >= 130) continue;
            const int c = c0 - 1 + col;
            sx[lr][col] = (row_in && c >= 0 && c < nc) ? xg(rb + c) : 0.0f;
        }
    }
    __syncthreads();
}

// The PCG loops' state beside the coefficients scal[0] (alpha), scal[1] (beta).
struct HsnLoop
{
    double rel;
    int iters, done;
    unsigned arrived, pad;
};

// Ap = A p and p.Ap into *pap_out, from which the last block forms
// alpha = *rz / p.Ap (scal[0]), over strips as in the linear step (10.9 us at
// 1024 x 1000; 21 us over 128 x 32 tiles, whose edge warps resolved each
// neighbour by loads and of which there were only 256). With kFuse
// the direction update of the previous iteration, p = z + beta p
// (beta = scal[1]), is formed on the way: p_src is read, p_dst written.
template <bool kFuse, int RW>
__global__ void __launch_bounds__(256) hsn_apply_t(HsN P, float inv_dt, float DA, const std::uint8_t* __restrict__ mask,
                                                   const std::uint8_t* __restrict__ dof,
                                                   const float4* __restrict__ alpha, float* __restrict__ scal,
                                                   const float* __restrict__ zz, const float* __restrict__ p_src,
                                                   float* __restrict__ p_dst, float* __restrict__ Ap,
                                                   double* __restrict__ part, HsnLoop* __restrict__ L,
                                                   const double* __restrict__ rz, double* __restrict__ pap_out)
{
    LSDTT_COUNT();
    if (L->done) return;
    const int nr = P.H.nr, nc = P.H.nc;
    const Strip t(P.H, RW);
    const float beta = kFuse ? scal[1] : 0.0f;
    float pv[RW + 2], zv[RW + 2];
    float4 av[RW];
    unsigned kd[RW];
#pragma unroll
    for (int k = 0; k < RW + 2; ++k)
    {
        const int row = t.row(k);
        const bool in = row >= 0;
        const std::int64_t i = static_cast<std::int64_t>(row) * nc + t.c;
        pv[k] = in ? p_src[i] : 0.0f;
        zv[k] = (kFuse && in) ? zz[i] : 0.0f;
        if (k >= 1 && k <= RW)
        {
            const bool mine = t.own && t.r0 - 1 + k < nr;
            kd[k - 1] = mine ? dof[i] : 0u;
            av[k - 1] = mine ? alpha[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    if (kFuse)
    {
#pragma unroll
        for (int k = 0; k < RW + 2; ++k) pv[k] = zv[k] + beta * pv[k];
    }
    Sum2 v[1];
#pragma unroll
    for (int k = 1; k <= RW; ++k)
    {
        const float pe = __shfl_down_sync(0xffffffffu, pv[k], 1), pw = __shfl_up_sync(0xffffffffu, pv[k], 1);
        const int row = t.r0 - 1 + k;
        if (!t.own || row >= nr) continue;
        const std::int64_t i = static_cast<std::int64_t>(row) * nc + t.c;
        const float pi = pv[k];
        const float4 a = av[k - 1];
        const unsigned cl = kd[k - 1];
        float s = 0.0f;
        s += (cl & 4u) ? a.x * (pi - pv[k - 1]) : 0.0f;
        s += (cl & 8u) ? a.y * (pi - pe) : 0.0f;
        s += (cl & 16u) ? a.z * (pi - pv[k + 1]) : 0.0f;
        s += (cl & 32u) ? a.w * (pi - pw) : 0.0f;
        const float o = cl ? inv_dt * pi + DA * s : 0.0f;
        if (kFuse) p_dst[i] = pi;
        Ap[i] = o;
        if (cl) v[0].add(pi * o);
    }
    const unsigned nblk = gridDim.x;
    block_partials<1>(v, part, nblk);
    if (!last_block(&L->arrived, nblk)) return;
    double s[1];
    total_partials<1>(part, nblk, s);
    if (threadIdx.x == 0)
    {
        *pap_out = s[0];
        scal[0] = s[0] > 0.0 ? static_cast<float>(*rz / s[0]) : 0.0f;
    }
}

// The smoothing step of the learned preconditioner over one tile per block:
// y = [DOF] ynet (staged), t = A y, z = y + D^-1 (r - t) into zz; partials
// part_rz[tile] = r.z and part_roz[tile] = z.(r - r_old). Same arithmetic as
// masking, applying the operator and smoothing in three passes.
__global__ void __launch_bounds__(256) hsf_smooth_t(HsN P, float inv_dt, float DA, const std::uint8_t* __restrict__ mask,
                                                    const std::uint8_t* __restrict__ dof,
                                                    const float4* __restrict__ alpha, const float* __restrict__ ynet,
                                                    const float* __restrict__ invd, const float* __restrict__ r,
                                                    const float* __restrict__ ro, float* __restrict__ zz,
                                                    double* __restrict__ part_rz, double* __restrict__ part_roz)
{
    LSDTT_COUNT();
    __shared__ float sx[kHsTR + 2][132];
    const int nr = P.H.nr, nc = P.H.nc;
    const int ntx = (nc + kHsTC - 1) / kHsTC;
    const int c0 = (blockIdx.x % ntx) * kHsTC, r0 = (blockIdx.x / ntx) * kHsTR;
    auto yg = [&](std::int64_t k) { return dof[k] ? ynet[k] : 0.0f; };
    hs_stage_tile(sx, nr, nc, r0, c0, yg);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double rz_d = 0.0, roz_d = 0.0;
#pragma unroll 1
    for (int qr = 0; qr < 4; ++qr)
    {
        const int lr = 1 + w * 4 + qr, rw = r0 + lr - 1;
        if (rw >= nr) break;  // warp-uniform
        const std::int64_t rb = static_cast<std::int64_t>(rw) * nc;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const int lc = 1 + 32 * k + lane, c = c0 + lc - 1;
            float rz = 0.0f, roz = 0.0f;
            if (c < nc)
            {
                const std::int64_t i = rb + c;
                const float t = hs_op_cell(P, inv_dt, DA, mask, dof, alpha, sx, lr, lc, rw, c, i, dof[i], yg);
                const float ri = r[i];
                const float zi = sx[lr][lc] + invd[i] * (ri - t);
                zz[i] = zi;
                rz = ri * zi;
                roz = zi * (ri - ro[i]);
            }
            rz = warp_sum_f(rz);
            roz = warp_sum_f(roz);
            if (lane == 0)
            {
                rz_d += static_cast<double>(rz);
                roz_d += static_cast<double>(roz);
            }
        }
    }
    block_store_d(rz_d, part_rz + blockIdx.x);
    block_store_d(roz_d, part_roz + blockIdx.x);
}

// Jacobi-PCG update with alpha = scal[0]: x += alpha p; r -= alpha Ap;
// zz = D^-1 r; r.z and r.r into out[0], out[1] (FP32 over four cells, two
// words beyond), from which the last block forms beta = r.z / *rz (scal[1]) and
// tests convergence every fourth iteration. Four cells a thread and access.
__global__ void __launch_bounds__(256) hs_update_g(std::int64_t n, float* __restrict__ scal,
                                                  const float* __restrict__ inv_diag, const float* __restrict__ p,
                                                  const float* __restrict__ Ap, float* __restrict__ x,
                                                  float* __restrict__ r, float* __restrict__ zz,
                                                  double* __restrict__ part, HsnLoop* __restrict__ L,
                                                  const double* __restrict__ rz, double* __restrict__ out, double bnorm,
                                                  double rel_tol, int max_iter)
{
    LSDTT_COUNT();
    if (L->done) return;
    const float alpha = scal[0];
    Sum2 v[2];
    const std::int64_t t0 = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const std::int64_t stride = static_cast<std::int64_t>(gridDim.x) * blockDim.x, n4 = n >> 2;
    for (std::int64_t q = t0; q < n4; q += stride)
    {
        const float4 pv = reinterpret_cast<const float4*>(p)[q], av = reinterpret_cast<const float4*>(Ap)[q];
        const float4 dv = reinterpret_cast<const float4*>(inv_diag)[q];
        float4 xv = reinterpret_cast<float4*>(x)[q], rv = reinterpret_cast<float4*>(r)[q];
        xv.x += alpha * pv.x;
        xv.y += alpha * pv.y;
        xv.z += alpha * pv.z;
        xv.w += alpha * pv.w;
        rv.x -= alpha * av.x;
        rv.y -= alpha * av.y;
        rv.z -= alpha * av.z;
        rv.w -= alpha * av.w;
        const float4 zv = make_float4(rv.x * dv.x, rv.y * dv.y, rv.z * dv.z, rv.w * dv.w);
        reinterpret_cast<float4*>(x)[q] = xv;
        reinterpret_cast<float4*>(r)[q] = rv;
        reinterpret_cast<float4*>(zz)[q] = zv;
        v[0].add((rv.x * zv.x + rv.y * zv.y) + (rv.z * zv.z + rv.w * zv.w));
        v[1].add((rv.x * rv.x + rv.y * rv.y) + (rv.z * rv.z + rv.w * rv.w));
    }
    if (t0 < (n & 3))
    {
        const std::int64_t i = 4 * n4 + t0;
        x[i] += alpha * p[i];
        const float ri = r[i] - alpha * Ap[i], zi = ri * inv_diag[i];
        r[i] = ri;
        zz[i] = zi;
        v[0].add(ri * zi);
        v[1].add(ri * ri);
    }
    const unsigned nblk = gridDim.x;
    block_partials<2>(v, part, nblk);
    if (!last_block(&L->arrived, nblk)) return;
    double t[2];
    total_partials<2>(part, nblk, t);
    if (threadIdx.x == 0)
    {
        out[0] = t[0];
        out[1] = t[1];
        scal[1] = *rz > 0.0 ? static_cast<float>(t[0] / *rz) : 0.0f;
        const int it = ++L->iters;
        if (it % 4 == 0 || it >= max_iter)
        {
            L->rel = sqrt(t[1]) / bnorm;
            if (L->rel <= rel_tol) L->done = 1;
        }
    }
}

// Flexible-PCG update with alpha = scal[0]: x += alpha p; r_old = r;
// r -= alpha Ap; q = D^-1 r (the network's input); part[blk] = r.r.
__global__ void __launch_bounds__(256) hsf_update_g(std::int64_t n, const float* __restrict__ scal,
                                                   const float* __restrict__ invd, const float* __restrict__ p,
                                                   const float* __restrict__ Ap, float* __restrict__ x,
                                                   float* __restrict__ r, float* __restrict__ ro,
                                                   float* __restrict__ q, double* __restrict__ part)
{
    LSDTT_COUNT();
    const float alpha = scal[0];
    const int lane = threadIdx.x & 31;
    double rr_d = 0.0;
    const std::int64_t stride = static_cast<std::int64_t>(gridDim.x) * blockDim.x;
    for (std::int64_t b = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + (threadIdx.x & ~31); b < n;
         b += stride)
    {
        const std::int64_t i = b + lane;
        float rr = 0.0f;
        if (i < n)
        {
            x[i] += alpha * p[i];
            const float r0 = r[i];
            ro[i] = r0;
            const float ri = r0 - alpha * Ap[i];
            r[i] = ri;
            q[i] = invd[i] * ri;
            rr = ri * ri;
        }
        rr = warp_sum_f(rr);
        if (lane == 0) rr_d += static_cast<double>(rr);
    }
    block_store_d(rr_d, part + blockIdx.x);
}

// One block: dst[q] = sum of part[q][0 .. count[q]) in a fixed order (each
// thread a strided run, then the warps' shuffle trees in order), for the
// quantities with a partial array; then scal = float(num / den) when den > 0
// (else 0), the PCG step or direction coefficient.
struct HsRed
{
    const double* part[4];
    int count[4];
    double* dst[4];
    const double* num;
    const double* den;
    float* scal;
};

__global__ void __launch_bounds__(512) hs_reduce(HsRed R)
{
    LSDTT_COUNT();
    __shared__ double sh[4][16];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        if (!R.part[q]) continue;
        double s = 0.0;
        for (int k = threadIdx.x; k < R.count[q]; k += blockDim.x) s += R.part[q][k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) sh[q][w] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int q = 0; q < 4; ++q)
        {
            if (!R.part[q]) continue;
            double t = sh[q][0];
            for (int k = 1; k < static_cast<int>(blockDim.x >> 5); ++k) t += sh[q][k];
            *R.dst[q] = t;
        }
        if (R.scal)
        {
            const double den = *R.den;
            *R.scal = (den > 0.0) ? static_cast<float>(*R.num / den) : 0.0f;
        }
    }
}

// z_try = z + lambda * dz on DOFs (double)
__global__ void hsn_axpy(std::int64_t n, const std::uint8_t* __restrict__ dof, const double* __restrict__ z,
                         const float* __restrict__ dz, double lambda, double* __restrict__ zt)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    zt[i] = dof[i] ? z[i] + lambda * static_cast<double>(dz[i]) : z[i];
}

__global__ void hsn_to_double(std::int64_t n, const float* __restrict__ a, double* __restrict__ b)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[i];
}

__global__ void hsn_to_float(std::int64_t n, const double* __restrict__ a, float* __restrict__ b)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) b[i] = static_cast<float>(a[i]);
}

// ---- flexible PCG with the learned preconditioner --------------------------
// Per-iteration reduction slot (4 doubles): [0] p.Ap, [1] r.z, [2] r.r,
// [3] z.(r - r_old). beta = z.(r - r_old) / r_old.z_old (Polak-Ribiere),
// which keeps conjugacy when M^-1 changes from one iteration to the next.

// The network's input: the Jacobi-scaled residual D^-1 r (metres), which
// carries the local stiffness of the lagged-coefficient operator.
__global__ void hsf_input(std::int64_t n, const float* __restrict__ invd, const float* __restrict__ r,
                          float* __restrict__ q)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) q[i] = invd[i] * r[i];
}

// Explicit residual res = b - A x, evaluated in FP64 from the FP32 iterate and
// stored (FP32) in r. acc[0] += ||res||^2; acc[1] += sum_i (diag_i |x_i|
// 2^-24)^2, the residual that rounding x to FP32 alone can leave (the
// representation floor the acceptance check allows for).
__global__ void hsn_explicit(HsN P, const std::uint8_t* __restrict__ mask, const std::uint8_t* __restrict__ dof,
                             const float4* __restrict__ alpha, const float* __restrict__ b,
                             const float* __restrict__ x, float* __restrict__ r, double* __restrict__ acc)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const std::int64_t n = static_cast<std::int64_t>(P.H.nr) * P.H.nc;
    double rr = 0.0, fl = 0.0;
    if (i < n)
    {
        double res = 0.0;
        if (dof[i])
        {
            const int rw = static_cast<int>(i / P.H.nc), cl = static_cast<int>(i % P.H.nc);
            const float4 a = alpha[i];
            const float av[4] = {a.x, a.y, a.z, a.w};
            const double xi = x[i];
            double diag = P.H.inv_dt, off = 0.0;
#pragma unroll
            for (int f = 0; f < 4; ++f)
            {
                const std::int64_t j = hs_nb(P.H, mask, rw, cl, kDr[f], kDc[f]);
                if (j == i) continue;
                diag += P.H.DA * av[f];
                if (dof[j]) off += P.H.DA * av[f] * static_cast<double>(x[j]);
            }
            res = static_cast<double>(b[i]) - (diag * xi - off);
            const double u = diag * fabs(xi) * 5.9604644775390625e-8;
            fl = u * u;
        }
        r[i] = static_cast<float>(res);
        rr = res * res;
    }
    block_atomic_add(&acc[0], rr);
    block_atomic_add(&acc[1], fl);
}

// Jacobi-PCG restart from the residual in r: z = p = D^-1 r, acc[0] = r.z
__global__ void hsn_restart(std::int64_t n, const float* __restrict__ invd, const float* __restrict__ r,
                            float* __restrict__ p, double* __restrict__ acc)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    double rz = 0.0;
    if (i < n)
    {
        const float zi = r[i] * invd[i];
        p[i] = zi;
        rz = static_cast<double>(r[i]) * zi;
    }
    block_atomic_add(&acc[0], rz);
}

__global__ void hsn_pair_finish(std::int64_t n, const float* __restrict__ x_final, const float* __restrict__ invd,
                                float* __restrict__ r_slot, float* __restrict__ e_slot)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r_slot[i] = invd[i] * r_slot[i];
    e_slot[i] = x_final[i] - e_slot[i];
}

struct HsnBuf
{
    std::uint8_t* dof;
    double *z, *zn, *zt, *F, *acc;
    float4* alpha;
    float *invd, *b, *x, *r, *p, *zz, *Ap, *ro;
    float* p2;     // the other direction buffer of the fused apply
    double* part;  // block partials (HsParts)
    float* scal;   // [0] alpha, [1] beta of the current iteration
    HsnLoop* loop; // the loop's state, in the same 256 bytes
    double* hacc;
};

// Device bytes of p2, the partials and the scalars for an n-cell grid
// (256-byte aligned pieces).
inline std::size_t hsn_pcg_bytes(int nr, int nc)
{
    const std::size_t n = static_cast<std::size_t>(nr) * nc;
    return (4 * n + 255) / 256 * 256 +
           (sizeof(double) * hs_parts(nr, nc).total + 255) / 256 * 256 + 256;
}

template <class Carve>
void hsn_pcg_carve(HsnBuf& B, int nr, int nc, Carve carve)
{
    const std::size_t n = static_cast<std::size_t>(nr) * nc;
    B.p2 = reinterpret_cast<float*>(carve(4 * n));
    B.part = reinterpret_cast<double*>(carve(sizeof(double) * hs_parts(nr, nc).total));
    B.scal = reinterpret_cast<float*>(carve(256));
    B.loop = reinterpret_cast<HsnLoop*>(B.scal + 16);
}

// Statistics of the linear solves of one hillslope call.
struct SolveStats
{
    int solves = 0, net_apps = 0, rejected = 0, fallback_its = 0;
    double explicit_max = 0.0;
};

// Reductions of one linear solve: a header of 16 doubles, then kSlot
// doubles per iteration.
constexpr int kSlot = 4;
inline std::size_t solve_acc_doubles(int max_iter) { return 16 + static_cast<std::size_t>(kSlot) * (max_iter + 2); }

// One evaluation of alpha, F and the norms at z (device), read back.
cudaError_t hsn_evaluate(const HsN& P, const std::uint8_t* mask, HsnBuf& B, const double* z, std::int64_t n,
                         cudaStream_t st, double out[3])
{
    cudaMemsetAsync(B.acc, 0, sizeof(double) * 3, st);
    hsn_eval<<<grid_blocks(n, 256), 256, 0, st>>>(P, mask, B.dof, z, B.zn, B.alpha, B.F, B.acc);
    cudaMemcpyAsync(B.hacc, B.acc, sizeof(double) * 3, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    out[0] = B.hacc[0];
    out[1] = B.hacc[1];
    out[2] = B.hacc[2];
    return e;
}

// Jacobi-PCG iterations from the state (x, r, p) with r.z in *rz0 until
// ||r||_2 <= rel_tol * bnorm or max_iter. With snap_at (ascending), x and r
// after iteration snap_at[j] are copied to x_snap + j*n and r_snap + j*n.
cudaError_t jacobi_loop(const HsN& P, const std::uint8_t* mask, HsnBuf& B, std::int64_t n, double bnorm,
                        double rel_tol, int max_iter, cudaStream_t st, double* slots, const double* rz0, int* iters,
                        double* rel, const std::vector<int>* snap_at = nullptr, float* x_snap = nullptr,
                        float* r_snap = nullptr, bool check = true)
{
    const float inv_dt = static_cast<float>(P.H.inv_dt), DA = static_cast<float>(P.H.DA);
    float* pbuf[2] = {B.p, B.p2};
    const HsParts parts = hs_parts(P.H.nr, P.H.nc);
    double* part_ap = B.part + parts.ap;
    double* part_up = B.part + parts.up;
    const bool tall = strip_long(P.H.nr, P.H.nc);
    const unsigned nt = strip_blocks(P.H.nr, P.H.nc, tall ? 16 : 8);
    const unsigned ub = static_cast<unsigned>(std::min<std::int64_t>(kHsUpdBlocks, (n + 1023) / 1024));
    cudaMemsetAsync(B.loop, 0, sizeof(HsnLoop), st);
    auto apply = [&](const float* src, float* dst, const double* rz, double* pap, bool fuse) {
#define LSDTT_APPLY(F, TR)                                                                                            \
    hsn_apply_t<F, TR><<<nt, 256, 0, st>>>(P, inv_dt, DA, mask, B.dof, B.alpha, B.scal, B.zz, src, dst, B.Ap, part_ap, \
                                           B.loop, rz, pap)
        if (tall && fuse) LSDTT_APPLY(true, 16);
        else if (tall) LSDTT_APPLY(false, 16);
        else if (fuse) LSDTT_APPLY(true, 8);
        else LSDTT_APPLY(false, 8);
#undef LSDTT_APPLY
    };
    int it = 0, step = 4;
    std::size_t next_snap = 0;
    HsnLoop H{};
    cudaError_t e = cudaSuccess;
    while (it < max_iter)
    {
        const int batch = std::min(step, max_iter - it);
        for (int k = 0; k < batch; ++k, ++it)
        {
            double* cur = slots + kSlot * it;
            const double* rz_prev = (it == 0) ? rz0 : slots + kSlot * (it - 1) + 1;
            // the direction p = z + beta p of the previous iteration is
            // formed inside the apply (the first iteration's p is given)
            float* p = pbuf[it & 1];
            LSDTT_TIMED("hillslope_apply", 8.0 * static_cast<double>(n), st,
                        (apply(it == 0 ? p : pbuf[(it - 1) & 1], p, rz_prev, cur, it > 0)));
            hs_update_g<<<ub, 256, 0, st>>>(n, B.scal, B.invd, p, B.Ap, B.x, B.r, B.zz, part_up, B.loop, rz_prev,
                                            cur + 1, bnorm, check ? rel_tol : -1.0, max_iter);
            while (snap_at && next_snap < snap_at->size() && (*snap_at)[next_snap] == it)
            {
                cudaMemcpyAsync(x_snap + next_snap * n, B.x, sizeof(float) * n, cudaMemcpyDeviceToDevice, st);
                cudaMemcpyAsync(r_snap + next_snap * n, B.r, sizeof(float) * n, cudaMemcpyDeviceToDevice, st);
                ++next_snap;
            }
        }
        if (!check) continue;
        // (a batch launched past convergence returns at once)
        cudaMemcpyAsync(&H, B.loop, sizeof(H), cudaMemcpyDeviceToHost, st);
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        *rel = H.rel;
        if (H.done) break;
        step = std::min(16, step + 4);
    }
    *iters = check ? H.iters : it;
    return cudaGetLastError();
}

// ||b - A x||_2 and the FP32 representation floor, both relative to bnorm;
// leaves the explicit residual in B.r.
cudaError_t explicit_residual(const HsN& P, const std::uint8_t* mask, HsnBuf& B, std::int64_t n, double bnorm,
                              double* acc2, cudaStream_t st, double* rel_exp, double* rel_floor)
{
    cudaMemsetAsync(acc2, 0, sizeof(double) * 2, st);
    hsn_explicit<<<grid_blocks(n, 256), 256, 0, st>>>(P, mask, B.dof, B.alpha, B.b, B.x, B.r, acc2);
    cudaMemcpyAsync(B.hacc, acc2, sizeof(double) * 2, cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    *rel_exp = std::sqrt(B.hacc[0]) / bnorm;
    *rel_floor = std::sqrt(B.hacc[1]) / bnorm;
    return e;
}

// The acceptance check's tolerance on the explicit residual: the requested relative
// residual, or 4x the floor that rounding the iterate to FP32 leaves,
// whichever is larger.
constexpr double kAcceptFloor = 4.0;

// Solve A(alpha) dz = -F to rel_tol: Jacobi-PCG, or flexible PCG with the
// network when net is given (then checked, and finished by Jacobi-PCG when
// rejected). Sets *iters (all PCG iterations) and *rel (final recurrence
// residual).
cudaError_t hsn_pcg(const HsN& P, const std::uint8_t* mask, HsnBuf& B, std::int64_t n, double rel_tol, int max_iter,
                    cudaStream_t st, int* iters, double* rel, double* acc, lsdtt_gpu_unet* net, SolveStats& S)
{
    // After two rejected learned solves the rest of the call is plain Jacobi-PCG.
    constexpr int kMaxRejected = 2;
    if (S.rejected >= kMaxRejected) net = nullptr;
    const unsigned nb = grid_blocks(n, 256);
    cudaMemsetAsync(acc, 0, sizeof(double) * solve_acc_doubles(max_iter), st);
    hsn_pcg_init<<<nb, 256, 0, st>>>(P, mask, B.dof, B.alpha, B.F, B.invd, B.b, B.x, B.r, B.p, acc);
    cudaMemcpyAsync(B.hacc, acc, sizeof(double) * 2, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    const double bnorm = std::sqrt(B.hacc[1]);
    *rel = 0.0;
    *iters = 0;
    ++S.solves;
    if (bnorm == 0.0) return cudaSuccess;
    double* slots = acc + 16;
    double rel_exp = 0.0, rel_floor = 0.0;
    if (!net)
    {
        e = jacobi_loop(P, mask, B, n, bnorm, rel_tol, max_iter, st, slots, acc, iters, rel);
        if (e == cudaSuccess) e = explicit_residual(P, mask, B, n, bnorm, acc + 4, st, &rel_exp, &rel_floor);
        if (e == cudaSuccess) S.explicit_max = std::max(S.explicit_max, rel_exp);
        return e;
    }
    // Flexible PCG. Initial slot acc[8..11]; iteration slots from acc + 16.
    const int H = P.H.nr, W = P.H.nc;
    const int tiles = hs_tiles(H, W);
    const float inv_dt = static_cast<float>(P.H.inv_dt), DA = static_cast<float>(P.H.DA);
    float* pbuf[2] = {B.p, B.p2};
    const HsParts parts = hs_parts(H, W);
    double* part_ap = B.part + parts.ap;
    double* part_rz = B.part + parts.rz;
    double* part_roz = B.part + parts.roz;
    const unsigned nt = strip_blocks(H, W, 8);
    double* part_rr = B.part + parts.up;
    // z = y + D^-1 (r - A y), y = the network applied to q = D^-1 r (in zz),
    // masked to the DOFs; partials of r.z and z.(r - r_old)
    auto precondition = [&]() -> cudaError_t {
        const float* ynet = nullptr;
        cudaError_t pe = unet_forward_dev(net, B.zz, H, W, st, &ynet);
        ++S.net_apps;
        hsf_smooth_t<<<tiles, 256, 0, st>>>(P, inv_dt, DA, mask, B.dof, B.alpha, ynet, B.invd, B.r, B.ro, B.zz,
                                            part_rz, part_roz);
        return pe;
    };
    cudaMemsetAsync(B.loop, 0, sizeof(HsnLoop), st);
    cudaMemcpyAsync(B.ro, B.r, sizeof(float) * n, cudaMemcpyDeviceToDevice, st);
    hsf_input<<<nb, 256, 0, st>>>(n, B.invd, B.r, B.zz);
    e = precondition();
    hs_reduce<<<1, 512, 0, st>>>(HsRed{{nullptr, part_rz, nullptr, part_roz}, {0, tiles, 0, tiles},
                                       {nullptr, acc + 9, nullptr, acc + 11}, nullptr, nullptr, nullptr});
    cudaMemcpyAsync(B.p, B.zz, sizeof(float) * n, cudaMemcpyDeviceToDevice, st);
    int it = 0;
    bool converged = false, broke = false;
    const int kCheck = 4;
    const int kStall = 16;  // iterations over which the residual must at least halve
    std::vector<double> hist;
    while (e == cudaSuccess && !converged && !broke && it < max_iter)
    {
        const int batch = std::min(kCheck, max_iter - it);
        for (int k = 0; k < batch && e == cudaSuccess; ++k, ++it)
        {
            double* cur = slots + kSlot * it;
            const double* rz_prev = (it == 0) ? acc + 9 : slots + kSlot * (it - 1) + 1;
            // p = z + beta p of the previous iteration inside the apply
            float* p = pbuf[it & 1];
            // (with p.Ap and alpha = rz_prev / p.Ap)
            if (it == 0)
                LSDTT_TIMED("hillslope_apply", 8.0 * static_cast<double>(n), st,
                            (hsn_apply_t<false, 8><<<nt, 256, 0, st>>>(P, inv_dt, DA, mask, B.dof, B.alpha,
                                                                              B.scal, B.zz, p, p, B.Ap, part_ap, B.loop,
                                                                              rz_prev, cur)));
            else
                LSDTT_TIMED("hillslope_apply", 8.0 * static_cast<double>(n), st,
                            (hsn_apply_t<true, 8><<<nt, 256, 0, st>>>(P, inv_dt, DA, mask, B.dof, B.alpha, B.scal,
                                                                             B.zz, pbuf[(it - 1) & 1], p, B.Ap, part_ap,
                                                                             B.loop, rz_prev, cur)));
            hsf_update_g<<<kHsUpdBlocks, 256, 0, st>>>(n, B.scal, B.invd, p, B.Ap, B.x, B.r, B.ro, B.zz, part_rr);
            e = precondition();
            // r.z, r.r, z.(r - r_old); beta = z.(r - r_old) / rz_prev (Polak-Ribiere)
            hs_reduce<<<1, 512, 0, st>>>(HsRed{{nullptr, part_rz, part_rr, part_roz}, {0, tiles, kHsUpdBlocks, tiles},
                                               {nullptr, cur + 1, cur + 2, cur + 3}, cur + 3, rz_prev, B.scal + 1});
        }
        if (e != cudaSuccess) break;
        cudaMemcpyAsync(B.hacc, slots + kSlot * (it - 1), sizeof(double) * 4, cudaMemcpyDeviceToHost, st);
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) break;
        *rel = std::sqrt(B.hacc[2]) / bnorm;
        if (!std::isfinite(*rel) || !(B.hacc[0] > 0.0) || !(B.hacc[1] > 0.0)) broke = true;
        converged = !broke && *rel <= rel_tol;
        hist.push_back(*rel);
        const std::size_t back = kStall / kCheck;
        if (!converged && hist.size() > back && *rel > 0.5 * hist[hist.size() - 1 - back]) broke = true;
    }
    if (e != cudaSuccess) return e;
    *iters = it;
    // The acceptance check: explicit FP64 residual of the learned iterate.
    e = explicit_residual(P, mask, B, n, bnorm, acc + 4, st, &rel_exp, &rel_floor);
    if (e != cudaSuccess) return e;
    const bool finite = std::isfinite(rel_exp);
    if (converged && finite && rel_exp <= std::max(rel_tol, kAcceptFloor * rel_floor))
    {
        S.explicit_max = std::max(S.explicit_max, rel_exp);
        return cudaSuccess;
    }
    // Rejected: Jacobi-PCG finishes from the learned iterate (from zero if
    // it is not finite), with the explicit residual as its start.
    ++S.rejected;
    if (!finite)
    {
        cudaMemsetAsync(B.x, 0, sizeof(float) * n, st);
        cudaMemcpyAsync(B.r, B.b, sizeof(float) * n, cudaMemcpyDeviceToDevice, st);
    }
    cudaMemsetAsync(acc + 12, 0, sizeof(double), st);
    cudaMemsetAsync(slots, 0, sizeof(double) * kSlot * (max_iter + 1), st);
    hsn_restart<<<nb, 256, 0, st>>>(n, B.invd, B.r, B.p, acc + 12);
    int fit = 0;
    e = jacobi_loop(P, mask, B, n, bnorm, rel_tol, max_iter, st, slots, acc + 12, &fit, rel);
    S.fallback_its += fit;
    *iters += fit;
    if (e == cudaSuccess) e = explicit_residual(P, mask, B, n, bnorm, acc + 4, st, &rel_exp, &rel_floor);
    if (e == cudaSuccess) S.explicit_max = std::max(S.explicit_max, rel_exp);
    return e;
}

}  // namespace
}  // namespace lsdtt_gb300

namespace lsdtt_gb300
{
namespace
{

// Shared body of the plain and learned entry points (net may be null).
int hillslope_implicit_impl(const std::string& who, const lsdtt_gpu_grid* grid, const float* z_dev,
                            const std::uint8_t* mask_dev, const std::uint8_t* is_channel_dev, float D, float Sc,
                            int32_t nonlinear, float dt_total, double rel_tol, int32_t max_pcg_iter,
                            double residual_tol, int32_t max_outer, lsdtt_gpu_unet* net, float* z_out_dev,
                            lsdtt_gpu_solve_report* report, void* stream)
{
    if (!grid || !z_dev || !mask_dev || !z_out_dev) return fail(LSDTT_GPU_EINVAL, who + ": null argument");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        return fail(LSDTT_GPU_ENODEV, who + ": no CUDA device");
    if (!(grid->n_rows > 0 && grid->n_cols > 0 && grid->cell_size > 0.0))
        return fail(LSDTT_GPU_EINVAL, who + ": raster metadata is invalid");
    if (net)
        if (int sc = unet_check_shape(net, grid->n_rows, grid->n_cols)) return sc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const std::int64_t n = static_cast<std::int64_t>(grid->n_rows) * grid->n_cols;
    const unsigned nb = grid_blocks(n, 256);
    HsN P{};
    P.H.nr = grid->n_rows;
    P.H.nc = grid->n_cols;
    const char* bc = grid->boundary_conditions;
    P.H.bn = bc[0]; P.H.be = bc[1]; P.H.bs = bc[2]; P.H.bw = bc[3];
    P.h = grid->cell_size;
    P.H.DA = static_cast<double>(D) / (P.h * P.h);
    P.H.U = 0.0;
    P.Sc2 = static_cast<double>(Sc) * static_cast<double>(Sc);
    P.cap = 0.9999;
    hsn_reciprocals(P);
    P.nonlinear = nonlinear ? 1 : 0;
    const int kPcg = max_pcg_iter > 0 ? max_pcg_iter : 2000;
    const int kOuter = max_outer > 0 ? max_outer : 200;
    const double ftol = residual_tol > 0 ? residual_tol : 1e-12;
    const double rtol = rel_tol > 0 ? rel_tol : 1e-8;
    if (!(dt_total > 0.0f))
    {
        // dt_total <= 0: nothing to integrate (newton_cpu.cpp:700-706).
        cudaMemcpyAsync(z_out_dev, z_dev, sizeof(float) * n, cudaMemcpyDeviceToDevice, st);
        const cudaError_t e0 = cudaStreamSynchronize(st);
        if (report) *report = lsdtt_gpu_solve_report{};
        return e0 == cudaSuccess ? LSDTT_GPU_OK : cuda_fail(e0, who.c_str());
    }
    // Buffers: doubles z, zn, zt, F; float4 alpha; 8 floats; dof; reductions.
    HsnBuf B{};
    const std::size_t need = static_cast<std::size_t>(n) * (4 * 8 + 16 + 8 * 4 + 1) + 64 * 256 +
                             sizeof(double) * (8 + solve_acc_doubles(kPcg)) + hsn_pcg_bytes(P.H.nr, P.H.nc);
    char* base = nullptr;
    cudaError_t e = cudaMallocAsync(&base, need, st);
    if (e == cudaSuccess) e = cudaMallocHost(&B.hacc, sizeof(double) * 8);
    if (e != cudaSuccess)
    {
        if (base) cudaFreeAsync(base, st);
        return cuda_fail(e, who.c_str());
    }
    char* cur = base;
    auto carve = [&](std::size_t bytes) {
        char* p = cur;
        cur += (bytes + 255) & ~std::size_t(255);
        return p;
    };
    B.z = reinterpret_cast<double*>(carve(8 * n));
    B.zn = reinterpret_cast<double*>(carve(8 * n));
    B.zt = reinterpret_cast<double*>(carve(8 * n));
    B.F = reinterpret_cast<double*>(carve(8 * n));
    B.alpha = reinterpret_cast<float4*>(carve(16 * n));
    B.invd = reinterpret_cast<float*>(carve(4 * n));
    B.b = reinterpret_cast<float*>(carve(4 * n));
    B.x = reinterpret_cast<float*>(carve(4 * n));
    B.r = reinterpret_cast<float*>(carve(4 * n));
    B.p = reinterpret_cast<float*>(carve(4 * n));
    B.zz = reinterpret_cast<float*>(carve(4 * n));
    B.Ap = reinterpret_cast<float*>(carve(4 * n));
    B.ro = reinterpret_cast<float*>(carve(4 * n));
    B.dof = reinterpret_cast<std::uint8_t*>(carve(n));
    B.acc = reinterpret_cast<double*>(carve(sizeof(double) * 8));
    double* acc_it = reinterpret_cast<double*>(carve(sizeof(double) * solve_acc_doubles(kPcg)));
    hsn_pcg_carve(B, P.H.nr, P.H.nc, carve);
    SolveStats S;
    {
        hs_dofs<<<nb, 256, 0, st>>>(P.H, mask_dev, is_channel_dev, B.dof);
    }
    hsn_to_double<<<nb, 256, 0, st>>>(n, z_dev, B.z);
    cudaMemcpyAsync(B.zn, B.z, 8 * n, cudaMemcpyDeviceToDevice, st);

    const double total = static_cast<double>(dt_total);
    double dt = total, remaining = total;
    const double dt_min = total * 1e-9;
    int n_sub = 0, rejects = 0, total_outer = 0, total_pcg = 0;
    double last_rel = 0.0, last_finf = 0.0;
    int status = LSDTT_GPU_OK;
    const double feasible = std::sqrt(P.cap);
    while (remaining > 0.0 && status == LSDTT_GPU_OK)
    {
        const double step = std::min(dt, remaining);
        P.H.inv_dt = 1.0 / step;
        // z starts from the previous accepted field (== zn).
        cudaMemcpyAsync(B.z, B.zn, 8 * n, cudaMemcpyDeviceToDevice, st);
        double ev[3];
        e = hsn_evaluate(P, mask_dev, B, B.z, n, st, ev);
        if (e != cudaSuccess) break;
        double fnorm = ev[0];
        bool converged = false;
        int it = 0;
        for (; it < kOuter; ++it)
        {
            if (fnorm <= ftol) { converged = true; break; }
            int pit = 0;
            double rel = 0.0;
            e = hsn_pcg(P, mask_dev, B, n, rtol, kPcg, st, &pit, &rel, acc_it, net, S);
            if (e != cudaSuccess) break;
            total_pcg += pit;
            last_rel = rel;
            // Line search on the true residual (alpha/F buffers are reused:
            // re-evaluate at z before leaving).
            const double ratio_now = P.nonlinear ? ev[2] : 0.0;
            const bool restoring = P.nonlinear && ratio_now > feasible;
            double lambda = 1.0;
            bool accepted = false;
            double evt[3] = {0, 0, 0};
            for (int ls = 0; ls < 30; ++ls)
            {
                hsn_axpy<<<nb, 256, 0, st>>>(n, B.dof, B.z, B.x, lambda, B.zt);
                e = hsn_evaluate(P, mask_dev, B, B.zt, n, st, evt);
                if (e != cudaSuccess) break;
                if (P.nonlinear)
                {
                    if (restoring)
                    {
                        if (evt[2] >= ratio_now) { lambda *= 0.5; continue; }
                        accepted = true;
                        break;
                    }
                    if (evt[2] > feasible) { lambda *= 0.5; continue; }
                }
                if (evt[0] < fnorm) { accepted = true; break; }
                lambda *= 0.5;
            }
            if (e != cudaSuccess) break;
            if (!accepted)
            {
                // restore alpha/F at z for a clean state
                e = hsn_evaluate(P, mask_dev, B, B.z, n, st, ev);
                break;
            }
            std::swap(B.z, B.zt);
            ev[0] = evt[0];
            ev[1] = evt[1];
            ev[2] = evt[2];
            fnorm = ev[0];
            if (fnorm <= ftol) { converged = true; ++it; break; }
        }
        if (e != cudaSuccess) break;
        total_outer += it;
        last_finf = fnorm;
        if (!converged)
        {
            ++rejects;
            if (rejects > 40 || step <= dt_min)
            {
                status = LSDTT_GPU_ENOCONV;
                break;
            }
            dt = std::max(dt_min, step * 0.5);
            continue;
        }
        cudaMemcpyAsync(B.zn, B.z, 8 * n, cudaMemcpyDeviceToDevice, st);
        remaining -= step;
        ++n_sub;
        if (it <= 4) dt = std::min(total, step * 1.7);
        else if (it >= 15) dt = std::max(dt_min, step * 0.5);
    }
    if (e == cudaSuccess)
    {
        hsn_to_float<<<nb, 256, 0, st>>>(n, B.zn, z_out_dev);
        e = cudaStreamSynchronize(st);
    }
    cudaFreeAsync(base, st);
    cudaFreeHost(B.hacc);
    if (e != cudaSuccess) return cuda_fail(e, who.c_str());
    if (report)
    {
        *report = lsdtt_gpu_solve_report{};
        report->iterations = total_pcg;
        report->converged = status == LSDTT_GPU_OK ? 1 : 0;
        report->relative_residual = last_rel;
        report->initial_residual_inf = last_finf;
        report->linear_solves = S.solves;
        report->network_applications = S.net_apps;
        report->rejected_solves = S.rejected;
        report->fallback_iterations = S.fallback_its;
        report->explicit_relative_residual = S.explicit_max;
    }
    if (status != LSDTT_GPU_OK) return fail(status, who + ": Newton failed at the minimum sub-step");
    (void)n_sub;
    (void)total_outer;
    return LSDTT_GPU_OK;
}

}  // namespace
}  // namespace lsdtt_gb300

extern "C" int lsdtt_gpu_hillslope_implicit(const lsdtt_gpu_grid* grid, const float* z_dev, const std::uint8_t* mask_dev,
                                            const std::uint8_t* is_channel_dev, float D, float Sc, int32_t nonlinear,
                                            float dt_total, double rel_tol, int32_t max_pcg_iter, double residual_tol,
                                            int32_t max_outer, float* z_out_dev, lsdtt_gpu_solve_report* report,
                                            void* stream)
{
    return lsdtt_gb300::hillslope_implicit_impl("lsdtt_gpu_hillslope_implicit", grid, z_dev, mask_dev, is_channel_dev,
                                                D, Sc, nonlinear, dt_total, rel_tol, max_pcg_iter, residual_tol,
                                                max_outer, nullptr, z_out_dev, report, stream);
}

extern "C" int lsdtt_gpu_hillslope_implicit_learned(const lsdtt_gpu_grid* grid, const float* z_dev,
                                                    const std::uint8_t* mask_dev, const std::uint8_t* is_channel_dev,
                                                    float D, float Sc, int32_t nonlinear, float dt_total,
                                                    double rel_tol, int32_t max_pcg_iter, double residual_tol,
                                                    int32_t max_outer, lsdtt_gpu_unet* net, float* z_out_dev,
                                                    lsdtt_gpu_solve_report* report, void* stream)
{
    if (!net) return lsdtt_gb300::fail(LSDTT_GPU_EINVAL, "lsdtt_gpu_hillslope_implicit_learned: net is null");
    return lsdtt_gb300::hillslope_implicit_impl("lsdtt_gpu_hillslope_implicit_learned", grid, z_dev, mask_dev,
                                                is_channel_dev, D, Sc, nonlinear, dt_total, rel_tol, max_pcg_iter,
                                                residual_tol, max_outer, net, z_out_dev, report, stream);
}

// Residual/correction pairs from the plain Jacobi-PCG solve of the first
// linear system of a step of length dt (see the header for the layout).
extern "C" int lsdtt_gpu_hillslope_capture_pairs(const lsdtt_gpu_grid* grid, const float* z_dev,
                                                 const std::uint8_t* mask_dev, const std::uint8_t* is_channel_dev,
                                                 float D, float Sc, int32_t nonlinear, float dt, double rel_tol,
                                                 int32_t max_iter, int32_t n_pairs, float* r_out_dev,
                                                 float* e_out_dev, int32_t* n_written, void* stream)
{
    using namespace lsdtt_gb300;
    const char* who = "lsdtt_gpu_hillslope_capture_pairs";
    if (!grid || !z_dev || !mask_dev || !r_out_dev || !e_out_dev || !n_written)
        return fail(LSDTT_GPU_EINVAL, std::string(who) + ": null argument");
    *n_written = 0;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        return fail(LSDTT_GPU_ENODEV, std::string(who) + ": no CUDA device");
    if (!(grid->n_rows > 0 && grid->n_cols > 0 && grid->cell_size > 0.0) || !(dt > 0.0f) || n_pairs <= 0)
        return fail(LSDTT_GPU_EINVAL, std::string(who) + ": invalid grid, dt or pair count");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const std::int64_t n = static_cast<std::int64_t>(grid->n_rows) * grid->n_cols;
    const unsigned nb = grid_blocks(n, 256);
    HsN P{};
    P.H.nr = grid->n_rows;
    P.H.nc = grid->n_cols;
    const char* bc = grid->boundary_conditions;
    P.H.bn = bc[0]; P.H.be = bc[1]; P.H.bs = bc[2]; P.H.bw = bc[3];
    P.h = grid->cell_size;
    P.H.DA = static_cast<double>(D) / (P.h * P.h);
    P.H.U = 0.0;
    P.H.inv_dt = 1.0 / static_cast<double>(dt);
    P.Sc2 = static_cast<double>(Sc) * static_cast<double>(Sc);
    P.cap = 0.9999;
    hsn_reciprocals(P);
    P.nonlinear = nonlinear ? 1 : 0;
    const int kPcg = max_iter > 0 ? max_iter : 2000;
    const double rtol = rel_tol > 0 ? rel_tol : 1e-8;
    HsnBuf B{};
    const std::size_t need = static_cast<std::size_t>(n) * (2 * 8 + 16 + 8 * 4 + 1) + 64 * 256 +
                             sizeof(double) * (8 + solve_acc_doubles(kPcg)) + hsn_pcg_bytes(P.H.nr, P.H.nc);
    char* base = nullptr;
    cudaError_t e = cudaMallocAsync(&base, need, st);
    if (e == cudaSuccess) e = cudaMallocHost(&B.hacc, sizeof(double) * 8);
    if (e != cudaSuccess)
    {
        if (base) cudaFreeAsync(base, st);
        return cuda_fail(e, who);
    }
    char* cur = base;
    auto carve = [&](std::size_t bytes) {
        char* p = cur;
        cur += (bytes + 255) & ~std::size_t(255);
        return p;
    };
    B.z = reinterpret_cast<double*>(carve(8 * n));
    B.F = reinterpret_cast<double*>(carve(8 * n));
    B.zn = B.z;
    B.alpha = reinterpret_cast<float4*>(carve(16 * n));
    B.invd = reinterpret_cast<float*>(carve(4 * n));
    B.b = reinterpret_cast<float*>(carve(4 * n));
    B.x = reinterpret_cast<float*>(carve(4 * n));
    B.r = reinterpret_cast<float*>(carve(4 * n));
    B.p = reinterpret_cast<float*>(carve(4 * n));
    B.zz = reinterpret_cast<float*>(carve(4 * n));
    B.Ap = reinterpret_cast<float*>(carve(4 * n));
    B.ro = reinterpret_cast<float*>(carve(4 * n));
    B.dof = reinterpret_cast<std::uint8_t*>(carve(n));
    B.acc = reinterpret_cast<double*>(carve(sizeof(double) * 8));
    double* acc = reinterpret_cast<double*>(carve(sizeof(double) * solve_acc_doubles(kPcg)));
    hsn_pcg_carve(B, P.H.nr, P.H.nc, carve);
    hs_dofs<<<nb, 256, 0, st>>>(P.H, mask_dev, is_channel_dev, B.dof);
    hsn_to_double<<<nb, 256, 0, st>>>(n, z_dev, B.z);
    double ev[3];
    e = hsn_evaluate(P, mask_dev, B, B.z, n, st, ev);
    int K = 0, written = 0;
    double rel = 0.0;
    auto init = [&]() -> double {
        cudaMemsetAsync(acc, 0, sizeof(double) * solve_acc_doubles(kPcg), st);
        hsn_pcg_init<<<nb, 256, 0, st>>>(P, mask_dev, B.dof, B.alpha, B.F, B.invd, B.b, B.x, B.r, B.p, acc);
        cudaMemcpyAsync(B.hacc, acc, sizeof(double) * 2, cudaMemcpyDeviceToHost, st);
        e = cudaStreamSynchronize(st);
        return std::sqrt(B.hacc[1]);
    };
    if (e == cudaSuccess)
    {
        const double bnorm = init();
        if (e == cudaSuccess && bnorm > 0.0)
            e = jacobi_loop(P, mask_dev, B, n, bnorm, rtol, kPcg, st, acc + 16, acc, &K, &rel);
        if (e == cudaSuccess && bnorm > 0.0 && K > 0)
        {
            // Second, identical solve with snapshots at n_pairs evenly spaced iterations.
            std::vector<int> snaps;
            for (int j = 0; j < n_pairs; ++j)
            {
                const int k = static_cast<int>(static_cast<std::int64_t>(j) * K / n_pairs);
                if (snaps.empty() || k > snaps.back()) snaps.push_back(k);
            }
            init();
            int k2 = 0;
            if (e == cudaSuccess)
                e = jacobi_loop(P, mask_dev, B, n, bnorm, rtol, K, st, acc + 16, acc, &k2, &rel, &snaps, e_out_dev,
                                r_out_dev, false);
            for (std::size_t j = 0; e == cudaSuccess && j < snaps.size(); ++j)
                hsn_pair_finish<<<nb, 256, 0, st>>>(n, B.x, B.invd, r_out_dev + j * n, e_out_dev + j * n);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            written = static_cast<int>(snaps.size());
        }
    }
    cudaFreeAsync(base, st);
    cudaFreeHost(B.hacc);
    if (e != cudaSuccess) return cuda_fail(e, who);
    *n_written = written;
    return LSDTT_GPU_OK;
}
