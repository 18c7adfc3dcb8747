// fill_tile.cuh -- the epsilon-fill relaxation rules, shared by the
// single-grid fill (fill.cu) and the packed ensemble (ensemble.cu).
// See fill.cu for the algorithm and its relation to the reference's
// priority flood.
#pragma once

#include <cmath>

#include "common.cuh"

namespace lsdtt_gb300
{
namespace
{

constexpr int kT = 32;                                   // tile edge (cells)
constexpr int kH = kT + 2;                               // with halo
constexpr int kMaxLocal = 4 * kT;
constexpr int kFillThreads = 256;                        // threads per tile (32 x 8 block)
constexpr int kFillBlocks = (kT / 2) * (kT / 2) / kFillThreads;  // 2 x 2 blocks per thread

// Tile colours of a fill pass. A pass relaxes its active tiles one colour
// after another, in place; no two tiles of one colour are neighbours
// (including diagonal and periodic ones), so a tile reads every neighbour
// either settled in an earlier colour of this pass or untouched since the
// last pass: the result depends only on the inputs, not on which tiles ran
// first (the discoverer rule is not monotone, so halos read from a field
// that neighbours update meanwhile made it depend on scheduling), and a
// change can still cross several tiles in one pass. Colour = cx + 3 cy with
// cx the parity of the tile column, or 2 for the last column of a periodic
// axis with an odd tile count (it neighbours column 0); cy likewise.
constexpr int kFillColours = 9;

// Bit c set: colour c can hold tiles of an ntx x nty tile grid (host side:
// the passes launch only those colours; four for a grid without wrap).
inline unsigned fill_colour_mask(int ntx, int nty, bool per_ns, bool per_ew)
{
    unsigned mx = 1u | (ntx > 1 ? 2u : 0u) | ((per_ew && (ntx & 1) && ntx > 1) ? 4u : 0u);
    unsigned my = 1u | (nty > 1 ? 2u : 0u) | ((per_ns && (nty & 1) && nty > 1) ? 4u : 0u);
    unsigned m = 0;
    for (int cy = 0; cy < 3; ++cy)
        for (int cx = 0; cx < 3; ++cx)
            if (((mx >> cx) & 1u) && ((my >> cy) & 1u)) m |= 1u << (cx + 3 * cy);
    return m;
}

__host__ __device__ __forceinline__ int fill_colour(int tx, int ty, int ntx, int nty, bool per_ns, bool per_ew)
{
    const int cx = (per_ew && (ntx & 1) && ntx > 1 && tx == ntx - 1) ? 2 : (tx & 1);
    const int cy = (per_ns && (nty & 1) && nty > 1 && ty == nty - 1) ? 2 : (ty & 1);
    return cx + 3 * cy;
}

__device__ __forceinline__ float raise_from(float zeta, float min_slope, float d)
{
    // min_slope <= 0: the neighbour takes the spill value itself (:491-494).
    if (!(min_slope > 0.0f)) return zeta;
    // max(zeta + min_slope*d, nextafter(zeta, +inf)) in float, no contraction
    const float requested = __fadd_rn(zeta, __fmul_rn(min_slope, d));
    const float strict = nextafterf(zeta, INFINITY);
    return fmaxf(requested, strict);
}

// Resolve a neighbour for the fill: periodic wrap on periodic axes only,
// otherwise off-grid = none.
__device__ __forceinline__ bool fill_nb(int nr, int nc, bool per_ns, bool per_ew, int r, int c, int d, int& rr,
                                        int& cc)
{
    rr = r + d8_dr(d);
    cc = c + d8_dc(d);
    if (per_ns) { if (rr < 0) rr += nr; else if (rr >= nr) rr -= nr; }
    if (per_ew) { if (cc < 0) cc += nc; else if (cc >= nc) cc -= nc; }
    return rr >= 0 && rr < nr && cc >= 0 && cc < nc;
}

// Initial state of one cell (row-major index i of an nr x nc grid): seeds
// (and NaN cells) hold z and are fixed, other valid cells +inf, invalid cells hold the nodata
// value (and are never read as neighbours).
__device__ __forceinline__ void fill_init_cell(int nr, int nc, bool per_ns, bool per_ew, const float* __restrict__ z,
                                               const std::uint8_t* __restrict__ mask, double nodata, int interior_nd,
                                               float* __restrict__ F, std::uint8_t* __restrict__ kind, std::int64_t i)
{
    const int r = static_cast<int>(i / nc);
    const int c = static_cast<int>(i - static_cast<std::int64_t>(r) * nc);
    auto valid_at = [&](std::int64_t k) {
        return mask[k] != 0 && !(isnan(nodata) ? isnan(z[k]) : static_cast<double>(z[k]) == nodata);
    };
    if (!valid_at(i))
    {
        F[i] = static_cast<float>(nodata);
        kind[i] = 0;  // invalid
        return;
    }
    bool seed = (!per_ns && (r == 0 || r == nr - 1)) || (!per_ew && (c == 0 || c == nc - 1));
    if (!seed && interior_nd)
        for (int d = 0; d < 8 && !seed; ++d)
        {
            const int rr = r + d8_dr(d), cc = c + d8_dc(d);
            if (rr >= 0 && rr < nr && cc >= 0 && cc < nc && !valid_at(static_cast<std::int64_t>(rr) * nc + cc))
                seed = true;
        }
    // A NaN elevation in a valid cell is kept as it is and never raised;
    // its neighbours' minimum skips it (fminf ignores NaN), so nothing
    // spills through it. (The reference's heap
    // orders a NaN key arbitrarily; its output there is not defined by
    // the algorithm.)
    const bool nan_cell = isnan(z[i]);
    F[i] = (seed || nan_cell) ? z[i] : INFINITY;
    kind[i] = (seed || nan_cell) ? 2 : 1;  // 2 seed or NaN (fixed), 1 free
}

// Does cell i of an nr x nc grid flag interior nodata (an invalid cell off
// the outer ring)?
__device__ __forceinline__ bool fill_interior_invalid(int nr, int nc, const float* __restrict__ z,
                                                      const std::uint8_t* __restrict__ mask, double nodata,
                                                      std::int64_t i)
{
    const int r = static_cast<int>(i / nc), c = static_cast<int>(i % nc);
    if (r < 1 || r >= nr - 1 || c < 1 || c >= nc - 1) return false;
    const bool valid = mask[i] != 0 && !(isnan(nodata) ? isnan(z[i]) : static_cast<double>(z[i]) == nodata);
    return !valid;
}

// One relaxation pass over tile (tx, ty) of an nr x nc grid tiled ntx x nty,
// run by one 32 x 8 thread block (kFillThreads). dirty_in / dirty_out are the grid's
// per-tile activity planes (ntx * nty entries).
__device__ __forceinline__ void fill_relax_tile(int nr, int nc, bool per_ns, bool per_ew, float L, float Ld,
                                                float min_slope, const float* __restrict__ z,
                                                const std::uint8_t* __restrict__ kind, float* __restrict__ F,
                                                int* __restrict__ changed, const std::uint8_t* __restrict__ dirty_in,
                                                std::uint8_t* __restrict__ dirty_out, const int tx, const int ty,
                                                const int ntx, const int nty, const bool gate = true)
{
    // Active-tile gate: a tile can only change if it or one of its eight
    // neighbouring tiles changed in the previous pass (periodic axes wrap).
    // Callers that list the active tiles beforehand skip it (gate = false).
    if (gate)
    {
        bool active = false;
        for (int dy = -1; dy <= 1 && !active; ++dy)
            for (int dx = -1; dx <= 1; ++dx)
            {
                int yy = ty + dy, xx = tx + dx;
                if (per_ns) yy = (yy + nty) % nty;
                if (per_ew) xx = (xx + ntx) % ntx;
                if (yy < 0 || yy >= nty || xx < 0 || xx >= ntx) continue;
                if (dirty_in[yy * ntx + xx]) { active = true; break; }
            }
        if (!active)
        {
            if (threadIdx.x == 0 && threadIdx.y == 0) dirty_out[ty * ntx + tx] = 0;
            return;
        }
    }
    // Staged tile: filled values with +inf at invalid and off-grid cells (so
    // they never win a minimum).
    __shared__ float sF[kH][kH];
    const int r0 = ty * kT - 1, c0 = tx * kT - 1;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    // Each thread owns kFillBlocks 2 x 2 blocks of the tile (block b: local
    // rows 2*(b / (kT/2))+1 .. +2, columns 2*(b % (kT/2))+1 .. +2, b = tid +
    // j * kFillThreads), so it holds kFillBlocks cells of each colour.
    unsigned free_mask = 0;  // bit 4j + k: block j's cell of colour k is free (kind 1)
    for (int k = tid; k < kH * kH; k += blockDim.x * blockDim.y)
    {
        const int lr = k / kH, lcc = k % kH;
        int r = r0 + lr, c = c0 + lcc;
        if (per_ns) { if (r < 0) r += nr; else if (r >= nr) r -= nr; }
        if (per_ew) { if (c < 0) c += nc; else if (c >= nc) c -= nc; }
        float f = INFINITY;
        if (r >= 0 && r < nr && c >= 0 && c < nc)
        {
            const std::int64_t g = static_cast<std::int64_t>(r) * nc + c;
            if (kind[g] != 0) f = F[g];
        }
        sF[lr][lcc] = f;
    }
    // The thread's own cells (its 2 x 2 blocks) live in registers as well:
    // only the owner writes them, so its copies are always the values other
    // threads read from sF. Three of a cell's eight neighbours, its own value
    // and its elevation come from the registers.
    float own[kFillBlocks][4], zown[kFillBlocks][4];
#pragma unroll
    for (int j = 0; j < kFillBlocks; ++j)
    {
        const int b = tid + j * kFillThreads, bx = b % (kT / 2), by = b / (kT / 2);
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const int lr = 2 * by + 1 + (k >> 1), lc = 2 * bx + 1 + (k & 1);
            const int r = r0 + lr, c = c0 + lc;
            zown[j][k] = INFINITY;
            if (r < nr && c < nc)
            {
                const std::int64_t g = static_cast<std::int64_t>(r) * nc + c;
                if (kind[g] == 1)
                {
                    free_mask |= 1u << (4 * j + k);
                    zown[j][k] = z[g];
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kFillBlocks; ++j)
    {
        const int b = tid + j * kFillThreads, bx = b % (kT / 2), by = b / (kT / 2);
#pragma unroll
        for (int k = 0; k < 4; ++k) own[j][k] = sF[2 * by + 1 + (k >> 1)][2 * bx + 1 + (k & 1)];
    }
    // Each local iteration updates the four colours of the 2 x 2 colouring
    // (local row parity, column parity) in turn, a barrier between them:
    // cells of one colour are never neighbours, so every update reads
    // settled values and the result depends only on the tile's inputs (the
    // discoverer rule is not monotone, so in-place updates racing with their
    // neighbours' reads could settle on different values run to run).
    bool tile_changed = false;
    for (int it = 0; it < kMaxLocal; ++it)
    {
        bool local = false;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
#pragma unroll
            for (int j = 0; j < kFillBlocks; ++j)
            {
            const int b = tid + j * kFillThreads, bx = b % (kT / 2), by = b / (kT / 2);
            const int R = 2 * by + 1, C = 2 * bx + 1;  // the block's top-left cell
            const int lr = R + (k >> 1), lc = C + (k & 1);
            if ((free_mask >> (4 * j + k)) & 1u)
            {
                // neighbour (dy, dx): a register when it lies in this block
                // (resolved at compile time: k, dy and dx are constants)
                auto nb = [&](int dy, int dx) -> float {
                    const int yy = (k >> 1) + dy, xx = (k & 1) + dx;
                    if (yy >= 0 && yy <= 1 && xx >= 0 && xx <= 1) return own[j][2 * yy + xx];
                    return sF[R + yy][C + xx];
                };
                const float vN = nb(-1, 0), vNE = nb(-1, 1), vE = nb(0, 1);
                const float vSE = nb(1, 1), vS = nb(1, 0), vSW = nb(1, -1);
                const float vW = nb(0, -1), vNW = nb(-1, -1);
                // lowest neighbour; +inf: none reached yet (or none valid)
                const float cmin = fminf(fminf(vN, vE), fminf(vS, vW));
                const float dmin = fminf(fminf(vNE, vSE), fminf(vSW, vNW));
                const float m = fminf(cmin, dmin);
                if (m < INFINITY)
                {
                    const float zc = zown[j][k];
                    float nv = zc;
                    if (!(zc > m))
                    {
                        // the first neighbour in direction order N, NE, ...,
                        // NW at m decides the step length
                        bool diag = dmin < cmin;
                        if (cmin == dmin)
                            diag = !(vN == m) && ((vNE == m) || (!(vE == m) && ((vSE == m) ||
                                                    (!(vS == m) && ((vSW == m) || (!(vW == m)))))));
                        nv = raise_from(m, min_slope, diag ? Ld : L);
                    }
                    if (nv < own[j][k])
                    {
                        own[j][k] = nv;
                        sF[lr][lc] = nv;
                        local = true;
                    }
                }
            }
            }
            if (k < 3) __syncthreads();
        }
        if (!__syncthreads_or(local)) break;
        tile_changed = true;
    }
#pragma unroll
    for (int j = 0; j < kFillBlocks; ++j)
    {
        const int b = tid + j * kFillThreads, bx = b % (kT / 2), by = b / (kT / 2);
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            if (!((free_mask >> (4 * j + k)) & 1u)) continue;
            const int lr = 2 * by + 1 + (k >> 1), lc = 2 * bx + 1 + (k & 1);
            const std::int64_t g = static_cast<std::int64_t>(r0 + lr) * nc + (c0 + lc);
            if (own[j][k] < F[g]) F[g] = own[j][k];
        }
    }
    if (tid == 0)
    {
        dirty_out[ty * ntx + tx] = tile_changed ? 1 : 0;
        if (tile_changed) atomicOr(changed, 1);
    }
}

// ---- relaxation by line scans -----------------------------------------------
// At raise step 0 a cell's rule F = max(z, lowest neighbour) maps a neighbour's
// value x to min(F, max(z, x)), and such maps compose into one of the same
// form, so a line of 32 cells takes a value from one end to the other in a
// warp scan of five steps where a colour step moves it one cell. A tile
// alternates row and column scans (both ways; the two lines beside each line
// enter first, so diagonals count) until a row pass changes nothing: two
// barriers an alternation, and a handful of alternations where the four-colour
// rounds took tens of four barriers each.
//
// The maps are monotone and start from +inf, so the fixed point (the epsilon-0
// fill, bit for bit) does not depend on the order in which tiles are relaxed.
// (fmaxf and fminf order -0 below +0 and the rule does not: relax_fill takes a
// surface with a -0 through the colours.)
// A pass takes all its tiles in one launch, without colours, and a tile that
// changed cells on its rim queues just the neighbours beyond them for the next
// pass. 4099 x 4000 pitted fractal, wrapped: 24.0 ms in 696 launches, now about
// 10 in 130 to 140.
//
// With a raise step the tile runs the four-colour rounds of fill_relax_tile
// (a cell above its lowest neighbour keeps its elevation, however little: a
// rule without a composed form, and rounding it up to one merged the windows
// of LEM surfaces into a few long ones, 16 times the time of a step), queued
// the same way: 512 x 512 LEM surface 1.43 ms, now 0.64 with the step-0 pass;
// 1500 x 1403 fractal 6.5 ms, now 3.1. Its fixed point then depends on the
// schedule where the discoverer rule is not monotone; it is only the estimate
// that chooses window starts (fill_window.cuh), never a result.
struct ScanTile
{
    float F[kH][kH + 1];
    float Z[kT][kT + 1];
    unsigned rim;
};

// Queue of a relaxation: the lists of this pass and the next, their counts
// (of three, in turn), and a word per tile that is set while it is queued.
struct TileQueue
{
    std::int32_t* list[2];
    unsigned* cnt;     // [3] (and a flag of the caller's)
    unsigned* queued;  // [tiles]
};

__device__ __forceinline__ float scan_line(float f, float zc, float x0, float x1)
{
    const int lane = threadIdx.x & 31;
    float A = f, B = zc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const float pa = __shfl_up_sync(0xffffffffu, A, o), pb = __shfl_up_sync(0xffffffffu, B, o);
        if (lane >= o)
        {
            A = fminf(A, fmaxf(B, pa));
            B = fmaxf(B, pb);
        }
    }
    A = fminf(A, fmaxf(B, x0));
    B = zc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const float pa = __shfl_down_sync(0xffffffffu, A, o), pb = __shfl_down_sync(0xffffffffu, B, o);
        if (lane + o < 32)
        {
            A = fminf(A, fmaxf(B, pa));
            B = fmaxf(B, pb);
        }
    }
    return fminf(A, fmaxf(B, x1));
}

// The tile's row and column scans to its fixed point; false if it ran out of
// rounds.
__device__ __forceinline__ bool scan_rounds(ScanTile& S)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int it = 0;; ++it)
    {
        bool any = false;
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            const int r = w * 4 + q + 1;
            const float f = S.F[r][lane + 1], zc = S.Z[r - 1][lane];
            const float v = fminf(fminf(fminf(S.F[r - 1][lane], S.F[r - 1][lane + 1]),
                                        fminf(S.F[r - 1][lane + 2], S.F[r + 1][lane])),
                                  fminf(S.F[r + 1][lane + 1], S.F[r + 1][lane + 2]));
            const float g = scan_line(fminf(f, fmaxf(zc, v)), zc, S.F[r][0], S.F[r][kT + 1]);
            any |= g < f;
            S.F[r][lane + 1] = g;
        }
        if (!__syncthreads_or(any)) return true;
        if (it == 2 * kT) return false;
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            const int c = w * 4 + q + 1;
            const float f = S.F[lane + 1][c], zc = S.Z[lane][c - 1];
            const float v = fminf(fminf(fminf(S.F[lane][c - 1], S.F[lane + 1][c - 1]),
                                        fminf(S.F[lane + 2][c - 1], S.F[lane][c + 1])),
                                  fminf(S.F[lane + 1][c + 1], S.F[lane + 2][c + 1]));
            S.F[lane + 1][c] = scan_line(fminf(f, fmaxf(zc, v)), zc, S.F[0][c], S.F[kT + 1][c]);
        }
        __syncthreads();
    }
}

// The four-colour rounds of fill_relax_tile on the staged tile (thread: the
// 2 x 2 block at row 2 (tid / 16), column 2 (tid % 16)). A cell that is not
// free has Z = F and never changes.
__device__ __forceinline__ bool colour_rounds(ScanTile& S, unsigned free_mask, float L, float Ld, float eps)
{
    const int R = 2 * (static_cast<int>(threadIdx.x) / (kT / 2)) + 1, C = 2 * (static_cast<int>(threadIdx.x) % (kT / 2)) + 1;
    float own[4], zown[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        own[k] = S.F[R + (k >> 1)][C + (k & 1)];
        zown[k] = S.Z[R - 1 + (k >> 1)][C - 1 + (k & 1)];
    }
    for (int it = 0; it < kMaxLocal; ++it)
    {
        bool local = false;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            if ((free_mask >> k) & 1u)
            {
                auto nb = [&](int dy, int dx) -> float {
                    const int yy = (k >> 1) + dy, xx = (k & 1) + dx;
                    if (yy >= 0 && yy <= 1 && xx >= 0 && xx <= 1) return own[2 * yy + xx];
                    return S.F[R + yy][C + xx];
                };
                const float vN = nb(-1, 0), vNE = nb(-1, 1), vE = nb(0, 1);
                const float vSE = nb(1, 1), vS = nb(1, 0), vSW = nb(1, -1);
                const float vW = nb(0, -1), vNW = nb(-1, -1);
                const float cmin = fminf(fminf(vN, vE), fminf(vS, vW));
                const float dmin = fminf(fminf(vNE, vSE), fminf(vSW, vNW));
                const float m = fminf(cmin, dmin);
                if (m < INFINITY)
                {
                    float nv = zown[k];
                    if (!(nv > m))
                    {
                        bool diag = dmin < cmin;
                        if (cmin == dmin)
                            diag = !(vN == m) && ((vNE == m) || (!(vE == m) && ((vSE == m) ||
                                                    (!(vS == m) && ((vSW == m) || (!(vW == m)))))));
                        nv = raise_from(m, eps, diag ? Ld : L);
                    }
                    if (nv < own[k])
                    {
                        own[k] = nv;
                        S.F[R + (k >> 1)][C + (k & 1)] = nv;
                        local = true;
                    }
                }
            }
            if (k < 3) __syncthreads();
        }
        if (!__syncthreads_or(local)) return true;
    }
    return false;
}

// Relax tile (tx, ty) of an nr x nc grid tiled ntx x nty to its own fixed
// point, by one 256-thread block. `next` and `next_cnt`: the next pass's list.
template <bool kStep>
__device__ __forceinline__ void fill_scan_tile(ScanTile& S, int nr, int nc, bool per_ns, bool per_ew, float L, float Ld,
                                               float eps, const float* __restrict__ z,
                                               const std::uint8_t* __restrict__ kind, float* F, int tx, int ty, int ntx,
                                               int nty, const TileQueue& Q, std::int32_t* __restrict__ next, unsigned* __restrict__ next_cnt)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int r0 = ty * kT - 1, c0 = tx * kT - 1;
    const std::int32_t t = ty * ntx + tx;
    unsigned free_mask = 0;  // (kStep) free cells of the thread's 2 x 2 block
    if (tid == 0)
    {
        // from here on a neighbour that changes queues the tile again
        atomicExch(&Q.queued[t], 0u);
        __threadfence();
        S.rim = 0u;
    }
    __syncthreads();
    for (int k = tid; k < kH * kH; k += 256)
    {
        const int lr = k / kH, lc = k - lr * kH;
        int r = r0 + lr, c = c0 + lc;
        // (a wrapped axis continues one row or column past the grid, in a
        // ragged last tile too; what lies beyond takes no part)
        if (per_ns) r = r < 0 ? r + nr : (r == nr ? 0 : r);
        if (per_ew) c = c < 0 ? c + nc : (c == nc ? 0 : c);
        float f = INFINITY, zc = INFINITY;
        if (r >= 0 && r < nr && c >= 0 && c < nc)
        {
            const std::int64_t g = static_cast<std::int64_t>(r) * nc + c;
            const std::uint8_t kd = kind[g];
            if (kd)
            {
                // (other blocks write F meanwhile: read past the L1)
                f = __ldcg(F + g);
                if (isnan(f)) f = INFINITY;  // a NaN cell is no neighbour
                zc = kd == 1 ? z[g] : f;     // a seed is a constant
            }
        }
        const bool own = lr >= 1 && lr <= kT && lc >= 1 && lc <= kT;
        S.F[lr][lc] = f;
        // a wrapped copy inside a ragged tile is a constant too
        if (own) S.Z[lr - 1][lc - 1] = (r0 + lr < nr && c0 + lc < nc) ? zc : f;
    }
    __syncthreads();
    // the thread's own cells: four rows of a column, or a 2 x 2 block
    auto own_row = [&](int q) { return kStep ? 2 * (tid / (kT / 2)) + 1 + (q >> 1) : w * 4 + q + 1; };
    auto own_col = [&](int q) { return kStep ? 2 * (tid % (kT / 2)) + 1 + (q & 1) : lane + 1; };
    float f0[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) f0[q] = S.F[own_row(q)][own_col(q)];
    bool unsettled;
    if (kStep)
    {
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            const int r = r0 + own_row(q), c = c0 + own_col(q);
            if (r < nr && c < nc && kind[static_cast<std::int64_t>(r) * nc + c] == 1) free_mask |= 1u << q;
        }
        unsettled = !colour_rounds(S, free_mask, L, Ld, eps);
    }
    else
        unsettled = !scan_rounds(S);
    // cells that changed, and the rim they are on: bits N, NE, ..., NW
    const int rb = min(kT, nr - ty * kT), cb = min(kT, nc - tx * kT);  // the tile's own rows and columns
    unsigned rim = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        const int r = own_row(q), c = own_col(q);
        const float f = S.F[r][c];
        if (r > rb || c > cb || !(f < f0[q])) continue;
        F[static_cast<std::int64_t>(r0 + r) * nc + (c0 + c)] = f;
        const bool n = r == 1, s = r == rb, west = c == 1, east = c == cb;
        rim |= (n ? 1u : 0u) | (n && east ? 2u : 0u) | (east ? 4u : 0u) | (s && east ? 8u : 0u) | (s ? 16u : 0u) |
               (s && west ? 32u : 0u) | (west ? 64u : 0u) | (n && west ? 128u : 0u);
    }
    __threadfence();
    rim = __reduce_or_sync(0xffffffffu, rim);
    if (lane == 0 && rim) atomicOr(&S.rim, rim);
    __syncthreads();
    if (tid < 9)
    {
        const unsigned all = S.rim;
        const bool go = tid < 8 ? ((all >> tid) & 1u) != 0 : unsettled;
        int yy = ty, xx = tx;
        if (tid < 8)
        {
            yy += d8_dr(tid);
            xx += d8_dc(tid);
            if (per_ns) yy = yy < 0 ? nty - 1 : (yy >= nty ? 0 : yy);
            if (per_ew) xx = xx < 0 ? ntx - 1 : (xx >= ntx ? 0 : xx);
        }
        if (go && yy >= 0 && yy < nty && xx >= 0 && xx < ntx)
        {
            const std::int32_t u = yy * ntx + xx;
            if (atomicExch(&Q.queued[u], 1u) == 0u) next[atomicAdd(next_cnt, 1u)] = u;
        }
    }
    __syncthreads();  // the arrays are staged again for the next tile
}

}  // namespace
}  // namespace lsdtt_gb300
