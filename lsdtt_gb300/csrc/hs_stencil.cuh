// hs_stencil.cuh -- the hillslope operator's neighbour rules, shared by
// the single-grid solvers (hillslope.cu) and the packed ensemble
// (ensemble.cu). lsdtt_hillslope_domain::neighbour
// (src/cpu/lsdtt_hillslope_operator_cpu.hpp:163-175): 'p' wraps, every other
// edge and every masked neighbour resolves to the cell itself (zero flux).
#pragma once

#include "common.cuh"

namespace lsdtt_gb300
{
namespace
{

struct Hs
{
    int nr, nc;
    char bn, be, bs, bw;
    double DA;      // D / h^2
    double inv_dt;
    double U;
};

__device__ __forceinline__ bool hs_valid(const std::uint8_t* mask, int nc, int r, int c)
{
    return mask[static_cast<std::int64_t>(r) * nc + c] != 0;
}

// lsdtt_hillslope_domain::neighbour (operator_cpu.hpp:163-175)
__device__ __forceinline__ std::int64_t hs_nb(const Hs& H, const std::uint8_t* mask, int r, int c, int dr, int dc)
{
    int rr = r + dr, cc = c + dc;
    if (rr < 0) rr = (H.bn == 'p') ? H.nr - 1 : r;
    else if (rr >= H.nr) rr = (H.bs == 'p') ? 0 : r;
    if (cc < 0) cc = (H.bw == 'p') ? H.nc - 1 : c;
    else if (cc >= H.nc) cc = (H.be == 'p') ? 0 : c;
    if (!hs_valid(mask, H.nc, rr, cc)) { rr = r; cc = c; }
    return static_cast<std::int64_t>(rr) * H.nc + cc;
}

__device__ __forceinline__ bool hs_dirichlet_edge(const Hs& H, int r, int c)
{
    return (r == 0 && H.bn == 'o') || (r == H.nr - 1 && H.bs == 'o') || (c == 0 && H.bw == 'o') ||
           (c == H.nc - 1 && H.be == 'o');
}

// ---- shapes of the single-grid solvers' passes -------------------------------
// Blocks of a strip pass.
inline unsigned strip_blocks(int nr, int nc, int rw)
{
    const std::int64_t g = static_cast<std::int64_t>((nc + 29) / 30) * ((nr + rw - 1) / rw);
    return static_cast<unsigned>((g + 7) / 8);
}
// Rows a warp walks: 16 where that leaves every SM 32 warps (two halo rows in
// 18 loaded, not two in 10), else 8.
inline bool strip_long(int nr, int nc) { return strip_blocks(nr, nc, 16) >= 4 * 152; }

// Tiles of the learned preconditioner's smoothing, and the grid of the
// grid-stride update kernels.
constexpr int kHsTC = 128, kHsTR = 32;
constexpr int kHsUpdBlocks = 152 * 8;

inline int hs_tiles(int nr, int nc) { return ((nc + kHsTC - 1) / kHsTC) * ((nr + kHsTR - 1) / kHsTR); }

// Where the Roering solver's block partials lie (doubles): p.Ap (a strip pass,
// 8 rows at least), r.z and z.(r - r_old) (the smoothing), and the updates' two.
struct HsParts
{
    std::size_t ap, rz, roz, up, total;
};

inline HsParts hs_parts(int nr, int nc)
{
    const std::size_t strips = strip_blocks(nr, nc, 8), tiles = static_cast<std::size_t>(hs_tiles(nr, nc));
    const std::size_t up = strips + 2 * tiles;
    return HsParts{0, strips, strips + tiles, up, up + 2 * kHsUpdBlocks};
}

__device__ constexpr int kDr[4] = {-1, 0, 1, 0};  // N, E, S, W
__device__ constexpr int kDc[4] = {0, 1, 0, -1};

}  // namespace
}  // namespace lsdtt_gb300
