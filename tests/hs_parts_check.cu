// Host-only check of the Roering solver's partial-sum layout
// (lsdtt_gb300/csrc/hs_stencil.cuh): for a range of grid sizes, every pass's
// partials (one double a block) lie in a region of their own. Runs no kernel.
#include <cstdio>

#include "hs_stencil.cuh"

using namespace lsdtt_gb300;

int main()
{
    const int sides[] = {1, 2, 3, 7, 8, 9, 15, 16, 17, 29, 30, 31, 32, 33, 60, 61, 64, 97, 127, 128, 129, 150, 256, 257,
                         500, 511, 512, 513, 1000, 1023, 1024, 1025, 1408, 2048, 2051, 4096, 4097, 8192, 16384, 20011};
    long checked = 0;
    for (int nr : sides)
        for (int nc : sides)
        {
            const HsParts p = hs_parts(nr, nc);
            const std::size_t tiles = static_cast<std::size_t>(hs_tiles(nr, nc));
            const std::size_t strips = strip_blocks(nr, nc, strip_long(nr, nc) ? 16 : 8);
            // (the flexible solver runs 8-row strips whatever the grid)
            if (p.ap + strips > p.rz || p.ap + strip_blocks(nr, nc, 8) > p.rz || p.rz + tiles > p.roz ||
                p.roz + tiles > p.up || p.up + 2 * kHsUpdBlocks > p.total)
            {
                std::printf("%d x %d: partials overlap\n", nr, nc);
                return 1;
            }
            ++checked;
        }
    std::printf("%ld sizes OK\n", checked);
    return 0;
}
