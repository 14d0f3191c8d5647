// Column passes: loads and stores walk across neighbouring transforms, so a
// warp touches C consecutive columns of each row it reads or writes.
// Transforms of up to 512 points.
#include "tile_table.cuh"

namespace mgb {

void register_tiles_across_short(std::vector<TileKernel> &out)
{
    add_tile<2, 2, 256, 1, ACROSS, ACROSS>(out);
    add_tile<4, 4, 256, 1, ACROSS, ACROSS>(out);
    add_tile<8, 8, 256, 1, ACROSS, ACROSS>(out);
    add_tile<16, 16, 256, 1, ACROSS, ACROSS>(out);
    add_tile<32, 16, 128, 1, ACROSS, ACROSS>(out);
    add_tile<64, 16, 64, 1, ACROSS, ACROSS>(out);
    add_tile<128, 16, 32, 1, ACROSS, ACROSS>(out);
    add_tile<256, 16, 16, 1, ACROSS, ACROSS>(out);
    add_tile<256, 16, 32, 1, ACROSS, ACROSS>(out);
    add_tile<512, 16, 8, 1, ACROSS, ACROSS>(out);
    // further shapes, chosen by size (choose_tile)
    add_tile<64, 16, 32, 1, ACROSS, ACROSS>(out);
    add_tile<128, 16, 16, 1, ACROSS, ACROSS>(out);
    add_tile<256, 16, 8, 1, ACROSS, ACROSS>(out);
    add_tile<512, 32, 16, 1, ACROSS, ACROSS>(out);
    add_tile<512, 32, 8, 1, ACROSS, ACROSS>(out);
}

}  // namespace mgb
