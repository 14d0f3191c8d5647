// Column passes: loads and stores walk across neighbouring transforms, so a
// warp touches C consecutive columns of each row it reads or writes.
// Transforms of 1024 and more points.
#include "tile_table.cuh"

namespace mgb {

void register_tiles_across_long(std::vector<TileKernel> &out)
{
    add_tile<1024, 16, 8, 1, ACROSS, ACROSS>(out);
    add_tile<1024, 16, 16, 1, ACROSS, ACROSS>(out);
    add_tile<2048, 16, 4, 1, ACROSS, ACROSS>(out);
    add_tile<2048, 16, 8, 1, ACROSS, ACROSS>(out);
    add_tile<4096, 16, 4, 1, ACROSS, ACROSS>(out);       // default: measured fastest for the 4096 x 4096 four-step
    add_tile<4096, 16, 4, 4, ACROSS, ACROSS>(out);  // the same tile spread over a 4-CTA cluster
    add_tile<4096, 16, 2, 1, ACROSS, ACROSS>(out);
    add_tile<4096, 32, 4, 1, ACROSS, ACROSS>(out);
    add_tile<4096, 32, 2, 1, ACROSS, ACROSS>(out);
    add_tile<8192, 32, 2, 1, ACROSS, ACROSS>(out);
    add_tile<16384, 32, 1, 1, ACROSS, ACROSS>(out);
    add_tile<1024, 32, 8, 1, ACROSS, ACROSS>(out);
    add_tile<2048, 32, 4, 1, ACROSS, ACROSS>(out);
}

}  // namespace mgb
