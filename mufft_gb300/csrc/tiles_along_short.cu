// Contiguous batched transforms: loads and stores walk along each transform.
// Transforms of up to 512 points.
#include "tile_table.cuh"

namespace mgb {

void register_tiles_along_short(std::vector<TileKernel> &out)
{
    add_tile<2, 2, 256, 1, ALONG, ALONG>(out);
    add_tile<4, 4, 256, 1, ALONG, ALONG>(out);
    add_tile<8, 8, 256, 1, ALONG, ALONG>(out);
    add_tile<16, 16, 256, 1, ALONG, ALONG>(out);
    add_tile<32, 16, 128, 1, ALONG, ALONG>(out);
    add_tile<64, 16, 64, 1, ALONG, ALONG>(out);
    add_tile<128, 16, 32, 1, ALONG, ALONG>(out);
    add_tile<256, 16, 16, 1, ALONG, ALONG>(out);
    add_tile<512, 16, 8, 1, ALONG, ALONG>(out);
    // further shapes, for the choices by size (choose_tile), the autotuner and
    // explicit tile choices
    add_tile<16, 16, 64, 1, ALONG, ALONG>(out);
    add_tile<32, 16, 64, 1, ALONG, ALONG>(out);
    add_tile<64, 16, 16, 1, ALONG, ALONG>(out);
    add_tile<128, 16, 8, 1, ALONG, ALONG>(out);
    add_tile<256, 16, 4, 1, ALONG, ALONG>(out);
    add_tile<512, 32, 2, 1, ALONG, ALONG>(out);
}

}  // namespace mgb
