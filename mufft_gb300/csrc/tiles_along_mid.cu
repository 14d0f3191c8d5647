// Contiguous batched transforms: loads and stores walk along each transform.
// Transforms of 1024 to 2048 points.
#include "tile_table.cuh"

namespace mgb {

void register_tiles_along_mid(std::vector<TileKernel> &out)
{
    // one transform per tile from 1024 points: measured faster than several
    // on GB300 for batches of every size (c2c 2048 x 1024: 12.4 -> 10.4 us,
    // c2r 4096 x 16384: 140.2 -> 132.7 us, r2c 4096 x 16: 6.2 -> 4.3 us) and for
    // the row passes of 2D transforms (4096^2 c2r 94.4 -> 91.1 us)
    add_tile<1024, 16, 1, 1, ALONG, ALONG>(out);
    add_tile<2048, 16, 1, 1, ALONG, ALONG>(out);
    add_tile<1024, 32, 1, 1, ALONG, ALONG>(out);
    add_tile<1024, 16, 4, 1, ALONG, ALONG>(out);
    add_tile<1024, 16, 2, 1, ALONG, ALONG>(out);
    add_tile<2048, 16, 2, 1, ALONG, ALONG>(out);
}

}  // namespace mgb
