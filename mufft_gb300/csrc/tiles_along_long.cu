// Contiguous batched transforms: loads and stores walk along each transform.
// Transforms of 4096 and more points.
#include "tile_table.cuh"

namespace mgb {

void register_tiles_along_long(std::vector<TileKernel> &out)
{
    add_tile<4096, 16, 1, 1, ALONG, ALONG>(out);
    // 32 elements a thread and radix-32 stages: one exchange fewer than with 16
    // (c2c 2048 x 8192: 62.6 -> 46.7 us, c2r 3001 x 16384 reals 109.5 -> 91.3,
    // r2c 2048 x 16384 reals 70.6 -> 60.7, c2c 1024 x 16384: 78.0 -> 71.1; one
    // transform alone the same)
    add_tile<8192, 32, 1, 1, ALONG, ALONG>(out);
    add_tile<8192, 16, 1, 1, ALONG, ALONG>(out);
    add_tile<8192, 16, 1, 2, ALONG, ALONG>(out);  // clusters: the transform is spread over Q SMs
    add_tile<16384, 32, 1, 1, ALONG, ALONG>(out);
    add_tile<16384, 16, 1, 1, ALONG, ALONG>(out);
    add_tile<16384, 16, 1, 4, ALONG, ALONG>(out);
    add_tile<32768, 16, 1, 8, ALONG, ALONG>(out);
    add_tile<65536, 16, 1, 8, ALONG, ALONG>(out);
}

}  // namespace mgb
