// Row passes with transposed stores (second pass of the four-step FFT): loads
// walk along each row, stores walk across neighbouring rows.
#include "tile_table.cuh"

namespace mgb {

void register_tiles_transpose(std::vector<TileKernel> &out)
{
    add_tile<32, 16, 128, 1, ALONG, ACROSS>(out);
    add_tile<64, 16, 64, 1, ALONG, ACROSS>(out);
    add_tile<128, 16, 32, 1, ALONG, ACROSS>(out);
    add_tile<256, 16, 16, 1, ALONG, ACROSS>(out);
    add_tile<256, 16, 32, 1, ALONG, ACROSS>(out);
    add_tile<512, 16, 8, 1, ALONG, ACROSS>(out);
    add_tile<1024, 16, 8, 1, ALONG, ACROSS>(out);
    add_tile<1024, 16, 16, 1, ALONG, ACROSS>(out);
    add_tile<2048, 16, 4, 1, ALONG, ACROSS>(out);
    add_tile<2048, 16, 8, 1, ALONG, ACROSS>(out);
    add_tile<4096, 16, 4, 1, ALONG, ACROSS>(out);       // default: measured fastest for the 4096 x 4096 four-step
    add_tile<4096, 16, 4, 4, ALONG, ACROSS>(out);  // the same tile spread over a 4-CTA cluster
    add_tile<4096, 16, 2, 1, ALONG, ACROSS>(out);
    add_tile<4096, 32, 4, 1, ALONG, ACROSS>(out);
    add_tile<4096, 32, 2, 1, ALONG, ACROSS>(out);
    add_tile<8192, 32, 2, 1, ALONG, ACROSS>(out);
    add_tile<16384, 32, 1, 1, ALONG, ACROSS>(out);
    // further shapes, chosen by size (choose_tile)
    add_tile<256, 16, 8, 1, ALONG, ACROSS>(out);
    add_tile<512, 32, 8, 1, ALONG, ACROSS>(out);
    add_tile<1024, 32, 8, 1, ALONG, ACROSS>(out);
    add_tile<2048, 32, 4, 1, ALONG, ACROSS>(out);
}

}  // namespace mgb
