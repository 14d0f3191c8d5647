// Entry of one tile-FFT instantiation in the kernel table.
#pragma once

#include "fft_device.cuh"
#include "registry.h"

namespace mgb {

// Tile of C transforms of L points, R elements per thread, Q CTAs.
template <int L, int R, int C, int Q, int LMAP, int SMAP> void add_tile(std::vector<TileKernel> &out)
{
    TileKernel k{L, R, C, Q, LMAP, SMAP, (const void *)&tile_fft<L, R, C, Q, LMAP, SMAP>, C * (L / (R * Q)),
                 tile_smem_bytes<L, R, C, Q, LMAP, SMAP>(), tile_has_thi<L, R, C, Q, LMAP, SMAP>(),
                 tile_exchange_bytes<L, R, C, Q, LMAP, SMAP>(), tile_flavours<L, R, C, Q, LMAP, SMAP>()};
    if constexpr (LMAP == ALONG && SMAP == ALONG)
        k.fn_c2r = tile_c2r_rows_fn<L, R, C, Q>();
    out.push_back(k);
}

}  // namespace mgb
