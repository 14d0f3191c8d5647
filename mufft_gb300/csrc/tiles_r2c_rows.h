// Row passes of a four-step that resolve the real transform's bins
// (tiles_r2c_rows.cu).
#pragma once

#include <stddef.h>
#include <vector>

namespace mgb {

struct R2cRowsKernel {
    int L;           // row length (N2)
    int R;           // elements per thread
    int C;           // rows per tile: C / 2 and their mirror rows
    const void *fn;  // kernel(TileArgs a), grid (N1 / C, batch)
    int threads;
    size_t smem;
};

void register_tiles_r2c_rows(std::vector<R2cRowsKernel> &out);

}  // namespace mgb
