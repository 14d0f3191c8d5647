// Table of compiled tile-FFT instantiations, filled by the kernel translation
// units and searched by the planner.
#pragma once

#include <stddef.h>
#include <vector>

namespace mgb {

// A tile kernel compiled for one prologue and epilogue (fft_device.cuh,
// Flavour), named by them.
struct TileFlavours {
    const void *plain = nullptr;   // plain stores
    const void *plain_many = nullptr;  // the same in fewer registers, for launches of many CTAs
    const void *colpow = nullptr;  // four-step twiddle by column powers
    const void *byrow = nullptr;   // four-step twiddle by grid row
    const void *r2c = nullptr;     // r2c fix-up, M + 1 bins
    // zero-padded inputs
    const void *half_plain = nullptr, *half_r2c = nullptr, *half_colpow = nullptr;
    // inputs times a second spectrum, and c2r fix-ups of inputs or such products
    const void *mul_plain = nullptr, *mul_colpow = nullptr, *c2r_colpow = nullptr, *mul_c2r_colpow = nullptr;
};

struct TileKernel {
    int L;          // transform length
    int R;          // elements per thread
    int C;          // transforms per tile
    int Q;          // CTAs per tile (thread-block cluster size)
    int lmap, smap; // thread maps of the load and store phases
    const void *fn;
    int threads;    // per CTA
    size_t smem;    // per CTA
    bool has_thi;   // column pass that takes the four-step twiddle table tw_lo
    size_t smem_ex; // per CTA without the four-step table region (launches with tw_lo == null)
    TileFlavours fl = {};          // fn for one prologue and epilogue each
    const void *fn_c2r = nullptr;  // row tiles: variant staging c2r fix-up rows in shared memory
};

void register_tiles_along_short(std::vector<TileKernel> &out);
void register_tiles_along_mid(std::vector<TileKernel> &out);
void register_tiles_along_long(std::vector<TileKernel> &out);
void register_tiles_across_short(std::vector<TileKernel> &out);
void register_tiles_across_long(std::vector<TileKernel> &out);
void register_tiles_transpose(std::vector<TileKernel> &out);

// Returns the instantiation for (L, lmap, smap): the one matching the
// nonzero of C (transforms per tile), R (elements per thread) and Q (cluster
// size), else the one the options of the plan being built prefer, else the
// first registered.  nullptr if none exists.
const TileKernel *find_tile(int L, int lmap, int smap, int C = 0, int R = 0, int Q = 0);

// The instantiation for a pass of `rows` grid rows of `ntrans` transforms:
// find_tile's where the plan's options prefer one (or ask for a form that
// only some tiles have), else the measured choice for the pass's size.
// real: the one pass of a batch of r2c or c2r transforms (with the fix-up).
const TileKernel *choose_tile(int L, int lmap, int smap, unsigned long long ntrans, unsigned long long rows,
                              bool real = false);

}  // namespace mgb
