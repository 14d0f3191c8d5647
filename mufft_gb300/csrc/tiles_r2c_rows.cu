// Second pass of a four-step r2c transform with the fix-up in its stores.
//
// The complex transform Z of the packed reals, M = N1 x N2, leaves this pass as
// Z[k1 + N1*k2], row k1 of the scratch giving the outputs k2.  Bin k of the real
// transform needs Z[k] and Z[M - k] (kernel.c:47-82), and M - k sits in row
// N1 - k1 at position N2 - 1 - k2 (row 0: row 0, position N2 - k2).  So a tile
// takes C / 2 rows and their mirror rows -- row 0 beside row N1 / 2, its own
// mirror -- and after its last stage, where the threads walk across the
// tile's rows, position tl + TL*j of a row (j < R / 2) meets position
// TL - 1 - tl + TL*(R - 1 - j) of its mirror row: every thread leaves its upper
// half in shared memory, reads its mirror's and resolves both bins.
//
// It replaces a row pass with plain stores and an in-place fix-up sweep (16
// bytes read and written per bin): r2c 61 x 2^18 55.7 -> 45.8 us, 64 x 2^16 28.6 ->
// 13.2 (with the tile choices), 100 x 2^19 247 -> 144.  Rows of up to 512 points: from 1024 a 16-row tile fills an SM alone, and narrower ones
// store 32-byte segments.
#include "fft_device.cuh"
#include "tiles_r2c_rows.h"

namespace mgb {

namespace {

template <int L, int R, int C>
__global__ void __launch_bounds__(tile_threads<L, R, C, 1>(), tile_min_blocks<L, R, C, 1>()) r2c_rows(const TileArgs a)
{
    using S = Sched<L, R>;
    constexpr int TL = L / R, NST = S::NST, rl = S::radix(NST - 1), NBL = R / rl, PS = S::PS;
    constexpr int RS = region_stride<L, C, true, PS>();
    static_assert(NST > 1, "a row tile with an exchange");
    extern __shared__ float2 smem[];
    dependent_start();
    const float2 *in = a.in + (long long)blockIdx.y * a.in_batch;
    float2 *out = a.out + (long long)blockIdx.y * a.out_batch;
    const unsigned N1 = a.ntrans;
    auto row_of = [&](int c) -> unsigned {
        const unsigned lo = blockIdx.x * (C / 2) + (c & (C / 2 - 1));
        return c < C / 2 ? lo : (lo == 0 ? N1 / 2 : N1 - lo);
    };
    float2 v[R];
    int c, tl;
    split_tid<ALONG, C, TL>(threadIdx.x, c, tl);
    load_stage0<L, R, 1, ALONG, false, FL_PLAIN>(a, in, nullptr, row_of(c), 0, tl, v);
    stage_compute<L, R, 1, 0>(v, 0, tl, a.tw);
    run_stages<L, R, C, 1, ALONG, ACROSS, 1>(v, 0, c, tl, smem, a.tw);
    // register u*rl + m holds position tl + TL*(u + NBL*m): at(j) in order of position
    auto at = [&](int j) { return v[(j % NBL) * rl + j / NBL]; };
    __syncthreads();  // every thread has read its last stage's inputs
    if (a.l2 & L2_DISCARD_IN) {
        // the tile's rows have been read: their lines leave L2 without write-back
        constexpr int LINES = L / 16;
        for (int idx = threadIdx.x; idx < C * LINES; idx += tile_threads<L, R, C, 1>()) {
            const float2 *line = in + (long long)row_of(idx / LINES) * a.in_dist + 16 * (idx % LINES);
            asm volatile("discard.global.L2 [%0], 128;" ::"l"(line) : "memory");
        }
    }
    float2 *mine = smem + c * RS;
#pragma unroll
    for (int j = R / 2; j < R; j++)
        mine[padpos<PS>(tl + TL * j)] = at(j);
    __syncthreads();
    const unsigned k1 = row_of(c);
    const bool self = k1 == 0 || k1 == N1 / 2;
    const float2 *theirs = smem + (self ? c : c ^ (C / 2)) * RS;
    const long long M = (long long)N1 * L, step = (long long)N1 * TL;
    const bool full = a.epilogue == EPI_R2C_FULL;
    const unsigned long long pol = (a.l2 & L2_STORE_FIRST) ? l2_evict_first() : l2_evict_normal();
    const long long kb = k1 + (long long)N1 * tl;
    float2 *lo = out + kb, *hi = out + (M - kb);
    const float2 *w = a.rtw + kb;
    const int mtop = k1 == 0 ? L - tl : L - 1 - tl;  // mirror of position tl
#pragma unroll
    for (int j = 0; j < R / 2; j++) {
        const float2 zk = at(j);
        if (k1 == 0 && tl == 0 && j == 0) {
            st_policy(out, make_float2(zk.x + zk.y, 0.f), pol);
            st_policy(out + M, make_float2(zk.x - zk.y, 0.f), pol);
            const float2 zh = at(R / 2);  // the middle bin pairs with itself
            float2 x, xh;
            r2c_bins(zh, zh, __ldg(a.rtw + M / 2), x, xh);
            st_policy(out + M / 2, x, pol);
            if (full)
                st_policy(out + M / 2 + M, xh, pol);
        } else {
            float2 x, xh;
            r2c_bins(zk, theirs[padpos<PS>(mtop - TL * j)], __ldg(w), x, xh);
            st_policy(lo, x, pol);
            st_policy(hi, cconj(xh), pol);
            if (full) {
                st_policy(lo + M, xh, pol);
                st_policy(hi + M, cconj(x), pol);
            }
        }
        lo += step;
        hi -= step;
        w += step;
    }
}

template <int L, int R, int C> void add(std::vector<R2cRowsKernel> &out)
{
    out.push_back(R2cRowsKernel{L, R, C, (const void *)&r2c_rows<L, R, C>, tile_threads<L, R, C, 1>(),
                                (size_t)C * region_stride<L, C, true, Sched<L, R>::PS>() * sizeof(float2)});
}

}  // namespace

// widest first
void register_tiles_r2c_rows(std::vector<R2cRowsKernel> &out)
{
    add<256, 16, 16>(out);
    add<256, 16, 8>(out);
    add<512, 32, 16>(out);
    add<512, 32, 8>(out);
}

}  // namespace mgb
