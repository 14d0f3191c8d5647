// Ragged batched fast convolution: many muFFT convolution requests of mixed
// power-of-two sizes in one persistent launch.
//
// A request is the reference's per-block convolution (fft.c:794-809): the
// first block is transformed (zero-padded input allowed), multiplied by the
// already transformed second block (a filter spectrum from
// mufft_execute_conv_input), scaled by 1/N and transformed back.  MONO_MONO
// goes through an N/2-point complex FFT with the r2c/c2r fix-ups,
// STEREO_MONO through an N-point complex FFT (fft.c:585-599).
//
// Every CTA (512 threads) takes the next work item from a global counter.
// The host orders the items (longest requests first) and decides which
// requests are split: a split request of L = L1 x L2 >= 16384 points runs as
// five phases of tasks (F1 column tiles, F2 row tiles, multiply chunks, I1 row
// tiles, I2 column tiles) that any CTA may take, each task waiting (bounded)
// on a per-request counter until the previous phase is complete; phases are
// queued phase-major across requests, so the waits are rarely long, and every
// awaited task was dequeued earlier by a running CTA (no deadlock).  A request
// that is not split runs whole in one CTA:
//   L <= 8192 complex points: one forward tile (r2c fix-up fused into its
//     store for mono) writes the spectrum to the request's scratch, which
//     stays in L2; one inverse tile reads it back with the multiply and the
//     c2r pre-pass fused into its loads.
//   L = 16384 .. 65536: an in-CTA four-step over the request's scratch,
//     L = L1 x L2.  The forward half stops at the transposed spectrum
//     X^T[k1][k2] = X[k1 + L1*k2] (no transpose), the multiply (and for mono
//     the r2c fix-up, product and c2r pre-pass of each bin pair k, L-k) runs
//     on that layout, and the inverse four-step consumes it directly:
//       F1 columns of L1 with W_L^(n2*k1) -> F2 rows of L2 -> multiply ->
//       I1 rows of L2 (inverse) with W_L^(-n2*k1) -> I2 columns of L1 -> output.
#include "../../include/fft.h"
#include "conv_ragged.h"
#include "fft_device.cuh"

namespace mgb {

namespace {

constexpr int kThreads = 512;

template <int L> __host__ __device__ constexpr int single_r() { return L > 8192 ? 32 : 16; }
template <int L> __host__ __device__ constexpr int single_c() { return kThreads * single_r<L>() / L; }

// The two tiles of a whole request (or a group of them: TAB), each compiled
// for its form.
template <int L, int R, int C, bool TAB, int FL, bool COH>
__device__ __forceinline__ void conv_tile(const TileArgs &a, float2 *smem)
{
    tile_body<L, R, C, 1, ALONG, ALONG, COH, false, false, false, TAB, FL>(a, 0, 0, 0, 0, smem);
}

template <int L, int R, int C, bool TAB>
__device__ __forceinline__ void conv_forward(const TileArgs &f, bool mono, float2 *smem)
{
    if (mono && f.half)
        conv_tile<L, R, C, TAB, FL_HALF_R2C, false>(f, smem);
    else if (mono)
        conv_tile<L, R, C, TAB, FL_R2C, false>(f, smem);
    else if (f.half)
        conv_tile<L, R, C, TAB, FL_HALF_PLAIN, false>(f, smem);
    else
        conv_tile<L, R, C, TAB, FL_PLAIN, false>(f, smem);
}

template <int L, int R, int C, bool TAB>
__device__ __forceinline__ void conv_inverse(const TileArgs &b, bool mono, float2 *smem)
{
    if (mono)
        conv_tile<L, R, C, TAB, FL_MUL_C2R_PLAIN, true>(b, smem);
    else
        conv_tile<L, R, C, TAB, FL_MUL_PLAIN, true>(b, smem);
}

// Forward tile into the spectrum scratch, then the fused multiply + inverse
// tile into the output.
template <int L>
__device__ void conv_single(const RaggedReq &q, float2 *smem, const float2 *tw, const float2 *rtw_fwd,
                            const float2 *rtw_inv)
{
    constexpr int C = single_c<L>(), R = single_r<L>();
    const bool mono = q.stereo == 0;
    TileArgs f{};
    f.in = q.in;
    f.out = q.spec;
    f.in_stride = f.out_stride = 1;
    f.in_dist = f.out_dist = L + 1;
    f.ntrans = 1;
    f.half = q.zero_pad;
    f.epilogue = mono ? EPI_R2C : EPI_PLAIN;
    f.tw = tw;
    f.rtw = rtw_fwd;
    f.scale = 1.0f;
    conv_forward<L, R, C, false>(f, mono, smem);
    __syncthreads();  // spectrum complete and visible to the whole CTA

    TileArgs b{};
    b.in = q.spec;
    b.in2 = q.h;
    b.out = q.out;
    b.in_stride = b.out_stride = 1;
    b.in_dist = b.out_dist = L + 1;
    b.ntrans = 1;
    b.prologue = mono ? PRO_MUL_C2R : PRO_MUL;
    b.mirror_len = L;
    b.rtw = rtw_inv;
    b.scale = q.scale;
    b.conj = 3;
    b.tw = tw;
    conv_inverse<L, R, C, false>(b, mono, smem);
    __syncthreads();
}

// A group of n whole requests of one class: the n transforms of one tile pair
// (the tile's C transforms each take one request's buffers from the tables).
template <int L>
__device__ void conv_group(const RaggedReq &q, const float2 *const *tab, unsigned n, float2 *smem, const float2 *tw,
                           const float2 *rtw_fwd, const float2 *rtw_inv)
{
    constexpr int C = single_c<L>(), R = single_r<L>();
    const bool mono = q.stereo == 0;
    const float2 *const *t_in = tab, *const *t_h = tab + n;
    float2 *const *t_out = (float2 *const *)(tab + 2 * n), *const *t_spec = (float2 *const *)(tab + 3 * n);
    TileArgs f{};
    f.in = q.in;
    f.out = q.spec;
    f.in_tab = t_in;
    f.out_tab = t_spec;
    f.in_stride = f.out_stride = 1;
    f.ntrans = n;
    f.half = q.zero_pad;
    f.epilogue = mono ? EPI_R2C : EPI_PLAIN;
    f.tw = tw;
    f.rtw = rtw_fwd;
    f.scale = 1.0f;
    conv_forward<L, R, C, true>(f, mono, smem);
    __syncthreads();  // spectra complete and visible to the whole CTA

    TileArgs b{};
    b.in = q.spec;
    b.in2 = q.h;
    b.out = q.out;
    b.in_tab = (const float2 *const *)t_spec;
    b.in2_tab = t_h;
    b.out_tab = t_out;
    b.in_stride = b.out_stride = 1;
    b.ntrans = n;
    b.prologue = mono ? PRO_MUL_C2R : PRO_MUL;
    b.mirror_len = L;
    b.rtw = rtw_inv;
    b.scale = q.scale;
    b.conj = 3;
    b.tw = tw;
    conv_inverse<L, R, C, true>(b, mono, smem);
    __syncthreads();
}

// Multiply phase of the four-step path on the transposed spectrum, for the
// chunk `chunk` of `nchunks` (pairs k, L-k for mono; elements for stereo).
template <int L1, int L2>
__device__ void conv_multiply(const RaggedReq &q, const float2 *rtw_fwd, const float2 *rtw_inv, unsigned chunk,
                              unsigned nchunks)
{
    constexpr int L = L1 * L2;
    float2 *s = q.spec;
    auto at = [](int k) { return (k % L1) * L2 + k / L1; };  // X[k] lives at X^T[k % L1][k / L1]
    if (q.stereo) {
        const int i0 = (int)((long long)L * chunk / nchunks), i1 = (int)((long long)L * (chunk + 1) / nchunks);
        for (int idx = i0 + threadIdx.x; idx < i1; idx += kThreads) {
            const int k = (idx / L2) + L1 * (idx % L2);
            s[idx] = cscale(cmul(__ldcg(&s[idx]), __ldcg(&q.h[k])), q.scale);
        }
        return;
    }
    // mono: Z (forward complex FFT of the packed reals) -> r2c bins X -> Y = s*X*H
    // -> c2r pre-pass Zi, pair by pair (kernel.c:36-82).
    constexpr int NP = L / 2 + 1;
    const int k0 = (int)((long long)NP * chunk / nchunks), k1 = (int)((long long)NP * (chunk + 1) / nchunks);
    for (int k = k0 + threadIdx.x; k < k1; k += kThreads) {
        if (k == 0) {
            const float2 z0 = __ldcg(&s[0]);
            const float2 x0 = make_float2(z0.x + z0.y, 0.f), xm = make_float2(z0.x - z0.y, 0.f);
            const float2 y0 = cscale(cmul(x0, __ldcg(&q.h[0])), q.scale);
            const float2 ym = cscale(cmul(xm, __ldcg(&q.h[L])), q.scale);
            s[0] = c2r_fixup(y0, ym, __ldg(&rtw_inv[0]));
            continue;
        }
        const int km = L - k;
        const int ik = at(k), im = at(km);
        const float2 zk = __ldcg(&s[ik]), zm = __ldcg(&s[im]);
        float2 xk, xk_hi, xm, xm_hi;
        r2c_bins(zk, zm, __ldg(&rtw_fwd[k]), xk, xk_hi);
        r2c_bins(zm, zk, __ldg(&rtw_fwd[km]), xm, xm_hi);
        const float2 yk = cscale(cmul(xk, __ldcg(&q.h[k])), q.scale);
        const float2 ym = cscale(cmul(xm, __ldcg(&q.h[km])), q.scale);
        s[ik] = c2r_fixup(yk, ym, __ldg(&rtw_inv[k]));
        if (km != k)
            s[im] = c2r_fixup(ym, yk, __ldg(&rtw_inv[km]));
    }
}

template <int L1, int L2> __host__ __device__ constexpr int c1_of() { return kThreads * 16 / L1; }
template <int L1, int L2> __host__ __device__ constexpr int c2_of() { return kThreads * 16 / L2; }

// Tile arguments of the four phases that transform (F1, F2, I1, I2).
template <int L1, int L2>
__device__ TileArgs multi_args(const RaggedReq &q, const float2 *tw, int phase)
{
    constexpr int L = L1 * L2;
    TileArgs a{};
    a.tw = tw;
    a.scale = 1.0f;
    a.tw_scale = 2.0f / (float)L;
    a.tw_mask = L - 1;
    if (phase == 0 || phase == 4) {
        // columns of length L1 (n1), stride L2, twiddle W_L^(k1*n2) on the way in
        a.in = phase == 0 ? q.in : q.spec;
        a.out = phase == 0 ? q.spec : q.out;
        a.in_stride = a.out_stride = L2;
        a.in_dist = a.out_dist = 1;
        a.ntrans = L2;
        a.half = phase == 0 ? q.zero_pad : 0;
        a.epilogue = phase == 0 ? EPI_TWIDDLE : EPI_PLAIN;
        a.conj = phase == 0 ? 0 : 2;  // I2: inverse over k1 of conj(Z), conjugated out
    } else {
        // rows of length L2, in place; I1: inverse over k2 (conj in, forward FFT,
        // W_L^(n2*k1)) -> conj(Z)
        a.in = q.spec;
        a.out = q.spec;
        a.in_stride = a.out_stride = 1;
        a.in_dist = a.out_dist = L2;
        a.ntrans = L1;
        a.conj = phase == 3 ? 1 : 0;
        a.epilogue = phase == 3 ? EPI_TWIDDLE : EPI_PLAIN;
    }
    return a;
}

// Out of line: inside the kernel, beside all the other forms, the 32-element
// tile spilled 1.7 KB a thread; alone it takes its 128 registers without (300
// stereo requests of 16384 without class pipelines 61.5 -> 53.5 us).
__device__ __noinline__ void conv_single_16384(const RaggedReq &q, float2 *smem, const float2 *tw,
                                               const float2 *rtw_fwd, const float2 *rtw_inv)
{
    conv_single<16384>(q, smem, tw, rtw_fwd, rtw_inv);
}

// One phase task of a split request (or, with index < 0, the whole phase).
template <int L1, int L2>
__device__ void multi_phase(const RaggedReq &q, float2 *smem, const float2 *tw, const float2 *rtw_fwd,
                            const float2 *rtw_inv, int phase, int index)
{
    constexpr int C1 = c1_of<L1, L2>(), C2 = c2_of<L1, L2>();
    if (phase == 2) {
        if (index < 0)
            conv_multiply<L1, L2>(q, rtw_fwd, rtw_inv, 0, 1);
        else
            conv_multiply<L1, L2>(q, rtw_fwd, rtw_inv, (unsigned)index, kRaggedMulChunks);
        return;
    }
    const TileArgs a = multi_args<L1, L2>(q, tw, phase);
    if (phase == 0 || phase == 4) {
        const int t0 = index < 0 ? 0 : index, t1 = index < 0 ? L2 / C1 : index + 1;
        for (int t = t0; t < t1; t++) {
            if (phase == 0)
                tile_body<L1, 16, C1, 1, ACROSS, ACROSS, false>(a, t, 0, 0, 0, smem);
            else
                tile_body<L1, 16, C1, 1, ACROSS, ACROSS, true>(a, t, 0, 0, 0, smem);
            __syncthreads();
        }
    } else {
        const int t0 = index < 0 ? 0 : index, t1 = index < 0 ? L1 / C2 : index + 1;
        for (int t = t0; t < t1; t++) {
            tile_body<L2, 16, C2, 1, ALONG, ALONG, true>(a, t, 0, 0, 0, smem);
            __syncthreads();
        }
    }
}

// Whole request through the in-CTA four-step.
template <int L1, int L2>
__device__ void conv_multi(const RaggedReq &q, float2 *smem, const float2 *tw, const float2 *rtw_fwd,
                           const float2 *rtw_inv)
{
    for (int phase = 0; phase < 5; phase++) {
        multi_phase<L1, L2>(q, smem, tw, rtw_fwd, rtw_inv, phase, -1);
        __syncthreads();
    }
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Thread 0 waits (bounded) until *ctr >= target; CTA-uniform result.
__device__ bool wait_tasks(const unsigned *ctr, unsigned target, int *err)
{
    int ok = 1;
    if (threadIdx.x == 0) {
        for (unsigned i = 0; ld_acquire_u32(ctr) < target; i++) {
            if (i > (1u << 24) || *(volatile int *)err) {
                atomicExch(err, 1);
                ok = 0;
                break;
            }
            __nanosleep(128);
        }
    }
    return __syncthreads_and(ok) != 0;
}

}  // namespace

unsigned ragged_phase_tasks(unsigned lg, unsigned phase)
{
    // four-step split L1 x L2 of the in-CTA path: 2^14 = 128 x 128, 2^15 = 128 x 256, 2^16 = 256 x 256
    const unsigned l1 = lg == 16 ? 256 : 128, l2 = lg == 14 ? 128 : 256;
    const unsigned c1 = kThreads * 16 / l1, c2 = kThreads * 16 / l2;
    switch (phase) {
    case 0:
    case 4: return l2 / c1;
    case 1:
    case 3: return l1 / c2;
    default: return kRaggedMulChunks;
    }
}

__global__ void __launch_bounds__(kThreads, 1) conv_ragged_kernel(const RaggedArgs args)
{
    extern __shared__ float2 smem[];
    __shared__ unsigned s_idx;
    for (;;) {
        if (threadIdx.x == 0)
            s_idx = atomicAdd(args.next, 1u);
        __syncthreads();
        const unsigned i = s_idx;
        __syncthreads();
        if (i >= args.count)
            return;
        const RaggedTask task = args.tasks[i];
        const RaggedReq q = args.reqs[task.req];
        const float2 *rf = args.rtw + args.rtw_off[q.lg];
        const float2 *ri = rf + (1u << q.lg);
        if (q.split) {
            if (task.wait && !wait_tasks(&args.counters[q.counter], task.wait, args.err))
                return;
            switch (q.lg) {
            case 14: multi_phase<128, 128>(q, smem, args.tw, rf, ri, task.phase, task.index); break;
            case 15: multi_phase<128, 256>(q, smem, args.tw, rf, ri, task.phase, task.index); break;
            case 16: multi_phase<256, 256>(q, smem, args.tw, rf, ri, task.phase, task.index); break;
            default: break;
            }
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0)
                atomicAdd(&args.counters[q.counter], 1u);
            continue;
        }
        if (task.phase == kRaggedGroupTask) {
            const float2 *const *tab = args.tab + task.pad;
            switch (q.lg) {
            case 4: conv_group<16>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 5: conv_group<32>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 6: conv_group<64>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 7: conv_group<128>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 8: conv_group<256>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 9: conv_group<512>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 10: conv_group<1024>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 11: conv_group<2048>(q, tab, task.index, smem, args.tw, rf, ri); break;
            case 12: conv_group<4096>(q, tab, task.index, smem, args.tw, rf, ri); break;
            default: break;
            }
            continue;
        }
        // whole requests up to 4096 points always come as group tasks (above)
        switch (q.lg) {
        case 13: conv_single<8192>(q, smem, args.tw, rf, ri); break;
        case 14: conv_single_16384(q, smem, args.tw, rf, ri); break;
        case 15: conv_multi<128, 256>(q, smem, args.tw, rf, ri); break;
        case 16: conv_multi<256, 256>(q, smem, args.tw, rf, ri); break;
        default: break;
        }
    }
}

unsigned ragged_group_size(unsigned lg)
{
    switch (lg) {
    case 4: return single_c<16>();
    case 5: return single_c<32>();
    case 6: return single_c<64>();
    case 7: return single_c<128>();
    case 8: return single_c<256>();
    case 9: return single_c<512>();
    case 10: return single_c<1024>();
    case 11: return single_c<2048>();
    case 12: return single_c<4096>();
    default: return 1;
    }
}

template <int L> constexpr size_t single_bytes()
{
    return tile_exchange_bytes<L, single_r<L>(), single_c<L>(), 1, ALONG, ALONG>();
}
template <int L1, int L2> constexpr size_t multi_bytes()
{
    constexpr size_t a = tile_exchange_bytes<L1, 16, kThreads * 16 / L1, 1, ACROSS, ACROSS>();
    constexpr size_t b = tile_exchange_bytes<L2, 16, kThreads * 16 / L2, 1, ALONG, ALONG>();
    return a > b ? a : b;
}

size_t conv_ragged_smem()
{
    // every tile conv_ragged_kernel instantiates
    const size_t v[] = {single_bytes<16>(),   single_bytes<32>(),   single_bytes<64>(),   single_bytes<128>(),
                        single_bytes<256>(),  single_bytes<512>(),  single_bytes<1024>(), single_bytes<2048>(),
                        single_bytes<4096>(), single_bytes<8192>(), single_bytes<16384>(),
                        multi_bytes<128, 128>(), multi_bytes<128, 256>(), multi_bytes<256, 256>()};
    size_t m = 0;
    for (size_t x : v)
        m = x > m ? x : m;
    return m;
}

namespace {

// Column passes of class pipelines (see conv_ragged.h): F1 reads the request's
// input (FL: with the twiddle, zero-padded or whole), I2 (FL_PLAIN) writes its
// output; the spectrum scratch is the other side.
template <int L, int C, int FL>
__global__ void __launch_bounds__(tile_threads<L, 16, C, 1>(), tile_min_blocks<L, 16, C, 1>())
    class_columns(const TileArgs tmpl, const ClassEntry *tab)
{
    extern __shared__ float2 smem[];
    const ClassEntry e = tab[blockIdx.y];
    TileArgs a = tmpl;
    a.in = FL == FL_PLAIN ? e.spec : e.in;
    a.out = FL == FL_PLAIN ? e.out : e.spec;
    tile_body<L, 16, C, 1, ACROSS, ACROSS, false, false, false, false, false, FL>(a, blockIdx.x, 0, 0, 0, smem);
}

// The rows of a class pipeline in one pass over the scratch: forward row
// transforms of C rows (F2), the spectral multiply and the inverse ones with
// the W_L^(n2*k1) twiddle (I1).  Row k1 of the scratch holds X^T[k1][k2] =
// X[k1 + L1*k2]; the forward tile's last stage leaves positions tl + TL*j of a
// row in registers, which is what the inverse tile's first stage wants, so
// the spectrum itself never leaves them.  There the threads walk across the
// tile's rows, so the filter spectrum and the fix-up twiddles, indexed by k =
// k1 + L1*k2, are read along k1.
//   stereo: X[k] * H[k].
//   mono: the packed reals' spectrum Z pairs k with L - k, which sits in row
//     L1 - k1 at column L2 - 1 - k2 (row 0: row 0, L2 - k2): a tile takes C / 2
//     rows and their mirror rows (row 0 beside row L1 / 2, its own mirror), and
//     the threads exchange Z through shared memory once more.  X[k] and X[L-k]
//     come from one fix-up (r2c_bins), then the products, then the c2r one.
// Against three launches (stereo two) with the spectrum through L2 between
// them the 512-request mix takes 66.2 us instead of 86.9, 200 requests of 2^7
// .. 2^15 27.6 instead of 40.2.  Bound by latency: a class is a few hundred CTAs.
template <int L2, int C, bool MONO>
__global__ void __launch_bounds__(256, 3)
    class_rows(const ClassEntry *tab, unsigned L1, float scale, const float2 *tw, const float2 *rtw)
{
    using S = Sched<L2, 16>;
    constexpr int R = 16, TL = L2 / R, NST = S::NST, rl = S::radix(NST - 1), NBL = R / rl, PS = S::PS;
    constexpr int RS = region_stride<L2, C, true, PS>();
    static_assert(TL * C == 256 && NST > 1, "256-thread row tile");
    extern __shared__ float2 smem[];
    float2 *thi = smem + C * RS;
    const ClassEntry e = tab[blockIdx.y];
    const unsigned L = L1 * L2;
    // row of the tile's transform c
    auto row_of = [&](int c) -> unsigned {
        if (!MONO)
            return blockIdx.x * C + c;
        const unsigned lo = blockIdx.x * (C / 2) + (c & (C / 2 - 1));
        return c < C / 2 ? lo : (lo == 0 ? L1 / 2 : L1 - lo);
    };
    float2 v[R];
    int c, tl;
    split_tid<ALONG, C, TL>(threadIdx.x, c, tl);
    const float2 *in = e.spec + (size_t)row_of(c) * L2 + tl;
#pragma unroll
    for (int m = 0; m < R; m++)
        v[m] = ld_data(in + TL * m);
    // the inverse's twiddle while the loads are in flight: W_L^(row * off) for
    // the R output offsets of each row, and this thread's W_L^(row * tl)
    const float tws = 2.0f / (float)L;
    for (int idx = threadIdx.x; idx < C * R; idx += 256) {
        const int i = idx / C;
        thi[idx] = fourstep_twiddle(row_of(idx % C) * (unsigned)(TL * (i / rl) + (i % rl) * (L2 / rl)), tws, L - 1);
    }
    const float2 wbase = fourstep_twiddle(row_of(c) * (unsigned)tl, tws, L - 1);
    stage_compute<L2, R, 1, 0>(v, 0, tl, tw);
    run_stages<L2, R, C, 1, ALONG, ACROSS, 1>(v, 0, c, tl, smem, tw);
    // register u*rl + m holds position tl + TL*(u + NBL*m): in order of position
    float2 z[R];
#pragma unroll
    for (int j = 0; j < R; j++)
        z[j] = v[(j % NBL) * rl + j / NBL];
    const unsigned k1 = row_of(c);
    const float2 *h = e.h + k1 + (size_t)L1 * tl;
    const size_t hstep = (size_t)L1 * TL;
    __syncthreads();  // every thread has read its last stage's inputs
    if constexpr (MONO) {
        float2 *mine = smem + c * RS;
#pragma unroll
        for (int j = 0; j < R; j++)
            mine[padpos<PS>(tl + TL * j)] = z[j];
        __syncthreads();
        const bool self = k1 == 0 || k1 == L1 / 2;
        const float2 *theirs = smem + (self ? c : c ^ (C / 2)) * RS;
        const float2 *w = rtw + k1 + (size_t)L1 * tl;
        const float2 *hm = e.h + (L - k1 - (size_t)L1 * tl);
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int pos = tl + TL * j;
            const int mp = k1 == 0 ? ((L2 - pos) & (L2 - 1)) : L2 - 1 - pos;
            const float2 zm = theirs[padpos<PS>(mp)];
            const float2 wf = __ldg(w + hstep * j);
            float2 xk, xm;
            if (k1 == 0 && pos == 0) {  // X[0] and X[L] from one value
                xk = make_float2(z[j].x + z[j].y, 0.f);
                xm = make_float2(z[j].x - z[j].y, 0.f);
            } else {
                r2c_bins(z[j], zm, wf, xk, xm);
                xm = cconj(xm);
            }
            const float2 yk = cscale(cmul(xk, ld_data(h + hstep * j)), scale);
            const float2 ym = cscale(cmul(xm, ld_data(hm - hstep * j)), scale);
            z[j] = cconj(c2r_fixup(yk, ym, cconj(wf)));  // the c2r twiddle is the r2c one's conjugate
        }
        __syncthreads();  // the slices are free again
    } else {
#pragma unroll
        for (int j = 0; j < R; j++)
            z[j] = cconj(cscale(cmul(z[j], ld_data(h + hstep * j)), scale));
    }
    stage_compute<L2, R, 1, 0>(z, 0, tl, tw);
    run_stages<L2, R, C, 1, ACROSS, ALONG, 1, true>(z, 0, c, tl, smem, tw, wbase);
    float2 *out = e.spec + (size_t)row_of(c) * L2 + tl;
#pragma unroll
    for (int u = 0; u < NBL; u++)
#pragma unroll
        for (int m = 0; m < rl; m++)
            out[TL * u + m * (L2 / rl)] = cmul(z[u * rl + m], thi[(u * rl + m) * C + c]);
}

template <int L2, int C> constexpr size_t class_rows_bytes()
{
    return ((size_t)C * region_stride<L2, C, true, Sched<L2, 16>::PS>() + (size_t)C * 16) * sizeof(float2);
}

template <int L, int C> ClassTile column_tile(int form)
{
    const void *fn = form == 0   ? (const void *)&class_columns<L, C, FL_COLPOW>
                     : form == 1 ? (const void *)&class_columns<L, C, FL_HALF_COLPOW>
                                 : (const void *)&class_columns<L, C, FL_PLAIN>;
    return ClassTile{fn, L, C, tile_threads<L, 16, C, 1>(), tile_smem_bytes<L, 16, C, 1, ACROSS, ACROSS>()};
}

}  // namespace

ClassTile class_column_tile(int L1, bool first, bool zero_pad)
{
    const int form = first ? (zero_pad ? 1 : 0) : 2;
    return L1 == 128 ? column_tile<128, 32>(form) : column_tile<256, 16>(form);
}

ClassTile class_row_tile(int L2, bool mono)
{
    if (L2 == 128)
        return ClassTile{mono ? (const void *)&class_rows<128, 32, true> : (const void *)&class_rows<128, 32, false>, 128,
                         32, 256, class_rows_bytes<128, 32>()};
    return ClassTile{mono ? (const void *)&class_rows<256, 16, true> : (const void *)&class_rows<256, 16, false>, 256, 16,
                     256, class_rows_bytes<256, 16>()};
}

const void *conv_ragged_fn() { return (const void *)&conv_ragged_kernel; }
int conv_ragged_threads() { return kThreads; }

}  // namespace mgb
