// Split-precision FFT stages on the 5th-generation tensor cores (tcgen05).
//
// Same mathematics as split_tc.cu (radix-16 Stockham stages of N = 256 / 4096
// as Y = F16 X with BF16 limbs and FP32 accumulation; here three limbs of X
// are cut by truncation, so they represent X exactly), laid out for
// tcgen05.mma: per stage the 256 DFT columns of a CTA's 4096 points form the
// M dimension, so each product is
//   D[j][n] += sum_kk A[j][kk] B[n][kk],   M = 128 columns j, N = 32, K = 32,
// with A = the columns' inputs [Xr(0..15) | Xi(0..15)] (one BF16 limb) and
// B = the real form of F16^T (one limb): B[k][m] = Re F, B[k][16+m] = -Im F,
// B[16+k][m] = Im F, B[16+k][16+m] = Re F.  D (FP32, 32 TMEM columns per
// 128 DFT columns) holds Yr(0..15) | Yi(0..15) of column j in TMEM lane j.
//
// A comes from TMEM as well: row j of A is lane j, two BF16 values to a
// 32-bit column, so the thread of a column writes each limb of it with one
// tcgen05.st of 16 registers -- no operand layout, no shared-memory traffic for
// the 96 bytes of limbs per point pair, and the products read A at TMEM rate.
//
// Per stage: every thread gathers its column, applies the stage twiddle in
// FP32, splits into limbs and stores them to TMEM; each half of the CTA owns
// one M = 128 tile, and one thread of it issues the products x 2 K-halves and
// commits them to an mbarrier; after the wait every thread reads its D row with
// tcgen05.ld.  The first stage gathers straight from the block's input (staged
// by bulk copies, the next block's as soon as this gather is done; or from
// global memory where the copies' alignment does not hold), the last one
// stores straight to the output (outputs k of neighbouring columns are
// neighbours); only the exchanges between stages go through shared memory.
// Persistent CTAs (two per SM) allocate 256 TMEM columns once.  Waits are
// bounded: on timeout the kernel records an error, waits (bounded) for its
// MMAs, frees TMEM, returns.
//
// 16384 x 4096 with three limbs: 457.8 us with the operands in shared memory (and
// the input and output passing through it once more), 352.1 with TMEM operands,
// 337.8 with two exchange buffers (three barriers a block instead of seven), bit
// for bit the same.  Bound by the chain of each stage -- limbs, products,
// read-back -- with two CTAs of eight warps per SM: 45 % of the issue slots, the
// tensor pipe 17 % busy.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>

#include "fft_device.cuh"
#include "split_tc.h"

namespace mgb {

namespace {

constexpr int kUThreads = 256;
// two 128 x 32 FP32 accumulators (64 columns), two 128 x 32 BF16 operands of
// three limbs (48 columns each); allocations are powers of two
constexpr int kTmemCols = 256;
constexpr unsigned kTmemA = 64;

// shared-memory layout (bytes)
constexpr int kInOff = 0;                          // staged input: 4096 points
constexpr int kBOff = kInOff + 4096 * 8;           // [limb] B operands: 3 x 2 KB
constexpr int kXOff = kBOff + 3 * 2048;            // two exchange buffers, 4096 points padded each
constexpr int kXElems = 4096 + 256;                // upad(4095) + 1
constexpr int kTwOff = kXOff + 2 * kXElems * 8;        // 512 stage twiddle factors
constexpr int kBarOff = kTwOff + 512 * 8;          // 3 mbarriers (24 B) + TMEM address (4 B)
constexpr int kUSmem = kBarOff + 64;

__device__ __forceinline__ int upad(int e) { return e + (e >> 4); }

__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor: canonical K-major layout, no swizzle.
__device__ __forceinline__ unsigned long long umma_desc(unsigned saddr)
{
    unsigned long long d = 0;
    d |= (unsigned long long)((saddr >> 4) & 0x3FFFu);
    d |= (unsigned long long)((128u >> 4) & 0x3FFFu) << 16;  // leading: K-adjacent core matrices
    d |= (unsigned long long)((512u >> 4) & 0x3FFFu) << 32;  // stride: 8-row groups
    d |= 1ull << 46;                                          // descriptor version
    return d;                                                 // base offset 0, no swizzle
}

// kind::f16 instruction descriptor: D F32, A and B BF16, both K-major, N = 32, M = 128.
constexpr unsigned kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

// D (TMEM) (+)= A (TMEM) x B (shared memory)
__device__ __forceinline__ void umma(unsigned dtmem, unsigned atmem, unsigned long long bd, unsigned acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(dtmem),
        "r"(atmem), "l"(bd), "r"(kIdesc), "r"(acc)
        : "memory");
}

// One limb of this thread's row of A: 16 registers of two BF16 values.
__device__ __forceinline__ void tmem_st16(unsigned taddr, const unsigned (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void umma_commit(unsigned bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ bool bar_try_wait(unsigned bar, unsigned parity)
{
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded wait for phase `parity` of the mbarrier.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity)
{
    for (unsigned i = 0; i < (1u << 22); i++)
        if (bar_try_wait(bar, parity))
            return true;
    return false;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(unsigned taddr, float (&d)[32])
{
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++)
        d[i] = __uint_as_float(r[i]);
}

// (a, b) as LIMBS bf16x2 pairs by truncation: each limb keeps the top 8
// significant bits of what is left, the residual is exact, and three limbs
// hold an FP32 value exactly (24 bits); two keep 16 bits.  The pair of high
// halves is one byte permute.
// Two limbs round to nearest instead (truncation would bias the 16 bits kept).
template <int LIMBS>
__device__ __forceinline__ void split2(float a, float b, unsigned (&o)[LIMBS])
{
    if constexpr (LIMBS == 3) {
        unsigned ua = __float_as_uint(a), ub = __float_as_uint(b);
#pragma unroll
        for (int l = 0; l < LIMBS; l++) {
            o[l] = __byte_perm(ua, ub, 0x7632);  // high half of a (low), high half of b (high)
            if (l + 1 < LIMBS) {
                ua = __float_as_uint(__uint_as_float(ua) - __uint_as_float(ua & 0xFFFF0000u));
                ub = __float_as_uint(__uint_as_float(ub) - __uint_as_float(ub & 0xFFFF0000u));
            }
        }
    } else {
#pragma unroll
        for (int l = 0; l < LIMBS; l++) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            memcpy(&o[l], &h, 4);
            if (l + 1 < LIMBS) {
                const float2 f = __bfloat1622float2(h);
                a -= f.x;
                b -= f.y;
            }
        }
    }
}

// Bulk copy of `bytes` contiguous bytes into shared memory, completing on `bar`.
__device__ __forceinline__ void bulk_copy(unsigned dst, const void *src, unsigned bytes, unsigned bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Issues the copies of block `blk`'s transforms into the staging area (thread 0).
template <int N, int T>
__device__ __forceinline__ void prefetch_block(const SplitArgs &a, long long blk, unsigned stage, unsigned bar)
{
    const long long tr0 = blk * T;
    const unsigned nt = (unsigned)((a.ntrans - tr0) < T ? (a.ntrans - tr0) : T);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"(nt * (unsigned)(N * sizeof(float2)))
                 : "memory");
    for (unsigned t = 0; t < nt; t++)
        bulk_copy(stage + t * (unsigned)(N * sizeof(float2)), a.in + (tr0 + t) * a.in_dist,
                  (unsigned)(N * sizeof(float2)), bar);
}

template <int S, int LIMBS>
__global__ void __launch_bounds__(kUThreads, 2) split_umma_fft(const SplitArgs a)
{
    constexpr int N = S == 2 ? 256 : 4096;
    constexpr int T = 4096 / N;  // transforms per block of 4096 points
    constexpr int Q = N / 16;    // columns per transform
    constexpr int NT = LIMBS == 3 ? 6 : 3;
    constexpr int ta[6] = {LIMBS == 3 ? 2 : 1, LIMBS == 3 ? 1 : 0, 0, 1, 0, 0};  // F limb
    constexpr int tb[6] = {0, 1, LIMBS == 3 ? 2 : 0, 0, 1, 0};                    // X limb

    extern __shared__ __align__(1024) unsigned char sm[];
    float2 *X = (float2 *)(sm + kXOff);
    float2 *t1 = (float2 *)(sm + kTwOff), *t2 = t1 + 256;
    // mbarriers: [0], [1] MMA completion of tiles 0 and 1, [2] input prefetch
    const unsigned bar0 = smem_u32(sm + kBarOff), bar_in = bar0 + 16;
    unsigned *tmem_slot = (unsigned *)(sm + kBarOff + 24);
    const float2 *stage_in = (const float2 *)(sm + kInOff);
    const int tid = threadIdx.x, warp = tid >> 5, half = tid >> 7;
    const bool bulk = a.bulk != 0;

    // B operands (F limbs, already in core-matrix order) and stage twiddles
    for (int i = tid; i < 3 * 2048 / 16; i += kUThreads)
        ((uint4 *)(sm + kBOff))[i] = __ldg(&((const uint4 *)a.bfrag)[i]);
    for (int i = tid; i < 512; i += kUThreads)
        t1[i] = __ldg(&a.tw[i]);
    if (tid == 0) {
        for (int b = 0; b < 3; b++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0 + 8 * b), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the B operands above are read by the tensor cores (async proxy)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // the tables above are the plan's; what follows reads the caller's input.
    // Before the allocation: a CTA that holds TMEM waits for no other kernel
    dependent_start();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem = *tmem_slot;
    unsigned phase = 0, in_phase = 0;
    // pending: this thread's wait for its tile's products ran out; in_flight:
    // (thread 0) a copy of a block's input is under way
    bool ok = true, in_flight = false, pending = false;

    const long long nblocks = ((long long)a.ntrans + T - 1) / T;
    if (bulk && tid == 0 && (long long)blockIdx.x < nblocks) {
        prefetch_block<N, T>(a, blockIdx.x, smem_u32(stage_in), bar_in);
        in_flight = true;
    }
    for (long long blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x) {
        const long long tr0 = blk * T;
        // this thread's waits so far; all threads' are brought together at the
        // barriers below (a thread whose wait ran out goes on to them)
        bool good = true;
        if (bulk) {
            good = bar_wait(bar_in, in_phase & 1);
            if (good) {
                in_phase++;
                in_flight = false;
            }
        }

#pragma unroll 1
        for (int s = 0; s < S && ok; s++) {
            // the stages scatter into the two exchange buffers in turn, so a
            // scatter never meets the gathers of its own stage
            const float2 *from = X + (s & 1 ? 0 : kXElems);
            float2 *to = X + (s & 1 ? kXElems : 0);
            const int p = 1 << (4 * s);
            // this thread's column: jj = tid (rows of the two M = 128 tiles)
            const int jj = tid, tt = jj / Q, j = jj % Q;
            const bool valid = tr0 + tt < a.ntrans;
            float2 x[16];
            if (s == 0) {
#pragma unroll
                for (int m = 0; m < 16; m++)
                    x[m] = make_float2(0.f, 0.f);
                if (valid && bulk) {
                    const float2 *src = stage_in + tt * N + j;
#pragma unroll
                    for (int m = 0; m < 16; m++)
                        x[m] = src[Q * m];
                } else if (valid) {
                    const float2 *src = a.in + (tr0 + tt) * a.in_dist + j;
#pragma unroll
                    for (int m = 0; m < 16; m++)
                        x[m] = ld_data(src + Q * m);
                }
                if (a.conj) {
#pragma unroll
                    for (int m = 0; m < 16; m++)
                        x[m].y = -x[m].y;
                }
            } else {
#pragma unroll
                for (int m = 0; m < 16; m++) {
                    float2 v = from[upad(tt * N + j + Q * m)];
                    if (s == 1)
                        v = cmul(v, t1[m * 16 + (j & 15)]);
                    else
                        v = cmul(v, cmul(t1[m * 16 + (j >> 4)], t2[m * 16 + (j & 15)]));
                    x[m] = v;
                }
            }
            // A row of this column: registers 0-7 Xr, 8-15 Xi, two values each
            unsigned w[LIMBS][16];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                unsigned o[LIMBS];
                split2<LIMBS>(x[2 * q].x, x[2 * q + 1].x, o);
#pragma unroll
                for (int l = 0; l < LIMBS; l++)
                    w[l][q] = o[l];
                split2<LIMBS>(x[2 * q].y, x[2 * q + 1].y, o);
#pragma unroll
                for (int l = 0; l < LIMBS; l++)
                    w[l][8 + q] = o[l];
            }
            const unsigned lanes = (unsigned)((warp & 3) * 32) << 16;
#pragma unroll
            for (int l = 0; l < LIMBS; l++)
                tmem_st16(tmem + lanes + kTmemA + half * 48 + l * 16, w[l]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            fence_before();
            // each half of the CTA owns one M = 128 tile: its products start as
            // soon as that half has written its operands
            asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
            if ((tid & 127) == 0) {
                fence_after();
#pragma unroll
                for (int q = 0; q < NT; q++)
#pragma unroll
                    for (int kh = 0; kh < 2; kh++) {
                        const unsigned baddr = smem_u32(sm + kBOff + ta[q] * 2048 + kh * 256);
                        umma(tmem + half * 32, tmem + kTmemA + half * 48 + tb[q] * 16 + kh * 8, umma_desc(baddr),
                             (q | kh) ? 1u : 0u);
                    }
                umma_commit(bar0 + 8 * half);
            }
            const bool done = bar_wait(bar0 + 8 * half, phase & 1);
            if (done)
                phase++;
            else
                good = false;
            pending = !done;
            fence_after();
            if (__all_sync(0xFFFFFFFFu, done)) {
                // D row of this thread's column: lane group (warp & 3), tile (warp >> 2)
                float d[32];
                tmem_ld32(tmem + lanes + (warp >> 2) * 32, d);
                fence_before();  // before the next products of this tile (the half's barrier above)
                if (s == S - 1) {
                    // p = Q: output k of column j is j + k*Q
                    if (valid && good) {
                        float2 *dst = a.out + (tr0 + tt) * a.out_dist + j;
                        const float sg = a.conj ? -1.f : 1.f;
#pragma unroll
                        for (int k = 0; k < 16; k++)
                            dst[Q * k] = make_float2(d[k], sg * d[16 + k]);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 16; k++) {
                        const int pos = tt * N + (j / p) * 16 * p + (j & (p - 1)) + k * p;
                        to[upad(pos)] = make_float2(d[k], d[16 + k]);
                    }
                }
            }
            // the scatter is complete, or (last stage) the block is
            ok = __syncthreads_and(good) != 0;
            if (s == 0 && ok && bulk && tid == 0 && blk + gridDim.x < nblocks) {
                // every thread has gathered the staged input
                prefetch_block<N, T>(a, blk + gridDim.x, smem_u32(stage_in), bar_in);
                in_flight = true;
            }
        }
        if (!ok && tid == 0 && a.err)
            atomicExch(a.err, 1);
    }
    if (!ok) {
        // let this CTA's products and copies drain before TMEM is released
        // (bounded): the timed-out phases are still `phase` / `in_phase`, each
        // half's of its own tile
        if ((tid & 127) == 0 && pending)
            bar_wait(bar0 + 8 * half, phase & 1);
        if (tid == 0 && in_flight)
            bar_wait(bar_in, in_phase & 1);
        __syncthreads();
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
    }
}

double bf16r(double v)
{
    float f = (float)v;
    unsigned u;
    std::memcpy(&u, &f, 4);
    u = (u + 0x7FFFu + ((u >> 16) & 1u)) & 0xFFFF0000u;
    std::memcpy(&f, &u, 4);
    return (double)f;
}

}  // namespace

const void *split_umma_kernel(int stages, int limbs)
{
    if (stages == 2)
        return limbs == 3 ? (const void *)&split_umma_fft<2, 3> : (const void *)&split_umma_fft<2, 2>;
    if (stages == 3)
        return limbs == 3 ? (const void *)&split_umma_fft<3, 3> : (const void *)&split_umma_fft<3, 2>;
    return nullptr;
}

size_t split_umma_smem_bytes() { return (size_t)kUSmem; }
int split_umma_threads() { return kUThreads; }

std::vector<unsigned short> split_umma_bfrag_table()
{
    // [limb][core matrix (g = n/8, c = kk/8) at (4g + c) * 128 B][row n % 8][kk % 8], bf16 bits
    std::vector<unsigned short> t(3 * 1024);
    for (int n = 0; n < 32; n++)
        for (int kk = 0; kk < 32; kk++) {
            const int k = n & 15, m = kk & 15;
            const double ph = -2.0 * M_PI * (double)((k * m) % 16) / 16.0;
            const double re = std::cos(ph), im = std::sin(ph);
            double v = (n < 16) ? (kk < 16 ? re : -im) : (kk < 16 ? im : re);
            for (int l = 0; l < 3; l++) {
                const double h = bf16r(v);
                v -= h;
                float f = (float)h;
                unsigned u;
                std::memcpy(&u, &f, 4);
                const int idx = l * 1024 + ((n >> 3) * 4 + (kk >> 3)) * 64 + (n & 7) * 8 + (kk & 7);
                t[idx] = (unsigned short)(u >> 16);
            }
        }
    return t;
}

}  // namespace mgb
