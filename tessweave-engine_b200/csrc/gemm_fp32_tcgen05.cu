// 32-bit matrix products of many rows on the 5th-generation tensor cores: out = x @ w.T, all fp32.
//
// A 32-bit number is the sum of three bf16 numbers (8 bits each; the last one rounds at 2^-27 of the number).  Of the nine products
// of two such sums the six that matter are made, x_h w_h, x_h w_m, x_m w_h, x_h w_l, x_l w_h and x_m w_m; what is left out lies
// below 2^-26 of a product.  The tensor cores truncate when they add: a chain of such additions over all of k would err more than
// the FMAs of a plain fp32 product do.  So the leading products are chained over 64 values of k only and these sums are added up
// in registers, by additions that round to nearest; the five small ones may stay in tensor memory until the end.
//
//   * a block computes a tile of 128 rows of x by 128 rows of w.  Sixteen warps read both as they are, 64 values of k at a time and
//     the next 64 under way, cut each number into its terms and leave these in shared memory in the 128-byte swizzle;
//   * one thread issues the MMAs (tcgen05.mma, M = N = 128), 24 for 64 values of k, into one of two accumulators for the leading
//     products and the one for the others;
//   * four warps add the accumulator of the last 64 values to their registers (tcgen05.ld), a row of the tile per thread.
//
// A sum that is not finite is made again as a chain of plain fp32 multiply-adds: an infinite number has no three terms, and a
// finite one above the largest bf16 would give infinities.  The block's cutting warps make the whole tile again then, so that a
// matrix full of NaN takes a few times the product's time and not a thousand times.  Numbers are taken times 2^16 on the
// way in, so that the last bits of the smallest ones do not fall below what a term can hold.
//
// What bounds it is the data port of shared memory and L1: the MMAs' operands take 48 KB of it per 16 values of k, the terms' stores
// and the loads half as much again, and 64 values of k take 3,100 cycles of which the tensor pipe is busy for 1,540.  (N = 256 for x_h
// against two terms of w at once, and eight warps instead of sixteen, change nothing.)  us here and in the library's fp32 product, which
// runs on the FMA units: 1,814 rows by 896 x 1,152 28 and 77, by 896 x 896 28 and 68, by 1,536 x 2,048 84 and 236, by 4,864 x 896 125
// and 324; 777 rows by 896 x 1,152 28 and 42 (caches warm).  A matrix of NaN: 777 rows by 4,864 x 896 0.92 ms, the library 0.20.
// Relative error against 64 bits (2-norms), here and there: k = 896 1.0e-7 and 5.4e-7, k = 1,536 1.2e-7 and 7.0e-7, k = 4,864 1.9e-7 and
// 6.3e-7; numbers spread over 60 powers of two: k = 256 9.4e-8 and 9.0e-8, k = 896 1.1e-7 and 1.6e-7, k = 4,864 1.8e-7 and 1.9e-7, k =
// 8,960 2.4e-7 and 2.1e-7; numbers of 2^-126: 9.0e-8 and 4.1e-7 (not scaled 2.3e-3).  (Halving what grows with k, by a second level of sums
// in tensor memory, costs 2 to 5 % of the time.)
//
// Every wait on an mbarrier is bounded; a wait that runs out sets TW_ERR_WAIT in the status word, every role stops, and the block
// frees its tensor memory and returns.
//
// The reference runs these products through a library (nn.Linear: flow_engine/model.py:39-43,71-73).
#include "tcgen05.cuh"

namespace {

using namespace tc5;

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int CUTTERS = 16, ADDERS = 4, MMA_WARP = CUTTERS + ADDERS, THREADS = 768;     // (three warps of the last group have nothing to do)
// registers by role: 512 x 64 + 128 x 168 + 128 x 56 = 768 x 80, which the block is launched with
constexpr int CUT_REGS = 64, ADD_REGS = 168, MMA_REGS = 56, LAUNCH_REGS = 80;
static_assert(CUTTERS * 32 * CUT_REGS + ADDERS * 32 * ADD_REGS + 128 * MMA_REGS <= THREADS * LAUNCH_REGS, "registers of the block");
constexpr int TERM = 128 * BK * 2;                 // bytes of a term of 128 rows: [128 rows][64 values], swizzled
constexpr int STAGE = 6 * TERM;                    // x: high, middle, low; w: high, middle, low
constexpr int SMEM = 2 * STAGE + 1024;
constexpr int TMEM_COLS = 512, LOW_COL = 256;      // leading sums: columns 0 and 128; the others: 256
constexpr int VALS = 2 * 128 * BK / 4 / (CUTTERS * 32);    // groups of four numbers a thread carries: 8

// Four numbers that nobody on this SM reads again: past L1, whose data port the stores of the terms and the MMAs' operands fill.
__device__ __forceinline__ float4 load_once(const float* p) {
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
// (x, y) less the two bf16 numbers of `h`, as one packed multiply-add
__device__ __forceinline__ float2 less(float2 v, uint32_t h) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\tmov.b64 rc, {%5, %6};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(__uint_as_float(h << 16)), "f"(__uint_as_float(h & 0xffff0000u)), "f"(-1.f), "f"(v.x), "f"(v.y));
    return d;
}
__device__ __forceinline__ uint32_t round2(float2 v) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// (x, y) times 2^UP.  The smallest 32-bit number's last bit, 2^-149, becomes 2^-133 so, the smallest that a bf16 number has; a number
// or a sum that this takes out of range is not finite and made again.  The sums are taken back by 2^-2 UP.
constexpr int UP = 16;
__device__ __forceinline__ float2 scaled(float x, float y) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(x), "f"(y), "f"((float)(1 << UP)));
    return d;
}
__device__ __forceinline__ void split3(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
    float2 v = scaled(x, y);
    a = round2(v);
    v = less(v, a);
    b = round2(v);
    c = round2(less(v, b));
}

// Sums of the tile that are not finite, again, by the cutting warps: every sum of the tile on the FMA units, in one chain over k
// (fmaf(x, w, sum) from zero on), and those that were not finite take the place of what stands in `sums` (see the kernel).
// 128 rows of 32 values of k of x and of w at a time in `area`, transposed; a warp has eight rows, a lane four columns.
constexpr int AGAIN_K = 32, AGAIN_STRIDE = 128 + 4;
static_assert(128 * 512 <= STAGE && 2 * AGAIN_K * AGAIN_STRIDE * 4 <= STAGE && CUTTERS * 8 == 128, "the sums take the first stage, their factors the second");
__device__ __forceinline__ void cutters_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CUTTERS * 32) : "memory"); }
__device__ __forceinline__ unsigned char* sum_place(unsigned char* sums, int row, int col4) {
    return sums + (row >> 5) * (32 * 512) + (row & 31) * 512 + ((col4 ^ (row & 31)) << 4);
}
__device__ __forceinline__ void make_again(unsigned char* sums, float* area, const float* __restrict__ x, int x_stride, const float* __restrict__ w,
                                        int w_stride, int row0, int col0, int M, int N, int K) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* xs = area;
    float* ws = area + AGAIN_K * AGAIN_STRIDE;
    float acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
    for (int k0 = 0; k0 < K; k0 += AGAIN_K) {
        cutters_sync();                                     // nobody reads the values before these any more
        for (int half = 0; half < 2; ++half)
            for (int i = threadIdx.x; i < 128 * (AGAIN_K / 4); i += CUTTERS * 32) {
                const int r = i / (AGAIN_K / 4), q = i % (AGAIN_K / 4) * 4, at = (half ? col0 : row0) + r;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k0 + q < K && at < (half ? N : M))
                    v = *reinterpret_cast<const float4*>((half ? w + (size_t)at * w_stride : x + (size_t)at * x_stride) + k0 + q);
                float* p = (half ? ws : xs) + q * AGAIN_STRIDE + r;
                p[0] = v.x; p[AGAIN_STRIDE] = v.y; p[2 * AGAIN_STRIDE] = v.z; p[3 * AGAIN_STRIDE] = v.w;
            }
        cutters_sync();
        const int most = min(AGAIN_K, K - k0);
        for (int k = 0; k < most; ++k) {
            const float4 xa = *reinterpret_cast<const float4*>(xs + k * AGAIN_STRIDE + warp * 8);
            const float4 xb = *reinterpret_cast<const float4*>(xs + k * AGAIN_STRIDE + warp * 8 + 4);
            const float4 wv = *reinterpret_cast<const float4*>(ws + k * AGAIN_STRIDE + lane * 4);
            const float xr[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w}, wc[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(xr[r], wc[c], acc[r][c]);
        }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        float* p = reinterpret_cast<float*>(sum_place(sums, warp * 8 + r, lane));
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (!isfinite(p[c])) p[c] = acc[r][c];
    }
}
// the sums stand in shared memory: the adding warps say so, the cutting warps wait for it
__device__ __forceinline__ void sums_there() { asm volatile("bar.arrive 2, %0;" ::"n"((CUTTERS + ADDERS) * 32) : "memory"); }
__device__ __forceinline__ void wait_for_sums() { asm volatile("bar.sync 2, %0;" ::"n"((CUTTERS + ADDERS) * 32) : "memory"); }

__global__ void __launch_bounds__(THREADS, 1)
gemm_fp32_kernel(float* __restrict__ out, int out_stride, const float* __restrict__ x, int x_stride, const float* __restrict__ w,
                 int w_stride, int M, int N, int K, int* status) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[2], done[2], read[2], made_again;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_aborted, s_again;
    unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    volatile int* aborted = &s_aborted;
    volatile int* again = &s_again;
    tw_grid_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_m = (M + BM - 1) / BM;
    const int row0 = (int)(blockIdx.x % tiles_m) * BM, col0 = (int)(blockIdx.x / tiles_m) * BN;
    const int num_kb = (K + BK - 1) / BK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(&full[s], CUTTERS); mbar_init(&done[s], 1); mbar_init(&read[s], ADDERS); }
        mbar_init(&made_again, CUTTERS);
        s_aborted = s_again = 0;
        mbar_fence_init();
    }
    if (warp == MMA_WARP) tmem_alloc(&tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp >= MMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MMA_REGS));
        if (warp == MMA_WARP && lane == 0) {
            const uint32_t idesc = instr_desc(BN);
            const uint64_t base = smem_desc(stages, 0);
            bool ok = true;
            for (int kb = 0; ok && kb < num_kb; ++kb) {
                const int s = kb & 1;
                ok = (kb < 2 || mbar_wait(&read[s], ((kb >> 1) - 1) & 1, status)) && mbar_wait(&full[s], (kb >> 1) & 1, status);
                if (!ok) break;
                tc_fence_after();
                const uint64_t a = base + (uint64_t)(s * (STAGE >> 4)), b = a + (uint64_t)(3 * (TERM >> 4));
                constexpr int TA[5] = {0, 2, 1, 0, 1}, TB[5] = {2, 0, 1, 1, 0};
#pragma unroll
                for (int p = 0; p < 5; ++p)
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma_bf16(tmem + LOW_COL, a + (uint64_t)(TA[p] * (TERM >> 4) + 2 * k), b + (uint64_t)(TB[p] * (TERM >> 4) + 2 * k),
                                  idesc, (kb > 0 || p > 0 || k > 0) ? 1u : 0u);
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_bf16(tmem + s * BN, a + (uint64_t)(2 * k), b + (uint64_t)(2 * k), idesc, k > 0 ? 1u : 0u);
                umma_commit(&done[s]);
            }
            if (!ok) *aborted = 1;
        }
        __syncwarp();
    } else if (warp < CUTTERS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CUT_REGS));
        // a thread's numbers: four neighbouring values of k of four rows of x and of four rows of w
        const int quad = threadIdx.x & 15, r0 = threadIdx.x >> 4;
        constexpr int STEP = CUTTERS * 2;                    // rows between two of them
        float4 v[VALS];
        const bool whole = row0 + BM <= M && col0 + BN <= N && (K & (BK - 1)) == 0;
        const float* px = x + (size_t)min(row0 + r0, M - 1) * x_stride + quad * 4;
        const float* pw = w + (size_t)min(col0 + r0, N - 1) * w_stride + quad * 4;
        const size_t step_x = (size_t)STEP * x_stride, step_w = (size_t)STEP * w_stride;
        auto load = [&](int half, int kb) {
            const float* p = (half ? pw : px) + kb * BK;
            if (whole) {
#pragma unroll
                for (int j = 0; j < VALS / 2; ++j) {
                    v[half * (VALS / 2) + j] = load_once(p);
                    p += half ? step_w : step_x;
                }
                return;
            }
            // (a row behind the last one reads this thread's first: nobody looks at its sums; a value of k behind the last is a zero)
            const bool in = kb * BK + quad * 4 < K;
#pragma unroll
            for (int j = 0; j < VALS / 2; ++j) {
                const bool there = (half ? col0 : row0) + r0 + STEP * j < (half ? N : M);
                const float* from = p + (there ? j * (half ? step_w : step_x) : 0);
                v[half * (VALS / 2) + j] = in ? load_once(from) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        bool ok = true;
        load(0, 0);
        load(1, 0);
        for (int kb = 0; kb < num_kb; ++kb) {
            const int s = kb & 1;
            if (kb >= 2) {
                ok = !*aborted && mbar_wait(&done[s], ((kb >> 1) - 1) & 1, status);
                if (!ok) break;
            }
            unsigned char* st = stages + s * STAGE;
            // Half of the numbers at a time, their successors asked for together as soon as they are cut.  (One by one, each wait
            // for a number is a wait for the ones just asked for as well: 100 us where this takes 33.)
#pragma unroll
            for (int j0 = 0; j0 < VALS; j0 += VALS / 2) {
#pragma unroll
                for (int j = j0; j < j0 + VALS / 2; ++j) {
                    const int r = r0 + STEP * (j & (VALS / 2 - 1));
                    uint2 h, m, l;
                    split3(v[j].x, v[j].y, h.x, m.x, l.x);
                    split3(v[j].z, v[j].w, h.y, m.y, l.y);
                    unsigned char* p = st + (j0 ? 3 * TERM : 0) + r * 128 + (((quad >> 1) ^ (r & 7)) << 4) + (quad & 1) * 8;
                    *reinterpret_cast<uint2*>(p) = h;
                    *reinterpret_cast<uint2*>(p + TERM) = m;
                    *reinterpret_cast<uint2*>(p + 2 * TERM) = l;
                }
                asm volatile("" ::: "memory");
                if (kb + 1 < num_kb) load(j0 ? 1 : 0, kb + 1);
                asm volatile("" ::: "memory");
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
        if (!ok) *aborted = 1;
        __syncwarp();
        wait_for_sums();
        if (*again) {
            make_again(stages, reinterpret_cast<float*>(stages + STAGE), x, x_stride, w, w_stride, row0, col0, M, N, K);
            __syncwarp();
            if (lane == 0) mbar_arrive(&made_again);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ADD_REGS));
        // a thread adds up the sums of one row
        const int quarter = warp & 3;
        const uint32_t mine = tmem + ((uint32_t)(quarter * 32) << 16);
        float acc[BN];
#pragma unroll
        for (int e = 0; e < BN; ++e) acc[e] = 0.f;
        auto add = [&](uint32_t at) {
#pragma unroll
            for (int c = 0; c < BN; c += 16) {
                uint32_t t[16];
                tmem_ld16(at + c, t);
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[c + e] += __uint_as_float(t[e]);
            }
        };
        bool ok = true, finite = true;
        for (int kb = 0; kb < num_kb; ++kb) {
            const int s = kb & 1;
            ok = !*aborted && mbar_wait(&done[s], (kb >> 1) & 1, status);
            if (!ok) break;
            tc_fence_after();
            add(mine + s * BN);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&read[s]);
        }
        if (!ok) {
            *aborted = 1;
        } else {
            add(mine + LOW_COL);
#pragma unroll
            for (int e = 0; e < BN; ++e) acc[e] *= 1.f / (1ll << 2 * UP);
#pragma unroll
            for (int e = 0; e < BN; ++e) finite = finite && isfinite(acc[e]);
            if (!finite) *again = 1;                        // (what is behind the last row or column has the numbers of one that is not)
            // through shared memory (every MMA has retired), so that a warp writes whole rows: 32 rows of 128 sums a warp
#pragma unroll
            for (int c = 0; c < BN / 4; ++c)
                *reinterpret_cast<float4*>(sum_place(stages, quarter * 32 + lane, c)) = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
        }
        __syncwarp();
        sums_there();
        if (__any_sync(0xffffffffu, !finite) && !mbar_wait(&made_again, 0, status)) ok = false;
        if (ok) {
            const int gcol = col0 + 4 * lane;
            const bool wide = (N & 3) == 0 && (out_stride & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll 8
            for (int r = 0; r < 32; ++r) {
                const int grow = row0 + quarter * 32 + r;
                const float4 o = *reinterpret_cast<const float4*>(sum_place(stages, quarter * 32 + r, lane));
                if (grow >= M || gcol >= N) continue;
                float* dst = out + (size_t)grow * out_stride + gcol;
                if (wide) {
                    *reinterpret_cast<float4*>(dst) = o;
                } else {
                    const float f[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (gcol + e < N) dst[e] = f[e];
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_dealloc(tmem, TMEM_COLS);
}

}  // namespace

// 1 if the compiler gave the kernel the registers that its roles are split from, 0 if not (the product belongs to the library then), a
// negative number if the driver could not say.
TW_EXPORT int tw_gemm_fp32_built() { return tw_registers_are<gemm_fp32_kernel>(LAUNCH_REGS); }

// out[m, n] = x[m, k] @ w[n, k].T, fp32; rows of x and w on 16-byte boundaries, k a multiple of 4.
TW_EXPORT int tw_gemm_fp32(float* out, int out_stride, const float* x, int x_stride, const float* w, int w_stride, int m, int n, int k,
                           int* status, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0 || (k & 3) || (x_stride & 3) || (w_stride & 3) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15))
        return (int)cudaErrorInvalidValue;
    const long long blocks = ((long long)(m + BM - 1) / BM) * ((n + BN - 1) / BN);
    if (blocks > 0x7fffffffll) return (int)cudaErrorInvalidValue;
    if (const int e = tw_allow_shared<gemm_fp32_kernel, SMEM>()) return e;
    static std::atomic<bool> known{false};
    if (!known.load(std::memory_order_relaxed)) {
        const int built = tw_gemm_fp32_built();
        if (built != 1) return built < 0 ? -built : (int)cudaErrorInvalidConfiguration;
        known.store(true, std::memory_order_relaxed);
    }
    return tw_launch(gemm_fp32_kernel, dim3((unsigned)blocks), dim3(THREADS), (size_t)SMEM, stream, 1, out, out_stride, x, x_stride, w,
                     w_stride, m, n, k, status);
}
