// The products of routed experts in steps with few rows (decode): every expert's rows times its matrices, in bf16 with fp32 sums.
//
// The pairs (row, chosen expert) come sorted by expert (tw_moe_sort); expert e's places are ends[e - 1] .. ends[e] - 1.  What
// bounds such a step is reading the matrices of the experts that were chosen, once: as in gemm_smallm.cu they stream from
// memory straight into tensor-core fragments as the 16-row operand, and the expert's rows -- up to 8 or 16 a pass -- are
// the other one, read through the sorted order where they lie (nothing is gathered).  Gate rows and their up rows share a tile
// (eight each), so act(gate) * up is made of the sums in registers.  Experts that nobody chose cost a block nothing but its
// launch.
//
//   tw_moe_rows_in    act[place] = glu(Wg_e h, Wu_e h), or f(Wu_e h) for experts without a gate
//   tw_moe_rows_out   ys[place] = Wd_e act[place]
//
// 8 rows, two of 8 experts of 4,736 x 3,584 each: 75 us (gate and up) and 43 us (down) for the 7.2 experts that are chosen on
// average, 6.5 and 5.7 TB/s; the library's grouped product took 186 us for both, and the pairs' rows and the activation two
// launches more.
#include "moe_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int WARPS = 4, CHUNK = 64;            // values of k per step: a thread reads 32 contiguous bytes of each of its rows

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ld_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
struct Frag { uint4 lo, hi; };                  // 16 consecutive values of k of one row

enum : int { ROWS_GLU = 0, ROWS_ACT = 1, ROWS_OUT = 2 };

struct MoeRows {
    const bf16* w;              // glu: [E, 2, N, K]; else [E, N, K]
    const bf16* x; int x_stride;
    const int* order; int top;  // the rows of x by place: order[place] / top (null: the place itself)
    const int* ends;
    bf16* out;                  // [places, N]
    int N, K, how;              // how: the glu or the activation
    float limit, alpha;
};

template <int MODE, int NT>
__global__ void __launch_bounds__(WARPS * 32, (NT == 1 ? 4 : 1))
moe_rows_kernel(MoeRows a) {
    tw_grid_wait();
    tw_grid_launch_dependents();
    const int e = blockIdx.y;
    const int begin = e > 0 ? a.ends[e - 1] : 0, end = a.ends[e];
    if (begin >= end) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int tile = blockIdx.x * WARPS + warp;
    // glu: eight outputs per tile, a gate row and its up row in a thread; else sixteen outputs
    const int ra = MODE == ROWS_GLU ? tile * 8 + g : tile * 16 + g, rb = MODE == ROWS_GLU ? ra : ra + 8;
    const int N = a.N, K = a.K;
    if (tile * (MODE == ROWS_GLU ? 8 : 16) >= N) return;
    const bool va = ra < N, vb = rb < N;
    const bf16* w = a.w + (size_t)e * (MODE == ROWS_GLU ? 2 : 1) * N * K;
    const bf16* wa = w + (size_t)(va ? ra : 0) * K;
    const bf16* wb = w + (MODE == ROWS_GLU ? (size_t)N * K : 0) + (size_t)(vb ? rb : 0) * K;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    auto load_w = [&](const bf16* row, bool valid, int k0) -> Frag {
        const int kk = k0 + 16 * c;
        Frag f;
        f.lo = (valid && kk < K) ? ld_stream(row + kk) : zero;
        f.hi = (valid && kk + 8 < K) ? ld_stream(row + kk + 8) : zero;
        return f;
    };
    auto load_x = [&](const bf16* row, bool valid, int k0) -> Frag {
        const int kk = k0 + 16 * c;
        Frag f;
        f.lo = (valid && kk < K) ? *reinterpret_cast<const uint4*>(row + kk) : zero;
        f.hi = (valid && kk + 8 < K) ? *reinterpret_cast<const uint4*>(row + kk + 8) : zero;
        return f;
    };
    for (int p0 = begin; p0 < end; p0 += 8 * NT) {
        const bf16* xr[NT];
        bool vx[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int place = p0 + t * 8 + g;
            vx[t] = place < end;
            const int row = !vx[t] ? 0 : (a.order ? a.order[place] / a.top : place);
            xr[t] = a.x + (size_t)row * a.x_stride;
        }
        float acc[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t) { acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f; }
        Frag a_cur = load_w(wa, va, 0), b_cur = load_w(wb, vb, 0);
        Frag a_nxt = load_w(wa, va, CHUNK), b_nxt = load_w(wb, vb, CHUNK);
        Frag x_nxt = load_x(xr[0], vx[0], 0);
        for (int k = 0; k < K; k += CHUNK) {
            const Frag a_far = load_w(wa, va, k + 2 * CHUNK), b_far = load_w(wb, vb, k + 2 * CHUNK);
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const Frag xf = NT == 1 ? x_nxt : load_x(xr[t], vx[t], k);
                if (NT == 1) x_nxt = load_x(xr[0], vx[0], k + CHUNK);
                mma_bf16(acc[t], a_cur.lo.x, b_cur.lo.x, a_cur.lo.y, b_cur.lo.y, xf.lo.x, xf.lo.y);
                mma_bf16(acc[t], a_cur.lo.z, b_cur.lo.z, a_cur.lo.w, b_cur.lo.w, xf.lo.z, xf.lo.w);
                mma_bf16(acc[t], a_cur.hi.x, b_cur.hi.x, a_cur.hi.y, b_cur.hi.y, xf.hi.x, xf.hi.y);
                mma_bf16(acc[t], a_cur.hi.z, b_cur.hi.z, a_cur.hi.w, b_cur.hi.w, xf.hi.z, xf.hi.w);
            }
            a_cur = a_nxt; b_cur = b_nxt;
            a_nxt = a_far; b_nxt = b_far;
        }
        // acc[t][0..1]: weight row ra, places p0 + 8 t + 2 c, + 1;  acc[t][2..3]: weight row rb
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int place = p0 + t * 8 + 2 * c + x;
                if (place >= end) continue;
                bf16* o = a.out + (size_t)place * N;
                if (MODE == ROWS_GLU) {
                    if (va) o[ra] = __float2bfloat16_rn(tw_glu(acc[t][x], acc[t][2 + x], a.how, a.limit, a.alpha));
                } else {
                    const float ya = MODE == ROWS_ACT ? tw_activate(acc[t][x], a.how) : acc[t][x];
                    const float yb = MODE == ROWS_ACT ? tw_activate(acc[t][2 + x], a.how) : acc[t][2 + x];
                    if (va) o[ra] = __float2bfloat16_rn(ya);
                    if (vb) o[rb] = __float2bfloat16_rn(yb);
                }
            }
    }
}

template <int MODE>
int launch_rows(const MoeRows& a, int E, int most, cudaStream_t stream) {
    const int per = WARPS * (MODE == ROWS_GLU ? 8 : 16);
    const dim3 grid((a.N + per - 1) / per, E);
    return most <= 8 ? tw_launch(moe_rows_kernel<MODE, 1>, grid, dim3(WARPS * 32), 0, stream, 1, a)
                     : tw_launch(moe_rows_kernel<MODE, 2>, grid, dim3(WARPS * 32), 0, stream, 1, a);
}

bool fits(const void* w, const void* x, int x_stride, int K, int E) {
    return !((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(x)) & 15) && (x_stride & 7) == 0 && K > 0 && (K & 7) == 0
           && E > 0 && E <= 65535;
}

}  // namespace

// `most`: no expert has more rows than this (more cost further passes over the matrices, nothing else).  gated: w [E, 2, N, K] and
// `how` a glu (tw_glu, with limit and alpha); else w [E, N, K] and `how` an activation.  act bf16 [places, N].
TW_EXPORT int tw_moe_rows_in(void* act, const void* h, int h_stride, const void* w, const int* order, const int* ends, int N, int K, int E,
                             int top, int most, int gated, int how, float limit, float alpha, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (!fits(w, h, h_stride, K, E) || top <= 0 || (!gated && (how < TW_ACT_NONE || how > TW_ACT_RELU_SQUARED))) return (int)cudaErrorInvalidValue;
    const MoeRows a{(const bf16*)w, (const bf16*)h, h_stride, order, top, ends, (bf16*)act, N, K, how, limit, alpha};
    return gated ? launch_rows<ROWS_GLU>(a, E, most, stream) : launch_rows<ROWS_ACT>(a, E, most, stream);
}

// ys bf16 [places, N] from act bf16 [places, K] and w [E, N, K].
TW_EXPORT int tw_moe_rows_out(void* ys, const void* act, const void* w, const int* ends, int N, int K, int E, int most, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (!fits(w, act, K, K, E)) return (int)cudaErrorInvalidValue;
    const MoeRows a{(const bf16*)w, (const bf16*)act, K, nullptr, 1, ends, (bf16*)ys, N, K, 0, 0.f, 0.f};
    return launch_rows<ROWS_OUT>(a, E, most, stream);
}
