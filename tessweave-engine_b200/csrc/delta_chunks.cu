// Prompt portions of the gated delta rule (TW_REC_DELTA of linear_recurrence.cu, one decay per head) in chunks of 64 tokens.
//
// With F_t the sum of the log decays up to token t of its chunk, S the state before the chunk and u_t what token t writes,
//
//   u_t = beta_t (v_t - e^(F_t) S^T k_t - sum over s < t of e^(F_t - F_s) (k_t . k_s) u_s)
//   o_t = e^(F_t) S^T q_t + sum over s <= t of e^(F_t - F_s) (q_t . k_s) u_s
//   S' = e^(F_64) S + sum over s of e^(F_64 - F_s) k_s u_s^T
//
// The first line is a unit lower triangular system, (I + A) U = diag(beta) V - diag(beta e^F) K S.  Its matrix does not know
// S, so U = U0 - W S with (I + A) U0 = diag(beta) V and (I + A) W = diag(beta e^F) K.  Three launches:
//   (1) every chunk: the products k . k, then W and U0 by forward substitution in fp32, a thread per column;
//   (2) the walk over the chunks, the columns of S shared out: U = U0 - W S, S' = e^(F_64) S + K^T (e^(F_64 - F) U);
//   (3) every chunk: the outputs.
//
// What bounded the rule token by token is its chain (0.23 us a token, whatever the GPU could do beside it); now it is the
// walk's, two products and two barriers a chunk, and the reads of W and K (96 KB a chunk and block) from L2.
// 14 heads of 128 x 128 over 2,048 tokens: 482 us token by token, 202 in chunks (59 + 96 + 47 for the launches); portions of
// 777, 1,024 and 201 tokens: 378 and 184 (58 + 77 + 49); 14 heads of 64 x 64, 2,048 tokens: 413 and 118 (37 + 57 + 21).
// Against 64 bits: outputs 1.8e-7 (token by token 6.5e-7), state 2.0e-7 (6.1e-7).
//
// Precision: q, k, v, the state and everything in between are 32-bit numbers here.  They enter a product on the tensor
// cores as the sum of three bf16 terms (24 bits), with a product for each of the six pairs of terms that matter; the
// leading pair is added by fp32 additions that round to nearest.  The substitution is plain fp32.
#include "recurrence_chunks.cuh"

namespace {

struct DcArgs {
    float* out;                                             // [rows, H * DV]
    const float* q; const float* k; const float* v; int q_stride, k_stride, v_stride;
    const float* pre; int pre_stride;                       // projected decay [rows, H]
    const float* write; int write_stride;                   // write strength before its sigmoid [rows, H]
    const float* rate_log; const float* dt_bias;            // [H]
    float q_scale, k_scale;
    float* state; long long state_stride;
    const int* seq_slot; const int* seq_q_start; const int* seq_q_len;
    int n_seqs, H, qk_group, min_len, write_state;
    // scratch, per chunk and head unless it says otherwise
    float* before;                                          // the state before the chunk: [DV / 8][KT][32 lanes][4]
    float* u;                                               // U0, then U: [DV / 8][4][32 lanes][4], see below
    bf16* w;                                                // W: [3][L][DK]
    bf16* keys;                                             // k, per chunk and head of q and k: [3][L][DK]
    float2* decay;                                          // F_t as a float and what it leaves: [L]
};

// Of U (tokens x values) a lane holds what the tensor cores want of it as an operand: of a tile of 8 values and 16 tokens
// lane 4 v + p holds tokens 2 p, 2 p + 1, 2 p + 8, 2 p + 9 of value v.
__device__ __forceinline__ size_t u_at(int value, int token16) { return ((size_t)((value >> 3) * (L / 16) + token16) * 32 + (value & 7) * 4) * 4; }

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

// fp32 rows (zeros from `ct` on) as three bf16 terms, four channels per thread and step
__device__ __forceinline__ void stage_rows(bf16* dst, const float* src, int stride, int ct, float scale) {
    constexpr int N = L * (DK / 4) / THREADS;
    float4 v[N];
#pragma unroll
    for (int e = 0; e < N; ++e) {
        const int x = threadIdx.x + e * THREADS, t = x / (DK / 4), i = x % (DK / 4) * 4;
        v[e] = t < ct ? *reinterpret_cast<const float4*>(src + (size_t)t * stride + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int e = 0; e < N; ++e) {
        const int x = threadIdx.x + e * THREADS, t = x / (DK / 4), i = x % (DK / 4) * 4;
        put3(dst, t, i, v[e].x * scale, v[e].y * scale);
        put3(dst, t, i + 2, v[e].z * scale, v[e].w * scale);
    }
}

// The tiles half, half + 2 (of 16 columns, at or before the diagonal) of rows 16 rt .. of x y^T, x and y in three terms.
__device__ __forceinline__ void triangle(float (&G)[2][2][4], const bf16* x, const bf16* y, int rt, int half, int lane) {
    float low[2][2][2][4];                                  // (the smaller products, in two sums)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) G[i][j][e] = low[0][i][j][e] = low[1][i][j][e] = 0.f;
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        uint32_t A[3][4];
#pragma unroll
        for (int t = 0; t < 3; ++t) ldmatrix_x4(A[t], x + (t * L + rt * 16 + (lane & 15)) * RS + k * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = half + 2 * i;
            if (j > rt) continue;
#pragma unroll
            for (int u = 2; u >= 0; --u) {
                uint32_t B[4];
                ldmatrix_x4(B, y + (u * L + j * 16 + (lane & 7) + ((lane >> 4) << 3)) * RS + k * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
                for (int t = 2 - u; t >= 0; --t) {
                    if (t + u == 0) { mma_top(G[i][0], A[t], B[0], B[1]); mma_top(G[i][1], A[t], B[2], B[3]); }
                    else { mma_bf16(low[t & 1][i][0], A[t], B[0], B[1]); mma_bf16(low[t & 1][i][1], A[t], B[2], B[3]); }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) G[i][j][e] += low[0][i][j][e] + low[1][i][j][e];
}

// ---- (1) a chunk's W and U0.  A thread owns a column: a key channel of W or a value of U0, all 64 tokens of it in registers;
// as soon as a token is known it is taken out of all later ones, so that the multiply-adds of a step do not wait for one
// another (2,016 a column, the matrix read from shared memory by all threads alike).
template <int DV>
__global__ void __launch_bounds__(THREADS, 2) delta_solve_kernel(DcArgs a) {
    extern __shared__ __align__(16) unsigned char dc_smem[];
    bf16* ks = reinterpret_cast<bf16*>(dc_smem);            // [3][L][RS]
    float* at = reinterpret_cast<float*>(ks + 3 * L * RS);  // [L][L + 4]: column s of A, then its rows t
    constexpr int AS = L + 4;
    __shared__ float2 f[L];
    __shared__ float ef[L], beta[L];
    tw_grid_wait();
    tw_grid_launch_dependents();
    const int c = blockIdx.x, h = blockIdx.y, s = blockIdx.z;
    const int len = a.seq_q_len[s];
    if (len < a.min_len || c * L >= len) return;
    const int ct = min(L, len - c * L), hq = h / a.qk_group;
    const size_t row0 = (size_t)a.seq_q_start[s] + c * L;
    const size_t chunk = (size_t)first_chunk(a.seq_q_len, s, a.min_len) + c, place = chunk * a.H + h;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const float* krows = a.k + row0 * a.k_stride + (size_t)hq * DK;
    // this thread's column, as it comes
    const int col = threadIdx.x;
    const bool of_w = col < DK, live = col < DK + DV;
    const float* src = of_w ? krows + col : a.v + row0 * a.v_stride + (size_t)h * DV + (col - DK);
    const int src_stride = of_w ? a.k_stride : a.v_stride;
    float X[L];
#pragma unroll
    for (int t = 0; t < L; ++t) X[t] = live && t < ct ? src[(size_t)t * src_stride] : 0.f;
    if (warp == 0) {
        // (a token behind the last neither decays nor writes)
        const float rate = expf(a.rate_log[h]), bias = a.dt_bias[h];
        double d[2];
        float b[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = lane + 32 * e;
            d[e] = 0.0; b[e] = 0.f;
            if (t < ct) {
                d[e] = -rate * softplus(a.pre[(row0 + t) * a.pre_stride + h] + bias);
                if (d[e] < -1000.0) d[e] = -1000.0;         // (nothing is left either way, and differences of sums stay numbers)
                b[e] = 1.0f / (1.0f + expf(-a.write[(row0 + t) * a.write_stride + h]));
            }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double u0 = __shfl_up_sync(0xffffffffu, d[0], o), u1 = __shfl_up_sync(0xffffffffu, d[1], o);
            if (lane >= o) { d[0] += u0; d[1] += u1; }
        }
        d[1] += __shfl_sync(0xffffffffu, d[0], 31);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = lane + 32 * e;
            const float hi = (float)d[e];
            f[t] = make_float2(hi, (float)(d[e] - (double)hi));
            ef[t] = (float)exp(d[e]);
            beta[t] = b[e];
            a.decay[place * L + t] = f[t];
        }
    }
    stage_rows(ks, krows, a.k_stride, ct, a.k_scale);
    __syncthreads();
    if (h % a.qk_group == 0) {                              // the keys themselves, for the walk
        bf16* dst = a.keys + (chunk * (a.H / a.qk_group) + hq) * (3 * L * DK);
        for (int e = threadIdx.x; e < 3 * L * (DK / 8); e += THREADS) {
            const int r = e / (DK / 8), i = e % (DK / 8) * 8;
            *reinterpret_cast<uint4*>(dst + (size_t)r * DK + i) = *reinterpret_cast<const uint4*>(ks + r * RS + i);
        }
    }
    {
        const int half = warp >> 2, rt = half ? 3 - (warp & 3) : (warp & 3);
        float G[2][2][4];
        triangle(G, ks, ks, rt, half, lane);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int j = half + 2 * x;
            if (j > rt) continue;
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = rt * 16 + g + (e < 2 ? 0 : 8), from = j * 16 + y * 8 + 2 * tq + (e & 1);
                    at[from * AS + t] = from < t ? G[x][y][e] * (beta[t] * expf((f[t].x - f[from].x) + (f[t].y - f[from].y))) : 0.f;
                }
        }
    }
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int t = 0; t < L; ++t) X[t] = X[t] * (of_w ? a.k_scale * (beta[t] * ef[t]) : beta[t]);
    // (tokens in pairs, so that one instruction takes a token out of two later ones: half the instructions to fetch and to issue, on
    // which the warps waited most; the layers of three portions and of 2,048 tokens 301.2 -> 298 and 289.5 -> 284.5 us)
    unsigned long long X2[L / 2];
#pragma unroll
    for (int p = 0; p < L / 2; ++p) X2[p] = pack2(X[2 * p], X[2 * p + 1]);
#pragma unroll
    for (int from = 0; from < L - 1; ++from) {
        const float2 own = unpack2(X2[from / 2]);
        const float taken = -((from & 1) ? own.y : own.x);
        const unsigned long long both = pack2(taken, taken);
        // (tokens of the same group of four at or before `from` are left out)
#pragma unroll
        for (int t4 = (from + 1) / 4; t4 < L / 4; ++t4) {
            const ulonglong2 m = *reinterpret_cast<const ulonglong2*>(at + from * AS + 4 * t4);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int p = 2 * t4 + e;
                if (2 * p > from) X2[p] = fma2(e ? m.y : m.x, both, X2[p]);
                else if (2 * p + 1 > from) X2[p] = pack2(own.x, fmaf(unpack2(e ? m.y : m.x).y, taken, own.y));     // (from is 2 p)
            }
        }
    }
#pragma unroll
    for (int p = 0; p < L / 2; ++p) {
        const float2 x = unpack2(X2[p]);
        X[2 * p] = x.x; X[2 * p + 1] = x.y;
    }
    if (of_w) {
        // neighbouring columns in pairs: the even one writes the even tokens, the odd one the odd tokens
        bf16* dst = a.w + place * (3 * L * DK);
        const bool odd = col & 1;
#pragma unroll
        for (int t = 0; t < L; t += 2) {
            const float other = __shfl_xor_sync(0xffffffffu, odd ? X[t] : X[t + 1], 1);
            uint32_t hi, mid, lo;
            if (odd) split3(other, X[t + 1], hi, mid, lo);
            else split3(X[t], other, hi, mid, lo);
            bf16* p = dst + (size_t)(t + odd) * DK + (col & ~1);
            *reinterpret_cast<uint32_t*>(p) = hi;
            *reinterpret_cast<uint32_t*>(p + L * DK) = mid;
            *reinterpret_cast<uint32_t*>(p + 2 * L * DK) = lo;
        }
    } else {
        float* dst = a.u + place * ((size_t)L * DV);
        const int value = col - DK;
#pragma unroll
        for (int i = 0; i < L / 16; ++i)
#pragma unroll
            for (int p = 0; p < 4; ++p)
                *reinterpret_cast<float4*>(dst + u_at(value, i) + 4 * p) =
                    make_float4(X[16 * i + 2 * p], X[16 * i + 2 * p + 1], X[16 * i + 2 * p + 8], X[16 * i + 2 * p + 9]);
    }
}

// ---- (2) the walk.  A block owns 16 VT values of a head's state, transposed (rows are values): warp w the key channels 16 w ...
// of it, in its accumulators.  S and the weighted U go through shared memory as three terms, which all warps read as the row
// operand; the W and K of the chunks stand in a ring of four places, or of three where the state takes more room, the next ones on
// their way while one is used.
//
// What bounds it is the chain of a chunk (its products, on mma.sync, and two barriers), 3.0 us with 16 values and 4.5 with 32 (keys of
// 128), and one block fits an SM: 16 unless that gives more rounds of blocks than 32 by more than this (ops.delta_walk_values).  14 heads
// of 128 x 128: portions of 777, 1,024 and 201 tokens 89 us and 77 (336 blocks in two rounds, 168 whose longest start first), of 2,048
// tokens and 30 single ones 97 and 147, of 1,500 and 300 tokens 74 and 111.
template <int DV, int VT>
__global__ void __launch_bounds__(THREADS, 1) delta_walk_kernel(DcArgs a) {
    constexpr int NT = DK / 64;                             // tiles of 8 key channels per warp
    constexpr int TERMS = 3 * L * RS, SS = DK + 8, V = 16 * VT, PLACES = VT == 1 ? 4 : 3;
    extern __shared__ __align__(16) unsigned char dc_smem[];
    bf16* ring = reinterpret_cast<bf16*>(dc_smem);          // [PLACES][3][L][RS]: W of chunk 0, K of chunk 0, W of chunk 1, ...
    bf16* st = ring + PLACES * TERMS;                            // [3][V][SS] the state
    bf16* ut = st + 3 * V * SS;                             // [3][V][MS] the weighted U
    __shared__ __align__(16) float2 f[2][L];
    tw_grid_wait();
    tw_grid_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int h = blockIdx.y, v0 = blockIdx.x * V;
    int s = blockIdx.z;
    if (a.n_seqs <= 32) {                                   // the longest request's blocks start first (ops.DELTA_WALK_SORTED)
        const int mine = lane < a.n_seqs ? a.seq_q_len[lane] : -1;
        int rank = 0;
        for (int r = 0; r < a.n_seqs; ++r) {
            const int other = __shfl_sync(0xffffffffu, mine, r);
            rank += other > mine || (other == mine && r < lane);
        }
        s = __ffs(__ballot_sync(0xffffffffu, lane < a.n_seqs && rank == s)) - 1;
    }
    const int len = a.seq_q_len[s];
    if (len < a.min_len) return;
    const int chunks = (len + L - 1) / L, hq = h / a.qk_group, Hq = a.H / a.qk_group;
    const size_t first = first_chunk(a.seq_q_len, s, a.min_len);
    float* slot = a.state + (size_t)a.seq_slot[s] * a.state_stride + (size_t)h * ((size_t)DK * DV);

    auto copy = [&](int place, const bf16* src) {
        bf16* dst = ring + place * TERMS;
        for (int e = threadIdx.x; e < 3 * L * (DK / 8); e += THREADS) {
            const int r = e / (DK / 8), i = e % (DK / 8) * 8;
            tw_attn::cp_async16(dst + r * RS + i, src + (size_t)r * DK + i, 16);
        }
    };
    auto fetch_w = [&](int c) {                             // with the chunk's decays
        if (c < chunks) {
            copy((2 * c) % PLACES, a.w + ((first + c) * a.H + h) * (size_t)(3 * L * DK));
            if (threadIdx.x < L / 2)
                tw_attn::cp_async16(&f[c & 1][2 * threadIdx.x], a.decay + ((first + c) * a.H + h) * L + 2 * threadIdx.x, 16);
        }
        tw_attn::cp_async_commit();
    };
    auto fetch_k = [&](int c) {
        if (c < chunks) copy((2 * c + 1) % PLACES, a.keys + ((first + c) * Hq + hq) * (size_t)(3 * L * DK));
        tw_attn::cp_async_commit();
    };
    // U of this block's values and warp w's tokens 8 w ..: pairs of tokens of values v0 + 8 x + g
    auto u_place = [&](int c, int x) {
        return reinterpret_cast<float2*>(a.u + ((first + c) * a.H + h) * ((size_t)L * DV) + u_at(v0 + 8 * x, warp >> 1) + lane * 4 + (warp & 1) * 2);
    };

    float S[VT][NT][4];                                     // values 16 z + g, + 8; key channels 8 (NT w + n) + 2 tq, + 1
#pragma unroll
    for (int z = 0; z < VT; ++z)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                S[z][n][e] = slot[(size_t)((warp * NT + n) * 8 + 2 * tq + (e & 1)) * DV + v0 + 16 * z + g + (e < 2 ? 0 : 8)];
    fetch_w(0);
    fetch_k(0);
    float2 u0[2 * VT];
#pragma unroll
    for (int x = 0; x < 2 * VT; ++x) u0[x] = *u_place(0, x);
    for (int c = 0; c < chunks; ++c) {
        // the state before this chunk: for the outputs, and as terms for everybody
        float* keep = a.before + ((first + c) * a.H + h) * ((size_t)DK * DV);
#pragma unroll
        for (int z = 0; z < VT; ++z)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int k8 = warp * NT + n;
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    *reinterpret_cast<float2*>(keep + (((size_t)((v0 >> 3) + 2 * z + x) * KT + (k8 >> 1)) * 32 + lane) * 4 + (k8 & 1) * 2) =
                        make_float2(S[z][n][2 * x], S[z][n][2 * x + 1]);
                    uint32_t hi, mid, lo;
                    split3(S[z][n][2 * x], S[z][n][2 * x + 1], hi, mid, lo);
                    bf16* p = st + (16 * z + g + 8 * x) * SS + k8 * 8 + 2 * tq;
                    *reinterpret_cast<uint32_t*>(p) = hi;
                    *reinterpret_cast<uint32_t*>(p + V * SS) = mid;
                    *reinterpret_cast<uint32_t*>(p + 2 * V * SS) = lo;
                }
            }
        tw_attn::cp_async_wait<1>();
        __syncthreads();                                    // the state, W and the decays are there; nobody reads the keys before these
        fetch_w(c + 1);
        if constexpr (PLACES == 4) fetch_k(c + 1);
        const bf16* ws = ring + (2 * c) % PLACES * TERMS;
        const bf16* ks = ring + (2 * c + 1) % PLACES * TERMS;
        // ---- U^T = U0^T - S^T W^T, this warp's eight tokens
        // (the smaller products in sums of their own)
        float top[VT][4], low[VT][6][4];
#pragma unroll
        for (int z = 0; z < VT; ++z) {
            top[z][0] = top[z][1] = top[z][2] = top[z][3] = 0.f;
#pragma unroll
            for (int x = 0; x < 6; ++x) low[z][x][0] = low[z][x][1] = low[z][x][2] = low[z][x][3] = 0.f;
        }
#pragma unroll
        for (int k = 0; k < KT; k += 2) {
            uint32_t B[3][4];                               // two steps of k: (k, first and last eight), (k + 1, ...)
#pragma unroll
            for (int u = 0; u < 3; ++u) ldmatrix_x4(B[u], ws + (u * L + warp * 8 + (lane & 7)) * RS + k * 16 + (lane >> 3) * 8);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int z = 0; z < VT; ++z) {
                    uint32_t A[3][4];
#pragma unroll
                    for (int t = 0; t < 3; ++t) ldmatrix_x4(A[t], st + (t * V + 16 * z + (lane & 15)) * SS + (k + x) * 16 + (lane >> 4) * 8);
#pragma unroll
                    for (int u = 2; u >= 0; --u)
#pragma unroll
                        for (int t = 2 - u; t >= 0; --t) {
                            if (t + u == 0) mma_top(top[z], A[t], B[u][2 * x], B[u][2 * x + 1]);
                            else mma_bf16(low[z][3 * x + u], A[t], B[u][2 * x], B[u][2 * x + 1]);
                        }
                }
        }
        const float2 fl = f[c & 1][L - 1];
        const float whole = expf(fl.x + fl.y);
        {
            const int t0 = warp * 8 + 2 * tq;
            const float2 fa = f[c & 1][t0], fb = f[c & 1][t0 + 1];
            const float wa = expf((fl.x - fa.x) + (fl.y - fa.y)), wb = expf((fl.x - fb.x) + (fl.y - fb.y));
#pragma unroll
            for (int z = 0; z < VT; ++z) {
                float U[4] = {u0[2 * z].x, u0[2 * z].y, u0[2 * z + 1].x, u0[2 * z + 1].y};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    U[e] -= top[z][e] + (((low[z][0][e] + low[z][3][e]) + (low[z][1][e] + low[z][4][e])) + (low[z][2][e] + low[z][5][e]));
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    *u_place(c, 2 * z + x) = make_float2(U[2 * x], U[2 * x + 1]);
                    uint32_t hi, mid, lo;
                    split3(U[2 * x] * wa, U[2 * x + 1] * wb, hi, mid, lo);
                    bf16* p = ut + (16 * z + g + 8 * x) * MS + t0;
                    *reinterpret_cast<uint32_t*>(p) = hi;
                    *reinterpret_cast<uint32_t*>(p + V * MS) = mid;
                    *reinterpret_cast<uint32_t*>(p + 2 * V * MS) = lo;
                }
            }
        }
        if (c + 1 < chunks) {
#pragma unroll
            for (int x = 0; x < 2 * VT; ++x) u0[x] = *u_place(c + 1, x);
        }
        tw_attn::cp_async_wait<PLACES - 2>();
        __syncthreads();                                    // the weighted U and the keys are there, and nobody reads W or the old state any more
        if constexpr (PLACES == 3) fetch_k(c + 1);
        // ---- S^T = e^F S^T + (w U)^T K, this warp's key channels
        float lo2[VT][3][NT][4];
#pragma unroll
        for (int z = 0; z < VT; ++z)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) { S[z][n][e] *= whole; lo2[z][0][n][e] = lo2[z][1][n][e] = lo2[z][2][n][e] = 0.f; }
#pragma unroll
        for (int k = 0; k < L / 16; ++k) {
            uint32_t B[3][4];
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const bf16* base = ks + (u * L + k * 16 + (lane & 15)) * RS + warp * NT * 8;
                if constexpr (NT == 2) {
                    ldmatrix_x4_trans(B[u], base + (lane >> 4) * 8);
                } else {
                    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                                 : "=r"(B[u][0]), "=r"(B[u][1]) : "r"((uint32_t)__cvta_generic_to_shared(base)));
                }
            }
#pragma unroll
            for (int z = 0; z < VT; ++z) {
                uint32_t A[3][4];
#pragma unroll
                for (int t = 0; t < 3; ++t) ldmatrix_x4(A[t], ut + (t * V + 16 * z + (lane & 15)) * MS + k * 16 + (lane >> 4) * 8);
#pragma unroll
                for (int u = 2; u >= 0; --u)
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int t = 2 - u; t >= 0; --t) {
                            if (t + u == 0) mma_top(S[z][n], A[t], B[u][2 * n], B[u][2 * n + 1]);
                            else mma_bf16(lo2[z][u][n], A[t], B[u][2 * n], B[u][2 * n + 1]);
                        }
            }
        }
#pragma unroll
        for (int z = 0; z < VT; ++z)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[z][n][e] += (lo2[z][0][n][e] + lo2[z][1][n][e]) + lo2[z][2][n][e];
    }
    tw_attn::cp_async_wait<0>();
    if (!a.write_state) return;
#pragma unroll
    for (int z = 0; z < VT; ++z)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                slot[(size_t)((warp * NT + n) * 8 + 2 * tq + (e & 1)) * DV + v0 + 16 * z + g + (e < 2 ? 0 : 8)] = S[z][n][e];
}

// ---- (3) a chunk's outputs, as in recurrence_chunks.cu; U is read like the state, in the order the tensor cores want.
template <int DV>
__global__ void __launch_bounds__(THREADS, 2) delta_outputs_kernel(DcArgs a) {
    constexpr int NTW = DV / 64;
    extern __shared__ __align__(16) unsigned char dc_smem[];
    bf16* qs = reinterpret_cast<bf16*>(dc_smem);            // [3][L][RS]
    bf16* ks = qs + 3 * L * RS;                             // [3][L][RS]; later the coefficients times q . k: [3][L][MS]
    bf16* ms = ks;
    __shared__ float2 f[L];
    __shared__ float in[L];
    tw_grid_wait();
    tw_grid_launch_dependents();
    const int c = blockIdx.x, h = blockIdx.y, s = blockIdx.z;
    const int len = a.seq_q_len[s];
    if (len < a.min_len || c * L >= len) return;
    const int ct = min(L, len - c * L), hq = h / a.qk_group;
    const size_t row0 = (size_t)a.seq_q_start[s] + c * L;
    const size_t place = ((size_t)first_chunk(a.seq_q_len, s, a.min_len) + c) * a.H + h;
    const float4* state = reinterpret_cast<const float4*>(a.before + place * ((size_t)DK * DV));
    const float* urows = a.u + place * ((size_t)L * DV);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    if (threadIdx.x < L) {
        const float2 x = a.decay[place * L + threadIdx.x];
        f[threadIdx.x] = x;
        in[threadIdx.x] = (float)exp((double)x.x + (double)x.y);
    }
    stage_rows(qs, a.q + row0 * a.q_stride + (size_t)hq * DK, a.q_stride, ct, a.q_scale);
    stage_rows(ks, a.k + row0 * a.k_stride + (size_t)hq * DK, a.k_stride, ct, a.k_scale);
    __syncthreads();
    const int half = warp >> 2, rt = half ? 3 - (warp & 3) : (warp & 3);
    float G[2][2][4];
    triangle(G, qs, ks, rt, half, lane);
    __syncthreads();                                        // nobody reads k any more: its place is the coefficients'
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int j = half + 2 * x;
        if (j > rt) continue;
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const int s0 = j * 16 + y * 8 + 2 * tq;
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                const int t = rt * 16 + g + 8 * z;
                float m[2];
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    m[e] = s0 + e <= t ? G[x][y][2 * z + e] * expf((f[t].x - f[s0 + e].x) + (f[t].y - f[s0 + e].y)) : 0.f;
                uint32_t hi, mid, lo;
                split3(m[0], m[1], hi, mid, lo);
                *reinterpret_cast<uint32_t*>(ms + t * MS + s0) = hi;
                *reinterpret_cast<uint32_t*>(ms + (L + t) * MS + s0) = mid;
                *reinterpret_cast<uint32_t*>(ms + (2 * L + t) * MS + s0) = lo;
            }
        }
    }
    float acc[L / 16][NTW][4], low[L / 16][NTW][4];
#pragma unroll
    for (int r = 0; r < L / 16; ++r)
#pragma unroll
        for (int n = 0; n < NTW; ++n) {
            acc[r][n][0] = acc[r][n][1] = acc[r][n][2] = acc[r][n][3] = 0.f;
            low[r][n][0] = low[r][n][1] = low[r][n][2] = low[r][n][3] = 0.f;
        }
    float4 next[NTW];
#pragma unroll
    for (int n = 0; n < NTW; ++n) next[n] = state[((warp * NTW + n) * KT) * 32 + lane];
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        uint32_t B[NTW][3][2];
#pragma unroll
        for (int n = 0; n < NTW; ++n) {
            const float4 v = next[n];
            if (k + 1 < KT) next[n] = state[((warp * NTW + n) * KT + k + 1) * 32 + lane];
            split3(v.x, v.y, B[n][0][0], B[n][1][0], B[n][2][0]);
            split3(v.z, v.w, B[n][0][1], B[n][1][1], B[n][2][1]);
        }
#pragma unroll
        for (int r = 0; r < L / 16; ++r)
#pragma unroll
            for (int t = 2; t >= 0; --t) {
                uint32_t A[4];
                ldmatrix_x4(A, qs + (t * L + r * 16 + (lane & 15)) * RS + k * 16 + (lane >> 4) * 8);
#pragma unroll
                for (int n = 0; n < NTW; ++n)
#pragma unroll
                    for (int u = 2 - t; u >= 0; --u) {
                        if (t + u == 0) mma_top(acc[r][n], A, B[n][u][0], B[n][u][1]);
                        else mma_bf16(low[r][n], A, B[n][u][0], B[n][u][1]);
                    }
            }
    }
#pragma unroll
    for (int r = 0; r < L / 16; ++r) {
        const float ia = in[r * 16 + g], ib = in[r * 16 + g + 8];
#pragma unroll
        for (int n = 0; n < NTW; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc[r][n][e] = (acc[r][n][e] + low[r][n][e]) * (e < 2 ? ia : ib);
                low[r][n][e] = 0.f;
            }
    }
    __syncthreads();                                        // the coefficients are there
    // ---- plus the chunk's own tokens.  (What a token writes that is not finite must not reach the tokens before it, with
    // which it shares a tile of the product: it is left out and added token by token.)
    bool loud = false;
#pragma unroll
    for (int j = 0; j < L / 16; ++j) {
        uint32_t B[NTW][3][2];
#pragma unroll
        for (int n = 0; n < NTW; ++n) {
            float4 v = *reinterpret_cast<const float4*>(urows + u_at((warp * NTW + n) * 8, j) + lane * 4);
            if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w))) {
                loud = true;
                v.x = isfinite(v.x) ? v.x : 0.f; v.y = isfinite(v.y) ? v.y : 0.f; v.z = isfinite(v.z) ? v.z : 0.f; v.w = isfinite(v.w) ? v.w : 0.f;
            }
            split3(v.x, v.y, B[n][0][0], B[n][1][0], B[n][2][0]);
            split3(v.z, v.w, B[n][0][1], B[n][1][1], B[n][2][1]);
        }
#pragma unroll
        for (int r = j; r < L / 16; ++r)
#pragma unroll
            for (int t = 2; t >= 0; --t) {
                uint32_t A[4];
                ldmatrix_x4(A, ms + (t * L + r * 16 + (lane & 15)) * MS + j * 16 + (lane >> 4) * 8);
#pragma unroll
                for (int n = 0; n < NTW; ++n)
#pragma unroll
                    for (int u = 2 - t; u >= 0; --u) {
                        if (t + u == 0) mma_top(acc[r][n], A, B[n][u][0], B[n][u][1]);
                        else mma_bf16(low[r][n], A, B[n][u][0], B[n][u][1]);
                    }
            }
    }
#pragma unroll
    for (int r = 0; r < L / 16; ++r)
#pragma unroll
        for (int n = 0; n < NTW; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][n][e] += low[r][n][e];
    if (__any_sync(0xffffffffu, loud)) {
        for (int src = 0; src < ct; ++src) {
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int value = (warp * NTW + n) * 8 + 2 * tq + e, in16 = src & 15;
                    const float v = urows[u_at(value, src >> 4) + (size_t)((in16 & 7) >> 1) * 4 + (in16 >> 3) * 2 + (in16 & 1)];
                    if (isfinite(v)) continue;
#pragma unroll
                    for (int r = 0; r < L / 16; ++r)
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const int t = r * 16 + g + 8 * x;
                            if (t >= src)
                                acc[r][n][2 * x + e] += v * ((__bfloat162float(ms[t * MS + src]) + __bfloat162float(ms[(L + t) * MS + src]))
                                                             + __bfloat162float(ms[(2 * L + t) * MS + src]));
                        }
                }
        }
    }
#pragma unroll
    for (int r = 0; r < L / 16; ++r)
#pragma unroll
        for (int n = 0; n < NTW; ++n) {
            const int ta = r * 16 + g, tb = ta + 8;
            float* dst = a.out + (row0 + ta) * ((size_t)a.H * DV) + (size_t)h * DV + (warp * NTW + n) * 8 + 2 * tq;
            if (ta < ct) *reinterpret_cast<float2*>(dst) = make_float2(acc[r][n][0], acc[r][n][1]);
            if (tb < ct) *reinterpret_cast<float2*>(dst + (size_t)8 * a.H * DV) = make_float2(acc[r][n][2], acc[r][n][3]);
        }
}

template <int DV>
int launch_delta(const DcArgs& a, int max_q_len, int walk_values, cudaStream_t stream) {
    constexpr size_t terms = (size_t)3 * L * RS * 2;
    constexpr size_t smem1 = terms + (size_t)L * (L + 4) * 4, smem3 = 2 * terms;
    constexpr auto smem2 = [](int vt) constexpr { return (vt == 1 ? 4 : 3) * terms + (size_t)3 * 16 * vt * (DK + 8 + MS) * 2; };
    static_assert(smem2(1) + 2 * L * 8 <= 227 * 1024 && smem2(2) + 2 * L * 8 <= 227 * 1024 && smem1 <= 112 * 1024 && smem3 <= 112 * 1024, "shared memory");
    if (const int e = tw_allow_shared<delta_solve_kernel<DV>, (int)smem1>()) return e;
    if (const int e = tw_allow_shared<delta_walk_kernel<DV, 1>, (int)smem2(1)>()) return e;
    if (const int e = tw_allow_shared<delta_walk_kernel<DV, 2>, (int)smem2(2)>()) return e;
    if (const int e = tw_allow_shared<delta_outputs_kernel<DV>, (int)smem3>()) return e;
    const dim3 grid((max_q_len + L - 1) / L, a.H, a.n_seqs);
    int code = tw_launch(delta_solve_kernel<DV>, grid, dim3(THREADS), smem1, stream, 1, a);
    if (code) return code;
    if (walk_values == 32)
        code = tw_launch(delta_walk_kernel<DV, 2>, dim3(DV / 32, a.H, a.n_seqs), dim3(THREADS), smem2(2), stream, 1, a);
    else
        code = tw_launch(delta_walk_kernel<DV, 1>, dim3(DV / 16, a.H, a.n_seqs), dim3(THREADS), smem2(1), stream, 1, a);
    if (code) return code;
    return tw_launch(delta_outputs_kernel<DV>, grid, dim3(THREADS), smem3, stream, 1, a);
}

}  // namespace

// Requests with at least `min_len` rows (the others are left to tw_linear_recurrence).  Operands as tw_linear_recurrence has them
// for the delta rule with a decay per head: q, k, v fp32 rows on 16-byte boundaries; Dk as compiled (64 or 128), Dv 64 or 128.
// `scratch`: for each of `chunks` (at least the sum of ceil(rows / 64) over those requests)
// H (Dk Dv + 64 Dv + 96 Dk + 128) + H / qk_group x 96 Dk floats.  `walk_values`: values a block of the walk takes, 16 or 32; the bits
// do not depend on it.
TW_EXPORT int tw_delta_chunks(float* out, const float* q, int q_stride, const float* k, int k_stride, const float* v, int v_stride,
                              const float* pre, int pre_stride, const float* write, int write_stride, const float* rate_log,
                              const float* dt_bias, float q_scale, float k_scale, float* state, long long state_stride, const int* seq_slot,
                              const int* seq_q_start, const int* seq_q_len, int n_seqs, int H, int Dk, int Dv, int qk_group, int min_len,
                              int max_q_len, int write_state, int walk_values, float* scratch, int chunks, cudaStream_t stream) {
    if (n_seqs <= 0 || H <= 0 || max_q_len <= 0) return 0;
    auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (Dk != DK || (Dk != 64 && Dk != 128) || (Dv != 64 && Dv != 128) || min_len < 1 || qk_group <= 0 || H % qk_group || (q_stride & 3)
        || (k_stride & 3) || !a16(q) || !a16(k) || !a16(scratch) || !pre || !write || !rate_log || !dt_bias || chunks < 1
        || (reinterpret_cast<uintptr_t>(out) & 7) || n_seqs > 65535 || H > 65535 || (walk_values != 16 && walk_values != 32))
        return (int)cudaErrorInvalidValue;
    DcArgs a;
    a.out = out; a.q = q; a.k = k; a.v = v; a.q_stride = q_stride; a.k_stride = k_stride; a.v_stride = v_stride;
    a.pre = pre; a.pre_stride = pre_stride; a.write = write; a.write_stride = write_stride; a.rate_log = rate_log; a.dt_bias = dt_bias;
    a.q_scale = q_scale; a.k_scale = k_scale; a.state = state; a.state_stride = state_stride;
    a.seq_slot = seq_slot; a.seq_q_start = seq_q_start; a.seq_q_len = seq_q_len;
    a.n_seqs = n_seqs; a.H = H; a.qk_group = qk_group; a.min_len = min_len; a.write_state = write_state;
    const size_t n = (size_t)chunks * H;
    a.before = scratch;
    a.u = a.before + n * Dk * Dv;
    a.w = (bf16*)(a.u + n * L * Dv);
    a.decay = (float2*)(a.w + n * 3 * L * Dk);
    a.keys = (bf16*)(a.decay + n * L);
#if TW_DK == 64 || TW_DK == 128
    return Dv == 128 ? launch_delta<128>(a, max_q_len, walk_values, stream) : launch_delta<64>(a, max_q_len, walk_values, stream);
#else
    return (int)cudaErrorInvalidValue;
#endif
}
