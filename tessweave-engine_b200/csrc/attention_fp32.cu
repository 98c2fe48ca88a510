// Paged causal attention of prompt portions in 32 bits: tiles of queries against tiles of keys.
//
// The same arithmetic as attention_generic.cu -- fp32 scores, expf, fp32 online softmax and sums, nothing rounded in
// between -- for requests that bring two tokens or more; that kernel keeps the rows of requests that bring one.
//
// What bounds it: the fp32 multiply-add units and shared memory.  The row kernel reads every key and value once per
// (token, head) from L2 and spends a warp reduction on every score.  Portions of 777, 1,000 and 37
// tokens, 14 heads of 64 on 2 key/value heads: 1,995 us by rows, 167 us by tiles (12 heads of 128, 2,048 tokens: 4,817 and
// 516).  ncu of the first: FMA pipe 46 % of its active cycles, shared-memory wavefronts 68 %, 16 warps per SM.
// A block owns 64 (token, head) rows of one key/value head, the heads of a group side by side, so a key tile of 64 that
// was copied once serves all of them.  The threads form a grid, TXN along the keys; a thread holds the scores of
// RPT rows x CPT keys and of the output RPT rows x DP / TXN columns (256 threads, 16 along the keys; for small heads 128
// and 8, which read less from shared memory per multiply-add: 160 us against 192 with 16 heads of 32 and 1,400 tokens, but
// 666 against 516 with heads of 128, where four warps cannot hide a tile's latencies).  Multiply-adds are packed pairs (fma.rn.f32x2):
// pairs of neighbouring channels for the scores, pairs of neighbouring output columns for P V, for which the
// probabilities lie in shared memory twice.  64 rows and not 128: a portion of 1,000 tokens then still gives more blocks
// than the GPU has SMs, and the longest block, which sets the time, is half as long.  The latest rows of all requests,
// which have the most keys, start first.
//
// A query's sums run over tiles of 64 keys counted from position 0 and, inside a tile, in one fixed order, so they do
// not depend on how a prompt was cut or on what else is in the step.  No chain of additions is long (16 channels, one
// tile of keys): the error against 64 bits is that of the row kernel, or below it where there are many keys.
#include "attention_common.cuh"

namespace {

using tw_attn::cp_async16;
using tw_attn::cp_async_commit;
using tw_attn::cp_async_wait;

constexpr int BR = 64, BK = 64;

struct TileArgs {
    float* out; int out_stride;
    const float* q; int q_stride;
    const int* seq_q_start; const int* seq_q_len; const int* seq_kv_len; const int* seq_slot;
    const int* block_table; int table_stride;
    const float* k_cache; const float* v_cache;
    int Hq, Hkv, D, page_size, num_pages, window;
    float scale;
    const float* dist_bias; int bias_rows;
    const float* sink; const float* gate;
    int* status;
};

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
struct Whole { __device__ constexpr operator bool() const { return false; } };
struct Masked { __device__ constexpr operator bool() const { return true; } };

// DP: the head size rounded up to 32, 64 or 128; channels from D on are zeros.
template <int DP, int THREADS, int TXN>
__global__ void __launch_bounds__(THREADS) attn_fp32_tile_kernel(TileArgs a) {
    constexpr int RG = THREADS / TXN, RPT = BR / RG, CPT = BK / TXN;   // threads down the rows; rows and keys of a thread
    constexpr int QS = DP + 4, PS = 2 * BK + 4;     // padded rows: neighbouring rows start four banks apart
    constexpr int OT = DP / (4 * TXN);              // groups of four output columns per thread
    static_assert(RPT >= 1 && CPT >= 1 && OT >= 1 && THREADS >= BK, "thread grid");
    extern __shared__ __align__(16) float fsm[];
    float* qs = fsm;                                // [BR][QS]
    float* ks = qs + BR * QS;                       // [BK][QS]
    float* vs = ks + BK * QS;                       // [BK][DP]
    float* ps = vs + BK * DP;                       // [BR][PS]: every probability twice
    __shared__ long long key_at[2][BK];             // where a key's row starts in the cache; -1: no such key
    tw_grid_wait();
    tw_grid_launch_dependents();
    const int s = blockIdx.x / a.Hkv, kvh = blockIdx.x - s * a.Hkv;
    const int len = a.seq_q_len[s], group = a.Hq / a.Hkv;
    const int r0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * BR, rows = len * group;
    if (len <= 1 || r0 >= rows) return;
    const int tid = threadIdx.x, tx = tid % TXN, ty = tid / TXN;
    const int q0 = a.seq_q_start[s], p0 = a.seq_kv_len[s] - len;       // first row of the request, its position
    const int* table = a.block_table + (size_t)a.seq_slot[s] * a.table_stride;
    const int t_first = r0 / group, t_last = (min(r0 + BR, rows) - 1) / group;
    const int key_end = p0 + t_last, key_first = tw_first_key(p0 + t_first, a.window);     // the keys any row of the block sees
    const int kt0 = key_first / BK, kt1 = key_end / BK;
    // only tiles that lie wholly among the keys of every row of the block have no key that some row must not see
    const int all_first = tw_first_key(key_end, a.window), all_end = p0 + t_first;
    const int D = a.D;

    int page = -1;                                  // of key `tid` of the tile that is looked up next (threads 0 .. BK - 1)
    auto look_up = [&](int kt) {
        const int blk = (kt * BK + tid) / a.page_size;
        page = tid < BK && kt <= kt1 && blk < a.table_stride ? table[blk] : -1;
    };
    auto find_keys = [&](int kt) {                  // the rows of key tile kt in the cache, from the pages looked up a tile before
        if (tid < BK && kt <= kt1) {
            const int p = kt * BK + tid;
            long long at = -1;
            if (p >= key_first && p <= key_end) {
                if (page >= 0 && page < a.num_pages)
                    at = ((long long)page * a.Hkv + kvh) * a.page_size + p % a.page_size;
                else
                    atomicOr(a.status, TW_ERR_PAGE);
            }
            key_at[kt & 1][tid] = at;
        }
    };
    auto fetch = [&](int kt, const float* cache, float* dst, int stride) {
        constexpr int CH = DP / 4;
        if (kt <= kt1) {
            for (int e = tid; e < BK * CH; e += THREADS) {
                const int r = e / CH, c = (e - r * CH) * 4;
                const long long at = key_at[kt & 1][r];
                const bool live = at >= 0 && c < D;
                cp_async16(dst + r * stride + c, live ? cache + at * D + c : cache, live ? 16 : 0);
            }
        }
        cp_async_commit();
    };

    look_up(kt0);
    find_keys(kt0);
    look_up(kt0 + 1);
    for (int e = tid; e < BR * DP; e += THREADS) {
        const int r = e / DP, c = e - r * DP, gr = r0 + r;
        float v = 0.f;
        if (gr < rows && c < D) v = a.q[(size_t)(q0 + gr / group) * a.q_stride + (size_t)(kvh * group + gr % group) * D + c];
        qs[r * QS + c] = v;
    }
    __syncthreads();
    fetch(kt0, a.k_cache, ks, QS);
    fetch(kt0, a.v_cache, vs, DP);

    int pos[RPT], low[RPT];                         // what each of the thread's rows (ty + RG i) sees
    float m[RPT], l[RPT];
    unsigned long long o[RPT][2 * OT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int gr = r0 + ty + RG * i;
        pos[i] = gr < rows ? p0 + gr / group : -1;
        low[i] = gr < rows ? tw_first_key(pos[i], a.window) : 0;
        m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 2 * OT; ++j) o[i][j] = 0ull;
    }

    for (int kt = kt0; kt <= kt1; ++kt) {
        find_keys(kt + 1);
        look_up(kt + 2);
        cp_async_wait<1>();
        __syncthreads();                            // the tile's keys are there
        float dot[RPT][CPT];
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int j = 0; j < CPT; ++j) dot[i][j] = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < DP; c0 += 16) {       // sums of 16 channels at a time, so that no chain of additions is long
            unsigned long long s2[RPT][CPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int j = 0; j < CPT; ++j) s2[i][j] = 0ull;
#pragma unroll
            for (int c = c0; c < c0 + 16; c += 4) {
                ulonglong2 kk[CPT];
#pragma unroll
                for (int j = 0; j < CPT; ++j) kk[j] = *reinterpret_cast<const ulonglong2*>(ks + (tx + TXN * j) * QS + c);
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(qs + (ty + RG * i) * QS + c);
#pragma unroll
                    for (int j = 0; j < CPT; ++j) s2[i][j] = fma2(qq.y, kk[j].y, fma2(qq.x, kk[j].x, s2[i][j]));
                }
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int j = 0; j < CPT; ++j) {
                    const float2 two = unpack2(s2[i][j]);
                    dot[i][j] += two.x + two.y;
                }
        }
        __syncthreads();                            // nobody reads these keys any more
        fetch(kt + 1, a.k_cache, ks, QS);
        float keep[RPT];
        bool there[CPT];
#pragma unroll
        for (int j = 0; j < CPT; ++j) there[j] = key_at[kt & 1][tx + TXN * j] >= 0;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            float sc[CPT], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                const int p = kt * BK + tx + TXN * j;
                float v = dot[i][j] * a.scale;
                if (a.dist_bias && p <= pos[i])
                    v += a.dist_bias[(size_t)min(pos[i] - p, a.bias_rows - 1) * a.Hq + kvh * group + (r0 + ty + RG * i) % group];
                sc[j] = there[j] && p >= low[i] && p <= pos[i] ? v : -INFINITY;
                top = fmaxf(top, sc[j]);
            }
#pragma unroll
            for (int d = TXN / 2; d > 0; d >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
            const float m_new = fmaxf(m[i], top);
            const float base = m_new == -INFINITY ? 0.f : m_new;       // (no key so far: every exponential below is 0)
            keep[i] = expf(m[i] - base);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                const float p = expf(sc[j] - base);
                sum += p;
                *reinterpret_cast<float2*>(ps + (ty + RG * i) * PS + 2 * (tx + TXN * j)) = make_float2(p, p);
            }
            l[i] = l[i] * keep[i] + sum;
            m[i] = m_new;
        }
        cp_async_wait<1>();
        __syncthreads();                            // the probabilities and the tile's values are there
        unsigned long long n[RPT][2 * OT];          // the tile's own sums: added to the running ones once
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int j = 0; j < 2 * OT; ++j) n[i][j] = 0ull;
        auto add_values = [&](auto masked) {
#pragma unroll 4
            for (int key = 0; key < BK; key += 2) {
                ulonglong2 va[OT], vb[OT];
#pragma unroll
                for (int j = 0; j < OT; ++j) {
                    va[j] = *reinterpret_cast<const ulonglong2*>(vs + key * DP + tx * 4 + 4 * TXN * j);
                    vb[j] = *reinterpret_cast<const ulonglong2*>(vs + (key + 1) * DP + tx * 4 + 4 * TXN * j);
                }
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const ulonglong2 pp = *reinterpret_cast<const ulonglong2*>(ps + (ty + RG * i) * PS + 2 * key);
                    // (a value that a row does not see must not reach it, be it infinite or not a number)
                    const bool use_a = !masked || pp.x != 0ull, use_b = !masked || pp.y != 0ull;
#pragma unroll
                    for (int j = 0; j < OT; ++j) {
                        if (use_a) {
                            n[i][2 * j] = fma2(pp.x, va[j].x, n[i][2 * j]);
                            n[i][2 * j + 1] = fma2(pp.x, va[j].y, n[i][2 * j + 1]);
                        }
                        if (use_b) {
                            n[i][2 * j] = fma2(pp.y, vb[j].x, n[i][2 * j]);
                            n[i][2 * j + 1] = fma2(pp.y, vb[j].y, n[i][2 * j + 1]);
                        }
                    }
                }
            }
        };
        if (kt * BK >= all_first && kt * BK + BK - 1 <= all_end) add_values(Whole{});
        else add_values(Masked{});
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int j = 0; j < 2 * OT; ++j) o[i][j] = fma2(o[i][j], pack2(keep[i], keep[i]), n[i][j]);
        __syncthreads();                            // nobody reads these values and probabilities any more
        fetch(kt + 1, a.v_cache, vs, DP);
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int gr = r0 + ty + RG * i;
        float total = l[i];
#pragma unroll
        for (int d = TXN / 2; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
        if (gr >= rows) continue;
        const int head = kvh * group + gr % group;
        const size_t row = (size_t)q0 + gr / group;
        float f = 1.f;
        if (a.sink) {
            const float top = fmaxf(m[i], a.sink[head]);
            f = m[i] == -INFINITY ? 0.f : expf(m[i] - top);
            total = total * f + expf(a.sink[head] - top);
        }
        const float gate = a.gate ? a.gate[row * a.Hq + head] : 1.f;
        const bool any = total > 0.f;               // (as in the row kernel: no visible key, or a sum that is not a number, gives 0)
        const float by = any ? f / total * gate : 0.f;
        float* dst = a.out + row * a.out_stride + (size_t)head * D;
#pragma unroll
        for (int j = 0; j < OT; ++j) {
            const float2 x = unpack2(o[i][2 * j]), y = unpack2(o[i][2 * j + 1]);
            const float v[4] = {x.x * by, x.y * by, y.x * by, y.y * by};
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (tx * 4 + 4 * TXN * j + c < D) dst[tx * 4 + 4 * TXN * j + c] = any ? v[c] : 0.f;
        }
    }
}

template <int DP, int THREADS, int TXN>
int launch_tiles(const TileArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
    constexpr size_t smem = ((size_t)(BR + BK) * (DP + 4) + (size_t)BK * DP + (size_t)BR * (2 * BK + 4)) * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(attn_fp32_tile_kernel<DP, THREADS, TXN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int blocks = (int)(((long long)max_q_len * (a.Hq / a.Hkv) + BR - 1) / BR);
    return tw_launch(attn_fp32_tile_kernel<DP, THREADS, TXN>, dim3(a.Hkv * n_seqs, blocks), dim3(THREADS), smem, stream, 1, a);
}

}  // namespace

// Rows of requests with seq_q_len of 2 or more (the others are left alone).  q, out: fp32 rows, head h at column h * D;
// pages [num_pages, Hkv, page_size, D] on 16-byte boundaries; D a multiple of 4 up to 128, keys and values alike.
TW_EXPORT int tw_attn_fp32_tiles(float* out, int out_stride, const float* q, int q_stride, const int* seq_q_start,
                                 const int* seq_q_len, const int* seq_kv_len, const int* seq_slot, const int* block_table,
                                 int table_stride, const float* k_cache, const float* v_cache, int n_seqs, int max_q_len, int Hq,
                                 int Hkv, int D, int page_size, int num_pages, int window, float scale, const float* dist_bias,
                                 int bias_rows, const float* sink, const float* gate, int* status, cudaStream_t stream) {
    if (n_seqs <= 0 || max_q_len <= 0) return 0;
    if (dist_bias && bias_rows <= 0) return (int)cudaErrorInvalidValue;
    if (D <= 0 || D > 128 || (D & 3) || Hkv <= 0 || Hq % Hkv || page_size <= 0 || (long long)max_q_len * (Hq / Hkv) > 65535ll * BR
        || (reinterpret_cast<uintptr_t>(k_cache) & 15) || (reinterpret_cast<uintptr_t>(v_cache) & 15))
        return (int)cudaErrorInvalidValue;
    TileArgs a;
    a.out = out; a.out_stride = out_stride; a.q = q; a.q_stride = q_stride;
    a.seq_q_start = seq_q_start; a.seq_q_len = seq_q_len; a.seq_kv_len = seq_kv_len; a.seq_slot = seq_slot;
    a.block_table = block_table; a.table_stride = table_stride; a.k_cache = k_cache; a.v_cache = v_cache;
    a.Hq = Hq; a.Hkv = Hkv; a.D = D; a.page_size = page_size; a.num_pages = num_pages; a.window = window; a.scale = scale;
    a.dist_bias = dist_bias; a.bias_rows = bias_rows; a.sink = sink; a.gate = gate; a.status = status;
    if (D <= 32) return launch_tiles<32, 128, 8>(a, n_seqs, max_q_len, stream);
    if (D <= 64) return launch_tiles<64, 256, 16>(a, n_seqs, max_q_len, stream);
    return launch_tiles<128, 256, 16>(a, n_seqs, max_q_len, stream);
}
