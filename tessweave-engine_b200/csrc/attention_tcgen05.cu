// Paged causal attention for prompt portions on the 5th-generation tensor cores, for one head
// size (compile with -DTW_HEAD_DIM=64 or 128; values of another size: -DTW_V_DIM=32, 64 or 128).
//
// A block serves up to 256 rows of one (request, key/value head), a row being a (token, query
// head of the group) pair, as two tiles of 128 rows, and walks the request's keys in tiles of
// 128.  Per key tile and row tile:
//     S = Q K^T        tcgen05.mma, both operands K-major in shared memory, S (fp32) in tensor memory
//     P = 2^(S c - m)  four warps, one row (one TMEM lane) per thread: tcgen05.ld, fp32 maximum
//                      and sum, P rounded to bf16 and stored over S in tensor memory (tcgen05.st)
//     O += P V         tcgen05.mma with P as the operand in tensor memory and V read "MN-major"
//                      straight from the page layout [key][d]; O (fp32) stays in tensor memory
//                      for the whole walk
// The two row tiles alternate, so the tensor cores work on one while the softmax warps work on
// the other.  Keys and values travel by TMA (cp.async.bulk.tensor.2d, no multicast), one box
// per page and 64 columns of d, into the swizzled layout the MMAs read; a warp each
// issues them.  Another warp issues every MMA.
//
// What bounds it: a key tile takes 3,600 cycles of which the tensor pipe is busy for 2,048; a tile's chain is its softmax
// (1,650: 1,024 for its exponentials), its products (1,250) and the hand-overs between the two, and the longest blocks of a
// prompt run through 16 such tiles one behind the other.  So what shortens the chain counts: exponentials that do not wait
// for the tile's own maximum, one wait and no commits beside the products', copies from two warps, query rows whose loads
// hang on no condition (8,500 -> 2,500 cycles), results written by whole rows (5,300 -> 2,400), masks off the path that all
// tiles take (the first tile of a block fetches its instructions: 6,600 -> 3,000).  us before and after: 2,048 tokens of
// 28 heads of 128 50.4 and 42.4, of 14 heads of 64 39.3 and 37.2; 777 + 300 + 201 tokens of 12 heads behind 0, 512 and 1,030
// keys 30.9 and 27.0; 400 tokens of 28 heads 21.5 and 16.5; 301 + 182 of 40 heads 25.2 and 23.4.
//
// O is only rescaled when a row's maximum grows by more than 2^8 (the sums carry the same
// stale maximum, so the quotient is exact); rows of values beyond the request's last key are
// zeroed in shared memory, so stale page contents cannot reach a product.  Pages that lie wholly before the first key
// any row of the block sees (a window or a chunk has moved on, and the pages may have been given back) are not read:
// their boxes are asked for beyond the end of the cache, which the copy engine answers with zeros.
//
//   score = (q . k) * scale,  visible iff  tw_first_key(position, window) <= p <= position
//   (`gate`: fp32 [rows][Hq] or null; head h's output is multiplied by its entry)
// Reference: flow_engine/model.py:193-200 (the reference calls a library's attention here).
//
// Every wait on an mbarrier is bounded; a wait that runs out sets TW_ERR_WAIT in the status
// word, every role stops, the block waits (bounded) for its copies in flight, frees its tensor
// memory and returns.
#include "tcgen05_softmax.cuh"

#ifndef TW_HEAD_DIM
#define TW_HEAD_DIM 128
#endif
#ifndef TW_V_DIM
#define TW_V_DIM TW_HEAD_DIM
#endif

namespace {

using namespace tc5;

constexpr int D = TW_HEAD_DIM;
static_assert(D == 64 || D == 128, "the tcgen05 attention is built for head sizes 64 and 128");

constexpr int BM = 128;                       // rows of a query tile = TMEM lanes
constexpr int NQ = 2;                         // query tiles per block
constexpr int BN = 128;                       // keys per tile
constexpr int DV = TW_V_DIM;
static_assert(DV == 32 || DV == 64 || DV == 128, "the tcgen05 attention is built for value sizes 32, 64 and 128");
constexpr int KB = D / 64;                    // 64-column blocks of a row of q or k
constexpr int VB = (DV + 63) / 64;            // 64-column blocks of a row of v (32 values: the copy fills the rest with zeros)
constexpr int BLK = 128 * 128;                // bytes of a [128 rows][64 columns] swizzled block
constexpr int KV_STAGES = D == 64 && DV <= 64 ? 4 : 2;   // K and V have rings of their own
constexpr int Q_BYTES = NQ * KB * BLK;
constexpr int K_STAGE_BYTES = KB * BLK, V_STAGE_BYTES = VB * BLK;
constexpr int SMEM_TILES = Q_BYTES + KV_STAGES * (K_STAGE_BYTES + V_STAGE_BYTES);
constexpr int SMEM = SMEM_TILES + 1024 /* alignment slack */ + 256 /* barriers */;
constexpr int THREADS = 384;                  // warps 0-3 / 4-7: softmax of tile 0 / 1, warps 8 / 9: copies of K / V, warp 10: every MMA; warp 11 helps with the query rows and fills up the group that gives registers back
constexpr int K_WARP = 8, V_WARP = 9, MMA_WARP = 10;
// A softmax thread holds a row of 128 scores; the others need few registers.  256 x 200 + 128 x 104 = 384 x 168, which the
// block is launched with.
constexpr int SOFTMAX_REGS = 200, OTHER_REGS = 104, LAUNCH_REGS = 168;
static_assert(256 * SOFTMAX_REGS + 128 * OTHER_REGS <= THREADS * LAUNCH_REGS, "registers of the block");
constexpr int TMEM_COLS = 512;                // S of both tiles (2 x 128 columns; P over its first 64), O of both tiles (2 x DV)
constexpr int O_COL = 256;
constexpr float RESCALE_THRESHOLD = 8.f;      // log2 units
#define NEG_INF (-INFINITY)

// -DTW_TRACE: block (0, 0, 0) records clock64() at the hand-over points of its roles, for a
// timeline of one block (tw_attn_tc5_trace_ptr gives the buffer).  Off in the product.
#ifdef TW_TRACE
constexpr int TRACE_SLOTS = 12, TRACE_TILES = 80, TRACE_ROLES = 12;     // a role: a softmax warp, 8 the MMA warp, 9 and 10 the copies, 11 the block
__device__ long long g_trace[TRACE_ROLES * TRACE_TILES * TRACE_SLOTS];
#define TW_TRACE_AT(role, tile, slot)                                                              \
    do {                                                                                           \
        if (blockIdx.x == 0 && blockIdx.y == 0 && (tile) < TRACE_TILES)         \
            g_trace[((role) * TRACE_TILES + (tile)) * TRACE_SLOTS + (slot)] = clock64();           \
    } while (0)
#else
#define TW_TRACE_AT(role, tile, slot) do {} while (0)
#endif

__global__ void __launch_bounds__(THREADS, 1)
attn_prefill_tc5_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        bf16* __restrict__ out, int out_stride, const bf16* __restrict__ q, int q_stride,
                        const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                        const int* __restrict__ seq_kv_len, const int* __restrict__ seq_slot,
                        const int* __restrict__ block_table, int table_stride, int Hq, int Hkv, int page_size,
                        int num_pages, int window, float scale_log2e, int skip_single, const float* __restrict__ gate,
                        int* status, int n_seqs, int* word) {
    extern __shared__ unsigned char smem_raw[];
    TW_TIMELINE_SCOPE(TW_K_ATTN_PREFILL);
    tw_grid_wait();
    // The decode attention of the same step writes other rows: it may run beside this kernel, on the SMs that have no block of it.
    if (skip_single) {
        tw_say_ready(word);
        tw_launch_dependents_now();
    }
    if (threadIdx.x == 0) TW_TRACE_AT(11, 0, 5);
    TW_TIMELINE_MARK();
    // Blocks start in the order of blockIdx.x, and a block's work grows with the position of its rows: x counts
    // (row tile, key/value head) with the head fastest and the last row tile first, so that the longest blocks of
    // all heads start first and the short ones fill the gaps (with the head as blockIdx.y, the long blocks of
    // the last heads started late: 78 us against 58 us for 2,048 tokens).
    const int G = Hq / Hkv, kvh = (int)blockIdx.x % Hkv;
    int s = blockIdx.y, xt = (int)blockIdx.x / Hkv, q_len = 0;
    auto served = [&](int len) { return len <= 0 || (skip_single && len == 1) ? 0 : len; };
    auto tiles_of = [&](int len) { return (len * G + NQ * BM - 1) / (NQ * BM); };
    if (n_seqs > 0) {
        // the grid holds the row tiles of all requests one behind the other: which request's is this one?  (With a grid of
        // every request's largest number of tiles, 1,440 of 1,520 blocks of a step of 2 prompts and 30 single tokens had
        // nothing to do, one per SM at a time, and the decode attention could not start beside this kernel for 18 us.)
        const int lane = threadIdx.x & 31;
        int before = 0;
        s = -1;
        for (int r0 = 0; r0 < n_seqs && s < 0; r0 += 32) {
            const int len = r0 + lane < n_seqs ? served(seq_q_len[r0 + lane]) : 0, mine = tiles_of(len);
            int upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += below;
            }
            const uint32_t beyond = __ballot_sync(0xffffffffu, xt < before + upto);
            if (beyond) {
                const int at = __ffs(beyond) - 1;
                s = r0 + at;
                q_len = __shfl_sync(0xffffffffu, len, at);
                xt -= before + __shfl_sync(0xffffffffu, upto - mine, at);
            } else {
                before += __shfl_sync(0xffffffffu, upto, 31);
            }
        }
        if (s < 0) return;
    } else {
        q_len = served(seq_q_len[s]);
    }
    const int rows_total = q_len * G;
    const int mtiles = tiles_of(q_len);
    if (xt >= mtiles) return;
    const int row0 = (mtiles - 1 - xt) * (NQ * BM);                  // the rows with the most keys first
    const int kv_len = seq_kv_len[s];
    const int pos0 = kv_len - q_len;                                 // position of the first token of this portion
    const int n0 = seq_q_start[s];
    const int* table = block_table + (size_t)seq_slot[s] * table_stride;
    const int row_end = min(rows_total, row0 + NQ * BM);
    const int nq = row_end - row0 > BM ? 2 : 1;
    const int pos_first = pos0 + row0 / G, pos_last = pos0 + (row_end - 1) / G;
    const int lo_block = tw_first_key(pos_first, window);             // no row of the block sees a key before this one
    const int j_begin = lo_block / BN;
    const int ntiles = pos_last / BN + 1 - j_begin;
    const int tail_rows = max(0, (j_begin + ntiles) * BN - kv_len);  // rows of the last tile that hold no key

    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* q_s = tiles;                                      // [NQ][KB][128 rows][128 B]
    unsigned char* k_s = q_s + Q_BYTES;                              // [KV_STAGES][KB][128 keys][128 B]
    unsigned char* v_s = k_s + KV_STAGES * K_STAGE_BYTES;            // [KV_STAGES][VB][128 keys][128 B]
    uint64_t* k_first = reinterpret_cast<uint64_t*>(tiles + SMEM_TILES);   // K of the first tile has landed
    uint64_t* v_last = k_first + 1;                                  // V of the last tile has (where rows of it are zeroed)
    // Of tile i's products P V and the next tile's S: P of query tile 0 is written, V of tile i and K of tile i + 1 have landed.
    // One barrier for all three, since each wait costs the thread that issues the MMAs some 170 cycles even if it is over.
    uint64_t* ready = v_last + 1;                                    // [stage]
    uint64_t* p_full = ready + KV_STAGES;                            // P of query tile 1 is written, S read, O rescaled
    // [query tile][stage]: S of the tile is complete, its P V products have retired.  The producers take them as the sign that
    // a stage is free as well (commits to barriers of their own took 200 cycles each).
    uint64_t* s_full = p_full + 1;
    uint64_t* o_done = s_full + NQ * KV_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + NQ * KV_STAGES);
    volatile int* aborted = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(k_first, 1);
        mbar_init(v_last, 1);
        mbar_init(p_full, BM / 32);
        for (int i = 0; i < KV_STAGES; ++i) mbar_init(&ready[i], BM / 32 + 2);
        for (int i = 0; i < NQ * KV_STAGES; ++i) { mbar_init(&s_full[i], 1); mbar_init(&o_done[i], 1); }
        *aborted = 0;
        mbar_fence_init();
    }
    // A producer's work for key tile i: one TMA box per page and 64 columns of d; lane b owns box b of the tile (one lane
    // that issues them all takes 160 cycles a copy, eight lanes 100).  Keys and values have a warp each: the 32 copies of
    // both take one warp as long as the products of the tile take.  False if a wait ran out.
    const int box_rows = min(page_size, BN);
    const int boxes = BN / box_rows;
    auto issue_tile = [&](int i, const CUtensorMap* map, unsigned char* ring, int stage_bytes, int blocks, uint64_t* full, uint64_t* freed) -> bool {
        const int st = i % KV_STAGES;
        int row_coord = -1;
        if (lane < boxes) {
            const int key0 = (j_begin + i) * BN + lane * box_rows;
            if (key0 < kv_len && key0 + box_rows <= lo_block) {
                row_coord = num_pages * Hkv * page_size;              // beyond the cache: zeros
            } else if (key0 < kv_len) {
                const int blk = key0 / page_size;
                const int page = blk < table_stride ? table[blk] : -1;
                if (page < 0 || page >= num_pages) atomicOr(status, TW_ERR_PAGE);
                else row_coord = (page * Hkv + kvh) * page_size + (key0 - blk * page_size);
            }
        }
        const uint32_t box_bytes = (uint32_t)__popc(__ballot_sync(0xffffffffu, row_coord >= 0)) * box_rows * 128;
        int ok = 1;
        if (lane == 0) {
            ok = (!*aborted && (i < KV_STAGES || mbar_wait(&freed[st], (i / KV_STAGES - 1) & 1, status))) ? 1 : 0;
            if (ok) mbar_expect_tx(full, box_bytes * blocks); else *aborted = 1;
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) return false;
        if (lane == 0) TW_TRACE_AT(ring == k_s ? 9 : 10, i, 0);
        if (row_coord >= 0) {
            for (int b = 0; b < blocks; ++b)
                tma_load_2d(ring + st * stage_bytes + b * BLK + lane * box_rows * 128, map, full, b * 64, row_coord);
        }
        return true;
    };
    // the barrier that tells of tile i's keys, of its values
    auto k_full = [&](int i) { return i == 0 ? k_first : &ready[(i - 1) % KV_STAGES]; };
    auto v_full = [&](int i) { return i == ntiles - 1 && tail_rows ? v_last : &ready[i % KV_STAGES]; };
    auto issue_k = [&](int i) { return issue_tile(i, &map_k, k_s, K_STAGE_BYTES, KB, k_full(i), s_full + (nq - 1) * KV_STAGES); };
    auto issue_v = [&](int i) { return issue_tile(i, &map_v, v_s, V_STAGE_BYTES, VB, v_full(i), o_done + (nq - 1) * KV_STAGES); };
    // The first key and value tiles need nothing of what follows: their producers ask for them as soon as the barriers
    // stand, and the other warps bring the query rows in meanwhile.
    __syncthreads();
    if (warp == MMA_WARP) tmem_alloc(tmem_slot, TMEM_COLS);
    int issued = 0;
    if (warp == K_WARP) {
        while (issued < ntiles && issued < KV_STAGES && issue_k(issued)) ++issued;
    } else if (warp == V_WARP) {
        while (issued < ntiles && issued < KV_STAGES && issue_v(issued)) ++issued;
    }

    // the block's query rows into shared memory, in the swizzled K-major layout (rows beyond the portion are zero).
    // All of a thread's loads are issued before the first store: one round trip to L2, not thirteen in a row
    // (which was 9 of the 13 us a block spent outside its key tiles).
    if (warp != K_WARP && warp != V_WARP) {
        constexpr int Q_ITEMS = NQ * BM * (D / 8);
        constexpr int Q_THREADS = THREADS - 64;                          // every warp but the producers
        constexpr int Q_PER_THREAD = (Q_ITEMS + Q_THREADS - 1) / Q_THREADS;
        constexpr int STEP = Q_THREADS / (D / 8);                        // rows between two of a thread's loads: its columns stay
        static_assert(Q_THREADS % (D / 8) == 0, "a thread keeps its columns");
        const int first = (warp < K_WARP ? warp : warp - 2) * 32 + lane;
        const int c = first % (D / 8), rr0 = first / (D / 8), step_t = STEP / G, step_h = STEP - step_t * G;
        int t = (row0 + rr0) / G, hg = row0 + rr0 - t * G;
        const bf16* src = q + (size_t)n0 * q_stride + (size_t)kvh * G * D + c * 8;
        uint4 vals[Q_PER_THREAD];
#pragma unroll
        for (int j = 0; j < Q_PER_THREAD; ++j) {
            // no load hangs on a condition (a row behind the last reads the last token's): all of them are under way at once
            vals[j] = *reinterpret_cast<const uint4*>(src + (size_t)min(t, q_len - 1) * q_stride + hg * D);
            t += step_t; hg += step_h;
            if (hg >= G) { hg -= G; ++t; }
        }
#pragma unroll
        for (int j = 0; j < Q_PER_THREAD; ++j) {
            const int rr = rr0 + j * STEP;
            if (rr < NQ * BM) {
                const int x = rr / BM, rt = rr - x * BM;
                if (row0 + rr >= rows_total) vals[j] = make_uint4(0u, 0u, 0u, 0u);
                *reinterpret_cast<uint4*>(q_s + (x * KB + (c >> 3)) * BLK + rt * 128 + (((c & 7) ^ (rt & 7)) << 4)) = vals[j];
            }
        }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0) TW_TRACE_AT(11, 0, 6);

    if (warp >= K_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OTHER_REGS));
        if (warp < MMA_WARP) {
        // ---- producers: the remaining tiles, each as soon as its stage is free
        if (warp == K_WARP) {
            while (issued < ntiles && !*aborted && issue_k(issued)) ++issued;
        } else {
            while (issued < ntiles && !*aborted && issue_v(issued)) ++issued;
        }
        if (warp == K_WARP && issued == ntiles && ntiles > 0 && lane == 0) {
            // no keys behind the last tile's: its barrier gets the arrival alone, once the phase before is over there
            if (ntiles < KV_STAGES || mbar_wait(&s_full[(nq - 1) * KV_STAGES + ntiles % KV_STAGES], (ntiles / KV_STAGES - 1) & 1, status))
                mbar_arrive(&ready[(ntiles - 1) % KV_STAGES]);
            else *aborted = 1;
        }
        if (warp == V_WARP && tail_rows && issued == ntiles) {
            // The last tile reaches past the request's last key.  What its value rows hold there (the rest
            // of a page, or whatever the stage held before) must not reach a product, since 0 x NaN is NaN:
            // zero them once the copies have landed, then tell the MMA thread.
            const int last = ntiles - 1;
            if (mbar_wait(v_last, 0, status)) {
                unsigned char* vt = v_s + (last % KV_STAGES) * V_STAGE_BYTES;
                for (int idx = lane; idx < tail_rows * VB * 8; idx += 32) {
                    const int r = BN - tail_rows + idx / (VB * 8), rest = idx % (VB * 8);
                    *reinterpret_cast<uint4*>(vt + (rest >> 3) * BLK + r * 128 + ((rest & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ready[last % KV_STAGES]);
            } else {
                *aborted = 1;
            }
        }
        if (*aborted && lane == 0) {
            // wait (bounded) for the copies already in flight, so that none lands after the block has gone
            for (int i = max(0, issued - KV_STAGES); i < issued; ++i) {
                if (warp == K_WARP) mbar_wait(k_full(i), i == 0 ? 0 : ((i - 1) / KV_STAGES) & 1, status);
                else mbar_wait(v_full(i), i == ntiles - 1 && tail_rows ? 0 : (i / KV_STAGES) & 1, status);
            }
        }
        } else {
        // ---- tensor cores: lane 0 issues every MMA of the block.  The tensor pipe runs dry as soon as
        // this thread does anything else, so it waits once for all that a group of MMAs needs.  (A thread for each
        // query tile was no faster: left alone the tiles fall into step, both in their softmax at a time and both at the
        // tensor pipe at a time, 5,080 cycles a key tile; taking turns, 3,700, they are as fast as with one thread.)
        if (warp == MMA_WARP && lane == 0 && ntiles > 0) {
            const uint32_t idesc_s = instr_desc(BN), idesc_o = instr_desc(DV, true);
            // Descriptors are built once; per MMA only a constant is added to the address field (a thread
            // that computes a descriptor from scratch before each MMA issues them slower than they execute).
            const uint64_t q_desc = smem_desc(q_s, 0), k_desc = smem_desc(k_s, 0), v_desc = smem_desc_mn_major(v_s, BLK);
            auto issue_s = [&](int x, int i) {
                const uint64_t kd = k_desc + (uint64_t)((i % KV_STAGES) * (K_STAGE_BYTES >> 4));
                const uint64_t qd = q_desc + (uint64_t)(x * KB * (BLK >> 4));
#pragma unroll
                for (int kb = 0; kb < KB; ++kb)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base + x * BN, qd + (uint64_t)(kb * (BLK >> 4) + k * 2), kd + (uint64_t)(kb * (BLK >> 4) + k * 2),
                                  idesc_s, (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(&s_full[x * KV_STAGES + i % KV_STAGES]);
            };
            auto issue_o = [&](int x, int i) {
                const uint64_t vd = v_desc + (uint64_t)((i % KV_STAGES) * (V_STAGE_BYTES >> 4));
#pragma unroll
                for (int k = 0; k < BN / 16; ++k)
                    umma_bf16_ts(tmem_base + O_COL + x * DV, tmem_base + x * BN + k * 8, vd + (uint64_t)(k * (2048 >> 4)),
                                 idesc_o, (i > 0 || k > 0) ? 1u : 0u);
                umma_commit(&o_done[x * KV_STAGES + i % KV_STAGES]);
            };
            bool ok = mbar_wait(k_first, 0, status);
            if (ok) {
                tc_fence_after();
                for (int x = 0; x < nq; ++x) issue_s(x, 0);
            }
            for (int i = 0; ok && i < ntiles; ++i) {
                for (int x = 0; ok && x < nq; ++x) {
                    TW_TRACE_AT(8, i, x * 6 + 1);
                    ok = x == 0 ? mbar_wait(&ready[i % KV_STAGES], (i / KV_STAGES) & 1, status) : mbar_wait(p_full, i & 1, status);
                    if (!ok) break;
                    TW_TRACE_AT(8, i, x * 6 + 2);
                    tc_fence_after();
                    issue_o(x, i);
                    if (i + 1 < ntiles) issue_s(x, i + 1);
                    TW_TRACE_AT(8, i, x * 6 + 4);
                }
            }
            if (!ok) *aborted = 1;
        }
        __syncwarp();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SOFTMAX_REGS));
        if (warp / 4 < nq) {
        // ---- softmax: thread = row rt of tile x = TMEM lane rt
        const int x = warp / 4;
        const int quarter = warp & 3;                        // the TMEM lanes this warp may touch
        const int rt = quarter * 32 + lane;
        const int r = row0 + x * BM + rt;
        const bool valid = r < rows_total;
        const int t = valid ? r / G : (rows_total - 1) / G;
        const int pos = pos0 + t;
        const int lo = tw_first_key(pos, window);
        const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const uint32_t s_addr = lane_addr + x * BN, o_addr = lane_addr + O_COL + x * DV;
        float m_used = NEG_INF, l = 0.f;
        bool ok = true;
        for (int i = 0; i < ntiles; ++i) {
            const int kbase = (j_begin + i) * BN;
            if (lane == 0) TW_TRACE_AT(warp, i, 0);
            ok = !*aborted && mbar_wait(&s_full[x * KV_STAGES + i % KV_STAGES], (i / KV_STAGES) & 1, status);
            if (!ok) break;
            if (lane == 0) TW_TRACE_AT(warp, i, 1);
            tc_fence_after();
            uint32_t v[2][32], packed[BN / 2];
            if (!__all_sync(0xffffffffu, kbase + BN - 1 <= pos && kbase >= lo)) {
                // keys that the row does not see: -infinity in tensor memory, so that what follows, which every tile runs
                // through, need not ask (its instructions are fetched anew by every block's first tile)
#pragma unroll 1
                for (int c = 0; c < BN; c += 32) {
                    tmem_ld32_nowait(s_addr + c, v[0]);
                    tmem_wait_ld_of(v[0]);
#pragma unroll
                    for (int e = 0; e < 32; ++e)
                        if ((unsigned)(kbase + c + e - lo) > (unsigned)(pos - lo)) v[0][e] = __float_as_uint(NEG_INF);
                    tmem_st32_nowait(s_addr + c, v[0]);
                }
                tmem_wait_st();
            }
            // four independent chains of three-input maxima
            auto maxima = [&](float (&mx)[4], const uint32_t (&v)[32]) {
#pragma unroll
                for (int c = 0; c < 32; c += 8)
#pragma unroll
                    for (int k = 0; k < 4; ++k) mx[k] = max3(mx[k], __uint_as_float(v[c + 2 * k]), __uint_as_float(v[c + 2 * k + 1]));
            };
            auto largest = [&](const float (&mx)[4]) {      // scale > 0: the maximum commutes with it
                return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2e;
            };
            if (i == 0) {
                float mx[4] = {NEG_INF, NEG_INF, NEG_INF, NEG_INF};
#pragma unroll 1
                for (int c = 0; c < BN; c += 32) {
                    tmem_ld32_nowait(s_addr + c, v[0]);
                    tmem_wait_ld_of(v[0]);
                    maxima(mx, v[0]);
                }
                m_used = largest(mx);
            }
            // The exponentials are taken against the maximum as it was, 32 scores at a time while the next 32 come in, and the
            // tile's own maximum is found beside them: waiting for it first took 400 of the 1,830 cycles between S and P.  Only
            // where a row's maximum has grown by more than the threshold (the first tiles of a request) are they taken again.
            bool rescale = false;
            float factor = 1.f, sum;
            while (true) {
                float mx[4] = {NEG_INF, NEG_INF, NEG_INF, NEG_INF};
                const float neg_mu = m_used == NEG_INF ? 0.f : -m_used;
                // p = 2^(s c - m) two at a time (packed fp32 multiply-add and add), four independent sums of pairs
                float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                tmem_ld32_nowait(s_addr, v[0]);
#pragma unroll
                for (int c = 0; c < BN; c += 32) {
                    uint32_t (&w)[32] = v[(c >> 5) & 1];
                    tmem_wait_ld_of(w);
                    if (c + 32 < BN) tmem_ld32_nowait(s_addr + c + 32, v[((c >> 5) & 1) ^ 1]);
                    maxima(mx, w);
#pragma unroll
                    for (int e8 = 0; e8 < 32; e8 += 8) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            float2 e = fma2(__uint_as_float(w[e8 + 2 * k]), __uint_as_float(w[e8 + 2 * k + 1]), scale_log2e, neg_mu);
                            e.x = ex2(e.x);
                            e.y = ex2(e.y);
                            acc[k] = add2(acc[k], e);
                            packed[((c + e8) >> 1) + k] = pack_bf16(e.x, e.y);
                        }
                    }
                }
                sum = ((acc[0].x + acc[0].y) + (acc[1].x + acc[1].y)) + ((acc[2].x + acc[2].y) + (acc[3].x + acc[3].y));
                const float mt = largest(mx);
                const bool grown = mt > m_used + RESCALE_THRESHOLD;
                if (!__any_sync(0xffffffffu, grown)) break;
                rescale = true;
                if (grown) {
                    factor = m_used == NEG_INF ? 0.f : ex2(m_used - mt);
                    m_used = mt;
                }
            }
            if (lane == 0) TW_TRACE_AT(warp, i, 2);
            l = l * factor + sum;
            if (i > 0 && rescale) {
                // P V of the tile before has retired (it was issued before the S just read): O is complete up to it
                ok = mbar_wait(&o_done[x * KV_STAGES + (i - 1) % KV_STAGES], ((i - 1) / KV_STAGES) & 1, status);
                if (!ok) break;
                tc_fence_after();
                {
#pragma unroll
                    for (int c = 0; c < DV; c += 32) {
                        uint32_t o[32];
                        tmem_ld32_nowait(o_addr + c, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * factor);
                        tmem_st32_nowait(o_addr + c, o);
                    }
                    tmem_wait_st();
                }
            }
            if (lane == 0) TW_TRACE_AT(warp, i, 3);
            // P over the first 64 columns of S: the whole row of S is in registers by now
            tmem_st32_nowait(s_addr, packed);
            tmem_st32_nowait(s_addr + 32, packed + 32);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(x == 0 ? &ready[i % KV_STAGES] : p_full);      // one arrival per warp: 128 arrivals on one barrier take 450 cycles
            if (lane == 0) TW_TRACE_AT(warp, i, 4);
        }
        if (ok && ntiles > 0) ok = mbar_wait(&o_done[x * KV_STAGES + (ntiles - 1) % KV_STAGES], ((ntiles - 1) / KV_STAGES) & 1, status);
        if (lane == 0) TW_TRACE_AT(warp, TRACE_TILES - 1, 0);
        if (!ok) {
            *aborted = 1;
        } else if (ntiles > 0) {
            tc_fence_after();
            float inv = l > 0.f ? 1.f / l : 0.f;
            if (gate && valid) inv *= __ldg(gate + (size_t)(n0 + t) * Hq + kvh * G + (r - t * G));
            const long long at = (long long)(n0 + t) * out_stride + (long long)(kvh * G + (r - t * G)) * DV;
            if constexpr (DV <= D) {
                // through the tile's query rows, which nobody reads any more, so that a warp writes whole rows: with a row per
                // thread, 16 bytes at a time, the stores of a block took 5,000 cycles
                unsigned char* stage = q_s + x * KB * BLK + quarter * 32 * (DV * 2);
#pragma unroll
                for (int c = 0; c < DV; c += 32) {
                    uint32_t o[32];
                    tmem_ld32_nowait(o_addr + c, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int k = 0; k < 32; k += 8) {
                        uint4 w;
                        w.x = pack_bf16(__uint_as_float(o[k]) * inv, __uint_as_float(o[k + 1]) * inv);
                        w.y = pack_bf16(__uint_as_float(o[k + 2]) * inv, __uint_as_float(o[k + 3]) * inv);
                        w.z = pack_bf16(__uint_as_float(o[k + 4]) * inv, __uint_as_float(o[k + 5]) * inv);
                        w.w = pack_bf16(__uint_as_float(o[k + 6]) * inv, __uint_as_float(o[k + 7]) * inv);
                        *reinterpret_cast<uint4*>(stage + lane * (DV * 2) + ((((c + k) >> 3) ^ (lane & (DV / 8 < 8 ? DV / 8 - 1 : 7))) << 4)) = w;
                    }
                }
                __syncwarp();
                constexpr int LANES = DV / 8, ROWS = 32 / LANES;         // lanes a row, rows a store
                const uint32_t live = __ballot_sync(0xffffffffu, valid);
                const int c = lane % LANES;
#pragma unroll
                for (int j = 0; j < 32 / ROWS; ++j) {
                    const int row = j * ROWS + lane / LANES;
                    const long long dst = __shfl_sync(0xffffffffu, at, row);
                    const uint4 w = *reinterpret_cast<const uint4*>(stage + row * (DV * 2) + ((c ^ (row & (LANES < 8 ? LANES - 1 : 7))) << 4));
                    if ((live >> row) & 1) *reinterpret_cast<uint4*>(out + dst + c * 8) = w;
                }
            } else {
                bf16* orow = out + at;
#pragma unroll
                for (int c = 0; c < DV; c += 32) {
                    uint32_t o[32];
                    tmem_ld32_nowait(o_addr + c, o);
                    tmem_wait_ld();
                    if (valid) {
#pragma unroll
                        for (int k = 0; k < 32; k += 8) {
                            uint4 w;
                            w.x = pack_bf16(__uint_as_float(o[k]) * inv, __uint_as_float(o[k + 1]) * inv);
                            w.y = pack_bf16(__uint_as_float(o[k + 2]) * inv, __uint_as_float(o[k + 3]) * inv);
                            w.z = pack_bf16(__uint_as_float(o[k + 4]) * inv, __uint_as_float(o[k + 5]) * inv);
                            w.w = pack_bf16(__uint_as_float(o[k + 6]) * inv, __uint_as_float(o[k + 7]) * inv);
                            *reinterpret_cast<uint4*>(orow + c + k) = w;
                        }
                    }
                }
            }
        }
    }
    }
    if (lane == 0 && warp < K_WARP) TW_TRACE_AT(warp, TRACE_TILES - 1, 1);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_dealloc(tmem_base, TMEM_COLS);
    if (threadIdx.x == 0) TW_TRACE_AT(11, 0, 7);
}

}  // namespace

TW_EXPORT int tw_attn_tc5_head_dim() { return D; }

#ifdef TW_TRACE
TW_EXPORT int tw_attn_tc5_trace_ptr(long long** ptr, int* roles, int* tiles, int* slots) {
    *roles = TRACE_ROLES; *tiles = TRACE_TILES; *slots = TRACE_SLOTS;
    return (int)cudaGetSymbolAddress((void**)ptr, g_trace);
}
#endif

// Whether the kernel takes this page size: a key tile is a whole number of pages, or a page a
// whole number of key tiles, and a tile has at most 32 boxes.
TW_EXPORT int tw_attn_prefill_tc5_supported(int page_size) {
    if (page_size < 4) return 0;
    return (BN % page_size == 0 || page_size % BN == 0) ? 1 : 0;
}

// 1 if the compiler gave the kernel the registers that its roles are split from, 0 if not (the shape belongs to the mma.sync kernel then),
// a negative number if the driver could not say.
TW_EXPORT int tw_attn_prefill_tc5_built() { return tw_registers_are<attn_prefill_tc5_kernel>(LAUNCH_REGS); }

// Attention for the requests of the batch that bring several tokens (with skip_single, requests
// with one token are left to the decode kernel).  q [tokens, Hq * D] and out [tokens, Hq * D] are
// bf16 with 16-byte aligned rows; the cache is [pages, Hkv, page_size, D] bf16 (values and out: heads of DV).  `row_tiles`: the sum of
// ceil(rows x Hq / Hkv / 256) over the requests that are served, where the caller knows it, else 0.  `ready` (or null; with
// skip_single): a word that tw_attn_decode_tma is given next, see tw_say_ready.
TW_EXPORT int tw_attn_prefill_tc5(void* out, int out_stride, const void* q, int q_stride, const int* seq_q_start,
                                  const int* seq_q_len, const int* seq_kv_len, const int* seq_slot,
                                  const int* block_table, int table_stride, const void* k_cache, const void* v_cache,
                                  int n_seqs, int max_q_len, int Hq, int Hkv, int page_size, int num_pages, int window,
                                  float scale, int skip_single, const float* gate, int row_tiles, int* status, int* ready,
                                  cudaStream_t stream) {
    if (n_seqs <= 0 || max_q_len <= 0) return 0;
    if (Hkv <= 0 || Hq % Hkv || !tw_attn_prefill_tc5_supported(page_size) || scale <= 0.f) return (int)cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(q) & 15) || (out_stride & 7) || (q_stride & 7) ||
        (reinterpret_cast<uintptr_t>(k_cache) & 15) || (reinterpret_cast<uintptr_t>(v_cache) & 15))
        return (int)cudaErrorMisalignedAddress;
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc5_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        const int built = tw_attn_prefill_tc5_built();
        if (built != 1) return built < 0 ? -built : (int)cudaErrorInvalidConfiguration;
        attr_set = true;
    }
    const int box_rows = page_size < BN ? page_size : BN;
    const long long rows = (long long)num_pages * Hkv * page_size;
    if (rows >= (1ll << 31) - 1) return (int)cudaErrorInvalidValue;
    CUtensorMap mk, mv;
    if (int e = get_map(k_cache, rows, D, box_rows, &mk)) return e;
    if (int e = get_map(v_cache, rows, DV, box_rows, &mv)) return e;
    const int G = Hq / Hkv;
    const bool counted = row_tiles > 0;
    const long long blocks = (long long)(counted ? row_tiles : (max_q_len * G + NQ * BM - 1) / (NQ * BM)) * Hkv;
    if (blocks > 0x7fffffffll || (!counted && n_seqs > 65535)) return (int)cudaErrorInvalidValue;
    dim3 grid((unsigned)blocks, counted ? 1 : n_seqs);
    return tw_launch(attn_prefill_tc5_kernel, grid, dim3(THREADS), (size_t)SMEM, stream, 1, mk, mv, (bf16*)out, out_stride,
                     (const bf16*)q, q_stride, seq_q_start, seq_q_len, seq_kv_len, seq_slot, block_table, table_stride,
                     Hq, Hkv, page_size, num_pages, window, scale * 1.4426950408889634f, skip_single, gate, status, counted ? n_seqs : 0, ready);
}
